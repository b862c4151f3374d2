// Exact-tier kernels in float (a translation unit per type: they compile side by side).
#include "deform_exact.cuh"

namespace d2c {
namespace exact {

#define D2C_EXACT(Coords, FieldOut)                                                                                            \
  template int launch_fwd<float, Coords<float>>(const Geom&, const Coords<float>&, const float*, const float*, const float*, const float*, \
                                            float*, void*, cudaStream_t);                                                        \
  template int launch_bwd<float, Coords<float>, FieldOut>(const Geom&, const Coords<float>&, const float*, const float*, const float*,   \
                                                      const float*, float*, float*, size_t, float*, float*, float*, void*,               \
                                                      unsigned long long, cudaStream_t);
D2C_EXACT(OffsetCoords, false)
D2C_EXACT(FieldCoords, true)
D2C_EXACT(Offset1dCoords, false)
#undef D2C_EXACT

}  // namespace exact
}  // namespace d2c
