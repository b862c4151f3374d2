// Exact-tier kernels in double (a translation unit per type: they compile side by side).
#include "deform_exact.cuh"

namespace d2c {
namespace exact {

#define D2C_EXACT(Coords, FieldOut)                                                                                            \
  template int launch_fwd<double, Coords<double>>(const Geom&, const Coords<double>&, const double*, const double*, const double*, const double*, \
                                            double*, void*, cudaStream_t);                                                        \
  template int launch_bwd<double, Coords<double>, FieldOut>(const Geom&, const Coords<double>&, const double*, const double*, const double*,   \
                                                      const double*, double*, double*, size_t, double*, double*, double*, void*,               \
                                                      unsigned long long, cudaStream_t);
D2C_EXACT(OffsetCoords, false)
D2C_EXACT(FieldCoords, true)
D2C_EXACT(Offset1dCoords, false)
#undef D2C_EXACT

}  // namespace exact
}  // namespace d2c
