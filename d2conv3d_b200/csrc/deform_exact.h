// Exact tier of the deformable convolutions (deform_exact.cuh): entry points and workspace sizes.
#pragma once

#include "d2c_common.cuh"

namespace d2c {
namespace exact {

constexpr int kTK = 16;            // contraction rows per step
constexpr int kMinChannelsCl = 16; // fewer channels than this fill less than two sectors of a staged voxel

// Where samples come from: a channels-last copy of x, x itself four channels at a time, x itself row by row (channel
// counts per group that four does not divide).
enum Route { kChannelsLast = 0, kDirect = 1, kAny = 2 };

inline Route route_of(const Geom& g, bool one_d) {
  if (g.cpg % 4 || g.cin_g % 4) return kAny;
  return !one_d && g.Cin >= kMinChannelsCl ? kChannelsLast : kDirect;
}

// Output channels of a block tile.
template <typename T>
inline int tile_n(const Geom& g) { return g.cout_g <= 32 ? 32 : (g.cout_g <= 64 || sizeof(T) == 8 ? 64 : 128); }

template <typename T>
inline size_t x_cl_bytes(const Geom& g) { return align_up(sizeof(T) * (size_t)g.B * g.Vin * g.Cin, 256); }
template <typename T>
inline size_t w_fwd_bytes(const Geom& g) {
  return align_up(sizeof(T) * (size_t)g.groups * align_up((size_t)g.cin_g * g.K, kTK) * align_up(g.cout_g, tile_n<T>(g)), 256);
}
template <typename T>
inline size_t w_bwd_bytes(const Geom& g) {
  return align_up(sizeof(T) * (size_t)g.groups * align_up(g.cout_g, kTK) * align_up((size_t)g.cin_g * g.K, 128), 256);
}

// Clips per backward slice under the intermediate-element cap.
inline int slice_clips(const Geom& g, unsigned long long cap) {
  const unsigned long long per = (unsigned long long)g.Cin * g.K * g.V;
  unsigned long long nb = per ? cap / per : 1;
  if (nb < 1) nb = 1;
  if (nb > (unsigned long long)g.B) nb = g.B;
  return (int)nb;
}

template <typename T>
inline size_t fwd_workspace(const Geom& g) {
  return route_of(g, false) == kChannelsLast ? x_cl_bytes<T>(g) + w_fwd_bytes<T>(g) : 0;
}
template <typename T>
inline size_t bwd_workspace(const Geom& g, unsigned long long cap) {
  const size_t dcol = align_up(sizeof(T) * (size_t)slice_clips(g, cap) * g.Cin * g.K * g.V, 256);
  return dcol + (route_of(g, false) == kChannelsLast ? 2 * x_cl_bytes<T>(g) + w_bwd_bytes<T>(g) : 0);
}

// Instantiated for float and double (deform_exact_f32.cu, deform_exact_f64.cu) and the three coordinate sources.  The 1-D
// source needs no workspace in the forward.  FieldOut: grad_coord is the dilation field's gradient.
template <typename T, typename Coords>
int launch_fwd(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* w, const T* bias, T* y, void* ws,
               cudaStream_t st);
template <typename T, typename Coords, bool FieldOut>
int launch_bwd(const Geom& g, const Coords& coords, const T* gy, const T* x, const T* mask, const T* w, T* grad_x, T* grad_coord,
               size_t grad_coord_elems, T* grad_mask, T* grad_w, T* grad_bias, void* ws, unsigned long long cap, cudaStream_t st);

}  // namespace exact
}  // namespace d2c
