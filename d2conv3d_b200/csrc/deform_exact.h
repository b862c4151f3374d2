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
  // the channels-last kernels address a clip in 31 bits
  return !one_d && g.Cin >= kMinChannelsCl && g.Vin * g.Cin <= 0x7fffffffLL ? kChannelsLast : kDirect;
}

// Output channels of a block tile.
template <typename T>
inline int tile_n(const Geom& g) { return g.cout_g <= 32 ? 32 : (g.cout_g <= 64 || sizeof(T) == 8 ? 64 : 128); }

template <typename T>
inline size_t x_cl_bytes(const Geom& g) { return align_up(sizeof(T) * (size_t)g.B * g.Vin * g.Cin, 256); }
template <int TN> constexpr int kPitchB = TN + 4;     // row pitch of a B tile in elements
template <typename T> constexpr int kDcolN = sizeof(T) == 4 ? 128 : 64;      // column rows of a gradient-column tile

// Staged weights: B-tile images of 16 x (columns + 4) elements.
template <typename T>
inline size_t w_image_bytes(const Geom& g, int rows, int cols, int tn) {
  return align_up(sizeof(T) * (size_t)g.groups * ((cols + tn - 1) / tn) * align_up((size_t)rows, kTK) * (tn + 4), 256);
}
template <typename T>
inline size_t w_fwd_bytes(const Geom& g) { return w_image_bytes<T>(g, g.cin_g * g.K, g.cout_g, tile_n<T>(g)); }
template <typename T>
inline size_t w_bwd_bytes(const Geom& g) { return w_image_bytes<T>(g, g.cout_g, g.cin_g * g.K, kDcolN<T>); }

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
