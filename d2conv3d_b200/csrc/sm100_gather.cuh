// Sampling records and the gather producer shared by the tensor-core forward, the weight-gradient and
// the sampling-gradient kernels.
//
// Everything that depends only on (clip, offset group, tap, output voxel) -- the sampling position exactly
// as the reference forms it (integer base converted once + offset, one fp add; csrc/ops/dconv3d_gpu.cu:192-194,
// or the dilation-field synthesis of utils/grid.py:97), its floor corners, which corners are readable, the
// eight trilinear weights and the modulation value -- is computed ONCE per call by sample_records_kernel with
// the same make_sample() as every other kernel (so integer corners stay bit-identical across tiers), and the
// inner loops of the consumers contain no integer division, no strided offset read and no weight arithmetic.
//
// Two record streams, both [B][G][K][V]:
//   pos  float4 {z, y, x, mask}                                    -> sampling-gradient kernel
//   gat  3 x uint4 (48 B): {voff, steps, -, -}, w0..w3, w4..w7      -> gather producers (forward, dW)
//        voff  = element offset (no channel term) of the CLAMPED corner 000 inside the clip's channels-last
//                staging: per axis the floor index if it is inside the volume, else the ceil index if that is,
//                else 0
//        steps = bit 0/1/2 set when the x/y/z neighbour (+1) exists AND the floor index is inside, i.e. when
//                corner 1 of that axis is a different, readable voxel; otherwise both corners of the axis read
//                the same (readable) voxel;
//                bit 3 + j set when corner j has a weight other than zero
//        wj    = half2 {a_j*mask, a_j*mask}: trilinear weight x modulation, rounded to fp16, duplicated; ZERO
//                for every corner that does not contribute to the forward sample.  fp32 a_j*mask in
//                the fp32-parity mode
// A dilation field gives all offset groups the same positions: with more than one group its forward takes the record once per
// (clip, tap, voxel), with the plain weights, and the activated modulation separately (fp32 [B][G][K][V padded to 4]), which the
// producer multiplies the blended sample by.  Eight groups: 80 instead of 384 bytes written and read per tap and voxel.
// A producer reads only the corners that weigh anything and blends all eight, the others as zero: zero times their weight, where
// what a register held before may be a NaN of another voxel, tile or clip.  The 16-byte gathers clear a register before each
// load (256 channels in 8 groups on 2 x 8 x 60 x 107, bf16: weight gradient that gathers 0.97 ms; 1.19 with registers that kept
// their contents from item to item, which spilled).  The forward, whose 32-byte gathers have a register file's worth in flight,
// clears them only where the staged input holds a NaN (deform_sm100_fwd_kernel.cuh).
// Corners of zero weight are those outside the volume and, for a dilation field, the upper neighbour along every axis on which
// the tap sits at the kernel's centre: 4.6 corners a tap instead of 8 with 3 x 3 x 3 taps.  Leaving them out took the forward of
// such a layer, 256 channels on 2 x 8 x 60 x 107, from 2.71 to 2.27 ms (1.85 now) and, with free offsets, where they are the corners
// outside the volume, 512 channels on 2 x 8 x 30 x 54 from 1.68 to 1.55 ms (1.32 now).
#pragma once

#include <cuda_fp16.h>

#include "d2c_common.cuh"
#include "sm100_ptx.cuh"

namespace d2c {
namespace {

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// Row of the separate modulation values: 16-byte copies of any tile start on a boundary.
__host__ __device__ inline int mask_row(int V) { return (V + 3) / 4 * 4; }

// kShared: the coordinates do not depend on the offset group (dilation field): a thread serves one (voxel, tap)
// and all groups, computing the position, corners and weights once and applying each group's modulation.
// nan_flag (nullable): cleared for the staging of x, which sets it when this kernel is done (stage_input_cl_kernel).
template <typename Coords, bool kShared>
static __global__ void __launch_bounds__(256)
sample_records_kernel(Geom g, Coords coords, const float* __restrict__ mask, long long mask_bstride, int mask_act,
                      float4* __restrict__ pos, uint4* __restrict__ gat, int f32_weights, float* __restrict__ masks,
                      int* __restrict__ nan_flag) {
  next_kernel_may_start();
  const int v = blockIdx.x * 256 + threadIdx.x;
  if (nan_flag && v == 0 && blockIdx.y == 0 && blockIdx.z == 0) *nan_flag = 0;
  if (v >= g.V) return;
  const int tap = kShared ? blockIdx.y : blockIdx.y % g.K, b = blockIdx.z;
  const int grp_beg = kShared ? 0 : blockIdx.y / g.K, grp_end = kShared ? g.G : grp_beg + 1;
  int bz, by, bx;
  voxel_tap_base(g, v, tap, bz, by, bx);
  float z, y, x;
  coords.get(g, b, grp_beg, tap, v, bz, by, bx, z, y, x);
  const Sample<float> s = make_sample(g, z, y, x);
  float a[8];
  sample_weights(s, a);
  const unsigned valid = s.inside ? s.valid : 0u;
  int cz, cy, cx;
  unsigned steps = 0;
  {
    const bool z0ok = s.z0 >= 0 && s.z0 < g.D, z1ok = s.z0 + 1 >= 0 && s.z0 + 1 < g.D;
    const bool y0ok = s.y0 >= 0 && s.y0 < g.H, y1ok = s.y0 + 1 >= 0 && s.y0 + 1 < g.H;
    const bool x0ok = s.x0 >= 0 && s.x0 < g.W, x1ok = s.x0 + 1 >= 0 && s.x0 + 1 < g.W;
    cz = z0ok ? s.z0 : (z1ok ? s.z0 + 1 : 0);
    cy = y0ok ? s.y0 : (y1ok ? s.y0 + 1 : 0);
    cx = x0ok ? s.x0 : (x1ok ? s.x0 + 1 : 0);
    steps = (x0ok && x1ok ? 1u : 0u) | (y0ok && y1ok ? 2u : 0u) | (z0ok && z1ok ? 4u : 0u);
  }
  const int voff = ((cz * g.H + cy) * g.W + cx) * g.Cin;
  for (int grp = grp_beg; grp < grp_end; ++grp) {
    const long long i = (((long long)b * g.G + grp) * g.K + tap) * g.V + v;
    // the mask as the op receives it, or the predictor's logits read in place and activated here
    const float m = mask ? mask_act_value(mask_act, __ldg(mask + (mask_bstride ? (long long)b * mask_bstride +
                                                          ((long long)grp * g.K + tap) * g.V + v : i)))
                         : 1.f;
    if (pos) pos[i] = make_float4(z, y, x, m);
    if (masks) masks[(((long long)b * g.G + grp) * g.K + tap) * mask_row(g.V) + v] = m;
    if (gat && (!masks || grp == grp_beg)) {
      uint4* o = gat + 3 * (masks ? ((long long)b * g.K + tap) * g.V + v : i);
      const float m_w = masks ? 1.f : m;
      if (f32_weights) {
        // fp32-parity mode: the 48 bytes hold the eight products a_j*mask in fp32
        uint32_t f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = ((valid >> j) & 1u) ? __float_as_uint(a[j] * m_w) : 0u;
        uint32_t weighs = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) weighs |= (f[j] << 1) ? 8u << j : 0u;      // +-0 alike
        o[0] = make_uint4((uint32_t)voff, steps | weighs, 0u, 0u);
        o[1] = make_uint4(f[0], f[1], f[2], f[3]);
        o[2] = make_uint4(f[4], f[5], f[6], f[7]);
      } else {
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = ((valid >> j) & 1u) ? h2_bits(__float2half2_rn(a[j] * m_w)) : 0u;
        uint32_t weighs = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) weighs |= (w[j] & 0x7fffu) ? 8u << j : 0u;
        o[0] = make_uint4((uint32_t)voff, steps | weighs, 0u, 0u);
        o[1] = make_uint4(w[0], w[1], w[2], w[3]);
        o[2] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
  }
}

template <typename Coords>
struct CoordsSharedAcrossGroups { static constexpr bool value = false; };
template <typename T>
struct CoordsSharedAcrossGroups<FieldCoords<T>> { static constexpr bool value = true; };

template <typename Coords>
static int launch_sample_records(const Geom& g, const Coords& coords, const float* mask, const HeadCfg& head, float4* pos,
                                 uint4* gat, cudaStream_t st, bool f32_weights = false, float* masks = nullptr, int* nan_flag = nullptr) {
  constexpr bool kShared = CoordsSharedAcrossGroups<Coords>::value;
  dim3 grid((unsigned)((g.V + 255) / 256), (unsigned)(kShared ? g.K : g.G * g.K), (unsigned)g.B);
  if (grid.y > 65535 || grid.z > 65535) return D2C_ERR_TOO_LARGE;
  sample_records_kernel<Coords, kShared><<<grid, 256, 0, st>>>(g, coords, mask, head.mask_bstride, head.mask_act, pos, gat,
                                                              f32_weights ? 1 : 0, masks, nan_flag);
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

inline size_t pos_records_bytes(const Geom& g) {
  return align_up((size_t)g.B * g.G * g.K * g.V * sizeof(float4), 256);
}
inline size_t gather_records_bytes(const Geom& g) {
  return align_up((size_t)g.B * g.G * g.K * g.V * 3 * sizeof(uint4), 256);
}

// Element strides of the channels-last staging of x within one clip.
struct ClStrides {
  int dz, dy, dx;   // H*W*Cin, W*Cin, Cin
};

// One A-tile item = the 8 channels [ch0, ch0+8) of one modulated trilinear sample, blended in packed fp16
// (the weights already carry the modulation), converted to bf16 and stored (16 bytes) in the swizzled A tile.
// The work is split in two so that a producer can put the corners of several items in flight before the first
// blend: load_corners issues the corner loads of one item (those that weigh anything, see the record format above),
// blend_store consumes them.   xb_ch: channels-last fp16 staging of the clip, advanced to the item's channel.
__device__ __forceinline__ void load_corners(const __half* __restrict__ xb_ch, ClStrides cs, uint32_t voff,
                                             uint32_t steps, uint4 (&c)[8]) {
  const int dx = (steps & 1u) ? cs.dx : 0, dy = (steps & 2u) ? cs.dy : 0, dz = (steps & 4u) ? cs.dz : 0;
  const __half* p0 = xb_ch + voff;
  const __half* p1 = p0 + dz;
  ptx::ldg_nc_v4_or_zero(c[0], p0, steps & 8u);
  ptx::ldg_nc_v4_or_zero(c[1], p0 + dx, steps & 16u);
  ptx::ldg_nc_v4_or_zero(c[2], p0 + dy, steps & 32u);
  ptx::ldg_nc_v4_or_zero(c[3], p0 + dy + dx, steps & 64u);
  ptx::ldg_nc_v4_or_zero(c[4], p1, steps & 128u);
  ptx::ldg_nc_v4_or_zero(c[5], p1 + dx, steps & 256u);
  ptx::ldg_nc_v4_or_zero(c[6], p1 + dy, steps & 512u);
  ptx::ldg_nc_v4_or_zero(c[7], p1 + dy + dx, steps & 1024u);
}

// Returns the 16 bytes it stored (a caller that also keeps the samples for the backward writes them to global).
__device__ __forceinline__ uint4 blend_store(const uint4 (&c)[8], uint4 w03, uint4 w47, uint32_t dst) {
  const uint32_t w[8] = {w03.x, w03.y, w03.z, w03.w, w47.x, w47.y, w47.z, w47.w};
  __half2 acc[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = __float2half2_rn(0.f);
#pragma unroll
  for (int j = 0; j < 8; ++j) {   // corner order 000..111, as the reference's interpolation chain
    const __half2 wj = bits_h2(w[j]);
    acc[0] = __hfma2(bits_h2(c[j].x), wj, acc[0]);
    acc[1] = __hfma2(bits_h2(c[j].y), wj, acc[1]);
    acc[2] = __hfma2(bits_h2(c[j].z), wj, acc[2]);
    acc[3] = __hfma2(bits_h2(c[j].w), wj, acc[3]);
  }
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __half22float2(acc[e]);
    o[e] = ptx::pack_bf16x2(f.x, f.y);
  }
  const uint4 out = make_uint4(o[0], o[1], o[2], o[3]);
  ptx::sts_v4(dst, out);
  return out;
}

// ---- fp32-parity mode ("bf16x3"): fp32 staging, fp32 blend, bf16 hi/lo split -------------------------------
// One item = 4 channels (16 bytes of fp32) of one sample.  The blended value v is written twice into the
// 128-byte A row of a 32-channel unit: hi = bf16(v) at channel column c, lo = bf16(v - hi) at column 32 + c,
// so that the MMA issuer can form a_hi*b_hi + a_lo*b_hi + a_hi*b_lo from K sub-blocks of ONE tile pair.
__device__ __forceinline__ void load_corners_f32(const float* __restrict__ xb_ch, ClStrides cs, uint32_t voff,
                                                 uint32_t steps, uint4 (&c)[8]) {
  const int dx = (steps & 1u) ? cs.dx : 0, dy = (steps & 2u) ? cs.dy : 0, dz = (steps & 4u) ? cs.dz : 0;
  const float* p0 = xb_ch + voff;
  const float* p1 = p0 + dz;
  ptx::ldg_nc_v4_or_zero(c[0], p0, steps & 8u);
  ptx::ldg_nc_v4_or_zero(c[1], p0 + dx, steps & 16u);
  ptx::ldg_nc_v4_or_zero(c[2], p0 + dy, steps & 32u);
  ptx::ldg_nc_v4_or_zero(c[3], p0 + dy + dx, steps & 64u);
  ptx::ldg_nc_v4_or_zero(c[4], p1, steps & 128u);
  ptx::ldg_nc_v4_or_zero(c[5], p1 + dx, steps & 256u);
  ptx::ldg_nc_v4_or_zero(c[6], p1 + dy, steps & 512u);
  ptx::ldg_nc_v4_or_zero(c[7], p1 + dy + dx, steps & 1024u);
}

// w: the eight fp32 products a_j*mask (corner order 000..111, the reference's interpolation chain).
// dst_hi / dst_lo: shared-memory addresses of the 8-byte hi and lo slots of this item.
// Returns {hi (8 bytes), lo (8 bytes)} as stored.
__device__ __forceinline__ uint4 blend_split_store(const uint4 (&c)[8], const float (&w)[8], uint32_t dst_hi,
                                                   uint32_t dst_lo) {
  float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[0] = __fmaf_rn(__uint_as_float(c[j].x), w[j], v[0]);
    v[1] = __fmaf_rn(__uint_as_float(c[j].y), w[j], v[1]);
    v[2] = __fmaf_rn(__uint_as_float(c[j].z), w[j], v[2]);
    v[3] = __fmaf_rn(__uint_as_float(c[j].w), w[j], v[3]);
  }
  const uint32_t h01 = ptx::pack_bf16x2(v[0], v[1]), h23 = ptx::pack_bf16x2(v[2], v[3]);
  const uint32_t l01 = ptx::pack_bf16x2(v[0] - ptx::bf16_lo(h01), v[1] - ptx::bf16_hi(h01));
  const uint32_t l23 = ptx::pack_bf16x2(v[2] - ptx::bf16_lo(h23), v[3] - ptx::bf16_hi(h23));
  ptx::sts_v2(dst_hi, make_uint2(h01, h23));
  ptx::sts_v2(dst_lo, make_uint2(l01, l23));
  return make_uint4(h01, h23, l01, l23);
}

}  // namespace
}  // namespace d2c
