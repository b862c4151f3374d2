// Sampling gradient of the tensor-core tier: grad_input, grad_offset (or the gradient of the dilation field) and grad_mask from
// the gradient columns, with the contributions to a voxel of the input added up in the block before they leave it.
//
// Replaces deformable_col2im_coord_gpu_kernel (csrc/ops/dconv3d_gpu.cu:756-864) and deformable_col2im_gpu_kernel (:562-643).
#pragma once

#include <type_traits>

#include "sm100_gather.cuh"

namespace d2c {
namespace {

// Order in which the blocks walk a clip's output voxels.  Position i is voxel at(i): slabs of bz frames, in them strips of by
// rows, along a strip bricks of 8 columns, in a brick row by row.  The last slab, strip and brick are as small as the volume
// leaves them, without padding.  Neighbouring positions are neighbours along every axis, and what they sample overlaps.
struct VoxelOrder {
  int D, H, W, bz, by;
  __host__ __device__ __forceinline__ int at(int i) const {
    const unsigned slab = (unsigned)(bz * H * W);
    const unsigned zb = (unsigned)i / slab;
    unsigned r = (unsigned)i - zb * slab;
    const unsigned dz = (unsigned)(D - (int)zb * bz < bz ? D - (int)zb * bz : bz);
    const unsigned strip = dz * (unsigned)(by * W);
    const unsigned yb = r / strip;
    r -= yb * strip;
    const unsigned dy = (unsigned)(H - (int)yb * by < by ? H - (int)yb * by : by);
    const unsigned brick = dz * dy * 8u;
    const unsigned xb = r / brick;
    r -= xb * brick;
    const unsigned wx = (unsigned)(W - (int)xb * 8 < 8 ? W - (int)xb * 8 : 8);
    const unsigned row = r / wx, x = xb * 8u + (r - row * wx);
    const unsigned zr = row / dy, z = zb * (unsigned)bz + zr, y = yb * (unsigned)by + (row - zr * dy);
    return (int)((z * (unsigned)H + y) * (unsigned)W + x);
  }
};
// Bricks of 4 rows of 8 columns, the 32 voxels of a block: 2 frames x 2 rows where there are two of each.
inline VoxelOrder voxel_order(const Geom& g) {
  VoxelOrder o{g.Do, g.Ho, g.Wo, g.Do > 1 ? 2 : 1, 0};
  o.by = 4 / o.bz < g.Ho ? 4 / o.bz : g.Ho;
  return o;
}

// Tap positions per dim of the dilation-field variant, by value (a kernel parameter: no copy to the device).
struct FieldAxes {
  float pos[3][kMaxFieldKernelDim];
};

constexpr int kSgVox = 32;             // output voxels of a block
constexpr int kSgThreads = 256;
constexpr int kSgMaxTaps = 27;         // taps of a block
constexpr int kSgRounds = (kSgVox * kSgMaxTaps + kSgThreads - 1) / kSgThreads;   // samples of a thread
constexpr int kSgCells = 8192;         // input voxels that a block keeps lists for

// Shared memory: per sample eight values (scatter weights, then the corner dot products; their sums apart where a group has several
// slices), {row of the gradient columns, offset of corner 000}, the list entries, and the 16-bit list starts of the cells.
inline size_t sample_grad_smem(int taps, int nh) {
  const size_t n = (size_t)kSgVox * taps;
  return n * (8 * 4 * (nh > 1 ? 2 : 1) + 8 + 8 * 2) + kSgCells * 2;
}

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  // volatile (must not be dropped) but no memory clobber: read-only loads may move across it
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d));
}
// Loads under a predicate; the register keeps its contents otherwise.
__device__ __forceinline__ void ldg_if(float4& r, const float* p, bool on) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "+f"(r.x), "+f"(r.y), "+f"(r.z), "+f"(r.w) : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ldg_if(uint2& r, const __half* p, bool on) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t@q ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t}"
      : "+r"(r.x), "+r"(r.y) : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void red_add_v4_if(float* addr, float4 v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n\t}"
               ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"((int)on));
}
__device__ __forceinline__ float4 to_f32(const float4& x) { return x; }
__device__ __forceinline__ float4 to_f32(const uint2& x) {
  const float2 lo = __half22float2(bits_h2(x.x)), hi = __half22float2(bits_h2(x.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
// acc += a * b where it counts (a weight of zero is no substitute: the columns may hold infinities)
__device__ __forceinline__ void fma_v4_if(float4& acc, const float4& a, const float4& b, bool on) {
  if (on) { acc.x += a.x * b.x; acc.y += a.y * b.y; acc.z += a.z * b.z; acc.w += a.w * b.w; }
}
// A load that is not merged with an earlier one of the same address.
__device__ __forceinline__ float4 ldg_again(const float4* p) {
  float4 r;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p));
  return r;
}

// Corners of a sample that are inside the volume and can matter.  A tap at the kernel's centre on an axis does not move along it, and
// no tap does where the field has no channel for the axis: the upper corners of that axis weigh nothing and the axis takes no
// gradient (with 3 x 3 x 3 taps 4.6 corners a tap instead of 8, and 2.8 where the field scales rows and columns alone; the latter, one
// group of 256 channels on 2 x 8 x 30 x 54: 531 us with the first of the two rules alone, 374 with both).
template <bool FieldOut>
__device__ __forceinline__ unsigned live_corners(const Geom& g, const Sample<float>& s, int tap, int3 field_ch, const FieldAxes& axes) {
  unsigned valid = s.valid;
  if constexpr (FieldOut) {
    const int kx = tap % g.kw, ky = (tap / g.kw) % g.kh, kz = tap / (g.kw * g.kh);
    if (valid) {
      if ((field_ch.x < 0 || axes.pos[0][kz] == 0.f) && !(s.gz < 1.f)) valid &= 0x0fu;
      if ((field_ch.y < 0 || axes.pos[1][ky] == 0.f) && !(s.gy < 1.f)) valid &= 0x33u;
      if ((field_ch.z < 0 || axes.pos[2][kx] == 0.f) && !(s.gx < 1.f)) valid &= 0x55u;
    }
  }
  return valid;
}
// Those that weigh something in the scatter (a corner at distance exactly 1 does not, dconv3d_gpu.cu:626-637).
__device__ __forceinline__ unsigned weighing_corners(const Sample<float>& s, unsigned valid) {
  return valid & (s.gz < 1.f ? 0xffu : 0x0fu) & (s.gy < 1.f ? 0xffu : 0x33u) & (s.gx < 1.f ? 0xffu : 0x55u);
}

// Which kernel takes a call's positions (below): asked of 256 records, evenly spread over the clips at hand, by one block of a kernel
// that runs before both.
struct PositionAsk {
  Geom g;
  const float4* recs;          // of the first clip at hand
  long long n_recs;            // 0: not asked
  VoxelOrder order;
  int taps;                    // of a block
  int field;
  int3 field_ch;
  FieldAxes field_axes;
  int* direct;                 // the answer
};
// Sums win where contributions meet and weigh something.  (us, sums / direct, two clips of 8 x 60 x 107 and one group of 256 channels
// unless it says otherwise; measured with each kernel taking all.)
//   offsets    few corners weigh: the direct kernel sends fewer, the lists are as long as ever.  All offsets zero (one corner of
//              eight) 2700 / 1620, whole along one axis (a half) 2980 / 2370, along none 2900 / 3470; single pass 2760 / 1390, 2860 /
//              2170, 2830 / 3320.  The line lies a little above a half.
//   fields     a field of ones over three axes (0.22 of the corners left) 2190 / 1740; over two (0.36) 1440 / 1680; so 0.3.  Groups of one
//              slice are not asked: there the lists win at 0.22 too (two groups of 64: 1110 / 1230).
//   scattered  contributions of a brick that rarely meet: two groups of 64 channels on 8 x 120 x 214, offsets of sigma 16 in the plane
//              and 0.5 across (13 cells a contribution) 4310 / 3720, sigma 8 (4) 3850 / 3840, sigma 4 3590 / 3870; the line at 7.
//   outside    the lists hold nothing for samples outside the volume, while the direct kernel reads every gradient column: 512
//              channels on 2 x 8 x 30 x 54, sigma 64, 270 / 1070.  So the direct kernel needs three quarters of the samples inside.
__device__ __forceinline__ bool direct_by_positions(const PositionAsk& q, const int* sums) {
  const Geom& g = q.g;
  const int n_in = sums[0], n = sums[1], n_weigh = sums[2];
  if (4 * n_in < 3 * kSgThreads) return false;
  if (q.field) return 10 * n_weigh <= 3 * n;
  if (16 * n_weigh <= 9 * n) return true;
  // cells of a brick's box (864 samples reach about 8 times their mean distance from end to end) against its contributions
  auto cells = [&](int size, int brick, int stride, int k, int dil, int spread) {
    const float ext = (float)((brick - 1) * stride + (k - 1) * dil + 2) + 8.f / (16.f * kSgThreads) * (float)spread;
    return fminf(ext, (float)size);
  };
  const float box = cells(g.D, q.order.bz, g.sd, g.kd, g.dd, sums[3]) * cells(g.H, q.order.by, g.sh, g.kh, g.dh, sums[4]) *
                    cells(g.W, 8, g.sw, g.kw, g.dw, sums[5]);
  return box > 7.f * (float)n * ((float)(kSgVox * q.taps) / (float)kSgThreads);
}
__device__ __forceinline__ void ask_positions(const PositionAsk& q) {
  __shared__ int sums[6];      // samples in the volume, their corners, those that weigh; |position - tap| in 1/16 voxel
  const Geom& g = q.g;
  if (threadIdx.x < 6) sums[threadIdx.x] = 0;
  __syncthreads();
  const long long i = (2 * (long long)threadIdx.x + 1) * q.n_recs / (2 * kSgThreads);
  const int v = (int)(i % g.V), tap = (int)(i / g.V % g.K);
  const float4 rec = __ldg(q.recs + i);
  const Sample<float> s = make_sample(g, rec.x, rec.y, rec.z);
  const unsigned valid = q.field ? live_corners<true>(g, s, tap, q.field_ch, q.field_axes) : s.valid;
  int base[3];
  voxel_tap_base(g, v, tap, base[0], base[1], base[2]);
  const float at[3] = {rec.x, rec.y, rec.z};
  int own[6] = {valid != 0, __popc(valid), __popc(weighing_corners(s, valid))};
#pragma unroll
  for (int d = 0; d < 3; ++d) own[3 + d] = (int)(16.f * fminf(fabsf(at[d] - (float)base[d]), 4096.f));
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int t = __reduce_add_sync(0xffffffffu, own[k]);
    if ((threadIdx.x & 31) == 0) atomicAdd(sums + k, t);
  }
  __syncthreads();
  if (threadIdx.x == 0) *q.direct = direct_by_positions(q, sums);
}

// How a call's sampling gradient is split, and which kernel may take it.
struct SampleGradPlan {
  dim3 grid;                   // voxels / 32, clips x groups, tap ranges
  int taps;                    // of a block
  bool lists, ask;             // may be sample_grad_taps_kernel's; the positions decide
};
// Asking costs a call 1 to 2 us (a launch that ends at once and the wait for it): from this many (32 voxels, tap, slice) on, about 30 us
// of kernel.  us of forward and backward kernels, not asked / asked (single pass):
//   offsets of two voxels   64 channels, 4 x 4 x 16 x 16 175 / 174 (155 / 155); 128, 8 x 15 x 27 240 / 242 (207 / 207); 256 in 4 groups
//                           there 388 / 390 (313 / 316); 128, 8 x 30 x 54 571 / 571 (455 / 456)
//   all offsets zero        180 / 168 (161 / 150); 233 / 216 (205 / 186); 374 / 352 (310 / 292), in one group 383 / 332 (322 / 264);
//                           546 / 495 (453 / 403)
constexpr long long kSgAskFrom = 2048;
// A block lists and adds up the contributions of 32 voxels; the more taps it has, the more of them meet.  Small volumes share
// the taps out over up to nine blocks, so that there are three for every multiprocessor, also for the kernels of which two fit on one
// (256 channels on 8 x 15 x 27: 107 us with three, six or twelve a multiprocessor; 64 channels on 4 x 16 x 16: 17.6 us with nine
// blocks, 19.5 with 14).
// Which kernel, by what the host knows (us, direct / sums; offsets of two voxels):
//   few taps           the lists' fixed cost, and little meets.  256 channels in 4 groups on 2 x 8 x 30 x 54, 1 tap 54 / 87, 3 taps 115 /
//                      133, 5 taps 179 / 182, 6 taps 215 / 209; fp16 staging, 6 taps 196 / 205, 7 taps 218 / 223, 8 taps 280 / 266.
//                      One group, 5 taps 160 / 154.  A field has fewer corners a tap: 1 tap 43 / 75, 3 taps 90 / 94 (one group 64
//                      / 61, groups of 32 channels 148 / 170), 5 taps 137 / 117 (groups of 32 channels 223 / 209).
//   few taps a block   64 channels on 4 x 16 x 16, 3 taps a block 16 / 19; on 8 x 16 x 16, 4 taps 31 / 27; 2 groups of 32 there, 7 taps 33 / 37.
//   strides            the voxels of a brick lie apart.  512 channels in 8 groups, 8 x 60 x 107 with stride 2 on every axis 970 / 1000 (fp16
//                      836 / 892), with stride 3 in the plane 454 / 502 (4 groups of 64).  Groups of several slices win with sums all the
//                      same (one of 256: 628 / 499).
//   32 channels a group, offsets: half the sums' gain for the same lists.  256 channels on 8 x 60 x 107 2310 / 2230, 9 taps on 2 x 8 x
//                      30 x 54 400 / 432, stride 2 there 625 / 681; fp16 staging 2110 / 2267, but 57 / 50 on 4 x 16 x 16, where the taps
//                      are shared out.
inline SampleGradPlan sample_grad_plan(const Geom& g, int nbc, int nh, bool field, bool f32x, bool narrow, int sm_count) {
  const long long vblocks = (long long)((g.V + kSgVox - 1) / kSgVox) * nbc * g.G;
  const int min_split = (g.K + kSgMaxTaps - 1) / kSgMaxTaps;
  long long split = (3LL * sm_count + vblocks - 1) / vblocks;
  const bool full = split == 1;
  if (split > 9) split = 9;
  if (split < min_split) split = min_split;
  if (split > g.K) split = g.K;
  SampleGradPlan p;
  p.taps = (g.K + (int)split - 1) / (int)split;
  p.grid = dim3((unsigned)((g.V + kSgVox - 1) / kSgVox), (unsigned)(nbc * g.G), (unsigned)((g.K + p.taps - 1) / p.taps));
  if (field) {
    p.lists = g.K >= (narrow ? 5 : 3);
  } else {
    p.lists = g.K >= (f32x || nh > 1 ? 5 : 8) && p.taps >= (narrow ? 8 : 4);
    if (nh == 1 && g.sd * g.sh * g.sw >= (narrow ? 2 : 8)) p.lists = false;
    if (narrow && (g.K < 16 || (!f32x && full))) p.lists = false;
  }
  p.ask = p.lists && (!field || nh > 1) && vblocks * g.K * nh >= kSgAskFrom;
  return p;
}

// Block = 32 output voxels (a brick) and up to 27 taps of one (clip, offset group).  A sample is one (voxel, tap); each of its
// corners inside the volume is a contribution: weight x gradient column is due to the input voxel there, and (gradient column .
// input) is due to the sample's coordinate and modulation gradients.
//   1  the block lists its contributions by input voxel ("cell"): count, start of each cell's list, entry;
//   2  groups of 8 lanes walk equal shares of the lists, a lane with 8 channels: the gradient columns of every entry are read, the
//      input only when the cell changes, the sum over a cell stays in registers and leaves as one reduction;
//   3  a thread per sample turns the eight corner sums into the gradients of offset (field) and modulation.
// Reducing every contribution into L2 by itself sends 8.15 GB for 512 channels in 8 groups on 2 x 8 x 30 x 54, offsets of two voxels:
// 1.20 ms at L2's rate of fp32 additions (6.8 TB/s, measured alone), 1.68 ms with the corners' loads and the products beside it.  A
// brick of 32 voxels and 27 taps meets the same input voxel 4.2 times, so that 1.9 GB of sums leave it and 2 GB of input are read
// instead of 8.15; what bounds it now are the instructions of step 2 (about 110 a warp for four entries) and the steps' barriers.
// Measured there: fp32 staging 1.68 -> 1.38 ms, fp16 staging 1.55 -> 1.35; field layer of one group of 256 channels on 2 x 8 x 60 x 107
// 2.16 -> 1.90; 32 channels a group there, one clip of 8 x 120 x 214, 9.1 -> 7.7; 256 channels in 4 groups, 4 x 16 x 16, 39.6 -> 37.1
// us.  Where it is slower, sample_grad_plan and direct_by_positions send the call to sample_grad_direct_kernel.  Not faster: a warp per
// entry with two channels a lane (35 instructions an entry), entries filled up so that none is out of range, the input read with every
// entry, three entries ahead, packed FMAs.
// Three blocks a multiprocessor with one entry ahead (80 registers) beat two blocks with two ahead, 1.38 to 1.43 ms; where a group has
// several slices shared memory allows two blocks, and the field's kernels would spill.
// kMulti: the offset group has several slices of 64 channels (nh > 1).
template <bool FieldOut, bool kF32X, bool kNarrow, bool kMulti>
__global__ void __launch_bounds__(kSgThreads, kMulti || FieldOut ? 2 : 3)
sample_grad_taps_kernel(Geom g, VoxelOrder order, ClStrides cs, int b0, int nh, const float4* __restrict__ recs,
                         const float* __restrict__ dcol, const void* __restrict__ x_cl_v, bool has_mask,
                         float* __restrict__ grad_coord, float* __restrict__ grad_mask, float* __restrict__ gx_cl,
                         int field_nch, int3 field_ch, const __grid_constant__ FieldAxes field_axes, int taps_per_block,
                         HeadCfg head, const int* __restrict__ direct) {
  extern __shared__ __align__(16) uint8_t sg_smem[];
  __shared__ int s_box[6], s_total, s_single, s_delta[8];
  if (direct) {                        // started beside sample_grad_direct_kernel, which is the other answer's
    wait_for_kernels_before();
    if (*direct) return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = blockIdx.y % g.G, bl = blockIdx.y / g.G, b = b0 + bl;
  const int tap_beg = blockIdx.z * taps_per_block, n_tap = min(g.K - tap_beg, taps_per_block);
  const int n_max = kSgVox * taps_per_block;
  uint32_t* cnt = reinterpret_cast<uint32_t*>(sg_smem);                       // two cells a word
  float* vals = reinterpret_cast<float*>(sg_smem + kSgCells * 2);             // [sample][corner]
  float* sums = kMulti ? vals + n_max * 8 : vals;
  int2* tab = reinterpret_cast<int2*>(sums + n_max * 8);                      // [sample]
  uint16_t* ent = reinterpret_cast<uint16_t*>(tab + n_max);                   // sample * 8 + corner, bit 14: weighs nothing, bit 15: first

  // ---- 1: lists.  Lane = voxel, a warp's samples are taps warp, warp + 8, ...
  const bool active = (int)blockIdx.x * kSgVox + lane < g.V;
  const int v = order.at(active ? (int)blockIdx.x * kSgVox + lane : g.V - 1);
  if (tid < 3) s_box[tid] = 0x7fffffff;
  else if (tid < 6) s_box[tid] = -1;
  else if (tid == 6) s_total = s_single = 0;
  else if (tid >= 8 && tid < 16) s_delta[tid - 8] = ((tid & 4) ? cs.dz : 0) + ((tid & 2) ? cs.dy : 0) + ((tid & 1) ? cs.dx : 0);
  const float4* recp = recs + (((long long)b * g.G + grp) * g.K + tap_beg) * g.V + v;
  unsigned corners[kSgRounds];         // bits 0-7: count, 8-15: weigh something, 16-23: in the box
  {
  float4 rec[kSgRounds];
#pragma unroll
  for (int k = 0; k < kSgRounds; ++k) {
    const int t = k * 8 + warp;
    rec[k] = t < n_tap ? __ldg(recp + (long long)t * g.V) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  {
    int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
#pragma unroll
    for (int k = 0; k < kSgRounds; ++k) {
      const int tap = tap_beg + k * 8 + warp;
      const Sample<float> s = make_sample(g, rec[k].x, rec[k].y, rec[k].z);
      unsigned valid = active && k * 8 + warp < n_tap ? s.valid : 0u;
      if constexpr (FieldOut) {          // live_corners, written out: as a call this kernel's code comes out up to 12 % slower
        const int kx = tap % g.kw, ky = (tap / g.kw) % g.kh, kz = tap / (g.kw * g.kh);
        if (valid) {
          if ((field_ch.x < 0 || field_axes.pos[0][kz] == 0.f) && !(s.gz < 1.f)) valid &= 0x0fu;
          if ((field_ch.y < 0 || field_axes.pos[1][ky] == 0.f) && !(s.gy < 1.f)) valid &= 0x33u;
          if ((field_ch.z < 0 || field_axes.pos[2][kx] == 0.f) && !(s.gx < 1.f)) valid &= 0x55u;
        }
      }
      corners[k] = valid;
      if (valid) {
        lo[0] = min(lo[0], max(s.z0, 0)); hi[0] = max(hi[0], min(s.z0 + 1, g.D - 1));
        lo[1] = min(lo[1], max(s.y0, 0)); hi[1] = max(hi[1], min(s.y0 + 1, g.H - 1));
        lo[2] = min(lo[2], max(s.x0, 0)); hi[2] = max(hi[2], min(s.x0 + 1, g.W - 1));
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int l = __reduce_min_sync(0xffffffffu, lo[d]), h = __reduce_max_sync(0xffffffffu, hi[d]);
      if (lane == 0) { atomicMin(&s_box[d], l); atomicMax(&s_box[3 + d], h); }
    }
  }
  __syncthreads();
  int bz = s_box[0], by = s_box[1], bx = s_box[2];
  int nz = s_box[3] - bz + 1, ny = s_box[4] - by + 1, nx = s_box[5] - bx + 1;
  if (s_box[3] < 0) { nz = ny = nx = 0; }
  // a box with more cells than there are lists is cut at both ends; what lies outside is a list of its own each
  bool cut = false;
  while ((long long)nz * ny * nx > kSgCells) {
    int& n = nx >= ny && nx >= nz ? nx : (ny >= nz ? ny : nz);
    int& at = nx >= ny && nx >= nz ? bx : (ny >= nz ? by : bz);
    const int less = (n + 3) / 4;
    at += less / 2;
    n -= less;
    cut = true;
  }
  const int words = (nz * ny * nx + 1) / 2;
  for (int i = tid; i < words; i += kSgThreads) cnt[i] = 0u;
  __syncthreads();

  int cell0[kSgRounds];                // of corner 000 (which need not be one)
  uint32_t place[kSgRounds][4];        // 16 bits a corner: its place in the cell's list
#pragma unroll
  for (int k = 0; k < kSgRounds; ++k) {
    if (k * 8 + warp >= n_tap) continue;
    const int i = k * kSgThreads + tid;
    const float4 rk = ldg_again(recp + (long long)(k * 8 + warp) * g.V);      // (held, it would spill)
    const Sample<float> s = make_sample(g, rk.x, rk.y, rk.z);
    const int cz = s.z0 - bz, cy = s.y0 - by, cx = s.x0 - bx;
    cell0[k] = (cz * ny + cy) * nx + cx;
    unsigned in = 0xffu;
    if (cut) {
      if ((unsigned)cz >= (unsigned)nz) in &= 0xf0u;
      if ((unsigned)(cz + 1) >= (unsigned)nz) in &= 0x0fu;
      if ((unsigned)cy >= (unsigned)ny) in &= 0xccu;
      if ((unsigned)(cy + 1) >= (unsigned)ny) in &= 0x33u;
      if ((unsigned)cx >= (unsigned)nx) in &= 0xaau;
      if ((unsigned)(cx + 1) >= (unsigned)nx) in &= 0x55u;
    }
    // scatter weights of the reference's col2im: (1-|z-zp|)(1-|y-yp|)(1-|x-xp|), corners at distance
    // exactly 1 excluded (dconv3d_gpu.cu:626-637)
    const float wz[2] = {sub_rn(1.f, s.fz), sub_rn(1.f, s.gz)};
    const float wy[2] = {sub_rn(1.f, s.fy), sub_rn(1.f, s.gy)};
    const float wx[2] = {sub_rn(1.f, s.fx), sub_rn(1.f, s.gx)};
    const unsigned weigh = corners[k] & (s.gz < 1.f ? 0xffu : 0x0fu) & (s.gy < 1.f ? 0xffu : 0x33u) & (s.gx < 1.f ? 0xffu : 0x55u);
    float w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      w[q] = (weigh >> q) & 1u ? mul_rn(mul_rn(wz[q >> 2], wy[(q >> 1) & 1]), wx[q & 1]) * rk.w : 0.f;
      uint32_t r = 0u;
      if ((corners[k] >> q) & 1u) {
        const int cell = cell0[k] + (q >> 2) * (ny * nx) + ((q >> 1) & 1) * nx + (q & 1), sh = (cell & 1) * 16;
        if ((in >> q) & 1u)
          r = (atomicAdd(&cnt[cell >> 1], 1u << sh) >> sh) & 0xffffu;
        else
          r = (uint32_t)atomicAdd(&s_single, 1);
      }
      if (q & 1) place[k][q >> 1] |= r << 16;
      else place[k][q >> 1] = r;
    }
    corners[k] |= (weigh << 8) | (in << 16);
    reinterpret_cast<float4*>(vals)[2 * i] = make_float4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<float4*>(vals)[2 * i + 1] = make_float4(w[4], w[5], w[6], w[7]);
    // (rows of a clip's columns: 31 bits of them would be 512 GB)
    tab[i] = make_int2(((kNarrow ? grp >> 1 : grp) * g.K + tap_beg + k * 8 + warp) * (kMulti ? nh : 1) * g.V + v,
                       ((s.z0 * g.H + s.y0) * g.W + s.x0) * g.Cin + grp * g.cpg);
  }
  __syncthreads();
  for (int base = warp * 32; base < words; base += kSgThreads) {
    const uint32_t c = base + lane < words ? cnt[base + lane] : 0u;
    const int first = (int)(c & 0xffffu), both = first + (int)(c >> 16);
    int incl = both;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    int start = 0;
    if (lane == 31) start = atomicAdd(&s_total, incl);
    start = __shfl_sync(0xffffffffu, start, 31) + incl - both;
    if (base + lane < words) cnt[base + lane] = (uint32_t)start | ((uint32_t)(start + first) << 16);
  }
  __syncthreads();
  const uint16_t* start = reinterpret_cast<const uint16_t*>(cnt);
#pragma unroll
  for (int k = 0; k < kSgRounds; ++k) {
    if (k * 8 + warp >= n_tap) continue;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if ((corners[k] >> q) & 1u) {
        const int r = (int)((place[k][q >> 1] >> ((q & 1) * 16)) & 0xffffu);
        const bool in = (corners[k] >> (16 + q)) & 1u;
        const int cell = cell0[k] + (q >> 2) * (ny * nx) + ((q >> 1) & 1) * nx + (q & 1);
        const int at = r + (in ? (int)start[cell] : s_total);
        ent[at] = (uint16_t)(((k * kSgThreads + tid) * 8 + q) | ((corners[k] >> (8 + q)) & 1u ? 0 : 0x4000) | (!in || r == 0 ? 0x8000 : 0));
      }
    }
  }
  }
  __syncthreads();

  // ---- 2: sums.  Lane j of a group owns channels [4j, 4j+4) and [32+4j, 32+4j+4) of a slice (kNarrow: [4j, 4j+4) of the offset
  // group's half of it), so that a warp's access covers whole 32-byte sectors.
  {
    const int n_ent = s_total + s_single;
    const int j = lane & 7, share = (n_ent + kSgThreads / 8 - 1) / (kSgThreads / 8);
    const int beg = min(n_ent, (tid >> 3) * share), end = min(n_ent, beg + share);
    using XT = typename std::conditional<kF32X, float, __half>::type;
    using XV = typename std::conditional<kF32X, float4, uint2>::type;        // four channels
    const long long slices = kNarrow ? (long long)(g.G / 2) * g.K : (long long)g.G * g.K * (kMulti ? nh : 1);
    constexpr int kParts = kNarrow ? 1 : 2;
    constexpr int kRing = kMulti || FieldOut ? 2 : 1;              // entries requested ahead
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    struct Item {
      uint32_t id;
      int off;                         // of the cell
      float w;
      float4 d[kParts];
      XV x[kParts];
    };
    for (int h = 0; h < (kMulti ? nh : 1); ++h) {
      const XT* xb = reinterpret_cast<const XT*>(x_cl_v) + (long long)b * g.Vin * g.Cin + h * 64 + j * 4;
      float* gxb = gx_cl + (long long)b * g.Vin * g.Cin + h * 64 + j * 4;
      const float* dp = dcol + ((long long)bl * slices + h) * g.V * 64 + (kNarrow ? (grp & 1) * 32 : 0) + j * 4;
      auto fetch = [&](int e, Item& it) {
        const bool in = e < end;
        it.id = 0x4000u;
        if (in) it.id = ent[e];
        if (e == beg && in) it.id |= 0x8000u;
        const int2 t = tab[(it.id >> 3) & 0x3ffu];
        it.off = t.y + s_delta[it.id & 7u];
        it.w = vals[it.id & 0x1fffu];
        const float* row = dp + (long long)t.x * 64;
#pragma unroll
        for (int i = 0; i < kParts; ++i) {
          ldg_if(it.d[i], row + 32 * i, in);
          ldg_if(it.x[i], xb + it.off + 32 * i, it.id & 0x8000u);
        }
      };
      float4 acc[kParts], xc[kParts];
#pragma unroll
      for (int i = 0; i < kParts; ++i) acc[i] = xc[i] = zero4;
      int cell = -1;
      auto take = [&](const Item& it) -> float {
        const bool first = it.id & 0x8000u, weighs = !(it.id & 0x4000u);
#pragma unroll
        for (int i = 0; i < kParts; ++i) {
          red_add_v4_if(gxb + cell + 32 * i, acc[i], first && cell >= 0);
          const float4 x = to_f32(it.x[i]);
          acc[i].x = first ? 0.f : acc[i].x; acc[i].y = first ? 0.f : acc[i].y;
          acc[i].z = first ? 0.f : acc[i].z; acc[i].w = first ? 0.f : acc[i].w;
          xc[i].x = first ? x.x : xc[i].x; xc[i].y = first ? x.y : xc[i].y;
          xc[i].z = first ? x.z : xc[i].z; xc[i].w = first ? x.w : xc[i].w;
        }
        cell = first ? it.off : cell;
        float4 dot = zero4;
#pragma unroll
        for (int i = 0; i < kParts; ++i) {
          fma_v4_if(acc[i], it.d[i], make_float4(it.w, it.w, it.w, it.w), weighs);
          fma_v4_if(dot, it.d[i], xc[i], true);
        }
        return (dot.x + dot.y) + (dot.z + dot.w);
      };
      Item a[kRing];
#pragma unroll
      for (int i = 0; i < kRing; ++i)
#pragma unroll
        for (int q = 0; q < kParts; ++q) { a[i].d[q] = zero4; a[i].x[q] = XV{}; }
#pragma unroll
      for (int i = 0; i < kRing; ++i) fetch(beg + i, a[i]);
#pragma unroll 1
      for (int e = beg; e < beg + share; e += 2) {     // the same count for all groups of a warp
        const uint32_t id0 = a[0].id;
        const float d0 = take(a[0]);
        fetch(e + kRing, a[0]);
        const uint32_t id = j & 1 ? a[kRing - 1].id : id0;
        const float d1 = take(a[kRing - 1]);
        fetch(e + kRing + 1, a[kRing - 1]);
        // both dot products over the group's 8 lanes: the even lanes end up with the first, the odd ones with the second
        float d = (j & 1 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, j & 1 ? d0 : d1, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        d += __shfl_xor_sync(0xffffffffu, d, 4);
        if (j < 2 && e + j < end) {
          if (kMulti && h > 0) d += sums[id & 0x1fffu];
          sums[id & 0x1fffu] = d;
        }
      }
#pragma unroll
      for (int i = 0; i < kParts; ++i) red_add_v4_if(gxb + cell + 32 * i, acc[i], cell >= 0);
    }
  }
  __syncthreads();

  // ---- 3: gradients of the sampling position and of the modulation
  float fsum[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < kSgRounds; ++k) {
    if (!active || k * 8 + warp >= n_tap) continue;
    const int i = k * kSgThreads + tid, tap = tap_beg + k * 8 + warp;
    const float4 rec = __ldg(recp + (long long)(k * 8 + warp) * g.V);
    const Sample<float> s = make_sample(g, rec.x, rec.y, rec.z);
    const float m = rec.w;
    const float4 lo = reinterpret_cast<const float4*>(sums)[2 * i], hi = reinterpret_cast<const float4*>(sums)[2 * i + 1];
    float G[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int q = 0; q < 8; ++q) G[q] = (corners[k] >> q) & 1u ? G[q] : 0.f;
    float wts[3];
    coord_weights(G, s, wts);    // linear in the corner values: applies to the channel-summed corners
    // head.*_bstride != 0: the gradients go into the gradient of the predictor's raw output (clip stride = all of
    // its channels), the mask's through the derivative of its activation (taken from the activated value m)
    if (has_mask && grad_mask) {
      float a[8];
      sample_weights(s, a);
      const long long ri = head.mask_bstride ? (long long)b * head.mask_bstride + ((long long)grp * g.K + tap) * g.V + v
                                             : (((long long)b * g.G + grp) * g.K + tap) * g.V + v;
      grad_mask[ri] = s.inside ? blend(G, a) * mask_act_slope(head.mask_act, m) : 0.f;
    }
    if constexpr (!FieldOut) {
      float* go = grad_coord + (head.geo_bstride ? (long long)b * head.geo_bstride + ((long long)grp * 3 * g.K + 3 * tap) * g.V + v
                                                 : (((long long)b * g.G + grp) * 3 * g.K + 3 * tap) * g.V + v);
      go[0] = m * wts[0];
      go[g.V] = m * wts[1];
      go[2 * (long long)g.V] = m * wts[2];
    } else {
      // the field's gradient sums over taps (and groups): taps are summed here, one atomic per group after
      const int kx = tap % g.kw, ky = (tap / g.kw) % g.kh, kz = tap / (g.kw * g.kh);
      fsum[0] += field_axes.pos[0][kz] * (m * wts[0]);
      fsum[1] += field_axes.pos[1][ky] * (m * wts[1]);
      fsum[2] += field_axes.pos[2][kx] * (m * wts[2]);
    }
  }
  if constexpr (FieldOut) {
    float* part = reinterpret_cast<float*>(cnt);       // [axis][thread]: the lists are done with
#pragma unroll
    for (int d = 0; d < 3; ++d) part[d * kSgThreads + tid] = fsum[d];
    __syncthreads();
    if (warp < 3 && active) {
      const int ch = warp == 0 ? field_ch.x : (warp == 1 ? field_ch.y : field_ch.z);
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += part[warp * kSgThreads + i * 32 + lane];
      if (ch >= 0)
        atomicAdd(grad_coord + (long long)b * (head.geo_bstride ? head.geo_bstride : (long long)field_nch * g.V) + (long long)ch * g.V + v, sum);
    }
  }
}

// The same without lists: every corner of every sample is read, and reduced into L2, by itself.  Eight threads a voxel, thread j with
// channels [4j, 4j + 4) and [32 + 4j, 32 + 4j + 4) of a slice (two lanes cover a 32-byte sector); the block walks its taps, the record
// and the gradient columns of the next tap requested before the present one is worked on.  Bound by L2's rate of fp32 additions where
// all corners weigh.  Voxels in storage order: in bricks, whose threads add to the same voxels at the same time, it is up to 15 % slower.
// Small volumes share the taps out as there (1024 voxels, 27 taps: 46.9 us with one block per 32 voxels, 10.6 with nine).
template <bool FieldOut, bool kF32X, bool kNarrow>
__device__ __forceinline__ void
sample_grad_direct(Geom g, ClStrides cs, int b0, int nh, const float4* __restrict__ recs,
                   const float* __restrict__ dcol, const void* __restrict__ x_cl_v, bool has_mask,
                   float* __restrict__ grad_coord, float* __restrict__ grad_mask, float* __restrict__ gx_cl,
                   int field_nch, int3 field_ch, const FieldAxes& field_axes, int taps_per_block,
                   HeadCfg head, unsigned blk_x, unsigned blk_y, unsigned blk_z) {
  const int j = threadIdx.x & 7;
  const int v = blk_x * kSgVox + (threadIdx.x >> 3);
  const int grp = blk_y % g.G, bl = blk_y / g.G;
  const int b = b0 + bl;
  const bool active = v < g.V;
  const int vc = active ? v : g.V - 1;                       // clamped: inactive threads load valid memory
  const long long S = kNarrow ? (long long)(g.G / 2) * g.K : (long long)g.G * g.K * nh;
  const float4* recp = recs + (((long long)b * g.G + grp) * g.K) * g.V + vc;
  // thread j owns channels [4j, 4j+4) and [32+4j, 32+4j+4) of a slice: one warp-wide 16-byte access then
  // covers whole 32-byte sectors (two lanes each), which halves the sector operations of the reductions
  const float* dp = kNarrow
      ? dcol + (((long long)bl * S + (long long)(grp >> 1) * g.K) * g.V + vc) * 64 + (grp & 1) * 32 + j * 4
      : dcol + (((long long)bl * S + (long long)grp * g.K * nh) * g.V + vc) * 64 + j * 4;
  const long long slice_stride = (long long)g.V * 64;
  using XT = typename std::conditional<kF32X, float, __half>::type;
  const XT* xb = reinterpret_cast<const XT*>(x_cl_v) + (long long)b * g.Vin * g.Cin;
  float* gxb = gx_cl + (long long)b * g.Vin * g.Cin;
  const int chbase = grp * g.cpg + j * 4;

  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float fsum[3] = {0.f, 0.f, 0.f};
  auto ld_cols = [&](const float* q, float4& a, float4& b) {
    a = __ldg(reinterpret_cast<const float4*>(q));
    b = kNarrow ? zero4 : __ldg(reinterpret_cast<const float4*>(q + 32));
  };
  const int tap_beg = blk_z * taps_per_block, tap_end = min(g.K, tap_beg + taps_per_block);
  float4 rec_n = __ldg(recp + (long long)tap_beg * g.V);
  float4 d0_n, d1_n;
  ld_cols(dp + (long long)tap_beg * nh * slice_stride, d0_n, d1_n);
  for (int tap = tap_beg; tap < tap_end; ++tap) {
    const float4 rec = rec_n;
    float4 d0 = d0_n, d1 = d1_n;
    if (tap + 1 < tap_end) {
      rec_n = __ldg(recp + (long long)(tap + 1) * g.V);
      ld_cols(dp + (long long)(tap + 1) * nh * slice_stride, d0_n, d1_n);
    }
    const float m = rec.w;
    const Sample<float> s = make_sample(g, rec.x, rec.y, rec.z);
    // scatter weights of the reference's col2im: (1-|z-zp|)(1-|y-yp|)(1-|x-xp|), corners at distance
    // exactly 1 excluded (dconv3d_gpu.cu:626-637)
    const float wz[2] = {sub_rn(1.f, s.fz), sub_rn(1.f, s.gz)};
    const float wy[2] = {sub_rn(1.f, s.fy), sub_rn(1.f, s.gy)};
    const float wx[2] = {sub_rn(1.f, s.fx), sub_rn(1.f, s.gx)};
    const bool okz[2] = {true, s.gz < 1.f}, oky[2] = {true, s.gy < 1.f}, okx[2] = {true, s.gx < 1.f};
    // (Not the field's dead corners where a thread has 4 channels of fp16: it issues its loads either way, a corner left out
    // reads the stand-in below, and finding out which to leave out costs it more than the cache hits give back.)
    const unsigned valid = active ? live_corners<FieldOut && (kF32X || !kNarrow)>(g, s, tap, field_ch, field_axes) : 0u;
    const int off0 = ((s.z0 * g.H + s.y0) * g.W + s.x0) * g.Cin + chbase;
    float G[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) G[q] = 0.f;
    for (int h = 0; h < nh; ++h) {
      if (h > 0) {
        ld_cols(dp + ((long long)tap * nh + h) * slice_stride, d0, d1);
      }
      // corner values of this thread's 8 channels ([4j, 4j+4) and [32+4j, 32+4j+4)), as loaded.  fp16 staging:
      // the loads are unconditional -- a corner outside the volume reads the clip's first voxel instead and its
      // dot product is discarded by a select after the slice loop (a select, so a non-finite stand-in cannot
      // leak); measured 0.13 ms per step faster than predicated loads.  fp32 staging: predicated loads (twice
      // the bytes per corner; fetching the stand-ins measured 0.08 ms slower).
      uint4 c[8], chi[kF32X ? 8 : 1];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int off_in = off0 + h * 64 + (q >> 2) * cs.dz + ((q >> 1) & 1) * cs.dy + (q & 1) * cs.dx;
        if constexpr (kF32X) {
          if ((valid >> q) & 1u) {
            c[q] = ptx::ldg_nc_v4(xb + off_in);
            chi[q] = kNarrow ? make_uint4(0u, 0u, 0u, 0u) : ptx::ldg_nc_v4(xb + off_in + 32);
          } else {
            c[q] = chi[q] = make_uint4(0u, 0u, 0u, 0u);
          }
        } else {
          const int off = ((valid >> q) & 1u) ? off_in : chbase + h * 64;
          const uint2 lo = ptx::ldg_nc_v2(xb + off);
          const uint2 hi = kNarrow ? make_uint2(0u, 0u) : ptx::ldg_nc_v2(xb + off + 32);
          c[q] = make_uint4(lo.x, lo.y, hi.x, hi.y);
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int dz = q >> 2, dy = (q >> 1) & 1, dx = q & 1;
        if constexpr (kF32X) {
          if constexpr (kNarrow)
            G[q] += d0.x * __uint_as_float(c[q].x) + d0.y * __uint_as_float(c[q].y) +
                    d0.z * __uint_as_float(c[q].z) + d0.w * __uint_as_float(c[q].w);
          else
            G[q] += d0.x * __uint_as_float(c[q].x) + d0.y * __uint_as_float(c[q].y) +
                    d0.z * __uint_as_float(c[q].z) + d0.w * __uint_as_float(c[q].w) +
                    d1.x * __uint_as_float(chi[q].x) + d1.y * __uint_as_float(chi[q].y) +
                    d1.z * __uint_as_float(chi[q].z) + d1.w * __uint_as_float(chi[q].w);
        } else {
          const float2 x0 = __half22float2(bits_h2(c[q].x)), x1 = __half22float2(bits_h2(c[q].y));
          const float2 x2 = __half22float2(bits_h2(c[q].z)), x3 = __half22float2(bits_h2(c[q].w));
          if constexpr (kNarrow)
            G[q] += d0.x * x0.x + d0.y * x0.y + d0.z * x1.x + d0.w * x1.y;
          else
            G[q] += d0.x * x0.x + d0.y * x0.y + d0.z * x1.x + d0.w * x1.y + d1.x * x2.x + d1.y * x2.y +
                    d1.z * x3.x + d1.w * x3.y;
        }
        if (((valid >> q) & 1u) && okz[dz] && oky[dy] && okx[dx]) {
          const float sw = mul_rn(mul_rn(wz[dz], wy[dy]), wx[dx]) * m;
          float* dst = gxb + (off0 + h * 64 + dz * cs.dz + dy * cs.dy + dx * cs.dx);
          red_add_v4(dst, sw * d0.x, sw * d0.y, sw * d0.z, sw * d0.w);
          if (!kNarrow) red_add_v4(dst + 32, sw * d1.x, sw * d1.y, sw * d1.z, sw * d1.w);
        }
      }
    }
    // channel reduction of the 8 corner dot-products across the voxel's 8 threads (corners outside: zero)
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (!kF32X) G[q] = ((valid >> q) & 1u) ? G[q] : 0.f;
      G[q] += __shfl_xor_sync(0xffffffffu, G[q], 1);
      G[q] += __shfl_xor_sync(0xffffffffu, G[q], 2);
      G[q] += __shfl_xor_sync(0xffffffffu, G[q], 4);
    }
    if (active && j == 0) {
      float wts[3];
      coord_weights(G, s, wts);    // linear in the corner values: applies to the channel-summed corners
      // head.*_bstride != 0: the gradients go into the gradient of the predictor's raw output (clip stride = all of
      // its channels), the mask's through the derivative of its activation (taken from the activated value m)
      if (has_mask && grad_mask) {
        float a[8];
        sample_weights(s, a);
        const long long ri = head.mask_bstride ? (long long)b * head.mask_bstride + ((long long)grp * g.K + tap) * g.V + v
                                               : (((long long)b * g.G + grp) * g.K + tap) * g.V + v;
        grad_mask[ri] = s.inside ? blend(G, a) * mask_act_slope(head.mask_act, m) : 0.f;
      }
      if constexpr (!FieldOut) {
        float* go = grad_coord + (head.geo_bstride ? (long long)b * head.geo_bstride + ((long long)grp * 3 * g.K + 3 * tap) * g.V + v
                                                   : (((long long)b * g.G + grp) * 3 * g.K + 3 * tap) * g.V + v);
        go[0] = m * wts[0];
        go[g.V] = m * wts[1];
        go[2 * (long long)g.V] = m * wts[2];
      } else {
        // the field's gradient sums over taps (and groups): taps are summed here, one atomic per group after
        const int k = tap % g.kw, jj = (tap / g.kw) % g.kh, i = tap / (g.kw * g.kh);
        fsum[0] += field_axes.pos[0][i] * (m * wts[0]);
        fsum[1] += field_axes.pos[1][jj] * (m * wts[1]);
        fsum[2] += field_axes.pos[2][k] * (m * wts[2]);
      }
    }
  }
  if constexpr (FieldOut) {
    if (active && j == 0) {
      float* gs = grad_coord + (long long)b * (head.geo_bstride ? head.geo_bstride : (long long)field_nch * g.V) + v;
      if (field_ch.x >= 0) atomicAdd(gs + (long long)field_ch.x * g.V, fsum[0]);
      if (field_ch.y >= 0) atomicAdd(gs + (long long)field_ch.y * g.V, fsum[1]);
      if (field_ch.z >= 0) atomicAdd(gs + (long long)field_ch.z * g.V, fsum[2]);
    }
  }
}
// kAsk: only where the positions were asked and this is the answer; a few blocks that take turns, so that it costs little where not
// (in turns it takes 3 to 8 % longer; fp16, 8 channels a thread, spills at three blocks a multiprocessor then).
template <bool FieldOut, bool kF32X, bool kNarrow, bool kAsk>
__global__ void __launch_bounds__(kSgThreads, kF32X || (kAsk && !kNarrow) ? 2 : 3)
sample_grad_direct_kernel(Geom g, ClStrides cs, int b0, int nh, const float4* __restrict__ recs,
                          const float* __restrict__ dcol, const void* __restrict__ x_cl_v, bool has_mask,
                          float* __restrict__ grad_coord, float* __restrict__ grad_mask, float* __restrict__ gx_cl,
                          int field_nch, int3 field_ch, const __grid_constant__ FieldAxes field_axes, int taps_per_block,
                          HeadCfg head, int3 blocks, const int* __restrict__ direct) {
  auto block = [&](int x, int y, int z) {
    sample_grad_direct<FieldOut, kF32X, kNarrow>(g, cs, b0, nh, recs, dcol, x_cl_v, has_mask, grad_coord, grad_mask, gx_cl, field_nch,
                                                 field_ch, field_axes, taps_per_block, head, x, y, z);
  };
  if constexpr (kAsk) {
    if (!*direct) return;
    const int n_blocks = blocks.x * blocks.y * blocks.z;
    for (int i = blockIdx.x; i < n_blocks; i += gridDim.x) block(i % blocks.x, i / blocks.x % blocks.y, i / (blocks.x * blocks.y));
  } else {
    block(blockIdx.x, blockIdx.y, blockIdx.z);
  }
}

}  // namespace
}  // namespace d2c
