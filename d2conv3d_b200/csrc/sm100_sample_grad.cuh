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

// Block = 32 output voxels (a brick) and up to 27 taps of one (clip, offset group).  A sample is one (voxel, tap); each of its
// corners inside the volume is a contribution: weight x gradient column is due to the input voxel there, and (gradient column .
// input) is due to the sample's coordinate and modulation gradients.
//   1  the block lists its contributions by input voxel ("cell"): count, start of each cell's list, entry;
//   2  groups of 8 lanes walk equal shares of the lists, a lane with 8 channels: the gradient columns of every entry are read, the
//      input only when the cell changes, the sum over a cell stays in registers and leaves as one reduction;
//   3  a thread per sample turns the eight corner sums into the gradients of offset (field) and modulation.
// Reducing every contribution into L2 by itself is bound by L2's rate of fp32 additions (6.8 TB/s): 512 channels in 8 groups on
// 2 x 8 x 30 x 54, offsets of two voxels, sends 8.15 GB, 1.68 ms with 16-byte reductions per corner.  A brick of 32 voxels and 27
// taps meets the same input voxel 4.2 times, so that 1.9 GB of sums leave it and 2 GB of input are read instead of 8.15; what bounds
// it now are the instructions of step 2 (about 110 a warp for four entries) and the steps' barriers.  Measured there: fp32 staging
// 1.68 -> 1.38 ms, fp16 staging 1.55 -> 1.35; field layer of one group of 256 channels on 2 x 8 x 60 x 107 2.16 -> 1.90; 32 channels
// a group, one clip of 8 x 120 x 214, 9.1 -> 7.7.  The smallest layers pay for the lists: 64 channels, 4 x 16 x 16, 15.7 -> 17.6 us,
// 256 channels in 4 groups 39.6 -> 37.1.  Not faster: a warp per entry with two channels a lane (35 instructions an entry),
// entries filled up so that none is out of range, the input read with every entry, three entries ahead, packed FMAs.
// Three blocks a multiprocessor with one entry ahead (80 registers) beat two blocks with two ahead, 1.38 to 1.43 ms; where a group has
// several slices shared memory allows two blocks, and the field's kernels would spill.
// kMulti: the offset group has several slices of 64 channels (nh > 1).
template <bool FieldOut, bool kF32X, bool kNarrow, bool kMulti>
__global__ void __launch_bounds__(kSgThreads, kMulti || FieldOut ? 2 : 3)
sample_grad_taps_kernel(Geom g, VoxelOrder order, ClStrides cs, int b0, int nh, const float4* __restrict__ recs,
                         const float* __restrict__ dcol, const void* __restrict__ x_cl_v, bool has_mask,
                         float* __restrict__ grad_coord, float* __restrict__ grad_mask, float* __restrict__ gx_cl,
                         int field_nch, int3 field_ch, const __grid_constant__ FieldAxes field_axes, int taps_per_block,
                         HeadCfg head) {
  extern __shared__ __align__(16) uint8_t sg_smem[];
  __shared__ int s_box[6], s_total, s_single, s_delta[8];
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
      if constexpr (FieldOut) {
        // A tap at the kernel's centre on an axis does not move along it, and no tap does where the field has no channel for the
        // axis: the upper corners of that axis weigh nothing and the axis takes no gradient (with 3 x 3 x 3 taps 4.6
        // corners a tap instead of 8, and 2.8 where the field scales rows and columns alone; the latter, one group of 256 channels
        // on 2 x 8 x 30 x 54: 531 us with the first of the two rules alone, 374 with both, 494 with every corner reduced by itself).
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

}  // namespace
}  // namespace d2c
