// Exact tier of the deformable convolutions: any geometry, fp32 / fp64, every product and sum on the FMA pipe (the
// results of an S/Dgemm up to summation order; fp64 supports gradcheck).  The tensor-core tier (deform_sm100_*.cu)
// replaces these kernels for the shapes it takes.
//
// Forward, gradient columns and weight gradient are one register-blocked GEMM each, 128 x N block tiles of 8 x N/16 per
// thread, 16 contraction rows per step, double-buffered in shared memory.  In the forward and the weight gradient the
// 128-wide operand is SAMPLED: the threads that multiply step s issue the corner loads of step s+1 before the arithmetic
// and blend them after it, so no column matrix exists.  Only the backward's gradient columns are written to memory.
//
// Two things make that fit the machine (B200: 128 fp32 FMA per clock and SM, one issue slot per scheduler and clock):
//   * fp32 products are packed (fma.rn.f32x2): half the issue slots of the FMA pipe stay free for coordinates, corner
//     loads and blends.  The pairs run along the output channel; the sampled operand is stored as broadcast pairs
//     {s, s}, because a pair built in registers costs a move per use.
//   * the input is staged channels-last (route kChannelsLast), so a 16-byte load fetches four channels of a corner and
//     the four corners' loads of neighbouring threads are one 64-byte run.  Below 16 channels, and for the 1-D op, whose
//     positions are already neighbours along a row, the samples are taken from the NCDHW tensor itself (kDirect).
//
// 128 -> 128 channels, one clip of 8 x 30 x 54, 4 offset groups, forward + backward: 6.37 ms with a scalar 64 x 64 tile and
// separate coordinate / scatter passes over channel-major columns.  What bounds the kernels now is the FMA pipe
// (forward, columns, weight gradient) and the L2's reduction rate (sampling gradient).
#pragma once

#include <cooperative_groups.h>

#include "deform_exact.h"

namespace d2c {
namespace exact {

namespace cg = cooperative_groups;

constexpr int kTM = 128;        // rows of a block tile (voxels, or column rows in the weight gradient)
constexpr int kThreads = 256;
constexpr int kPitchA = kTM + 2;   // in 8-byte elements; + 2 keeps 16-byte alignment and spreads the stores

// ---- element types -----------------------------------------------------------------------------------

using u64 = unsigned long long;

// What the 128-wide operand is stored as (8 bytes for both types) and how an accumulator row is kept.
template <typename T> struct Pair;
template <> struct Pair<float> {
  using type = u64;
  static __device__ __forceinline__ u64 bcast(float a) {
    u64 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
  }
  static __device__ __forceinline__ ulonglong2 two(float a, float b) { return make_ulonglong2(bcast(a), bcast(b)); }
};
template <> struct Pair<double> {
  using type = double;
  static __device__ __forceinline__ double bcast(double a) { return a; }
  static __device__ __forceinline__ ulonglong2 two(double a, double b) {
    return make_ulonglong2((u64)__double_as_longlong(a), (u64)__double_as_longlong(b));
  }
};

// One thread's accumulators: 8 rows x N columns.
template <typename T, int N> struct Acc;
template <int N> struct Acc<float, N> {
  u64 v[8][N / 2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < N / 2; ++j) v[i][j] = 0ull;
  }
  __device__ __forceinline__ void fma(int i, u64 a, const float (&b)[N]) {
#pragma unroll
    for (int j = 0; j < N / 2; ++j) {
      u64 bb;
      asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b[2 * j]), "f"(b[2 * j + 1]));
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[i][j]) : "l"(a), "l"(bb));
    }
  }
  __device__ __forceinline__ float at(int i, int j) const {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[i][j / 2]));
    return (j & 1) ? hi : lo;
  }
};
template <int N> struct Acc<double, N> {
  double v[8][N];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) v[i][j] = 0.0;
  }
  __device__ __forceinline__ void fma(int i, double a, const double (&b)[N]) {
#pragma unroll
    for (int j = 0; j < N; ++j) v[i][j] = __fma_rn(a, b[j], v[i][j]);
  }
  __device__ __forceinline__ double at(int i, int j) const { return v[i][j]; }
};

// Thread position in the 16 x 16 grid of a block tile.  A warp covers 8 x 4 threads, so that its A and B fragments are
// 128 and 64 contiguous bytes.
struct Lane {
  int tx, ty;
  __device__ __forceinline__ Lane() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    tx = (lane & 7) + 8 * (warp & 1);
    ty = (lane >> 3) + 4 * (warp >> 1);
  }
  // row i (0..7) of the thread inside the tile
  __device__ __forceinline__ int row(int i) const { return (i >> 1) * 32 + tx * 2 + (i & 1); }
  // column j of the thread's TN/16 columns: runs of four (two where there are only two)
  template <int TN>
  __device__ __forceinline__ int col(int j) const {
    return TN == 128 ? (j >> 2) * 64 + ty * 4 + (j & 3) : (TN == 64 ? ty * 4 + j : ty * 2 + j);
  }
};

// Row pitch of the B tile: the four elements of padding spread the transposing stores.
template <int TN> constexpr int kPitchB = TN + 4;

// two stages of both tiles
template <typename T, int TN>
constexpr size_t gemm_smem() { return 2 * (size_t)kTK * (kPitchA * 8 + kPitchB<TN> * sizeof(T)); }

// Resident blocks the sampling kernels are compiled for: 128 registers hold the accumulators of up to 64 fp32 columns.
template <typename T, int TN> constexpr int kBlocksPerSm = sizeof(T) == 4 && TN < 128 ? 2 : 1;

// acc += A[k][rows] * B[k][cols] for k in [k0, k0 + KN)
template <typename T, int TN, int KN>
__device__ __forceinline__ void tile_fma(const typename Pair<T>::type* As, const T* Bs, int k0, const Lane& L, Acc<T, TN / 16>& acc) {
  constexpr int N = TN / 16;
  constexpr int kVecB = 16 / sizeof(T);
#pragma unroll
  for (int kk = 0; kk < KN; ++kk) {
    const int k = k0 + kk;
    typename Pair<T>::type a[8];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const auto q = *reinterpret_cast<const ulonglong2*>(As + k * kPitchA + m * 32 + L.tx * 2);
      if constexpr (sizeof(T) == 4) {
        a[2 * m] = q.x; a[2 * m + 1] = q.y;
      } else {
        a[2 * m] = __longlong_as_double((long long)q.x); a[2 * m + 1] = __longlong_as_double((long long)q.y);
      }
    }
    T b[N];
    const T* brow = Bs + k * kPitchB<TN>;
    if constexpr (N == 2) {
      b[0] = brow[L.ty * 2]; b[1] = brow[L.ty * 2 + 1];
    } else {
#pragma unroll
      for (int h = 0; h < N / 4; ++h)
#pragma unroll
        for (int q = 0; q < 4 / kVecB; ++q) {
          const T* src = brow + h * 64 + L.ty * 4 + q * kVecB;
          if constexpr (sizeof(T) == 4) {
            const float4 f = *reinterpret_cast<const float4*>(src);
            b[4 * h] = f.x; b[4 * h + 1] = f.y; b[4 * h + 2] = f.z; b[4 * h + 3] = f.w;
          } else {
            const double2 f = *reinterpret_cast<const double2*>(src);
            b[4 * h + 2 * q] = f.x; b[4 * h + 2 * q + 1] = f.y;
          }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) acc.fma(i, a[i], b);
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- index arithmetic ----------------------------------------------------------------------------------

// Division of 0 <= n < 2^31 by a divisor known on the host.
struct FastDiv {
  uint32_t d, mul, shift;
  static FastDiv of(int d) {
    FastDiv f;
    f.d = (uint32_t)d;
    f.shift = 0;
    while ((1ull << f.shift) < (unsigned long long)d) ++f.shift;
    f.mul = (uint32_t)(((1ull << 32) * ((1ull << f.shift) - (unsigned long long)d)) / (unsigned long long)d + 1);
    return f;
  }
  __device__ __forceinline__ int div(int n) const { return (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shift); }
  __device__ __forceinline__ int divmod(int n, int& rem) const {
    const int q = div(n);
    rem = n - q * (int)d;
    return q;
  }
};

struct Index {
  FastDiv V, Wo, Ho, kw, kh, cpg, cin_g;
  static Index of(const Geom& g) {
    return {FastDiv::of(g.V), FastDiv::of(g.Wo), FastDiv::of(g.Ho), FastDiv::of(g.kw), FastDiv::of(g.kh), FastDiv::of(g.cpg),
            FastDiv::of(g.cin_g)};
  }
};

// An output voxel n of the flattened (clip, voxel) range, or nothing (n past the end).
struct Voxel {
  int b, v, bz, by, bx;    // clip, voxel inside it, integer base coordinates of tap 0
  bool ok;
  __device__ __forceinline__ void set(const Geom& g, const Index& ix, long long n, long long n_end, int b0) {
    ok = n < n_end;
    const int nn = ok ? (int)n : 0;
    int ox, oy;
    b = b0 + ix.V.divmod(nn, v);
    const int r = ix.Wo.divmod(v, ox), oz = ix.Ho.divmod(r, oy);
    bz = oz * g.sd - g.pd; by = oy * g.sh - g.ph; bx = ox * g.sw - g.pw;
  }
};

// A chunk of four column rows: one tap, channels [c, c+4) (c counts from the first channel of the weight group).
struct Chunk {
  int tap, i, j, k, c, grp;
  __device__ __forceinline__ void set(const Geom& g, const Index& ix, int row, int wg) {
    tap = ix.cin_g.divmod(row, c);
    const int r = ix.kw.divmod(tap, k);
    i = ix.kh.divmod(r, j);
    grp = ix.cpg.div(wg * g.cin_g + c);
  }
};

template <typename T> struct Pos { T z, y, x, m; };

template <typename T, typename Coords>
__device__ __forceinline__ Pos<T> position(const Geom& g, const Coords& coords, const T* __restrict__ mask, const Voxel& vx,
                                           const Chunk& ck) {
  Pos<T> p;
  coords.get_at(g, vx.b, ck.grp, ck.tap, ck.i, ck.j, ck.k, vx.v, vx.bz + ck.i * g.dd, vx.by + ck.j * g.dh, vx.bx + ck.k * g.dw,
                p.z, p.y, p.x);
  p.m = mask ? __ldg(mask + (((long long)vx.b * g.G + ck.grp) * g.K + ck.tap) * g.V + vx.v) : (T)1;
  return p;
}

// ---- sampling of one item: four channels of one (voxel, tap) ------------------------------------------------

template <typename T> struct Corners { T c[8][4]; };

// Issues the corner loads (0 where a corner does not contribute).  1-D: corners 0 and 1 only.
template <typename T, int kRoute, bool k1d>
__device__ __forceinline__ void load_corners(const Geom& g, const T* __restrict__ x, int b, int ch, const Pos<T>& p, bool ok,
                                             Corners<T>& out) {
  const Sample<T> s = make_sample(g, p.z, p.y, p.x);
  const unsigned valid = (ok && s.inside) ? s.valid : 0u;
  const long long lin = ((long long)s.z0 * g.H + s.y0) * g.W + s.x0;
#pragma unroll
  for (int q = 0; q < (k1d ? 2 : 8); ++q) {
    const long long at = lin + (q >> 2) * ((long long)g.H * g.W) + ((q >> 1) & 1) * g.W + (q & 1);
    const bool on = (valid >> q) & 1u;
    if constexpr (kRoute == kChannelsLast) {
      const T* src = x + ((long long)b * g.Vin + at) * g.Cin + ch;
      if constexpr (sizeof(T) == 4) {
        const float4 f = on ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
        out.c[q][0] = f.x; out.c[q][1] = f.y; out.c[q][2] = f.z; out.c[q][3] = f.w;
      } else {
        const double2 f = on ? __ldg(reinterpret_cast<const double2*>(src)) : make_double2(0.0, 0.0);
        const double2 h = on ? __ldg(reinterpret_cast<const double2*>(src) + 1) : make_double2(0.0, 0.0);
        out.c[q][0] = f.x; out.c[q][1] = f.y; out.c[q][2] = h.x; out.c[q][3] = h.y;
      }
    } else {
      const T* src = x + ((long long)b * g.Cin + ch) * g.Vin + at;
#pragma unroll
      for (int e = 0; e < 4; ++e) out.c[q][e] = on ? __ldg(src + e * g.Vin) : (T)0;
    }
  }
}

// mask * trilinear(x, p) of the four channels; the interpolation chain and roundings of the reference
// (csrc/ops/dconv3d_gpu.cu:48-109, 184-199)
template <typename T, bool k1d>
__device__ __forceinline__ void blend_item(const Geom& g, const Pos<T>& p, bool ok, const Corners<T>& c, T (&out)[4]) {
  const Sample<T> s = make_sample(g, p.z, p.y, p.x);
  T a[8];
  sample_weights(s, a);
  const bool in = ok && s.inside;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    T r = (T)0;
#pragma unroll
    for (int q = 0; q < (k1d ? 2 : 8); ++q) r = fma_rn(c.c[q][e], a[q], r);
    out[e] = in ? mul_rn(p.m, r) : (T)0;
  }
}

// Route kAny: four column rows that may belong to different taps and groups (channel counts not divisible by four);
// nothing is prefetched.
template <typename T, typename Coords>
__device__ __forceinline__ void sample_any(const Geom& g, const Index& ix, const Coords& coords, const T* __restrict__ x,
                                           const T* __restrict__ mask, const Voxel& vx, int row, int R, int wg, T (&out)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    out[e] = (T)0;
    if (!vx.ok || row + e >= R) continue;
    Chunk ck;
    ck.set(g, ix, row + e, wg);
    const Pos<T> p = position(g, coords, mask, vx, ck);
    const Sample<T> s = make_sample(g, p.z, p.y, p.x);
    if (!s.inside) continue;
    T a[8], cv[8];
    sample_weights(s, a);
    gather_corners(g, x + ((long long)vx.b * g.Cin + wg * g.cin_g + ck.c) * g.Vin, s, cv);
    out[e] = mul_rn(p.m, blend(cv, a));
  }
}

// ---- staging ---------------------------------------------------------------------------------------------------

template <typename T>
struct StageArgs {
  const T* x; T* x_cl;                 // [B][C][Vin] -> [B][Vin][C]
  const T* w; T* w_st;                 // see `transposed`
  int transposed;                      // 0: [wg][Rp rows][Np] (forward), 1: [wg][co padded][Rp] (gradient columns)
  int Rp, Np;                          // padded column rows, padded output channels
  long long x_blocks;
  ZeroFill zero[3];
};

// One launch: blocks below x_blocks transpose 32 voxels x 32 channels of x, the rest 32 x 32 pieces of the weights into
// column-row order (tap, channel), zero-padded so that the GEMM's loads need no bounds.
template <typename T>
__global__ void __launch_bounds__(256) stage_kernel(Geom g, StageArgs<T> p) {
  __shared__ T tile[32][33];
#pragma unroll
  for (int z = 0; z < 3; ++z) zero_fill(p.zero[z], blockIdx.x, gridDim.x);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (blockIdx.x < p.x_blocks) {
    const int cb = (g.Cin + 31) / 32;
    const long long vb = (g.Vin + 31) / 32;
    const long long blk = blockIdx.x;
    const int c0 = (int)(blk % cb) * 32;
    const long long v0 = ((blk / cb) % vb) * 32, b = blk / (cb * vb);
    for (int cc = ty; cc < 32; cc += 8)
      tile[cc][tx] = (v0 + tx < g.Vin && c0 + cc < g.Cin) ? __ldg(p.x + (b * g.Cin + c0 + cc) * g.Vin + v0 + tx) : (T)0;
    __syncthreads();
    for (int vv = ty; vv < 32; vv += 8)
      if (v0 + vv < g.Vin && c0 + tx < g.Cin) p.x_cl[(b * g.Vin + v0 + vv) * g.Cin + c0 + tx] = tile[tx][vv];
    return;
  }
  const int R = g.cin_g * g.K;
  const int rb = (p.Rp + 31) / 32, nb = (p.Np + 31) / 32;
  const long long blk = blockIdx.x - p.x_blocks;
  const int r0 = (int)(blk % rb) * 32, n0 = (int)((blk / rb) % nb) * 32, wg = (int)(blk / ((long long)rb * nb));
  // column row r = tap * cin_g + c; the source runs over (c, tap)
  for (int nn = ty; nn < 32; nn += 8) {
    const int r = r0 + tx, n = n0 + nn;
    T v = (T)0;
    if (r < R && n < g.cout_g) {
      const int tap = r / g.cin_g, c = r - tap * g.cin_g;
      v = __ldg(p.w + ((long long)(wg * g.cout_g + n)) * R + (long long)c * g.K + tap);
    }
    tile[nn][tx] = v;
  }
  __syncthreads();
  if (p.transposed) {
    for (int nn = ty; nn < 32; nn += 8)
      if (r0 + tx < p.Rp && n0 + nn < p.Np) p.w_st[((long long)wg * p.Np + n0 + nn) * p.Rp + r0 + tx] = tile[nn][tx];
  } else {
    for (int rr = ty; rr < 32; rr += 8)
      if (r0 + rr < p.Rp && n0 + tx < p.Np) p.w_st[((long long)wg * p.Rp + r0 + rr) * p.Np + n0 + tx] = tile[tx][rr];
  }
}

// ---- forward: y[b, co, v] = sum_r W[co, r] * sample(b, r, v) + bias[co] ------------------------------------------

template <typename T>
struct FwdArgs {
  const T* x;          // NCDHW, or its channels-last copy
  const T* mask;
  const T* w;          // the weights as given, or staged [wg][Rp][Np]
  const T* bias;
  T* y;
  int Rp, Np, steps;   // steps: 16-row steps of the whole contraction
};

// Grid (voxel tiles x cluster, output-channel tiles, weight groups); the CTAs of a cluster share a tile's contraction and
// add their accumulators through distributed shared memory in rank order (no atomics, no workspace, reproducible).
template <typename T, int TN, typename Coords, int kRoute>
__global__ void __launch_bounds__(kThreads, (kBlocksPerSm<T, TN>))
fwd_kernel(const __grid_constant__ Geom g, const __grid_constant__ Index ix, const __grid_constant__ Coords coords,
           const __grid_constant__ FwdArgs<T> p) {
  using P = typename Pair<T>::type;
  constexpr bool k1d = CoordsIs1d<Coords>::value;
  constexpr int N = TN / 16;
  constexpr int kA = kTK * kPitchA, kB = kTK * kPitchB<TN>;
  constexpr int kDirW = kTK * TN / kThreads;          // weights a thread fetches per step when they are not staged
  extern __shared__ __align__(16) unsigned char smem[];
  P* As = reinterpret_cast<P*>(smem);                                 // [2][16][kPitchA]
  T* Bs = reinterpret_cast<T*>(smem + 2 * kA * sizeof(P));            // [2][16][kPitchB]
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int t = threadIdx.x;
  const Lane L;
  const int R = g.cin_g * g.K, wg = blockIdx.z, n0 = blockIdx.y * TN;
  const long long total = (long long)g.B * g.V, v0 = (long long)(blockIdx.x / ranks) * kTM;
  const int s_beg = (int)((long long)p.steps * rank / ranks), s_end = (int)((long long)p.steps * (rank + 1) / ranks);

  // a thread samples chunk q (four of the step's 16 rows) of voxels vr and vr + 64
  const int q = kRoute == kChannelsLast ? (t & 3) : (t >> 6), vr = kRoute == kChannelsLast ? (t >> 2) : (t & 63);
  Voxel vx[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) vx[h].set(g, ix, v0 + vr + 64 * h, total, 0);
  Acc<T, N> acc;
  acc.clear();

  Pos<T> pos[2];
  Corners<T> cor;
  T wreg[kDirW];
  auto chunk_of = [&](int s, Chunk& ck) {
    const int row = s * kTK + q * 4;
    ck.set(g, ix, min(row, R - 4 < 0 ? 0 : R - 4), wg);
    return row < R;
  };
  auto positions = [&](int s, int h) {
    if constexpr (kRoute != kAny) {
      Chunk ck;
      if (s < s_end && chunk_of(s, ck) && vx[h].ok) pos[h] = position(g, coords, p.mask, vx[h], ck);
    }
  };
  auto issue = [&](int s, int h) {
    if constexpr (kRoute != kAny) {
      Chunk ck;
      const bool ok = chunk_of(s, ck) && vx[h].ok;
      load_corners<T, kRoute, k1d>(g, p.x, vx[h].b, wg * g.cin_g + ck.c, pos[h], ok, cor);
    }
  };
  auto finish = [&](int s, int h, int buf) {
    T out[4];
    if constexpr (kRoute == kAny)
      sample_any<T, Coords>(g, ix, coords, p.x, p.mask, vx[h], s * kTK + q * 4, R, wg, out);
    else
      blend_item<T, k1d>(g, pos[h], vx[h].ok && s * kTK + q * 4 < R, cor, out);
#pragma unroll
    for (int e = 0; e < 4; ++e) As[buf * kA + (q * 4 + e) * kPitchA + vr + 64 * h] = Pair<T>::bcast(out[e]);
  };
  auto weights_begin = [&](int s, int buf) {
    if constexpr (kRoute == kChannelsLast) {
      constexpr int kVec = 16 / sizeof(T), kPer = TN / kVec;
      const T* src = p.w + ((long long)wg * p.Rp + (long long)s * kTK) * p.Np + n0;
      for (int e = t; e < kTK * kPer; e += kThreads)
        cp_async16(Bs + buf * kB + (e / kPer) * kPitchB<TN> + (e % kPer) * kVec, src + (long long)(e / kPer) * p.Np + (e % kPer) * kVec);
    } else {
#pragma unroll
      for (int j = 0; j < kDirW; ++j) {
        const int row = s * kTK + (t & 15), n = n0 + (t >> 4) + 16 * j;
        int c;
        const int tap = ix.cin_g.divmod(min(row, R - 1), c);
        wreg[j] = (row < R && n < g.cout_g) ? __ldg(p.w + ((long long)(wg * g.cout_g + n)) * R + (long long)c * g.K + tap) : (T)0;
      }
    }
  };
  auto weights_end = [&](int buf) {
    if constexpr (kRoute == kChannelsLast) {
      cp_async_wait();
    } else {
#pragma unroll
      for (int j = 0; j < kDirW; ++j) Bs[buf * kB + (t & 15) * kPitchB<TN> + (t >> 4) + 16 * j] = wreg[j];
    }
  };

  if (s_beg < s_end) {
    weights_begin(s_beg, 0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      positions(s_beg, h);
      issue(s_beg, h);
      finish(s_beg, h, 0);
      positions(s_beg + 1, h);
    }
    weights_end(0);
    __syncthreads();
    for (int s = s_beg; s < s_end; ++s) {
      const int cur = (s - s_beg) & 1;
      const bool more = s + 1 < s_end;
      if (more) weights_begin(s + 1, cur ^ 1);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (more) issue(s + 1, h);
        tile_fma<T, TN, kTK / 2>(As + cur * kA, Bs + cur * kB, h * (kTK / 2), L, acc);
        if (more) {
          finish(s + 1, h, cur ^ 1);
          positions(s + 2, h);
        }
      }
      if (more) weights_end(cur ^ 1);
      __syncthreads();
    }
  }

  auto store = [&](int row, int n, T v) {
    const long long vox = v0 + row;
    if (vox < total && n < g.cout_g) {
      int vv;
      const int b = ix.V.divmod((int)vox, vv);
      const int co = wg * g.cout_g + n;
      p.y[((long long)b * g.Cout + co) * g.V + vv] = v + (p.bias ? __ldg(p.bias + co) : (T)0);
    }
  };
  if (ranks == 1) {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < 8; ++i) store(L.row(i), n0 + L.template col<TN>(j), acc.at(i, j));
    return;
  }
  T* part = reinterpret_cast<T*>(smem);                // [TN][kTM + 4]
  constexpr int kPitchC = kTM + 4;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) part[L.template col<TN>(j) * kPitchC + L.row(i)] = acc.at(i, j);
  cluster.sync();
  for (int e = rank * kThreads + t; e < TN * kTM; e += ranks * kThreads) {
    const int n = e / kTM, row = e % kTM;
    T v = (T)0;
    for (int r = 0; r < ranks; ++r) v += cluster.map_shared_rank(part, r)[n * kPitchC + row];
    store(row, n0 + n, v);
  }
  cluster.sync();                                      // nobody leaves while its tile is being read
}

template <typename T, int TN>
constexpr size_t fwd_smem() {
  const size_t loop = gemm_smem<T, TN>();
  const size_t out = (size_t)TN * (kTM + 4) * sizeof(T);
  return loop > out ? loop : out;
}

// ---- gradient columns: dcol = sum_co W[co, r] * gy[b, co, v]  (reference dconv3d_gpu.cu:981-999) ------------------

template <typename T>
struct DcolArgs {
  const T* gy;
  const T* w;          // staged [wg][Np][Rp] in (tap, channel) row order, or the weights as given (rows (channel, tap))
  T* dcol;             // kChannelsLast: [clip][tap][v][Cin]; otherwise [clip][Cin*K][v]
  int Rp, Np, b0, nb;
};

template <typename T> constexpr int kDcolN = sizeof(T) == 4 ? 128 : 64;      // column rows of a block tile

template <typename T, int kRoute>
__global__ void __launch_bounds__(kThreads, 2)
dcol_kernel(const __grid_constant__ Geom g, const __grid_constant__ Index ix, const __grid_constant__ DcolArgs<T> p) {
  constexpr int TN = kDcolN<T>;
  using P = typename Pair<T>::type;
  constexpr int N = TN / 16;
  constexpr int kA = kTK * kPitchA, kB = kTK * kPitchB<TN>;
  constexpr int kLdA = kTK * kTM / kThreads, kLdB = kTK * TN / kThreads;
  extern __shared__ __align__(16) unsigned char smem[];
  P* As = reinterpret_cast<P*>(smem);                                 // [2][16 channels][kPitchA voxels]
  T* Bs = reinterpret_cast<T*>(smem + 2 * kA * sizeof(P));            // [2][16 channels][kPitchB column rows]
  const int t = threadIdx.x;
  const Lane L;
  const int R = g.cin_g * g.K, wg = blockIdx.y, rtiles = (R + TN - 1) / TN;
  const int r0 = (int)(blockIdx.x % rtiles) * TN;
  const long long total = (long long)p.nb * g.V, v0 = (long long)(blockIdx.x / rtiles) * kTM;
  const int steps = (g.cout_g + kTK - 1) / kTK;

  // this thread's voxel column and its rows (co) of the A tile
  const int va = t & 127, ca = t >> 7;
  const long long na = v0 + va;
  const bool va_ok = na < total;
  int vva = 0, bla = 0;
  if (va_ok) bla = ix.V.divmod((int)na, vva);
  const T* gyp = p.gy + ((long long)(p.b0 + bla) * g.Cout + wg * g.cout_g) * g.V + vva;
  T areg[kLdA], breg[kLdB];
  Acc<T, N> acc;
  acc.clear();
  auto begin = [&](int s, int buf) {
#pragma unroll
    for (int j = 0; j < kLdA; ++j) {
      const int co = s * kTK + ca + 2 * j;
      areg[j] = (va_ok && co < g.cout_g) ? __ldg(gyp + (long long)co * g.V) : (T)0;
    }
    if constexpr (kRoute == kChannelsLast) {
      constexpr int kVec = 16 / sizeof(T), kPer = TN / kVec;
      const T* src = p.w + ((long long)wg * p.Np + (long long)s * kTK) * p.Rp + r0;
      for (int e = t; e < kTK * kPer; e += kThreads)
        cp_async16(Bs + buf * kB + (e / kPer) * kPitchB<TN> + (e % kPer) * kVec, src + (long long)(e / kPer) * p.Rp + (e % kPer) * kVec);
    } else {
#pragma unroll
      for (int j = 0; j < kLdB; ++j) {
        const int e = t + j * kThreads, co = s * kTK + e / TN, r = r0 + e % TN;
        breg[j] = (co < g.cout_g && r < R) ? __ldg(p.w + ((long long)(wg * g.cout_g + co)) * R + r) : (T)0;
      }
    }
  };
  auto end = [&](int buf) {
#pragma unroll
    for (int j = 0; j < kLdA; ++j) As[buf * kA + (ca + 2 * j) * kPitchA + va] = Pair<T>::bcast(areg[j]);
    if constexpr (kRoute == kChannelsLast) {
      cp_async_wait();
    } else {
#pragma unroll
      for (int j = 0; j < kLdB; ++j) {
        const int e = t + j * kThreads;
        Bs[buf * kB + (e / TN) * kPitchB<TN> + e % TN] = breg[j];
      }
    }
  };
  begin(0, 0);
  end(0);
  __syncthreads();
  for (int s = 0; s < steps; ++s) {
    const int cur = s & 1;
    const bool more = s + 1 < steps;
    if (more) begin(s + 1, cur ^ 1);
    tile_fma<T, TN, kTK>(As + cur * kA, Bs + cur * kB, 0, L, acc);
    if (more) end(cur ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const long long n = v0 + L.row(i);
    if (n >= total) continue;
    int v;
    const int bl = ix.V.divmod((int)n, v);
#pragma unroll
    for (int h = 0; h < N / 4; ++h) {
      const int r = r0 + L.template col<TN>(4 * h);
      if (r >= R) continue;
      if constexpr (kRoute == kChannelsLast) {
        int c;
        const int tap = ix.cin_g.divmod(r, c);          // four rows of one tap: channel counts are multiples of four
        T* dst = p.dcol + (((long long)bl * g.K + tap) * g.V + v) * g.Cin + wg * g.cin_g + c;
        if constexpr (sizeof(T) == 4)
          *reinterpret_cast<float4*>(dst) = make_float4(acc.at(i, 4 * h), acc.at(i, 4 * h + 1), acc.at(i, 4 * h + 2), acc.at(i, 4 * h + 3));
        else {
          reinterpret_cast<double2*>(dst)[0] = make_double2(acc.at(i, 4 * h), acc.at(i, 4 * h + 1));
          reinterpret_cast<double2*>(dst)[1] = make_double2(acc.at(i, 4 * h + 2), acc.at(i, 4 * h + 3));
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (r + e < R) p.dcol[((long long)bl * g.Cin * g.K + (long long)wg * R + r + e) * g.V + v] = acc.at(i, 4 * h + e);
      }
    }
  }
}

// ---- weight gradient: dW[co, r] = sum_{b, v} gy[b, co, v] * sample(b, r, v)  (reference dconv3d_gpu.cu:1037-1088) ---

template <typename T>
struct DwArgs {
  const T* x;
  const T* mask;
  const T* gy;
  T* grad_w;           // zeroed beforehand when `add`
  T* grad_bias;        // nullable; zeroed beforehand
  int steps, splits, add;
};

// Grid (column-row tiles x voxel ranges, output-channel tiles, weight groups).  The blocks of the first column-row tile
// also sum grad_out over their voxels: grad_bias.
template <typename T, int TN, typename Coords, int kRoute>
__global__ void __launch_bounds__(kThreads, (kBlocksPerSm<T, TN>))
dw_kernel(const __grid_constant__ Geom g, const __grid_constant__ Index ix, const __grid_constant__ Coords coords,
          const __grid_constant__ DwArgs<T> p) {
  using P = typename Pair<T>::type;
  constexpr bool k1d = CoordsIs1d<Coords>::value;
  constexpr int N = TN / 16;
  constexpr int kA = kTK * kPitchA, kB = kTK * kPitchB<TN>;
  constexpr int kLdB = kTK * TN / kThreads;
  extern __shared__ __align__(16) unsigned char smem[];
  P* As = reinterpret_cast<P*>(smem);                                 // [2][16 voxels][kPitchA column rows]
  T* Bs = reinterpret_cast<T*>(smem + 2 * kA * sizeof(P));            // [2][16 voxels][kPitchB]
  const int t = threadIdx.x;
  const Lane L;
  const int R = g.cin_g * g.K, wg = blockIdx.z, n0 = blockIdx.y * TN;
  const int rtile = blockIdx.x / p.splits, split = blockIdx.x % p.splits, r0 = rtile * kTM;
  const long long total = (long long)g.B * g.V;
  const int s_beg = (int)((long long)p.steps * split / p.splits), s_end = (int)((long long)p.steps * (split + 1) / p.splits);
  const bool want_bias = p.grad_bias != nullptr && rtile == 0;

  // channels-last: a warp takes the 32 chunks of one voxel (512 contiguous bytes where a tap has 128 channels), voxels
  // warp and warp + 8; otherwise 16 voxels x 2 chunks per warp, chunks t/16 and t/16 + 16
  auto chunk_row = [&](int h) { return r0 + 4 * (kRoute == kChannelsLast ? (t & 31) : (t >> 4) + 16 * h); };
  auto voxel_of = [&](int h) { return kRoute == kChannelsLast ? (t >> 5) + 8 * h : (t & 15); };
  Pos<T> pos[2];
  Corners<T> cor;
  T breg[kLdB], bsum[kLdB];
#pragma unroll
  for (int j = 0; j < kLdB; ++j) bsum[j] = (T)0;
  Acc<T, N> acc;
  acc.clear();
  auto item = [&](int s, int h, Chunk& ck, Voxel& vx) {
    ck.set(g, ix, min(chunk_row(h), R - 4 < 0 ? 0 : R - 4), wg);
    vx.set(g, ix, (long long)s * kTK + voxel_of(h), total, 0);
    return vx.ok && chunk_row(h) < R;
  };
  auto positions = [&](int s, int h) {
    if constexpr (kRoute != kAny) {
      Chunk ck;
      Voxel vx;
      if (s < s_end && item(s, h, ck, vx)) pos[h] = position(g, coords, p.mask, vx, ck);
    }
  };
  auto issue = [&](int s, int h) {
    if constexpr (kRoute != kAny) {
      Chunk ck;
      Voxel vx;
      const bool ok = item(s, h, ck, vx);
      load_corners<T, kRoute, k1d>(g, p.x, vx.b, wg * g.cin_g + ck.c, pos[h], ok, cor);
    }
  };
  auto finish = [&](int s, int h, int buf) {
    T out[4];
    const bool in_range = (long long)s * kTK + voxel_of(h) < total && chunk_row(h) < R;
    if constexpr (kRoute == kAny) {
      Voxel vx;
      vx.set(g, ix, (long long)s * kTK + voxel_of(h), total, 0);
      sample_any<T, Coords>(g, ix, coords, p.x, p.mask, vx, chunk_row(h), R, wg, out);
    } else {
      blend_item<T, k1d>(g, pos[h], in_range, cor, out);
    }
    P* dst = As + buf * kA + voxel_of(h) * kPitchA + (chunk_row(h) - r0);
    reinterpret_cast<ulonglong2*>(dst)[0] = Pair<T>::two(out[0], out[1]);
    reinterpret_cast<ulonglong2*>(dst)[1] = Pair<T>::two(out[2], out[3]);
  };
  auto grads_begin = [&](int s) {
    int v = 0, b = 0;
    const long long n = (long long)s * kTK + (t & 15);
    const bool ok = n < total;
    if (ok) b = ix.V.divmod((int)n, v);
    const T* src = p.gy + ((long long)b * g.Cout + wg * g.cout_g) * g.V + v;
#pragma unroll
    for (int j = 0; j < kLdB; ++j) {
      const int co = n0 + (t >> 4) + 16 * j;
      breg[j] = (ok && co < g.cout_g) ? __ldg(src + (long long)co * g.V) : (T)0;
    }
  };
  auto grads_end = [&](int buf) {
#pragma unroll
    for (int j = 0; j < kLdB; ++j) Bs[buf * kB + (t & 15) * kPitchB<TN> + (t >> 4) + 16 * j] = breg[j];
    if (want_bias) {
#pragma unroll
      for (int j = 0; j < kLdB; ++j) bsum[j] += breg[j];
    }
  };

  if (s_beg < s_end) {
    grads_begin(s_beg);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      positions(s_beg, h);
      issue(s_beg, h);
      finish(s_beg, h, 0);
      positions(s_beg + 1, h);
    }
    grads_end(0);
    __syncthreads();
    for (int s = s_beg; s < s_end; ++s) {
      const int cur = (s - s_beg) & 1;
      const bool more = s + 1 < s_end;
      if (more) grads_begin(s + 1);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (more) issue(s + 1, h);
        tile_fma<T, TN, kTK / 2>(As + cur * kA, Bs + cur * kB, h * (kTK / 2), L, acc);
        if (more) {
          finish(s + 1, h, cur ^ 1);
          positions(s + 2, h);
        }
      }
      if (more) grads_end(cur ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + L.row(i);
    if (r >= R) continue;
    int c;
    const int tap = ix.cin_g.divmod(r, c);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int n = n0 + L.template col<TN>(j);
      if (n >= g.cout_g) continue;
      T* dst = p.grad_w + ((long long)(wg * g.cout_g + n)) * R + (long long)c * g.K + tap;
      if (p.add)
        atomicAdd(dst, acc.at(i, j));
      else
        *dst = acc.at(i, j);
    }
  }
  if (want_bias) {
#pragma unroll
    for (int j = 0; j < kLdB; ++j) {
      T s = bsum[j];
#pragma unroll
      for (int o = 8; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int co = n0 + (t >> 4) + 16 * j;
      if ((t & 15) == 0 && co < g.cout_g) atomicAdd(p.grad_bias + wg * g.cout_g + co, s);
    }
  }
}

// ---- sampling gradient + scatter -------------------------------------------------------------------------------------

// Offset / mask / field gradients and the scatter of grad_input in one pass over the gradient columns
// (reference dconv3d_gpu.cu:562-643, 756-864).
template <typename T>
struct GradArgs {
  const T* dcol;
  const T* x;
  const T* mask;
  T* grad_coord;       // offsets, or the field (zeroed beforehand)
  T* grad_mask;
  T* grad_x;           // zeroed beforehand; kChannelsLast: [B][Vin][Cin]
  int b0, nb, taps_per_block;
};

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void red_add4(double* p, double a, double b, double c, double d) {
  atomicAdd(p, a); atomicAdd(p + 1, b); atomicAdd(p + 2, c); atomicAdd(p + 3, d);
}
template <typename T> __device__ __forceinline__ void load4(const T* p, T (&o)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
  } else {
    const double2 f = __ldg(reinterpret_cast<const double2*>(p)), h = __ldg(reinterpret_cast<const double2*>(p) + 1);
    o[0] = f.x; o[1] = f.y; o[2] = h.x; o[3] = h.y;
  }
}

// weights of the reference's col2im; a corner at distance exactly 1 fails its `< 1` test and is skipped (:626-637)
template <typename T>
__device__ __forceinline__ bool scatter_weight(const Sample<T>& s, int q, T& w) {
  const bool ok = !((q & 4) && !(s.gz < (T)1)) && !((q & 2) && !(s.gy < (T)1)) && !((q & 1) && !(s.gx < (T)1));
  const T wz = sub_rn((T)1, (q & 4) ? s.gz : s.fz), wy = sub_rn((T)1, (q & 2) ? s.gy : s.fy), wx = sub_rn((T)1, (q & 1) ? s.gx : s.fx);
  w = mul_rn(mul_rn(wz, wy), wx);
  return ok;
}

// Writes the gradients of one (voxel, tap, group) from the channel-summed corner products G and sample product.
template <typename T, typename Coords, bool FieldOut>
__device__ __forceinline__ void write_coord_grads(const Geom& g, const GradArgs<T>& p, const Coords& coords, int b, int grp, int tap,
                                                  int i, int j, int k, int v, T m, const Sample<T>& s, const T (&G)[8], T (&fsum)[3]) {
  T wts[3], a[8];
  coord_weights(G, s, wts);            // linear in the corner values: applies to the channel-summed corners
  const long long mi = (((long long)b * g.G + grp) * g.K + tap) * g.V + v;
  if (p.mask && p.grad_mask) {
    sample_weights(s, a);
    p.grad_mask[mi] = s.inside ? blend(G, a) : (T)0;
  }
  if constexpr (!FieldOut) {
    T* go = p.grad_coord + (((long long)b * g.G + grp) * 3 * g.K + 3 * tap) * g.V + v;
    go[0] = m * wts[0];
    go[g.V] = m * wts[1];
    go[2 * (long long)g.V] = m * wts[2];
  } else {
    fsum[0] += coords.axis[0][i] * (m * wts[0]);
    fsum[1] += coords.axis[1][j] * (m * wts[1]);
    fsum[2] += coords.axis[2][k] * (m * wts[2]);
  }
}

template <typename T, typename Coords>
__device__ __forceinline__ void add_field_grads(const Geom& g, const GradArgs<T>& p, const Coords& coords, int b, int v, const T (&fsum)[3]) {
  T* gs = p.grad_coord + (long long)b * coords.nch * g.V + v;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (coords.ch[d] >= 0) atomicAdd(gs + (long long)coords.ch[d] * g.V, fsum[d]);
}

// Channels-last route: TPV threads per voxel, each four channels at a time of its group; the block walks its taps.
// grid (voxel blocks x clips x groups, tap ranges).
template <typename T, typename Coords, bool FieldOut, int TPV>
__global__ void __launch_bounds__(256)
grad_cl_kernel(const __grid_constant__ Geom g, const __grid_constant__ Index ix, const __grid_constant__ Coords coords,
               const __grid_constant__ GradArgs<T> p) {
  const int vblocks = (g.V + 256 / TPV - 1) / (256 / TPV), bg = blockIdx.x / vblocks;
  const int j4 = threadIdx.x % TPV, n = (blockIdx.x % vblocks) * (256 / TPV) + threadIdx.x / TPV;
  const int bl = bg / g.G, grp = bg % g.G, b = p.b0 + bl;
  Voxel vx;
  vx.set(g, ix, n < g.V ? n : 0, g.V, 0);
  const bool live = n < g.V;
  vx.b = b;
  const int chunks = g.cpg / 4;
  const T* xb = p.x + (long long)b * g.Vin * g.Cin + grp * g.cpg;
  T* gxb = p.grad_x + (long long)b * g.Vin * g.Cin + grp * g.cpg;
  T fsum[3] = {(T)0, (T)0, (T)0};
  const int tap_end = min(g.K, (int)(blockIdx.y + 1) * p.taps_per_block);
  for (int tap = blockIdx.y * p.taps_per_block; tap < tap_end; ++tap) {
    Chunk ck;
    ck.tap = tap; ck.grp = grp; ck.c = 0;
    const int r = ix.kw.divmod(tap, ck.k);
    ck.i = ix.kh.divmod(r, ck.j);
    const Pos<T> pos = position(g, coords, p.mask, vx, ck);
    const Sample<T> s = make_sample(g, pos.z, pos.y, pos.x);
    const unsigned valid = live ? s.valid : 0u;
    const long long lin = (((long long)s.z0 * g.H + s.y0) * g.W + s.x0) * g.Cin;
    const T* dc = p.dcol + (((long long)bl * g.K + tap) * g.V + vx.v) * g.Cin + grp * g.cpg;
    T G[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) G[q] = (T)0;
    for (int c4 = j4; c4 < chunks; c4 += TPV) {
      T d[4], xv[8][4];
      load4(dc + 4 * c4, d);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const long long at = lin + ((q >> 2) * ((long long)g.H * g.W) + ((q >> 1) & 1) * g.W + (q & 1)) * g.Cin + 4 * c4;
        if ((valid >> q) & 1u) load4(xb + at, xv[q]);
        else xv[q][0] = xv[q][1] = xv[q][2] = xv[q][3] = (T)0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        G[q] += (d[0] * xv[q][0] + d[1] * xv[q][1]) + (d[2] * xv[q][2] + d[3] * xv[q][3]);
        T w;
        if (scatter_weight(s, q, w) && ((valid >> q) & 1u)) {
          w *= pos.m;
          const long long at = lin + ((q >> 2) * ((long long)g.H * g.W) + ((q >> 1) & 1) * g.W + (q & 1)) * g.Cin + 4 * c4;
          red_add4(gxb + at, w * d[0], w * d[1], w * d[2], w * d[3]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int o = TPV / 2; o >= 1; o >>= 1) G[q] += __shfl_xor_sync(0xffffffffu, G[q], o);
    if (live && j4 == 0)
      write_coord_grads<T, Coords, FieldOut>(g, p, coords, b, grp, tap, ck.i, ck.j, ck.k, vx.v, pos.m, s, G, fsum);
  }
  if constexpr (FieldOut) {
    if (live && j4 == 0) add_field_grads(g, p, coords, b, vx.v, fsum);
  }
}

// NCDHW routes (few channels, odd channel counts, 1-D): a block takes 32 neighbouring voxels of one (clip, group, tap), its
// eight warps share the group's channels; columns are [Cin*K][v].  The 1-D op has its own rule for the gradient of the
// position: at a position within 1e-8 of an integer the LEFT neighbour moves one further left while the right one stays
// (reference csrc/ops/dconv1d_gpu.cu:300-349, with its lerp, line 13-15).
template <typename T, typename Coords, bool FieldOut>
__global__ void __launch_bounds__(256)
grad_direct_kernel(const __grid_constant__ Geom g, const __grid_constant__ Index ix, const __grid_constant__ Coords coords,
                   const __grid_constant__ GradArgs<T> p) {
  constexpr bool k1d = CoordsIs1d<Coords>::value;
  __shared__ T part[8][8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int vblocks = (g.V + 31) / 32;
  const int blk = blockIdx.x, vb = blk % vblocks, bgt = blk / vblocks;
  const int tap = bgt % g.K, grp = (bgt / g.K) % g.G, bl = bgt / (g.K * g.G), b = p.b0 + bl;
  const int n = vb * 32 + lane;
  const bool live = n < g.V;
  Voxel vx;
  vx.set(g, ix, live ? n : 0, g.V, 0);
  vx.b = b;
  Chunk ck;
  ck.tap = tap; ck.grp = grp; ck.c = 0;
  const int r = ix.kw.divmod(tap, ck.k);
  ck.i = ix.kh.divmod(r, ck.j);
  const Pos<T> pos = position(g, coords, p.mask, vx, ck);
  const Sample<T> s = make_sample(g, pos.z, pos.y, pos.x);
  const unsigned valid = live ? s.valid : 0u;
  const long long lin = ((long long)s.z0 * g.H + s.y0) * g.W + s.x0;
  T G[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) G[q] = (T)0;
  // 1-D: G[0] = sum of (right - left) * column, G[1] = sum of lerp * column
  int x0 = s.x0;
  T lerp_t = s.fx;
  if constexpr (k1d) {
    if (sub_rn(pos.x, (T)x0) < (T)1e-8) x0 -= 1;
    lerp_t = sub_rn(pos.x, (T)x0);
  }
  for (int c = warp; c < g.cpg; c += 8) {
    const long long ch = (long long)grp * g.cpg + c;
    const T* plane = p.x + ((long long)b * g.Cin + ch) * g.Vin;
    T* gplane = p.grad_x + ((long long)b * g.Cin + ch) * g.Vin;
    const T d = live ? __ldg(p.dcol + (((long long)bl * g.Cin + ch) * g.K + tap) * g.V + vx.v) : (T)0;
    if constexpr (k1d) {
      const T l = (live && x0 >= 0 && x0 < g.W) ? __ldg(plane + x0) : (T)0;
      const T h = (live && s.x0 + 1 >= 0 && s.x0 + 1 < g.W) ? __ldg(plane + s.x0 + 1) : (T)0;
      G[0] += (h - l) * d * pos.m;
      G[1] += d * fma_rn(lerp_t, h, fma_rn(-lerp_t, l, l));
    }
#pragma unroll
    for (int q = 0; q < (k1d ? 2 : 8); ++q) {
      if (!((valid >> q) & 1u)) continue;
      const long long at = lin + (q >> 2) * ((long long)g.H * g.W) + ((q >> 1) & 1) * g.W + (q & 1);
      if constexpr (!k1d) G[q] += d * __ldg(plane + at);
      T w;
      if (scatter_weight(s, q, w)) atomicAdd(gplane + at, w * (pos.m * d));
    }
  }
#pragma unroll
  for (int q = 0; q < (k1d ? 2 : 8); ++q) part[warp][q][lane] = G[q];
  __syncthreads();
  if (warp != 0 || !live) return;
#pragma unroll
  for (int q = 0; q < (k1d ? 2 : 8); ++q)
    for (int wp = 1; wp < 8; ++wp) G[q] += part[wp][q][lane];
  if constexpr (k1d) {
    const long long mi = (((long long)b * g.G + grp) * g.K + tap) * g.V + vx.v;
    p.grad_coord[mi] = G[0];
    if (p.mask && p.grad_mask) p.grad_mask[mi] = G[1];
  } else {
    T fsum[3] = {(T)0, (T)0, (T)0};
    write_coord_grads<T, Coords, FieldOut>(g, p, coords, b, grp, tap, ck.i, ck.j, ck.k, vx.v, pos.m, s, G, fsum);
    if constexpr (FieldOut) add_field_grads(g, p, coords, b, vx.v, fsum);
  }
}

// channels-last gradient of x -> NCDHW
template <typename T>
__global__ void __launch_bounds__(256) unstage_kernel(Geom g, const T* __restrict__ gx_cl, T* __restrict__ gx) {
  __shared__ T tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long v0 = (long long)blockIdx.x * 32, b = blockIdx.z;
  const int c0 = blockIdx.y * 32;
  for (int vv = ty; vv < 32; vv += 8)
    tile[vv][tx] = (v0 + vv < g.Vin && c0 + tx < g.Cin) ? __ldg(gx_cl + (b * g.Vin + v0 + vv) * g.Cin + c0 + tx) : (T)0;
  __syncthreads();
  for (int cc = ty; cc < 32; cc += 8)
    if (v0 + tx < g.Vin && c0 + cc < g.Cin) gx[(b * g.Cin + c0 + cc) * g.Vin + v0 + tx] = tile[tx][cc];
}

// ---- host side -----------------------------------------------------------------------------------------------------------

// the kernels count flattened voxels in 31 bits
inline bool too_large(const Geom& g) { return (long long)g.B * g.V > 0x7fffff00LL || (long long)g.cin_g * g.K > 0x7fffff00LL; }

template <typename T>
int launch_stage(const Geom& g, StageArgs<T> a, cudaStream_t st) {
  a.x_blocks = (long long)((g.Cin + 31) / 32) * ((g.Vin + 31) / 32) * g.B;
  const long long wblocks = (long long)((a.Rp + 31) / 32) * ((a.Np + 31) / 32) * g.groups;
  if (a.x_blocks + wblocks > 0x7fffffffLL) return D2C_ERR_TOO_LARGE;
  stage_kernel<T><<<(unsigned)(a.x_blocks + wblocks), 256, 0, st>>>(g, a);
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

// CTAs that share a tile's contraction: the size (1, 2, 4, 8) with the shortest expected time.  A wave takes the steps of
// one CTA plus, where there is something to combine, about six steps' worth of filling the pipeline and adding tiles.
inline int pick_cluster(long long tiles, int steps, int sm_count, int per_sm) {
  int best = 1;
  double best_t = 0;
  for (int s = 1; s <= 8; s *= 2) {
    if (s > 1 && steps < 2 * s) break;
    const long long waves = (tiles * s + (long long)sm_count * per_sm - 1) / ((long long)sm_count * per_sm);
    const double t = (double)waves * ((double)((steps + s - 1) / s) + (s > 1 ? 6.0 : 2.0));
    if (s == 1 || t < best_t) { best_t = t; best = s; }
  }
  return best;
}

template <typename T, int TN, typename Coords, int kRoute>
int launch_fwd_tn(const Geom& g, const Coords& coords, const FwdArgs<T>& a, cudaStream_t st) {
  constexpr auto kern = fwd_kernel<T, TN, Coords, kRoute>;
  constexpr int smem = (int)fwd_smem<T, TN>();
  int rc = allow_dynamic_smem<kern>(smem), sm_count = 0;
  if (rc || (rc = device_sm_count(&sm_count))) return rc;
  const long long vtiles = ((long long)g.B * g.V + kTM - 1) / kTM;
  const int ntiles = (g.cout_g + TN - 1) / TN;
  const int s = pick_cluster(vtiles * ntiles * g.groups, a.steps, sm_count, kBlocksPerSm<T, TN>);
  if (vtiles * s > 0x7fffffffLL || ntiles > 65535 || g.groups > 65535) return D2C_ERR_TOO_LARGE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(vtiles * s), (unsigned)ntiles, (unsigned)g.groups);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)s; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  D2C_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, g, Index::of(g), coords, a));
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

template <typename T, typename Coords, int kRoute>
int launch_fwd_route(const Geom& g, const Coords& coords, const FwdArgs<T>& a, cudaStream_t st) {
  switch (tile_n<T>(g)) {
    case 32: return launch_fwd_tn<T, 32, Coords, kRoute>(g, coords, a, st);
    case 64: return launch_fwd_tn<T, 64, Coords, kRoute>(g, coords, a, st);
    default:
      if constexpr (sizeof(T) == 4) return launch_fwd_tn<T, 128, Coords, kRoute>(g, coords, a, st);
      return D2C_ERR_SHAPE;
  }
}

template <typename T, typename Coords>
int launch_fwd(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* w, const T* bias, T* y, void* ws,
               cudaStream_t st) {
  constexpr bool k1d = CoordsIs1d<Coords>::value;
  if (too_large(g)) return D2C_ERR_TOO_LARGE;
  const Route route = route_of(g, k1d);
  FwdArgs<T> a{x, mask, w, bias, y, 0, 0, (g.cin_g * g.K + kTK - 1) / kTK};
  prof_mark(st, "fwd_generic");
  int rc;
  if (route == kChannelsLast) {
    if constexpr (!k1d) {
      a.Rp = (int)align_up((size_t)g.cin_g * g.K, kTK);
      a.Np = (int)align_up(g.cout_g, tile_n<T>(g));
      T* x_cl = reinterpret_cast<T*>(ws);
      T* w_st = reinterpret_cast<T*>(reinterpret_cast<uint8_t*>(ws) + x_cl_bytes<T>(g));
      if ((rc = launch_stage<T>(g, StageArgs<T>{x, x_cl, w, w_st, 0, a.Rp, a.Np, 0, {}}, st))) return rc;
      a.x = x_cl; a.w = w_st;
      rc = launch_fwd_route<T, Coords, kChannelsLast>(g, coords, a, st);
    } else {
      rc = D2C_ERR_SHAPE;
    }
  } else if (route == kDirect) {
    rc = launch_fwd_route<T, Coords, kDirect>(g, coords, a, st);
  } else {
    rc = launch_fwd_route<T, Coords, kAny>(g, coords, a, st);
  }
  if (rc) return rc;
  prof_mark(st, nullptr);
  return D2C_OK;
}

template <typename T, int TN, typename Coords, int kRoute>
int launch_dw_tn(const Geom& g, const Coords& coords, DwArgs<T> a, int splits, cudaStream_t st) {
  constexpr auto kern = dw_kernel<T, TN, Coords, kRoute>;
  constexpr int smem = (int)gemm_smem<T, TN>();
  const int rc = allow_dynamic_smem<kern>(smem);
  if (rc) return rc;
  const int rtiles = (g.cin_g * g.K + kTM - 1) / kTM, ntiles = (g.cout_g + TN - 1) / TN;
  if ((long long)rtiles * splits > 0x7fffffffLL || ntiles > 65535 || g.groups > 65535) return D2C_ERR_TOO_LARGE;
  a.splits = splits;
  kern<<<dim3((unsigned)(rtiles * splits), (unsigned)ntiles, (unsigned)g.groups), kThreads, smem, st>>>(g, Index::of(g), coords, a);
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

template <typename T, typename Coords, int kRoute>
int launch_dw_route(const Geom& g, const Coords& coords, const DwArgs<T>& a, int splits, cudaStream_t st) {
  switch (tile_n<T>(g)) {
    case 32: return launch_dw_tn<T, 32, Coords, kRoute>(g, coords, a, splits, st);
    case 64: return launch_dw_tn<T, 64, Coords, kRoute>(g, coords, a, splits, st);
    default:
      if constexpr (sizeof(T) == 4) return launch_dw_tn<T, 128, Coords, kRoute>(g, coords, a, splits, st);
      return D2C_ERR_SHAPE;
  }
}

// Voxel ranges of the weight gradient: as pick_cluster, a range costs its steps plus about eight steps' worth of
// pipeline fill and reductions into grad_w.
inline int pick_splits(long long tiles, int steps, int sm_count, int per_sm) {
  int best = 1;
  double best_t = 0;
  const long long slots = (long long)sm_count * per_sm;
  for (int s = 1; s <= steps && s <= 256; ++s) {
    const long long waves = (tiles * s + slots - 1) / slots;
    const double t = (double)waves * ((double)((steps + s - 1) / s) + (s > 1 ? 8.0 : 4.0));
    if (s == 1 || t < best_t * 0.999) { best_t = t; best = s; }
  }
  return best;
}

template <typename T, typename Coords, bool FieldOut>
int launch_grad_cl(const Geom& g, const Coords& coords, GradArgs<T> a, int sm_count, cudaStream_t st) {
  const int chunks = g.cpg / 4;
  const int tpv = chunks >= 8 ? 8 : (chunks >= 4 ? 4 : (chunks >= 2 ? 2 : 1));
  const int vpb = 256 / tpv;
  const long long vblocks = (long long)((g.V + vpb - 1) / vpb) * a.nb * g.G;
  int split = (int)((4LL * sm_count + vblocks - 1) / vblocks);       // taps over blocks while the GPU is not full
  if (split > g.K) split = g.K;
  if (split > 9) split = 9;
  a.taps_per_block = (g.K + split - 1) / split;
  if (vblocks > 0x7fffffffLL) return D2C_ERR_TOO_LARGE;
  dim3 grid((unsigned)vblocks, (unsigned)((g.K + a.taps_per_block - 1) / a.taps_per_block));
  const Index ix = Index::of(g);
  switch (tpv) {
    case 8: grad_cl_kernel<T, Coords, FieldOut, 8><<<grid, 256, 0, st>>>(g, ix, coords, a); break;
    case 4: grad_cl_kernel<T, Coords, FieldOut, 4><<<grid, 256, 0, st>>>(g, ix, coords, a); break;
    case 2: grad_cl_kernel<T, Coords, FieldOut, 2><<<grid, 256, 0, st>>>(g, ix, coords, a); break;
    default: grad_cl_kernel<T, Coords, FieldOut, 1><<<grid, 256, 0, st>>>(g, ix, coords, a); break;
  }
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

template <typename T, typename Coords, bool FieldOut>
int launch_bwd(const Geom& g, const Coords& coords, const T* gy, const T* x, const T* mask, const T* w, T* grad_x, T* grad_coord,
               size_t grad_coord_elems, T* grad_mask, T* grad_w, T* grad_bias, void* ws, unsigned long long cap, cudaStream_t st) {
  constexpr bool k1d = CoordsIs1d<Coords>::value;
  if (too_large(g)) return D2C_ERR_TOO_LARGE;
  const Route route = route_of(g, k1d);
  const int R = g.cin_g * g.K, nb_max = slice_clips(g, cap);
  const bool cl = route == kChannelsLast;
  int sm_count = 0, rc;
  if ((rc = device_sm_count(&sm_count))) return rc;
  uint8_t* wsp = reinterpret_cast<uint8_t*>(ws);
  T* dcol = reinterpret_cast<T*>(wsp); wsp += align_up(sizeof(T) * (size_t)nb_max * g.Cin * g.K * g.V, 256);
  T *x_cl = nullptr, *gx_cl = nullptr, *w_st = nullptr;
  if (cl) {
    x_cl = reinterpret_cast<T*>(wsp); wsp += x_cl_bytes<T>(g);
    gx_cl = reinterpret_cast<T*>(wsp); wsp += x_cl_bytes<T>(g);
    w_st = reinterpret_cast<T*>(wsp);
  }
  const int dw_steps = (int)(((long long)g.B * g.V + kTK - 1) / kTK);
  const int tn = tile_n<T>(g);
  const long long dw_tiles = (long long)((R + kTM - 1) / kTM) * ((g.cout_g + tn - 1) / tn) * g.groups;
  const int splits = pick_splits(dw_tiles, dw_steps, sm_count, sizeof(T) == 4 && tn < 128 ? 2 : 1);

  prof_mark(st, "bwd_stage_generic");
  const long long gw_bytes = splits > 1 ? (long long)sizeof(T) * g.Cout * R : 0;
  const int Rp = (int)align_up((size_t)R, 128), Np = (int)align_up(g.cout_g, kTK);
  if (FieldOut) D2C_CUDA_TRY(cudaMemsetAsync(grad_coord, 0, sizeof(T) * grad_coord_elems, st));
  if (cl) {
    StageArgs<T> sa{x, x_cl, w, w_st, 1, Rp, Np, 0,
                    {{gx_cl, (long long)sizeof(T) * g.B * g.Vin * g.Cin}, {grad_w, gw_bytes},
                     {grad_bias, grad_bias ? (long long)sizeof(T) * g.Cout : 0}}};
    if ((rc = launch_stage<T>(g, sa, st))) return rc;
  } else {
    D2C_CUDA_TRY(cudaMemsetAsync(grad_x, 0, sizeof(T) * (size_t)g.B * g.Cin * g.Vin, st));
    if (gw_bytes) D2C_CUDA_TRY(cudaMemsetAsync(grad_w, 0, (size_t)gw_bytes, st));
    if (grad_bias) D2C_CUDA_TRY(cudaMemsetAsync(grad_bias, 0, sizeof(T) * g.Cout, st));
  }

  prof_mark(st, "bwd_dw_generic");
  {
    const DwArgs<T> a{cl ? x_cl : x, mask, gy, grad_w, grad_bias, dw_steps, 1, splits > 1 ? 1 : 0};
    if (route == kAny) rc = launch_dw_route<T, Coords, kAny>(g, coords, a, splits, st);
    else if (route == kDirect) rc = launch_dw_route<T, Coords, kDirect>(g, coords, a, splits, st);
    else if constexpr (!k1d) rc = launch_dw_route<T, Coords, kChannelsLast>(g, coords, a, splits, st);
    if (rc) return rc;
  }

  const Index ix = Index::of(g);
  for (int b0 = 0; b0 < g.B; b0 += nb_max) {
    const int nb = (g.B - b0 < nb_max) ? g.B - b0 : nb_max;
    prof_mark(st, "bwd_dcol_generic");
    const long long vtiles = ((long long)nb * g.V + kTM - 1) / kTM;
    const long long dblocks = vtiles * ((R + kDcolN<T> - 1) / kDcolN<T>);
    if (dblocks > 0x7fffffffLL || g.groups > 65535) return D2C_ERR_TOO_LARGE;
    dim3 grid((unsigned)dblocks, (unsigned)g.groups);
    const DcolArgs<T> da{gy, cl ? w_st : w, dcol, Rp, Np, b0, nb};
    constexpr int smem = (int)gemm_smem<T, kDcolN<T>>();
    if ((rc = cl ? allow_dynamic_smem<dcol_kernel<T, kChannelsLast>>(smem) : allow_dynamic_smem<dcol_kernel<T, kDirect>>(smem)))
      return rc;
    if (cl) dcol_kernel<T, kChannelsLast><<<grid, kThreads, smem, st>>>(g, ix, da);
    else dcol_kernel<T, kDirect><<<grid, kThreads, smem, st>>>(g, ix, da);
    D2C_LAUNCH_CHECK();
    prof_mark(st, "bwd_sample_grad_generic");
    const GradArgs<T> ga{dcol, cl ? x_cl : x, mask, grad_coord, grad_mask, cl ? gx_cl : grad_x, b0, nb, 0};
    if (cl) {
      if constexpr (!k1d) {
        if ((rc = launch_grad_cl<T, Coords, FieldOut>(g, coords, ga, sm_count, st))) return rc;
      }
    } else {
      const long long blocks = (long long)((g.V + 31) / 32) * nb * g.G * g.K;
      if (blocks > 0x7fffffffLL) return D2C_ERR_TOO_LARGE;
      grad_direct_kernel<T, Coords, FieldOut><<<(unsigned)blocks, 256, 0, st>>>(g, ix, coords, ga);
      D2C_LAUNCH_CHECK();
    }
  }
  if (cl) {
    prof_mark(st, "bwd_unstage_generic");
    dim3 grid((unsigned)((g.Vin + 31) / 32), (unsigned)((g.Cin + 31) / 32), (unsigned)g.B);
    if (grid.y > 65535 || grid.z > 65535) return D2C_ERR_TOO_LARGE;
    unstage_kernel<T><<<grid, 256, 0, st>>>(g, gx_cl, grad_x);
    D2C_LAUNCH_CHECK();
  }
  prof_mark(st, nullptr);
  return D2C_OK;
}

}  // namespace exact
}  // namespace d2c
