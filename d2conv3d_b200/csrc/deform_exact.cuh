// Exact tier of the deformable convolutions: any geometry, fp32 / fp64, every product and sum on the FMA pipe (the
// results of an S/Dgemm up to summation order; fp64 supports gradcheck).  The tensor-core tier (deform_sm100_*.cu)
// replaces these kernels for the shapes it takes.
//
// Forward, gradient columns and weight gradient are one persistent GEMM kernel with three operand sources: block tiles of
// 256 x N, 16 contraction rows per step, a ring of stages in shared memory, eight warps that multiply and eight that
// produce operands.  In the forward and the weight gradient the 256-wide operand is SAMPLED by the producers (an item =
// four channels of one voxel and tap: position, eight corner loads, blend), so no column matrix exists; only the
// backward's gradient columns are written to memory.  Forward: the CTAs of a cluster share a tile's contraction and add
// their accumulators through distributed shared memory in rank order (reproducible, no workspace).  Gradient columns: a CTA
// takes a range of whole tiles.  Weight gradient: a CTA takes a range of (tile, step) units, shared tiles are added up with
// reductions.
//
// What shapes it (B200: 128 fp32 FMA per clock and SM, one issue slot per scheduler and clock, 32 registers per clock
// delivered by the load-store unit):
//   * fp32 products are packed (fma.rn.f32x2): a warp that multiplies leaves half the issue slots to the producers.  The
//     pairs run along the sampled operand, the other one is broadcast in registers.
//   * a thread owns 16 x 8 accumulators and reads 16 + 8 registers per contraction row: 96 load cycles per SM and row beside
//     128 FMA cycles.  With broadcast pairs read from shared memory it was 128, with 8 x 8 accumulators 192, and the
//     load-store unit was the limit (gradient columns below: 407 and 318 us).
//   * sampling in the threads that multiply kept the FMA pipe at 37 % (two warps per scheduler, each waiting for its own
//     corners); separate warps hide the gather, and hand-over is one mbarrier per stage.
//   * the input is staged channels-last (route kChannelsLast), so a 16-byte load fetches four channels of a corner and
//     the loads of four neighbouring threads are one 64-byte run.  Below 16 channels, and for the 1-D op, whose
//     positions are already neighbours along a row, the samples are taken from the NCDHW tensor itself (kDirect).
//
// 128 -> 128 channels, one clip of 8 x 30 x 54, 4 offset groups, forward + backward: 6.37 ms with scalar 64 x 64 tiles and
// separate coordinate / scatter passes over channel-major columns; 1.45 ms now (forward 0.49, weight gradient 0.39, columns
// 0.26, sampling gradient 0.27).  What bounds it: the producers' gather latency in the forward (51 tiles shared by pairs of
// CTAs) and the weight gradient, the FMA pipe in the columns, L2 reductions in the sampling gradient.
#pragma once

#include <algorithm>

#include "deform_exact.h"
#include "sm100_ptx.cuh"

namespace d2c {
namespace exact {

constexpr int kTM = 256;          // rows of a block tile (voxels, or column rows in the weight gradient)
constexpr int kRows = 16;         // rows per multiplying thread
constexpr int kStages = 4;
constexpr int kConsumers = 256, kProducers = 256, kThreads = kConsumers + kProducers;
constexpr int kPitchA = kTM + 4;                      // elements; keeps 16-byte alignment and spreads the stores

// ---- element types -----------------------------------------------------------------------------------

using u64 = unsigned long long;

// One thread's accumulators: 16 rows x N columns.
template <typename T, int N> struct Acc;
template <int N> struct Acc<float, N> {
  u64 v[kRows / 2][N];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < kRows / 2; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) v[i][j] = 0ull;
  }
  __device__ __forceinline__ float at(int i, int j) const {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[i / 2][j]));
    return (i & 1) ? hi : lo;
  }
};
template <int N> struct Acc<double, N> {
  double v[kRows][N];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < kRows; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) v[i][j] = 0.0;
  }
  __device__ __forceinline__ double at(int i, int j) const { return v[i][j]; }
};

// Place of a multiplying thread: half of the rows, 8 x 16 threads inside it; a warp covers 8 x 4.
struct Lane {
  int half, tx, ty;
  __device__ __forceinline__ explicit Lane(int t) : half(t >> 7), tx(t & 7), ty((t >> 3) & 15) {}
  // row i (0..15) of the thread inside the tile: runs of four
  __device__ __forceinline__ int row(int i) const { return half * 128 + (i >> 2) * 32 + tx * 4 + (i & 3); }
  // column j of the thread's TN/16 columns: runs of four (two where there are only two)
  template <int TN>
  __device__ __forceinline__ int col(int j) const {
    return TN == 128 ? (j >> 2) * 64 + ty * 4 + (j & 3) : (TN == 64 ? ty * 4 + j : ty * 2 + j);
  }
};

// {a, a}; volatile, so that it is made once and not again before every use
__device__ __forceinline__ u64 bcast2(float a) {
  u64 r;
  asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

// acc += A[k][rows] * B[k][cols] over the 16 rows of a stage
template <typename T, int TN>
__device__ __forceinline__ void stage_fma(const T* As, const T* Bs, const Lane& L, Acc<T, TN / 16>& acc) {
  constexpr int N = TN / 16;
  const T* arow = As + L.half * 128 + L.tx * 4;
#pragma unroll 4
  for (int k = 0; k < kTK; ++k) {
    T b[N];
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      const T* src = Bs + k * kPitchB<TN> + L.template col<TN>(j);
      if constexpr (sizeof(T) == 4 && N >= 4) {
        if (j % 4 == 0) {
          const float4 q = *reinterpret_cast<const float4*>(src);
          b[j] = q.x; b[j + 1] = q.y; b[j + 2] = q.z; b[j + 3] = q.w;
        }
      } else if constexpr (sizeof(T) == 4) {
        const float2 q = *reinterpret_cast<const float2*>(src);
        b[j] = q.x; b[j + 1] = q.y;
      } else {
        const double2 q = *reinterpret_cast<const double2*>(src);
        b[j] = q.x; b[j + 1] = q.y;
      }
    }
    if constexpr (sizeof(T) == 4) {
      u64 bb[N];
#pragma unroll
      for (int j = 0; j < N; ++j) bb[j] = bcast2(b[j]);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(arow + k * kPitchA + m * 32);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc.v[2 * m][j]) : "l"(a.x), "l"(bb[j]));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc.v[2 * m + 1][j]) : "l"(a.y), "l"(bb[j]));
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const double2 a = *reinterpret_cast<const double2*>(arow + k * kPitchA + (m >> 1) * 32 + (m & 1) * 2);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          acc.v[2 * m][j] = __fma_rn(a.x, b[j], acc.v[2 * m][j]);
          acc.v[2 * m + 1][j] = __fma_rn(a.y, b[j], acc.v[2 * m + 1][j]);
        }
      }
    }
  }
}

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  // volatile (must not be dropped) but no memory clobber: read-only loads may move across it
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d));
}
__device__ __forceinline__ void red_add4(double* p, double a, double b, double c, double d) {
  atomicAdd(p, a); atomicAdd(p + 1, b); atomicAdd(p + 2, c); atomicAdd(p + 3, d);
}

// ---- the GEMM ------------------------------------------------------------------------------------------

// Units of one launch: unit u = step u % steps of tile u / steps.
struct Units {
  long long tiles;
  int steps;
};
// How CTAs share them: one range of units each; one range of whole tiles each; the CTAs of a cluster one tile.
enum class Split { units, tiles, cluster };

template <typename T, int TN>
constexpr size_t gemm_ring() { return (size_t)kStages * kTK * (kPitchB<TN> + kPitchA) * sizeof(T); }

template <typename T, int TN>
constexpr size_t gemm_smem() {
  const size_t part = (size_t)TN * kPitchA * sizeof(T);
  return gemm_ring<T, TN>() > part ? gemm_ring<T, TN>() : part;
}

// Registers: the launch gives every thread 128 (512 threads x 128 = the whole file) and the two roles re-divide them.  A
// multiplying thread holds up to 128 registers of accumulators, a producing one 32 (fp64: 64) of corner values per item.
// Register split for a tile of TN columns.  Wide fp32 tiles: the gradient columns' producers only copy and leave 200 to
// the multiplying warps (fragments of the next row in flight: 356 -> 262 us at the size named at the top).
template <typename T, int TN, typename Op>
constexpr int kConsumerRegs = TN * (int)sizeof(T) == 512 ? (Op::kSplit == Split::tiles ? 200 : 168)
                                                         : TN * (int)sizeof(T) == 256 ? 120 : 96;
template <typename T, int TN, typename Op> constexpr int kProducerRegs = 256 - kConsumerRegs<T, TN, Op>;
static_assert(kConsumers == kProducers && kThreads * 128 == 65536, "the two shares add up to the register file");

template <int kRegs>
__device__ __forceinline__ void set_registers() {
  if constexpr (kRegs > 128) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
  else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// Op: `units`; Producer with begin(tile, s_beg, s_end), fill(step, As, Bs), end(); kBulk: the B tile of a step is one
// contiguous image b_image(tile, step) and arrives by bulk copy; epilogue(tile, first, last, lane, acc), or for clusters
// store(tile, row, column, 16 bytes of consecutive rows).
template <typename T, int TN, typename Op>
__global__ void __launch_bounds__(kThreads, 1) gemm_kernel(const __grid_constant__ Op op) {
  constexpr int kA = kTK * kPitchA, kB = kTK * kPitchB<TN>;
  extern __shared__ __align__(128) unsigned char smem[];
  T* const Bs = reinterpret_cast<T*>(smem);
  T* const As = reinterpret_cast<T*>(smem + (size_t)kStages * kB * sizeof(T));
  __shared__ __align__(8) u64 bars[2 * kStages];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(full(s), kProducers / 32 + (Op::kBulk ? 1 : 0));
      ptx::mbar_init(empty(s), kConsumers / 32);
    }
    abort_word = 0;
    ptx::fence_mbar_init();
  }
  __syncthreads();
  const int steps = op.units.steps;
  int ranks = 1;
  if constexpr (Op::kSplit == Split::cluster) ranks = op.ranks;
  const int rank = (int)(blockIdx.x % ranks);
  long long u_beg, u_end;
  if constexpr (Op::kSplit == Split::cluster) {
    u_beg = (long long)(blockIdx.x / ranks) * steps + (long long)steps * rank / ranks;
    u_end = (long long)(blockIdx.x / ranks) * steps + (long long)steps * (rank + 1) / ranks;
  } else if constexpr (Op::kSplit == Split::tiles) {
    u_beg = op.units.tiles * blockIdx.x / gridDim.x * steps;
    u_end = op.units.tiles * (blockIdx.x + 1) / gridDim.x * steps;
  } else {
    u_beg = op.units.tiles * steps * blockIdx.x / gridDim.x;
    u_end = op.units.tiles * steps * (blockIdx.x + 1) / gridDim.x;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < kConsumers / 32) {
    set_registers<kConsumerRegs<T, TN, Op>>();
    const Lane L(threadIdx.x);
    Acc<T, TN / 16> acc;
    uint32_t q = 0;
    bool ok = true;
    for (long long u = u_beg; ok && u < u_end;) {
      const long long tile = u / steps;
      const int s_beg = (int)(u - tile * steps), s_end = (int)min((long long)steps, s_beg + (u_end - u));
      acc.clear();
      for (int s = s_beg; s < s_end; ++s, ++q) {
        const int st = q % kStages;
        if (!ptx::mbar_wait(full(st), (q / kStages) & 1, abort_flag)) { ok = false; break; }
        stage_fma<T, TN>(As + st * kA, Bs + st * kB, L, acc);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(empty(st));
      }
      if constexpr (Op::kSplit == Split::cluster) {
        // the ring becomes the CTA's partial tile [column][row]: every multiplying warp is done with it
        asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory");
        T* part = reinterpret_cast<T*>(smem);
        if (ok) {
#pragma unroll
          for (int j = 0; j < TN / 16; ++j)
#pragma unroll
            for (int i = 0; i < kRows; ++i) part[L.template col<TN>(j) * kPitchA + L.row(i)] = acc.at(i, j);
        }
      } else {
        if (ok) op.epilogue(tile, s_beg == 0, s_end == steps, L, acc);
      }
      u += s_end - s_beg;
    }
  } else {
    set_registers<kProducerRegs<T, TN, Op>>();
    const int t = threadIdx.x - kConsumers;
    typename Op::Producer prod(op, t);
    uint32_t q = 0;
    bool ok = true;
    for (long long u = u_beg; ok && u < u_end;) {
      const long long tile = u / steps;
      const int s_beg = (int)(u - tile * steps), s_end = (int)min((long long)steps, s_beg + (u_end - u));
      prod.begin(tile, s_beg, s_end);
      for (int s = s_beg; s < s_end; ++s, ++q) {
        const int st = q % kStages;
        if (!ptx::mbar_wait(empty(st), ((q / kStages) & 1) ^ 1, abort_flag)) { ok = false; break; }
        if constexpr (Op::kBulk) {
          if (t == 0) {
            ptx::mbar_arrive_expect_tx(full(st), kB * sizeof(T));
            ptx::bulk_g2s(ptx::smem_u32(Bs + st * kB), op.b_image(tile, s), kB * sizeof(T), full(st));
          }
        }
        prod.fill(s, As + st * kA, Bs + st * kB);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(full(st));
      }
      if (ok) prod.end();
      u += s_end - s_beg;
    }
    if (Op::kBulk && t == 0) {       // never leave with a bulk copy in flight
      for (uint32_t w = (q > (uint32_t)kStages ? q - kStages : 0); w < q; ++w) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(full(w % kStages), (w / kStages) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
    }
  }
  if constexpr (Op::kSplit == Split::cluster) {
    if (ranks > 1) ptx::cluster_sync();
    else __syncthreads();
    // rank by rank, so that the sum does not depend on timing
    const uint32_t part = ptx::smem_u32(smem);
    constexpr int kVec = 16 / sizeof(T);
    for (int e = rank * kThreads + threadIdx.x; e < TN * (kTM / kVec); e += ranks * kThreads) {
      const int col = e / (kTM / kVec), row = e % (kTM / kVec) * kVec;
      T sum[kVec];
#pragma unroll
      for (int i = 0; i < kVec; ++i) sum[i] = (T)0;
      for (int r = 0; r < ranks; ++r) {
        T v[kVec];
        ptx::ld_cluster_16(ptx::mapa_shared(part + (uint32_t)((col * kPitchA + row) * sizeof(T)), (uint32_t)r), v);
#pragma unroll
        for (int i = 0; i < kVec; ++i) sum[i] += v[i];
      }
      op.store(blockIdx.x / ranks, row, col, sum);
    }
    if (ranks > 1) ptx::cluster_sync();        // nobody leaves while its tile is being read
    else __syncthreads();
  } else {
    __syncthreads();
  }
  if (threadIdx.x == 0 && abort_word) ptx::report_device_timeout();
}

// ---- index arithmetic ----------------------------------------------------------------------------------

// Division of 0 <= n < 2^31 by a divisor known on the host: multiply by its scaled reciprocal and shift (Granlund and Montgomery,
// "Division by Invariant Integers using Multiplication", PLDI 1994).
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

template <typename T> __device__ __forceinline__ void load4(const T* p, T (&o)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
  } else {
    const double2 f = __ldg(reinterpret_cast<const double2*>(p)), h = __ldg(reinterpret_cast<const double2*>(p) + 1);
    o[0] = f.x; o[1] = f.y; o[2] = h.x; o[3] = h.y;
  }
}

// ---- sampling of one item: four channels of one (voxel, tap) ------------------------------------------------

template <typename T> struct Corners { T c[8][4]; };

// Issues the corner loads from the NCDHW tensor (0 where a corner does not contribute).  1-D: corners 0 and 1 only.
template <typename T, bool k1d>
__device__ __forceinline__ void load_corners(const Geom& g, const T* __restrict__ x, int b, int ch, const Pos<T>& p, bool ok,
                                             Corners<T>& out) {
  const Sample<T> s = make_sample(g, p.z, p.y, p.x);
  const unsigned valid = (ok && s.inside) ? s.valid : 0u;
  const long long lin = ((long long)s.z0 * g.H + s.y0) * g.W + s.x0;
#pragma unroll
  for (int q = 0; q < (k1d ? 2 : 8); ++q) {
    const long long at = lin + (q >> 2) * ((long long)g.H * g.W) + ((q >> 1) & 1) * g.W + (q & 1);
    const bool on = (valid >> q) & 1u;
    const T* src = x + ((long long)b * g.Cin + ch) * g.Vin + at;
#pragma unroll
    for (int e = 0; e < 4; ++e) out.c[q][e] = on ? __ldg(src + e * g.Vin) : (T)0;
  }
}

// Channels-last sampling, four items at a time.  The S = 4, 2 or 1 neighbouring threads whose chunks have the tap and the
// offset group in common (16, 8 or 4 channels) share positions, corners and weights: each works out 4 / S of the four
// items and the others get them by shuffles (10 per item instead of about 100 instructions).
template <typename T>
struct SharedSample {
  int off;             // element offset of corner 000 inside the clip, without the channel
  int b;               // clip
  unsigned valid;      // corners to read; none: the sample is zero
  T a[8], m;
  __device__ __forceinline__ void set(const Geom& g, const Pos<T>& p, const Voxel& vx, bool ok) {
    const Sample<T> s = make_sample(g, p.z, p.y, p.x);
    const bool in = ok && s.inside;
    valid = in ? s.valid : 0u;
    off = ((s.z0 * g.H + s.y0) * g.W + s.x0) * g.Cin;
    b = vx.b;
    sample_weights(s, a);
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = in ? a[q] : (T)0;
    m = in ? p.m : (T)0;
  }
};
// kBuf: items whose corners are in flight.
template <typename T, int S, int kBuf>
struct SharedSampler {
  SharedSample<T> mine[4 / S];
  Corners<T> cor[kBuf];
  __device__ __forceinline__ int owner(int h) const { return ((threadIdx.x & 31) & ~(S - 1)) | (h & (S - 1)); }
  template <typename V> __device__ __forceinline__ V from(V v, int h) const {
    return S == 1 ? v : __shfl_sync(0xffffffffu, v, owner(h));
  }
  __device__ __forceinline__ void load(const Geom& g, const T* __restrict__ x, int ch, int h) {
    const SharedSample<T>& sh = mine[h / S];
    const int off = from(sh.off, h), b = from(sh.b, h);
    const unsigned valid = from(sh.valid, h);
    const T* src = x + (long long)b * g.Vin * g.Cin + (off + ch);
    const int dx = g.Cin, dy = g.W * g.Cin, dz = g.H * g.W * g.Cin;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      T (&c)[4] = cor[h % kBuf].c[q];
      if ((valid >> q) & 1u) load4(src + ((q >> 2) * dz + ((q >> 1) & 1) * dy + (q & 1) * dx), c);
      else c[0] = c[1] = c[2] = c[3] = (T)0;
    }
  }
  // the interpolation chain and roundings of the reference (csrc/ops/dconv3d_gpu.cu:48-109, 184-199)
  __device__ __forceinline__ void blend(int h, T (&out)[4]) const {
    const SharedSample<T>& sh = mine[h / S];
    T r[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const T a = from(sh.a[q], h);
#pragma unroll
      for (int e = 0; e < 4; ++e) r[e] = fma_rn(cor[h % kBuf].c[q][e], a, r[e]);
    }
    const T m = from(sh.m, h);
#pragma unroll
    for (int e = 0; e < 4; ++e) out[e] = mul_rn(m, r[e]);
  }
};

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
  int transposed;                      // contraction runs over 0: column rows (forward), 1: output channels (gradient columns)
  int tn, steps;                       // columns of a B tile, 16-row steps
  long long x_blocks;
  ZeroFill zero[3];
};

// One launch: blocks below x_blocks transpose 32 voxels x 32 channels of x, the rest 32 x 32 pieces of the weights into the
// images of the GEMM's B tiles, [weight group][column tile][step][16 rows][tn + 4], zero-padded at the ends.  Column rows
// run (tap, channel).
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
  const int cols = p.transposed ? R : g.cout_g, ctiles = (cols + p.tn - 1) / p.tn;
  const int rb = (p.steps * kTK + 31) / 32, nb = ctiles * (p.tn / 32);       // blocks of contraction rows, of columns
  const long long blk = blockIdx.x - p.x_blocks;
  const int k0 = (int)(blk % rb) * 32, n0 = (int)((blk / rb) % nb) * 32, wg = (int)(blk / ((long long)rb * nb));
  // read with neighbouring threads on neighbouring column rows of the source
  for (int yy = ty; yy < 32; yy += 8) {
    const int r = (p.transposed ? n0 : k0) + tx, n = (p.transposed ? k0 : n0) + yy;
    T v = (T)0;
    if (r < R && n < g.cout_g) {
      const int tap = r / g.cin_g, c = r - tap * g.cin_g;
      v = __ldg(p.w + ((long long)(wg * g.cout_g + n)) * R + (long long)c * g.K + tap);
    }
    if (p.transposed) tile[yy][tx] = v;
    else tile[tx][yy] = v;
  }
  __syncthreads();
  for (int kk = ty; kk < 32; kk += 8) {
    const int k = k0 + kk, n = n0 + tx;
    if (k < p.steps * kTK)
      p.w_st[((((long long)wg * ctiles + n / p.tn) * p.steps + k / kTK) * kTK + k % kTK) * (p.tn + 4) + n % p.tn] = tile[kk][tx];
  }
}

// ---- forward: y[b, co, v] = sum_r W[co, r] * sample(b, r, v) + bias[co] ------------------------------------------

// Tiles: 256 voxels of the flattened (clip, voxel) range x TN output channels of a weight group, voxels fastest.
template <typename T, int TN, typename Coords, int kRoute>
struct FwdOp {
  static constexpr bool k1d = CoordsIs1d<Coords>::value;
  static constexpr bool kBulk = kRoute == kChannelsLast;
  static constexpr Split kSplit = Split::cluster;
  Units units;
  int ranks;           // CTAs of a cluster
  Geom g;
  Index ix;
  Coords coords;
  const T* x;          // NCDHW, or its channels-last copy
  const T* mask;
  const T* w;          // the weights as given ...
  const T* w_st;       // ... or their tile images
  const T* bias;
  T* y;
  int vtiles, ntiles, vec;   // vec: 16 bytes of consecutive voxels lie in one clip, 16-byte aligned
  int share;                 // neighbouring threads that share samples (kChannelsLast)

  __device__ __forceinline__ void split_tile(long long tile, long long& v0, int& n0, int& wg) const {
    const int vt = (int)(tile % vtiles), r = (int)(tile / vtiles);
    v0 = (long long)vt * kTM;
    n0 = (r % ntiles) * TN;
    wg = r / ntiles;
  }
  __device__ __forceinline__ const T* b_image(long long tile, int s) const {
    return w_st + ((tile / vtiles) * units.steps + s) * (kTK * kPitchB<TN>);
  }

  struct Producer {
    static constexpr int kDirW = kTK * TN / kProducers;     // weights a thread fetches per step when they are not staged
    // next to a 128-column tile one item in flight spills already (offsets, channels-last: 544 bytes stored, 548 loaded) and two
    // spill twice that: 492 us with one, 545 with two
    static constexpr int kBuf = sizeof(T) == 8 || TN == 128 ? 1 : 2;
    const FwdOp& op;
    const int t, R;
    int n0, wg, s_end;
    long long v0;
    Voxel vx;            // kDirect, kAny: the thread's voxel
    Pos<T> pos[4];       // of the next items: four (fewer where threads share), kDirect: one
    __device__ __forceinline__ Producer(const FwdOp& o, int tt) : op(o), t(tt), R(o.g.cin_g * o.g.K) {}
    __device__ __forceinline__ void begin(long long tile, int s_beg, int s_last) {
      op.split_tile(tile, v0, n0, wg);
      s_end = s_last;
      vx.set(op.g, op.ix, v0 + t, (long long)op.g.B * op.g.V, 0);
      if constexpr (kRoute == kDirect) fetch_direct(s_beg, 0);
      if constexpr (kRoute == kChannelsLast) {
        switch (op.share) {
          case 4: fetch_cl<4>(s_beg); break;
          case 2: fetch_cl<2>(s_beg); break;
          default: fetch_cl<1>(s_beg); break;
        }
      }
    }
    __device__ __forceinline__ void fill(int s, T* As, T* Bs) {
      if constexpr (kRoute == kChannelsLast) {
        switch (op.share) {
          case 4: fill_cl<4>(s, As); break;
          case 2: fill_cl<2>(s, As); break;
          default: fill_cl<1>(s, As); break;
        }
      } else {
        fill_direct(s, As, Bs);
      }
    }
    __device__ __forceinline__ void end() {}

    // Channels-last: chunk t % 4 of the step's four, voxels t / 4 + 64 h: neighbouring threads read neighbouring channels.
    template <int S> __device__ __forceinline__ bool own_item(int s, int i, Voxel& v, Chunk& ck) const {
      const int row = s * kTK + 4 * (t & 3), h = i * S + (t & (S - 1));
      v.set(op.g, op.ix, v0 + (t >> 2) + 64 * h, (long long)op.g.B * op.g.V, 0);
      ck.set(op.g, op.ix, row < R ? row : 0, wg);
      return s < s_end && row < R && v.ok;
    }
    template <int S> __device__ __forceinline__ void fetch_cl(int s) {
#pragma unroll
      for (int i = 0; i < 4 / S; ++i) {
        Voxel v;
        Chunk ck;
        if (own_item<S>(s, i, v, ck)) pos[i] = position(op.g, op.coords, op.mask, v, ck);
      }
    }
    template <int S> __device__ __forceinline__ void fill_cl(int s, T* As) {
      SharedSampler<T, S, kBuf> sm;
      int ch = 0;
#pragma unroll
      for (int i = 0; i < 4 / S; ++i) {
        Voxel v;
        Chunk ck;
        const bool ok = own_item<S>(s, i, v, ck);
        sm.mine[i].set(op.g, pos[i], v, ok);
        ch = wg * op.g.cin_g + ck.c;
      }
      if constexpr (kBuf == 2) sm.load(op.g, op.x, ch, 0);
      fetch_cl<S>(s + 1);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        if constexpr (kBuf == 1) sm.load(op.g, op.x, ch, h);
        else if (h < 3) sm.load(op.g, op.x, ch, h + 1);
        T out[4];
        sm.blend(h, out);
#pragma unroll
        for (int e = 0; e < 4; ++e) As[(4 * (t & 3) + e) * kPitchA + (t >> 2) + 64 * h] = out[e];
      }
    }

    // Otherwise: chunks 0 .. 3 of voxel t: neighbouring threads read neighbouring voxels.
    __device__ __forceinline__ void fetch_direct(int s, int h) {
      const int row = s * kTK + 4 * h;
      if (s < s_end && row < R && vx.ok) {
        Chunk ck;
        ck.set(op.g, op.ix, row, wg);
        pos[0] = position(op.g, op.coords, op.mask, vx, ck);
      }
    }
    __device__ __forceinline__ void fill_direct(int s, T* As, T* Bs) {
      T wreg[kDirW];
      {
        const int row = s * kTK + (t & 15);
        int c;
        const int tap = op.ix.cin_g.divmod(min(row, R - 1), c);
#pragma unroll
        for (int j = 0; j < kDirW; ++j) {
          const int n = n0 + (t >> 4) + 16 * j;
          wreg[j] = (row < R && n < op.g.cout_g) ? __ldg(op.w + ((long long)(wg * op.g.cout_g + n)) * R + (long long)c * op.g.K + tap) : (T)0;
        }
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int row = s * kTK + 4 * h;
        T out[4];
        if constexpr (kRoute == kAny) {
          sample_any<T, Coords>(op.g, op.ix, op.coords, op.x, op.mask, vx, row, R, wg, out);
        } else {
          const bool ok = vx.ok && row < R;
          int c;
          op.ix.cin_g.divmod(ok ? row : 0, c);
          Corners<T> cor;
          load_corners<T, k1d>(op.g, op.x, vx.b, wg * op.g.cin_g + c, pos[0], ok, cor);
          const Pos<T> cur = pos[0];
          fetch_direct(h < 3 ? s : s + 1, (h + 1) & 3);
          blend_item<T, k1d>(op.g, cur, ok, cor, out);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) As[(4 * h + e) * kPitchA + t] = out[e];
        if (h == 0) {
#pragma unroll
          for (int j = 0; j < kDirW; ++j) Bs[(t & 15) * kPitchB<TN> + (t >> 4) + 16 * j] = wreg[j];
        }
      }
    }
  };

  template <int kVec>
  __device__ __forceinline__ void store(long long tile, int row, int col, T (&a)[kVec]) const {
    long long v0;
    int n0, wg;
    split_tile(tile, v0, n0, wg);
    const long long total = (long long)g.B * g.V, vox = v0 + row;
    if (vox >= total || n0 + col >= g.cout_g) return;
    int v;
    const int b = ix.V.divmod((int)vox, v);
    const int co = wg * g.cout_g + n0 + col;
    const T bb = bias ? __ldg(bias + co) : (T)0;
    T* dst = y + ((long long)b * g.Cout + co) * g.V + v;
#pragma unroll
    for (int e = 0; e < kVec; ++e) a[e] += bb;
    if (vec) {
      if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(dst) = make_float4(a[0], a[1], a[2], a[3]);
      else *reinterpret_cast<double2*>(dst) = make_double2(a[0], a[1]);
      return;
    }
#pragma unroll
    for (int e = 0; e < kVec; ++e) {
      if (vox + e < total) *dst = a[e];
      ++dst;
      if (++v == g.V) { v = 0; dst += ((long long)g.Cout - 1) * g.V; }   // the next clip's first voxel
    }
  }
};

// ---- gradient columns: dcol = sum_co W[co, r] * gy[b, co, v]  (reference dconv3d_gpu.cu:981-999) ------------------

// Tiles: 256 voxels of the flattened clips [b0, b0 + nb) x TN column rows of a weight group, column rows fastest (they share
// the grad_out tile, which then comes from L2).
template <typename T, int TN, int kRoute>
struct DcolOp {
  static constexpr bool kBulk = kRoute == kChannelsLast;
  static constexpr Split kSplit = Split::tiles;
  Units units;
  Geom g;
  Index ix;
  const T* gy;
  const T* w;          // the weights as given (column rows (channel, tap)) ...
  const T* w_st;       // ... or their tile images (column rows (tap, channel))
  T* dcol;             // kChannelsLast: [clip][tap][v][Cin]; otherwise [clip][Cin*K][v]
  int b0, nb, rtiles;
  long long vtiles;

  __device__ __forceinline__ void split_tile(long long tile, long long& v0, int& r0, int& wg) const {
    r0 = (int)(tile % rtiles) * TN;
    const long long r = tile / rtiles;
    v0 = (r % vtiles) * kTM;
    wg = (int)(r / vtiles);
  }
  __device__ __forceinline__ const T* b_image(long long tile, int s) const {
    const long long wg = tile / rtiles / vtiles;
    return w_st + ((wg * rtiles + tile % rtiles) * units.steps + s) * (kTK * kPitchB<TN>);
  }

  struct Producer {
    static constexpr int kDirW = kTK * TN / kProducers;
    const DcolOp& op;
    const int t, R;
    int r0, wg;
    bool ok;
    const T* src;
    __device__ __forceinline__ Producer(const DcolOp& o, int tt) : op(o), t(tt), R(o.g.cin_g * o.g.K) {}
    __device__ __forceinline__ void begin(long long tile, int, int) {
      long long v0;
      op.split_tile(tile, v0, r0, wg);
      ok = v0 + t < (long long)op.nb * op.g.V;
      int v = 0, bl = 0;
      if (ok) bl = op.ix.V.divmod((int)(v0 + t), v);
      src = op.gy + ((long long)(op.b0 + bl) * op.g.Cout + wg * op.g.cout_g) * op.g.V + v;
    }
    __device__ __forceinline__ void fill(int s, T* As, T* Bs) {
      T a[kTK];
      const T* p = src + (long long)s * kTK * op.g.V;
      if (ok && (s + 1) * kTK <= op.g.cout_g) {
#pragma unroll
        for (int j = 0; j < kTK; ++j) { a[j] = __ldg(p); p += op.g.V; }
      } else {
#pragma unroll
        for (int j = 0; j < kTK; ++j) { a[j] = ok && s * kTK + j < op.g.cout_g ? __ldg(p) : (T)0; p += op.g.V; }
      }
      if constexpr (!kBulk) {
#pragma unroll
        for (int j = 0; j < kDirW; ++j) {
          const int e = t + j * kProducers, co = s * kTK + e / TN, r = r0 + e % TN;
          const T v = (co < op.g.cout_g && r < R) ? __ldg(op.w + ((long long)(wg * op.g.cout_g + co)) * R + r) : (T)0;
          Bs[(e / TN) * kPitchB<TN> + e % TN] = v;
        }
      }
#pragma unroll
      for (int j = 0; j < kTK; ++j) As[j * kPitchA + t] = a[j];
    }
    __device__ __forceinline__ void end() {}
  };

  __device__ __forceinline__ void epilogue(long long tile, bool, bool, const Lane& L, const Acc<T, TN / 16>& acc) const {
    long long v0;
    int r0, wg;
    split_tile(tile, v0, r0, wg);
    const long long total = (long long)nb * g.V;
    const int R = g.cin_g * g.K;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const long long n = v0 + L.row(i);
      if (n >= total) continue;
      int v;
      const int bl = ix.V.divmod((int)n, v);
#pragma unroll
      for (int j = 0; j < TN / 16; j += 4) {
        const int r = r0 + L.template col<TN>(j);
        if (r >= R) continue;
        if constexpr (kRoute == kChannelsLast) {
          int c;
          const int tap = ix.cin_g.divmod(r, c);          // four rows of one tap: channel counts are multiples of four
          T* dst = dcol + (((long long)bl * g.K + tap) * g.V + v) * g.Cin + wg * g.cin_g + c;
          if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(dst) = make_float4(acc.at(i, j), acc.at(i, j + 1), acc.at(i, j + 2), acc.at(i, j + 3));
          } else {
            reinterpret_cast<double2*>(dst)[0] = make_double2(acc.at(i, j), acc.at(i, j + 1));
            reinterpret_cast<double2*>(dst)[1] = make_double2(acc.at(i, j + 2), acc.at(i, j + 3));
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (r + e < R) dcol[((long long)bl * g.Cin * g.K + (long long)wg * R + r + e) * g.V + v] = acc.at(i, j + e);
        }
      }
    }
  }
};

// ---- weight gradient: dW[co, r] = sum_{b, v} gy[b, co, v] * sample(b, r, v)  (reference dconv3d_gpu.cu:1037-1088) ---

// Tiles: 256 column rows x TN output channels of a weight group; the contraction runs over all voxels.  The tiles of the
// first column rows also sum grad_out over their voxels: grad_bias.
template <typename T, int TN, typename Coords, int kRoute>
struct DwOp {
  static constexpr bool k1d = CoordsIs1d<Coords>::value;
  static constexpr bool kBulk = false;
  static constexpr Split kSplit = Split::units;
  Units units;
  Geom g;
  Index ix;
  Coords coords;
  const T* x;
  const T* mask;
  const T* gy;
  T* grad_w;           // zeroed beforehand where tiles are shared
  T* grad_bias;        // nullable; zeroed beforehand
  int rtiles, ntiles;
  int share;           // neighbouring threads that share samples (kChannelsLast)

  __device__ __forceinline__ void split_tile(long long tile, int& r0, int& n0, int& wg) const {
    r0 = (int)(tile % rtiles) * kTM;
    const int r = (int)(tile / rtiles);
    n0 = (r % ntiles) * TN;
    wg = r / ntiles;
  }

  struct Producer {
    static constexpr int kLdB = kTK * TN / kProducers;
    static constexpr int kBuf = sizeof(T) == 8 ? 1 : 2;     // items in flight (392 us with two, 435 with one)
    const DwOp& op;
    const int t, R, total;
    int r0, n0, wg, s_end;
    bool want_bias;
    Chunk ck;            // kChannelsLast: the thread's chunk
    Pos<T> pos[4];       // of the next items: four (fewer where threads share), kDirect: one
    T bsum[kLdB];
    __device__ __forceinline__ Producer(const DwOp& o, int tt) : op(o), t(tt), R(o.g.cin_g * o.g.K), total(o.g.B * o.g.V) {}
    __device__ __forceinline__ void begin(long long tile, int s_beg, int s_last) {
      op.split_tile(tile, r0, n0, wg);
      s_end = s_last;
      want_bias = op.grad_bias != nullptr && r0 == 0;
#pragma unroll
      for (int j = 0; j < kLdB; ++j) bsum[j] = (T)0;
      if constexpr (kRoute == kDirect) fetch_direct(s_beg, 0);
      if constexpr (kRoute == kChannelsLast) {
        const int row = r0 + 4 * (t & 63);
        ck.set(op.g, op.ix, row < R ? row : 0, wg);
        switch (op.share) {
          case 4: fetch_cl<4>(s_beg); break;
          case 2: fetch_cl<2>(s_beg); break;
          default: fetch_cl<1>(s_beg); break;
        }
      }
    }
    __device__ __forceinline__ void fill(int s, T* As, T* Bs) {
      T breg[kLdB];
      {
        const int n = s * kTK + (t & 15);
        int v = 0, b = 0;
        const bool ok = n < total;
        if (ok) b = op.ix.V.divmod(n, v);
        const T* src = op.gy + ((long long)b * op.g.Cout + wg * op.g.cout_g + n0 + (t >> 4)) * op.g.V + v;
#pragma unroll
        for (int j = 0; j < kLdB; ++j) {
          breg[j] = (ok && n0 + (t >> 4) + 16 * j < op.g.cout_g) ? __ldg(src) : (T)0;
          src += 16 * (long long)op.g.V;
        }
      }
      if constexpr (kRoute == kChannelsLast) {
        switch (op.share) {
          case 4: fill_cl<4>(s, As); break;
          case 2: fill_cl<2>(s, As); break;
          default: fill_cl<1>(s, As); break;
        }
      } else {
        fill_direct(s, As);
      }
#pragma unroll
      for (int j = 0; j < kLdB; ++j) Bs[(t & 15) * kPitchB<TN> + (t >> 4) + 16 * j] = breg[j];
      if (want_bias) {
#pragma unroll
        for (int j = 0; j < kLdB; ++j) bsum[j] += breg[j];
      }
    }
    static __device__ __forceinline__ void store4(T* dst, const T (&out)[4]) {
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(dst) = make_float4(out[0], out[1], out[2], out[3]);
      } else {
        reinterpret_cast<double2*>(dst)[0] = make_double2(out[0], out[1]);
        reinterpret_cast<double2*>(dst)[1] = make_double2(out[2], out[3]);
      }
    }

    // Channels-last: chunk t % 64 (a warp reads 512 contiguous bytes where a tap has 128 channels) of voxels t / 64 + 4 h.
    template <int S> __device__ __forceinline__ bool own_item(int s, int i, Voxel& v) const {
      v.set(op.g, op.ix, s * kTK + (t >> 6) + 4 * (i * S + (t & (S - 1))), total, 0);
      return s < s_end && r0 + 4 * (t & 63) < R && v.ok;
    }
    template <int S> __device__ __forceinline__ void fetch_cl(int s) {
#pragma unroll
      for (int i = 0; i < 4 / S; ++i) {
        Voxel v;
        if (own_item<S>(s, i, v)) pos[i] = position(op.g, op.coords, op.mask, v, ck);
      }
    }
    template <int S> __device__ __forceinline__ void fill_cl(int s, T* As) {
      SharedSampler<T, S, kBuf> sm;
#pragma unroll
      for (int i = 0; i < 4 / S; ++i) {
        Voxel v;
        const bool ok = own_item<S>(s, i, v);
        sm.mine[i].set(op.g, pos[i], v, ok);
      }
      const int ch = wg * op.g.cin_g + ck.c;
      if constexpr (kBuf == 2) sm.load(op.g, op.x, ch, 0);
      fetch_cl<S>(s + 1);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        if constexpr (kBuf == 1) sm.load(op.g, op.x, ch, h);
        else if (h < 3) sm.load(op.g, op.x, ch, h + 1);
        T out[4];
        sm.blend(h, out);
        store4(As + ((t >> 6) + 4 * h) * kPitchA + 4 * (t & 63), out);
      }
    }

    // Otherwise: voxel t % 16, chunks t / 16 + 16 h.
    __device__ __forceinline__ int row_of(int h) const { return r0 + 4 * ((t >> 4) + 16 * h); }
    __device__ __forceinline__ void fetch_direct(int s, int h) {
      const int n = s * kTK + (t & 15);
      if (s < s_end && row_of(h) < R && n < total) {
        Voxel v;
        Chunk c;
        v.set(op.g, op.ix, n, total, 0);
        c.set(op.g, op.ix, row_of(h), wg);
        pos[0] = position(op.g, op.coords, op.mask, v, c);
      }
    }
    __device__ __forceinline__ void fill_direct(int s, T* As) {
      const int n = s * kTK + (t & 15);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        T out[4];
        if constexpr (kRoute == kAny) {
          Voxel v;
          v.set(op.g, op.ix, n, total, 0);
          sample_any<T, Coords>(op.g, op.ix, op.coords, op.x, op.mask, v, row_of(h), R, wg, out);
        } else {
          const bool ok = row_of(h) < R && n < total;
          int c;
          op.ix.cin_g.divmod(ok ? row_of(h) : 0, c);
          Corners<T> cor;
          load_corners<T, k1d>(op.g, op.x, op.ix.V.div(ok ? n : 0), wg * op.g.cin_g + c, pos[0], ok, cor);
          const Pos<T> cur = pos[0];
          fetch_direct(h < 3 ? s : s + 1, (h + 1) & 3);
          blend_item<T, k1d>(op.g, cur, ok, cor, out);
        }
        store4(As + (t & 15) * kPitchA + 4 * ((t >> 4) + 16 * h), out);
      }
    }
    __device__ __forceinline__ void end() {
      if (!want_bias) return;
#pragma unroll
      for (int j = 0; j < kLdB; ++j) {
        T sum = bsum[j];
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const int co = n0 + (t >> 4) + 16 * j;
        if ((t & 15) == 0 && co < op.g.cout_g) atomicAdd(op.grad_bias + wg * op.g.cout_g + co, sum);
      }
    }
  };

  __device__ __forceinline__ void epilogue(long long tile, bool first, bool last, const Lane& L, const Acc<T, TN / 16>& acc) const {
    int r0, n0, wg;
    split_tile(tile, r0, n0, wg);
    const int R = g.cin_g * g.K;
    const bool whole = first && last;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int r = r0 + L.row(i);
      if (r >= R) continue;
      int c;
      const int tap = ix.cin_g.divmod(r, c);
#pragma unroll
      for (int j = 0; j < TN / 16; ++j) {
        const int n = n0 + L.template col<TN>(j);
        if (n >= g.cout_g) continue;
        T* dst = grad_w + ((long long)(wg * g.cout_g + n)) * R + (long long)c * g.K + tap;
        if (whole) *dst = acc.at(i, j);
        else atomicAdd(dst, acc.at(i, j));
      }
    }
  }
};

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

// What the threads of a voxel need of one tap, made by one of them and passed on by shuffles.
template <typename T>
struct TapShare {
  int off;             // element offset of corner 000 inside the clip's channels-last tensors, without the channel
  unsigned bits;       // corners inside the volume (0-7), corners that take part in the scatter (8-15)
  T w[8];              // scatter weights x modulation
};

template <typename T, int TPV>
__device__ __forceinline__ TapShare<T> tap_from(const TapShare<T>& mine, int lane_of_voxel) {
  if constexpr (TPV == 1) return mine;
  TapShare<T> s;
  s.off = __shfl_sync(0xffffffffu, mine.off, lane_of_voxel, TPV);
  s.bits = __shfl_sync(0xffffffffu, mine.bits, lane_of_voxel, TPV);
#pragma unroll
  for (int q = 0; q < 8; ++q) s.w[q] = __shfl_sync(0xffffffffu, mine.w[q], lane_of_voxel, TPV);
  return s;
}

// Corner products of TPV taps, summed over the TPV threads of a voxel so that thread j ends with the eight sums of tap j:
// a reduce-scatter over the taps (7 shuffles per tap for eight threads; reducing every tap to all threads takes 24).
// body(tap, G) leaves the thread's own contribution in G.
template <typename T, int TPV, int kBit, typename Body>
__device__ __forceinline__ void reduce_taps(int tap, int j4, const Body& body, T (&G)[8]) {
  if constexpr (kBit == TPV) {
    body(tap, G);
  } else {
    T other[8];
    reduce_taps<T, TPV, kBit * 2>(tap, j4, body, G);
    reduce_taps<T, TPV, kBit * 2>(tap | kBit, j4, body, other);
    const bool hi = j4 & kBit;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const T keep = hi ? other[q] : G[q], give = hi ? G[q] : other[q];
      G[q] = keep + __shfl_xor_sync(0xffffffffu, give, kBit);
    }
  }
}

// Channels-last route: TPV threads per voxel, each four channels at a time of its group.  The block walks its taps TPV at a
// time: thread j works out position, corners and weights of tap j once for the whole voxel, then all of them go through the
// TPV taps (columns read, corner products, scatter), and thread j writes the gradients of tap j.  With every thread working
// out every tap the kernel spent 690 instructions per warp and tap and 373 us at the size named at the top.
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
  const T* dcol = p.dcol + ((long long)bl * g.K * g.V + vx.v) * g.Cin + grp * g.cpg;
  const long long dcol_tap = (long long)g.V * g.Cin;
  const int dx = g.Cin, dy = g.W * g.Cin, dz = g.H * g.W * g.Cin;
  T fsum[3] = {(T)0, (T)0, (T)0};
  const int tap_beg = blockIdx.y * p.taps_per_block, tap_end = min(g.K, tap_beg + p.taps_per_block);
  for (int tap0 = tap_beg; tap0 < tap_end; tap0 += TPV) {
    const int my_tap = tap0 + j4;
    Pos<T> pos{};
    Sample<T> s{};
    Chunk ck;
    ck.tap = min(my_tap, tap_end - 1); ck.grp = grp; ck.c = 0;
    ck.i = ix.kh.divmod(ix.kw.divmod(ck.tap, ck.k), ck.j);
    pos = position(g, coords, p.mask, vx, ck);
    s = make_sample(g, pos.z, pos.y, pos.x);
    TapShare<T> mine;
    mine.off = ((s.z0 * g.H + s.y0) * g.W + s.x0) * g.Cin;
    mine.bits = live ? s.valid : 0u;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      T w;
      if (scatter_weight(s, q, w) && ((mine.bits >> q) & 1u)) mine.bits |= 256u << q;
      mine.w[q] = w * pos.m;
    }
    auto body = [&](int t, T (&G)[8]) {
#pragma unroll
      for (int q = 0; q < 8; ++q) G[q] = (T)0;
      if (tap0 + t >= tap_end) return;                 // the same for the whole block
      const TapShare<T> ts = tap_from<T, TPV>(mine, t);
      const T* dc = dcol + (tap0 + t) * dcol_tap;
      for (int c4 = j4; c4 < chunks; c4 += TPV) {
        T d[4], xv[8][4];
        load4(dc + 4 * c4, d);
        const int at = ts.off + 4 * c4;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if ((ts.bits >> q) & 1u) load4(xb + at + ((q >> 2) * dz + ((q >> 1) & 1) * dy + (q & 1) * dx), xv[q]);
          else xv[q][0] = xv[q][1] = xv[q][2] = xv[q][3] = (T)0;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          G[q] += (d[0] * xv[q][0] + d[1] * xv[q][1]) + (d[2] * xv[q][2] + d[3] * xv[q][3]);
          if ((ts.bits >> (8 + q)) & 1u)
            red_add4(gxb + at + ((q >> 2) * dz + ((q >> 1) & 1) * dy + (q & 1) * dx), ts.w[q] * d[0], ts.w[q] * d[1], ts.w[q] * d[2],
                     ts.w[q] * d[3]);
        }
      }
    };
    T G[8];
    reduce_taps<T, TPV, 1>(0, j4, body, G);
    if (live && my_tap < tap_end)
      write_coord_grads<T, Coords, FieldOut>(g, p, coords, b, grp, my_tap, ck.i, ck.j, ck.k, vx.v, pos.m, s, G, fsum);
  }
  if constexpr (FieldOut) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int o = TPV / 2; o >= 1; o >>= 1) fsum[d] += __shfl_xor_sync(0xffffffffu, fsum[d], o);
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
  const int cols = a.transposed ? g.cin_g * g.K : g.cout_g;
  const long long wblocks = (long long)((a.steps * kTK + 31) / 32) * ((cols + a.tn - 1) / a.tn) * (a.tn / 32) * g.groups;
  if (a.x_blocks + wblocks > 0x7fffffffLL) return D2C_ERR_TOO_LARGE;
  stage_kernel<T><<<(unsigned)(a.x_blocks + wblocks), 256, 0, st>>>(g, a);
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

// Neighbouring chunks of four channels that are certain to have tap and offset group in common.
inline int sharing_threads(const Geom& g) {
  return g.cpg % 16 == 0 && g.cin_g % 16 == 0 ? 4 : (g.cpg % 8 == 0 && g.cin_g % 8 == 0 ? 2 : 1);
}

// CTAs of a launch that splits by units: one per multiprocessor, at least two steps each.
inline long long units_grid(const Units& u, int sm_count) {
  const long long most = (u.tiles * u.steps + 1) / 2;
  return most < sm_count ? most : sm_count;
}
// Whether some CTA of it ends inside a tile (then the output is accumulated).
inline bool shares_tiles(const Units& u, int sm_count) { return u.tiles % units_grid(u, sm_count) != 0; }

// Shared memory, and once per kernel and process (whose GPUs are alike) a register check and how many clusters of each size fit.
struct GemmSetup {
  int rc;
  int clusters[9];     // [size]: resident clusters, 0 where the size is not used
};
template <typename T, int TN, typename Op>
int setup_gemm(int sm_count, GemmSetup* out) {
  constexpr auto kern = gemm_kernel<T, TN, Op>;
  constexpr int smem = (int)gemm_smem<T, TN>();
  const int rc = allow_dynamic_smem<kern>(smem);
  if (rc) return rc;
  static const GemmSetup setup = [sm_count] {
    GemmSetup s{};
    // The roles divide 128 registers per thread between them; a build that launches with fewer would leave the
    // multiplying warps waiting for registers that never come.
    cudaFuncAttributes fa;
    s.rc = cudaFuncGetAttributes(&fa, kern) == cudaSuccess && fa.numRegs == 128 ? D2C_OK : D2C_ERR_CUDA;
    s.clusters[1] = sm_count;
    if (Op::kSplit == Split::cluster)
      for (int c = 2; c <= 8; ++c) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)c; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(c * sm_count), 1, 1);
        cfg.blockDim = dim3(kThreads, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &attr; cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&s.clusters[c], kern, &cfg) != cudaSuccess) {
          s.clusters[c] = 0;
          (void)cudaGetLastError();
        }
      }
    return s;
  }();
  ptx::bind_status_sink();
  *out = setup;
  return setup.rc;
}

// CTAs that share a tile's contraction: the cluster size with the shortest expected time.  A wave takes the steps of one
// CTA plus about four steps' worth of filling the ring and adding tiles; fewer than two steps per CTA do not pay.
inline int pick_cluster(long long tiles, int steps, const GemmSetup& setup) {
  int best = 1;
  double best_t = 0;
  for (int c = 1; c <= 8 && (c == 1 || steps >= 2 * c); ++c) {
    if (!setup.clusters[c]) continue;
    const double t = (double)((tiles + setup.clusters[c] - 1) / setup.clusters[c]) * ((steps + c - 1) / c + 4.0 + 0.25 * c);
    if (c == 1 || t < best_t) { best_t = t; best = c; }
  }
  return best;
}

template <typename T, int TN, typename Op>
int launch_gemm(Op& op, int sm_count, cudaStream_t st) {
  GemmSetup setup;
  const int rc = setup_gemm<T, TN, Op>(sm_count, &setup);
  if (rc) return rc;
  constexpr int smem = (int)gemm_smem<T, TN>();
  constexpr auto kern = gemm_kernel<T, TN, Op>;
  if constexpr (Op::kSplit == Split::cluster) {
    op.ranks = pick_cluster(op.units.tiles, op.units.steps, setup);
    if (op.units.tiles * op.ranks > 0x7fffffffLL) return D2C_ERR_TOO_LARGE;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)op.ranks; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(op.units.tiles * op.ranks), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    D2C_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, op));
  } else {
    const long long grid = Op::kSplit == Split::tiles ? std::min<long long>(op.units.tiles, sm_count) : units_grid(op.units, sm_count);
    kern<<<(unsigned)grid, kThreads, smem, st>>>(op);
  }
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

template <typename T, int TN, typename Coords, int kRoute>
int launch_fwd_tn(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* w, const T* bias, T* y, void* ws,
                  int sm_count, cudaStream_t st) {
  using Op = FwdOp<T, TN, Coords, kRoute>;
  constexpr int kVec = 16 / sizeof(T);
  const int vtiles = (int)(((long long)g.B * g.V + kTM - 1) / kTM), ntiles = (g.cout_g + TN - 1) / TN;
  const Units units{(long long)vtiles * ntiles * g.groups, (g.cin_g * g.K + kTK - 1) / kTK};
  Op op{units, 1, g, Index::of(g), coords, x, mask, w, nullptr, bias, y, vtiles, ntiles,
        g.V % kVec == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0, sharing_threads(g)};
  if constexpr (kRoute == kChannelsLast) {
    T* x_cl = reinterpret_cast<T*>(ws);
    T* w_st = reinterpret_cast<T*>(reinterpret_cast<uint8_t*>(ws) + x_cl_bytes<T>(g));
    const int rc = launch_stage<T>(g, StageArgs<T>{x, x_cl, w, w_st, 0, TN, units.steps, 0, {}}, st);
    if (rc) return rc;
    op.x = x_cl; op.w_st = w_st;
  }
  return launch_gemm<T, TN>(op, sm_count, st);
}

template <typename T, typename Coords, int kRoute>
int launch_fwd_route(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* w, const T* bias, T* y, void* ws,
                     int sm_count, cudaStream_t st) {
  switch (tile_n<T>(g)) {
    case 32: return launch_fwd_tn<T, 32, Coords, kRoute>(g, coords, x, mask, w, bias, y, ws, sm_count, st);
    case 64: return launch_fwd_tn<T, 64, Coords, kRoute>(g, coords, x, mask, w, bias, y, ws, sm_count, st);
    default:
      if constexpr (sizeof(T) == 4) return launch_fwd_tn<T, 128, Coords, kRoute>(g, coords, x, mask, w, bias, y, ws, sm_count, st);
      return D2C_ERR_SHAPE;
  }
}

template <typename T, typename Coords>
int launch_fwd(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* w, const T* bias, T* y, void* ws,
               cudaStream_t st) {
  constexpr bool k1d = CoordsIs1d<Coords>::value;
  if (too_large(g)) return D2C_ERR_TOO_LARGE;
  int sm_count = 0, rc;
  if ((rc = device_sm_count(&sm_count))) return rc;
  prof_mark(st, "fwd_generic");
  const Route route = route_of(g, k1d);
  if (route == kAny) rc = launch_fwd_route<T, Coords, kAny>(g, coords, x, mask, w, bias, y, ws, sm_count, st);
  else if (route == kDirect) rc = launch_fwd_route<T, Coords, kDirect>(g, coords, x, mask, w, bias, y, ws, sm_count, st);
  else if constexpr (!k1d) rc = launch_fwd_route<T, Coords, kChannelsLast>(g, coords, x, mask, w, bias, y, ws, sm_count, st);
  if (rc) return rc;
  prof_mark(st, nullptr);
  return D2C_OK;
}

// The weight gradient's units for a tile width (needed before the launch: shared tiles start from zero).
inline Units dw_units(const Geom& g, int tn) {
  return {(long long)((g.cin_g * g.K + kTM - 1) / kTM) * ((g.cout_g + tn - 1) / tn) * g.groups,
          (int)(((long long)g.B * g.V + kTK - 1) / kTK)};
}

template <typename T, int TN, typename Coords, int kRoute>
int launch_dw_tn(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* gy, T* grad_w, T* grad_bias,
                 int sm_count, cudaStream_t st) {
  DwOp<T, TN, Coords, kRoute> op{dw_units(g, TN), g, Index::of(g), coords, x, mask, gy, grad_w, grad_bias,
                                 (g.cin_g * g.K + kTM - 1) / kTM, (g.cout_g + TN - 1) / TN, sharing_threads(g)};
  return launch_gemm<T, TN>(op, sm_count, st);
}

template <typename T, typename Coords, int kRoute>
int launch_dw_route(const Geom& g, const Coords& coords, const T* x, const T* mask, const T* gy, T* grad_w, T* grad_bias,
                    int sm_count, cudaStream_t st) {
  switch (tile_n<T>(g)) {
    case 32: return launch_dw_tn<T, 32, Coords, kRoute>(g, coords, x, mask, gy, grad_w, grad_bias, sm_count, st);
    case 64: return launch_dw_tn<T, 64, Coords, kRoute>(g, coords, x, mask, gy, grad_w, grad_bias, sm_count, st);
    default:
      if constexpr (sizeof(T) == 4) return launch_dw_tn<T, 128, Coords, kRoute>(g, coords, x, mask, gy, grad_w, grad_bias, sm_count, st);
      return D2C_ERR_SHAPE;
  }
}

template <typename T, int kRoute>
int launch_dcol(const Geom& g, const T* gy, const T* w, const T* w_st, T* dcol, int b0, int nb, int sm_count,
                cudaStream_t st) {
  constexpr int TN = kDcolN<T>;
  const int rtiles = (g.cin_g * g.K + TN - 1) / TN;
  const long long vtiles = ((long long)nb * g.V + kTM - 1) / kTM;
  DcolOp<T, TN, kRoute> op{{vtiles * rtiles * g.groups, (g.cout_g + kTK - 1) / kTK}, g, Index::of(g), gy, w, w_st, dcol,
                           b0, nb, rtiles, vtiles};
  return launch_gemm<T, TN>(op, sm_count, st);
}

template <typename T, typename Coords, bool FieldOut>
int launch_grad_cl(const Geom& g, const Coords& coords, GradArgs<T> a, int sm_count, cudaStream_t st) {
  const int chunks = g.cpg / 4;
  const int tpv = chunks >= 8 ? 8 : (chunks >= 4 ? 4 : (chunks >= 2 ? 2 : 1));
  const int vpb = 256 / tpv;
  const long long vblocks = (long long)((g.V + vpb - 1) / vpb) * a.nb * g.G;
  int split = (int)((4LL * sm_count + vblocks - 1) / vblocks);       // taps over blocks while the GPU is not full,
  const int max_split = (g.K + tpv - 1) / tpv;                       // as many at a time as a voxel has threads
  if (split > max_split) split = max_split;
  a.taps_per_block = ((g.K + split - 1) / split + tpv - 1) / tpv * tpv;
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

  prof_mark(st, "bwd_stage_generic");
  const long long gw_bytes = shares_tiles(dw_units(g, tile_n<T>(g)), sm_count) ? (long long)sizeof(T) * g.Cout * R : 0;
  if (FieldOut) D2C_CUDA_TRY(cudaMemsetAsync(grad_coord, 0, sizeof(T) * grad_coord_elems, st));
  if (cl) {
    StageArgs<T> sa{x, x_cl, w, w_st, 1, kDcolN<T>, (g.cout_g + kTK - 1) / kTK, 0,
                    {{gx_cl, (long long)sizeof(T) * g.B * g.Vin * g.Cin}, {grad_w, gw_bytes},
                     {grad_bias, grad_bias ? (long long)sizeof(T) * g.Cout : 0}}};
    if ((rc = launch_stage<T>(g, sa, st))) return rc;
  } else {
    D2C_CUDA_TRY(cudaMemsetAsync(grad_x, 0, sizeof(T) * (size_t)g.B * g.Cin * g.Vin, st));
    if (gw_bytes) D2C_CUDA_TRY(cudaMemsetAsync(grad_w, 0, (size_t)gw_bytes, st));
    if (grad_bias) D2C_CUDA_TRY(cudaMemsetAsync(grad_bias, 0, sizeof(T) * g.Cout, st));
  }

  prof_mark(st, "bwd_dw_generic");
  if (route == kAny) rc = launch_dw_route<T, Coords, kAny>(g, coords, x, mask, gy, grad_w, grad_bias, sm_count, st);
  else if (route == kDirect) rc = launch_dw_route<T, Coords, kDirect>(g, coords, x, mask, gy, grad_w, grad_bias, sm_count, st);
  else if constexpr (!k1d) rc = launch_dw_route<T, Coords, kChannelsLast>(g, coords, x_cl, mask, gy, grad_w, grad_bias, sm_count, st);
  if (rc) return rc;

  const Index ix = Index::of(g);
  for (int b0 = 0; b0 < g.B; b0 += nb_max) {
    const int nb = (g.B - b0 < nb_max) ? g.B - b0 : nb_max;
    prof_mark(st, "bwd_dcol_generic");
    rc = cl ? launch_dcol<T, kChannelsLast>(g, gy, w, w_st, dcol, b0, nb, sm_count, st)
            : launch_dcol<T, kDirect>(g, gy, w, w_st, dcol, b0, nb, sm_count, st);
    if (rc) return rc;
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
