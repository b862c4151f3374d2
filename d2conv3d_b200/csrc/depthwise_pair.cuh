// fp32 / fp16 depthwise 3x3x3 kernels (stride 1, dilation 1, padding 1, channel multiplier 1, any size whose rows fit a
// block): a forward and a fused backward that produces grad_x and grad_w from one pass over grad_out and x.
//
// What shapes them (B200): per element the forward moves 8 (fp16: 4) bytes against 27 FMA, the backward 12 (6) against 54;
// at 23 bytes and 128 FMA per clock and SM neither side may waste its half.
//   * packed fp32 FMA (fma.rn.f32x2) over CHANNEL pairs: element and weight pairs are {channel c, channel c+1} at the same
//     place, so no tap needs a pair shifted by one column (x-adjacent pairs cost 4 moves and 2 selects per input row).
//   * a thread owns R = 4 rows of one column of one channel pair and marches along z: each plane's 6 x 3 neighbourhood is
//     read from shared memory once and scattered into the accumulators of three output planes.  Lanes run along x.
//   * the backward needs only grad_out's neighbourhood: grad_x(q) and grad_w both multiply the SAME neighbour grad_out(q - k),
//     by w(k) and by x(q).  Half of a block's compute warps form grad_x (the forward's code, weights reflected), the other
//     half grad_w (x straight into registers), from the same staged planes: three tensors of traffic for the two gradients
//     instead of five.  One thread for both would hold 108 registers of weights and sums; with two roles the kernel spills a
//     little (fp16 backward: 64 bytes stored, 100 loaded).
//   * planes arrive in two rings.  Every band of rows of a plane of one channel is one contiguous byte range; it is bulk
//     copied from the 16-byte boundary below its start (any width, offset and pointer alignment: the remainder is added to
//     the reader's address; vectors that the tensor's first or last byte cuts are fetched by elements) into a raw stage.  Two warps turn the raw bands of a channel pair into one stage of fp32 pairs
//     {c, c+1} with zeros around it, once per plane: a compute thread's plane is then 18 conflict-free 8-byte loads and 108
//     packed FMA.  (Reading the channels' separate bands from the compute threads cost 36 loads, 24 selects and as many
//     moves as FMA; pairing in the compute threads instead of two warps of their own gave 445 instructions per 108 FMA.)
// Work is ordered channel pair, clip, band: a warp keeps its 54 weight-gradient sums over clips and bands of a pair and
// reduces them (31 shuffles of pairs, one atomic per lane and channel) when the pair changes.
//
// fp16, 4 x 256 channels, 8 x 60 x 107 (rows that cannot be bulk-copied one by one): forward 0.36 -> 0.17 ms, backward 1.10 ->
// 0.32 ms against a register march from global memory.  fp32, 8 x 1024 channels, 8 x 30 x 54: 0.32 and 0.54 ms, where the
// kernels over x-adjacent pairs take 0.23 and 0.49 ms (they read a plane as it was copied; here the two pairing warps are the
// limit), so those keep the sizes that they can take.
// Reference: ops/fast-depthwise-conv3d/csrc/grouped_conv3d.cu:22-276.
#pragma once

#include <cuda_fp16.h>

#include "d2c_common.cuh"
#include "sm100_ptx.cuh"

namespace d2c {
namespace {

constexpr int kDwpRows = 4;             // R
constexpr int kDwpMaxStages = 6;
constexpr size_t kDwpSmemMax = 220 * 1024;
constexpr int kDwpThreads = 512;        // 128 registers a thread: 54 of weights (or sums), 24 of accumulators (or x)
constexpr int kDwpLoaders = 64;         // two warps: bulk copies, and raw bands into pairs
constexpr int kDwpRawStages = 4;        // raw planes on the way
struct DwPairPlan {
  int bands, band_rows;       // bands per plane, rows per band (a multiple of R)
  int patches, lanes;         // patches (row groups x W) per band, rounded up to whole warps
  int groups;                 // (pair, clip, band) groups a block works on at a time
  int n_groups, n_chunks;
  int buf;                    // pairs of one staged band, borders included
  int raw;                    // elements of one raw band (one channel)
  int stages, compute, blocks;        // compute: threads per role
  size_t smem;
};

// roles: 1 (forward, or one gradient alone) or 2 (grad_x and grad_w): thread sets over the same planes.
template <typename T>
inline bool dw_pair_plan(const Geom& g, int roles, int sm_count, DwPairPlan* p) {
  if (!(g.kd == 3 && g.kh == 3 && g.kw == 3 && g.sd == 1 && g.sh == 1 && g.sw == 1 && g.dd == 1 && g.dh == 1 && g.dw == 1 &&
        g.pd == 1 && g.ph == 1 && g.pw == 1 && g.Cout == g.Cin))
    return false;
  constexpr int R = kDwpRows;
  const int most = (kDwpThreads - kDwpLoaders) / roles / 32 * 32;
  if (g.W > most) return false;
  // rows per band: as many row groups as fit the block, evened out over the bands
  const int row_groups = (g.H + R - 1) / R, fit = most / g.W;
  p->bands = (row_groups + fit - 1) / fit;
  const int per_band = (row_groups + p->bands - 1) / p->bands;
  p->bands = (row_groups + per_band - 1) / per_band;
  p->band_rows = per_band * R;
  p->patches = per_band * g.W;
  p->lanes = (p->patches + 31) / 32 * 32;
  const long long n_groups = (long long)((g.Cin + 1) / 2) * g.B * p->bands;
  if (n_groups > 0x7fffffffLL) return false;
  p->n_groups = (int)n_groups;
  p->groups = most / p->lanes;
  // small planes: several groups per block, but not fewer blocks than multiprocessors
  while (p->groups > 1 && (p->n_groups + p->groups - 1) / p->groups < sm_count) --p->groups;
  p->n_chunks = (p->n_groups + p->groups - 1) / p->groups;
  p->buf = ((p->band_rows + 2) * (g.W + 1) + 2) / 2 * 2;
  p->raw = ((p->band_rows + 2) * g.W + 16 + 7) / 8 * 8;
  p->compute = p->groups * p->lanes;
  const size_t stage = (size_t)p->groups * p->buf * 2 * sizeof(float);
  const size_t raw = (size_t)kDwpRawStages * p->groups * 2 * p->raw * sizeof(T);
  if (raw + 2 * stage > kDwpSmemMax) return false;
  p->stages = (int)((kDwpSmemMax - raw) / stage);
  if (p->stages > kDwpMaxStages) p->stages = kDwpMaxStages;
  p->smem = p->stages * stage + raw;
  p->blocks = p->n_chunks < sm_count ? p->n_chunks : sm_count;
  return true;
}

using dwp_u64 = unsigned long long;
__device__ __forceinline__ dwp_u64 dwp_pair(float a, float b) {
  dwp_u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 dwp_split(dwp_u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void dwp_fma(dwp_u64& d, dwp_u64 a, dwp_u64 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float dwp_ld(const float* p) { return __ldg(p); }
__device__ __forceinline__ float dwp_ld(const __half* p) { return __half2float(__ldg(p)); }
__device__ __forceinline__ void dwp_st(float* p, float v) { *p = v; }
__device__ __forceinline__ void dwp_st(__half* p, float v) { *p = __float2half_rn(v); }

// A group's place in the tensors.
struct DwpGroup {
  int pair, b, y0;            // channel pair, clip, first row of the band
  __device__ __forceinline__ void set(int gid, int B, int bands, int band_rows) {
    y0 = gid % bands * band_rows;
    gid /= bands;
    b = gid % B;
    pair = gid / B;
  }
};

// Where a band of plane p of one channel starts: element index of its first readable row, rows to copy, and the part of a
// 16-byte vector that precedes it.
template <typename T>
struct DwpBand {
  static constexpr int kVec = 16 / sizeof(T);
  int row_beg, rows;
  __device__ __forceinline__ DwpBand(int y0, int band_rows, int H) {
    row_beg = max(y0 - 1, 0);
    rows = min(y0 + band_rows + 1, H) - row_beg;
  }
  static __device__ __forceinline__ int shift(const T* start) {
    return (int)((reinterpret_cast<uintptr_t>(start) / sizeof(T)) % kVec);
  }
};

// The 16-byte vectors that a bulk copy takes for the bytes [start, stop) of the tensor [base, end): those that hold any of them
// and lie inside the tensor.  What remains of [start, stop) is part of a vector that the tensor's first or last byte cuts.
struct DwpSpan {
  uintptr_t lo, hi;
  __host__ __device__ DwpSpan(uintptr_t start, uintptr_t stop, uintptr_t base, uintptr_t end) {
    const uintptr_t first = (base + 15) & ~(uintptr_t)15, last = end & ~(uintptr_t)15;
    lo = start & ~(uintptr_t)15;
    hi = (stop + 15) & ~(uintptr_t)15;
    if (lo < first) lo = first;
    if (hi > last) hi = last;
    if (hi < lo) hi = lo;
  }
};

// A staged pair; 32-bit shared-memory addresses (a generic pointer costs two registers and two adds per row).
template <int kOff>
__device__ __forceinline__ dwp_u64 dwp_lds(uint32_t addr) {
  dwp_u64 v;
  asm volatile("ld.shared.b64 %0, [%1+%2];" : "=l"(v) : "r"(addr), "n"(kOff));
  return v;
}
// A staged band holds input rows y0 - 1 .. y0 + band_rows of W + 1 pairs, the first of each row zero (column -1, and column W
// of the row before), rows outside the plane zero.
__device__ __forceinline__ void dwp_row(uint32_t at, dwp_u64 (&v)[3]) {
  v[0] = dwp_lds<0>(at);
  v[1] = dwp_lds<8>(at);
  v[2] = dwp_lds<16>(at);
}

// Forward, one plane: input plane p meets output planes p-1 (kz = 2), p (1), p+1 (0); the last starts from the bias.
__device__ __forceinline__ void dwp_conv_step(uint32_t at, uint32_t pitch, const dwp_u64 (&w)[27],
                                              dwp_u64 bias, dwp_u64 (&am1)[kDwpRows], dwp_u64 (&a0)[kDwpRows],
                                              dwp_u64 (&ap1)[kDwpRows]) {
#pragma unroll
  for (int r = 0; r < kDwpRows; ++r) ap1[r] = bias;
#pragma unroll
  for (int j = 0; j < kDwpRows + 2; ++j) {
    dwp_u64 v[3];
    dwp_row(at + j * pitch, v);
#pragma unroll
    for (int kx = 0; kx < 3; ++kx)
#pragma unroll
      for (int r = 0; r < kDwpRows; ++r) {
        const int ky = j - r;
        if (ky < 0 || ky > 2) continue;
        dwp_fma(am1[r], w[(2 * 3 + ky) * 3 + kx], v[kx]);
        dwp_fma(a0[r], w[(1 * 3 + ky) * 3 + kx], v[kx]);
        dwp_fma(ap1[r], w[(0 * 3 + ky) * 3 + kx], v[kx]);
      }
  }
}

// Weight gradient, one plane: grad_out plane p meets x planes p-1 (kz = 0), p (1), p+1 (2).
__device__ __forceinline__ void dwp_grad_step(uint32_t at, uint32_t pitch, dwp_u64 (&gw)[27],
                                              const dwp_u64 (&xm1)[kDwpRows], const dwp_u64 (&x0)[kDwpRows],
                                              const dwp_u64 (&xp1)[kDwpRows]) {
#pragma unroll
  for (int j = 0; j < kDwpRows + 2; ++j) {
    dwp_u64 v[3];
    dwp_row(at + j * pitch, v);
#pragma unroll
    for (int r = 0; r < kDwpRows; ++r)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int ky = r - j + 2, kx = 2 - i;
        if (ky < 0 || ky > 2) continue;
        dwp_fma(gw[(0 * 3 + ky) * 3 + kx], xm1[r], v[i]);
        dwp_fma(gw[(1 * 3 + ky) * 3 + kx], x0[r], v[i]);
        dwp_fma(gw[(2 * 3 + ky) * 3 + kx], xp1[r], v[i]);
      }
  }
}

// Sums of the 27 pair accumulators over the warp: lane t ends with tap t.  Halving exchange: 16 + 8 + 4 + 2 + 1 shuffles of
// pairs (each 64 bits) instead of 27 x 5.
__device__ __forceinline__ dwp_u64 dwp_warp_sums(const dwp_u64 (&acc)[27]) {
  const int lane = threadIdx.x & 31;
  dwp_u64 v[32];
#pragma unroll
  for (int t = 0; t < 32; ++t) v[t] = t < 27 ? acc[t] : 0ull;
#pragma unroll
  for (int bit = 16; bit >= 1; bit >>= 1) {
    const bool hi = lane & bit;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      if (t >= bit) continue;
      const dwp_u64 keep = hi ? v[t + bit] : v[t], give = hi ? v[t] : v[t + bit];
      const float2 a = dwp_split(keep), b = dwp_split(__shfl_xor_sync(0xffffffffu, give, bit));
      v[t] = dwp_pair(a.x + b.x, a.y + b.y);
    }
  }
  return v[0];
}

struct DwPairArgs {
  Geom g;
  DwPairPlan plan;
  const void* in;             // convolution: x or grad_out; weight gradient: grad_out
  const void* x;              // weight gradient
  const void* w;              // convolution
  const void* bias;           // convolution, nullable
  void* out;                  // convolution: y or grad_x
  float* grad_w;              // weight gradient, accumulated, [C][27]
  int flip;                   // convolution with the reflected kernel (grad_x)
};

// Reader of the staged planes, common to both roles.
template <typename T>
struct DwpReader {
  const DwPairArgs& a;
  const uint32_t smem, full0, empty0;       // staged bands, barriers
  volatile int* abort_flag;
  const int k, lane;          // group slot of the block
  const uint32_t off, pitch;  // bytes: the thread's patch in a staged band, one of its rows
  int stage = 0;
  uint32_t phase = 0;

  // waits for the next plane and gives the address of the thread's patch (column x - 1, row y0 - 1) in it
  __device__ __forceinline__ bool next(uint32_t& at) const {
    if (!ptx::mbar_wait(full0 + 8u * stage, phase, abort_flag)) return false;
    at = smem + (uint32_t)(stage * a.plan.groups + k) * (8u * (uint32_t)a.plan.buf) + off;
    return true;
  }
  __device__ __forceinline__ void release() {
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(empty0 + 8u * stage);
    if (++stage == a.plan.stages) { stage = 0; phase ^= 1u; }
  }
};

// The part of a chunk's bookkeeping that both roles need: the thread's patch in the tensors.
template <typename T>
struct DwpPatch {
  int pair, c0, c1, rows_ok;
  bool has2, group_ok;
  long long at0, at1;         // element index of row y0, column x, plane 0 in the two channels
  __device__ __forceinline__ void set(const DwPairArgs& a, int chunk, int k, int i) {
    const Geom& g = a.g;
    const DwPairPlan& pl = a.plan;
    const int gid = chunk * pl.groups + k;
    group_ok = gid < pl.n_groups;
    DwpGroup gr;
    gr.set(group_ok ? gid : 0, g.B, pl.bands, pl.band_rows);
    pair = gr.pair;
    c0 = 2 * pair;
    has2 = c0 + 1 < g.Cin;
    c1 = has2 ? c0 + 1 : c0;
    const int yg = i / g.W, x = i - yg * g.W, y0 = gr.y0 + yg * kDwpRows;
    const bool live = group_ok && i < pl.patches && y0 < g.H;
    rows_ok = live ? min(kDwpRows, g.H - y0) : 0;
    const long long HW = (long long)g.H * g.W, vol = g.D * HW;
    const long long b0 = ((long long)gr.b * g.Cin + c0) * vol, b1 = ((long long)gr.b * g.Cin + c1) * vol;
    at0 = b0 + (live ? (long long)y0 * g.W + x : 0);
    at1 = b1 + (live ? (long long)y0 * g.W + x : 0);
  }
};

template <typename T>
__device__ __forceinline__ void dwp_conv_role(const DwPairArgs& a, DwpReader<T>& rd, int i, int ch_beg, int ch_end) {
  constexpr int R = kDwpRows;
  const Geom& g = a.g;
  const int HW = g.H * g.W;
  T* out = reinterpret_cast<T*>(a.out);
  dwp_u64 w[27], bias = 0ull;
  int pair_open = -1;                     // channel pair whose weights the warp holds
  for (int ch = ch_beg; ch < ch_end; ++ch) {
    DwpPatch<T> pt;
    pt.set(a, ch, rd.k, i);
    if (pt.group_ok && pt.pair != pair_open) {     // the same for the whole warp
      pair_open = pt.pair;
      const T* wt = reinterpret_cast<const T*>(a.w);
#pragma unroll
      for (int t = 0; t < 27; ++t) {
        const int tw = a.flip ? 26 - t : t;
        w[t] = dwp_pair(dwp_ld(wt + (long long)pt.c0 * 27 + tw), dwp_ld(wt + (long long)pt.c1 * 27 + tw));
      }
      if (a.bias) {
        const T* bp = reinterpret_cast<const T*>(a.bias);
        bias = dwp_pair(dwp_ld(bp + pt.c0), dwp_ld(bp + pt.c1));
      }
    }
    T *o0 = out + pt.at0, *o1 = out + pt.at1;      // next output plane
    auto store = [&](const dwp_u64 (&v)[R]) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r < pt.rows_ok) {
          const float2 f = dwp_split(v[r]);
          dwp_st(o0 + r * g.W, f.x);
          if (pt.has2) dwp_st(o1 + r * g.W, f.y);
        }
      o0 += HW;
      o1 += HW;
    };
    uint32_t at;
    dwp_u64 A[R], B[R], C[R];
#pragma unroll
    for (int r = 0; r < R; ++r) A[r] = B[r] = C[r] = bias;
    // plane p completes output plane p-1; the accumulator roles rotate with period 3
    for (int p = 0; p < g.D; p += 3) {
      if (!rd.next(at)) return;
      dwp_conv_step(at, rd.pitch, w, bias, A, B, C);
      rd.release();
      if (p >= 1) store(A);
      if (p + 1 >= g.D) { store(B); break; }
      if (!rd.next(at)) return;
      dwp_conv_step(at, rd.pitch, w, bias, B, C, A);
      rd.release();
      store(B);
      if (p + 2 >= g.D) { store(C); break; }
      if (!rd.next(at)) return;
      dwp_conv_step(at, rd.pitch, w, bias, C, A, B);
      rd.release();
      store(C);
      if (p + 3 >= g.D) store(A);
    }
  }
}

template <typename T>
__device__ __forceinline__ void dwp_grad_role(const DwPairArgs& a, DwpReader<T>& rd, int i, int ch_beg, int ch_end) {
  constexpr int R = kDwpRows;
  const Geom& g = a.g;
  const int HW = g.H * g.W;
  dwp_u64 gw[27];
  int pair_open = -1;                     // channel pair whose sums the warp holds
  auto flush = [&]() {
    if (pair_open < 0) return;
    if (i >= a.plan.patches) {            // no patch: what it multiplied by x = 0 need not have been finite
#pragma unroll
      for (int t = 0; t < 27; ++t) gw[t] = 0ull;
    }
    const float2 s = dwp_split(dwp_warp_sums(gw));
    if (rd.lane < 27) {
      atomicAdd(a.grad_w + (long long)(2 * pair_open) * 27 + rd.lane, s.x);
      if (2 * pair_open + 1 < g.Cin) atomicAdd(a.grad_w + (long long)(2 * pair_open + 1) * 27 + rd.lane, s.y);
    }
  };
  for (int ch = ch_beg; ch < ch_end; ++ch) {
    DwpPatch<T> pt;
    pt.set(a, ch, rd.k, i);
    if (pt.group_ok && pt.pair != pair_open) {     // the same for the whole warp
      flush();
      pair_open = pt.pair;
#pragma unroll
      for (int t = 0; t < 27; ++t) gw[t] = 0ull;
    }
    const T *x0 = reinterpret_cast<const T*>(a.x) + pt.at0, *x1 = reinterpret_cast<const T*>(a.x) + pt.at1;
    int left = g.D;                       // planes of x not yet fetched
    T f0[R], f1[R];                       // the next plane of x, fetched a step ahead
    auto fetch = [&]() {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        f0[r] = f1[r] = T(0.f);
        if (left > 0 && r < pt.rows_ok) {
          f0[r] = __ldg(x0 + r * g.W);
          f1[r] = __ldg(x1 + r * g.W);
        }
      }
      --left;
      x0 += HW;
      x1 += HW;
    };
    auto take = [&](dwp_u64 (&v)[R]) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = dwp_pair(float(f0[r]), float(f1[r]));
    };
    uint32_t at;
    dwp_u64 xa[R], xb[R], xc[R];
    // one staged plane; the group slots that the last chunk leaves empty hold nothing to multiply
    auto step = [&](dwp_u64 (&xm1)[R], const dwp_u64 (&xz)[R], dwp_u64 (&xp1)[R]) {
      take(xp1);
      fetch();
      if (!rd.next(at)) return false;
      if (pt.group_ok) dwp_grad_step(at, rd.pitch, gw, xm1, xz, xp1);
      rd.release();
      return true;
    };
#pragma unroll
    for (int r = 0; r < R; ++r) xa[r] = 0ull;
    fetch();
    take(xb);
    fetch();
    // x planes p-1, p, p+1 are in xa, xb, xc (rotating)
    for (int p = 0; p < g.D; p += 3) {
      if (!step(xa, xb, xc)) return;
      if (p + 1 >= g.D) break;
      if (!step(xb, xc, xa)) return;
      if (p + 2 >= g.D) break;
      if (!step(xc, xa, xb)) return;
    }
  }
  flush();
}

// Copies the bands of successive planes into a ring of raw stages: lane 2k + c takes group k, channel c (at most 14 groups:
// 448 compute threads in whole warps).  One warp; step() issues one plane.
template <typename T>
struct DwpCopier {
  const DwPairArgs& a;
  const uint32_t ring, full0;       // raw bands of plan.raw elements
  const int lane, ch_end;
  int ch, p = 0, stage = 0;
  int rows_n = 0;
  bool mine = false;
  const T* src = nullptr;
  uintptr_t tensor_beg = reinterpret_cast<uintptr_t>(a.in);
  uintptr_t tensor_end = tensor_beg + (uintptr_t)((long long)a.g.B * a.g.Cin * a.g.D * a.g.H * a.g.W * sizeof(T));
  uint32_t issued = 0;
  __device__ __forceinline__ bool done() const { return ch >= ch_end; }
  __device__ __forceinline__ void open() {
    const Geom& g = a.g;
    const DwPairPlan& pl = a.plan;
    mine = lane < 2 * min(pl.groups, pl.n_groups - ch * pl.groups);
    DwpGroup gr;
    gr.set(mine ? ch * pl.groups + lane / 2 : 0, g.B, pl.bands, pl.band_rows);
    const DwpBand<T> band(gr.y0, pl.band_rows, g.H);
    const int chan = min(2 * gr.pair + (lane & 1), g.Cin - 1);
    src = reinterpret_cast<const T*>(a.in) + ((long long)gr.b * g.Cin + chan) * g.D * g.H * g.W + band.row_beg * g.W;
    rows_n = band.rows * g.W;
  }
  __device__ __forceinline__ void step() {
    if (p == 0) open();
    const uint32_t slot = ring + (uint32_t)((stage * a.plan.groups * 2 + lane) * a.plan.raw * (int)sizeof(T));
    const uintptr_t start = reinterpret_cast<uintptr_t>(src), stop = start + rows_n * sizeof(T), at0 = start & ~(uintptr_t)15;
    const DwpSpan span(start, stop, tensor_beg, tensor_end);
    const uint32_t len = mine ? (uint32_t)(span.hi - span.lo) : 0u;
    if (mine && (span.lo > start || span.hi < stop)) {       // the tensor's first or last band, where it is not aligned
      T* dst = reinterpret_cast<T*>(__cvta_shared_to_generic(slot + (uint32_t)(start - at0)));
      for (int i = 0; i < rows_n; ++i) {
        const uintptr_t e = start + i * sizeof(T);
        if (e < span.lo || e >= span.hi) dst[i] = __ldg(src + i);
        else i = (int)((span.hi - start) / sizeof(T)) - 1;
      }
      ptx::fence_proxy_async_smem();       // a bulk copy writes here the next time
    }
    __syncwarp();
    const uint32_t total = __reduce_add_sync(0xffffffffu, len);
    if (lane == 0) ptx::mbar_arrive_expect_tx(full0 + 8u * stage, total);
    __syncwarp();
    if (len) ptx::bulk_g2s(slot + (uint32_t)(span.lo - at0), reinterpret_cast<const void*>(span.lo), len, full0 + 8u * stage);
    src += (long long)a.g.H * a.g.W;
    ++issued;
    if (++stage == kDwpRawStages) stage = 0;
    if (++p == a.g.D) { p = 0; ++ch; }
  }
  // never leave with a bulk copy in flight
  __device__ __forceinline__ void drain() const {
    if (lane != 0) return;
    for (uint32_t k = (issued > (uint32_t)kDwpRawStages ? issued - kDwpRawStages : 0); k < issued; ++k) {
      const long long t0 = clock64();
      while (!ptx::mbar_try_wait(full0 + 8u * (k % kDwpRawStages), (k / kDwpRawStages) & 1))
        if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
    }
  }
};

__device__ __forceinline__ float dwp_f32(float v) { return v; }
__device__ __forceinline__ float dwp_f32(__half v) { return __half2float(v); }

// Two warps turn each raw plane into a stage of pairs; the second one also keeps the raw ring full.
template <typename T>
__device__ __forceinline__ void dwp_load(const DwPairArgs& a, const T* raw, float2* smem, uint32_t raw_full0, uint32_t raw_empty0,
                                         uint32_t full0, uint32_t empty0, volatile int* abort_flag, int t, int ch_beg, int ch_end) {
  const Geom& g = a.g;
  const DwPairPlan& pl = a.plan;
  const int lane = t & 31, HW = g.H * g.W, W = g.W, n = (pl.band_rows + 2) * W;
  const bool copies = t >= 32;
  DwpCopier<T> cp{a, ptx::smem_u32(raw), raw_full0, lane, ch_end, ch_beg};
  if (copies)
    for (int i = 0; i < kDwpRawStages && !cp.done(); ++i) cp.step();
  // element e of a band goes to pair e + e / W + 1; e advances by 64
  const int row0 = t / W, col0 = t - row0 * W, pos0 = t + row0 + 1;
  const int pos_step = 64 + 64 / W, col_step = 64 % W;
  int rs = 0, stage = 0;
  uint32_t rphase = 0, phase = 1;
  bool ok = true;
  for (int ch = ch_beg; ok && ch < ch_end; ++ch) {
    const int n_here = min(pl.groups, pl.n_groups - ch * pl.groups);
    // lane 2k + c knows where the band of group k, channel c starts
    DwpGroup gr;
    gr.set(lane < 2 * n_here ? ch * pl.groups + lane / 2 : 0, g.B, pl.bands, pl.band_rows);
    const DwpBand<T> band(gr.y0, pl.band_rows, g.H);
    const T* src = reinterpret_cast<const T*>(a.in) +
                   ((long long)gr.b * g.Cin + min(2 * gr.pair + (lane & 1), g.Cin - 1)) * g.D * HW + band.row_beg * W;
    const int my_skip = gr.y0 == 0 ? W : 0, my_rows = band.rows * W;    // elements of the row above the plane, of the raw band
    for (int p = 0; p < g.D; ++p, src += HW) {
      if (!ptx::mbar_wait(raw_full0 + 8u * rs, rphase, abort_flag) || !ptx::mbar_wait(empty0 + 8u * stage, phase, abort_flag)) ok = false;
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      const int my_shift = DwpBand<T>::shift(src);
      for (int k = 0; k < n_here; ++k) {
        const int skip = __shfl_sync(0xffffffffu, my_skip, 2 * k);
        const unsigned rows = (unsigned)__shfl_sync(0xffffffffu, my_rows, 2 * k);
        const T* in0 = raw + (rs * pl.groups + k) * 2 * pl.raw + __shfl_sync(0xffffffffu, my_shift, 2 * k);
        const T* in1 = raw + ((rs * pl.groups + k) * 2 + 1) * pl.raw + __shfl_sync(0xffffffffu, my_shift, 2 * k + 1);
        float2* out = smem + (stage * pl.groups + k) * pl.buf;
        int pos = pos0, col = col0;
        // eight loads of each channel in flight: the compiler may not move them over the stores
        for (int e = t; e < n; e += 8 * 64) {
          float2 v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int at = e + 64 * u - skip;
            v[u] = make_float2(0.f, 0.f);
            if ((unsigned)at < rows) v[u] = make_float2(dwp_f32(in0[at]), dwp_f32(in1[at]));
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (e + 64 * u < n) out[pos] = v[u];
            col += col_step;
            pos += pos_step;
            if (col >= W) { col -= W; ++pos; }
          }
        }
      }
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(full0 + 8u * stage);
        ptx::mbar_arrive(raw_empty0 + 8u * rs);
      }
      if (copies && !cp.done()) {        // the raw stage just read takes the plane kDwpRawStages ahead
        ok = ptx::mbar_wait(raw_empty0 + 8u * rs, rphase, abort_flag);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        cp.step();
      }
      if (++rs == kDwpRawStages) { rs = 0; rphase ^= 1u; }
      if (++stage == pl.stages) { stage = 0; phase ^= 1u; }
    }
  }
  if (copies) cp.drain();
}

// Threads: [convolution role][weight-gradient role][loaders]
template <typename T, bool kConv, bool kGrad>
__global__ void __launch_bounds__(kDwpThreads, 1) dw_pair_kernel(const __grid_constant__ DwPairArgs a) {
  const DwPairPlan& pl = a.plan;
  extern __shared__ __align__(128) float2 smem_pairs[];
  __shared__ __align__(8) dwp_u64 bars[2 * kDwpMaxStages + 2 * kDwpRawStages];
  __shared__ int abort_word;
  const uint32_t full0 = ptx::smem_u32(bars), empty0 = full0 + 8u * kDwpMaxStages;
  const uint32_t raw_full0 = empty0 + 8u * kDwpMaxStages, raw_empty0 = raw_full0 + 8u * kDwpRawStages;
  const int compute = pl.compute * ((kConv ? 1 : 0) + (kGrad ? 1 : 0));
  const int ch_beg = (int)((long long)pl.n_chunks * blockIdx.x / gridDim.x), ch_end = (int)((long long)pl.n_chunks * (blockIdx.x + 1) / gridDim.x);
  if (threadIdx.x == 0) {
    for (int s = 0; s < pl.stages; ++s) {
      ptx::mbar_init(full0 + 8u * s, kDwpLoaders / 32);
      ptx::mbar_init(empty0 + 8u * s, compute / 32);
    }
    for (int s = 0; s < kDwpRawStages; ++s) {
      ptx::mbar_init(raw_full0 + 8u * s, 1);
      ptx::mbar_init(raw_empty0 + 8u * s, kDwpLoaders / 32);
    }
    abort_word = 0;
    ptx::fence_mbar_init();
  }
  // the zero pairs between rows stay; everything else is written per plane
  for (int i = threadIdx.x; i < pl.stages * pl.groups * pl.buf; i += blockDim.x) smem_pairs[i] = make_float2(0.f, 0.f);
  __syncthreads();
  const int t = threadIdx.x, lane = t & 31;
  if (t >= compute) {
    dwp_load<T>(a, reinterpret_cast<const T*>(smem_pairs + pl.stages * pl.groups * pl.buf), smem_pairs, raw_full0, raw_empty0, full0,
                empty0, &abort_word, t - compute, ch_beg, ch_end);
  } else {
    const int tr = kConv && t >= pl.compute ? t - pl.compute : t, k = tr / pl.lanes, i = tr - k * pl.lanes;
    const int yg = i / a.g.W, pitch = a.g.W + 1;
    const uint32_t off = i < pl.patches ? 8u * (uint32_t)(yg * kDwpRows * pitch + i - yg * a.g.W) : 0u;
    DwpReader<T> rd{a, ptx::smem_u32(smem_pairs), full0, empty0, &abort_word, k, lane, off, 8u * (uint32_t)pitch};
    if (kConv && (!kGrad || t < pl.compute)) dwp_conv_role<T>(a, rd, i, ch_beg, ch_end);
    else if (kGrad) dwp_grad_role<T>(a, rd, i, ch_beg, ch_end);
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_word) ptx::report_device_timeout();
}

template <typename T, bool kConv, bool kGrad>
int dw_pair_launch(const DwPairArgs& a, cudaStream_t st) {
  const int rc = allow_dynamic_smem<dw_pair_kernel<T, kConv, kGrad>>((int)a.plan.smem);
  if (rc) return rc;
  const int threads = a.plan.compute * ((kConv ? 1 : 0) + (kGrad ? 1 : 0)) + kDwpLoaders;
  dw_pair_kernel<T, kConv, kGrad><<<a.plan.blocks, threads, a.plan.smem, st>>>(a);
  D2C_LAUNCH_CHECK();
  return D2C_OK;
}

}  // namespace
}  // namespace d2c
