// Tensor-core backward of the modulated deformable conv3d for sm_100a (data side):
//
//   (a) dcol_sm100_kernel   gradient columns dcol[b, v, (slice, c)] = sum_co grad_out[b, co, v] * W[co, c, tap]
//                           as a tcgen05 GEMM (bf16 operands, fp32 accumulate in TMEM), voxel-major
//                           rows so that the 64 channels of one (offset group, tap) slice are contiguous.
//                           Replaces the reference's cuBLAS call at csrc/ops/dconv3d_gpu.cu:981-999.
//   (b) sample_grad_taps_kernel  grad_offset / grad_mask and grad_input (channels-last fp32) from dcol; the contributions to an
//                           input voxel are added up per block and leave it as one reduction, or, where few would meet or
//                           weigh anything, each by itself (sample_grad_direct_kernel; sm100_sample_grad.cuh).
//                           Replaces deformable_col2im_coord_gpu_kernel (:756-864) and
//                           deformable_col2im_gpu_kernel (:562-643).
//   (c) unstage_grad_input_kernel  channels-last fp32 -> NCDHW.
//
// The weight gradient is in deform_sm100_dw.cu; sampling positions come from the records of
// sm100_gather.cuh, computed once per backward call.
#include <algorithm>
#include <type_traits>

#include "deform_exact.h"   // slice_clips
#include "deform_sm100.h"
#include "sm100_gather.cuh"
#include "sm100_ptx.cuh"
#include "sm100_sample_grad.cuh"
#include "sm100_stage.cuh"

namespace d2c {

namespace {

constexpr int kBM = 128;
constexpr int kABlockBytes = kBM * 128;       // one 64-wide K block of the grad_out tile: 16 KB
constexpr int kNBlock = 256;                  // dcol columns per accumulator (4 slices of 64 channels)
constexpr int kBStageBytes = kNBlock * 128;   // 32 KB
constexpr int kBStages = 3;
constexpr int kDcolEpiWarps = 8;              // warp w: TMEM lane quarter w%4, column half w/4
constexpr int kDcolMmaWarp = 8, kDcolLoadWarp = 9;
constexpr int kDcolThreads = 320;
constexpr int kSmemLimit = 227 * 1024;
constexpr size_t kWordBytes = 256;            // of the workspace: the answer of PositionAsk

// ---- staging ------------------------------------------------------------------------------------

// grad_out [B][Cout][V] fp32 -> per (tile, 64-wide co block) images of 128 rows (voxels) x 128 B (64 co,
// bf16), 16-byte chunks XOR-swizzled by (row & 7): the byte image of a K-major SW128 A tile.
// Rows past the end of the clip are zero.
// x3 = 1 (fp32-parity mode): a K block is 32 co and a row is [hi(32 co) | lo(32 co)], hi = bf16(g),
// lo = bf16(g - hi).
// x3 = 2 (fp32-parity mode, long contractions): K blocks of 64 co as in the single-pass mode, written twice: the hi
// parts as one image and the lo parts as a second image `lo_off` bytes further.
__device__ __forceinline__ float split_part(float f, bool lo) {
  return lo ? f - ptx::bf16_lo(ptx::pack_bf16x2(f, 0.f)) : f;
}

__global__ void __launch_bounds__(256)
stage_gy_img_kernel(int Cout, int V, int tiles_per_clip, int b0, int x3, const float* __restrict__ gy,
                    uint8_t* __restrict__ img, long long lo_off, const __grid_constant__ PositionAsk ask) {
  __shared__ float tile[64][129];
  const int asks = ask.n_recs > 0;               // then a column of blocks more, of which one asks, beside the others
  if (asks && blockIdx.x == 0) {
    if (blockIdx.y == 0) ask_positions(ask);
    return;
  }
  const int tile_id = blockIdx.x - asks, kb = blockIdx.y, KB = gridDim.y;
  const int bl = tile_id / tiles_per_clip, v0 = (tile_id % tiles_per_clip) * kBM;
  const int b = b0 + bl;
  const int nco = x3 == 1 ? 32 : 64;
  for (int e = threadIdx.x; e < nco * 128; e += 256) {
    const int co = e >> 7, r = e & 127, v = v0 + r;
    tile[co][r] = (v < V) ? __ldg(gy + ((long long)b * Cout + kb * nco + co) * V + v) : 0.f;
  }
  __syncthreads();
  uint8_t* dst = img + ((long long)tile_id * KB + kb) * kABlockBytes;
  for (int e = threadIdx.x; e < 128 * 8; e += 256) {
    const int r = e >> 3, j = e & 7;
    const bool lo = x3 == 1 && j >= 4;
    const int cb = x3 == 1 ? (j & 3) * 8 : j * 8;
    const long long at = (r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4);
    uint4 o;
    o.x = ptx::pack_bf16x2(split_part(tile[cb + 0][r], lo), split_part(tile[cb + 1][r], lo));
    o.y = ptx::pack_bf16x2(split_part(tile[cb + 2][r], lo), split_part(tile[cb + 3][r], lo));
    o.z = ptx::pack_bf16x2(split_part(tile[cb + 4][r], lo), split_part(tile[cb + 5][r], lo));
    o.w = ptx::pack_bf16x2(split_part(tile[cb + 6][r], lo), split_part(tile[cb + 7][r], lo));
    *reinterpret_cast<uint4*>(dst + at) = o;
    if (x3 == 2) {
      o.x = ptx::pack_bf16x2(split_part(tile[cb + 0][r], true), split_part(tile[cb + 1][r], true));
      o.y = ptx::pack_bf16x2(split_part(tile[cb + 2][r], true), split_part(tile[cb + 3][r], true));
      o.z = ptx::pack_bf16x2(split_part(tile[cb + 4][r], true), split_part(tile[cb + 5][r], true));
      o.w = ptx::pack_bf16x2(split_part(tile[cb + 6][r], true), split_part(tile[cb + 7][r], true));
      *reinterpret_cast<uint4*>(dst + lo_off + at) = o;
    }
  }
}

// W [Cout][Cin][K] fp32 -> per (N block of 4 slices, 64-wide co block) images of 256 rows x 128 B:
// row = slice_local*64 + c, 64 co (bf16) per row, swizzled as above (K-major SW128 B tile, K = co).
// Block = (64-wide co block kb, input channel cin): the 64 x K weights W[kb*64 + q][cin][0..K) are read
// as 64 contiguous runs of K floats into shared memory, then each tap's 64 co values are written as one
// 128-byte row (8 swizzled 16-byte chunks).
__global__ void __launch_bounds__(64)
stage_wt_img_kernel(int Cout, int Cin, int K, int cpg, int nh, int x3, const float* __restrict__ w,
                    uint8_t* __restrict__ img, long long lo_off) {
  extern __shared__ float wsm[];                    // [64 (x3: 32) co][K]
  const int kb = blockIdx.x, cin = blockIdx.y, KB = gridDim.x;
  const int nco = x3 == 1 ? 32 : 64;
  for (int i = threadIdx.x; i < nco * K; i += 64) {
    const int q = i / K, t = i - q * K;
    wsm[i] = __ldg(w + ((long long)(kb * nco + q) * Cin + cin) * K + t);
  }
  __syncthreads();
  const int grp = cin / cpg, h = (cin % cpg) / 64, c = cin & 63;
  for (int item = threadIdx.x; item < K * 8; item += 64) {
    const int tap = item >> 3, j = item & 7;
    const bool lo = x3 == 1 && j >= 4;
    const int cb = x3 == 1 ? (j & 3) * 8 : j * 8;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = split_part(wsm[(cb + q) * K + tap], lo);
    uint4 o;
    o.x = ptx::pack_bf16x2(v[0], v[1]); o.y = ptx::pack_bf16x2(v[2], v[3]);
    o.z = ptx::pack_bf16x2(v[4], v[5]); o.w = ptx::pack_bf16x2(v[6], v[7]);
    const int s = (grp * K + tap) * nh + h;
    const int nb = s >> 2, row = (s & 3) * 64 + c;
    uint8_t* dst = img + ((long long)nb * KB + kb) * kBStageBytes + (row >> 3) * 1024 + (row & 7) * 128 +
                   ((j ^ (row & 7)) << 4);
    *reinterpret_cast<uint4*>(dst) = o;
    if (x3 == 2) {
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = split_part(wsm[(cb + q) * K + tap], true);
      o.x = ptx::pack_bf16x2(v[0], v[1]); o.y = ptx::pack_bf16x2(v[2], v[3]);
      o.z = ptx::pack_bf16x2(v[4], v[5]); o.w = ptx::pack_bf16x2(v[6], v[7]);
      *reinterpret_cast<uint4*>(dst + lo_off) = o;
    }
  }
}

// ---- (a) dcol GEMM ------------------------------------------------------------------------------
// Work units are (tile, 256-column block); each CTA takes one contiguous range of them, so the last wave
// is as full as the others.  Within a range the grad_out tile (A, up to 128 KB) is loaded once per tile
// segment; B blocks stream through a 3-stage ring; two accumulators alternate so that the store epilogue
// (8 warps) overlaps the next block's MMAs.

struct DcolParams {
  const uint8_t* gy_img;   // [n_tiles][KB][16 KB]
  const uint8_t* wt_img;   // [NB][KB][32 KB]
  float* dcol;             // [clips_in_chunk * V][NT]
  int V, NT, KB, NB;       // KB: K blocks (128-byte rows) contracted by this launch
  int KBT, kb0;            // K blocks per image (image stride) and first block of this launch
  int tiles_per_clip, n_tiles;
  long long n_units;       // n_tiles * NB
  int tmem_cols;
  long long gy_lo_off, wt_lo_off;   // dcol_sm100_split_kernel: byte offsets of the lo images
};

// Store epilogue shared by the gradient-column kernels: warp w serves TMEM lane quarter w % 4 and column half w / 4 of
// the block's accumulator (two accumulators alternate; their full / empty barriers are 8 bytes apart).
__device__ __forceinline__ void dcol_epilogue(const DcolParams& p, int warp, int lane, long long u_beg, long long u_end,
                                              uint32_t tmem_base, uint32_t acc_full0, uint32_t acc_empty0,
                                              volatile int* abort_flag) {
    // ---- epilogue: TMEM -> dcol (a thread owns one voxel row and a 128-column half of the block)
    const int quarter = warp & 3, half = warp >> 2;
    uint32_t q = 0;
    for (long long u = u_beg; u < u_end; ++u, ++q) {
      const int tile = (int)(u / p.NB), nb = (int)(u % p.NB);
      const int bl = tile / p.tiles_per_clip, v0 = (tile % p.tiles_per_clip) * kBM;
      const int v = v0 + quarter * 32 + lane;
      // dcol is slice-major: [clip][slice][voxel][64 channels]; a 256-column block is 4 slices
      const long long S = p.NT / 64;
      float* row = p.dcol + (((long long)bl * S + nb * 4) * p.V + v) * 64;
      const long long slice_stride = (long long)p.V * 64;
      const int acc = q & 1;
      const int ncols = min(kNBlock, p.NT - nb * kNBlock);
      // Lanes 2i / 2i+1 hold rows v, v+1 (256 bytes apart).  They swap every other 16-byte chunk so that
      // each store instruction has the pair write one full 32-byte sector of ONE row (first the even
      // lane's row, then the odd lane's) instead of two half sectors of two rows.
      const bool odd = lane & 1;
      const bool ok_even = (v - (odd ? 1 : 0)) < p.V, ok_odd = (v + (odd ? 0 : 1)) < p.V;
      auto chunk_ptr = [&](int c0) {   // this lane's first 16-byte slot of the even row in the 32-column chunk c0
        return reinterpret_cast<float4*>(row - (odd ? 64 : 0) + (c0 >> 6) * slice_stride + (c0 & 63) + (odd ? 4 : 0));
      };
      const int c_beg = half * 128, c_end = min(ncols, half * 128 + 128);
      if (!ptx::mbar_wait(acc_full0 + 8u * acc, (q >> 1) & 1, abort_flag)) break;
      ptx::tc_fence_after();
      for (int c0 = c_beg; c0 < c_end; c0 += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * kNBlock + c0), r);
        ptx::tmem_ld_wait();
        float4* dst = chunk_ptr(c0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t send[4], recv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) send[e] = odd ? r[8 * i + e] : r[8 * i + 4 + e];
#pragma unroll
          for (int e = 0; e < 4; ++e) recv[e] = __shfl_xor_sync(0xffffffffu, send[e], 1);
          float4 first, second;   // first: even row's chunk (2i + odd); second: odd row's chunk (2i + odd)
          if (odd) {
            first = make_float4(__uint_as_float(recv[0]), __uint_as_float(recv[1]), __uint_as_float(recv[2]),
                                __uint_as_float(recv[3]));
            second = make_float4(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]),
                                 __uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
          } else {
            first = make_float4(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1]),
                                __uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
            second = make_float4(__uint_as_float(recv[0]), __uint_as_float(recv[1]), __uint_as_float(recv[2]),
                                 __uint_as_float(recv[3]));
          }
          if (ok_even) dst[2 * i] = first;
          if (ok_odd) dst[2 * i + 16] = second;    // next row: + 64 floats
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(acc_empty0 + 8u * acc);
    }
}

// kX3 = 1 (fp32-parity mode): a K block is 32 co with rows [hi | lo] in both operands and the issuer forms
// g_hi*w_hi + g_lo*w_hi + g_hi*w_lo from the 16-wide K sub-blocks.  The whole grad_out tile must be resident
// (at most 8 blocks): Cout <= 256 in this mode; longer contractions run dcol_sm100_split_kernel below.
template <int kX3>
__global__ void __launch_bounds__(kDcolThreads, 1)
dcol_sm100_kernel(const DcolParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const int a_bytes = p.KB * kABlockBytes;
  const uint32_t a_base = base, b_base = base + a_bytes, bar_base = b_base + kBStages * kBStageBytes;
  auto b_full = [&](int s) { return bar_base + 8u * s; };
  auto b_empty = [&](int s) { return bar_base + 8u * (kBStages + s); };
  auto acc_full = [&](int a) { return bar_base + 8u * (2 * kBStages + a); };
  auto acc_empty = [&](int a) { return bar_base + 8u * (2 * kBStages + 2 + a); };
  const uint32_t a_full = bar_base + 8u * (2 * kBStages + 4), a_empty = bar_base + 8u * (2 * kBStages + 5);
  const int slot_off = a_bytes + kBStages * kBStageBytes + 8 * (2 * kBStages + 6);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + slot_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + slot_off + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long u_beg = p.n_units * blockIdx.x / gridDim.x, u_end = p.n_units * (blockIdx.x + 1) / gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBStages; ++s) { ptx::mbar_init(b_full(s), 1); ptx::mbar_init(b_empty(s), 1); }
    for (int a = 0; a < 2; ++a) { ptx::mbar_init(acc_full(a), 1); ptx::mbar_init(acc_empty(a), kDcolEpiWarps); }
    ptx::mbar_init(a_full, 1);
    ptx::mbar_init(a_empty, 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32((const void*)tmem_slot), (uint32_t)p.tmem_cols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < kDcolEpiWarps) {
    dcol_epilogue(p, warp, lane, u_beg, u_end, tmem_base, acc_full(0), acc_empty(0), abort_flag);
  } else if (warp == kDcolMmaWarp) {
    if (lane == 0) {
      uint32_t q = 0, kbc = 0;
      int seg = 0;
      bool ok = true;
      for (long long u = u_beg; ok && u < u_end; ++seg) {
        const int nb_beg = (int)(u % p.NB);
        const int nb_end = (int)min((long long)p.NB, nb_beg + (u_end - u));
        u += nb_end - nb_beg;
        if (!ptx::mbar_wait(a_full, seg & 1, abort_flag)) break;
        ptx::tc_fence_after();
        for (int nb = nb_beg; ok && nb < nb_end; ++nb, ++q) {
          const int acc = q & 1;
          const int ncols = min(kNBlock, p.NT - nb * kNBlock);
          if (!ptx::mbar_wait(acc_empty(acc), ((q >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after();
          const uint32_t idesc = ptx::umma_idesc_bf16_f32(kBM, ncols);
          for (int kb = 0; kb < p.KB; ++kb, ++kbc) {
            const int sb = kbc % kBStages;
            if (!ptx::mbar_wait(b_full(sb), (kbc / kBStages) & 1, abort_flag)) { ok = false; break; }
            ptx::tc_fence_after();
            const uint64_t adesc = ptx::umma_desc_kmajor_sw128(a_base + kb * kABlockBytes);
            const uint64_t bdesc = ptx::umma_desc_kmajor_sw128(b_base + sb * kBStageBytes);
            constexpr int kSteps = kX3 ? 6 : 4;     // K sub-blocks that meet: bf16 (k,k); x3 hi*hi, lo*hi, hi*lo
            constexpr int ka_[6] = {0, 1, 2, 3, 0, 1};
            constexpr int kb_[6] = {0, 1, kX3 ? 0 : 2, kX3 ? 1 : 3, 2, 3};
#pragma unroll
            for (int k = 0; k < kSteps; ++k)
              ptx::umma_bf16(tmem_base + (uint32_t)(acc * kNBlock), adesc + (uint64_t)(2 * ka_[k]),
                             bdesc + (uint64_t)(2 * kb_[k]), idesc, (kb > 0 || k > 0) ? 1u : 0u);
            ptx::umma_commit(b_empty(sb));
          }
          if (ok) ptx::umma_commit(acc_full(acc));
        }
        if (ok) ptx::umma_commit(a_empty);
      }
    }
  } else if (warp == kDcolLoadWarp) {
    if (lane == 0) {
      uint32_t kbc = 0;
      int seg = 0;
      bool ok = true;
      for (long long u = u_beg; ok && u < u_end; ++seg) {
        const int tile = (int)(u / p.NB), nb_beg = (int)(u % p.NB);
        const int nb_end = (int)min((long long)p.NB, nb_beg + (u_end - u));
        u += nb_end - nb_beg;
        if (!ptx::mbar_wait(a_empty, (seg & 1) ^ 1, abort_flag)) break;
        ptx::mbar_arrive_expect_tx(a_full, (uint32_t)a_bytes);
        const uint8_t* asrc = p.gy_img + ((long long)tile * p.KBT + p.kb0) * kABlockBytes;
        for (int off = 0; off < a_bytes; off += 32768)
          ptx::bulk_g2s(a_base + off, asrc + off, (uint32_t)min(32768, a_bytes - off), a_full);
        for (int nb = nb_beg; ok && nb < nb_end; ++nb) {
          const int ncols = min(kNBlock, p.NT - nb * kNBlock);
          for (int kb = 0; kb < p.KB; ++kb, ++kbc) {
            const int sb = kbc % kBStages;
            if (!ptx::mbar_wait(b_empty(sb), ((kbc / kBStages) & 1) ^ 1, abort_flag)) { ok = false; break; }
            ptx::mbar_arrive_expect_tx(b_full(sb), (uint32_t)(ncols * 128));
            ptx::bulk_g2s(b_base + sb * kBStageBytes, p.wt_img + ((long long)nb * p.KBT + p.kb0 + kb) * kBStageBytes,
                          (uint32_t)(ncols * 128), b_full(sb));
          }
        }
      }
      // drain: never exit with a bulk copy in flight
      const uint32_t issued = kbc;
      for (uint32_t qq = (issued > (uint32_t)kBStages ? issued - kBStages : 0); qq < issued; ++qq) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(b_full(qq % kBStages), (qq / kBStages) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
      if (seg > 0) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(a_full, (seg - 1) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) ptx::report_device_timeout();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

// Fp32-parity contraction longer than the resident tile (Cout > 256) in ONE launch.  Operands come as separate hi and
// lo images of 64-wide K blocks.  The hi part of the grad_out tile stays resident (Cout/64 blocks of 16 KB); per
// (256-column block, K block) three ring entries arrive in this order
//     W_hi (up to 32 KB)   -> g_hi * w_hi
//     g_lo (16 KB)         -> g_lo * w_hi      (W_hi still in its stage)
//     W_lo (up to 32 KB)   -> g_hi * w_lo
// so every product accumulates into the block's accumulator before the epilogue stores it: the gradient columns are
// written once (two launches into two partial buffers wrote and re-read 1.4 GB more).  The lo part of the tile is
// re-streamed from L2 for every column block (+25 % bytes into shared memory).
__global__ void __launch_bounds__(kDcolThreads, 1)
dcol_sm100_split_kernel(const DcolParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const int a_bytes = p.KB * kABlockBytes;
  const uint32_t a_base = base, b_base = base + a_bytes, bar_base = b_base + kBStages * kBStageBytes;
  auto b_full = [&](int s) { return bar_base + 8u * s; };
  auto b_empty = [&](int s) { return bar_base + 8u * (kBStages + s); };
  auto acc_full = [&](int a) { return bar_base + 8u * (2 * kBStages + a); };
  auto acc_empty = [&](int a) { return bar_base + 8u * (2 * kBStages + 2 + a); };
  const uint32_t a_full = bar_base + 8u * (2 * kBStages + 4), a_empty = bar_base + 8u * (2 * kBStages + 5);
  const int slot_off = a_bytes + kBStages * kBStageBytes + 8 * (2 * kBStages + 6);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + slot_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + slot_off + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long u_beg = p.n_units * blockIdx.x / gridDim.x, u_end = p.n_units * (blockIdx.x + 1) / gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBStages; ++s) { ptx::mbar_init(b_full(s), 1); ptx::mbar_init(b_empty(s), 1); }
    for (int a = 0; a < 2; ++a) { ptx::mbar_init(acc_full(a), 1); ptx::mbar_init(acc_empty(a), kDcolEpiWarps); }
    ptx::mbar_init(a_full, 1);
    ptx::mbar_init(a_empty, 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32((const void*)tmem_slot), (uint32_t)p.tmem_cols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < kDcolEpiWarps) {
    dcol_epilogue(p, warp, lane, u_beg, u_end, tmem_base, acc_full(0), acc_empty(0), abort_flag);
  } else if (warp == kDcolMmaWarp) {
    if (lane == 0) {
      uint32_t q = 0, e = 0;            // column blocks and ring entries consumed so far
      int seg = 0;
      bool ok = true;
      auto wait_entry = [&](uint32_t idx) {
        return ptx::mbar_wait(b_full(idx % kBStages), (idx / kBStages) & 1, abort_flag);
      };
      for (long long u = u_beg; ok && u < u_end; ++seg) {
        const int nb_beg = (int)(u % p.NB);
        const int nb_end = (int)min((long long)p.NB, nb_beg + (u_end - u));
        u += nb_end - nb_beg;
        if (!ptx::mbar_wait(a_full, seg & 1, abort_flag)) break;
        ptx::tc_fence_after();
        for (int nb = nb_beg; ok && nb < nb_end; ++nb, ++q) {
          const int acc = q & 1;
          const int ncols = min(kNBlock, p.NT - nb * kNBlock);
          if (!ptx::mbar_wait(acc_empty(acc), ((q >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after();
          const uint32_t idesc = ptx::umma_idesc_bf16_f32(kBM, ncols);
          const uint32_t d = tmem_base + (uint32_t)(acc * kNBlock);
          for (int kb = 0; kb < p.KB; ++kb, e += 3) {
            const uint64_t a_hi = ptx::umma_desc_kmajor_sw128(a_base + kb * kABlockBytes);
            const uint32_t s_whi = e % kBStages, s_glo = (e + 1) % kBStages, s_wlo = (e + 2) % kBStages;
            const uint64_t w_hi = ptx::umma_desc_kmajor_sw128(b_base + s_whi * kBStageBytes);
            const uint64_t g_lo = ptx::umma_desc_kmajor_sw128(b_base + s_glo * kBStageBytes);
            const uint64_t w_lo = ptx::umma_desc_kmajor_sw128(b_base + s_wlo * kBStageBytes);
            if (!wait_entry(e)) { ok = false; break; }
            ptx::tc_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k)
              ptx::umma_bf16(d, a_hi + (uint64_t)(2 * k), w_hi + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
            if (!wait_entry(e + 1)) { ok = false; break; }
            ptx::tc_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k)
              ptx::umma_bf16(d, g_lo + (uint64_t)(2 * k), w_hi + (uint64_t)(2 * k), idesc, 1u);
            ptx::umma_commit(b_empty(s_whi));
            ptx::umma_commit(b_empty(s_glo));
            if (!wait_entry(e + 2)) { ok = false; break; }
            ptx::tc_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k)
              ptx::umma_bf16(d, a_hi + (uint64_t)(2 * k), w_lo + (uint64_t)(2 * k), idesc, 1u);
            ptx::umma_commit(b_empty(s_wlo));
          }
          if (ok) ptx::umma_commit(acc_full(acc));
        }
        if (ok) ptx::umma_commit(a_empty);
      }
    }
  } else if (warp == kDcolLoadWarp) {
    if (lane == 0) {
      uint32_t e = 0;
      int seg = 0;
      bool ok = true;
      auto push = [&](const uint8_t* src, uint32_t bytes) {
        const int sb = e % kBStages;
        if (!ptx::mbar_wait(b_empty(sb), ((e / kBStages) & 1) ^ 1, abort_flag)) return false;
        ptx::mbar_arrive_expect_tx(b_full(sb), bytes);
        ptx::bulk_g2s(b_base + sb * kBStageBytes, src, bytes, b_full(sb));
        ++e;
        return true;
      };
      for (long long u = u_beg; ok && u < u_end; ++seg) {
        const int tile = (int)(u / p.NB), nb_beg = (int)(u % p.NB);
        const int nb_end = (int)min((long long)p.NB, nb_beg + (u_end - u));
        u += nb_end - nb_beg;
        if (!ptx::mbar_wait(a_empty, (seg & 1) ^ 1, abort_flag)) break;
        ptx::mbar_arrive_expect_tx(a_full, (uint32_t)a_bytes);
        const uint8_t* asrc = p.gy_img + (long long)tile * p.KBT * kABlockBytes;
        for (int off = 0; off < a_bytes; off += 32768)
          ptx::bulk_g2s(a_base + off, asrc + off, (uint32_t)min(32768, a_bytes - off), a_full);
        for (int nb = nb_beg; ok && nb < nb_end; ++nb) {
          const uint32_t wbytes = (uint32_t)(min(kNBlock, p.NT - nb * kNBlock) * 128);
          for (int kb = 0; ok && kb < p.KB; ++kb) {
            const uint8_t* w_hi = p.wt_img + ((long long)nb * p.KBT + kb) * kBStageBytes;
            ok = push(w_hi, wbytes) && push(asrc + p.gy_lo_off + (long long)kb * kABlockBytes, (uint32_t)kABlockBytes) &&
                 push(w_hi + p.wt_lo_off, wbytes);
          }
        }
      }
      // drain: never exit with a bulk copy in flight
      const uint32_t issued = e;
      for (uint32_t qq = (issued > (uint32_t)kBStages ? issued - kBStages : 0); qq < issued; ++qq) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(b_full(qq % kBStages), (qq / kBStages) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
      if (seg > 0) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(a_full, (seg - 1) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) ptx::report_device_timeout();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

// ---- (c) channels-last fp32 -> NCDHW ----------------------------------------------------------------
// The staging of x the other way round, with the same reasons: 16-byte loads, all requested before the first is stored.
// 512 channels, 2 x 8 x 30 x 54: 37 us with 32 x 32 tiles and 4-byte loads, now 18.
template <int kVox>
__global__ void __launch_bounds__(256)
unstage_grad_input_kernel(int C, long long Vin, const float* __restrict__ gx_cl, float* __restrict__ gx) {
  __shared__ float tile[64][kVox + 1];
  const int b = blockIdx.z, c0 = blockIdx.y * 64;
  const long long v0 = (long long)blockIdx.x * kVox;
  const int c = (threadIdx.x & 15) * 4, vr = threadIdx.x >> 4;
  float4 f[kVox / 16];
#pragma unroll
  for (int i = 0; i < kVox / 16; ++i) {
    const long long v = v0 + vr + 16 * i;
    f[i] = (v < Vin && c0 + c < C) ? __ldg(reinterpret_cast<const float4*>(gx_cl + ((long long)b * Vin + v) * C + c0 + c))
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int i = 0; i < kVox / 16; ++i) {
    const int vv = vr + 16 * i;
    tile[c][vv] = f[i].x; tile[c + 1][vv] = f[i].y; tile[c + 2][vv] = f[i].z; tile[c + 3][vv] = f[i].w;
  }
  __syncthreads();
  const int tx = threadIdx.x % kVox;
  const long long v = v0 + tx;
#pragma unroll
  for (int cc = threadIdx.x / kVox; cc < 64; cc += 256 / kVox)
    if (v < Vin && c0 + cc < C) gx[((long long)b * C + c0 + cc) * Vin + v] = tile[cc][tx];
}

// grad[b, c, v] *= d size_act / d raw (raw[b, c, v]) for the field's channels (both tensors with clip stride bstride)
__global__ void __launch_bounds__(256)
field_act_grad_kernel(const float* __restrict__ raw, float* __restrict__ grad, long long bstride, int nch, int V, int B, int act) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)B * nch * V) return;
  const long long b = i / ((long long)nch * V), r = i % ((long long)nch * V);
  grad[b * bstride + r] *= size_act_slope(act, __ldg(raw + b * bstride + r));
}

template <typename Coords>
int field_nch_of(const Coords&) { return 0; }
template <>
int field_nch_of<FieldCoords<float>>(const FieldCoords<float>& c) { return c.nch; }

struct BwdPlan {
  int nh, S, NT, KB, KBT, NB, tiles_per_clip, tmem_cols, smem_bytes, clips_per_chunk;
  bool pairg;       // 32 channels per offset group: a 64-channel slice holds two neighbouring groups
  bool split;       // fp32-parity mode with Cout > 256: separate hi / lo operand images, dcol_sm100_split_kernel
  long long gy_lo_off, wt_lo_off;
  size_t x_cl_bytes, rec_bytes, gat_bytes, gy_img_bytes, wt_img_bytes, dcol_bytes, gx_cl_bytes;
};

bool make_bwd_plan(const Geom& g, unsigned long long cap, bool x3, BwdPlan* pl) {
  // 32 channels per group (an even number of groups): groups are contiguous channel ranges, so slices of 64
  // channels simply span two of them
  pl->pairg = g.cpg == 32 && g.G % 2 == 0;
  if (g.groups != 1 || (g.cpg % 64 != 0 && !pl->pairg) || g.Cout % 64 != 0 || g.Cout > 512) return false;
  if (g.Vin * g.Cin > 0x7fffffffLL) return false;
  if ((long long)g.G * g.K * g.B > 65535) return false;
  if (g.K * 64 * (int)sizeof(float) > 48 * 1024 || g.Cin > 65535) return false;   // weight staging kernel
  pl->nh = pl->pairg ? 1 : g.cpg / 64;
  pl->S = pl->pairg ? (g.G / 2) * g.K : g.G * g.K * pl->nh;
  pl->NT = pl->S * 64;
  pl->split = x3 && g.Cout > 256;
  pl->KBT = g.Cout / ((x3 && !pl->split) ? 32 : 64);     // K blocks per image
  pl->KB = pl->KBT;                                      // all resident (<= 8 blocks of 16 KB)
  pl->NB = (pl->NT + kNBlock - 1) / kNBlock;
  pl->tiles_per_clip = (g.V + kBM - 1) / kBM;
  pl->tmem_cols = 512;
  pl->smem_bytes = pl->KB * kABlockBytes + kBStages * kBStageBytes + 256 + 1024;
  if (pl->smem_bytes > kSmemLimit) return false;
  pl->clips_per_chunk = exact::slice_clips(g, cap);
  pl->x_cl_bytes = align_up((size_t)g.B * g.Vin * g.Cin * (x3 ? 4 : 2), 256);
  pl->rec_bytes = pos_records_bytes(g);
  pl->gat_bytes = gather_records_bytes(g);
  pl->gy_lo_off = (long long)pl->clips_per_chunk * pl->tiles_per_clip * pl->KBT * kABlockBytes;
  pl->wt_lo_off = (long long)pl->NB * pl->KBT * kBStageBytes;
  pl->gy_img_bytes = align_up((size_t)pl->gy_lo_off * (pl->split ? 2 : 1), 256);
  pl->wt_img_bytes = align_up((size_t)pl->wt_lo_off * (pl->split ? 2 : 1), 256);
  pl->dcol_bytes = align_up((size_t)pl->clips_per_chunk * g.V * pl->NT * 4, 256);
  pl->gx_cl_bytes = align_up((size_t)g.B * g.Vin * g.Cin * 4, 256);
  return true;
}

template <typename Coords, bool FieldOut>
int run_bwd(const Geom& g, bool x3, const Coords& coords, unsigned long long cap, const float* gy, const float* x,
            const float* mask, const float* w, float* grad_x, float* grad_coord, size_t grad_coord_elems,
            float* grad_mask, float* grad_w, float* grad_bias, void* ws, cudaStream_t st, cudaEvent_t params_ready,
            const HeadCfg& head, const float* raw_field) {
  BwdPlan pl;
  if (!make_bwd_plan(g, cap, x3, &pl)) return D2C_ERR_MODE;
  uint8_t* wsp = reinterpret_cast<uint8_t*>(ws);
  void* x_cl = wsp; wsp += pl.x_cl_bytes;
  float4* recs = reinterpret_cast<float4*>(wsp); wsp += pl.rec_bytes;
  uint4* gat = reinterpret_cast<uint4*>(wsp); wsp += pl.gat_bytes;
  uint8_t* gy_img = wsp; wsp += pl.gy_img_bytes;
  uint8_t* wt_img = wsp; wsp += pl.wt_img_bytes;
  float* dcol = reinterpret_cast<float*>(wsp); wsp += pl.dcol_bytes;
  float* gx_cl = reinterpret_cast<float*>(wsp); wsp += pl.gx_cl_bytes;
  int* direct_word = reinterpret_cast<int*>(wsp); wsp += kWordBytes;
  void* dw_ws = wsp;

  int sm_count = 0, rc;
  if ((rc = device_sm_count(&sm_count))) return rc;
  ptx::bind_status_sink();
  ClStrides cs;
  cs.dz = g.H * g.W * g.Cin; cs.dy = g.W * g.Cin; cs.dx = g.Cin;
  const void* sav = nullptr;

  // dilation-field variant: tap positions per dim, read by the kernel that accumulates grad_size_map
  int field_nch = 0;
  int3 field_ch = make_int3(-1, -1, -1);
  FieldAxes axes{};
  if constexpr (FieldOut) {
    field_nch = coords.nch;
    field_ch = make_int3(coords.ch[0], coords.ch[1], coords.ch[2]);
    for (int d = 0; d < 3; ++d)
      for (int i = 0; i < kMaxFieldKernelDim; ++i) axes.pos[d][i] = coords.axis[d][i];
  }

  prof_mark(st, "bwd_stage_operands");
  if (FieldOut) {
    if (head.geo_bstride)      // the field's gradient channels inside the raw gradient: nch planes per clip
      D2C_CUDA_TRY(cudaMemset2DAsync(grad_coord, sizeof(float) * head.geo_bstride, 0, sizeof(float) * field_nch_of(coords) * g.V,
                                     g.B, st));
    else
      D2C_CUDA_TRY(cudaMemsetAsync(grad_coord, 0, sizeof(float) * grad_coord_elems, st));
  }
  if (grad_bias) D2C_CUDA_TRY(cudaMemsetAsync(grad_bias, 0, sizeof(float) * g.Cout, st));
  // What the forward of this call kept in this mode's format: its operand tiles (the weight gradient streams them, no
  // gather records needed), the staged input and the position records -- nothing is staged a second time.
  if (SampleCache* sc = current_sample_cache()) {
    int np = 0;
    SampleCacheLayout lay{};
    if (sc->data && sc->format == (x3 ? 2 : 1) && sm100_sample_cache_layout(g, x3, &np, &lay) && sc->bytes >= lay.total()) {
      sav = sc->data;
      x_cl = reinterpret_cast<uint8_t*>(sc->data) + lay.image_bytes;
      recs = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(sc->data) + lay.image_bytes + lay.x_cl_bytes);
    }
  }
  if (!sav) {
    rc = x3 ? launch_stage_input(g, x, reinterpret_cast<float*>(x_cl), ZeroFill{nullptr, 0}, nullptr, sm_count, st)
            : launch_stage_input(g, x, reinterpret_cast<__half*>(x_cl), ZeroFill{nullptr, 0}, nullptr, sm_count, st);
    if (rc) return rc;
    if (!sav && (rc = launch_sample_records(g, coords, mask, head, recs, gat, st, x3))) return rc;
  }
  // The parameter gradients come first: the weight gradient (tensor-core implicit GEMM over the re-sampled tile)
  // needs only the records and the staged input, and its grad_out staging pass also sums grad_bias.  A caller that
  // reduces them across GPUs can start as soon as `params_ready` fires, under the data-side kernels below.
  if ((rc = sm100_dw(g, x3, gy, x_cl, gat, grad_w, grad_bias, dw_ws, st, ZeroFill{gx_cl, (long long)g.B * g.Vin * g.Cin * 4}, sav))) return rc;
  if (params_ready) D2C_CUDA_TRY(cudaEventRecord(params_ready, st));
  prof_mark(st, "bwd_stage_weights");
  const int img_mode = pl.split ? 2 : (x3 ? 1 : 0);
  stage_wt_img_kernel<<<dim3((unsigned)pl.KBT, (unsigned)g.Cin), 64, 64 * g.K * sizeof(float), st>>>(
      g.Cout, g.Cin, g.K, pl.pairg ? 64 : g.cpg, pl.nh, img_mode, w, wt_img, pl.wt_lo_off);
  D2C_LAUNCH_CHECK();
  rc = pl.split ? allow_dynamic_smem<dcol_sm100_split_kernel>(pl.smem_bytes)
                : (x3 ? allow_dynamic_smem<dcol_sm100_kernel<1>>(pl.smem_bytes) : allow_dynamic_smem<dcol_sm100_kernel<0>>(pl.smem_bytes));
  if (rc) return rc;

  for (int b0 = 0; b0 < g.B; b0 += pl.clips_per_chunk) {
    const int nbc = (g.B - b0 < pl.clips_per_chunk) ? g.B - b0 : pl.clips_per_chunk;
    const int n_tiles = nbc * pl.tiles_per_clip;
    const SampleGradPlan sp = sample_grad_plan(g, nbc, pl.nh, FieldOut, x3, pl.pairg, sm_count);
    const long long n_clip_recs = (long long)g.G * g.K * g.V;
    const PositionAsk ask{g, recs + b0 * n_clip_recs, sp.ask ? nbc * n_clip_recs : 0, voxel_order(g), sp.taps, FieldOut, field_ch, axes,
                          direct_word};
    prof_mark(st, "bwd_stage_grad_out");
    stage_gy_img_kernel<<<dim3((unsigned)(n_tiles + (sp.ask ? 1 : 0)), (unsigned)pl.KBT), 256, 0, st>>>(
        g.Cout, g.V, pl.tiles_per_clip, b0, img_mode, gy, gy_img, pl.gy_lo_off, ask);
    D2C_LAUNCH_CHECK();
    DcolParams p;
    p.gy_img = gy_img; p.wt_img = wt_img; p.dcol = dcol;
    p.V = g.V; p.NT = pl.NT; p.KB = pl.KB; p.NB = pl.NB;
    p.tiles_per_clip = pl.tiles_per_clip; p.n_tiles = n_tiles; p.n_units = (long long)n_tiles * pl.NB;
    p.tmem_cols = pl.tmem_cols;
    // a unit is 1-3 us of MMAs and stores, the grad_out tile that a CTA loads first less than one: units are spread over
    // all multiprocessors before any takes a second one
    long long grid = p.n_units;
    if (grid > sm_count) grid = sm_count;
    if (grid < 1) grid = 1;
    prof_mark(st, "bwd_dcol_sm100");
    p.KBT = pl.KBT; p.kb0 = 0; p.KB = pl.KB;
    p.gy_lo_off = pl.gy_lo_off; p.wt_lo_off = pl.wt_lo_off;
    if (pl.split)
      dcol_sm100_split_kernel<<<(unsigned)grid, kDcolThreads, pl.smem_bytes, st>>>(p);
    else if (x3)
      dcol_sm100_kernel<1><<<(unsigned)grid, kDcolThreads, pl.smem_bytes, st>>>(p);
    else
      dcol_sm100_kernel<0><<<(unsigned)grid, kDcolThreads, pl.smem_bytes, st>>>(p);
    D2C_LAUNCH_CHECK();
    prof_mark(st, "bwd_sample_grad");
    const size_t smem = sample_grad_smem(sp.taps, pl.nh);
    auto launch = [&](auto f32x, auto narrow, auto multi) -> int {
      constexpr bool kF32X = decltype(f32x)::value, kNarrow = decltype(narrow)::value, kMulti = decltype(multi)::value;
      constexpr bool kMayAsk = !FieldOut || kMulti;
      const int3 blocks = make_int3((int)sp.grid.x, (int)sp.grid.y, (int)sp.grid.z);
      auto direct = [&](auto kernel, const dim3& grid) -> int {
        kernel<<<grid, kSgThreads, 0, st>>>(g, cs, b0, pl.nh, recs, dcol, x_cl, mask != nullptr, grad_coord, grad_mask, gx_cl,
                                            field_nch, field_ch, axes, sp.taps, head, blocks, direct_word);
        D2C_LAUNCH_CHECK();
        return D2C_OK;
      };
      if (!sp.lists) return direct(sample_grad_direct_kernel<FieldOut, kF32X, kNarrow, false>, sp.grid);
      if constexpr (kMayAsk) {
        const int few = std::min((kF32X || !kNarrow ? 2 : 3) * sm_count, blocks.x * blocks.y * blocks.z);
        if (sp.ask && (rc = direct(sample_grad_direct_kernel<FieldOut, kF32X, kNarrow, true>, (unsigned)few))) return rc;
      }
      constexpr auto kernel = sample_grad_taps_kernel<FieldOut, kF32X, kNarrow, kMulti>;
      const int rc = allow_dynamic_smem<kernel>((int)smem);
      if (rc) return rc;
      if (sp.ask) {
        D2C_CUDA_TRY(launch_beside(kernel, sp.grid, kSgThreads, smem, st, g, voxel_order(g), cs, b0, pl.nh, recs, dcol, x_cl, mask != nullptr,
                                   grad_coord, grad_mask, gx_cl, field_nch, field_ch, axes, sp.taps, head, direct_word));
      } else {
        kernel<<<sp.grid, kSgThreads, smem, st>>>(g, voxel_order(g), cs, b0, pl.nh, recs, dcol, x_cl, mask != nullptr, grad_coord, grad_mask,
                                                  gx_cl, field_nch, field_ch, axes, sp.taps, head, nullptr);
      }
      D2C_LAUNCH_CHECK();
      return D2C_OK;
    };
    const std::true_type yes;
    const std::false_type no;
    if (pl.pairg)
      rc = x3 ? launch(yes, yes, no) : launch(no, yes, no);
    else if (pl.nh > 1)
      rc = x3 ? launch(yes, no, yes) : launch(no, no, yes);
    else
      rc = x3 ? launch(yes, no, no) : launch(no, no, no);
    if (rc) return rc;
  }
  if constexpr (FieldOut) {
    if (head.size_act != 0 && raw_field) {      // chain rule through the size activation, on the summed gradient
      const long long n = (long long)g.B * field_nch * g.V;
      field_act_grad_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
          raw_field, grad_coord, head.geo_bstride ? head.geo_bstride : (long long)field_nch * g.V, field_nch, g.V, g.B,
          head.size_act);
      D2C_LAUNCH_CHECK();
    }
  }
  prof_mark(st, "bwd_unstage_grad_input");
  {
    const dim3 grid((unsigned)((g.Vin + 63) / 64), (unsigned)((g.Cin + 63) / 64), (unsigned)g.B);
    if ((long long)grid.x * grid.y * grid.z >= 2LL * sm_count)
      unstage_grad_input_kernel<64><<<grid, 256, 0, st>>>(g.Cin, g.Vin, gx_cl, grad_x);
    else      // multiprocessors without a block
      unstage_grad_input_kernel<32><<<dim3((unsigned)((g.Vin + 31) / 32), grid.y, grid.z), 256, 0, st>>>(g.Cin, g.Vin, gx_cl, grad_x);
    D2C_LAUNCH_CHECK();
  }
  prof_mark(st, nullptr);
  return D2C_OK;
}

}  // namespace

// bf16 mode runs the single-pass kernels where their plans fit (32 channels per group: the weight gradient needs
// room for a second record set, i.e. Cout <= 256) and the fp32-parity kernels otherwise.
static bool bwd_use_x3(const Geom& g, int math_mode, unsigned long long cap) {
  if (math_mode != D2C_MATH_BF16) return true;
  BwdPlan pl;
  return !(make_bwd_plan(g, cap, false, &pl) && sm100_dw_workspace(g, false) > 0);
}

bool sm100_bwd_variant(const Geom& g, int math_mode, unsigned long long cap, bool* x3) {
  *x3 = bwd_use_x3(g, math_mode, cap);
  BwdPlan pl;
  return make_bwd_plan(g, cap, *x3, &pl) && sm100_dw_workspace(g, *x3) > 0;
}

bool sm100_bwd_supported(const Geom& g, int dtype, int math_mode, unsigned long long cap) {
  if (dtype != D2C_F32 || math_mode == D2C_MATH_FP32) return false;
  const bool x3 = bwd_use_x3(g, math_mode, cap);
  BwdPlan pl;
  return make_bwd_plan(g, cap, x3, &pl) && sm100_dw_workspace(g, x3) > 0;
}

size_t sm100_bwd_workspace(const Geom& g, int dtype, int math_mode, unsigned long long cap) {
  if (!sm100_bwd_supported(g, dtype, math_mode, cap)) return 0;
  const bool x3 = bwd_use_x3(g, math_mode, cap);
  BwdPlan pl;
  make_bwd_plan(g, cap, x3, &pl);
  return pl.x_cl_bytes + pl.rec_bytes + pl.gat_bytes + pl.gy_img_bytes + pl.wt_img_bytes + pl.dcol_bytes + pl.gx_cl_bytes + kWordBytes +
         sm100_dw_workspace(g, x3);
}

int sm100_bwd_offsets(const Geom& g, int math_mode, unsigned long long cap, const float* gy, const float* x, const float* offset,
                      const float* mask, const float* w, float* grad_x, float* grad_offset, float* grad_mask,
                      float* grad_w, float* grad_bias, void* ws, cudaStream_t st, cudaEvent_t params_ready,
                      const HeadCfg& head) {
  OffsetCoords<float> oc{offset, head.geo_bstride};
  return run_bwd<OffsetCoords<float>, false>(g, bwd_use_x3(g, math_mode, cap), oc, cap, gy, x, mask, w, grad_x, grad_offset, 0, grad_mask, grad_w,
                                             grad_bias, ws, st, params_ready, head, nullptr);
}

int sm100_bwd_field(const Geom& g, int math_mode, unsigned long long cap, const FieldCoords<float>& fc, const float* gy,
                    const float* x, const float* mask, const float* w, float* grad_x, float* grad_size_map,
                    size_t grad_size_elems, float* grad_mask, float* grad_w, float* grad_bias, void* ws,
                    cudaStream_t st, cudaEvent_t params_ready, const HeadCfg& head) {
  return run_bwd<FieldCoords<float>, true>(g, bwd_use_x3(g, math_mode, cap), fc, cap, gy, x, mask, w, grad_x, grad_size_map, grad_size_elems,
                                           grad_mask, grad_w, grad_bias, ws, st, params_ready, head, fc.size_map);
}

}  // namespace d2c
