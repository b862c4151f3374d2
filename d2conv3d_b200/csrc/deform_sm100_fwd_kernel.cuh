// The single-CTA forward kernel (included by deform_sm100_fwd.cu, whose constants, FwdParams and gather helpers it
// uses).  Warps: 4 epilogue | MMA, weight loader, record loader, one idle | 24 gather, of 64 registers a thread each.
// Optional instrumentation (compiled in with -DD2C_UNIT_TRACE, `python -m d2conv3d_b200.build --unit-trace`): every
// role of ONE CTA stamps clock64() at fixed points of its per-unit loop for a window of 64 units, and every CTA
// records its start / end (globaltimer), its SM and its unit count.  Read with `python -m d2conv3d_b200.unit_trace`.
// Layout of the buffer (long long): [role 0..4][unit 0..63][event 0..7], then [CTA][t0, t1, smid, units].
// Roles: 0 record loader, 1 weight loader, 2 MMA issuer, 3 / 4 first / last gather warp (lane 0).
#ifdef D2C_UNIT_TRACE
#define D2C_TR(role, k, e)                                                                                    \
  do {                                                                                                        \
    if (p.trace && (int)blockIdx.x == p.trace_cta && (int)(k) >= p.trace_k0 && (int)(k) < p.trace_k0 + 64)    \
      p.trace[((role) * 64 + ((int)(k) - p.trace_k0)) * 8 + (e)] = clock64();                                 \
  } while (0)
#else
#define D2C_TR(role, k, e) ((void)0)
#endif

constexpr int kThreadsFwd = 32 * 32;
constexpr int kGatherWarpsFwd = 24;
constexpr int kUnitItems = kBM / 8;               // a gather warp's item: 8 rows of a unit
constexpr int kMmaWarpFwd = 4, kLoadWarpFwd = 5, kRecWarpFwd = 6, kIdleWarpFwd = 7, kGatherWarp0Fwd = 8;

// kX3 = 0: math mode bf16 (a unit is 64 channels of one tap, one bf16 operand pair).
// kX3 = 1: math mode bf16x3, the fp32-parity mode: a unit is 32 channels; the A row holds [hi(32) | lo(32)] of
//          the fp32 blend, the weight row [hi(32) | lo(32)] of the fp32 weight, and the issuer forms
//          a_hi*b_hi + a_lo*b_hi + a_hi*b_lo from the 16-channel K sub-blocks of the same two tiles.
// kDual = 1 (single-pass mode only): 32 channels per offset group, a 64-channel unit spans two groups.
// kSave = 1: the blended tiles are also written to FwdParams::sav (a forward whose backward will follow).  A template
//          parameter, not a run-time test, so that the inference kernel carries neither the stores nor the registers
//          for their addresses.
// kShared = 1: records shared by the offset groups and separate modulation rows (sm100_gather.cuh).
template <int kX3, int kDual, int kSave, int kShared>
__global__ void __launch_bounds__(kThreadsFwd, 1)
fwd_sm100_kernel(const FwdParams p) {
  constexpr int kUnitCh = kX3 ? 32 : 64;
  constexpr int kRStage = kRStageBytesOf(kDual, kShared);
  constexpr int hdr_off = kRStage - 16;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const int rec_off = kAStages * kAStageBytes + p.b_stages * p.b_stage_bytes;
  const int bar_off = rec_off + kRStages * kRStage;
  const uint32_t a_base = base, b_base = base + kAStages * kAStageBytes, rec_base = base + rec_off,
                 bar_base = base + bar_off;
  auto a_full = [&](int s) { return bar_base + 8u * s; };
  auto a_empty = [&](int s) { return bar_base + 8u * (kAStages + s); };
  auto b_full = [&](int s) { return bar_base + 8u * (2 * kAStages + s); };
  auto b_empty = [&](int s) { return bar_base + 8u * (2 * kAStages + 4 + s); };
  const uint32_t acc_full = bar_base + 8u * (2 * kAStages + 8);
  const uint32_t acc_empty = bar_base + 8u * (2 * kAStages + 9);
  auto r_full = [&](int s) { return bar_base + 8u * (2 * kAStages + 11 + s); };
  auto r_empty = [&](int s) { return bar_base + 8u * (2 * kAStages + 11 + kRStages + s); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + bar_off + 8 * (2 * kAStages + 10));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + bar_off + 8 * (2 * kAStages + 10) + 4);

#ifdef D2C_UNIT_TRACE
  unsigned long long cta_t0;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(cta_t0));
#endif
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Geom& g = p.g;
  // A CTA's work is n_parts (<= 16) contiguous unit ranges, one inside every clip (cta_part_range in
  // deform_sm100_fwd.cu); ring slots, phases and segment counters run on across the parts, positions restart at every
  // part.  Thread 0 puts the ranges into shared memory once, so that the roles do no 64-bit division.
  // (unit indices fit 31 bits: checked by the host)
  int* part_tab = reinterpret_cast<int*>(base_ptr + bar_off + 256);      // [part][beg, end], the total, whether x holds a NaN
  // Large volumes (FwdParams::rr): whole tiles dealt round-robin instead -- at any time the CTAs then work on
  // gridDim.x CONSECUTIVE tiles, whose sampling neighbourhoods overlap, so the part of the staged input they gather
  // from is a few planes and not a few planes around 148 places spread over the whole volume (which L2 cannot hold:
  // the stride-4 decoder layer re-fetched its 210 MB input 22 times).
  auto part_range = [&](int part, int& beg, int& end) {
    if (p.rr) {
      const int tile = part * (int)gridDim.x + (int)blockIdx.x;
      beg = tile * p.S;
      end = tile < p.n_tiles ? beg + p.S : beg;
    } else {
      beg = part_tab[2 * part];
      end = part_tab[2 * part + 1];
    }
  };

  if (threadIdx.x == 0) {
    int total = 0;
    if (p.rr) {
      // round-robin tiles: part r is tile r * gridDim.x + blockIdx.x (computed where it is needed)
      for (int tile = (int)blockIdx.x; tile < p.n_tiles; tile += (int)gridDim.x) total += p.S;
    } else {
      for (int part = 0; part < p.n_parts; ++part) {
        long long pb, pe;
        cta_part_range(p, part, pb, pe);
        part_tab[2 * part] = (int)pb; part_tab[2 * part + 1] = (int)pe;
        total += (int)(pe - pb);
      }
    }
    part_tab[32] = total;
    for (int s = 0; s < kAStages; ++s) { ptx::mbar_init(a_full(s), kUnitItems); ptx::mbar_init(a_empty(s), 1); }
    for (int s = 0; s < p.b_stages; ++s) { ptx::mbar_init(b_full(s), 1); ptx::mbar_init(b_empty(s), 1); }
    for (int s = 0; s < kRStages; ++s) { ptx::mbar_init(r_full(s), 1); ptx::mbar_init(r_empty(s), kUnitItems); }
    ptx::mbar_init(acc_full, 1);
    ptx::mbar_init(acc_empty, kEpiWarps);
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  // by a warp without a role, beside the set-up (in the producers it would delay a call's first unit by up to 0.6 us).  A volatile
  // load: the staging kernel may write the word while this one already runs, so that it is not read-only for this kernel's life.
  if (threadIdx.x == kIdleWarpFwd * 32) {
    wait_for_kernels_before();
    part_tab[33] = *static_cast<const volatile int*>(p.nan_flag);
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32((const void*)tmem_slot), (uint32_t)p.tmem_cols);
    ptx::tmem_relinquish();
  }
  wait_for_kernels_before();         // what was staged is there from here on
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < kEpiWarps) {
    // ===================== epilogue: one pass per tile segment =====================
    int seg = 0;
    for (int part = 0; part < p.n_parts; ++part) {
    if (*abort_flag) break;
    int u_beg, u_end;
    part_range(part, u_beg, u_end);
    for (int u = u_beg; u < u_end; ++seg) {
      const int tile = u / p.S, s_beg = u % p.S;
      const int s_end = min(min(p.S, s_beg + (u_end - u)), s_beg + p.seg_cap);
      u += s_end - s_beg;
      const bool whole = (s_beg == 0 && s_end == p.S);
      const int b = tile / p.tiles_per_clip, v0 = (tile % p.tiles_per_clip) * kBM;
      if (!ptx::mbar_wait(acc_full, seg & 1, abort_flag, 2000)) break;
      ptx::tc_fence_after();
      const int v = v0 + warp * 32 + lane;
      float* yb = p.y + (long long)b * g.Cout * g.V + v;
      if ((g.V & 3) == 0) {
        // Each lane holds 32 channels of ONE voxel; y is [clip][channel][voxel], so a lane's values lie V floats
        // apart.  A 4 x 4 transpose inside every lane quad (two shuffle stages) gives lane q of the quad channel
        // 4i + q of the quad's four consecutive voxels: 16-byte stores / vector reductions, a quarter of the memory
        // instructions (the partial-tile epilogue was bound by their issue, not by bytes).
        const int q = lane & 3;
        const int vq = v0 + warp * 32 + (lane & ~3);
        float* yq = p.y + (long long)b * g.Cout * g.V + vq;
        const bool live = vq < g.V;                      // V is a multiple of 4: a quad is valid or invalid as a whole
        for (int c0 = 0; c0 < p.N; c0 += 32) {
          uint32_t r[32];
          ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint32_t* a = r + 4 * i;
            const uint32_t t0 = __shfl_xor_sync(0xffffffffu, (q & 1) ? a[0] : a[1], 1);
            const uint32_t t1 = __shfl_xor_sync(0xffffffffu, (q & 1) ? a[2] : a[3], 1);
            if (q & 1) { a[0] = t0; a[2] = t1; } else { a[1] = t0; a[3] = t1; }
            const uint32_t u0 = __shfl_xor_sync(0xffffffffu, (q & 2) ? a[0] : a[2], 2);
            const uint32_t u1 = __shfl_xor_sync(0xffffffffu, (q & 2) ? a[1] : a[3], 2);
            if (q & 2) { a[0] = u0; a[1] = u1; } else { a[2] = u0; a[3] = u1; }
            if (live) {
              const int c = c0 + 4 * i + q;
              const float bb = (p.bias && (whole || s_beg == 0)) ? __ldg(p.bias + c) : 0.f;
              float* dst = yq + (long long)c * g.V;
              const float f0 = __uint_as_float(a[0]) + bb, f1 = __uint_as_float(a[1]) + bb,
                          f2 = __uint_as_float(a[2]) + bb, f3 = __uint_as_float(a[3]) + bb;
              if (whole)
                *reinterpret_cast<float4*>(dst) = make_float4(f0, f1, f2, f3);
              else
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(f0), "f"(f1), "f"(f2), "f"(f3)
                             : "memory");
            }
          }
        }
      } else {
      for (int c0 = 0; c0 < p.N; c0 += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
        ptx::tmem_ld_wait();
        if (v < g.V) {
          if (whole) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float bb = p.bias ? __ldg(p.bias + c0 + j) : 0.f;
              yb[(long long)(c0 + j) * g.V] = __uint_as_float(r[j]) + bb;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float bb = (p.bias && s_beg == 0) ? __ldg(p.bias + c0 + j) : 0.f;
              atomicAdd(yb + (long long)(c0 + j) * g.V, __uint_as_float(r[j]) + bb);
            }
          }
        }
      }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(acc_empty);
    }
    }
  } else if (warp < kGatherWarp0Fwd) {
   if (warp == kMmaWarpFwd) {
    // ===================== MMA issuer =====================
    if (lane == 0) {
      // One thread drives the tensor core, so its own instruction latency is on the critical path of every unit:
      // no integer division or modulo by run-time values in the per-unit path (ring slots and phases are carried as
      // counters), descriptors are built from constants hoisted out of the loops.
      int seg = 0;
      uint32_t k = 0;           // units consumed so far
      int sb = 0;               // weight-ring slot and its phase
      uint32_t phb = 0;
      bool ok = true;
      constexpr int kSteps = kX3 ? 6 : 4;
      // K sub-blocks (16 channels = 32 bytes) of the A and B rows that meet in each MMA
      constexpr int ka_[6] = {0, 1, kX3 ? 2 : 2, kX3 ? 3 : 3, 0, 1};   // bf16: (k,k); x3: hi*hi, lo*hi, hi*lo
      constexpr int kb_[6] = {0, 1, kX3 ? 0 : 2, kX3 ? 1 : 3, 2, 3};
      const int n_blocks = (p.N + 255) / 256;      // N blocks of a slice, one weight stage each
      const uint32_t idesc_full = ptx::umma_idesc_bf16_f32(kBM, 256);
      const uint32_t idesc_last = ptx::umma_idesc_bf16_f32(kBM, p.N - (n_blocks - 1) * 256);
      const uint64_t adesc0 = ptx::umma_desc_kmajor_sw128(a_base), bdesc0 = ptx::umma_desc_kmajor_sw128(b_base);
      const uint64_t a_step = (uint64_t)(kAStageBytes >> 4), b_step = (uint64_t)(p.b_stage_bytes >> 4);
      for (int part = 0; ok && part < p.n_parts; ++part) {
      if (*abort_flag) break;
      int u_beg, u_end;
    part_range(part, u_beg, u_end);
      int s_beg = u_beg % p.S;                                          // once per part
      for (int u = u_beg; ok && u < u_end; ++seg) {
        const int s_end = min(min(p.S, s_beg + (u_end - u)), s_beg + p.seg_cap);
        u += s_end - s_beg;
        if (!ptx::mbar_wait(acc_empty, (seg & 1) ^ 1, abort_flag)) break;
        ptx::tc_fence_after();
        for (int s = s_beg; s < s_end; ++s, ++k) {
          const int sa = k & (kAStages - 1);
          D2C_TR(2, k, 0);
          if (!ptx::mbar_wait(a_full(sa), (k / kAStages) & 1, abort_flag)) { ok = false; break; }
          D2C_TR(2, k, 1);
          ptx::tc_fence_after();
          // descriptor address fields count 16-byte units: a stage further along adds stage_bytes / 16
          const uint64_t adesc = adesc0 + a_step * (uint64_t)sa;
          for (int h = 0; h < n_blocks; ++h) {
            if (!ptx::mbar_wait(b_full(sb), phb, abort_flag)) { ok = false; break; }
            D2C_TR(2, k, 2);
            ptx::tc_fence_after();
            const uint64_t bdesc = bdesc0 + b_step * (uint64_t)sb;
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk)
              ptx::umma_bf16(tmem_base + (uint32_t)(h * 256), adesc + (uint64_t)(2 * ka_[kk]), bdesc + (uint64_t)(2 * kb_[kk]),
                             h + 1 < n_blocks ? idesc_full : idesc_last, (s > s_beg || kk > 0) ? 1u : 0u);
            D2C_TR(2, k, 3);
            ptx::umma_commit(b_empty(sb));
            if (++sb == p.b_stages) { sb = 0; phb ^= 1u; }
          }
          if (!ok) break;
          ptx::umma_commit(a_empty(sa));
          D2C_TR(2, k, 4);
        }
        if (ok) ptx::umma_commit(acc_full);
        s_beg = s_end == p.S ? 0 : s_end;
      }
      }
    }
  } else if (warp == kLoadWarpFwd) {
    // ===================== weight-slice loader =====================
    if (lane == 0) {
      [[maybe_unused]] uint32_t k = 0;
      uint32_t issued = 0;
      int sb = 0;                       // ring slot and phase as counters: no division in the per-unit path
      uint32_t phb = 1;                 // the wait for a FREE slot looks at the previous phase
      for (int part = 0; part < p.n_parts; ++part) {
      if (*abort_flag) break;
      int u_beg, u_end;
    part_range(part, u_beg, u_end);
      int s = u_beg % p.S;              // once per part
      const uint8_t* src = p.w_sw + (long long)s * p.w_slice_bytes;
      const int n_part_units = u_end - u_beg;
      bool ok = true;
      for (int i = 0; ok && i < n_part_units; ++i, ++k) {
        D2C_TR(1, k, 0);
        for (int off = 0; off < p.w_slice_bytes; off += p.b_stage_bytes) {
          if (!ptx::mbar_wait(b_empty(sb), phb, abort_flag, 200)) { ok = false; break; }
          D2C_TR(1, k, 1);
          const uint32_t bytes = (uint32_t)min(p.b_stage_bytes, p.w_slice_bytes - off);
          ptx::mbar_arrive_expect_tx(b_full(sb), bytes);
          ptx::bulk_g2s(b_base + sb * p.b_stage_bytes, src + off, bytes, b_full(sb));
          ++issued;
          if (++sb == p.b_stages) { sb = 0; phb ^= 1u; }
        }
        src += p.w_slice_bytes;
        if (++s == p.S) { s = 0; src = p.w_sw; }
      }
      }
      // never leave with a bulk copy in flight: wait (bounded) for the last copies issued
      for (uint32_t q = (issued > (uint32_t)p.b_stages ? issued - p.b_stages : 0); q < issued; ++q) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(b_full(q % p.b_stages), (q / p.b_stages) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
    }
  } else if (warp == kRecWarpFwd) {
    // ===================== gather-record loader =====================
    // The records of a unit's rows are one contiguous run of the [B][G][K][V] stream: one bulk copy per unit, into a ring from which the
    // producers read them.  The ring has kRStages units; a copy starts once the one two units before it is there.
    if (lane == 0) {
      uint32_t k = 0;
      // position of the first unit, once per CTA; then everything advances by counters (this single thread's
      // instruction latency sits between "stage free" and "copy issued" for every unit: no division in the loop)
      const long long grp_ch = kDual ? 2 * g.cpg : g.cpg;
      const uint64_t pol_stream = ptx::l2_evict_first();       // records are read once
      for (int part = 0; part < p.n_parts; ++part) {
      if (*abort_flag) break;
      int u_beg, u_end;
    part_range(part, u_beg, u_end);
      int s = u_beg % p.S;
      const int tile0 = u_beg / p.S;
      int b = tile0 / p.tiles_per_clip, v0 = (tile0 % p.tiles_per_clip) * kBM;
      int tile = tile0;
      int tap = s % g.K, h = (s / g.K) % p.nh, grp = (s / g.K) / p.nh;   // dual: grp is the index of a group PAIR
      const int n_part_units = u_end - u_beg;
      for (int i = 0; i < n_part_units; ++i, ++k) {
        const int sr = k & (kRStages - 1);
        D2C_TR(0, k, 0);
        if (!ptx::mbar_wait(r_empty(sr), ((k / kRStages) & 1) ^ 1, abort_flag, 200)) break;
        // A gather warp leaves out one unit at most between two items, so that it may wait for unit k when it has seen k - 2.  The
        // parity it waits for is that of k only if the stage's last copy, k - 4, is there: copies are started in that order.
        if (k >= 2 && !ptx::mbar_wait(r_full((k - 2) % kRStages), ((k - 2) / kRStages) & 1, abort_flag)) break;
        D2C_TR(0, k, 1);
        const int rows = min(kBM, g.V - v0);
        // unit header for the gather warps (no index arithmetic there); ordered before their reads by the
        // release of the arrive below and the acquire of their wait
        uint8_t* hdr = base_ptr + rec_off + sr * kRStage + hdr_off;
        *reinterpret_cast<long long*>(hdr) = (long long)b * g.Vin * g.Cin + grp * grp_ch + h * kUnitCh;
        *reinterpret_cast<int*>(hdr + 8) = rows;
        if constexpr (kSave) {
          // where this unit's samples go in the image kept for the weight gradient (8 KB blocks, see FwdParams)
          int word;
          if constexpr (kX3) {
            // 64-channel slice of the weight gradient that holds this 32-channel unit, and which half of it
            const int s64 = p.sav_pairg ? (grp >> 1) * g.K + tap : (grp * g.K + tap) * (p.nh >> 1) + (h >> 1);
            const int half = p.sav_pairg ? (grp & 1) : (h & 1);
            word = (((tile * 2 * p.sav_np + (s64 >> 1)) * 4 + (s64 & 1)) << 1) | half;
          } else {
            word = tile * 2 * (2 * p.sav_np) + (grp * g.K + tap) * p.nh + h;
          }
          *reinterpret_cast<int*>(hdr + 12) = word;
        }
        const uint32_t bytes = (uint32_t)rows * 48u;
        if constexpr (kShared) {
          const uint32_t m_bytes = (uint32_t)(rows + 3) / 4 * 16;
          ptx::mbar_arrive_expect_tx(r_full(sr), bytes + m_bytes * (uint32_t)(1 + kDual));
          ptx::bulk_g2s(rec_base + sr * kRStage, p.recs + 3 * (((long long)b * g.K + tap) * g.V + v0), bytes, r_full(sr));
#pragma unroll
          for (int set = 0; set <= kDual; ++set)
            ptx::bulk_g2s_hint(rec_base + sr * kRStage + kRecBytes + set * kMaskBytes,
                               p.masks + (((long long)b * g.G + (kDual ? 2 * grp + set : grp)) * g.K + tap) * mask_row(g.V) + v0, m_bytes,
                               r_full(sr), pol_stream);
        } else {
        ptx::mbar_arrive_expect_tx(r_full(sr), bytes * (uint32_t)(1 + kDual));
#pragma unroll
        for (int set = 0; set <= kDual; ++set) {
          const int og = kDual ? 2 * grp + set : grp;      // offset group whose records fill this set
          ptx::bulk_g2s_hint(rec_base + sr * kRStage + set * kRecBytes,
                             p.recs + 3 * ((((long long)b * g.G + og) * g.K + tap) * g.V + v0), bytes, r_full(sr), pol_stream);
        }
        }
        // next unit: (tap, h, grp) count through the tile's slices, then the next tile of the clip / next clip
        if (++tap == g.K) {
          tap = 0;
          if (++h == p.nh) { h = 0; ++grp; }
        }
        if (++s == p.S) {
          s = 0; h = 0; tap = 0; grp = 0;
          ++tile;
          v0 += kBM;
          if (v0 >= p.tiles_per_clip * kBM) { v0 = 0; ++b; }
        }
      }
      }
      const uint32_t issued = k;
      for (uint32_t q = (issued > (uint32_t)kRStages ? issued - kRStages : 0); q < issued; ++q) {
        const long long t0 = clock64();
        while (!ptx::mbar_try_wait(r_full(q % kRStages), (q / kRStages) & 1))
          if (clock64() - t0 > ptx::kWaitBudgetCycles) break;
      }
    }
   }
  } else {
    // ===================== gather producers =====================
    // An item is 8 rows of a unit; a warp takes every 24th.  A thread owns 32 bytes (a quarter) of one row's 128: 8 fp32 or 16 fp16
    // channels, so that one record, one header and eight addresses serve 32 bytes of every corner and a row's 16-byte chunks of the
    // A tile need no exchange between lanes.  The corners of the z ceil half are requested as those of the z floor half are blended.
    // Bound by the latency of an item's chain (record, corners, corners, tile) over the warps there are: 24 warps that hold four
    // corners beat 16 that hold eight and look a unit ahead, whose instructions between loads added up instead of overlapping
    // (without its loads that kernel took half its time, with them half as much again).  Measured, 16 / 24 warps: 256-channel
    // field layer of one group on 2 x 8 x 60 x 107 1.36 / 1.27 ms, of eight groups on 8 x 120 x 214 2.99 / 2.55, 1024 -> 256
    // channels in 8 groups on 8 x 30 x 54 single pass 404 / 368 us, 512 channels in 8 groups on 2 x 8 x 30 x 54 1.06 / 1.04 ms, single
    // pass 0.50 / 0.48.  The last 3 % of it is one 8-byte read of the record that does not wait for the header.  Not faster:
    // corners of the next item requested under the blend (+6 %), the hand-over put off under the next item's loads, two slices
    // of one record an item (spills), the voxels of a tile in bricks (half the requests hit L1, but a request with one miss runs
    // at the rate of a miss).
    const int j = lane & 3;          // 32-byte quarter of the row
    // the two rows of a quarter warp (one shared-memory store phase) differ in the bit that keeps their chunks apart:
    // fp32-parity stores chunk j, then 4 + j (rows r and r + 4); single pass stores chunks 2j and 2j + 1 (rows r and r + 1)
    const int r8 = kX3 ? ((lane >> 3) & 3) | ((lane & 4)) : lane >> 2;
    const uint32_t chunk0 = (uint32_t)(((kX3 ? j : 2 * j) ^ r8) << 4), chunk1 = (uint32_t)(((kX3 ? 4 + j : 2 * j + 1) ^ r8) << 4);
    const uint64_t pol_stream = ptx::l2_evict_first();
    using XT = typename std::conditional<kX3 != 0, float, __half>::type;
    const uint32_t n_items = (uint32_t)part_tab[32] * kUnitItems;

    uint32_t c[4][8];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 8; ++e) c[q][e] = 0u;
#ifdef D2C_UNIT_TRACE
    const int trole = lane != 0 ? -1 : (warp == kGatherWarp0Fwd ? 3 : (warp == kGatherWarp0Fwd + kGatherWarpsFwd - 1 ? 4 : -1));
#define D2C_TG(e) do { if (trole >= 0) D2C_TR(trole, k, e); } while (0)
#else
#define D2C_TG(e) ((void)0)
#endif
    // Corners that weigh nothing are not read, and blended with weight zero: their registers hold zero or a corner of an earlier
    // item, of which only a NaN would show.  Where x holds a NaN they are cleared, in a loop of its own (in one loop, or always, it
    // cost 1 to 9 % of the kernel).
    auto work = [&](auto clear) {
    for (uint32_t i = (uint32_t)(warp - kGatherWarp0Fwd); i < n_items; i += kGatherWarpsFwd) {
      const uint32_t k = i / kUnitItems;
      const int sr = k % kRStages, sa = k % kAStages;
      const int r = (int)(i % kUnitItems) * 8 + r8;
      D2C_TG(0);
      if (!ptx::mbar_wait(r_full(sr), (k / kRStages) & 1, abort_flag)) break;
      D2C_TG(1);
      const uint8_t* st = base_ptr + rec_off + sr * kRStage;
      const uint8_t* rec = st + r * 48 + ((kDual && !kShared && j >= 2) ? kRecBytes : 0);
      const uint4 hdr = *reinterpret_cast<const uint4*>(st + hdr_off);         // {staging offset, rows, image word}
      const uint2 head = *reinterpret_cast<const uint2*>(rec);
      const bool live = r < (int)hdr.z;
      const uint32_t bits = live ? head.y : 0u;      // rows past the clip end have stale records: nothing is read for them
      const int dx = (bits & 1u) ? p.cs.dx : 0, dy = (bits & 2u) ? p.cs.dy : 0, dz = (bits & 4u) ? p.cs.dz : 0;
      const XT* p0 = reinterpret_cast<const XT*>(p.x_cl) + (long long)(((uint64_t)hdr.y << 32) | hdr.x) + j * (kX3 ? 8 : 16) + head.x;
      auto load = [&](int z, int q) {
        if constexpr (clear) {
          if (!(bits & (8u << (4 * z + q)))) ptx::clear_v8(c[q]);
        }
        ptx::ldg_v8_if(c[q], p0 + (z ? dz : 0) + ((q & 2) ? dy : 0) + ((q & 1) ? dx : 0), bits & (8u << (4 * z + q)));
      };
#pragma unroll
      for (int q = 0; q < 4; ++q) load(0, q);
      D2C_TG(2);
      auto weights = [&](int z) {
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (live) w = *reinterpret_cast<const uint4*>(rec + (z ? 32 : 16));
        return w;
      };
      // corner order 000..111, as the reference's interpolation chain; rows past the clip end have weight zero (their records
      // are stale bytes)
      uint64_t acc2[4];                // fp32-parity: 8 channels
      __half2 acch[8];                 // single pass: 16 channels
#pragma unroll
      for (int e = 0; e < 4; ++e) acc2[e] = 0ull;
#pragma unroll
      for (int e = 0; e < 8; ++e) acch[e] = __float2half2_rn(0.f);
      auto blend = [&](uint32_t w, const uint32_t (&cc)[8]) {
        if constexpr (kX3) {
          uint64_t w2;
          asm("mov.b64 %0, {%1, %1};" : "=l"(w2) : "r"(w));
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint64_t c2;
            asm("mov.b64 %0, {%1, %2};" : "=l"(c2) : "r"(cc[2 * e]), "r"(cc[2 * e + 1]));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[e]) : "l"(c2), "l"(w2));
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) acch[e] = __hfma2(bits_h2(cc[e]), bits_h2(w), acch[e]);
        }
      };
      uint4 w = weights(0);
      blend(w.x, c[0]); load(1, 0);
      blend(w.y, c[1]); load(1, 1);
      blend(w.z, c[2]); load(1, 2);
      blend(w.w, c[3]); load(1, 3);
      D2C_TG(3);
      w = weights(1);
      float m = 1.f;
      if constexpr (kShared) m = live ? *reinterpret_cast<const float*>(st + kRecBytes + ((kDual && j >= 2) ? kMaskBytes : 0) + r * 4) : 0.f;
      blend(w.x, c[0]); blend(w.y, c[1]); blend(w.z, c[2]); blend(w.w, c[3]);
      D2C_TG(4);
      uint4 o0, o1;                  // chunk0, chunk1
      if constexpr (kX3) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float v0, v1;
          asm("mov.b64 {%0, %1}, %2;" : "=f"(v0), "=f"(v1) : "l"(acc2[e]));
          if constexpr (kShared) { v0 *= m; v1 *= m; }
          h[e] = ptx::pack_bf16x2(v0, v1);
          l[e] = ptx::pack_bf16x2(v0 - ptx::bf16_lo(h[e]), v1 - ptx::bf16_hi(h[e]));
        }
        o0 = make_uint4(h[0], h[1], h[2], h[3]);
        o1 = make_uint4(l[0], l[1], l[2], l[3]);
      } else {
        uint32_t o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float2 f = __half22float2(acch[e]);
          if constexpr (kShared) { f.x *= m; f.y *= m; }
          o[e] = ptx::pack_bf16x2(f.x, f.y);
        }
        o0 = make_uint4(o[0], o[1], o[2], o[3]);
        o1 = make_uint4(o[4], o[5], o[6], o[7]);
      }
      if (!ptx::mbar_wait(a_empty(sa), ((k / kAStages) & 1) ^ 1, abort_flag)) break;
      D2C_TG(5);
      const uint32_t row_off = (uint32_t)(r * 128);
      const uint32_t row = a_base + sa * kAStageBytes + row_off;
      ptx::sts_v4(row + chunk0, o0);
      ptx::sts_v4(row + chunk1, o1);
      D2C_TG(6);
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(a_full(sa));
        ptx::mbar_arrive(r_empty(sr));
      }
      if constexpr (kSave) {
        // where the thread's bytes go in the kept image: block = (tile, 64-voxel block, slice) in the single-pass mode;
        // (tile, 64-voxel block, slice pair, {hi, lo}, slice of the pair) in the hi/lo mode, where a 64-channel row holds this
        // unit's 32 channels in its half `word & 1`, and the lo block lies two blocks further
        const int word = (int)hdr.w;
        const uint32_t in_blk = row_off & 8191u;
        if constexpr (kX3) {
          uint8_t* sd = p.sav + ((long long)((word >> 1) + (r >> 6) * p.sav_np * 4) << 13) + in_blk +
                        (uint32_t)(((4 * (word & 1) + j) ^ r8) << 4);
          ptx::stg_v4_hint(sd, o0, pol_stream);
          ptx::stg_v4_hint(sd + (2 << 13), o1, pol_stream);
        } else {
          uint8_t* sd = p.sav + ((long long)(word + (r >> 6) * 2 * p.sav_np) << 13) + in_blk;
          ptx::stg_v4_hint(sd + chunk0, o0, pol_stream);
          ptx::stg_v4_hint(sd + chunk1, o1, pol_stream);
        }
      }
      D2C_TG(7);
    }
    };
    if (part_tab[33]) work(std::true_type{});
    else work(std::false_type{});
  }

  // ---- teardown ----
  ptx::tc_fence_before();
  __syncthreads();
#ifdef D2C_UNIT_TRACE
  if (p.trace && threadIdx.x == 0) {
    unsigned long long t1;
    unsigned smid;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
    asm volatile("mov.u32 %0, %smid;" : "=r"(smid));
    long long* rec = p.trace + 5 * 64 * 8 + blockIdx.x * 4;
    rec[0] = (long long)cta_t0; rec[1] = (long long)t1; rec[2] = (long long)smid; rec[3] = (long long)part_tab[32];
  }
#endif
  if (threadIdx.x == 0 && *abort_flag) ptx::report_device_timeout();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

