// Split-K of the tile kernel's shapes with one tile per cluster: the CTAs (CG = 1) or CTA pairs (CG = 2) of a cluster take a
// part of K each and add their pieces in distributed shared memory. Included by gemm.cu, whose parameters and epilogue helpers
// it uses.
//
// What it replaces is the way of the pieces through L2: with split-K a product of 129 to 700 rows spends 4 us writing fp32
// copies and then a second launch that reads them. Here CTA `ks` of a cluster owns the ks-th slice of the tile's columns: the
// others send it theirs, 16 bytes per lane and 512 consecutive ones per warp, it adds them in the order of k with its own,
// which never leaves tensor memory, and applies the epilogue. The same sums in the same order as the two launches, bit for bit.
//
// us, two launches -> one, cold weights in a chain: 256 x 8192 x 8192 in two parts 42.8 -> 35.6, 256 x 8192 x 28672 106.8 -> 102.2,
// 333 x 4096 x 14336 50.2 -> 47.1, 256 x 4096 x 4096 (128 columns) 18.5 -> 16.1, 96 x 4096 x 4096 in four 14.6 -> 13.0. Clusters of
// four pairs stay two launches for 16 tiles and more: only 14 of them fit at once.
#pragma once

constexpr int kSplitMaxCluster = 8;                // the portable cluster size

struct SplitParams {
  DevParams d;
  int m_groups, kb_per, slice, early_weights;      // slice: columns of the tile that a CTA owns
};

struct SplitPlan {
  int cg, bn, split, kb_per, slice, stages, tmem_cols, smem_bytes, m_groups, tiles;
};

template <int CG>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_split_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ SplitParams sp) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_al = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_al);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* done_bar = full_bar + 2 * kMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_bar + 2 * kMaxStages + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* ring = smem_al + 1024;

  const DevParams& p = sp.d;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // uniform: see gemm_tcgen05_kernel
  const int lane = threadIdx.x & 31;
  const int BN = p.bn, S = p.split_k, STAGES = p.stages;
  const uint32_t crank = cluster_ctarank();
  const int half = CG == 2 ? static_cast<int>(crank & 1u) : 0;      // which CTA of the pair
  const int ks = static_cast<int>(crank) / CG;                      // which part of K
  const bool leader = half == 0;
  const uint32_t lead_rank = crank & ~static_cast<uint32_t>(CG - 1);
  const int tile = blockIdx.x / (S * CG);
  const int m_grp = tile % sp.m_groups, n_blk = tile / sp.m_groups;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = ks * sp.kb_per, kb1 = min(num_kb, kb0 + sp.kb_per);
  const int nkb = kb1 - kb0;                                        // at least one (split_plan)
  const NBlock nb = n_block(p, n_blk, BN);
  const int row0 = (m_grp * CG + half) * BM;
  const int B_BYTES = (BN / CG) * BK * 2;
  const int STAGE = A_TILE_BYTES + B_BYTES;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    if (CG == 2) {
      tmem_alloc_pair(tmem_slot, static_cast<uint32_t>(p.tmem_cols));
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, static_cast<uint32_t>(p.tmem_cols));
      tmem_relinquish();
    }
  }
  tc_fence_before();
  if (CG == 2) cluster_sync_all();   // the peer's barriers exist before anything signals them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  if (warp != 0) await_previous();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    uint32_t ph = 0;
    int s = 0, it = 0;
    bool ok = true;
    auto load = [&](int st, int i, bool weights, bool rows) {        // by one lane
      uint8_t* sa = ring + st * STAGE;
      const int k0 = (kb0 + i) * BK;
      if (CG == 2) {
        const uint32_t fb = mapa_shared(smem_u32(&full_bar[st]), lead_rank);   // both CTAs' bytes count on the leader's barrier
        if (weights) {
          if (leader) mbar_expect_tx(&full_bar[st], 2 * STAGE);
          tma_load_2d_pair(sa + A_TILE_BYTES, &tmB, fb, k0, nb.col0 + half * (BN / 2));
        }
        if (rows) tma_load_2d_pair(sa, &tmA, fb, nb.a_k0 + k0, row0);
      } else {
        if (weights) {
          mbar_expect_tx(&full_bar[st], STAGE);
          tma_load_2d(sa + A_TILE_BYTES, &tmB, &full_bar[st], k0, nb.col0);
        }
        if (rows) tma_load_2d(sa, &tmA, &full_bar[st], nb.a_k0 + k0, row0);
      }
    };
    // The ring is filled with weights while the kernel that computes the rows may still run.
    const int early = sp.early_weights ? min(STAGES, nkb) : 0;
    if (elect_one())
      for (int i = 0; i < early; ++i) load(i, i, true, false);
    __syncwarp();
    await_previous();
    for (; it < nkb; ++it, s = (s + 1 == STAGES) ? 0 : s + 1, ph ^= (s == 0)) {
      if (!__all_sync(0xffffffffu, wait_or_abort(&empty_bar[s], ph ^ 1, abort_flag))) {
        report_status(p.status, NF_ST_TIMEOUT_SMEM_EMPTY);
        *abort_flag = 1;
        ok = false;
        break;
      }
      if (elect_one()) load(s, it, it >= early, true);
      __syncwarp();
    }
    if (ok && CG == 2) {
      // every arrival that the leader's commits send to this CTA's slots has landed once each slot reads as free
      for (int j = 0; j < STAGES; ++j, s = (s + 1 == STAGES) ? 0 : s + 1, ph ^= (s == 0))
        if (!wait_or_abort(&empty_bar[s], ph ^ 1, abort_flag)) break;
    }
    if (!ok && leader) {
      // loads in flight get a bounded chance to land before the shared memory is given back
      const int back = it < STAGES ? it : STAGES;
      for (int j = it - back; j < it; ++j) (void)mbar_wait(&full_bar[j % STAGES], (j / STAGES) & 1);
    }
  } else if (warp == 1 && leader) {
    // ---------------- MMA issuer ----------------
    const uint32_t idesc = umma_idesc_bf16(BM * CG, BN);
    const uint32_t ring_addr = smem_u32(ring);
    uint32_t ph = 0;
    int s = 0;
    bool ok = true;
    for (int it = 0; it < nkb; ++it, s = (s + 1 == STAGES) ? 0 : s + 1, ph ^= (s == 0)) {
      if (!__all_sync(0xffffffffu, wait_or_abort(&full_bar[s], ph, abort_flag))) {
        report_status(p.status, NF_ST_TIMEOUT_SMEM_FULL);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      if (elect_one()) {
        const uint64_t a_desc = umma_desc_k_sw128(ring_addr + s * STAGE);
        const uint64_t b_desc = a_desc + (A_TILE_BYTES >> 4);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint32_t on = (it != 0 || k != 0) ? 1u : 0u;
          if (CG == 2) umma_bf16_ss_pair(tmem_base, a_desc + (k * UMMA_K * 2 >> 4), b_desc + (k * UMMA_K * 2 >> 4), idesc, on);
          else umma_bf16_ss(tmem_base, a_desc + (k * UMMA_K * 2 >> 4), b_desc + (k * UMMA_K * 2 >> 4), idesc, on);
        }
        if (CG == 2) umma_commit_pair_mask(&empty_bar[s], static_cast<uint16_t>(3u << lead_rank));
        else umma_commit(&empty_bar[s]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) {
      if (CG == 2) umma_commit_pair_mask(done_bar, static_cast<uint16_t>(3u << lead_rank));
      else umma_commit(done_bar);
    }
    __syncwarp();
  }

  // ---------------- pieces -> their owners -> epilogue (4 warps, a row of the tile per thread) ----------------
  bool have = true;
  if (warp >= 2) {
    have = __all_sync(0xffffffffu, wait_or_abort(done_bar, 0, abort_flag));
    if (!have) {
      if (lane == 0) report_status(p.status, NF_ST_TIMEOUT_TMEM_FULL);
      *abort_flag = 1;
    }
  }
  __syncwarp();
  cluster_sync_all();                  // all MMAs of the cluster are complete: the rings are free
  const int q = warp & 3;              // TMEM lane quarter this warp may read
  const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
  const uint32_t own = smem_u32(ring) + static_cast<uint32_t>(q * 32 + lane) * 16u;   // [part][4 columns][row] of 16 bytes
  const int piece_bytes = sp.slice * 512;
  const int row = row0 + q * 32 + lane;
  const int c0 = ks * sp.slice, c1 = min(BN, c0 + sp.slice);        // the columns that this CTA owns
  const bool row_ok = warp >= 2 && have && row < p.M;
  const __nv_bfloat16* crow = row_ok && p.C != nullptr ? p.C + static_cast<long long>(row) * p.ldc + nb.col0 : nullptr;
  uint4 c_next[2] = {};
  auto request_c = [&](int c) {        // what the residual adds to 16 columns, a chunk ahead
#pragma unroll
    for (int g8 = 0; g8 < 2; ++g8)
      if (nb.col0 + c + g8 * 8 < nb.col_end) c_next[g8] = *reinterpret_cast<const uint4*>(crow + c + g8 * 8);
  };
  if (warp >= 2 && have) {
    tc_fence_after();
    for (int i = 1; i < S; ++i) {
      const int o = ks + i < S ? ks + i : ks + i - S;
      const uint32_t dst = mapa_shared(own, static_cast<uint32_t>(o * CG + half)) + static_cast<uint32_t>(ks * piece_bytes);
      const int o0 = o * sp.slice, o1 = min(BN, o0 + sp.slice);
#pragma unroll 1
      for (int c = o0; c < o1; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16n(t_lane + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j)
          st_shared_cluster_v4(dst + static_cast<uint32_t>((c - o0) / 4 + j) * 2048u, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    }
    if (crow != nullptr && c0 < c1) request_c(c0);
  }
  __syncwarp();
  cluster_sync_all();                  // every piece has arrived
  if (warp >= 2 && have) {
#pragma unroll 1
    for (int c = c0; c < c1; c += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16n(t_lane + c, r);
      const uint4 c_now[2] = {c_next[0], c_next[1]};
      if (crow != nullptr && c + 16 < c1) request_c(c + 16);
      tmem_ld_wait();
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0.f;
      for (int s = 0; s < S; ++s) {
        if (s == ks) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
        } else {
          const uint32_t src = own + static_cast<uint32_t>(s * piece_bytes) + static_cast<uint32_t>((c - c0) / 4) * 2048u;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float x, y, z, w;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x), "=f"(y), "=f"(z), "=f"(w) : "r"(src + j * 2048u) : "memory");
            v[4 * j] += x;
            v[4 * j + 1] += y;
            v[4 * j + 2] += z;
            v[4 * j + 3] += w;
          }
        }
      }
      const int col = nb.col0 + c;
      if (!row_ok || col >= nb.col_end) continue;
#pragma unroll
      for (int g8 = 0; g8 < 2; ++g8) {
        if (col + g8 * 8 >= nb.col_end) continue;
        float* vv = v + g8 * 8;
        if (p.bias != nullptr) add_bias8(vv, p.bias + col + g8 * 8);
        if (crow != nullptr) {
          const uint32_t cw[4] = {c_now[g8].x, c_now[g8].y, c_now[g8].z, c_now[g8].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(cw[j]);
            vv[2 * j] += p.beta * f.x;
            vv[2 * j + 1] += p.beta * f.y;
          }
        }
      }
      store_cols16(p, row, col, nb.col_end, v);
    }
    tc_fence_before();
  }
  __syncwarp();
  if (CG == 2) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (CG == 2) tmem_dealloc_pair(tmem_base, static_cast<uint32_t>(p.tmem_cols));
    else tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
}

// The launch that sums a tile of `bn` columns in `split` parts within a cluster; stages 0 = not built for this shape.
inline SplitPlan split_plan(int M, int N, int K, int groups, int bn, int cg, int split) {
  SplitPlan s{};
  const int num_kb = (K + BK - 1) / BK;
  s.cg = cg;
  s.bn = bn;
  s.split = split;
  if (split < 2 || split * cg > kSplitMaxCluster || bn > 256 || bn % 32 != 0) return s;
  s.kb_per = (num_kb + split - 1) / split;
  if ((split - 1) * s.kb_per >= num_kb) return s;     // an empty part
  s.slice = ((bn + split - 1) / split + 15) / 16 * 16;
  const int stage = A_TILE_BYTES + (bn / cg) * BK * 2;
  s.stages = (kSmemMax - 2048) / stage;
  if (s.stages > kMaxStages) s.stages = kMaxStages;
  if (split * s.slice * 512 > s.stages * stage) {     // the pieces meet where the ring was
    s.stages = 0;
    return s;
  }
  s.tmem_cols = bn <= 32 ? 32 : bn <= 64 ? 64 : bn <= 128 ? 128 : 256;
  s.smem_bytes = s.stages * stage + 2048;
  s.m_groups = ((M + BM - 1) / BM + cg - 1) / cg;
  s.tiles = s.m_groups * n_block_count(groups, N / groups, bn);
  return s;
}
