// Products of few rows (decode batches, short prompts): the weights are the M operand of the tensor-core instruction and
// the activations its N operand, so a tile is 128 weight rows by exactly as many tokens as there are (a multiple of 16),
// and what streams through shared memory is weights. Included by gemm.cu, whose parameters and epilogue helpers it uses.
//
// What bounds it is reading the weight once from HBM. The tile kernel stages 128 activation rows per k-block however few
// there are, covers a small matrix with fewer CTAs than SMs, and adds split-K pieces up in a second launch. Here two CTAs
// share an SM (about 100 KB of copies in flight each), a matrix with few tiles is cut along K over the CTAs of a cluster,
// and the pieces meet in distributed shared memory: CTA s of a cluster takes the s-th share of the tokens, adds the
// pieces in the order of k and applies the epilogue. No workspace, no second launch, the same sum on every run.
// CG = 2: the two CTAs of a pair hold 128 weight rows each and half of the tokens each (tcgen05.mma.cta_group::2); for
// more than 128 tokens, where staging all tokens in every CTA would cost more than the weights.
//
// One tile per CTA: with two CTAs on an SM the set-up and the epilogue of one run under the copies of the other.
//
// Measured, cold weights, tile kernel -> this one (us; the weight at the copy bandwidth): 14336 x 2 x 4096, 1 row 79 -> 42
// (37), 48 rows 74 -> 46; 28672 x 2 x 8192, 1 row 207 -> 142 (147); 128256 x 4096, 1 row 179 -> 156 (163); 4096 x 14336
// 28 -> 23.5 (18); 4096 x 4096 with its second pass 14.5 -> 10.7 (5).
#pragma once

constexpr int kFewThreads = 192;
constexpr int kFewHeader = 1024;
constexpr int kFewSmem = 113 * 1024;               // two CTAs on an SM
constexpr int kFewWBytes = 128 * BK * 2;           // weight rows of a k-block

struct FewPlan {
  int cg, nt, tok_tiles, split, kb_per, stages, tmem_cols, smem_bytes, n_tiles, round_tokens;
};

struct FewParams {
  DevParams d;
  int nt, tok_tiles, split, kb_per, round_tokens, early_weights;
};

template <bool GATED, int CG>
__global__ void __launch_bounds__(kFewThreads, 2)
gemm_few_rows_kernel(const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                     const __grid_constant__ CUtensorMap tmX, const __grid_constant__ FewParams fp) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_al = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_al);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* done_bar = full_bar + 2 * kMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_bar + 2 * kMaxStages + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* ring = smem_al + kFewHeader;

  const DevParams& p = fp.d;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // uniform: see gemm_tcgen05_kernel
  const int lane = threadIdx.x & 31;
  const int NT = fp.nt, S = fp.split, STAGES = p.stages;
  const uint32_t crank = (S > 1 || CG == 2) ? cluster_ctarank() : 0u;
  const int half = CG == 2 ? static_cast<int>(crank & 1u) : 0;      // which CTA of the pair
  const int ks = static_cast<int>(crank) / CG;                      // which part of K
  const bool leader = half == 0;
  const uint32_t lead_rank = crank & ~static_cast<uint32_t>(CG - 1);
  const int unit = blockIdx.x / (S * CG);
  const int tt = unit % fp.tok_tiles, tile = unit / fp.tok_tiles;   // token tiles of a weight tile run side by side
  const int tok0 = tt * NT;
  const int tile_tokens = min(NT, p.M - tok0);
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = ks * fp.kb_per, kb1 = min(num_kb, kb0 + fp.kb_per);
  const int nkb = kb1 - kb0;                                        // at least one (few_rows_plan)
  constexpr int OUTW = GATED ? 64 : 128;                            // output columns of a CTA
  const NBlock nb = n_block(p, tile * CG + half, OUTW);
  const int X_BYTES = NT / CG * BK * 2;
  const int STAGE = kFewWBytes + X_BYTES;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmW0);
    if (GATED) tma_prefetch_desc(&tmW1);
    tma_prefetch_desc(&tmX);
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
    // Tiles start at different k-blocks: in step, all CTAs would read the same 128-byte columns of rows that lie a power
    // of two apart, and the same lines of the activations (14336 x 2 x 4096, 1 row: 44.6 -> 41.5 us).
    const int rot = (tile * 13) % nkb;
    auto load = [&](int st, int i, bool weights, bool tokens) {      // by one lane
      uint8_t* sw = ring + st * STAGE;
      const int k0 = (kb0 + (i + rot < nkb ? i + rot : i + rot - nkb)) * BK;
      if (CG == 2) {
        const uint32_t fb = mapa_shared(smem_u32(&full_bar[st]), lead_rank);   // both CTAs' bytes count on the leader's barrier
        if (weights) {
          if (leader) mbar_expect_tx(&full_bar[st], 2 * STAGE);
          tma_load_2d_pair(sw, &tmW0, fb, k0, nb.col0);
          if (GATED) tma_load_2d_pair(sw + kFewWBytes / 2, &tmW1, fb, k0, nb.col0);
        }
        if (tokens) tma_load_2d_pair(sw + kFewWBytes, &tmX, fb, k0, tok0 + half * (NT / 2));
      } else {
        if (weights) {
          mbar_expect_tx(&full_bar[st], STAGE);
          tma_load_2d(sw, &tmW0, &full_bar[st], k0, nb.col0);
          if (GATED) tma_load_2d(sw + kFewWBytes / 2, &tmW1, &full_bar[st], k0, nb.col0);
        }
        if (tokens) tma_load_2d(sw + kFewWBytes, &tmX, &full_bar[st], nb.a_k0 + k0, tok0);
      }
    };
    // The ring is filled with weights while the kernel that computes the tokens may still run.
    const int early = fp.early_weights ? min(STAGES, nkb) : 0;
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
    const uint32_t idesc = umma_idesc_bf16(128 * CG, NT);
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
        const uint64_t w_desc = umma_desc_k_sw128(ring_addr + s * STAGE);
        const uint64_t x_desc = w_desc + (kFewWBytes >> 4);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint32_t on = (it != 0 || k != 0) ? 1u : 0u;
          if (CG == 2) umma_bf16_ss_pair(tmem_base, w_desc + (k * UMMA_K * 2 >> 4), x_desc + (k * UMMA_K * 2 >> 4), idesc, on);
          else umma_bf16_ss(tmem_base, w_desc + (k * UMMA_K * 2 >> 4), x_desc + (k * UMMA_K * 2 >> 4), idesc, on);
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

  // ---------------- accumulators -> token shares -> epilogue ----------------
  bool have = true;
  if (warp >= 2) {
    have = __all_sync(0xffffffffu, wait_or_abort(done_bar, 0, abort_flag));
    if (!have) {
      if (lane == 0) report_status(p.status, NF_ST_TIMEOUT_TMEM_FULL);
      *abort_flag = 1;
    }
  }
  __syncwarp();
  // With all MMAs of the cluster complete, the rings are free: [part of K][token of the share][128 weight rows] fp32, in
  // rounds of as many tokens as the ring holds.
  if (S > 1) cluster_sync_all();
  float* red = reinterpret_cast<float*>(ring);
  for (int t0 = 0; t0 < tile_tokens; t0 += fp.round_tokens) {
    const int now = min(fp.round_tokens, tile_tokens - t0);
    const int tok_per = (now + S - 1) / S;
    if (warp >= 2 && have) {
      tc_fence_after();
      const int q = warp & 3;                    // TMEM lane quarter this warp may read
      const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + t0;
      const uint32_t slot0 = smem_u32(red) + static_cast<uint32_t>((ks * tok_per * 128 + q * 32 + lane) * 4);
      int owner = 0, tl = 0;
      uint32_t dst = S > 1 ? mapa_shared(slot0, static_cast<uint32_t>(half)) : slot0;
#pragma unroll 1
      for (int c = 0; c < now; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16n(t_lane + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c + j < now) {
            if (S > 1) st_shared_cluster_u32(dst, r[j]);
            else asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst), "r"(r[j]) : "memory");
            dst += 512;
            if (++tl == tok_per) {
              tl = 0;
              ++owner;
              if (S > 1) dst = mapa_shared(slot0, static_cast<uint32_t>(min(owner, S - 1) * CG + half));
            }
          }
        }
      }
      tc_fence_before();
    }
    __syncwarp();
    if (S > 1) cluster_sync_all();
    else __syncthreads();
    const int mine = min(tok_per, now - ks * tok_per);
    constexpr int GR = OUTW / 8;
    for (int i = threadIdx.x; i < mine * GR; i += kFewThreads) {
      const int t = i / GR, g = i % GR;
      const int col = nb.col0 + g * 8, row = tok0 + t0 + ks * tok_per + t;
      if (col >= nb.col_end) continue;
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, u[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int s = 0; s < S; ++s) {
        const float* src = red + (s * tok_per + t) * 128 + g * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += src[j];
        if (GATED) {
#pragma unroll
          for (int j = 0; j < 8; ++j) u[j] += src[64 + j];
        }
      }
      if (p.bias != nullptr) add_bias8(v, p.bias + col);
      if (GATED) {
        if (p.bias != nullptr) add_bias8(u, p.bias2 + col);
        gated_acts<8>(v, u, p.act);
      } else if (p.C != nullptr) {
        const uint4 cv = *reinterpret_cast<const uint4*>(p.C + static_cast<long long>(row) * p.ldc + col);
        const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(cw[j]);
          v[2 * j] += p.beta * f.x;
          v[2 * j + 1] += p.beta * f.y;
        }
      }
      store_cols8(p, row, col, v);
    }
    if (t0 + fp.round_tokens < tile_tokens) {    // the next round writes where this one is read
      __syncwarp();
      if (S > 1) cluster_sync_all();
      else __syncthreads();
    }
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

// Tile and split for M rows. `split` / `cg` 0 = choose.
inline FewPlan few_rows_plan(int M, int N, int K, bool gated, int groups, int cg, int split) {
  FewPlan f;
  f.cg = cg != 0 ? cg : M > 128 ? 2 : 1;
  const int gran = 16 * f.cg;
  f.tok_tiles = (M + 255) / 256;
  f.nt = ((M + f.tok_tiles - 1) / f.tok_tiles + gran - 1) / gran * gran;
  const int blocks = n_block_count(groups, N / groups, gated ? 64 : 128);
  f.n_tiles = (blocks + f.cg - 1) / f.cg;
  const int num_kb = (K + BK - 1) / BK;
  const int ctas = f.n_tiles * f.tok_tiles * f.cg;
  f.split = 1;
  if (split != 0) f.split = split;
  else
    while ((f.split + 1) * f.cg <= 8 && 4 * ctas * (f.split + 1) <= 7 * device_sm_count() && num_kb / (f.split + 1) >= 4) ++f.split;
  f.kb_per = (num_kb + f.split - 1) / f.split;
  f.split = (num_kb + f.kb_per - 1) / f.kb_per;       // no empty part
  const int stage = kFewWBytes + f.nt / f.cg * BK * 2;
  f.stages = (kFewSmem - 2048) / stage;
  if (f.stages > kMaxStages) f.stages = kMaxStages;
  f.tmem_cols = f.nt <= 32 ? 32 : f.nt <= 64 ? 64 : f.nt <= 128 ? 128 : 256;
  f.smem_bytes = f.stages * stage + 2048;
  // a round of the reduction: split * ceil(tokens / split) rows of 512 bytes in the ring; rounds start on an accumulator
  // chunk of 16 tokens
  f.round_tokens = (f.stages * stage / 512 - f.split + 1) / 16 * 16;
  return f;
}
