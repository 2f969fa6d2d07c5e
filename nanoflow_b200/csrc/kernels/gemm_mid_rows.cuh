// Products of more rows than the few-rows kernel takes and fewer than fill the tile kernel's 256-row tiles: again the weights
// are the M operand of the tensor-core instruction and the activations its N operand. Included by gemm.cu, whose parameters and
// epilogue helpers it uses.
//
// What bounds such a product is what enters an SM: 64 bytes a clock from L2, whatever the tile. A CTA pair that holds 256 weight
// rows and all tokens brings each weight byte into shared memory once and half of the tokens' bytes per CTA: at 352 tokens 38 KB
// for 0.38 us of products, where tiles of 128 rows by 256 columns fetch 48 KB for 0.28 us, and pair tiles of 256 rows work on 512
// rows for 333. Tokens are a multiple of 32, in one or two instructions (up to 256 tokens each) per k step. K is cut over the
// pairs of a cluster where a matrix has few tiles; the pieces meet in distributed shared memory and are added in the order of k,
// so the sums have the order of a tile kernel's split into as many parts, bit for bit.
//
// One tile per pair, one CTA on an SM, the whole shared memory for the ring. The finished tile is 128 output columns (64 gated
// ones) of each token per CTA; it leaves through the ring, [4 tokens][weight row] of 16 bytes, so that stores of all lanes of a
// warp are consecutive and loads of eight weight rows meet no bank twice (row w lies at w ^ (w / 8 % 8)).
//
// Tried and dropped: sending for the weights into L2 some blocks ahead of the ring (8192 x 28672 at 160 rows 87 -> 90 us with four
// blocks, 113 with 16): the ring holds enough. The second instruction behind a branch at run time cost a third of the loop's speed
// at one instruction (8192 x 28672 at 256 rows 113 -> 99 as a form of its own).
#pragma once

constexpr int kMidTokens = 512;                    // most tokens of a tile: the columns of tensor memory

struct MidPlan {
  int nb, nb2, tok_tiles, split, kb_per, stages, tmem_cols, smem_bytes, n_tiles, round_tokens;
};

struct MidParams {
  DevParams d;
  int nb, nb2, tok_tiles, split, kb_per, round_tokens, early_weights;     // nb, nb2: tokens of the two instructions (nb2: or 0)
};

template <bool GATED, bool TWO>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_mid_rows_kernel(const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                     const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmX2,
                     const __grid_constant__ MidParams mp) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_al = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_al);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* done_bar = full_bar + 2 * kMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_bar + 2 * kMaxStages + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* ring = smem_al + 1024;

  const DevParams& p = mp.d;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // uniform: see gemm_tcgen05_kernel
  const int lane = threadIdx.x & 31;
  const int NB = mp.nb, NB2 = TWO ? mp.nb2 : 0, S = mp.split, STAGES = p.stages;
  const uint32_t crank = cluster_ctarank();
  const int half = static_cast<int>(crank & 1u);                    // which CTA of the pair
  const int ks = static_cast<int>(crank >> 1);                      // which part of K
  const bool leader = half == 0;
  const uint32_t lead_rank = crank & ~1u;
  const int unit = blockIdx.x / (S * 2);
  const int tt = unit % mp.tok_tiles, tile = unit / mp.tok_tiles;   // token tiles of a weight tile run side by side
  const int tok0 = tt * (NB + NB2);
  const int tile_tokens = min(NB + NB2, p.M - tok0);                // at least one (mid_rows_plan)
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = ks * mp.kb_per, kb1 = min(num_kb, kb0 + mp.kb_per);
  const int nkb = kb1 - kb0;                                        // at least one
  constexpr int OUTW = GATED ? 64 : 128;                            // output columns of a CTA
  const NBlock nb = n_block(p, tile * 2 + half, OUTW);
  const int X_BYTES = NB / 2 * BK * 2;                              // tokens of the first instruction that this CTA stages
  const int STAGE = kFewWBytes + X_BYTES + NB2 / 2 * BK * 2;

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
    if (TWO) tma_prefetch_desc(&tmX2);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();                // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  if (warp != 0) await_previous();

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    uint32_t ph = 0;
    int s = 0, it = 0;
    bool ok = true;
    auto load = [&](int st, int i, bool weights, bool tokens) {      // by one lane
      uint8_t* sw = ring + st * STAGE;
      const int k0 = (kb0 + i) * BK;
      const uint32_t fb = mapa_shared(smem_u32(&full_bar[st]), lead_rank);     // both CTAs' bytes count on the leader's barrier
      if (weights) {
        if (leader) mbar_expect_tx(&full_bar[st], 2 * STAGE);
        tma_load_2d_pair(sw, &tmW0, fb, k0, nb.col0);
        if (GATED) tma_load_2d_pair(sw + kFewWBytes / 2, &tmW1, fb, k0, nb.col0);
      }
      if (tokens) {
        tma_load_2d_pair(sw + kFewWBytes, &tmX, fb, k0, tok0 + half * (NB / 2));
        if (TWO) tma_load_2d_pair(sw + kFewWBytes + X_BYTES, &tmX2, fb, k0, tok0 + NB + half * (NB2 / 2));
      }
    };
    // The ring is filled with weights while the kernel that computes the tokens may still run.
    const int early = mp.early_weights ? min(STAGES, nkb) : 0;
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
    if (ok) {
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
    const uint32_t idesc = umma_idesc_bf16(256, NB), idesc2 = umma_idesc_bf16(256, NB2);
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
        const uint64_t x2_desc = x_desc + static_cast<uint64_t>(X_BYTES >> 4);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint32_t on = (it != 0 || k != 0) ? 1u : 0u;
          umma_bf16_ss_pair(tmem_base, w_desc + (k * UMMA_K * 2 >> 4), x_desc + (k * UMMA_K * 2 >> 4), idesc, on);
          if (TWO)
            umma_bf16_ss_pair(tmem_base + NB, w_desc + (k * UMMA_K * 2 >> 4), x2_desc + (k * UMMA_K * 2 >> 4), idesc2, on);
        }
        umma_commit_pair_mask(&empty_bar[s], static_cast<uint16_t>(3u << lead_rank));
      }
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit_pair_mask(done_bar, static_cast<uint16_t>(3u << lead_rank));
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
  // With all MMAs of the cluster complete, the rings are free: [part of K][4 tokens of the share][weight row] of 16 bytes, in
  // rounds of as many tokens as the ring holds.
  cluster_sync_all();
  const uint32_t ring_addr = smem_u32(ring);
  for (int t0 = 0; t0 < tile_tokens; t0 += mp.round_tokens) {
    const int now = min(mp.round_tokens, tile_tokens - t0);
    const int share = (now + 4 * S - 1) / (4 * S);                  // groups of four tokens that a part of the cluster finishes
    const int first = ks * share * 4;                               // of this CTA's tokens in the round
    constexpr int GR = OUTW / 8;
    const int items = max(0, min(share, (now - first + 3) / 4)) * GR;     // eight columns of four tokens each
    // what the residual adds to an item is requested an item ahead, the first one's while the pieces are on their way
    uint4 c_next[4] = {};
    auto request_c = [&](int i) {
      if constexpr (!GATED) {
        const int col = nb.col0 + (i % GR) * 8, row = tok0 + t0 + first + i / GR * 4;
        if (p.C == nullptr || i >= items || col >= nb.col_end) return;
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (row + t < p.M) c_next[t] = *reinterpret_cast<const uint4*>(p.C + static_cast<long long>(row + t) * p.ldc + col);
      }
    };
    request_c(threadIdx.x);
    if (warp >= 2 && have) {
      tc_fence_after();
      const int q = warp & 3;                                       // TMEM lane quarter this warp may read
      const int w = q * 32 + lane;
      const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + t0;
      const uint32_t slot0 = ring_addr + static_cast<uint32_t>((ks * share * 128 + (w ^ ((w >> 3) & 7))) * 16);
      int owner = 0, left = share;
      uint32_t dst = mapa_shared(slot0, static_cast<uint32_t>(half));
#pragma unroll 1
      for (int c = 0; c < now; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_lane + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (c + 4 * j < now) {
            st_shared_cluster_v4(dst, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            dst += 2048;
            if (--left == 0) {
              left = share;
              ++owner;
              dst = mapa_shared(slot0, static_cast<uint32_t>(min(owner, S - 1) * 2 + half));
            }
          }
        }
      }
      tc_fence_before();
    }
    __syncwarp();
    cluster_sync_all();
    for (int i = threadIdx.x; i < items; i += kGemmThreads) {
      const int t4 = i / GR, g = i % GR;
      const int col = nb.col0 + g * 8, row = tok0 + t0 + first + t4 * 4;
      const uint4 c_in[4] = {c_next[0], c_next[1], c_next[2], c_next[3]};
      request_c(i + kGemmThreads);
      if (col >= nb.col_end) continue;
      const int rows = min(4, p.M - row);                           // (a round ends where its tile's tokens end)
      float v[4][8], u[4][8];
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int j = 0; j < 8; ++j) v[t][j] = u[t][j] = 0.f;
      for (int s = 0; s < S; ++s) {
        const uint32_t src = ring_addr + static_cast<uint32_t>((s * share + t4) * 2048);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float x0, x1, x2, x3;
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(x0), "=f"(x1), "=f"(x2), "=f"(x3) : "r"(src + (g * 8 + (j ^ (g & 7))) * 16) : "memory");
          v[0][j] += x0; v[1][j] += x1; v[2][j] += x2; v[3][j] += x3;
          if (GATED) {                                              // the up half: 64 weight rows on
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(x0), "=f"(x1), "=f"(x2), "=f"(x3) : "r"(src + 1024 + (g * 8 + (j ^ (g & 7))) * 16) : "memory");
            u[0][j] += x0; u[1][j] += x1; u[2][j] += x2; u[3][j] += x3;
          }
        }
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t >= rows) continue;
        if (p.bias != nullptr) add_bias8(v[t], p.bias + col);
        if (GATED) {
          if (p.bias != nullptr) add_bias8(u[t], p.bias2 + col);
          gated_acts<8>(v[t], u[t], p.act);
        } else if (p.C != nullptr) {
          const uint32_t cw[4] = {c_in[t].x, c_in[t].y, c_in[t].z, c_in[t].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(cw[j]);
            v[t][2 * j] += p.beta * f.x;
            v[t][2 * j + 1] += p.beta * f.y;
          }
        }
        store_cols8(p, row + t, col, v[t]);
      }
    }
    if (t0 + mp.round_tokens < tile_tokens) {    // the next round writes where this one is read
      __syncwarp();
      cluster_sync_all();
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
}

// Tiles of M rows with K in `split` parts; stages 0 = not built for this.
inline MidPlan mid_rows_plan(int M, int N, int K, bool gated, int split) {
  MidPlan f{};
  const int num_kb = (K + BK - 1) / BK;
  f.split = split;
  if (split < 1 || split * 2 > kSplitMaxCluster) return f;
  f.kb_per = (num_kb + split - 1) / split;
  if ((split - 1) * f.kb_per >= num_kb) return f;     // an empty part
  f.tok_tiles = (M + kMidTokens - 1) / kMidTokens;
  const int cols = ((M + f.tok_tiles - 1) / f.tok_tiles + 31) / 32 * 32;      // a pair's instruction takes a multiple of 32
  f.nb = cols <= 256 ? cols : (cols / 2 + 31) / 32 * 32;
  f.nb2 = cols - f.nb;
  f.tok_tiles = (M + cols - 1) / cols;
  f.n_tiles = (n_block_count(1, N, gated ? 64 : 128) + 1) / 2;
  const int stage = kFewWBytes + cols / 2 * BK * 2;
  f.stages = (kSmemMax - 2048) / stage;
  if (f.stages > kMaxStages) f.stages = kMaxStages;
  f.tmem_cols = cols <= 32 ? 32 : cols <= 64 ? 64 : cols <= 128 ? 128 : cols <= 256 ? 256 : 512;
  f.smem_bytes = f.stages * stage + 2048;
  // a round of the reduction: split * ceil(tokens / 4 / split) groups of four tokens, 2 KB each, in the ring; rounds start on
  // an accumulator chunk of 32 tokens
  f.round_tokens = (f.stages * stage / 2048 - split + 1) * 4 / 32 * 32;
  return f;
}
