// bf16 GEMM on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM), operands staged
// by TMA into 128B-swizzled shared memory, persistent over output tiles with an explicit CTA budget.
//
//   D[M,N] = A[M,K] * B[N,K]^T (+ bias[N]) (+ beta * C[M,N])            (linear epilogue)
//   D[M,F] = act(A * Bg[F,K]^T, A * Bu[F,K]^T)                           (gated epilogue, see gated_act.cuh)
//
// Columns from f32_col0 on can leave as fp32 into a second output (logits, gate pre-activations), and the
// product can be block diagonal: with `groups` > 1 output columns of group g see only A's columns
// [g * group_k, g * group_k + K), which is how per-head matrices are applied to all heads in one launch.
//
// Work units are whole output tiles, or with split-K (tile, k range) pairs whose fp32 partial tiles
// a second pass adds up; with the stream-K tail only the tiles left over after the full waves are
// cut, into equal k ranges. For small M one CTA can cover several M tiles with the same weight tile,
// so each weight byte is fetched into shared memory once; for larger M the two CTAs of a cluster
// share a 256-row tile (tcgen05.mma.cta_group::2) and each stages half of the weight tile. A cost
// model picks the shape; engines time the candidates on their own shapes (ops/autotune.py).
//
// Roles inside one 192-thread CTA: warp 0 = TMA producer, warp 1 = TMEM owner and MMA issuer (an elected
// lane of each issues), warps 2..5 = epilogue (TMEM -> registers -> global). Two TMEM accumulators are
// ping-ponged so the epilogue of tile i overlaps the main loop of tile i+1.
//
// Takes the place of the reference's CUTLASS Sm80 device::Gemm wrapper
// (pipeline/include/cutlassGemmWrapperImpl.cuh:68-125: D = alpha*A*B + beta*C, residual or
// replicated bias as C) and of its DualGemm + SiLU-mul epilogue (pipeline/include/dualWrapper.cuh:47-144).
#include "common.cuh"
#include "gated_act.cuh"
#include "kernels.h"

#include <algorithm>
#include <mutex>

namespace nf {

nf_encode_tiled_fn get_encode_tiled() {
  static nf_encode_tiled_fn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<nf_encode_tiled_fn>(p);
    }
  });
  return fn;
}

int device_slot() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return (dev >= 0 && dev < kMaxDevices) ? dev : 0;
}

int device_sm_count() {
  static int cached[kMaxDevices] = {0};
  const int slot = device_slot();
  int n = cached[slot];
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, slot) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      return 148;
    }
    cached[slot] = n;   // the same value from whichever thread gets here first
  }
  return n;
}

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols,
                      uint64_t ld, uint32_t box_rows, uint32_t box_cols) {
  nf_encode_tiled_fn enc = get_encode_tiled();
  if (enc == nullptr) return NF_ERR_CUDA;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld * 2) % 16 != 0) return NF_ERR_BAD_ARG;
  cuuint64_t gdim[2] = {cols, rows};
  cuuint64_t gstride[1] = {ld * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstride,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? NF_OK : NF_ERR_CUDA;
}

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int kGemmThreads = 192;
constexpr int kSmemBudget = 227 * 1024 - 2048;

// Tile geometry. The tile is 128*MT rows by `bn` weight rows (bn: multiple of 32 up to 256, a runtime
// value so that the tile count can be matched to the SM count); MT = number of 128-row M tiles one
// CTA covers with the same B tile (MT > 1 is the small-M, weight-streaming shape: every weight byte
// enters shared memory once). Shared memory: 1 KB of barriers, then `stages` ring slots of
// (MT*16 KB of A + bn*128 B of B). TMEM: MT*bn fp32 columns per accumulator set, two sets
// (epilogue of one tile under the main loop of the next) when they fit in 512 columns.
constexpr int kMaxStages = 8;
constexpr int A_TILE_BYTES = BM * BK * 2;
struct Geom {
  int bn, out_bn, stages, acc_bufs, tmem_cols, stage_bytes, b_bytes, smem_bytes;
};
// Reduce-scatter epilogue, staged form: each epilogue warp keeps a [32 rows][128 columns] bf16 piece of
// its rows in shared memory (row pitch 272 B, so that the 32 lanes' 16-byte stores spread over all
// banks) and sends each row's 256 bytes to its owner with one bulk copy.
constexpr int kRsRunCols = 128;
constexpr int kRsRowPitch = kRsRunCols * 2 + 16;
constexpr int kRsStageBytes = 4 * 32 * kRsRowPitch;     // four epilogue warps

inline Geom make_geom(int bn, int mt, bool swiglu, int smem_budget, int cg, int extra = 0) {
  Geom g;
  g.bn = bn;
  g.out_bn = swiglu ? bn / 2 : bn;
  g.b_bytes = (bn / cg) * BK * 2;      // a CTA pair splits the weight tile between its two CTAs
  g.stage_bytes = mt * A_TILE_BYTES + g.b_bytes;
  int st = (smem_budget - 2048 - extra) / g.stage_bytes;
  g.stages = st > kMaxStages ? kMaxStages : st;
  const int acc_cols = mt * bn;
  g.acc_bufs = acc_cols * 2 <= 512 ? 2 : 1;
  const int need = acc_cols * g.acc_bufs;
  g.tmem_cols = need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512;
  g.smem_bytes = g.stages * g.stage_bytes + 2048 + extra;   // the extra region follows the ring slots
  return g;
}

struct DevParams {
  __nv_bfloat16* D;
  const __nv_bfloat16* C;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* bias2;       // of the up half (gated epilogue)
  float* partial;   // split-K: fp32 [split_k][M][N] partial sums (second pass reduces them)
  long long ldd, ldc;
  float beta;
  int M, N, K;      // N = number of output columns
  int split_k;
  unsigned int* status;
  int bn, stages, acc_bufs, tmem_cols;   // tile geometry (see make_geom)
  // stream-K tail (see Walk): tiles from sk_tiles_dp on are cut into k-block ranges of sk_q
  float* sk_partial;          // fp32 [tile][piece][CTA of pair][rows per CTA][bn]
  int sk_tiles_dp, sk_q, sk_max_pieces;
  // RMSNorm of the result rows, fused into the split-K reduce pass
  const __nv_bfloat16* norm_w;
  __nv_bfloat16* norm_out;
  long long norm_ld;
  float norm_eps;
  // reduce-scatter epilogue (EPI == 2)
  char* rs_heap[8];
  int rs_rank, rs_nranks, rs_rows_cap, rs_epoch;
  long long rs_slab_off, rs_flag_off;
  int rs_staged;     // partial rows leave through shared memory and bulk copies instead of 16-byte stores
  // gated input: see nfk_gemm_params::gate_flags
  const unsigned int* gate_flags;
  int gate_epoch, gate_nranks;
  // columns from f32_col0 on go to D32 as fp32 (D32 null: none do)
  float* D32;
  long long ld32;
  int f32_col0;
  int d32_wide, d_wide, part_wide;  // rows of D32 / D / the fp32 partial copies start on 32-byte boundaries
  GatedAct act;                     // gated epilogue
  int lin_act;                      // linear epilogue: NFK_LIN_*
  int groups, group_n, group_k;     // block-diagonal product (groups 1: an ordinary one)
};

// First output column of column block `n_blk`, the column its group ends at, and where its group starts in
// A's columns. A column block never straddles two groups.
struct NBlock {
  int col0, col_end, a_k0;
};
__host__ __device__ __forceinline__ int n_block_count(int groups, int group_n, int out_bn) {
  return groups * ((group_n + out_bn - 1) / out_bn);
}
__device__ __forceinline__ NBlock n_block(const DevParams& p, int n_blk, int out_bn) {
  NBlock b;
  if (p.groups == 1) {
    b.col0 = n_blk * out_bn;
    b.a_k0 = 0;
    b.col_end = min(p.N, b.col0 + out_bn);
  } else {
    const int per = (p.group_n + out_bn - 1) / out_bn;
    const int g = n_blk / per;
    b.col0 = g * p.group_n + (n_blk - g * per) * out_bn;
    b.a_k0 = g * p.group_k;
    b.col_end = min((g + 1) * p.group_n, b.col0 + out_bn);
  }
  return b;
}

// v += the bias of eight columns.
__device__ __forceinline__ void add_bias8(float* v, uint4 bv) {
  const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(bw[j]);
    v[2 * j] += f.x;
    v[2 * j + 1] += f.y;
  }
}

__device__ __forceinline__ void add_bias8(float* v, const __nv_bfloat16* bias) {
  add_bias8(v, *reinterpret_cast<const uint4*>(bias));
}

// A thread holds columns of one row of its own, so a store of 16 bytes touches half a sector in each of 32 rows; 32 bytes make
// it whole.
__device__ __forceinline__ void store_32_bytes(void* dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f,
                                               uint32_t g, uint32_t h) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(a), "r"(b), "r"(c), "r"(d), "r"(e),
               "r"(f), "r"(g), "r"(h)
               : "memory");
}

// Eight fp32 partial sums of one row.
__device__ __forceinline__ void store_part8(float* dst, const float* v, bool wide) {
  if (wide) {
    store_32_bytes(dst, __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]),
                   __float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7]));
    return;
  }
  __stcg(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
  __stcg(reinterpret_cast<float4*>(dst) + 1, make_float4(v[4], v[5], v[6], v[7]));
}

// Eight finished columns of one row: bf16 to D, or fp32 to D32 from f32_col0 on (a multiple of 8).
__device__ __forceinline__ void store_cols8(const DevParams& p, int row, int col, float* v) {
  if (p.lin_act != NFK_LIN_NONE) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = lin_act_of(v[j], p.lin_act);
  }
  if (p.D32 != nullptr && col >= p.f32_col0) {
    float* out = p.D32 + static_cast<long long>(row) * p.ld32 + (col - p.f32_col0);
    if (p.d32_wide) {          // one store per 32-byte sector
      asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                   "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                   : "memory");
      return;
    }
    float4* dst = reinterpret_cast<float4*>(out);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
    return;
  }
  uint4 o;
  o.x = pack_bf16x2(v[0], v[1]);
  o.y = pack_bf16x2(v[2], v[3]);
  o.z = pack_bf16x2(v[4], v[5]);
  o.w = pack_bf16x2(v[6], v[7]);
  *reinterpret_cast<uint4*>(p.D + static_cast<long long>(row) * p.ldd + col) = o;
}

// Sixteen finished columns of one row, of which the first eight or all lie before `col_end`.
__device__ __forceinline__ void store_cols16(const DevParams& p, int row, int col, int col_end, float* v) {
  if (p.d_wide && p.D32 == nullptr && p.lin_act == NFK_LIN_NONE && (col & 15) == 0 && col + 8 < col_end) {
    store_32_bytes(p.D + static_cast<long long>(row) * p.ldd + col, pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                   pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]), pack_bf16x2(v[8], v[9]), pack_bf16x2(v[10], v[11]),
                   pack_bf16x2(v[12], v[13]), pack_bf16x2(v[14], v[15]));
    return;
  }
  store_cols8(p, row, col, v);
  if (col + 8 < col_end) store_cols8(p, row, col + 8, v + 8);
}

// Tile index -> (m group, n block). Normally m groups vary fastest, so CTAs that run together share
// weight panels in L2; with a gated input n blocks vary fastest, so the first wave of tiles needs only the
// first rows of A.
__device__ __forceinline__ void tile_coords(const DevParams& p, int tile, int m_groups, int n_blocks, int& m_grp,
                                            int& n_blk) {
  if (p.gate_flags != nullptr) {
    m_grp = tile / n_blocks;
    n_blk = tile - m_grp * n_blocks;
  } else {
    m_grp = tile % m_groups;
    n_blk = tile / m_groups;
  }
}

// Bounded wait until every rank has delivered its rows of 128-row block `m_tile` of A. The flags are
// written by remote stores (st.release.sys); the loads that follow are TMA copies (async proxy), hence
// the proxy fence after the acquire.
__device__ __forceinline__ bool wait_gate(const DevParams& p, int m_tile, volatile int* abort_flag) {
  const unsigned int* f = p.gate_flags + static_cast<long long>(m_tile) * 8;
  uint64_t t0 = 0;
  for (int r = 0; r < p.gate_nranks; ++r) {
    for (uint32_t it = 0;; ++it) {
      unsigned int v;
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(f + r) : "memory");
      if (static_cast<int>(v - static_cast<unsigned int>(p.gate_epoch)) >= 0) break;
      if ((it & 63u) == 63u) {
        if (*abort_flag) return false;
        if (p.status != nullptr && *reinterpret_cast<volatile unsigned int*>(p.status) != 0u) return false;
        uint64_t now;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (t0 == 0) t0 = now;
        if (now - t0 > 2000000000ull) return false;   // 2 s
        __nanosleep(64);
      }
    }
  }
  asm volatile("fence.proxy.async;" ::: "memory");
  return true;
}

// ---- work distribution -----------------------------------------------------------------------------
// The output is cut into tiles (m group x n block; m groups vary fastest so CTAs that run together
// share B panels in L2) and, with split-K, each tile's k-blocks into split_k equal ranges. A work
// unit is (tile, k range); CTA c takes units c, c+G, ... A k range that is only part of K is written
// as an fp32 partial tile and a second pass adds the partials and applies the epilogue.
struct Segment {
  int tile, ks, kb0, kb1;
  int sk_tile, piece, n_pieces;   // stream-K tail: index in the tail region, which piece, of how many
};
// Pieces that share tile t of the tail region: workers first..last (the ranges are q k-blocks long).
__host__ __device__ __forceinline__ void sk_tile_pieces(int t, int num_kb, int q, int sk_total, int& first, int& last) {
  first = (t * num_kb) / q;
  const int end = (t + 1) * num_kb < sk_total ? (t + 1) * num_kb : sk_total;
  last = (end - 1) / q;
}
// Units come in two phases. First whole tiles (with split-K: (tile, k range) pairs) dealt round-robin:
// worker w takes units w, w+W, ... Then, when the tile count is not a multiple of W, the k-blocks of
// the left-over tiles laid end to end and cut into W equal ranges, so that the last wave keeps every
// worker busy; the pieces of a tile cut that way are fp32 partial sums that sk_fixup_kernel adds up.
struct Walk {
  int cur, units, tiles_dp, num_kb, kb_per, step;
  int g, g_end, q, sk_total;
  __device__ __forceinline__ Walk(int w, int W, int tiles_, int num_kb_, int split_k, int tiles_dp_, int q_)
      : cur(w), units((q_ > 0 ? tiles_dp_ : tiles_) * split_k), tiles_dp(q_ > 0 ? tiles_dp_ : tiles_),
        num_kb(num_kb_), kb_per((num_kb_ + split_k - 1) / split_k), step(W), q(q_) {
    sk_total = q_ > 0 ? (tiles_ - tiles_dp_) * num_kb_ : 0;
    g = q_ > 0 ? min(w * q_, sk_total) : 0;
    g_end = q_ > 0 ? min(g + q_, sk_total) : 0;
  }
  __device__ __forceinline__ bool next(Segment& s) {
    if (cur < units) {
      s.tile = cur % tiles_dp;
      s.ks = cur / tiles_dp;
      s.kb0 = min(num_kb, s.ks * kb_per);
      s.kb1 = min(num_kb, s.kb0 + kb_per);
      s.sk_tile = 0;
      s.piece = 0;
      s.n_pieces = 1;
      cur += step;
      return true;
    }
    if (g < g_end) {
      const int t = g / num_kb;
      const int kb0 = g - t * num_kb;
      const int len = min(num_kb - kb0, g_end - g);
      s.tile = tiles_dp + t;
      s.ks = 0;
      s.kb0 = kb0;
      s.kb1 = kb0 + len;
      s.sk_tile = t;
      int first, last;
      sk_tile_pieces(t, num_kb, q, sk_total, first, last);
      s.n_pieces = last - first + 1;
      s.piece = g / q - first;
      g += len;
      return true;
    }
    return false;
  }
};

// CG = 1: one CTA per tile. CG = 2 (MT must be 1): the two CTAs of a cluster share a 256-row tile;
// each stages its own 128 rows of A and BN/2 of the weight rows, the even CTA issues
// tcgen05.mma.cta_group::2 for both, and each CTA drains its own 128 accumulator rows. Per SM that
// halves the weight bytes entering shared memory for the same tensor work.
// WIDE (CTA pairs, plain epilogue): a tile of more than 256 columns, computed as two pair MMAs of BN / 2 columns
// per k step into one accumulator of BN columns. A pair MMA takes half of its weight rows from each CTA, so
// each CTA stages quarter `rank` of both halves, one behind the other, and the accumulator columns come out in
// the order of the weight rows. A separate instantiation: the common kernel's instruction stream is untouched.
// Forms of the epilogue as template parameter: NFK_EPI_*, and the gated one with biases on both halves, which has kernels of
// its own so that the others keep their registers.
constexpr int kGatedBias = 3;
constexpr bool gated_epi(int epi) { return epi == 1 || epi == kGatedBias; }
// Most registers of a thread: what other streams' kernels find beside a GEMM's CTA hangs on it. An SM's registers are four banks
// of 16384 for the warps of one scheduler each, and two of the six warps share two of them. At 104 registers 9728 are left there:
// a decode CTA of three stages (232 registers a thread), or one of two stages (168) and a collective's of up to 136; at the 154
// that the plain epilogue would take 6144, one CTA of 168. (With known kernels: 192 threads of up to 88 registers leave room for two
// CTAs of 128 threads with 168, of 96 to 160 for one.) Gated epilogues: 120 (124 without the limit); those with a bias and those of
// several M tiles keep what they take (111 to 128).
constexpr int gemm_registers(int mt, int epi) { return epi == 0 ? (mt == 1 ? 104 : 120) : epi == 1 && mt == 1 ? 120 : 255; }

template <int MT, int EPI, int CG, bool WIDE>
__global__ void __maxnreg__(gemm_registers(MT, EPI))
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB0,
                    const __grid_constant__ CUtensorMap tmB1, DevParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_al = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_al);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kMaxStages;
  uint64_t* tmem_full = bars + 2 * kMaxStages;
  uint64_t* tmem_empty = bars + 2 * kMaxStages + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* smem = smem_al + 1024;     // ring slots

  // The warp number by a shuffle: the compiler then knows that a role's loop counters are the same in all lanes of a warp
  // and keeps the operands of TMA and tcgen05 instructions in uniform registers (see elect_one). With roles of one thread
  // (`lane == 0`) the issue of a k-block's four pair MMAs took longer than the MMAs: 2048 x 8192 x 28672 went from 745 to
  // 619 us (1.29 -> 1.55 PFLOP/s), 2048 x 10240 x 8192 from 255 to 228, 1024 x 8192 x 8192 from 121 to 104.
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  static_assert(CG == 1 || MT == 1, "CTA pairs cover one M tile per CTA");
  static_assert(!WIDE || (CG == 2 && EPI == 0), "wide tiles: CTA pairs, plain epilogue");
  const uint32_t rank = (CG == 2) ? cluster_ctarank() : 0u;   // position in the CTA pair
  const bool leader = rank == 0;
  const int BN = p.bn;                    // tile width = N of one MMA instruction
  const int STAGES = p.stages;
  const int ACC_BUFS = p.acc_bufs;
  const int ACC_COLS = MT * BN;
  const int B_BYTES = (BN / CG) * BK * 2; // weight rows this CTA stages per k-block
  // A CTA that gives up tells its peer too, so the pair unwinds together.
  auto raise_abort = [&]() {
    *abort_flag = 1;
    if (CG == 2)
      st_shared_cluster_u32(mapa_shared(smem_u32(const_cast<int*>(abort_flag)), rank ^ 1u), 1u);
  };
  const int STAGE_BYTES = MT * A_TILE_BYTES + B_BYTES;
  constexpr int A_BYTES = MT * A_TILE_BYTES;
  // Output tile width: the SwiGLU epilogue folds a gate half and an up half of BN/2 columns each.
  const int OUT_BN = gated_epi(EPI) ? BN / 2 : BN;
  const int m_tiles = (p.M + BM - 1) / BM;
  const int m_groups = (m_tiles + MT * CG - 1) / (MT * CG);
  const int n_blocks = n_block_count(p.groups, p.group_n, OUT_BN);
  const int num_kb = (p.K + BK - 1) / BK;
  const int tiles = m_groups * n_blocks;
  const int sk = p.split_k;
  const int worker = blockIdx.x / CG, workers = gridDim.x / CG;   // a CTA, or a CTA pair

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 4 * CG);   // the epilogue warps of every CTA that shares the tile
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB0);
    if (gated_epi(EPI)) tma_prefetch_desc(&tmB1);
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
  // With gated input this kernel waits for another stream's collective, whose CTAs still need their places on the SMs: the
  // next kernel starts when this one has ended.
  if (p.gate_flags == nullptr) let_next_start();
  await_previous();

  if (warp == 0) {
    // ---------------- TMA producer (the whole warp walks the tiles, an elected lane issues) ----------------
    // ring position kept as (slot, phase) counters: the stage count is a runtime value and a
    // division per k-block would sit on this thread's issue path
    uint32_t it = 0, ph = 0;
    int s = 0;
    bool ok = true;
    Walk walk(worker, workers, tiles, num_kb, sk, p.sk_tiles_dp, p.sk_q);
    Segment sg;
    int gate_seen = -1;     // M tiles up to this one have been seen complete (tiles are walked in row order)
    while (ok && walk.next(sg)) {
      int m_grp, n_blk;
      tile_coords(p, sg.tile, m_groups, n_blocks, m_grp, n_blk);
      const int mt_valid = min(MT, m_tiles - m_grp * MT);
      const NBlock nb = n_block(p, n_blk, OUT_BN);
      if (p.gate_flags != nullptr) {
        // last 128-row block of A that this CTA loads for the tile
        const int need = (CG == 2) ? min(m_tiles - 1, m_grp * 2 + static_cast<int>(rank)) : m_grp * MT + mt_valid - 1;
        const int first = (CG == 2) ? need : m_grp * MT;
        for (int mt_i = max(first, gate_seen + 1); mt_i <= need && ok; ++mt_i) {
          if (!__all_sync(0xffffffffu, wait_gate(p, mt_i, abort_flag))) {
            report_status(p.status, NF_ST_TIMEOUT_PEER_FLAG);
            raise_abort();
            ok = false;
          }
        }
        if (!ok) break;
        if (need > gate_seen) gate_seen = need;
      }
      for (int kb = sg.kb0; kb < sg.kb1; ++kb, ++it, s = (s + 1 == STAGES) ? 0 : s + 1, ph ^= (s == 0)) {
        if (!__all_sync(0xffffffffu, wait_or_abort(&empty_bar[s], ph ^ 1, abort_flag))) {
          report_status(p.status, NF_ST_TIMEOUT_SMEM_EMPTY);
          raise_abort();
          ok = false;
          break;
        }
        uint8_t* sa = smem + s * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        if (elect_one()) {
          if (CG == 2) {
            // Both CTAs' bytes are counted on the even CTA's barrier, which its MMA thread waits on.
            // A tile past the last row or column is still copied in full (zero filled).
            const uint32_t fb = mapa_shared(smem_u32(&full_bar[s]), 0);
            if (leader) mbar_expect_tx(&full_bar[s], 2 * (A_TILE_BYTES + B_BYTES));
            if (gated_epi(EPI))
              tma_load_2d_pair(sb, rank == 0 ? &tmB0 : &tmB1, fb, kb * BK, nb.col0);
            else if (WIDE) {
              const int qrows = BN / 4;
              tma_load_2d_pair(sb, &tmB0, fb, kb * BK, nb.col0 + static_cast<int>(rank) * qrows);
              tma_load_2d_pair(sb + qrows * (BK * 2), &tmB0, fb, kb * BK,
                               nb.col0 + BN / 2 + static_cast<int>(rank) * qrows);
            } else
              tma_load_2d_pair(sb, &tmB0, fb, kb * BK, nb.col0 + static_cast<int>(rank) * (BN / 2));
            tma_load_2d_pair(sa, &tmA, fb, nb.a_k0 + kb * BK, (m_grp * 2 + static_cast<int>(rank)) * BM);
          } else {
            mbar_expect_tx(&full_bar[s], mt_valid * A_TILE_BYTES + B_BYTES);
            if (gated_epi(EPI)) {
              tma_load_2d(sb, &tmB0, &full_bar[s], kb * BK, nb.col0);
              tma_load_2d(sb + B_BYTES / 2, &tmB1, &full_bar[s], kb * BK, nb.col0);
            } else {
              tma_load_2d(sb, &tmB0, &full_bar[s], kb * BK, nb.col0);
            }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
              if (mt < mt_valid)
                tma_load_2d(sa + mt * A_TILE_BYTES, &tmA, &full_bar[s], nb.a_k0 + kb * BK, (m_grp * MT + mt) * BM);
          }
        }
        __syncwarp();
      }
    }
    if (CG == 2 && ok) {
      // Every arrival that the even CTA's commits send to this CTA's slot barriers has landed once
      // each slot reads as free again.
      for (int j = 0; j < STAGES; ++j, s = (s + 1 == STAGES) ? 0 : s + 1, ph ^= (s == 0))
        if (!wait_or_abort(&empty_bar[s], ph ^ 1, abort_flag)) break;
    }
    if (!ok && leader) {
      // Drain: give loads already in flight a bounded chance to land before the CTA exits (a
      // pair's loads are all counted on the even CTA's barriers).
      const uint32_t issued = it;
      const uint32_t back = issued < static_cast<uint32_t>(STAGES) ? issued : STAGES;
      for (uint32_t j = issued - back; j < issued; ++j) {
        const int s = j % STAGES;
        const uint32_t ph = (j / STAGES) & 1;
        for (int spin = 0; spin < 100000; ++spin) {
          uint32_t done;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
              "selp.u32 %0, 1, 0, p;\n\t}"
              : "=r"(done)
              : "r"(smem_u32(&full_bar[s])), "r"(ph)
              : "memory");
          if (done) break;
        }
      }
    }
  } else if (warp == 1 && leader) {
    // ---------------- MMA issuer (the even CTA of a pair issues for both) ----------------
    const uint32_t idesc = umma_idesc_bf16(BM * CG, WIDE ? BN / 2 : BN);
    const uint32_t ring_addr = smem_u32(smem);
    uint32_t tcount = 0, ph = 0;
    int s = 0;
    bool ok = true;
    Walk walk(worker, workers, tiles, num_kb, sk, p.sk_tiles_dp, p.sk_q);
    Segment sg;
    while (ok && walk.next(sg)) {
      int m_grp, n_blk_unused;
      tile_coords(p, sg.tile, m_groups, n_blocks, m_grp, n_blk_unused);
      const int mt_valid = (CG == 2) ? 1 : min(MT, m_tiles - m_grp * MT);
      const uint32_t acc = (ACC_BUFS == 2) ? (tcount & 1) : 0;
      const uint32_t acc_ph = (ACC_BUFS == 2) ? ((tcount >> 1) & 1) : (tcount & 1);
      if (!__all_sync(0xffffffffu, wait_or_abort(&tmem_empty[acc], acc_ph ^ 1, abort_flag))) {
        report_status(p.status, NF_ST_TIMEOUT_TMEM_EMPTY);
        raise_abort();
        break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
      for (int kb = sg.kb0; kb < sg.kb1; ++kb, s = (s + 1 == STAGES) ? 0 : s + 1, ph ^= (s == 0)) {
        if (!__all_sync(0xffffffffu, wait_or_abort(&full_bar[s], ph, abort_flag))) {
          report_status(p.status, NF_ST_TIMEOUT_SMEM_FULL);
          raise_abort();
          ok = false;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t a_desc = umma_desc_k_sw128(ring_addr + s * STAGE_BYTES);
          const uint64_t b_desc = a_desc + (A_BYTES >> 4);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            if (mt < mt_valid) {
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; ++k) {
                const uint32_t on = (kb != sg.kb0 || k != 0) ? 1u : 0u;
                const uint64_t da = a_desc + ((mt * A_TILE_BYTES + k * UMMA_K * 2) >> 4);
                const uint64_t db = b_desc + (k * UMMA_K * 2 >> 4);
                if (CG == 2) umma_bf16_ss_pair(d_tmem, da, db, idesc, on);
                else umma_bf16_ss(d_tmem + mt * BN, da, db, idesc, on);
                if (WIDE)   // second half of the tile: the weight rows staged behind the first quarter
                  umma_bf16_ss_pair(d_tmem + BN / 2, da, db + static_cast<uint64_t>((BN / 4) * (BK * 2) >> 4), idesc, on);
              }
            }
          }
          // the stage is free (in both CTAs of a pair) once these MMAs have read it
          if (CG == 2) umma_commit_pair_both(&empty_bar[s]);
          else umma_commit(&empty_bar[s]);
        }
        __syncwarp();
      }
      if (ok && elect_one()) {
        if (CG == 2) umma_commit_pair_both(&tmem_full[acc]);
        else umma_commit(&tmem_full[acc]);
      }
      __syncwarp();
      ++tcount;
    }
  } else if (warp >= 2) {
    // ---------------- epilogue (4 warps, 128 threads) ----------------
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    uint32_t tcount = 0;
    Walk walk(worker, workers, tiles, num_kb, sk, p.sk_tiles_dp, p.sk_q);
    Segment sg;
    while (walk.next(sg)) {
      int m_grp, n_blk;
      tile_coords(p, sg.tile, m_groups, n_blocks, m_grp, n_blk);
      const int m_first = (m_grp * CG + static_cast<int>(rank)) * MT;   // first M tile this CTA drains
      const int mt_valid = min(MT, m_tiles - m_first);                  // <= 0: tile past the last row
      const uint32_t acc = (ACC_BUFS == 2) ? (tcount & 1) : 0;
      const uint32_t acc_ph = (ACC_BUFS == 2) ? ((tcount >> 1) & 1) : (tcount & 1);
      ++tcount;
      if (!wait_or_abort(&tmem_full[acc], acc_ph, abort_flag)) {
        if (lane == 0) report_status(p.status, NF_ST_TIMEOUT_TMEM_FULL);
        raise_abort();
        break;
      }
      __syncwarp();
      tc_fence_after();
      const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * ACC_COLS;
      // a k range that received no k-blocks contributes zeros (its accumulator was never written)
      const bool empty_range = sg.kb0 >= sg.kb1;
      // Stream-K tail: the fp32 partial copies of this tile (one slot per piece and CTA of a pair).
      const long long slot_floats = static_cast<long long>(MT) * BM * BN;
      float* const sk_tile_base = (EPI != 2 && sg.n_pieces > 1)
          ? p.sk_partial + (static_cast<long long>(sg.sk_tile) * p.sk_max_pieces * CG) * slot_floats
          : nullptr;
      // mode 0: epilogue to the output; mode 1: raw accumulators to this piece's slot.
      auto drain = [&](const int mode) {
#pragma unroll 1
        for (int mt = 0; mt < mt_valid; ++mt) {
          const int row = (m_first + mt) * BM + q * 32 + lane;
          const bool row_ok = row < p.M;
          const long long row_local = static_cast<long long>(mt * BM + q * 32 + lane) * BN;
          const NBlock nb = n_block(p, n_blk, OUT_BN);
          const int tile_col_end = nb.col_end;   // columns past it belong to the next tile
          if constexpr (gated_epi(EPI)) {
            // 16 gate and 16 up columns at a time: more would take 80 registers more, which a kernel beside this one needs. With
            // the activations' chains overlapped (gated_acts) a tile of 128 x 128 leaves in 4 us instead of 22, under the next
            // tile's loop; 14336 x 2 x 4096: 256 rows 71 -> 52 us, 333 100 -> 81, 700 163 -> 122, 1000 228 -> 164.
#pragma unroll 1
            for (int c = 0; c < OUT_BN; c += 16) {
              uint32_t r[16], uu[16];
              tmem_ld_32x32b_x16n(t_lane + mt * BN + c, r);
              tmem_ld_32x32b_x16n(t_lane + mt * BN + BN / 2 + c, uu);
              const int col = nb.col0 + c;
              uint4 bias_w[EPI == kGatedBias ? 2 : 1], bias2_w[EPI == kGatedBias ? 2 : 1];
              if constexpr (EPI == kGatedBias) {       // requested while the accumulators are on their way
#pragma unroll
                for (int g8 = 0; g8 < 2; ++g8) {
                  const bool in = col + g8 * 8 < tile_col_end;
                  bias_w[g8] = in ? *reinterpret_cast<const uint4*>(p.bias + col + g8 * 8) : make_uint4(0, 0, 0, 0);
                  bias2_w[g8] = in ? *reinterpret_cast<const uint4*>(p.bias2 + col + g8 * 8) : make_uint4(0, 0, 0, 0);
                }
              }
              tmem_ld_wait();
              float gsum[16], usum[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                gsum[j] = __uint_as_float(r[j]);
                usum[j] = __uint_as_float(uu[j]);
              }
              if (mode == 1) {
                if (row_ok) {
                  float* own = sk_tile_base + (static_cast<long long>(sg.piece) * CG + rank) * slot_floats + row_local;
#pragma unroll
                  for (int g8 = 0; g8 < 2; ++g8) {
                    store_part8(own + c + g8 * 8, gsum + g8 * 8, p.part_wide);
                    store_part8(own + BN / 2 + c + g8 * 8, usum + g8 * 8, p.part_wide);
                  }
                }
                continue;
              }
              if constexpr (EPI == kGatedBias) {
#pragma unroll
                for (int g8 = 0; g8 < 2; ++g8) {
                  add_bias8(gsum + g8 * 8, bias_w[g8]);
                  add_bias8(usum + g8 * 8, bias2_w[g8]);
                }
              }
              gated_acts<16>(gsum, usum, p.act);
              if (row_ok && col < tile_col_end) store_cols16(p, row, col, tile_col_end, gsum);
            }
          } else if constexpr (EPI == 0) {
            // Partial sums, of a split K or of a piece of a stream-K tail, as they are.
            if (mode == 1 || p.partial != nullptr) {
              float* prow = mode == 1 ? sk_tile_base + (static_cast<long long>(sg.piece) * CG + rank) * slot_floats + row_local
                                      : p.partial + (static_cast<long long>(sg.ks) * p.M + row) * p.N + nb.col0;
              const int end = !row_ok ? 0 : mode == 1 ? OUT_BN : tile_col_end - nb.col0;
#pragma unroll 1
              for (int c = 0; c < OUT_BN; c += 32) {
                uint32_t r[32];
                float v[32];
                tmem_ld_32x32b_x32(t_lane + mt * BN + c, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = empty_range ? 0.f : __uint_as_float(r[j]);
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8)
                  if (c + g8 * 8 < end) store_part8(prow + c + g8 * 8, v + g8 * 8, p.part_wide);
              }
              continue;
            }
            // What the residual adds to 16 columns is requested 32 columns ahead: D may be C itself, so the compiler cannot move
            // these loads over the stores before them, and each eight columns would wait for HBM. 16 columns at a time: 32 and the
            // residual of 64 took 154 registers (see gemm_registers).
            const __nv_bfloat16* crow = (p.C != nullptr && row_ok) ? p.C + static_cast<long long>(row) * p.ldc : nullptr;
            uint4 c_in[4] = {};
            auto request_c = [&](int h, int c) {
#pragma unroll
              for (int g8 = 0; g8 < 2; ++g8) {
                const int col = nb.col0 + c + g8 * 8;
                if (col < tile_col_end) c_in[h * 2 + g8] = *reinterpret_cast<const uint4*>(crow + col);
              }
            };
            if (crow != nullptr) {
              request_c(0, 0);
              request_c(1, 16);
            }
#pragma unroll 1
            for (int c0 = 0; c0 < OUT_BN; c0 += 32) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int c = c0 + h * 16, col0 = nb.col0 + c;
                uint32_t r[16];
                float v[16];
                tmem_ld_32x32b_x16n(t_lane + mt * BN + c, r);
                const uint4 c_now[2] = {c_in[h * 2], c_in[h * 2 + 1]};
                if (crow != nullptr && c + 32 < OUT_BN) request_c(h, c + 32);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = empty_range ? 0.f : __uint_as_float(r[j]);
                if (row_ok && col0 < tile_col_end) {
#pragma unroll
                  for (int g8 = 0; g8 < 2; ++g8) {
                    const int col = col0 + g8 * 8;
                    if (col < tile_col_end) {  // N is a multiple of 8
                      float* vv = v + g8 * 8;
                      if (p.bias != nullptr) add_bias8(vv, p.bias + col);
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
                  }
                  store_cols16(p, row, col0, tile_col_end, v);
                }
              }
            }
          } else {
#pragma unroll 1
            for (int c = 0; c * 32 < OUT_BN; ++c) {
              uint32_t r[32];
              float v[32];
              tmem_ld_32x32b_x32(t_lane + mt * BN + c * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = empty_range ? 0.f : __uint_as_float(r[j]);
              const int col0 = nb.col0 + c * 32;
              if (p.rs_staged) {
                // Staged push: this lane's 32 columns go to its row of the warp's staging piece; when a
                // run of 128 columns (or the tile's last columns) is complete, one bulk copy per lane
                // sends the row's run to the owner's slab. A lane only ever reads back what it wrote, so
                // the generic -> async proxy fence is all the ordering the copy needs.
                uint8_t* stage_row = smem + STAGES * STAGE_BYTES + (q * 32 + lane) * kRsRowPitch;
                // the bulk copy of the previous run reads this row: it must be done reading before the first
                // write of a new run (waiting here, not right after the copy, lets the copy run under the
                // accumulator loads in between)
                if ((c & 3) == 0) tma_store_wait_read<0>();
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8) {
                  const float* vv = v + g8 * 8;
                  uint4 o;
                  o.x = pack_bf16x2(vv[0], vv[1]);
                  o.y = pack_bf16x2(vv[2], vv[3]);
                  o.z = pack_bf16x2(vv[4], vv[5]);
                  o.w = pack_bf16x2(vv[6], vv[7]);
                  *reinterpret_cast<uint4*>(stage_row + (c & 3) * 64 + g8 * 16) = o;
                }
                const bool run_done = (c & 3) == 3 || (c + 1) * 32 >= OUT_BN;
                if (run_done) {
                  const int run_col0 = n_blk * OUT_BN + (c & ~3) * 32;
                  int run_end = n_blk * OUT_BN + (c + 1) * 32;
                  if (run_end > tile_col_end) run_end = tile_col_end;
                  fence_proxy_async_smem();
                  if (row_ok && run_end > run_col0) {
                    const int owner = row % p.rs_nranks;
                    __nv_bfloat16* srow = reinterpret_cast<__nv_bfloat16*>(p.rs_heap[owner] + p.rs_slab_off) +
                                          (static_cast<long long>(p.rs_rank) * p.rs_rows_cap + row / p.rs_nranks) * p.N;
                    bulk_store_1d(srow + run_col0, stage_row, static_cast<uint32_t>(run_end - run_col0) * 2u);
                  }
                  tma_store_commit();
                }
              } else if (row_ok && col0 < tile_col_end) {
                // push the partial row to its owner's slab (posted NVLink stores; the flag raised at
                // the end of the kernel orders them for the reader)
                const int owner = row % p.rs_nranks;
                __nv_bfloat16* srow = reinterpret_cast<__nv_bfloat16*>(p.rs_heap[owner] + p.rs_slab_off) +
                                      (static_cast<long long>(p.rs_rank) * p.rs_rows_cap + row / p.rs_nranks) * p.N;
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8) {
                  const int col = col0 + g8 * 8;
                  if (col < tile_col_end) {
                    const float* vv = v + g8 * 8;
                    uint4 o;
                    o.x = pack_bf16x2(vv[0], vv[1]);
                    o.y = pack_bf16x2(vv[2], vv[3]);
                    o.z = pack_bf16x2(vv[4], vv[5]);
                    o.w = pack_bf16x2(vv[6], vv[7]);
                    *reinterpret_cast<uint4*>(srow + col) = o;
                  }
                }
              }
            }
          }
        }
      };
      // A piece of a tile that several workers share leaves its partial sums in its slot; a second
      // kernel adds the pieces up and applies the epilogue.
      if (sk_tile_base != nullptr) drain(1);
      else drain(0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_cluster(mapa_shared(smem_u32(&tmem_empty[acc]), 0));
        else mbar_arrive(&tmem_empty[acc]);
      }
    }
  }

  if (EPI == 2) {
    tma_store_wait<0>();                    // bulk copies of the staged form have been written
    __threadfence_system();                 // this thread's pushes are ordered before the flag below
  }
  tc_fence_before();
  // Nothing of the pair may still signal this CTA's barriers or read its shared memory or TMEM once
  // it has exited, so the pair leaves together.
  __syncwarp();
  if (CG == 2) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (CG == 2) tmem_dealloc_pair(tmem_base, static_cast<uint32_t>(p.tmem_cols));
    else tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
  if (EPI == 2 && threadIdx.x == 0) {
    // The last CTA to get here tells every rank that this rank's partial rows have been pushed.
    // Flag block layout (collectives.cu): ready[8], done[8], cta_counter.
    unsigned int* mine = reinterpret_cast<unsigned int*>(p.rs_heap[p.rs_rank] + p.rs_flag_off);
    const unsigned int prev = atomicAdd(mine + 16, 1u);
    if (prev == gridDim.x - 1) {
      mine[16] = 0;
      __threadfence_system();
      for (int r = 0; r < p.rs_nranks; ++r) {
        unsigned int* flag = reinterpret_cast<unsigned int*>(p.rs_heap[r] + p.rs_flag_off) + p.rs_rank;
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(static_cast<unsigned int>(p.rs_epoch))
                     : "memory");
      }
    }
  }
}

// Reduce-scatter epilogue with nothing to push (an empty nano-batch): the consumer still waits for
// this rank's ready flag, so raise it.
__global__ void rs_signal_only_kernel(DevParams p) {
  if (threadIdx.x < p.rs_nranks) {
    unsigned int* flag = reinterpret_cast<unsigned int*>(p.rs_heap[threadIdx.x] + p.rs_flag_off) + p.rs_rank;
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(static_cast<unsigned int>(p.rs_epoch))
                 : "memory");
  }
}

inline int sm_count() { return device_sm_count(); }

// Split-K second passes: D = sum_s partial[s] (+ bias) (+ beta * C), fp32 -> bf16, the pieces added in the order of k.
// The pieces come from L2, so what counts is how many loads are on their way. With a norm a thread block has a row: up to four
// pieces are requested before the first is added, and the residual with them. One piece after the other, each behind the stores
// of the columns before, 333 rows of 4096 columns in three pieces took 13.4 us, now 10.4; of rows of 8200 to 16384 columns (241
// registers, one block to an SM) 140 x 10240 in three, with its product of depth 2048, 30.7 -> 24.3, 1000 x 16384 in two 149 -> 134.
template <int NV>
struct RowPart {
  float v[NV][8];
  uint4 c[NV];
};
// v[i] = the sum of the pieces of eight columns at column col[i] with bias and residual, for the `in` of them.
template <int NV>
__device__ __forceinline__ void sum_pieces(const DevParams& p, int row, const int (&col)[NV], const bool (&in)[NV], RowPart<NV>& r) {
  const long long slab = static_cast<long long>(p.M) * p.N;
  const float* base = p.partial + static_cast<long long>(row) * p.N;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    r.c[i] = make_uint4(0, 0, 0, 0);
    if (p.C != nullptr && in[i]) r.c[i] = *reinterpret_cast<const uint4*>(p.C + static_cast<long long>(row) * p.ldc + col[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) r.v[i][j] = 0.f;
  }
  constexpr int BATCH = NV >= 4 ? 1 : 4 / NV;                    // pieces requested at once: BATCH * NV * 32 bytes of a thread
  for (int s0 = 0; s0 < p.split_k; s0 += BATCH) {
    float4 a[BATCH][NV], b[BATCH][NV];
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const bool on = s0 + k < p.split_k;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (on && in[i]) {
          const float4* src = reinterpret_cast<const float4*>(base + (s0 + k) * slab + col[i]);
          a[k][i] = __ldcg(src);
          b[k][i] = __ldcg(src + 1);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      if (s0 + k < p.split_k) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          if (in[i]) {
            float* v = r.v[i];
            v[0] += a[k][i].x; v[1] += a[k][i].y; v[2] += a[k][i].z; v[3] += a[k][i].w;
            v[4] += b[k][i].x; v[5] += b[k][i].y; v[6] += b[k][i].z; v[7] += b[k][i].w;
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (in[i]) {
      if (p.bias != nullptr) add_bias8(r.v[i], p.bias + col[i]);
      if (p.C != nullptr) {
        const uint32_t cw[4] = {r.c[i].x, r.c[i].y, r.c[i].z, r.c[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(cw[j]);
          r.v[i][2 * j] += p.beta * f.x;
          r.v[i][2 * j + 1] += p.beta * f.y;
        }
      }
    }
  }
}

// Without a norm: a group of eight columns after the other, 64 registers, so that a thread block more fits an SM than with pieces
// and residual requested together (76 registers; no norm, tiles of 256 columns, K 4096: 16 x 2048 in eight parts 13.6 -> 13.3 us,
// 333 x 4096 in four 27.7 -> 26.0, 700 x 8192 in six 115 -> 95).
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(DevParams p) {
  let_next_start();
  await_previous();
  const long long total = static_cast<long long>(p.M) * (p.N >> 3);
  const long long slab = static_cast<long long>(p.M) * p.N;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += 256ll * gridDim.x) {
    const int row = static_cast<int>(i / (p.N >> 3));
    const int col = static_cast<int>(i % (p.N >> 3)) * 8;
    float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int s = 0; s < p.split_k; ++s) {
      const float4* src = reinterpret_cast<const float4*>(p.partial + s * slab + static_cast<long long>(row) * p.N + col);
      const float4 a = src[0], b = src[1];
      v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
      v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
    }
    if (p.bias != nullptr) add_bias8(v, p.bias + col);
    if (p.C != nullptr) {
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
}

// The same with the RMSNorm of the result folded in: one CTA per row (N <= 16384), every thread keeps its NV groups of eight
// columns of the row in registers, so the norm costs one block reduction and one more store instead of a kernel that reads the
// row back.
constexpr int kRowVec = 8;   // most groups per thread: 8 * 8 * 256 threads = 16384 columns
template <int NV>
__global__ void __launch_bounds__(256, NV == 1 ? 3 : NV <= 4 ? 2 : 1)
splitk_reduce_norm_kernel(DevParams p) {
  __shared__ float red[8];
  let_next_start();
  await_previous();
  const int nvec = p.N >> 3;
  int col[NV];
  bool in[NV];
  uint4 w[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int vi = threadIdx.x + i * 256;
    in[i] = vi < nvec;
    col[i] = vi * 8;
    w[i] = in[i] ? *reinterpret_cast<const uint4*>(p.norm_w + col[i]) : make_uint4(0, 0, 0, 0);
  }
  for (int row = blockIdx.x; row < p.M; row += gridDim.x) {
    RowPart<NV> r;
    sum_pieces<NV>(p, row, col, in, r);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (in[i]) {
        float* v = r.v[i];
        uint4 o;
        o.x = pack_bf16x2(v[0], v[1]);
        o.y = pack_bf16x2(v[2], v[3]);
        o.z = pack_bf16x2(v[4], v[5]);
        o.w = pack_bf16x2(v[6], v[7]);
        *reinterpret_cast<uint4*>(p.D + static_cast<long long>(row) * p.ldd + col[i]) = o;
        // normalise what was stored (bf16-rounded), as the standalone norm kernel would read it
        const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(ow[j]);
          v[2 * j] = f.x;
          v[2 * j + 1] = f.y;
          ss += f.x * f.x + f.y * f.y;
        }
      }
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = (threadIdx.x & 31) < 8 ? red[threadIdx.x & 31] : 0.f;
    tot = warp_sum(tot);
    __syncthreads();
    const float inv = rsqrtf(tot / static_cast<float>(p.N) + p.norm_eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (in[i]) {
        const uint32_t wv[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
        uint32_t ov[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 g = unpack_bf16x2(wv[j]);
          ov[j] = pack_bf16x2(r.v[i][2 * j] * inv * g.x, r.v[i][2 * j + 1] * inv * g.y);
        }
        *reinterpret_cast<uint4*>(p.norm_out + static_cast<long long>(row) * p.norm_ld + col[i]) =
            make_uint4(ov[0], ov[1], ov[2], ov[3]);
      }
    }
  }
}

// Stream-K tail, second pass: for every tile of the tail region that was cut into pieces, add the
// pieces' fp32 partial sums and apply the epilogue. One thread per 8 output columns of a row; the
// loads of the pieces are independent, so many are in flight per thread.
struct FixupGeom {
  int mt, cg, bn, out_bn, m_groups, num_kb, rest;
};
template <int EPI>
__global__ void __launch_bounds__(256)
sk_fixup_kernel(DevParams p, FixupGeom f) {
  let_next_start();
  await_previous();
  const int rows_cta = f.mt * BM;
  const int groups = f.out_bn / 8;
  const long long slot_floats = static_cast<long long>(rows_cta) * f.bn;
  const int sk_total = f.rest * f.num_kb;
  const long long per_cta = static_cast<long long>(rows_cta) * groups;
  const long long per_tile = per_cta * f.cg;
  const long long total = per_tile * f.rest;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += 256ll * gridDim.x) {
    const int t = static_cast<int>(i / per_tile);
    long long r = i - t * per_tile;
    const int rank = static_cast<int>(r / per_cta);
    r -= rank * per_cta;
    const int row_local = static_cast<int>(r / groups);
    const int gcol = static_cast<int>(r - static_cast<long long>(row_local) * groups) * 8;
    int first, last;
    sk_tile_pieces(t, f.num_kb, p.sk_q, sk_total, first, last);
    const int n_pieces = last - first + 1;
    if (n_pieces < 2) continue;   // written whole by its only piece
    const int tile = p.sk_tiles_dp + t;
    const int m_grp = tile % f.m_groups, n_blk = tile / f.m_groups;
    const int row = (m_grp * f.cg + rank) * rows_cta + row_local;
    const NBlock nb = n_block(p, n_blk, f.out_bn);
    const int col = nb.col0 + gcol;
    if (row >= p.M || col >= nb.col_end) continue;
    const float* base = p.sk_partial + (static_cast<long long>(t) * p.sk_max_pieces * f.cg + rank) * slot_floats +
                        static_cast<long long>(row_local) * f.bn + gcol;
    float a[8] = {0, 0, 0, 0, 0, 0, 0, 0}, u[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
    for (int pi = 0; pi < n_pieces; ++pi) {
      const float* src = base + static_cast<long long>(pi) * f.cg * slot_floats;
      const float4 x0 = __ldcg(reinterpret_cast<const float4*>(src));
      const float4 x1 = __ldcg(reinterpret_cast<const float4*>(src) + 1);
      a[0] += x0.x; a[1] += x0.y; a[2] += x0.z; a[3] += x0.w;
      a[4] += x1.x; a[5] += x1.y; a[6] += x1.z; a[7] += x1.w;
      if (EPI == 1) {
        const float4 y0 = __ldcg(reinterpret_cast<const float4*>(src + f.bn / 2));
        const float4 y1 = __ldcg(reinterpret_cast<const float4*>(src + f.bn / 2) + 1);
        u[0] += y0.x; u[1] += y0.y; u[2] += y0.z; u[3] += y0.w;
        u[4] += y1.x; u[5] += y1.y; u[6] += y1.z; u[7] += y1.w;
      }
    }
    if (EPI == 1) {
      if (p.bias != nullptr) {
        add_bias8(a, p.bias + col);
        add_bias8(u, p.bias2 + col);
      }
      gated_acts<8>(a, u, p.act);
    } else {
      if (p.bias != nullptr) add_bias8(a, p.bias + col);
      if (p.C != nullptr) {
        const uint4 cv = *reinterpret_cast<const uint4*>(p.C + static_cast<long long>(row) * p.ldc + col);
        const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 fl = unpack_bf16x2(cw[j]);
          a[2 * j] += p.beta * fl.x;
          a[2 * j + 1] += p.beta * fl.y;
        }
      }
    }
    store_cols8(p, row, col, a);
  }
}

constexpr int kSmemMax = 227 * 1024;

#include "gemm_few_rows.cuh"
#include "gemm_split_cluster.cuh"
#include "gemm_mid_rows.cuh"

// The caller's parameters as the kernels take them; geometry and work distribution are filled in by the launchers.
inline DevParams dev_params(const nfk_gemm_params& g, bool linear) {
  DevParams p{};
  p.D = reinterpret_cast<__nv_bfloat16*>(g.D);
  p.C = reinterpret_cast<const __nv_bfloat16*>(g.C);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(g.bias);
  p.bias2 = reinterpret_cast<const __nv_bfloat16*>(g.bias2);
  p.ldd = g.ldd;
  p.ldc = g.ldc;
  p.beta = g.beta;
  p.M = g.M;
  p.N = g.N;
  p.K = g.K;
  p.status = g.status;
  for (int r = 0; r < 8; ++r) p.rs_heap[r] = reinterpret_cast<char*>(g.rs_heap[r]);
  p.rs_rank = g.rs_rank;
  p.rs_nranks = g.rs_nranks;
  p.rs_rows_cap = g.rs_rows_cap;
  p.rs_epoch = g.rs_epoch;
  p.rs_slab_off = g.rs_slab_off;
  p.rs_flag_off = g.rs_flag_off;
  p.gate_flags = g.gate_flags;
  p.gate_epoch = g.gate_epoch;
  p.gate_nranks = g.gate_nranks;
  p.D32 = reinterpret_cast<float*>(g.D32);
  p.ld32 = g.ld32;
  p.f32_col0 = g.f32_col0;
  p.d32_wide = (reinterpret_cast<uintptr_t>(g.D32) & 31) == 0 && g.ld32 % 8 == 0;
  p.d_wide = (reinterpret_cast<uintptr_t>(g.D) & 31) == 0 && g.ldd % 16 == 0;
  p.part_wide = (reinterpret_cast<uintptr_t>(g.workspace) & 31) == 0;      // rows of N (a multiple of 8) or bn floats
  p.act = GatedAct{g.act, g.act_limit, g.act_alpha, g.act_shift};
  p.lin_act = linear ? g.lin_act : NFK_LIN_NONE;
  p.groups = g.groups > 1 ? g.groups : 1;
  p.group_n = g.N / p.groups;
  p.group_k = g.group_k;
  return p;
}

// The norm of finished rows as a launch of its own.
inline int rmsnorm_rows(const nfk_gemm_params& g, cudaStream_t stream) {
  const nfk_norm_params n{g.norm_out, g.D, g.norm_w, nullptr, g.M, g.N, g.norm_eps,
                          early_further(g.early_start) ? NFK_EARLY_FIRST : 0};
  return nfk_norm_p(&n, stream);
}

// Stream-K tail: with `tiles` tiles on `workers` workers, the tiles_dp tiles of the full waves are
// whole-tile units; the k-blocks of the rest are cut into ranges of q (>= 8, so a piece is worth its
// set-up), one per worker.
struct SkPlan {
  int tiles_dp, q, max_pieces, rest;
};
inline SkPlan plan_stream_k(int tiles, int workers, int num_kb) {
  SkPlan pl{tiles, 0, 0, 0};
  const int rest = tiles % workers;
  if (rest == 0 || num_kb < 2) return pl;
  int q = (static_cast<long long>(rest) * num_kb + workers - 1) / workers;
  const int q_min = num_kb < 8 ? num_kb : 8;
  if (q < q_min) q = q_min;
  if (q >= num_kb) return pl;           // nothing would be cut
  pl.tiles_dp = tiles - rest;
  pl.q = q;
  pl.max_pieces = (num_kb + q - 1) / q + 1;
  pl.rest = rest;
  return pl;
}

template <int MT, int EPI, int CG, bool WIDE>
int launch_impl(const nfk_gemm_params& g, int bn, int split_k, bool stream_k, cudaStream_t stream) {
  int budget = g.smem_budget_kb > 0 ? g.smem_budget_kb * 1024 : kSmemMax;
  if (budget > kSmemMax) budget = kSmemMax;
  const bool rs_staged = EPI == 2 && g.rs_staged != 0;
  const Geom geo = make_geom(bn, MT, gated_epi(EPI), budget, CG, rs_staged ? kRsStageBytes : 0);
  if (geo.stages < 2) return NF_ERR_BAD_ARG;      // shared-memory budget too small for this tile
  CUtensorMap tmA, tmB0, tmB1;
  const int groups = g.groups > 1 ? g.groups : 1;
  const int group_n = g.N / groups;
  // block-diagonal: a k block that runs past a group's K reads the next group's columns of A, which meet
  // the zeros that fill B past its K columns
  int rc = make_tmap_bf16_2d(&tmA, g.A, g.M, g.K + static_cast<uint64_t>(groups - 1) * g.group_k, g.lda, BM, BK);
  if (rc != NF_OK) return rc;
  // rows of B that one TMA copy brings in: a whole tile, a SwiGLU half, or a CTA pair's half
  // (wide tiles: a quarter of the tile per copy, two copies per CTA)
  const int b_box = gated_epi(EPI) ? geo.out_bn : (WIDE ? bn / 4 : bn / CG);
  rc = make_tmap_bf16_2d(&tmB0, g.B, g.N, g.K, g.ldb, b_box, BK);
  if (rc != NF_OK) return rc;
  if (gated_epi(EPI)) {
    rc = make_tmap_bf16_2d(&tmB1, g.B2, g.N, g.K, g.ldb, b_box, BK);
    if (rc != NF_OK) return rc;
  } else {
    tmB1 = tmB0;
  }
  // function attributes and occupancy are per device: one slot per device this process drives
  static bool attr_set_dev[kMaxDevices] = {false};
  static int max_workers_dev[kMaxDevices] = {0};    // CTAs (or CTA pairs) that can be resident at once
  bool& attr_set = attr_set_dev[device_slot()];
  int& max_workers = max_workers_dev[device_slot()];
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_tcgen05_kernel<MT, EPI, CG, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmemMax) != cudaSuccess)
      return NF_ERR_CUDA;
    // Always the largest shared-memory split: with a reduced budget (smem_budget_kb) the SM then
    // keeps room for the CTAs of a kernel that runs beside this one, whichever of the two came first.
    (void)cudaFuncSetAttribute(gemm_tcgen05_kernel<MT, EPI, CG, WIDE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    (void)cudaGetLastError();
    max_workers = sm_count() / CG;
    if (CG == 2) {
      // Pairs must sit on two SMs of one GPC; ask how many fit so that no pair waits for a second wave.
      cudaLaunchConfig_t qc = {};
      qc.gridDim = dim3(sm_count() / 2 * 2);
      qc.blockDim = dim3(kGemmThreads);
      qc.dynamicSmemBytes = kSmemMax;
      cudaLaunchAttribute qa[1];
      qa[0].id = cudaLaunchAttributeClusterDimension;
      qa[0].val.clusterDim.x = 2;
      qa[0].val.clusterDim.y = 1;
      qa[0].val.clusterDim.z = 1;
      qc.attrs = qa;
      qc.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_tcgen05_kernel<MT, EPI, CG, WIDE>, &qc) == cudaSuccess && n > 0 &&
          n < max_workers)
        max_workers = n;
      else
        (void)cudaGetLastError();
    }
    attr_set = true;
  }
  const int m_tiles = (g.M + BM - 1) / BM;
  const int m_groups = (m_tiles + MT * CG - 1) / (MT * CG);
  const int n_blocks = n_block_count(groups, group_n, geo.out_bn);
  const int units = m_groups * n_blocks * split_k;
  int workers = (g.num_ctas > 0 ? g.num_ctas : sm_count()) / CG;
  if (workers > max_workers) workers = max_workers;
  if (workers < 1) workers = 1;
  // stream_k 3: one work unit per CTA (or CTA pair), more CTAs than fit at once; the hardware block
  // scheduler deals the units out as CTAs retire, so an SM that another kernel's CTAs slow down takes
  // fewer of them instead of holding the launch back (no CTA of this kernel waits for another one)
  const bool hw_dealt = g.stream_k == 3 && g.gate_flags == nullptr;
  if (hw_dealt) {
    workers = units;
    stream_k = false;
  }
  SkPlan sk{m_groups * n_blocks, 0, 0, 0};
  if (stream_k && split_k == 1 && EPI != 2 && g.workspace != nullptr) {
    sk = plan_stream_k(m_groups * n_blocks, workers, (g.K + BK - 1) / BK);
    const long long need = static_cast<long long>(sk.rest) * sk.max_pieces * CG * MT * BM * bn * 4;
    if (sk.q > 0 && need > g.workspace_bytes)
      sk = SkPlan{m_groups * n_blocks, 0, 0, 0};
  }
  if (sk.q == 0 && workers > units) workers = units;
  const int ctas = workers * CG;
  DevParams p = dev_params(g, EPI == 0);
  p.partial = split_k > 1 ? reinterpret_cast<float*>(g.workspace) : nullptr;
  p.sk_partial = sk.q > 0 ? reinterpret_cast<float*>(g.workspace) : nullptr;
  p.sk_tiles_dp = sk.tiles_dp;
  p.sk_q = sk.q;
  p.sk_max_pieces = sk.max_pieces;
  p.split_k = split_k;
  p.bn = geo.bn;
  p.stages = geo.stages;
  p.acc_bufs = geo.acc_bufs;
  p.tmem_cols = geo.tmem_cols;
  p.rs_staged = rs_staged ? 1 : 0;
  const bool further = early_further(g.early_start);
  if (launch_kernel(early_first(g.early_start), gemm_tcgen05_kernel<MT, EPI, CG, WIDE>, ctas, kGemmThreads, geo.smem_bytes, stream, CG,
                    tmA, tmB0, tmB1, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return NF_ERR_CUDA;
  }
  if (sk.q > 0 && EPI != 2) {
    FixupGeom f{MT, CG, bn, geo.out_bn, m_groups, (g.K + BK - 1) / BK, sk.rest};
    const long long total = static_cast<long long>(sk.rest) * CG * MT * BM * (geo.out_bn / 8);
    long long blocks = (total + 255) / 256;
    if (blocks > sm_count() * 8) blocks = sm_count() * 8;
    if (launch_kernel(further, sk_fixup_kernel<gated_epi(EPI) ? 1 : 0>, static_cast<int>(blocks), 256, 0, stream, 1, p, f) !=
        cudaSuccess) {
      (void)cudaGetLastError();
      return NF_ERR_CUDA;
    }
  }
  p.norm_w = reinterpret_cast<const __nv_bfloat16*>(g.norm_w);
  p.norm_out = reinterpret_cast<__nv_bfloat16*>(g.norm_out);
  p.norm_ld = g.norm_ld;
  p.norm_eps = g.norm_eps;
  const bool want_norm = EPI == 0 && g.norm_w != nullptr;
  if (split_k > 1 && want_norm && g.N <= kRowVec * 8 * 256) {
    const int blocks = g.M < 16 * sm_count() ? g.M : 16 * sm_count();
    auto* kernel = g.N <= 2048 ? splitk_reduce_norm_kernel<1> : g.N <= 4096 ? splitk_reduce_norm_kernel<2>
                   : g.N <= 8192 ? splitk_reduce_norm_kernel<4> : splitk_reduce_norm_kernel<kRowVec>;
    if (launch_kernel(further, kernel, blocks, 256, 0, stream, 1, p) == cudaSuccess) return NF_OK;
    (void)cudaGetLastError();
    return NF_ERR_CUDA;
  }
  if (split_k > 1) {
    const long long total = static_cast<long long>(g.M) * (g.N >> 3);
    long long blocks = (total + 255) / 256;
    if (blocks > 4ll * sm_count()) blocks = 4ll * sm_count();
    if (launch_kernel(further, splitk_reduce_kernel, static_cast<int>(blocks), 256, 0, stream, 1, p) != cudaSuccess) {
      (void)cudaGetLastError();
      return NF_ERR_CUDA;
    }
  }
  if (want_norm) {
    // the result rows are complete in D (contiguous rows required): a plain norm launch follows
    if (g.ldd != g.N || g.norm_ld != g.N) return NF_ERR_UNSUPPORTED;
    return rmsnorm_rows(g, stream);
  }
  return NF_OK;
}

template <int MT, int EPI, int CG>
int launch(const nfk_gemm_params& g, int bn, int split_k, bool stream_k, cudaStream_t stream) {
  if constexpr (CG == 2 && EPI == 0 && MT == 1) {
    if (bn > 256) return launch_impl<MT, EPI, CG, true>(g, bn, split_k, stream_k, stream);
  }
  if (bn > 256) return NF_ERR_UNSUPPORTED;
  return launch_impl<MT, EPI, CG, false>(g, bn, split_k, stream_k, stream);
}

template <int EPI>
int launch_mt(const nfk_gemm_params& g, int bn, int mt, int cg, int split_k, bool stream_k, cudaStream_t stream) {
  if (cg == 2) return mt == 1 ? launch<1, EPI, 2>(g, bn, split_k, stream_k, stream) : NF_ERR_UNSUPPORTED;
  switch (mt) {
    case 1: return launch<1, EPI, 1>(g, bn, split_k, stream_k, stream);
    case 2: return launch<2, EPI, 1>(g, bn, split_k, stream_k, stream);
    case 4: return launch<4, EPI, 1>(g, bn, split_k, stream_k, stream);
    default: return NF_ERR_UNSUPPORTED;
  }
}

template <bool GATED, int CG>
int launch_few_rows(const nfk_gemm_params& g, const FewPlan& f, cudaStream_t stream) {
  const int groups = g.groups > 1 ? g.groups : 1;
  CUtensorMap tmW0, tmW1, tmX;
  int rc = make_tmap_bf16_2d(&tmW0, g.B, g.N, g.K, g.ldb, GATED ? 64 : 128, BK);
  if (rc != NF_OK) return rc;
  tmW1 = tmW0;
  if (GATED) {
    rc = make_tmap_bf16_2d(&tmW1, g.B2, g.N, g.K, g.ldb, 64, BK);
    if (rc != NF_OK) return rc;
  }
  rc = make_tmap_bf16_2d(&tmX, g.A, g.M, g.K + static_cast<uint64_t>(groups - 1) * g.group_k, g.lda, f.nt / CG, BK);
  if (rc != NF_OK) return rc;
  static bool attr_set_dev[kMaxDevices] = {false};
  bool& attr_set = attr_set_dev[device_slot()];
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_few_rows_kernel<GATED, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) !=
        cudaSuccess)
      return NF_ERR_CUDA;
    (void)cudaFuncSetAttribute(gemm_few_rows_kernel<GATED, CG>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    (void)cudaGetLastError();
    attr_set = true;
  }
  FewParams fp;
  fp.d = dev_params(g, !GATED);
  fp.d.stages = f.stages;
  fp.d.tmem_cols = f.tmem_cols;
  fp.nt = f.nt;
  fp.tok_tiles = f.tok_tiles;
  fp.split = f.split;
  fp.kb_per = f.kb_per;
  fp.round_tokens = f.round_tokens;
  fp.early_weights = g.weights_ready;
  if (launch_kernel(early_first(g.early_start), gemm_few_rows_kernel<GATED, CG>, f.n_tiles * f.tok_tiles * f.split * CG, kFewThreads,
                    f.smem_bytes, stream, f.split * CG, tmW0, tmW1, tmX, fp) != cudaSuccess) {
    (void)cudaGetLastError();
    return NF_ERR_CUDA;
  }
  if (!GATED && g.norm_w != nullptr) return rmsnorm_rows(g, stream);
  return NF_OK;
}

struct Shape {
  int bn, mt, split_k, cg;
  bool stream_k;
  double us = 0.0;      // of a chosen shape, by the model
};

// Clusters of `size` CTAs of `kernel`, with all the shared memory of an SM each, that can be resident at once; asked once per
// device, for which it also sets the kernel's attributes. `known` is that device's answer.
template <class Kernel>
int resident_clusters(Kernel* kernel, int size, int& known) {
  if (known == 0) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    (void)cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    cudaLaunchConfig_t qc = {};
    qc.gridDim = dim3(sm_count() / size * size);
    qc.blockDim = dim3(kGemmThreads);
    qc.dynamicSmemBytes = kSmemMax;
    cudaLaunchAttribute qa[1];
    qa[0].id = cudaLaunchAttributeClusterDimension;
    qa[0].val.clusterDim.x = size;
    qa[0].val.clusterDim.y = 1;
    qa[0].val.clusterDim.z = 1;
    qc.attrs = qa;
    qc.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &qc) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      return 0;
    }
    known = n;
  }
  return known;
}

// What one B200 answers (another 45, 33, 26, 22, 15, 15 from three CTAs on), for planning without one.
constexpr int kResidentClusters[kSplitMaxCluster + 1] = {0, 148, 74, 47, 35, 27, 22, 18, 14};

template <int CG>
int resident_split_clusters(int size) {
  static int known_dev[kMaxDevices][kSplitMaxCluster + 1] = {};
  const int n = resident_clusters(gemm_split_cluster_kernel<CG>, size, known_dev[device_slot()][size]);
  return n > 0 ? n : kResidentClusters[size];
}

// Calls that may run as clusters which add their parts of K among themselves. Those with a CTA or shared-memory budget keep the
// launches that leave places beside them, and so does a norm of rows that are not contiguous.
bool cluster_forms(const nfk_gemm_params& g) {
  return g.rows_kernel != 3 && g.epilogue != NFK_EPI_REDUCE_SCATTER && g.gate_flags == nullptr && g.num_ctas <= 0 && g.smem_budget_kb <= 0 &&
         g.stream_k != 3 && (g.norm_w == nullptr || (g.ldd == g.N && g.norm_ld == g.N));
}

// The split that one launch can do, from the shape that was chosen (or pinned): all tiles at once, since a cluster that waits
// for a place would make a second wave of a product that is one wave long.
SplitPlan split_in_cluster(const nfk_gemm_params& g, const Shape& s) {
  if (!cluster_forms(g) || g.epilogue != NFK_EPI_LINEAR || s.mt != 1 || s.split_k < 2) return SplitPlan{};
  SplitPlan f = split_plan(g.M, g.N, g.K, g.groups > 1 ? g.groups : 1, s.bn, s.cg, s.split_k);
  if (f.stages < 2) return SplitPlan{};
  const int size = s.split_k * s.cg;
  if (f.tiles > (s.cg == 2 ? resident_split_clusters<2>(size) : resident_split_clusters<1>(size))) f.stages = 0;
  return f;
}

template <int CG>
int launch_split(const nfk_gemm_params& g, const SplitPlan& f, cudaStream_t stream) {
  const int groups = g.groups > 1 ? g.groups : 1;
  CUtensorMap tmA, tmB;
  int rc = make_tmap_bf16_2d(&tmA, g.A, g.M, g.K + static_cast<uint64_t>(groups - 1) * g.group_k, g.lda, BM, BK);
  if (rc == NF_OK) rc = make_tmap_bf16_2d(&tmB, g.B, g.N, g.K, g.ldb, f.bn / CG, BK);
  if (rc != NF_OK) return rc;
  SplitParams sp;
  sp.d = dev_params(g, true);
  sp.d.split_k = f.split;
  sp.d.bn = f.bn;
  sp.d.stages = f.stages;
  sp.d.tmem_cols = f.tmem_cols;
  sp.m_groups = f.m_groups;
  sp.kb_per = f.kb_per;
  sp.slice = f.slice;
  sp.early_weights = g.weights_ready;
  if (launch_kernel(early_first(g.early_start), gemm_split_cluster_kernel<CG>, f.tiles * f.split * CG, kGemmThreads, f.smem_bytes, stream,
                    f.split * CG, tmA, tmB, sp) != cudaSuccess) {
    (void)cudaGetLastError();
    return NF_ERR_CUDA;
  }
  return g.norm_w != nullptr ? rmsnorm_rows(g, stream) : NF_OK;
}

template <bool GATED, bool TWO>
int resident_mid_clusters(int size) {
  static int known_dev[kMaxDevices][kSplitMaxCluster + 1] = {};
  const int n = resident_clusters(gemm_mid_rows_kernel<GATED, TWO>, size, known_dev[device_slot()][size]);
  return n > 0 ? n : kResidentClusters[size];
}

template <bool GATED, bool TWO>
int launch_mid_rows(const nfk_gemm_params& g, const MidPlan& f, cudaStream_t stream) {
  CUtensorMap tmW0, tmW1, tmX, tmX2;
  int rc = make_tmap_bf16_2d(&tmW0, g.B, g.N, g.K, g.ldb, GATED ? 64 : 128, BK);
  if (rc != NF_OK) return rc;
  tmW1 = tmW0;
  if (GATED) rc = make_tmap_bf16_2d(&tmW1, g.B2, g.N, g.K, g.ldb, 64, BK);
  if (rc == NF_OK) rc = make_tmap_bf16_2d(&tmX, g.A, g.M, g.K, g.lda, f.nb / 2, BK);
  if (rc != NF_OK) return rc;
  tmX2 = tmX;
  if (TWO) rc = make_tmap_bf16_2d(&tmX2, g.A, g.M, g.K, g.lda, f.nb2 / 2, BK);
  if (rc != NF_OK) return rc;
  (void)resident_mid_clusters<GATED, TWO>(2 * f.split);      // sets the kernel's attributes
  MidParams mp;
  mp.d = dev_params(g, !GATED);
  mp.d.stages = f.stages;
  mp.d.tmem_cols = f.tmem_cols;
  mp.nb = f.nb;
  mp.nb2 = f.nb2;
  mp.tok_tiles = f.tok_tiles;
  mp.split = f.split;
  mp.kb_per = f.kb_per;
  mp.round_tokens = f.round_tokens;
  mp.early_weights = g.weights_ready;
  if (launch_kernel(early_first(g.early_start), gemm_mid_rows_kernel<GATED, TWO>, f.n_tiles * f.tok_tiles * f.split * 2, kGemmThreads,
                    f.smem_bytes, stream, f.split * 2, tmW0, tmW1, tmX, tmX2, mp) != cudaSuccess) {
    (void)cudaGetLastError();
    return NF_ERR_CUDA;
  }
  if (!GATED && g.norm_w != nullptr) return rmsnorm_rows(g, stream);
  return NF_OK;
}

// Whether the few-rows kernel takes this call. Forms that fix how the tile kernel cuts its work (a pinned shape, a CTA or
// shared-memory budget, gated input, reduce-scatter) stay with it, and so do a norm of rows that are not contiguous and a
// caller without a workspace, who gets one sum in the order of k.
bool few_rows_takes(const nfk_gemm_params& g) {
  if (g.rows_kernel >= 2 || g.keep_order != 0 || g.epilogue == NFK_EPI_REDUCE_SCATTER || g.gate_flags != nullptr) return false;
  if (g.num_ctas > 0 || g.smem_budget_kb > 0 || g.stream_k != 0) return false;
  if (g.norm_w != nullptr && (g.ldd != g.N || g.norm_ld != g.N)) return false;
  if (g.rows_kernel == 1) return g.cta_group != 2 || g.groups <= 1;
  if (g.tile_n != 0 || g.tile_m != 0 || g.split_k != 0 || g.cta_group != 0 || g.workspace == nullptr) return false;
  // Measured in a chain with a small kernel between products, cold weights, both kernels fetching weights early (us, tile kernel
  // with its own rule -> this one). What it loses by is the tokens that each CTA stages beside its weights.
  //   Linear: 4096 x 4096 at 64 rows 14.3 -> 13.8, 96 14.5 -> 16.8; 8192 x 8192 at 64 32.6 -> 32.9, 96 31.4 -> 34.0; 32000 x 8192
  //   at 64 89.9 -> 89.1, 96 89.1 -> 93.7; 128256 x 4096 at 48 173 -> 167, 64 171 -> 189.
  //   Gated, all tiles at once (two CTAs on an SM): 14336 x 4096 at 64 rows 46.1 -> 46.9, 112 46.3 -> 51.9, 224 54.8 -> 66.1; 256,
  //   on the other side of the line, 55.5 -> 70.3; 18944 x 3584 at 64 49.7 -> 51.0, 224 57.9 -> 70.3.
  //   Gated, more than one round: 28672 x 8192 at 64 rows 150 -> 156, 112 153 -> 178, 144 183 -> 189, 192 189 -> 234; 22016 x 8192 at
  //   64 126 -> 141, 144 143 -> 168.
  // The lines are from before the tile kernel added its parts of K in a cluster and drained gated tiles without a branch per
  // element (14336 x 4096 at 112 rows then 75 -> 54); as the two kernels are now, all of them would lie at about 64 rows.
  const int groups = g.groups > 1 ? g.groups : 1;
  const bool gated = g.epilogue == NFK_EPI_SWIGLU;
  const int ctas = n_block_count(groups, g.N / groups, gated ? 64 : 128);    // before K is cut
  if (!gated) return g.M <= (g.N > 65536 ? 48 : 8 * ctas < sm_count() ? 64 : 96);
  if (ctas > 2 * sm_count()) return g.M <= 144 && g.M != 128;
  return g.M <= (8 * ctas < sm_count() ? 160 : 255);
}

int few_rows(const nfk_gemm_params& g, cudaStream_t stream) {
  const bool gated = g.epilogue == NFK_EPI_SWIGLU;
  const int groups = g.groups > 1 ? g.groups : 1;
  const FewPlan f = few_rows_plan(g.M, g.N, g.K, gated, groups, groups > 1 ? 1 : g.cta_group, g.split_k);
  if (f.split < 1 || f.split * f.cg > 8 || f.stages < 2) return NF_ERR_BAD_ARG;
  if (gated) return f.cg == 2 ? launch_few_rows<true, 2>(g, f, stream) : launch_few_rows<true, 1>(g, f, stream);
  return f.cg == 2 ? launch_few_rows<false, 2>(g, f, stream) : launch_few_rows<false, 1>(g, f, stream);
}

// Tile-shape choice when the caller leaves it open: a small cost model over the candidate shapes.
// A unit (tile x k range) costs its k-blocks times the per-k-block time of the tile shape (the
// larger of tensor time and shared-memory fill time) plus a fixed prologue/epilogue; the GEMM costs
// waves x unit cost, plus the reduce pass when K is split, and no less than the weight's way from HBM. MT > 1 shapes let
// one CTA cover several M tiles with one weight tile (each weight byte enters shared memory once), which wins when M is
// small and the GEMM is bound by streaming the weight.
//
// The constants (us, bytes, TFLOP/s of one SM) are fitted, with the gated epilogue and the split in a cluster as they are, to
// all candidate shapes of eleven products (4096 to 128256 columns, K 4096 to 28672, three of them gated) at 15 numbers of rows
// from 100 to 1500, by the time of the shape that is taken. Tiles of 224 columns are the best of the gated ones at most sizes.
//
// The earlier constants stay for calls with keep_order, the layer-list models' products: a recurrent layer carries every change
// of rounding into its state and on to the next tokens (logits of a second step moved by up to 0.9 of their size in an element,
// while either order is equally far from 64 bits: 0.0074), so these models keep the order of sums that the earlier shapes give.
struct ShapeModel {
  double mma, fill, least_single, least_pair;                 // TFLOP/s, GB/s of an SM; us per k-block at least
  double uneven, single;                                      // factors: gated tiles of uneven width, single CTAs
  double unit, per_col_single, per_col;                       // us per unit, and per accumulator column
  double reduce, reduce_rate, fix, fix_rate, copy_rate;       // us and TB/s of the second passes; GB/s of a CTA's partial copies
  double weight_rate;                                         // TB/s at which the weight arrives, 0 = no bound
  double tail_gain;                                           // a stream-K tail has to be below this share of the best without
  double cluster, cluster_col;                                // us, and per column sent, where parts meet in a cluster; 0 = as two launches
};
constexpr ShapeModel kModel{9.883, 129.2, 0.331, 0.295, 0.966, 1.095, 0.868, 0.0117, 0.00119, 7.28, 2.70, 2.47, 1.325, 177.0, 6.38, 1.0, 4.04, 0.01045};
constexpr ShapeModel kEarlierModel{11.0, 100.0, 0.0, 0.36, 1.0, 1.0, 2.0, 0.012, 0.003, 3.0, 4.0, 3.0, 3.0, 150.0, 0.0, 0.88, 0.0, 0.0};
// What one shape costs by the model, without a stream-K tail.
struct TileCost {
  double t_kb, unit_fixed, us;      // per k-block, per unit, the whole product
  int tiles, workers, mt_eff;
};
double weight_bound(const ShapeModel& m, const nfk_gemm_params& g, bool swiglu, double us) {
  if (m.weight_rate <= 0.0) return us;
  const double w = static_cast<double>(g.N) * g.K * (swiglu ? 4.0 : 2.0) / (m.weight_rate * 1e6) + 0.25 * us;
  return w > us ? w : us;
}
TileCost tile_cost(const ShapeModel& m, const nfk_gemm_params& g, bool swiglu, int bn, int mt, int sk, int cg) {
  TileCost c;
  const int ctas = g.num_ctas > 0 ? g.num_ctas : sm_count(), groups = g.groups > 1 ? g.groups : 1;
  const int m_tiles = (g.M + BM - 1) / BM, num_kb = (g.K + BK - 1) / BK;
  const int m_groups = (m_tiles + mt * cg - 1) / (mt * cg);
  c.tiles = m_groups * n_block_count(groups, g.N / groups, swiglu ? bn / 2 : bn);
  c.mt_eff = m_tiles < mt ? m_tiles : mt;
  // per k-block and SM (a CTA of a pair stages only half of the weight tile)
  const double t_mma = 2.0 * BM * c.mt_eff * bn * BK / (m.mma * 1e6);
  const double t_fill = (c.mt_eff * 16384.0 + bn * 128.0 / cg) / (m.fill * 1e3);
  c.t_kb = t_mma > t_fill ? t_mma : t_fill;
  const double t_least = cg == 2 ? m.least_pair : m.least_single;
  if (c.t_kb < t_least) c.t_kb = t_least;
  if (swiglu && bn % 64 != 0) c.t_kb *= m.uneven;
  if (cg == 1) c.t_kb *= m.single;
  // per unit: prologue + epilogue; the epilogue hides under the next main loop only when TMEM
  // holds two accumulator sets
  const bool single_acc = mt * bn * 2 > 512;
  c.unit_fixed = m.unit + (single_acc ? m.per_col_single : m.per_col) * c.mt_eff * bn;
  c.workers = ctas / cg > 0 ? ctas / cg : 1;
  const int units = c.tiles * sk, kb_per = (num_kb + sk - 1) / sk;
  double us = ((units + c.workers - 1) / c.workers) * (kb_per * c.t_kb + c.unit_fixed);
  if (sk > 1) {
    if (m.cluster > 0.0 && cluster_forms(g) && mt == 1 && sk * cg <= kSplitMaxCluster &&
        c.tiles <= (cg == 2 ? resident_split_clusters<2>(sk * cg) : resident_split_clusters<1>(sk * cg)))
      us += m.cluster + m.cluster_col * bn * (sk - 1) / sk;
    else
      us += m.reduce + (sk + 1.0) * g.M * static_cast<double>(g.N) * 4.0 / (m.reduce_rate * 1e6);  // partial write + reduce
  }
  c.us = weight_bound(m, g, swiglu, us);
  return c;
}

Shape search_shape(const nfk_gemm_params& g, bool swiglu) {
  const ShapeModel& m = g.keep_order != 0 ? kEarlierModel : kModel;
  const int m_tiles = (g.M + BM - 1) / BM, num_kb = (g.K + BK - 1) / BK;
  Shape best{256, 1, 1, 1, false}, best_tail{256, 1, 1, 1, true};
  double best_cost = 1e30, best_tail_cost = 1e30;
  const int cg_lo = g.cta_group == 2 ? 2 : 1, cg_hi = g.cta_group == 1 ? 1 : 2;
  for (int cg = cg_lo; cg <= cg_hi; ++cg) {
    for (int mt = 1; mt <= (cg == 2 ? 1 : 4); mt *= 2) {
      for (int bn = swiglu ? 128 : 64; bn <= 256; bn += 32) {
        if (mt * bn > 512) continue;
        if (swiglu && (bn / 2) % 16 != 0) continue;
        // Several M tiles per CTA only pay off when M is small (weight streaming); with many M tiles
        // the single TMEM accumulator set would serialise epilogue and main loop for nothing.
        if (mt > 1 && (m_tiles > 4 || m_tiles <= mt / 2)) continue;
        if (cg == 2 && m_tiles < 2) continue;    // a pair covers two M tiles
        const int max_sk = (swiglu || g.workspace == nullptr || g.epilogue == NFK_EPI_REDUCE_SCATTER) ? 1 : 8;
        for (int sk = 1; sk <= max_sk; ++sk) {
          if (sk > 1 && (num_kb / sk < 8 || static_cast<long long>(sk) * g.M * g.N * 4 > g.workspace_bytes)) break;
          const TileCost c = tile_cost(m, g, swiglu, bn, mt, sk, cg);
          if (c.us < best_cost) {
            best_cost = c.us;
            best = Shape{bn, mt, sk, cg, false};
          }
          // the same shape with a stream-K tail: full waves as above, then one round of k ranges whose
          // pieces are written out as fp32 and summed by a second pass
          if (sk == 1 && g.stream_k < 2 && g.workspace != nullptr && g.epilogue != NFK_EPI_REDUCE_SCATTER) {
            const SkPlan pl = plan_stream_k(c.tiles, c.workers, num_kb);
            const long long need = static_cast<long long>(pl.rest) * pl.max_pieces * cg * mt * BM * bn * 4;
            if (pl.q > 0 && need <= g.workspace_bytes) {
              const double tile_bytes = c.mt_eff * BM * bn * 4.0;          // one fp32 copy of a CTA's tile rows
              const double pieces = static_cast<double>(num_kb) / pl.q + 1.0;
              // a worker's range may straddle two tiles
              const double fix_us = m.fix + pl.rest * cg * pieces * tile_bytes / (m.fix_rate * 1e6);
              const double tail = pl.q * c.t_kb + 2.0 * c.unit_fixed + tile_bytes / (m.copy_rate * 1e3) + fix_us;
              const double c2 = weight_bound(m, g, swiglu, (c.tiles / c.workers) * (num_kb * c.t_kb + c.unit_fixed) + tail);
              if (c2 < best_tail_cost) {
                best_tail_cost = c2;
                best_tail = Shape{bn, mt, 1, cg, true};
              }
            }
          }
        }
      }
    }
  }
  const bool tail = (g.stream_k == 1 && best_tail_cost < 1e30) || best_tail_cost < m.tail_gain * best_cost;
  Shape s = tail ? best_tail : best;
  // What kModel says of a shape that the earlier one has chosen. Four M tiles of 128 columns, which it does not choose itself, take
  // 1.55 times that: 32000 x 8192 at 300 rows 295 us, said 189; 128256 x 4096 555, said 350.
  s.us = g.keep_order == 0 ? (tail ? best_tail_cost : best_cost)
                           : tile_cost(kModel, g, swiglu, s.bn, s.mt, s.split_k, s.cg).us * (s.mt == 4 ? 1.55 : 1.0);
  return s;
}

// The search looks at some 200 shapes, 4 us of a launch's host time, and the layers of an iteration ask for the same few
// products: a thread keeps the answers to its last questions, by everything that the search reads (sizes and forms, no address).
Shape choose_shape(const nfk_gemm_params& g, bool swiglu) {
  constexpr int kKept = 16;
  struct Question {
    long long workspace;
    int M, N, K, groups, num_ctas, cta_group, stream_k, device, forms;
    bool operator==(const Question& o) const {
      return workspace == o.workspace && M == o.M && N == o.N && K == o.K && groups == o.groups && num_ctas == o.num_ctas &&
             cta_group == o.cta_group && stream_k == o.stream_k && device == o.device && forms == o.forms;
    }
  };
  struct Kept {
    Question q;
    Shape s;
  };
  thread_local Kept kept[kKept];
  thread_local int n = 0, next = 0;
  const Question q{g.workspace != nullptr ? g.workspace_bytes : -1, g.M, g.N, g.K, g.groups, g.num_ctas, g.cta_group, g.stream_k, device_slot(),
                   (swiglu ? 1 : 0) | (g.keep_order != 0 ? 2 : 0) | (g.epilogue == NFK_EPI_REDUCE_SCATTER ? 4 : 0) | (cluster_forms(g) ? 8 : 0)};
  for (int i = 0; i < n; ++i)
    if (kept[i].q == q) return kept[i].s;
  const Shape s = search_shape(g, swiglu);
  kept[next] = Kept{q, s};
  next = (next + 1) % kKept;
  if (n < kKept) ++n;
  return s;
}

// us of `tiles` tiles of the mid-rows kernel at once, one to a cluster.
double mid_rows_round(const MidPlan& f, int cols, int tiles) {
  const double pairs = static_cast<double>(tiles) * f.split;
  const double pair_us = 1.33e-3 * cols;                                            // a pair's products, per k-block
  const double chip_us = pairs * cols * (2.0 * 256 * BK) / 1.42e9;                  // those of all pairs under the power limit: 1.42 PFLOP/s
  const double weight_us = 0.0964 + pairs * 2.0 * kFewWBytes / f.tok_tiles / 8.6e6;    // the weights' way from HBM
  return f.kb_per * std::max(std::max(pair_us, chip_us), weight_us) + 3.38 + 0.026 * cols;    // set-up; a token's way out
}

// Whether the mid-rows kernel takes a call for which the tile kernel would have shape `s`, and with how many parts of K (stages
// 0: it does not). rows_kernel 4 asks for it with split_k parts.
//
// The line is drawn by the two kernels' models; 8 % are in hand for their errors, and the tile kernel's counts 2.4 us less of
// what a product costs beside its loop. K is cut only where all tiles run at once (a second round of clusters starts late:
// 28672 x 2 x 8192 at 333 rows 328 us in two parts, 318 in one, tile kernel 278). The constants are those that choose best over
// 21 products (2048 to 128256 columns, K 2048 to 28672, five of them gated) at 30 numbers of rows from 64 to 1100, in a chain of
// products with cold weights, with the residual in place where a model has one, and over ten of them with the order kept and
// without a workspace. Beside the fastest of both kernels the choice is 0.2 % slower on average; 13 of 916 are more than 5 % behind,
// at worst 20 % (2048 x 8192 at 700 rows in the kept order's three parts: 33.4 us, tile kernel 27.9; 5120 x 5120 at 97 rows, which the
// tile kernel gets: 18.8, here 16.5). With no limit on the products of all pairs together it was 1.9 % and 29 %, up to 23 % slower
// than without this kernel.
// us, tile kernel -> this one where it is taken: 8192 x 28672 at 160 rows 99 -> 87, 288 156 -> 114, 384 161 -> 144, 576 257 -> 222;
// 8192 x 8192 at 160 37 -> 33, 288 51 -> 41, 576 81 -> 66; 4096 x 14336 at 288 45 -> 39, 576 70 -> 58; 32000 x 8192 at 288 152 -> 139;
// 18944 x 2 x 3584 at 288 84 -> 77. On the other side of the line: 8192 x 28672 at 256 rows 108 (here 112), 512 176 (188), 1000 325
// (370); 4096 x 4096 at 333 19 (24); 10240 x 8192 at 160 42 (44); 32000 x 8192 at 333 155 (168), 896 337 (377); 14336 x 2 x 4096 at 256
// 56 (74), 333 77 (90); 28672 x 2 x 8192 at 288 272 (274), 896 596 (781).
// Fewer rows come here where the few-rows kernel does not take them. Without a workspace (one sum in the order of k) 4096 x 4096
// at 8 rows 26.3 -> 19.5, 96 22.0 -> 21.1, 128 22.2 -> 21.9; 4096 x 14336 at 64 60.4 -> 51.4; from 129 to 256, where the tile kernel
// works in pairs of 256 rows, it stays: 160 20.2 (here 23.1), 4096 x 14336 51.4 (54.1). With keep_order 128256 x 4096 at 16
// rows stays (166; here 193).
//
// With keep_order K stays cut as the tile kernel's shape cuts it, which gives the same bits.
MidPlan mid_rows_takes(const nfk_gemm_params& g, const Shape& s) {
  const bool gated = g.epilogue == NFK_EPI_SWIGLU;
  if (!cluster_forms(g) || g.groups > 1) return MidPlan{};
  if (g.rows_kernel != 4 && (g.rows_kernel != 0 || g.M > 1024 || g.tile_n != 0 || g.tile_m != 0 || g.split_k != 0 || g.cta_group != 0 ||
                             g.stream_k != 0 || (g.keep_order != 0 && s.stream_k) || (g.workspace == nullptr && g.M > 128 && g.M <= 256)))
    return MidPlan{};
  MidPlan best{};
  double best_us = g.rows_kernel == 4 ? 1e30 : 0.92 * s.us + 2.4;
  const int lo = g.rows_kernel == 4 ? (g.split_k > 0 ? g.split_k : 1) : g.keep_order != 0 ? s.split_k : 1;
  const int hi = g.rows_kernel == 4 || g.keep_order != 0 ? lo : g.workspace == nullptr ? 1 : 4;   // without a workspace: one sum in the order of k
  for (int split = lo; split <= hi; ++split) {
    const MidPlan f = mid_rows_plan(g.M, g.N, g.K, gated, split);
    if (f.stages < 2 || f.round_tokens < 32) continue;
    const int fit = f.nb2 > 0 ? (gated ? resident_mid_clusters<true, true>(2 * split) : resident_mid_clusters<false, true>(2 * split))
                              : (gated ? resident_mid_clusters<true, false>(2 * split) : resident_mid_clusters<false, false>(2 * split));
    const int tiles = f.n_tiles * f.tok_tiles, cols = f.nb + f.nb2;
    if (g.rows_kernel != 4 && split > 1 && tiles > fit) continue;
    const double us = (tiles / fit) * mid_rows_round(f, cols, fit) + (tiles % fit != 0 ? mid_rows_round(f, cols, tiles % fit) : 0.0);
    if (us < best_us) {
      best_us = us;
      best = f;
    }
  }
  return best;
}

// A shape measured at another number of rows (tuned_rows) says little about this call: it holds for calls with as many
// 256-row groups of tiles, and the rules choose for the others. A shape tuned at 1024 rows took 50 us for 48 x 10240 x 8192,
// where the weight takes 26. Up to 256 rows that is too coarse: a shape holds for as many tiles of 128 rows, and only where
// the rules would not take the few-rows kernel, unless it was measured at exactly this number of rows.
//
// With keep_order a stopwatch must not decide where K is cut: a pick changes with the clock of the day, and the order of sums
// with it. Shapes that leave K whole all add up in the order of k, so a tuned one of them takes the place of a whole-K shape of
// the cost model; where the model cuts K for this M, or the tuned shape does, the model's shape stands.
nfk_gemm_params with_own_shape(const nfk_gemm_params& g) {
  nfk_gemm_params p = g;
  if (g.tuned_rows <= 0) return p;
  p.tile_m = p.tile_n = p.cta_group = p.split_k = p.stream_k = 0;
  if ((g.M + 255) / 256 != (g.tuned_rows + 255) / 256) return p;
  if (g.M <= 256 && g.M != g.tuned_rows && ((g.M + BM - 1) / BM != (g.tuned_rows + BM - 1) / BM || few_rows_takes(p))) return p;
  if (g.keep_order != 0) {
    const Shape own = choose_shape(p, g.epilogue == NFK_EPI_SWIGLU);
    if (own.split_k > 1 || own.stream_k || g.split_k > 1 || g.stream_k == 1) return p;
  }
  return g;
}

// Shape of this call: the cost model's, or the caller's pinned one, checked against what is built.
int resolve_shape(const nfk_gemm_params& gp, bool swiglu, bool rs, Shape& s) {
  const nfk_gemm_params* g = &gp;
  s = choose_shape(*g, swiglu);
  if (rs) s.split_k = 1;   // partial tiles go straight to their owners: no K split
  if (g->gate_flags != nullptr) {
    s.split_k = 1;         // gated input: whole tiles in row order only
    s.stream_k = false;
  }
  if (g->tile_n != 0 || g->tile_m != 0) {
    // pinned tile shape: fill in the other dimension with its default, split only on request
    s.bn = g->tile_n != 0 ? g->tile_n : 256;
    s.mt = g->tile_m != 0 ? g->tile_m : 1;
    s.split_k = 1;
    s.cg = g->cta_group == 2 ? 2 : 1;
    s.stream_k = false;
  }
  if (g->stream_k == 1) s.stream_k = true;
  if (g->stream_k >= 2 || s.split_k != 1 || g->gate_flags != nullptr) s.stream_k = false;
  if (s.cg == 2 && s.mt != 1) return NF_ERR_UNSUPPORTED;
  if (g->split_k != 0 && g->gate_flags == nullptr) s.split_k = g->split_k;
  if (s.split_k < 1 || s.split_k > 16) return NF_ERR_BAD_ARG;
  if (s.split_k > 1) {
    if (swiglu || g->workspace == nullptr ||
        static_cast<long long>(s.split_k) * g->M * g->N * 4 > g->workspace_bytes)
      return NF_ERR_BAD_ARG;
  }
  // Wider than one MMA instruction (256 columns): CTA pairs, one M tile, plain epilogue (the WIDE kernel).
  const bool wide_ok = s.bn > 256 && s.bn <= 512 && s.bn % 64 == 0 && s.cg == 2 && s.mt == 1 && !swiglu && !rs;
  if (s.bn < 32 || (s.bn > 256 && !wide_ok) || s.bn % 32 != 0 || (s.mt != 1 && s.mt != 2 && s.mt != 4) || s.mt * s.bn > 512)
    return NF_ERR_UNSUPPORTED;
  if (swiglu && (s.bn / 2) % 16 != 0) return NF_ERR_UNSUPPORTED;
  return NF_OK;
}

}  // namespace
}  // namespace nf

// What the tile kernel of nfk_gemm_bf16 would launch for these parameters, without launching: tile shape, number of
// tiles and workers, and the stream-K tail (first tile of the tail region, k-blocks per worker, most
// pieces a tile can be cut into). Needs no GPU (the SM count falls back to 148), so planners and
// tests can check the work distribution on any machine.
extern "C" int nfk_gemm_describe(const nfk_gemm_params* given, nfk_gemm_plan* out) {
  using namespace nf;
  if (given == nullptr || out == nullptr || given->M <= 0 || given->N <= 0 || given->K <= 0) return NF_ERR_BAD_ARG;
  const nfk_gemm_params own = with_own_shape(*given), *g = &own;
  const bool swiglu = g->epilogue == NFK_EPI_SWIGLU, rs = g->epilogue == NFK_EPI_REDUCE_SCATTER;
  Shape s;
  const int rc = resolve_shape(*g, swiglu, rs, s);
  if (rc != NF_OK) return rc;
  int budget = g->smem_budget_kb > 0 ? g->smem_budget_kb * 1024 : kSmemMax;
  if (budget > kSmemMax) budget = kSmemMax;
  const Geom geo = make_geom(s.bn, s.mt, swiglu, budget, s.cg, (rs && g->rs_staged) ? kRsStageBytes : 0);
  if (geo.stages < 2) return NF_ERR_BAD_ARG;
  const int m_tiles = (g->M + BM - 1) / BM;
  const int m_groups = (m_tiles + s.mt * s.cg - 1) / (s.mt * s.cg);
  const int n_blocks = n_block_count(g->groups > 1 ? g->groups : 1, g->N / (g->groups > 1 ? g->groups : 1), geo.out_bn);
  const int tiles = m_groups * n_blocks;
  int workers = (g->num_ctas > 0 ? g->num_ctas : sm_count()) / s.cg;
  if (workers > sm_count() / s.cg) workers = sm_count() / s.cg;
  if (workers < 1) workers = 1;
  SkPlan sk{tiles, 0, 0, 0};
  if (s.stream_k && s.split_k == 1 && !rs && g->workspace != nullptr) {
    sk = plan_stream_k(tiles, workers, (g->K + BK - 1) / BK);
    const long long need = static_cast<long long>(sk.rest) * sk.max_pieces * s.cg * s.mt * BM * s.bn * 4;
    if (sk.q > 0 && need > g->workspace_bytes) sk = SkPlan{tiles, 0, 0, 0};
  }
  if (sk.q == 0 && workers > tiles * s.split_k) workers = tiles * s.split_k;
  out->tile_n = s.bn;
  out->tile_m = s.mt;
  out->cta_group = s.cg;
  out->split_k = s.split_k;
  out->stream_k = sk.q > 0 ? 1 : 0;
  out->tiles = tiles;
  out->workers = workers;
  out->num_kb = (g->K + BK - 1) / BK;
  out->tail_first_tile = sk.tiles_dp;
  out->tail_range_kb = sk.q;
  out->tail_max_pieces = sk.max_pieces;
  out->stages = geo.stages;
  out->smem_bytes = geo.smem_bytes;
  out->few_rows = few_rows_takes(*g) ? 1 : 0;
  const MidPlan mid = out->few_rows != 0 ? MidPlan{} : mid_rows_takes(*g, s);
  out->mid_rows = mid.stages >= 2 ? mid.split : 0;
  const SplitPlan split = out->few_rows != 0 || out->mid_rows != 0 ? SplitPlan{} : split_in_cluster(*g, s);
  out->cluster_parts = split.stages >= 2 ? split.split : 0;
  return NF_OK;
}

extern "C" int nfk_gemm_bf16(const nfk_gemm_params* given, cudaStream_t stream) {
  using namespace nf;
  if (given == nullptr) return NF_ERR_BAD_ARG;
  const nfk_gemm_params own = with_own_shape(*given), *g = &own;
  if (g->M == 0 && g->epilogue == NFK_EPI_REDUCE_SCATTER) {
    if (g->rs_nranks < 1 || g->rs_nranks > 8 || g->rs_rank < 0 || g->rs_rank >= g->rs_nranks) return NF_ERR_BAD_ARG;
    DevParams p{};
    for (int r = 0; r < 8; ++r) p.rs_heap[r] = reinterpret_cast<char*>(g->rs_heap[r]);
    p.rs_rank = g->rs_rank;
    p.rs_nranks = g->rs_nranks;
    p.rs_epoch = g->rs_epoch;
    p.rs_flag_off = g->rs_flag_off;
    rs_signal_only_kernel<<<1, 32, 0, stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? NF_OK : NF_ERR_CUDA;
  }
  if (g->M == 0 || g->N == 0) return NF_OK;  // empty nano-batch: nothing to do
  if (g->A == nullptr || g->B == nullptr) return NF_ERR_BAD_ARG;
  if (g->D == nullptr && g->epilogue != NFK_EPI_REDUCE_SCATTER && !(g->D32 != nullptr && g->f32_col0 == 0))
    return NF_ERR_BAD_ARG;
  if (g->D32 != nullptr &&
      (g->epilogue != NFK_EPI_LINEAR || g->f32_col0 < 0 || g->f32_col0 % 8 != 0 || g->ld32 % 4 != 0 ||
       (reinterpret_cast<uintptr_t>(g->D32) & 15) != 0 || g->norm_w != nullptr))
    return NF_ERR_BAD_ARG;
  if (g->act < NFK_ACT_SILU || g->act > NFK_ACT_CAPPED || g->lin_act < NFK_LIN_NONE || g->lin_act > NFK_LIN_RELU2) return NF_ERR_BAD_ARG;
  if (g->groups > 1 && (g->epilogue != NFK_EPI_LINEAR || g->N % (8 * g->groups) != 0 || g->group_k % 8 != 0 ||
                        g->group_k < 0 || g->gate_flags != nullptr))
    return NF_ERR_BAD_ARG;
  if (g->M < 0 || g->N < 0 || g->K <= 0) return NF_ERR_BAD_ARG;
  if (g->K % 8 != 0 || g->N % 8 != 0 || g->lda % 8 != 0 || g->ldb % 8 != 0 || g->ldd % 8 != 0)
    return NF_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(g->D) & 15) != 0) return NF_ERR_BAD_ARG;
  if (g->C != nullptr && ((reinterpret_cast<uintptr_t>(g->C) & 15) != 0 || g->ldc % 8 != 0))
    return NF_ERR_BAD_ARG;
  if (g->workspace != nullptr && (reinterpret_cast<uintptr_t>(g->workspace) & 15) != 0) return NF_ERR_BAD_ARG;
  const bool swiglu = g->epilogue == NFK_EPI_SWIGLU;
  if (swiglu && (g->B2 == nullptr || (g->bias == nullptr) != (g->bias2 == nullptr))) return NF_ERR_BAD_ARG;
  const bool rs = g->epilogue == NFK_EPI_REDUCE_SCATTER;
  if (g->gate_flags != nullptr &&
      (rs || g->gate_nranks < 1 || g->gate_nranks > 8 || (reinterpret_cast<uintptr_t>(g->gate_flags) & 3) != 0))
    return NF_ERR_BAD_ARG;
  if (rs) {
    if (g->rs_nranks < 1 || g->rs_nranks > 8 || g->rs_rank < 0 || g->rs_rank >= g->rs_nranks ||
        g->rs_rows_cap * g->rs_nranks < g->M || g->rs_slab_off % 16 != 0 || g->rs_flag_off % 16 != 0 ||
        g->split_k > 1)
      return NF_ERR_BAD_ARG;
    for (int r = 0; r < g->rs_nranks; ++r)
      if (g->rs_heap[r] == nullptr) return NF_ERR_BAD_ARG;
  }

  if (few_rows_takes(*g)) return few_rows(*g, stream);
  Shape s;
  if (g->rows_kernel != 4) {
    const int rcs = resolve_shape(*g, swiglu, rs, s);
    if (rcs != NF_OK) return rcs;
  }
  const MidPlan mid = mid_rows_takes(*g, s);
  if (mid.stages >= 2) {
    if (mid.nb2 > 0) return swiglu ? launch_mid_rows<true, true>(*g, mid, stream) : launch_mid_rows<false, true>(*g, mid, stream);
    return swiglu ? launch_mid_rows<true, false>(*g, mid, stream) : launch_mid_rows<false, false>(*g, mid, stream);
  }
  if (g->rows_kernel == 4) return NF_ERR_UNSUPPORTED;
  if (swiglu) {
    if ((s.bn / 2) % 16 != 0) return NF_ERR_UNSUPPORTED;
    if (g->bias != nullptr) return launch_mt<kGatedBias>(*g, s.bn, s.mt, s.cg, 1, s.stream_k, stream);
    return launch_mt<1>(*g, s.bn, s.mt, s.cg, 1, s.stream_k, stream);
  }
  if (rs) return launch_mt<2>(*g, s.bn, s.mt, s.cg, 1, false, stream);
  const SplitPlan f = split_in_cluster(*g, s);
  if (f.stages >= 2) return s.cg == 2 ? launch_split<2>(*g, f, stream) : launch_split<1>(*g, f, stream);
  return launch_mt<0>(*g, s.bn, s.mt, s.cg, s.split_k, s.stream_k, stream);
}
