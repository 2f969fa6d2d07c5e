// Shared device/host helpers for the sm_100a kernels: error codes, a status word that bounded
// waits report into, PTX wrappers for mbarrier / TMA / tcgen05 / TMEM, and small vector utilities.
//
// Every spin in this library (mbarrier waits, flag polls on peer memory) is bounded. When a bound
// runs out the waiting thread records a code in the kernel's status word and the kernel unwinds:
// roles stop issuing work, the CTA re-converges, TMEM is released, and the host reads the status
// word after the launch. Nothing here traps or loops forever.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"

namespace nf {

// ---- host-visible error codes (returned by every extern "C" launcher) -------------------------
enum : int {
  NF_OK = 0,
  NF_ERR_BAD_ARG = 1,      // shape / alignment / size limit violated; nothing was launched
  NF_ERR_CUDA = 2,         // a CUDA runtime / driver call failed
  NF_ERR_UNSUPPORTED = 3,  // combination not built
};

// ---- device status word values -----------------------------------------------------------------
enum : unsigned int {
  NF_ST_OK = 0,
  NF_ST_TIMEOUT_SMEM_FULL = 0x100,   // consumer gave up waiting for a TMA stage
  NF_ST_TIMEOUT_SMEM_EMPTY = 0x200,  // producer gave up waiting for a free stage
  NF_ST_TIMEOUT_TMEM_FULL = 0x300,   // epilogue gave up waiting for an accumulator
  NF_ST_TIMEOUT_TMEM_EMPTY = 0x400,  // MMA issuer gave up waiting for a free accumulator
  NF_ST_TIMEOUT_PEER_FLAG = 0x500,   // a wait on a flag written by another rank ran out
  NF_ST_TIMEOUT_GRID_BARRIER = 0x600,
  NF_ST_BAD_INDEX = 0x700,           // a page / token index was out of range and was skipped
};

#ifdef __CUDACC__

#define NF_DEVICE __device__ __forceinline__

// Upper bound on mbarrier.try_wait attempts. Each attempt may sleep for a hardware-chosen time
// slice, so the wall-clock bound is of the order of a second.
static constexpr uint32_t kMbarSpinLimit = 1u << 22;

NF_DEVICE uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier ----------------------------------------------------------------------------------
NF_DEVICE void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
NF_DEVICE void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
NF_DEVICE void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
NF_DEVICE void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait. Returns false when the bound ran out (the caller must unwind).
NF_DEVICE bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < kMbarSpinLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Wait of a role of a persistent kernel: bounded by wall clock (globaltimer) and by the CTA abort flag.
NF_DEVICE bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t addr = smem_u32(bar);
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 255u) == 255u) {
      if (*abort_flag) return false;
      uint64_t now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      if (now - t0 > 2000000000ull || it > (1u << 30)) return false;  // 2 s
    }
  }
}

// One lane of a converged warp, known to the compiler as one: tcgen05 and TMA instructions take their operands from the
// warp's uniform registers, and inside `if (lane == 0)` every operand costs moves that an elected lane does not pay.
NF_DEVICE bool elect_one() {
  uint32_t on;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(on));
  return on != 0;
}

NF_DEVICE void report_status(unsigned int* status, unsigned int code) {
  if (status != nullptr) atomicCAS(status, 0u, code);
}

// ---- TMA (non-multicast only) --------------------------------------------------------------------
NF_DEVICE void tma_prefetch_desc(const CUtensorMap* tm) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tm)) : "memory");
}
NF_DEVICE void tma_load_2d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// Untiled bulk copy shared -> global (both addresses 16-byte aligned, size a multiple of 16 bytes),
// tracked by the issuing thread's bulk group like a tensor store.
NF_DEVICE void bulk_store_1d(void* gmem_dst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem_dst),
               "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
NF_DEVICE void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
NF_DEVICE void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
NF_DEVICE void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
NF_DEVICE void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- tcgen05 / TMEM -----------------------------------------------------------------------------
NF_DEVICE void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
NF_DEVICE void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
NF_DEVICE void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
NF_DEVICE void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
NF_DEVICE void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// One thread issues; D[tmem] (+)= A[smem desc] * B[smem desc].
NF_DEVICE void umma_bf16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with A in tensor memory (128 lanes = rows, each 32-bit column two consecutive k elements):
// D[tmem] (+)= A[tmem] * B[smem desc].
NF_DEVICE void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives once on `bar` when every tcgen05.mma issued so far by this thread has completed.
NF_DEVICE void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread t of the warp receives lane (base_lane + t).
NF_DEVICE void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 16 consecutive fp32 columns (tail chunk of tiles whose width is not a multiple of 32).
NF_DEVICE void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 16; i < 32; ++i) r[i] = 0u;
}
// 32 lanes x 16 consecutive fp32 columns into 16 registers.
NF_DEVICE void tmem_ld_32x32b_x16n(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
NF_DEVICE void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Registers -> TMEM, same shape as the x32 load: thread t writes lane (base_lane + t), 32 columns.
NF_DEVICE void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
      "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
NF_DEVICE void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- CTA pairs (cta_group::2): two CTAs of a 2-CTA cluster work on one 256-row tile --------------
// Each CTA stages its own 128 rows of A and half of the B tile; the even CTA issues the MMAs, which
// read both CTAs' shared memory and write 128 accumulator rows into each CTA's TMEM.
NF_DEVICE uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
NF_DEVICE uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
NF_DEVICE void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
NF_DEVICE void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
NF_DEVICE void st_shared_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
NF_DEVICE void st_shared_cluster_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// TMA load into this CTA's shared memory whose byte count is reported to a barrier that may live in
// the peer CTA (`bar_cluster_addr` from mapa_shared). No multicast: each CTA fetches its own tiles.
NF_DEVICE void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tm, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
NF_DEVICE void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
NF_DEVICE void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
NF_DEVICE void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
NF_DEVICE void umma_bf16_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives once on the barrier at `bar`'s offset in the CTAs of `mask` (both CTAs of the pair) when every pair MMA
// issued so far by this thread has completed.
NF_DEVICE void umma_commit_pair_mask(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)), "h"(mask)
      : "memory");
}
NF_DEVICE void umma_commit_pair_both(uint64_t* bar) { umma_commit_pair_mask(bar, 3); }

// Shared-memory matrix descriptor for a K-major tile stored with the 128-byte swizzle that TMA
// SWIZZLE_128B produces: rows of 128 bytes, 8-row groups 1024 bytes apart.
NF_DEVICE uint64_t umma_desc_k_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);        // start address
  d |= static_cast<uint64_t>(1) << 16;                            // leading byte offset (unused)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                    // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;                            // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                            // SWIZZLE_128B
  return d;
}
// Instruction descriptor: bf16 x bf16 -> fp32, both operands K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

// ---- launches that overlap the end of the kernel before them ------------------------------------------
// A kernel launched early (launch_kernel) may start while the kernel before it on the stream still runs, as soon as every
// CTA of that one has called let_next_start() (or has ended). await_previous() returns when all earlier work is complete and
// visible; every CTA calls it before its first access to memory that earlier work writes or reads, and no CTA ends
// without having called it, so that completion stays transitive along a stream. A kernel that allocates tensor memory
// calls let_next_start() after that: the next kernel cannot then take columns that it still needs. A kernel that waits for
// flags which another stream's or another GPU's kernel raises never calls it.
//
// Who launches early is the graph's choice (early_start of an op's parameters): CTAs that have started early hold threads,
// registers and shared memory of their SM while they wait, and where another stream's kernel is to run beside the one that
// they wait for, those are its places (a GEMM of 192 threads with four waiting CTAs of the rotary kernel, 256 threads each,
// leaves no registers for a collective's CTA).
NF_DEVICE void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
NF_DEVICE void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- misc -----------------------------------------------------------------------------------------
NF_DEVICE float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
NF_DEVICE uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
NF_DEVICE float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

#endif  // __CUDACC__

#ifdef __CUDACC__
inline bool early_first(int early_start) { return (early_start & NFK_EARLY_FIRST) != 0; }
inline bool early_further(int early_start) { return (early_start & NFK_EARLY_FURTHER) != 0; }
// kernel<<<grid, block, smem, stream>>>(args...) in clusters of `cluster` CTAs; `early`: see let_next_start.
template <class... P, class... A>
inline cudaError_t launch_kernel(bool early, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, int cluster,
                                 A... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(grid);
  lc.blockDim = dim3(block);
  lc.dynamicSmemBytes = smem;
  lc.stream = stream;
  cudaLaunchAttribute la[2];
  lc.attrs = la;
  lc.numAttrs = 0;
  if (early) {
    cudaLaunchAttribute& a = la[lc.numAttrs++];
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    cudaLaunchAttribute& a = la[lc.numAttrs++];
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = cluster;
    a.val.clusterDim.y = 1;
    a.val.clusterDim.z = 1;
  }
  return cudaLaunchKernelEx(&lc, kernel, static_cast<P>(args)...);
}
#endif

// ---- host: facts about the current device, asked once per device ----------------------------------
// Number of SMs of the current device (grids are sized from it). Falls back to a B200's 148 when no
// device can be asked (planning calls on a machine without a GPU).
int device_sm_count();
// Slot of the current device in per-device caches (0 when there is no device); kMaxDevices slots.
constexpr int kMaxDevices = 64;
int device_slot();

// ---- host: driver entry point for tensor-map encoding (no link-time libcuda dependency) -----------
typedef CUresult (*nf_encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                       const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                       const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
nf_encode_tiled_fn get_encode_tiled();

// Row-major bf16 matrix [rows, cols] with leading dimension ld (elements); box = box_rows x 64
// columns, 128-byte swizzle. Returns NF_OK or an error code.
int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols,
                      uint64_t ld, uint32_t box_rows, uint32_t box_cols);

}  // namespace nf
