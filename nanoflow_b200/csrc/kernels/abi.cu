// Uniform launch ABI: thin `int fn(const params*, cudaStream_t)` forms of the entry points that take
// scalar arguments, so an executor can store (function pointer, parameter block) pairs and replay
// them without knowing any kernel's signature.
#include "common.cuh"
#include "kernels.h"

using namespace nf;

namespace {

// What bounds it is the latency of the host link, a microsecond or two per read, so every thread has its 16 bytes on their way at
// once. The copies of an iteration (two to the device, two back, 3 to 8 us each as nodes of its graph with 2 to 6 us between
// them) became two launches: one request's iteration 682 -> 653 us with the merge in the decode attention, 96 Volarax requests
// 1321 -> 1303, a prompt of 333 tokens 1139 -> 1132.
__device__ __forceinline__ void copy_words(int* dst, const int* src, int count, int at, int step) {
  const bool wide = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0;
  const int whole = wide ? count / 4 : 0;
  for (int i = at; i < whole; i += step) reinterpret_cast<int4*>(dst)[i] = __ldcv(reinterpret_cast<const int4*>(src) + i);
  for (int i = whole * 4 + at; i < count; i += step) dst[i] = __ldcv(src + i);
}
__global__ void __launch_bounds__(256) word_copy_kernel(nfk_word_copy_params p) {
  let_next_start();
  await_previous();
  const int at = blockIdx.x * 256 + threadIdx.x, step = gridDim.x * 256;
  copy_words(p.dst, p.src, p.count, at, step);
  copy_words(p.dst2, p.src2, p.count2, at, step);
}

}  // namespace

extern "C" int nfk_argmax_combine_p(const nfk_argmax_combine_params* p, cudaStream_t s) {
  if (!p) return NF_ERR_BAD_ARG;
  return nfk_argmax_combine(p->idx_out, p->cand_val, p->cand_idx, p->shards, p->rows, s);
}
extern "C" int nfk_copy_cols_p(const nfk_copy_cols_params* p, cudaStream_t s) {
  if (!p) return NF_ERR_BAD_ARG;
  return nfk_copy_cols(p->out, p->ld_out, p->in, p->ld_in, p->rows, p->cols, s);
}
extern "C" int nfk_memcpy_p(const nfk_memcpy_params* p, cudaStream_t s) {
  if (!p || p->count < 0 || p->elem_bytes < 0) return NF_ERR_BAD_ARG;
  const long long bytes = p->elem_bytes * p->count;
  if (bytes == 0) return NF_OK;
  if (!p->dst || !p->src) return NF_ERR_BAD_ARG;
  return cudaMemcpyAsync(p->dst, p->src, static_cast<size_t>(bytes), cudaMemcpyDefault, s) == cudaSuccess
             ? NF_OK : NF_ERR_CUDA;
}
extern "C" int nfk_word_copy_p(const nfk_word_copy_params* p, cudaStream_t s) {
  if (!p || p->count < 0 || p->count2 < 0) return NF_ERR_BAD_ARG;
  if (p->count == 0 && p->count2 == 0) return NF_OK;
  if ((p->count > 0 && (!p->dst || !p->src)) || (p->count2 > 0 && (!p->dst2 || !p->src2))) return NF_ERR_BAD_ARG;
  const long long most = p->count > p->count2 ? p->count : p->count2;
  long long blocks = (most + 1023) / 1024;
  if (blocks > 2ll * device_sm_count()) blocks = 2ll * device_sm_count();
  return launch_kernel(early_first(p->early), word_copy_kernel, static_cast<int>(blocks), 256, 0, s, 1, *p) == cudaSuccess
             ? NF_OK : NF_ERR_CUDA;
}
extern "C" int nfk_memcpy2d_p(const nfk_memcpy2d_params* p, cudaStream_t s) {
  if (!p || p->height < 0 || p->width < 0 || p->dpitch < p->width || p->spitch < p->width) return NF_ERR_BAD_ARG;
  if (p->height == 0 || p->width == 0) return NF_OK;
  if (!p->dst || !p->src) return NF_ERR_BAD_ARG;
  return cudaMemcpy2DAsync(p->dst, static_cast<size_t>(p->dpitch), p->src, static_cast<size_t>(p->spitch),
                           static_cast<size_t>(p->width), static_cast<size_t>(p->height), cudaMemcpyDefault,
                           s) == cudaSuccess
             ? NF_OK : NF_ERR_CUDA;
}
extern "C" int nfk_sleep_p(const nfk_sleep_params* p, cudaStream_t s) {
  if (!p) return NF_ERR_BAD_ARG;
  return p->micros == 0 ? NF_OK : nfk_sleep(p->micros, s);
}
extern "C" int nfk_kv_move_p(const nfk_kv_move_params* p, cudaStream_t s) {
  if (!p) return NF_ERR_BAD_ARG;
  return nfk_kv_move_pages(p->pool, p->staging, p->page_ids, p->n_pages, p->page_bytes, p->num_pages,
                           p->direction, p->num_ctas, p->status, s);
}
