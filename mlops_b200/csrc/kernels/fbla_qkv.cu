// Launchers of the fused QKV step (bodies: fbla_qkv.cuh).
#include "fbla_qkv.cuh"
#include "fbla_close.cuh"
#include "fbla_launch.h"
#include <stdio.h>

namespace {
template <class K> cudaError_t pass_of(K kernel, int gx, int gy, int threads, size_t smem, const char *entry, fbla_k_pass *p) {
  cudaFuncAttributes fa;
  const cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
  if (e != cudaSuccess) return e;
  p->gx = gx; p->gy = gy; p->gz = 1; p->threads = threads; p->smem_bytes = (int)smem; p->regs = fa.numRegs;
  snprintf(p->entry, sizeof p->entry, "%s", entry);
  return cudaSuccess;
}
}  // namespace

namespace fbla {
// The whole one-token step of a (batch row, KV head): the group that the position closes is quantised from the open window,
// then the token takes its place. One launch: the close pass alone is a launch that finds nothing to do 127 times of 128.
template <int CB, int FB, bool NORM>
__global__ void __launch_bounds__(CLOSE_THREADS) qkv_step_kernel(const fbla_k_prefill closing, const fbla_k_token a) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  wait_previous_pass();
  const int bh = blockIdx.x;
  const Chunk ch = chunk_of(closing, bh / closing.kv_heads);
  const int g = closing_group(ch, 0);
  if (g >= 0) close_group<CB, FB>(closing, *reinterpret_cast<CloseSmem (*)[2]>(smem_raw), bh, g, ch.n0);
  // The decode behind this step is let in here, not at the top: launched together with this kernel, while neither's code was in L2 yet, it ran
  // 4 to 10 us longer (us of the step behind a read of 256 MB, 3+3, top / here: 16 rows of 240 to 2 400 tokens, 8 / 8 heads 53.2 / 41.5; 32 of 300
  // to 6 000, 32 / 8 heads 77.8 / 71.6; one of 1 999 27.7 / 19.5; nothing evicted between: 34.2 / 34.2, 67.2 / 66.9, 13.0 / 13.0).
  allow_next_pass();
  qkv_token_item<NORM>(a, nullptr);
}

template <bool NORM>
__global__ void __launch_bounds__(256) qkv_chunk_kernel(const fbla_k_token a) {
  wait_previous_pass();
  allow_next_pass();
  qkv_chunk_item<NORM>(a, nullptr);
}
}  // namespace fbla

template <int CB, int FB, bool NORM> static cudaError_t launch_step(const fbla_k_prefill &closing, const fbla_k_token &a, cudaStream_t stream) {
  static thread_local int configured[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(fbla::qkv_step_kernel<CB, FB, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * (int)sizeof(fbla::CloseSmem));
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = 1;
  }
  return fbla::launch(true, 1, fbla::qkv_step_kernel<CB, FB, NORM>, dim3(a.batch * a.kv_heads), fbla::CLOSE_THREADS, 2 * sizeof(fbla::CloseSmem), stream, closing, a);
}
extern "C" cudaError_t fbla_k_qkv_step_launch(const fbla_k_prefill *closing, const fbla_k_token *a, cudaStream_t stream) {
  if (closing->cb == 3) return a->q_norm ? launch_step<3, 3, true>(*closing, *a, stream) : launch_step<3, 3, false>(*closing, *a, stream);
  return a->q_norm ? launch_step<4, 2, true>(*closing, *a, stream) : launch_step<4, 2, false>(*closing, *a, stream);
}

extern "C" cudaError_t fbla_k_qkv_chunk_launch(const fbla_k_token *a, cudaStream_t stream) {
  const dim3 grid((a->max_count + fbla::TOK - 1) / fbla::TOK, a->kv_heads);
  return fbla::launch(true, 1, a->q_norm ? fbla::qkv_chunk_kernel<true> : fbla::qkv_chunk_kernel<false>, grid, 256, 0, stream, *a);
}

// (the registers of the kernel that runs the item here: the whole step)
extern "C" cudaError_t fbla_k_qkv_token_pass(const fbla_k_token *a, fbla_k_pass *info) {
  const int heads = a->batch * a->kv_heads;
  if (a->q_norm) return pass_of(fbla::qkv_step_kernel<3, 3, true>, heads, 1, 256, 0, "fbla::qkv_token_item<true>", info);
  return pass_of(fbla::qkv_step_kernel<3, 3, false>, heads, 1, 256, 0, "fbla::qkv_token_item<false>", info);
}

extern "C" cudaError_t fbla_k_qkv_chunk_pass(const fbla_k_token *a, fbla_k_pass *info) {
  const int tiles = (a->max_count + fbla::TOK - 1) / fbla::TOK;
  if (a->q_norm) return pass_of(fbla::qkv_chunk_kernel<true>, tiles, a->kv_heads, 256, 0, "fbla::qkv_chunk_item<true>", info);
  return pass_of(fbla::qkv_chunk_kernel<false>, tiles, a->kv_heads, 256, 0, "fbla::qkv_chunk_item<false>", info);
}
