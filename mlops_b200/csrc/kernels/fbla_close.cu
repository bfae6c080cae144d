// Launchers of the close / finish passes and of the chunk without queries (bodies: fbla_close.cuh).
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
template <int CB, int FB>
__global__ void __launch_bounds__(CLOSE_THREADS, 2) close_kernel(const fbla_k_prefill a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous_pass();
  allow_next_pass();
  close_item<CB, FB>(a, smem_raw);
}

template <int CB, int FB>
__global__ void __launch_bounds__(TENSOR_THREADS, 4) write_kernel(const fbla_k_prefill a, int blocks) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous_pass();
  // The next kernel is not let in before this one is through: a decode's CTAs want an SM each, and were placed as these CTAs left. us per append and
  // decode, 32 / 8 heads, let in at the top / not, and behind a read of 256 MB: 1 x 100 000 + 1 4+2 49.6 / 45.1, 59.4 / 49.2; 4 x 60 000 + 1 3+3
  // 122.5 / 111.7, 132.1 / 115.8; 4 x 3 000 + 1 3+3 26.3 / 26.9 (Python's), 33.8 / 23.6. At the end of a CTA: 129.0 at 4 x 60 000, behind the read.
  write_chunk<CB, FB>(a, smem_raw, blocks);
}

__global__ void __launch_bounds__(CLOSE_THREADS) finish_kernel(const fbla_k_prefill a) {
  wait_previous_pass();
  allow_next_pass();
  finish_item(a, nullptr);
}

// the write kernels' shared memory is above the default limit: asked for once per device and host thread; *sms: the device's SMs
static cudaError_t configure(int *sms) {
  static thread_local int configured[64] = {0};  // (its SMs, once configured)
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && configured[dev]) { *sms = configured[dev]; return cudaSuccess; }
  cudaError_t e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  for (auto kernel : {write_kernel<3, 3>, write_kernel<4, 2>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WriteSmem));
  if (e == cudaSuccess && dev >= 0 && dev < 64) configured[dev] = n;
  *sms = n;
  return e;
}
}  // namespace fbla

extern "C" cudaError_t fbla_k_close_launch(const fbla_k_prefill *a, int close_blocks, cudaStream_t stream) {
  if (close_blocks <= 0) return cudaSuccess;
  static_assert(2 * sizeof(fbla::CloseSmem) <= 48 * 1024, "within the default limit");
  const dim3 grid(close_blocks, a->batch * a->kv_heads);
  return fbla::launch(true, 1, a->cb == 3 ? fbla::close_kernel<3, 3> : fbla::close_kernel<4, 2>, grid, fbla::CLOSE_THREADS, 2 * sizeof(fbla::CloseSmem), stream, *a);
}

extern "C" cudaError_t fbla_k_write_launch(const fbla_k_prefill *a, int close_blocks, cudaStream_t stream) {
  int sms = 0;
  const cudaError_t e = fbla::configure(&sms);
  if (e != cudaSuccess) return e;
  // as many CTAs as the SMs hold at once (four each), no more than there are units to close or to clear
  const int blocks = close_blocks > 0 ? close_blocks : 1;
  const long long heads = (long long)a->batch * a->kv_heads, units = 2 * blocks * heads;
  const long long clear = a->clear_groups ? heads * (a->clear_groups - (a->count - 1) / fbla::G) : 0, work = units > clear ? units : clear;
  const int ctas = (int)(work < 4 * sms ? work : 4 * sms);
  return fbla::launch(true, 1, a->cb == 3 ? fbla::write_kernel<3, 3> : fbla::write_kernel<4, 2>, dim3(ctas), fbla::TENSOR_THREADS, sizeof(fbla::WriteSmem), stream, *a, blocks);
}

extern "C" cudaError_t fbla_k_finish_launch(const fbla_k_prefill *a, cudaStream_t stream) {
  return fbla::launch(true, 1, fbla::finish_kernel, dim3(a->batch * a->kv_heads), fbla::CLOSE_THREADS, 0, stream, *a);
}

extern "C" cudaError_t fbla_k_close_pass(const fbla_k_prefill *a, int close_blocks, fbla_k_pass *info) {
  const int heads = a->batch * a->kv_heads;
  if (a->cb == 3) return pass_of(fbla::close_kernel<3, 3>, close_blocks, heads, fbla::CLOSE_THREADS, 2 * sizeof(fbla::CloseSmem), "fbla::close_item<3, 3>", info);
  return pass_of(fbla::close_kernel<4, 2>, close_blocks, heads, fbla::CLOSE_THREADS, 2 * sizeof(fbla::CloseSmem), "fbla::close_item<4, 2>", info);
}

extern "C" cudaError_t fbla_k_finish_pass(const fbla_k_prefill *a, fbla_k_pass *info) {
  return pass_of(fbla::finish_kernel, a->batch * a->kv_heads, 1, fbla::CLOSE_THREADS, 0, "fbla::finish_item", info);
}
