// Launchers of the tensor-core prefill attention (body: fbla_prefill_tc.cuh).
#include "fbla_prefill_tc.cuh"
#include "fbla_launch.h"
#include <stdlib.h>
#include <string.h>
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
namespace tc {
template <int CB, int FB, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1) attend_tc_kernel(const fbla_k_prefill a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // A launch that the count does not ask for is gone before its turn: the close pass, which comes first in every call with a count on the
  // device, lets the next kernel begin behind its own wait, so count and length are what they will be. One CTA keeps the order: the kernel
  // after this one may not begin before the close pass is complete. (512 tokens at 128 in a cache with room for 64K, us: one launch 52;
  // two 59 with both waiting first, 54 so.)
  if (a.dcount && !serves(a)) {
    allow_next_pass();
    if (blockIdx.x == 0 && blockIdx.y == 0) wait_previous_pass();
    return;
  }
  wait_previous_pass();
  allow_next_pass();
  attend_tiles<CB, FB, SPLIT ? CLUSTER : WHOLE>(a, smem_raw);
}
}  // namespace tc
}  // namespace fbla

extern "C" int fbla_k_attend_tc_status(void) {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, fbla::tc::g_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(fbla::tc::g_status, &zero, sizeof(int));
  return v;
}

// The launches of a chunk (see fbla_kernels.h). A chunk of the ceiling's own size, at the end of the cache's room, has the fewest shares;
// where fewer tokens can have more, the larger clusters are a launch of their own, with as many tiles as can have them: for one
// launch with the largest cluster, a chunk of the ceiling's size would wait for SMs that its idle CTAs' clusters ask for.
extern "C" int fbla_k_attend_tc_deal(int heads, int tiles, int passes, int device_count, fbla_k_tc_deal deal[2]) {
  using fbla::tc::tile_shares;
  const int own = tile_shares((long long)tiles * heads, passes, FBLA_K_TILE_SHARES), most = device_count ? tile_shares(heads, passes, FBLA_K_TILE_SHARES) : own;
  int n = 0;
  if (most > own) {
    const int few = (148 - 8 * own) / ((own + 1) * heads);
    deal[n++] = fbla_k_tc_deal{most, own, few < tiles ? few : tiles};
  }
  deal[n++] = fbla_k_tc_deal{own, 0, tiles};
  return n;
}

extern "C" cudaError_t fbla_k_attend_tc_launch(const fbla_k_prefill *a, cudaStream_t stream) {
  using namespace fbla::tc;
  const int tiles = (a->count * (a->q_heads / a->kv_heads) + CTA_ROWS - 1) / CTA_ROWS, heads = a->batch * a->kv_heads;
  const size_t smem = sizeof(Smem) + 1024;
  static thread_local int configured[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    for (auto kernel : {attend_tc_kernel<3, 3, false>, attend_tc_kernel<3, 3, true>, attend_tc_kernel<4, 2, false>, attend_tc_kernel<4, 2, true>}) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    if (dev >= 0 && dev < 64) configured[dev] = 1;
  }
  fbla_k_tc_deal deal[2];
  const int launches = fbla_k_attend_tc_deal(heads, tiles, ((a->length ? a->room : a->n0 + a->count) - 1) / fbla::G + 1, a->dcount != nullptr, deal);
  for (int i = 0; i < launches; ++i) {
    fbla_k_prefill args = *a;
    args.cluster = deal[i].cluster;
    args.above = deal[i].above;
    const bool split = args.cluster > 1;
    const auto kernel = a->cb == 3 ? split ? attend_tc_kernel<3, 3, true> : attend_tc_kernel<3, 3, false> : split ? attend_tc_kernel<4, 2, true> : attend_tc_kernel<4, 2, false>;
    const int wide = deal[i].tiles * args.cluster;
    // launched dependent where one wave holds the grid (a 777-token prompt 69.5 -> 67.8 us), or where it is likely not the one that
    // works; several waves that began among the CTAs of the kernel before measured 3 % slower (batch 4 x 8192 4.55 -> 4.69 ms)
    const cudaError_t e = fbla::launch(wide * heads <= 148 || i + 1 < launches, args.cluster, kernel, dim3(wide, heads), THREADS, smem, stream, args);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

extern "C" int fbla_k_attend_plan(const fbla_k_prefill *a, fbla_k_prefill args[2], int tensor[2]) {
  static const bool rows_only = [] { const char *e = getenv("MLOPS_FBLA_PREFILL"); return e && !strcmp(e, "rows"); }();
  const int rows = a->count * (a->q_heads / a->kv_heads);  // (with a device count: the ceiling)
  args[0] = *a;
  args[0].tc_min_rows = 0;
  if (rows_only || rows < FBLA_K_TC_MIN_ROWS) { tensor[0] = 0; return 1; }
  tensor[0] = 1;
  if (!a->dcount) return 1;
  args[0].tc_min_rows = FBLA_K_TC_MIN_ROWS;
  args[1] = args[0];
  tensor[1] = 0;
  return 2;
}

extern "C" cudaError_t fbla_k_attend_launch(const fbla_k_prefill *a, cudaStream_t stream) {
  fbla_k_prefill args[2];
  int tensor[2];
  const int n = fbla_k_attend_plan(a, args, tensor);
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < n && e == cudaSuccess; ++i) e = tensor[i] ? fbla_k_attend_tc_launch(&args[i], stream) : fbla_k_attend_rows_launch(&args[i], stream);
  return e;
}

extern "C" cudaError_t fbla_k_attend_tc_pass(fbla_k_prefill *a, fbla_k_pass *info) {
  using namespace fbla::tc;
  a->cluster = 1;  // (an item takes a tile's shares in turn)
  const int qg = a->q_heads / a->kv_heads, rows = a->count * qg, heads = a->batch * a->kv_heads;
  const size_t smem = sizeof(Smem) + 1024;
  if (a->cb == 3) return pass_of(attend_tc_kernel<3, 3, false>, (rows + CTA_ROWS - 1) / CTA_ROWS, heads, THREADS, smem, "fbla::tc::attend_tc_item<3, 3>", info);
  return pass_of(attend_tc_kernel<4, 2, false>, (rows + CTA_ROWS - 1) / CTA_ROWS, heads, THREADS, smem, "fbla::tc::attend_tc_item<4, 2>", info);
}
