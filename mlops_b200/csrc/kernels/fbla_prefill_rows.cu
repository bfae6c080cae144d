// Launcher of the few-row prefill attention (body: fbla_prefill_rows.cuh).
#include "fbla_prefill_rows.cuh"
#include "fbla_launch.h"
#include <stdio.h>

namespace fbla {
template <int CB, int FB>
__global__ void __launch_bounds__(32 * rows::WARPS, 1) attend_rows_kernel(const fbla_k_prefill a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  wait_previous_pass();
  allow_next_pass();
  attend_rows_item<CB, FB>(a, smem_raw);
}

template <int CB, int FB> static cudaError_t launch_rows(const fbla_k_prefill &a, int bundles, cudaStream_t stream) {
  constexpr int smem = (int)sizeof(rows::RowSmem<CB, FB>);
  static thread_local int configured[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(attend_rows_kernel<CB, FB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = 1;
  }
  return launch(true, a.cluster, attend_rows_kernel<CB, FB>, dim3(bundles * a.cluster, a.batch * a.kv_heads), 32 * rows::WARPS, smem, stream, a);
}

// tiles of the launch: with a device count that goes to the tensor-core pass from tc_min_rows rows on, no more than it leaves here
static int row_tiles(const fbla_k_prefill &a) {
  const int rows = a.count * (a.q_heads / a.kv_heads), most = a.tc_min_rows && rows >= a.tc_min_rows ? a.tc_min_rows - 1 : rows;
  return (most + rows::COLS - 1) / rows::COLS;
}
}  // namespace fbla

extern "C" cudaError_t fbla_k_attend_rows_launch(const fbla_k_prefill *a, cudaStream_t stream) {
  int bundles = fbla::row_tiles(*a);
  fbla_k_prefill args = *a;
  if (a->length || a->dcount) {  // the deal follows from the device's length and count: the launch has room for what they can become
    const long long most = (a->room / fbla::G + fbla::rows::WARPS - 1) / fbla::rows::WARPS;
    args.cluster = most < 1 ? 1 : most > FBLA_K_ROW_SHARES ? FBLA_K_ROW_SHARES : (int)most;
  } else {
    const fbla::rows::RowDeal deal = fbla::rows::row_deal(bundles, a->batch * a->kv_heads, (a->n0 + a->count - 1) / fbla::G);
    bundles = (bundles + deal.tiles - 1) / deal.tiles;
    args.cluster = deal.shares;
  }
  return a->cb == 3 ? fbla::launch_rows<3, 3>(args, bundles, stream) : fbla::launch_rows<4, 2>(args, bundles, stream);
}

extern "C" cudaError_t fbla_k_attend_rows_pass(fbla_k_prefill *a, fbla_k_pass *info) {
  using namespace fbla;
  a->cluster = 1;
  cudaFuncAttributes fa;
  const cudaError_t e = a->cb == 3 ? cudaFuncGetAttributes(&fa, attend_rows_kernel<3, 3>) : cudaFuncGetAttributes(&fa, attend_rows_kernel<4, 2>);
  if (e != cudaSuccess) return e;
  info->gx = row_tiles(*a); info->gy = a->batch * a->kv_heads; info->gz = 1; info->threads = 32 * rows::WARPS;
  info->smem_bytes = (int)(a->cb == 3 ? sizeof(rows::RowSmem<3, 3>) : sizeof(rows::RowSmem<4, 2>)) + 128;
  info->regs = fa.numRegs;
  snprintf(info->entry, sizeof info->entry, "fbla::attend_rows_item<%d, %d>", a->cb, a->fb);
  return cudaSuccess;
}
