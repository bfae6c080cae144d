// Launchers of the dense decode (bodies: fbla_dense.cuh).
#include "fbla_dense.cuh"
#include "fbla_launch.h"
#include <stdio.h>

namespace fbla {
namespace dense {
template <int CB, int FB, int QG>
__global__ void __launch_bounds__(32 * SCORE_WARPS, 1) score_kernel(const fbla_k_decode a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  score_item<CB, FB, QG>(a, smem_raw);
}

template <int QG>
__global__ void __launch_bounds__(256) mass_kernel(const fbla_k_decode a) {
  mass_item<QG>(a, nullptr);
}

template <int CB, int FB, int QG>
__global__ void __launch_bounds__(32 * VALUE_WARPS, 1) value_kernel(const fbla_k_decode a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  value_item<CB, FB, QG>(a, smem_raw);
}

template <int QG>
__global__ void __launch_bounds__(128) gather_kernel(const fbla_k_decode a) {
  gather_item<QG>(a, nullptr);
}

template <int CB, int FB, int QG> struct Kernels {
  static constexpr size_t SCORE_SMEM = sizeof(ScoreSmem), VALUE_SMEM = sizeof(ValueSmem);
  static cudaError_t configure() {  // once per device and host thread
    static thread_local int configured[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && configured[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(score_kernel<CB, FB, QG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCORE_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(value_kernel<CB, FB, QG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VALUE_SMEM);
    if (e == cudaSuccess && dev >= 0 && dev < 64) configured[dev] = 1;
    return e;
  }
  static cudaError_t pass(const fbla_k_decode &a, int which, bool dependent, cudaStream_t stream) {
    const int vheads = a.batch * a.kv_heads * a.vg;
    switch (which) {
      case 0: return launch(dependent, 1, score_kernel<CB, FB, QG>, dim3(a.coarse_ctas), 32 * SCORE_WARPS, SCORE_SMEM, stream, a);
      case 1: return launch(dependent, 1, mass_kernel<QG>, dim3((vheads + 7) / 8), 256, 0, stream, a);
      case 2: return launch(dependent, 1, value_kernel<CB, FB, QG>, dim3(a.coarse_ctas), 32 * VALUE_WARPS, VALUE_SMEM, stream, a);
      case 3: return launch(dependent, 1, gather_kernel<QG>, dim3(vheads * QG), 128, 0, stream, a);
    }
    return cudaErrorInvalidValue;
  }
  static cudaError_t all(const fbla_k_decode &a, cudaStream_t stream) {
    cudaError_t e = configure();
    if (a.phase != 2 && e == cudaSuccess) e = pass(a, 0, true, stream);
    if (e != cudaSuccess) return e;
    if (a.phase == 1) return pass(a, 1, true, stream);
    e = pass(a, 2, true, stream);
    return e == cudaSuccess ? pass(a, 3, true, stream) : e;
  }
  template <class K> static cudaError_t describe(K kernel, int items, int threads, size_t smem, fbla_k_pass *p) {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    p->gx = items; p->gy = p->gz = 1; p->threads = threads; p->smem_bytes = (int)smem; p->regs = fa.numRegs;
    return cudaSuccess;
  }
  static cudaError_t passes(const fbla_k_decode &a, fbla_k_pass *p) {
    const int vheads = a.batch * a.kv_heads * a.vg;
    cudaError_t e = describe(score_kernel<CB, FB, QG>, a.coarse_ctas, 32 * SCORE_WARPS, SCORE_SMEM, p + 0);
    if (e == cudaSuccess) e = describe(mass_kernel<QG>, (vheads + 7) / 8, 256, 0, p + 1);
    if (e == cudaSuccess) e = describe(value_kernel<CB, FB, QG>, a.coarse_ctas, 32 * VALUE_WARPS, VALUE_SMEM + 128, p + 2);
    if (e == cudaSuccess) e = describe(gather_kernel<QG>, vheads * QG, 128, 0, p + 3);
    snprintf(p[0].entry, sizeof p[0].entry, "fbla::dense::score_item<%d, %d, %d>", CB, FB, QG);
    snprintf(p[1].entry, sizeof p[1].entry, "fbla::dense::mass_item<%d>", QG);
    snprintf(p[2].entry, sizeof p[2].entry, "fbla::dense::value_item<%d, %d, %d>", CB, FB, QG);
    snprintf(p[3].entry, sizeof p[3].entry, "fbla::dense::gather_item<%d>", QG);
    return e;
  }
};

template <class F> cudaError_t dispatch(const fbla_k_decode &a, F f) {
  if (a.cb == 3) return a.qg == 1 ? f(Kernels<3, 3, 1>{}) : a.qg == 2 ? f(Kernels<3, 3, 2>{}) : f(Kernels<3, 3, 4>{});
  return a.qg == 1 ? f(Kernels<4, 2, 1>{}) : a.qg == 2 ? f(Kernels<4, 2, 2>{}) : f(Kernels<4, 2, 4>{});
}
}  // namespace dense
}  // namespace fbla

extern "C" cudaError_t fbla_k_dense_launch(const fbla_k_decode *a, cudaStream_t stream) {
  return fbla::dense::dispatch(*a, [&](auto k) { return decltype(k)::all(*a, stream); });
}
extern "C" cudaError_t fbla_k_dense_pass_launch(const fbla_k_decode *a, int pass, cudaStream_t stream) {
  return fbla::dense::dispatch(*a, [&](auto k) { return decltype(k)::pass(*a, pass, false, stream); });
}
extern "C" cudaError_t fbla_k_dense_passes(const fbla_k_decode *a, fbla_k_pass info[4]) {
  return fbla::dense::dispatch(*a, [&](auto k) { return decltype(k)::passes(*a, info); });
}

// A sub-block of a row of N tokens holds 16 / N of the mass on average. Where that is not far below tau most sub-blocks are selected
// (how many beyond that the values decide), and adding each once is the faster way; else the coarse planes carry most of the sum and one
// sweep over them costs less than two. The host does not know the values, so the line lies where the worse of two kinds of values loses
// least: N(0, 1), few sub-blocks far above the average, and the same with four outlier channels, many. The two sweeps' work per group is the
// same for one query as for four, one sweep's is not: a line per query count. One sweep is a launch and a chain of round trips
// longer, some 8 us, so that with few groups per CTA the line lies further out. Measured on B200, us per step one sweep / two, N(0, 1)
// and outliers, 32 / 8 heads unless said; N tau in front:
//   batch 8, 3+3:  20: 309 / 227, 324 / 229    25: 264 / 261, 331 / 273    30: 242 / 294, 340 / 313    39: 263 / 367, 362 / 389
//   batch 8, 4+2:  20: 111 / 81, 114 / 81      25: 97 / 92, 116 / 94       30: 91 / 103, 119 / 106     39: 96 / 124, 123 / 127
//   batch 1, 3+3:  20: 77 / 55, 79 / 56        30: 66 / 62, 80 / 65        39: 63 / 72, 78 / 75        60: 79 / 95, 92 / 98
//   batch 1, 4+2:  20: 41 / 32, 42 / 32        30: 36 / 35, 41 / 36        39: 38 / 38, 42 / 39        60: 42 / 46, 46 / 46
//   batch 8, 16 / 8 heads, 3+3:  20: 238 / 237, 252 / 239    23: 220 / 259, 256 / 266     4+2:  16: 99 / 77, 92 / 77    23: 82 / 92, 93 / 93
//   batch 8, 8 / 8 heads, 3+3:   13: 222 / 178, 187 / 176    16: 207 / 205, 193 / 204     4+2:  13: 79 / 73, 70 / 73    16: 78 / 82, 72 / 82
// Rows of lengths of their own are shorter than the room that the host sees. Evenly spread up to it they break even at about twice these
// lines, all of them full at the lines themselves; the host asks with two thirds of the room, where either loses about as much (N tau of the
// room, us one / two, batch 8, 32 / 8 heads, 3+3, N(0, 1): spread 31: 262 / 188, 40: 264 / 235, 54: 278 / 303; full 31: 245 / 302, 40: 263 / 374).
extern "C" int fbla_k_two_sweeps(int batch, int vheads, int qg, long long tokens, float tau) {
  const long long groups = (tokens + fbla::G - 1) / fbla::G;
  const double n_tau = (double)tokens * tau;
  const int line = qg == 4 ? 28 : qg == 2 ? 22 : 15;
  const int few = qg == 4 ? 52 : qg == 2 ? 20 : 12, few_line = qg == 4 ? 40 : qg == 2 ? 30 : 20;  // groups per CTA of a B200, whatever the device
  return batch <= FBLA_K_DENSE_MAX_BATCH && (long long)vheads * groups * fbla::dense::PAIRS < (1ll << 29) &&
         (n_tau <= line || (n_tau <= few_line && (long long)vheads * groups <= few * 148));
}
