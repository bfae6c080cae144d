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

template <int CB, int FB, int QG>
__global__ void __launch_bounds__(32 * SCORE_WARPS, 1) head_kernel(const fbla_k_decode a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  head_passes<CB, FB, QG>(a, smem_raw);
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
    if (e == cudaSuccess) e = cudaFuncSetAttribute(head_kernel<CB, FB, QG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(HeadSmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(head_kernel<CB, FB, QG>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess && dev >= 0 && dev < 64) configured[dev] = 1;
    return e;
  }
  // clusters of `ctas` (1 .. 16) that are at work at once (0: such a cluster cannot be placed); asked for once per device and host thread, as
  // the attributes (every call: 0.3 us of a 12 us decode)
  static int clusters(int ctas) {
    static thread_local short held[64][17] = {};  // the answer + 1
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    const bool known = dev >= 0 && dev < 64;
    if (known && held[dev][ctas]) return held[dev][ctas] - 1;
    if (configure() != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(32 * SCORE_WARPS); cfg.dynamicSmemBytes = sizeof(HeadSmem);
    cudaLaunchAttribute size = {};
    size.id = cudaLaunchAttributeClusterDimension;
    size.val.clusterDim.x = ctas; size.val.clusterDim.y = size.val.clusterDim.z = 1;
    cfg.attrs = &size; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, head_kernel<CB, FB, QG>, &cfg) != cudaSuccess) {
      cudaGetLastError();  // (not the call's: it takes three kernels)
      n = 0;
    }
    if (known) held[dev][ctas] = (short)(n + 1);
    return n;
  }
  static cudaError_t whole(fbla_k_decode a, bool dependent, cudaStream_t stream) {
    a.mass_given = 0;
    return launch(dependent, a.head_ctas, head_kernel<CB, FB, QG>, dim3(a.head_ctas, a.kv_heads * a.vg, a.batch), 32 * SCORE_WARPS, sizeof(HeadSmem), stream, a);
  }
  static cudaError_t pass(const fbla_k_decode &a, int which, bool dependent, cudaStream_t stream) {
    const int vheads = a.batch * a.kv_heads * a.vg;
    if (a.head_ctas) return which == 0 ? whole(a, dependent, stream) : cudaSuccess;
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
    if (a.head_ctas && e == cudaSuccess) return whole(a, true, stream);
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
    if (a.head_ctas && e == cudaSuccess) {
      e = describe(head_kernel<CB, FB, QG>, a.head_ctas, 32 * SCORE_WARPS, sizeof(HeadScoreSmem), p + 0);
      if (e == cudaSuccess) e = describe(head_kernel<CB, FB, QG>, a.head_ctas, 32 * VALUE_WARPS, sizeof(HeadValueItemSmem), p + 2);
      for (int i = 0; i <= 2; i += 2) { p[i].gy = a.kv_heads * a.vg; p[i].gz = a.batch; }
      snprintf(p[0].entry, sizeof p[0].entry, "fbla::dense::score_item<%d, %d, %d, true>", CB, FB, QG);
      snprintf(p[2].entry, sizeof p[2].entry, "fbla::dense::value_item<%d, %d, %d, true>", CB, FB, QG);
    }
    snprintf(p[3].entry, sizeof p[3].entry, "fbla::dense::gather_item<%d>", QG);
    return e;
  }
};

template <class F> auto dispatch(const fbla_k_decode &a, F f) {
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
// longer, some 8 us, so that with few groups per CTA the line lies further out. Measured on B200 when the lines were set, us per step one sweep /
// two, N(0, 1) and outliers, 32 / 8 heads unless said; N tau in front (since then one sweep has become some 7 us shorter at batch 1, two in 3+3 by
// a tenth or more; the lines have stayed):
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

// A short decode is mostly launches and the chains of round trips at their borders. One kernel with a cluster per virtual head has neither,
// but its heads' CTAs leave SMs idle and a head's work cannot move to another's. CTAs per head: as many as let all clusters run at once (of n
// CTAs with an SM each a B200 holds n: 1: 148, 2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 8: 15, 10: 11, 16: 7). At most 20 groups per CTA of the room, 16 in
// clusters of 16. Device time on B200 behind a flush of L2, us, three kernels / one, 3+3, by heads and queries per head:
//   8 heads, 10 CTAs, 4:   3 groups per CTA 25.6 / 19.0    8: 31.8 / 24.4    13: 33.5 / 28.8    17: 35.9 / 32.9    20: 37.9 / 35.0    24: 37.9 / 38.9    (4+2  20: 36.2 / 34.5)
//   16 heads, 6 CTAs, 4:   3: 25.6 / 18.7    8: 29.7 / 24.8    13: 35.6 / 30.6    20: 37.9 / 36.4    (4+2  20: 37.9 / 35.1)
//   33 heads, 4 CTAs, 4:   3: 27.6 / 18.7    13: 37.9 / 30.7    20: 44.3 / 38.6    24: 46.9 / 43.0
//   74 heads, 2 CTAs, 4:   3: 25.6 / 20.5    13: 37.9 / 32.8    20: 45.8 / 40.9    2: 20: 44.5 / 43.0    148, 1 CTA, 4: 20: 48.4 / 42.7
//   75 heads, 1 CTA, 4:    3: 25.6 / 20.6    13: 33.8 / 30.9    17: 35.8 / 34.6    20: 37.2 / 38.8       7 heads, 16 CTAs, 4: 17: 37.9 / 34.9
extern "C" int fbla_k_head_ctas(int vheads, long long tokens) {
  static const struct { int ctas, vheads; } held[] = {{16, 7}, {10, 11}, {8, 15}, {6, 22}, {5, 26}, {4, 33}, {3, 45}, {2, 74}, {1, 148}};
  for (const auto &h : held)
    if (vheads <= h.vheads) return (tokens + fbla::G - 1) / fbla::G <= (h.ctas == 16 ? 16 : 20) * h.ctas ? h.ctas : 0;
  return 0;
}
// Fewer groups where the one kernel falls behind sooner: rows of lengths of their own (it waits for the longest; the three kernels deal what there
// is over all SMs), the more the more SMs its clusters leave idle; and one query per head, where a unit is a whole group, so that a CTA whose
// groups and window sub-blocks are more than its warps does them in two goes (`one`: what still fits). us, three kernels / one (and, 4+2, as
// three kernels were before there was one); rows evenly spread from a tenth of the room up to it:
//   8 heads, 10 CTAs, 4 queries:  13 groups per CTA 31.7 / 28.7    17: 30.7 / 32.3    20: 31.8 / 34.4       75 heads, 1 CTA:  13: 29.7 / 30.5    20: 31.5 / 36.3
//   8 heads, 2 queries:           12: 29.7 / 28.5    17: 30.0 / 33.8     75 heads:  10: 27.7 / 28.7    20: 31.1 / 37.9    27 heads, 4 CTAs:  12: 31.8 / 28.7    17: 34.8 / 34.9
//   8 heads, 1 query:             9: 29.7 / 28.7     13: 31.8 / 31.5     17: 32.8 / 38.9 (4+2 31.7 / 40.5, 32)            148 heads, 1 CTA: 13: 39.9 / 35.0    16: 38.0 / 38.7
//   27 heads, 4 CTAs, 1 query:    12: 33.8 / 32.5    13: 32.4 / 36.8 (4+2 31.8 / 38.6, 33)     75 heads:  9: 29.7 / 29.6    20: 33.8 / 45.0 (4+2 31.8 / 45.1, 34)
// One length, 1 query:  75 heads: 15: 37.9 / 36.7    20: 40.9 / 45.1    46 heads, 2 CTAs: 10: 35.8 / 30.8    13: 33.8 / 36.7    8 heads: 14: 33.8 / 32.9    15: 33.8 / 36.9    16 heads: 20: 42.0 / 41.3
// Last, where fewer clusters than heads run at once, or none can be placed, the three kernels are the way that always runs.
extern "C" int fbla_k_head_choice(const fbla_k_decode *a, int vheads, int qg, int own_lengths, long long tokens, int (*held)(const fbla_k_decode *a, int ctas)) {
  const int ctas = fbla_k_head_ctas(vheads, tokens), busy = ctas * vheads;
  if (ctas == 0) return 0;
  const bool few = busy < 96;  // SMs at work
  const int one = ctas == 16 ? 15 : ctas >= 8 ? 14 : ctas == 6 ? 13 : ctas >= 4 ? 12 : ctas >= 2 ? 10 : 15;
  const int line = !own_lengths ? (qg == 1 && few ? one : 20)
                   : qg == 4    ? (few ? 16 : 20)
                   : qg == 2    ? (few ? 12 : busy < 132 ? 16 : 20)
                                : (few ? 9 : one);
  return (tokens + fbla::G - 1) / fbla::G <= (long long)line * ctas && held(a, ctas) >= vheads ? ctas : 0;
}
extern "C" int fbla_k_head_clusters(const fbla_k_decode *a, int ctas) {
  return fbla::dense::dispatch(*a, [&](auto k) { return decltype(k)::clusters(ctas); });
}
