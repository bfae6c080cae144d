// Launchers of the decode passes (bodies: fbla_decode.cuh).
#include "fbla_decode.cuh"
#include "fbla_launch.h"
#include <stdio.h>

namespace fbla {
template <int CB, int FB, int QG, int DEAL, int SHAPE>
__global__ void __launch_bounds__(32 * CoarseShape<CB, SHAPE>::TOTAL, 1) coarse_kernel(const fbla_k_decode a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  coarse_item<CB, FB, QG, DEAL, SHAPE>(a, smem_raw);
}

template <int QG>
__global__ void __launch_bounds__(256) select_kernel(const fbla_k_decode a) {
  select_item<QG>(a, nullptr);
}

template <int CB, int FB, int QG>
__global__ void __launch_bounds__(32 * RefineShape<CB, FB>::WARPS, 1) refine_kernel(const fbla_k_decode a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  refine_item<CB, FB, QG>(a, smem_raw);
}

template <int QG>
__global__ void __launch_bounds__(512, 2) merge_kernel(const fbla_k_decode a) {
  merge_item<QG>(a, nullptr);
}

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

// the coarse kernel of a deal and a shape (a.deal, a.deep), its threads and shared memory
struct CoarseBuild { void (*kernel)(const fbla_k_decode); int threads; size_t smem; };
template <int CB, int FB, int QG, int SHAPE> CoarseBuild coarse_build(int deal) {
  return CoarseBuild{deal == FBLA_K_DEAL_LENGTHS ? coarse_kernel<CB, FB, QG, FBLA_K_DEAL_LENGTHS, SHAPE>
                     : deal == FBLA_K_DEAL_FIXED ? coarse_kernel<CB, FB, QG, FBLA_K_DEAL_FIXED, SHAPE> : coarse_kernel<CB, FB, QG, FBLA_K_DEAL_COST, SHAPE>,
                     32 * CoarseShape<CB, SHAPE>::TOTAL, sizeof(CoarseSmem<CB, SHAPE>)};
}
template <int CB, int FB, int QG> CoarseBuild coarse_build(int deal, int deep) {
  return deep ? coarse_build<CB, FB, QG, DEEP>(deal) : coarse_build<CB, FB, QG, WIDE>(deal);
}

constexpr int REFINE_SMEM_MAX = 220 * 1024;  // dynamic shared memory of the refine pass (its ring + the slice prefix + the first heads' row sets)
template <int CB, int FB> size_t refine_smem(const fbla_k_decode &a) {
  return (sizeof(RefineWarp<CB, FB>) + (a.refine_fold ? REFINE_SET_BYTES : 0)) * RefineShape<CB, FB>::WARPS + refine_prefix_bytes((size_t)a.batch * a.kv_heads * a.vg * a.nslices);
}
template <int CB, int FB, int QG> cudaError_t launch_all(const fbla_k_decode &a, cudaStream_t stream) {
  const int vheads = a.batch * a.kv_heads * a.vg;
  const size_t rsm = refine_smem<CB, FB>(a);
  static thread_local int configured[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaSuccess;
    for (const int deal : {FBLA_K_DEAL_LENGTHS, FBLA_K_DEAL_FIXED, FBLA_K_DEAL_COST})
      for (const int deep : {0, 1}) {
        const CoarseBuild c = coarse_build<CB, FB, QG>(deal, deep);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(c.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
      }
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(refine_kernel<CB, FB, QG>, cudaFuncAttributeMaxDynamicSharedMemorySize, REFINE_SMEM_MAX);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = 1;
  }
  if (rsm > REFINE_SMEM_MAX) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (a.phase != 2) {
    const CoarseBuild c = coarse_build<CB, FB, QG>(a.deal, a.deep);
    e = launch(true, 1, c.kernel, dim3(a.coarse_ctas), c.threads, c.smem, stream, a);
    if (e == cudaSuccess) e = launch(true, 1, select_kernel<QG>, dim3(a.phase == 1 ? 1 : a.nslices, vheads), 256, 0, stream, a);
    if (a.phase == 1) return e;
  } else {
    select_kernel<QG><<<dim3(a.nslices, vheads), 256, 0, stream>>>(a);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = launch(true, 1, refine_kernel<CB, FB, QG>, dim3(a.refine_ctas), 32 * RefineShape<CB, FB>::WARPS, rsm, stream, a);
  if (e == cudaSuccess) e = launch(true, 1, merge_kernel<QG>, dim3(vheads * QG), 512, 0, stream, a);
  return e;
}

// one pass alone, as an ordinary launch (no overlap with its neighbours): for measurements pass by pass
template <int CB, int FB, int QG> cudaError_t launch_one(const fbla_k_decode &a, int pass, cudaStream_t stream) {
  const int vheads = a.batch * a.kv_heads * a.vg;
  const size_t rsm = refine_smem<CB, FB>(a);
  if (rsm > REFINE_SMEM_MAX) return cudaErrorInvalidValue;
  switch (pass) {
    case 0: {
      const CoarseBuild c = coarse_build<CB, FB, QG>(a.deal, a.deep);
      c.kernel<<<a.coarse_ctas, c.threads, c.smem, stream>>>(a);
      break;
    }
    case 1: select_kernel<QG><<<dim3(a.nslices, vheads), 256, 0, stream>>>(a); break;
    case 2: refine_kernel<CB, FB, QG><<<a.refine_ctas, 32 * RefineShape<CB, FB>::WARPS, rsm, stream>>>(a); break;
    case 3: merge_kernel<QG><<<vheads * QG, 512, 0, stream>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int CB, int FB, int QG> cudaError_t passes_of(const fbla_k_decode &a, fbla_k_pass *p) {
  const int vheads = a.batch * a.kv_heads * a.vg;
  const size_t rsm = refine_smem<CB, FB>(a) + 128;
  if (rsm - 128 > REFINE_SMEM_MAX) return cudaErrorInvalidValue;
  char e[96];
  const CoarseBuild c = coarse_build<CB, FB, QG>(a.deal, a.deep);
  snprintf(e, sizeof e, "fbla::coarse_item<%d, %d, %d, %d, %d>", CB, FB, QG, (int)a.deal, (int)a.deep);
  cudaError_t st = pass_of(c.kernel, a.coarse_ctas, 1, c.threads, c.smem + 128, e, p + 0);
  snprintf(e, sizeof e, "fbla::select_item<%d>", QG);
  if (st == cudaSuccess) st = pass_of(select_kernel<QG>, a.nslices, vheads, 256, 0, e, p + 1);
  snprintf(e, sizeof e, "fbla::refine_item<%d, %d, %d>", CB, FB, QG);
  if (st == cudaSuccess) st = pass_of(refine_kernel<CB, FB, QG>, a.refine_ctas, 1, 32 * RefineShape<CB, FB>::WARPS, rsm, e, p + 2);
  snprintf(e, sizeof e, "fbla::merge_item<%d>", QG);
  if (st == cudaSuccess) st = pass_of(merge_kernel<QG>, vheads * QG, 1, 512, 0, e, p + 3);
  return st;
}

// a row's shares summed over the shards -> the BF16 output
__global__ void __launch_bounds__(128) combine_kernel(const float *partial, uint16_t *out) {
  const float *p = partial + (size_t)blockIdx.x * PSTRIDE;
  out[(size_t)blockIdx.x * D + threadIdx.x] = f32_to_bf16(__fdividef(p[threadIdx.x], p[D]));
}

// R_total[i] = log2 sum_s 2^(mass[s][i]) over the shards (masses of -inf contribute nothing)
__global__ void __launch_bounds__(128) total_mass_kernel(const float *mass, float *total, int shards, int rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows) return;
  float mx = -INFINITY;
  for (int s = 0; s < shards; ++s) mx = fmaxf(mx, mass[(size_t)s * rows + i]);
  float sum = 0.f;
  for (int s = 0; s < shards; ++s) { const float m = mass[(size_t)s * rows + i]; if (m != -INFINITY) sum += ex2(m - mx); }
  total[i] = mx + lg2(sum);
}

}  // namespace fbla

extern "C" cudaError_t fbla_k_total_mass_launch(const float *mass, float *total, int shards, int rows, cudaStream_t stream) {
  fbla::total_mass_kernel<<<(rows + 127) / 128, 128, 0, stream>>>(mass, total, shards, rows);
  return cudaGetLastError();
}

extern "C" cudaError_t fbla_k_combine_launch(const float *partial, uint16_t *out, int rows, cudaStream_t stream) {
  fbla::combine_kernel<<<rows, 128, 0, stream>>>(partial, out);
  return cudaGetLastError();
}

extern "C" long long fbla_k_refine_entry_limit(int cb, int fold) {
  using namespace fbla;
  const size_t ring = cb == 3 ? sizeof(RefineWarp<3, 3>) * RefineShape<3, 3>::WARPS : sizeof(RefineWarp<4, 2>) * RefineShape<4, 2>::WARPS;
  const size_t sets = fold ? REFINE_SET_BYTES * RefineShape<4, 2>::WARPS : 0;
  static_assert(REFINE_SMEM_MAX % 16 == 0 && REFINE_SET_BYTES % 16 == 0 && sizeof(RefineWarp<3, 3>) % 16 == 0 && sizeof(RefineWarp<4, 2>) % 16 == 0, "the prefix may fill its room");
  return (long long)((REFINE_SMEM_MAX - ring - sets) / sizeof(int)) - 1;
}

extern "C" cudaError_t fbla_k_decode_shape(fbla_k_decode *a) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  a->coarse_ctas = sms;
  a->coarse_warps = fbla::CoarseShape<4, fbla::WIDE>::TOTAL;  // (the larger of the two shapes: what the scratch is sized for)
  a->refine_ctas = sms;
  a->refine_warps = fbla::RefineShape<4, 2>::WARPS;
  return cudaSuccess;
}

// How the coarse CTAs' warps share the work (see split_of, deal_of), from the tokens a row has at most:
//   by the lengths when the BF16 windows would get three eighths of a CTA's warps or more (contexts up to about 4 700 tokens);
//   else all warps but one stream and one serves windows, or every warp has an equal cost share of windows and groups --
//   whichever leaves an eighth of a CTA fewer groups (whole groups), with 5 % against the deal by cost: a CTA whose every
//   warp streams runs a group that much slower. Measured on B200 with the eight warps of the deep shape, by cost against seven + one:
//   batch 1 x 128K tokens 80.0 -> 75.3 us per step in 3+3 and 65.7 -> 61.6 in 4+2 (7 groups per warp instead of 8), batch 64 x 1K..64K
//   2.07 -> 2.02 ms, but batch 8 x 16K 120.0 -> 123.9 (8 groups per warp either way). With the twelve warps of the wide shape, fixed
//   split / by cost: 1 x 128K 3+3 73.8 / 62.8, 1 x 512K 149 / 138, 8 x 128K 276 / 262; where the choice falls on the slower of the two
//   it costs up to 8 % (2 x 50 000, 4+2: 55.6 / 59.9).
// And the shape. A group takes a warp 1.4 times as long among twelve as among eight, so the wide shape pays where it leaves a warp less
// than three quarters of the groups (whole groups); with several queries and one or two groups per warp its shallower look-ahead costs more
// than that. Measured wide / deep, us per step, one sweep, N(0, 1), by (groups per warp deep, wide): 4+2 1 x 60 000 (4, 3) 46.9 / 41.6;
// 1 x 150 000 (8, 6) 71.2 / 61.3; 1 x 20 000 (2, 1) 44.2 / 41.4, with one query per head 31.2 / 32.6; 3+3 1 x 128K (7, 5) 62.5 / 63.5; 1 x 266 667
// (15, 10) 92.3 / 100.8; 2 x 66 667 (8, 5) 104 / 114. (Eight warps as they were before the pair's sub-blocks shared the score products'
// columns: 1 x 60 000 43.7, 1 x 150 000 63.4, 1 x 266 667 102.5.)
extern "C" void fbla_k_decode_split(fbla_k_decode *a, long long tokens) {
  constexpr int total = 8;  // (the choice is made in eighths of a CTA)
  const long long groups = (tokens + fbla::G - 1) / fbla::G, S = groups > 2 ? groups - 2 : 0;
  const long long W = groups <= 1 ? (tokens + fbla::S - 1) / fbla::S : 2 * fbla::SBG;  // (a full open window: the choice is monotone in tokens)
  const bool by_lengths = S == 0 || (2 * total * W + S + W) / (2 * (S + W)) >= 3;
  const long long heads = (long long)a->batch * a->kv_heads * a->vg, ctas = a->coarse_ctas > 0 ? a->coarse_ctas : 148;
  // groups an eighth of a CTA takes: seven eighths streaming; by cost (deal_of's share, a whole number of groups)
  const long long fixed = (heads * S + ctas * (total - 1) - 1) / (ctas * (total - 1));
  const long long cost = (fbla::GROUP_COST * heads * S + fbla::WINDOW_COST * heads * W + fbla::GROUP_COST * ctas * total - 1) / (fbla::GROUP_COST * ctas * total);
  a->deal = by_lengths ? FBLA_K_DEAL_LENGTHS : 21 * cost < 20 * fixed ? FBLA_K_DEAL_COST : FBLA_K_DEAL_FIXED;
  auto per_warp = [&](int warps) {  // groups of a streaming warp in a shape of `warps`
    const long long share = a->deal == FBLA_K_DEAL_COST ? fbla::GROUP_COST * ctas * warps : ctas * (warps - 1);
    const long long units = a->deal == FBLA_K_DEAL_COST ? fbla::GROUP_COST * heads * S + fbla::WINDOW_COST * heads * W : heads * S;
    return (units + share - 1) / share;
  };
  constexpr int eight = fbla::CoarseShape<4, fbla::DEEP>::TOTAL, twelve = fbla::CoarseShape<4, fbla::WIDE>::TOTAL;
  a->deep = 3 * per_warp(eight) <= 4 * per_warp(twelve) || 2 * per_warp(twelve) <= a->qg;
  a->coarse_warps = a->deep ? eight : twelve;
  // Folding the warps' partial rows per CTA costs the coarse pass a barrier and a few microseconds at its very end and saves
  // the later passes their walk over the rows: it pays when a virtual head is spread over many warps, i.e. when there are
  // few heads (measured on B200: batch 1 x 8 KV heads at 128K tokens -4.5 us per step, batch 8 x 8 heads at 16K +3 us).
  a->fold = !by_lengths && a->batch * a->kv_heads * a->vg <= 32;
}

extern "C" void fbla_k_decode_split_of(int cb, int batch, int kv_heads, int vg, long long tokens, int *deal, int *fold) {
  fbla_k_decode a = {};
  a.cb = cb; a.batch = batch; a.kv_heads = kv_heads; a.vg = vg;
  a.coarse_ctas = 148;  // (the shape of a B200; a caller with a device takes it from fbla_k_decode_shape)
  fbla_k_decode_split(&a, tokens);
  *deal = a.deal;
  *fold = a.fold;
}

extern "C" int fbla_k_decode_deep_of(int batch, int kv_heads, int vg, int qg, long long tokens) {
  fbla_k_decode a = {};
  a.cb = 4; a.batch = batch; a.kv_heads = kv_heads; a.vg = vg; a.qg = qg;
  a.coarse_ctas = 148;
  fbla_k_decode_split(&a, tokens);
  return a.deep;
}

extern "C" cudaError_t fbla_k_decode_launch(const fbla_k_decode *a, cudaStream_t stream) {
  if (a->dense) return fbla_k_dense_launch(a, stream);
  using namespace fbla;
  if (a->cb == 3) {
    switch (a->qg) {
      case 1: return launch_all<3, 3, 1>(*a, stream);
      case 2: return launch_all<3, 3, 2>(*a, stream);
      default: return launch_all<3, 3, 4>(*a, stream);
    }
  }
  switch (a->qg) {
    case 1: return launch_all<4, 2, 1>(*a, stream);
    case 2: return launch_all<4, 2, 2>(*a, stream);
    default: return launch_all<4, 2, 4>(*a, stream);
  }
}

// (after one whole fbla_k_decode_launch on this device: that call sets the kernels' shared-memory attributes)
extern "C" cudaError_t fbla_k_decode_pass_launch(const fbla_k_decode *a, int pass, cudaStream_t stream) {
  if (a->dense) return fbla_k_dense_pass_launch(a, pass, stream);
  using namespace fbla;
  if (a->cb == 3) {
    switch (a->qg) {
      case 1: return launch_one<3, 3, 1>(*a, pass, stream);
      case 2: return launch_one<3, 3, 2>(*a, pass, stream);
      default: return launch_one<3, 3, 4>(*a, pass, stream);
    }
  }
  switch (a->qg) {
    case 1: return launch_one<4, 2, 1>(*a, pass, stream);
    case 2: return launch_one<4, 2, 2>(*a, pass, stream);
    default: return launch_one<4, 2, 4>(*a, pass, stream);
  }
}

extern "C" cudaError_t fbla_k_decode_passes(const fbla_k_decode *a, fbla_k_pass info[4]) {
  if (a->dense) return fbla_k_dense_passes(a, info);
  using namespace fbla;
  if (a->cb == 3) {
    switch (a->qg) {
      case 1: return passes_of<3, 3, 1>(*a, info);
      case 2: return passes_of<3, 3, 2>(*a, info);
      default: return passes_of<3, 3, 4>(*a, info);
    }
  }
  switch (a->qg) {
    case 1: return passes_of<4, 2, 1>(*a, info);
    case 2: return passes_of<4, 2, 2>(*a, info);
    default: return passes_of<4, 2, 4>(*a, info);
  }
}
