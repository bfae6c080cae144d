// FBLA compressed-KV decode for sm_100a in two sweeps: every sub-block's scores, then every sub-block's values once.
//
//   * The score pass reads only the K half of the records, both planes (straight into registers, no staging), forms every
//     sub-block's coarse and full scores, its log2 mass and its integer weights p = round(255 * 2^(s - max)) under both, which it
//     leaves in the scratch (16 bytes per sub-block, query and set, beside the block maximum), and the rows' running (m, l); it
//     also serves the BF16 windows.
//   * The value pass knows every row's mass R before it starts, so it knows which (query, sub-block) pairs are selected. It
//     reads the V half of the coarse records, of the fine records where some query selected the sub-block, takes the weights
//     that the selection asks for and accumulates each sub-block once, in units of 2^-R -- no scores, no running maximum, no
//     correction of a coarse sum, no item list.
// For rows whose sub-blocks are mostly selected (fbla_k_two_sweeps); the decode of fbla_decode.cuh serves the others.
// Both passes put the columns of several sub-blocks into one product's eight columns (queries of sub-block b in columns
// b QG ..; its A fragments meet a B operand that is zero elsewhere, and all add into the same accumulators), so the softmax
// arithmetic runs once per eight (sub-block, query) columns on full warps. Semantics, formats and the definition of every
// number are fbla_decode.cuh's; only the order of the sums differs.
// Work is dealt in contiguous runs of the flattened (virtual head, group, piece of a group) list: first to CTAs, then to
// the CTA's warps, so that a head's partial rows are one per CTA, folded in warp order (reproducible bit for bit). Short rows: every head
// has CTAs of its own, and one kernel does both passes and the output rows (head_passes).
// Bound by latency: four warps per scheduler issue 0.44 to 0.5 instructions per cycle, waiting for loads and for their own results.
#pragma once
#include "fbla_decode.cuh"

namespace fbla {
namespace dense {

constexpr int SCORE_WARPS = FBLA_K_TWO_SCORE_WARPS, VALUE_WARPS = FBLA_K_TWO_VALUE_WARPS;
constexpr int MAX_BATCH = FBLA_K_DENSE_MAX_BATCH;
constexpr int PAIRS = SBG / 2;   // pairs of sub-blocks per group: the value pass's unit
// a window sub-block's time in the score pass, in pieces of a group (8 / QG sub-blocks: 1 / QG of the group)
template <int QG> __host__ __device__ constexpr int window_cost() { return QG == 4 ? 3 : QG; }

// ---- where the flattened lists begin for every batch row ------------------------------------------------------------------
// Rows of one length: closed forms. Per-row lengths: prefix sums over the batch, in shared memory.
struct Table {
  int closed[MAX_BATCH + 1], exact[MAX_BATCH + 1];  // sums of the rows before b (units of one virtual head)
  int warp_sum[2][32];
};
// (all threads of the CTA; ends with a barrier)
__device__ __forceinline__ void build_table(const fbla_k_decode &a, Table &t, int threads) {
  const int tid = FBLA_POS::tid(), lane = tid & 31, warp = tid >> 5;
  if (!a.lstride) return;
  int base0 = 0, base1 = 0;
  for (int b0 = 0; b0 < a.batch; b0 += threads) {
    const int b = b0 + tid;
    int v0 = 0, v1 = 0;
    if (b < a.batch) { const Row r = row_of(a, b); v0 = r.closed; v1 = r.exact; }
    int s0 = v0, s1 = v1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y0 = __shfl_up_sync(FULL, s0, o), y1 = __shfl_up_sync(FULL, s1, o);
      if (lane >= o) { s0 += y0; s1 += y1; }
    }
    if (lane == 31) { t.warp_sum[0][warp] = s0; t.warp_sum[1][warp] = s1; }
    __syncthreads();
    int p0 = base0, p1 = base1;
    for (int w = 0; w < threads / 32; ++w) {
      const int q0 = t.warp_sum[0][w], q1 = t.warp_sum[1][w];
      if (w < warp) { p0 += q0; p1 += q1; }
      base0 += q0; base1 += q1;
    }
    if (b < a.batch) { t.closed[b] = p0 + s0 - v0; t.exact[b] = p1 + s1 - v1; }
    __syncthreads();
  }
  if (tid == 0) { t.closed[a.batch] = base0; t.exact[a.batch] = base1; }
  __syncthreads();
}
// a head's units in one of the lists: its first (flattened over all heads) and their number
struct Span { int off, n; };
template <bool EXACT> __device__ __forceinline__ Span span_of(const fbla_k_decode &a, const int *prefix, int hpr, int b, int hir) {
  Span s;
  s.n = units_of<EXACT>(row_of(a, b));
  s.off = (a.lstride ? hpr * prefix[b] : b * hpr * s.n) + hir * s.n;
  return s;
}
template <bool EXACT> __device__ __forceinline__ int total_of(const fbla_k_decode &a, const int *prefix, int hpr) {
  return hpr * (a.lstride ? prefix[a.batch] : a.batch * units_of<EXACT>(row_of(a, 0)));
}
// the cursor of flattened unit u
template <bool EXACT> __device__ __forceinline__ Cursor find(const fbla_k_decode &a, const int *prefix, int hpr, int u) {
  Cursor c;
  int off;
  if (a.lstride) {
    int l = 0, h = a.batch;  // prefix[l] hpr <= u < prefix[h] hpr
    while (h - l > 1) { const int mid = (l + h) >> 1; if (prefix[mid] * hpr <= u) l = mid; else h = mid; }
    c.b = l; c.n = prefix[l + 1] - prefix[l];
    off = u - prefix[l] * hpr;
  } else {
    c.n = units_of<EXACT>(row_of(a, 0));
    c.b = u / (hpr * c.n);
    off = u - c.b * hpr * c.n;
  }
  c.hir = off / c.n;
  c.i = off - c.hir * c.n;
  return c;
}

// Where every virtual head has CTAs of its own (a.head_ctas of them: the grid is CTAs x heads of a batch row x batch rows): the head of this
// item's CTA, and the CTA's rank among the head's. `slot`: the CTA's number among all.
struct Own {
  int ctas, rank, hir, b, vh, slot;
  Row row;
  __device__ __forceinline__ explicit Own(const fbla_k_decode &a) : ctas(FBLA_POS::nx()), rank(FBLA_POS::x()), hir(FBLA_POS::y()), b(FBLA_POS::z()) {
    vh = b * (int)FBLA_POS::ny() + hir;
    slot = vh * ctas + rank;
    row = row_of(a, b);
  }
};
// the KV head of virtual head vh
__device__ __forceinline__ int kv_of(const fbla_k_decode &a, int vh) { return a.vg == 1 ? vh : vh / a.vg; }

// ---- scratch (`lse`; the rest inside the decode's `part` and `dpart` arrays) -----------------------------------------------------------------
// Window chunks: the flattened window sub-blocks in runs of `run`; chunk c leaves one (m, l, o) row per virtual head it meets, at
// slot c + vh. Value rows (o, l in units of 2^-R) and the score pass's (m, l) pairs: one per (CTA, virtual head), slot cta + vh.
__device__ __forceinline__ int window_run(const fbla_k_decode &a, int total) { return max(1, (total + a.coarse_ctas * SCORE_WARPS - 1) / (a.coarse_ctas * SCORE_WARPS)); }
__device__ __forceinline__ float *window_row(const fbla_k_decode &a, int slot) { return a.part + (size_t)slot * a.qg * PSTRIDE; }
__device__ __forceinline__ float *value_row(const fbla_k_decode &a, int slot) {
  return a.part + (size_t)(a.coarse_ctas * SCORE_WARPS + a.batch * a.kv_heads * a.vg + slot) * a.qg * PSTRIDE;
}
__device__ __forceinline__ float2 *mass_pair(const fbla_k_decode &a, int slot) {
  return reinterpret_cast<float2 *>(value_row(a, a.coarse_ctas + a.batch * a.kv_heads * a.vg)) + (size_t)slot * a.qg;
}
// prefix sums for the later passes: closed [batch + 1], exact [batch + 1]
__device__ __forceinline__ int *table_of(const fbla_k_decode &a) { return reinterpret_cast<int *>(mass_pair(a, a.coarse_ctas + a.batch * a.kv_heads * a.vg)); }

// lse: per cell (virtual head, sub-block, query) the log2 mass; behind it, per set of weights (0 coarse, 1 full), the block maxima,
// and then the sets' weights, 16 bytes per cell. (fbla_k_two_cells: cells, padded.)
__device__ __forceinline__ size_t cells_of(const fbla_k_decode &a) { return fbla_k_two_cells((size_t)a.batch * a.kv_heads * a.vg, a.nblocks, a.qg); }
__device__ __forceinline__ uint32_t *weights_of(const fbla_k_decode &a) { return reinterpret_cast<uint32_t *>(a.lse) + 3 * cells_of(a); }

// ---- quantisation of the virtual head's queries for one group (as quantize_query_word), into QG rows of qst, QST_ROW bytes apart ----
// am: the queries' max |z| (the same in every lane); dot: the lane's share of the result of a butterfly that hands half of the
// queries on in each of its first steps: q . base of query dot_query(lane).
template <int QG> __device__ __forceinline__ int dot_lane(int q) { return QG == 4 ? ((q >> 1) << 4) | ((q & 1) << 3) : QG == 2 ? q << 4 : 0; }
template <int QG>
__device__ __forceinline__ void quantize_group(uint4 km, const uint2 (&q)[QG], uint8_t *qst, int lane, float (&am)[QG], float &dot) {
  const float2 b0 = make_float2(bf_lo(km.x), bf_hi(km.x)), b1 = make_float2(bf_lo(km.y), bf_hi(km.y));
  const float2 s0 = make_float2(bf_lo(km.z), bf_hi(km.z)), s1 = make_float2(bf_lo(km.w), bf_hi(km.w));
  float d[QG];
#pragma unroll
  for (int i = 0; i < QG; ++i) {
    const float2 x0 = make_float2(bf_lo(q[i].x), bf_hi(q[i].x)), x1 = make_float2(bf_lo(q[i].y), bf_hi(q[i].y));
    const float2 z0 = __fmul2_rn(x0, s0), z1 = __fmul2_rn(x1, s1), t = __ffma2_rn(x1, b1, __fmul2_rn(x0, b0));
    d[i] = t.x + t.y;
    am[i] = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(max3_abs(max3_abs(z0.x, z0.y, z1.x), z1.y, z1.y))));
    const float2 r = splat(quotient_127(am[i])), mg = splat(MAGICF);
    const float2 c0 = __ffma2_rn(z0, r, mg), c1 = __ffma2_rn(z1, r, mg);
    reinterpret_cast<uint32_t *>(qst + QST_ROW * i)[lane] =
        __byte_perm(__byte_perm(__float_as_uint(c0.x), __float_as_uint(c0.y), 0x0040), __byte_perm(__float_as_uint(c1.x), __float_as_uint(c1.y), 0x0040), 0x5410);
  }
  int o = 16;
#pragma unroll
  for (int w = QG / 2; w; w >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < w; ++i) d[i] = (up ? d[i + w] : d[i]) + __shfl_xor_sync(FULL, up ? d[i] : d[i + w], o);
  }
#pragma unroll
  for (; o; o >>= 1) d[0] += __shfl_xor_sync(FULL, d[0], o);
  dot = d[0];
}

// ---- score pass -----------------------------------------------------------------------------------------------------------------
// K words of one sub-block in registers: what thread (gid, tig) supplies to the products, for tokens gid and gid + 8.
// 4 and 2 bits: the thread's slots are 4 t + i and 8 + 4 t + i (i = 0..3, t = tig % 2) of channel half tig / 2, so that a token's words
// come in 16-byte pieces (2 bits: both t read the same piece). 3 bits: the thread's words are W[2 t], W[2 t + 1] and W[4 + t] of half tig / 2:
// slots 2 t, + 1, 6 + 2 t, + 1, 12 + 2 t, + 1, 4 + t and 10 + t, whole. (Every thread on W[tig] of both halves took two words and twice the
// loads more; with the values' tails in shared memory: 32 sequences of 300 to 6 000 tokens 82.5 -> 75.8 us, 16 / 8 heads 16 x 4 000 54.2 -> 43.9.)
template <int BITS> struct KWords {
  uint4 a, a8;
  static __device__ __forceinline__ int offset(int gid, int tig) { return (BITS == 4 ? 512 * (tig & 1) : 0) + 256 * (tig >> 1) + 16 * gid; }
  __device__ __forceinline__ void load(const uint8_t *p, int) {  // p: the record + offset
    a = __ldg(reinterpret_cast<const uint4 *>(p));
    a8 = __ldg(reinterpret_cast<const uint4 *>(p + 128));
  }
};
template <> struct KWords<3> {
  uint2 a, a8;      // W[2 t], W[2 t + 1] of tokens gid and gid + 8
  uint32_t e, e8;   // W[4 + t]
  static __device__ __forceinline__ int offset(int gid, int tig) { return 256 * (tig >> 1) + 16 * gid + 8 * (tig & 1); }
  static __device__ __forceinline__ int tail(int tig) { return 1024 + 8 * (tig >> 1) + 4 * (tig & 1) - 256 * (tig >> 1) - 8 * (tig & 1); }  // from there to W[4 + t]
  __device__ __forceinline__ void load(const uint8_t *p, int tail) {
    a = __ldg(reinterpret_cast<const uint2 *>(p)); a8 = __ldg(reinterpret_cast<const uint2 *>(p + 128));
    e = __ldg(reinterpret_cast<const uint32_t *>(p + tail)); e8 = __ldg(reinterpret_cast<const uint32_t *>(p + tail + 128));
  }
};
// the qhat words matching KWords
template <int CB> __device__ __forceinline__ void score_frag(const uint8_t *qst, int row, int tig, uint32_t (&B)[8]) {
  if (CB == 4) {  // slots 4 t + i, then 8 + 4 t + i, of half tig / 2
    const uint8_t *p = qst + QST_ROW * row + 64 * (tig >> 1) + 16 * (tig & 1);
    const uint4 lo = lds128(p), hi = lds128(p + 32);
    B[0] = lo.x; B[1] = lo.y; B[2] = lo.z; B[3] = lo.w; B[4] = hi.x; B[5] = hi.y; B[6] = hi.z; B[7] = hi.w;
  } else {
    const uint8_t *p = qst + QST_ROW * row + 64 * (tig >> 1) + 8 * (tig & 1), *r = p - 4 * (tig & 1);
    const uint2 x = lds64(p), y = lds64(p + 24), z = lds64(p + 48);
    B[0] = x.x; B[1] = x.y; B[2] = y.x; B[3] = y.y; B[4] = z.x; B[5] = z.y; B[6] = lds32(r + 16); B[7] = lds32(r + 40);
  }
}
// The sub-block's products, in accumulators of the low and of the high class (times 16, 3 bits: 8): set (FIRST) or added to.
template <bool FIRST> __device__ __forceinline__ void mma_step(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (FIRST) mma_u8s8_k32_from(d, a0, a1, a2, a3, b0, b1, MAGIC);
  else mma_u8s8_k32(d, a0, a1, a2, a3, b0, b1);
}
template <int BITS, bool FIRST>
__device__ __forceinline__ void score_products(const KWords<BITS> &k, const uint32_t (&b)[8], int tig, uint32_t (&lo)[4], uint32_t (&hi)[4]) {
  if constexpr (BITS != 3) {
    constexpr uint32_t L = BITS == 4 ? 0x0f0f0f0fu : 0x03030303u, H = L << 4;
    const int sh = BITS == 2 ? 2 * (tig & 1) : 0;
    const uint4 a = BITS == 2 ? make_uint4(k.a.x >> sh, k.a.y >> sh, k.a.z >> sh, k.a.w >> sh) : k.a;
    const uint4 a8 = BITS == 2 ? make_uint4(k.a8.x >> sh, k.a8.y >> sh, k.a8.z >> sh, k.a8.w >> sh) : k.a8;
    mma_step<FIRST>(lo, a.x & L, a8.x & L, a.y & L, a8.y & L, b[0], b[1]);
    mma_step<FIRST>(hi, a.x & H, a8.x & H, a.y & H, a8.y & H, b[4], b[5]);
    mma_u8s8_k32(lo, a.z & L, a8.z & L, a.w & L, a8.w & L, b[2], b[3]);
    mma_u8s8_k32(hi, a.z & H, a8.z & H, a.w & H, a8.w & H, b[6], b[7]);
  } else {
    constexpr uint32_t L = 0x07070707u, M = 0x38383838u, T2 = 0x03030303u, T1 = 0x04040404u;
    mma_step<FIRST>(lo, k.a.x & L, k.a8.x & L, k.a.y & L, k.a8.y & L, b[0], b[1]);
    mma_step<FIRST>(hi, k.a.x & M, k.a8.x & M, k.a.y & M, k.a8.y & M, b[2], b[3]);
    mma_u8s8_k32(lo, ((k.a.x >> 6) & T2) | ((k.e >> 4) & T1), ((k.a8.x >> 6) & T2) | ((k.e8 >> 4) & T1),
                 ((k.a.y >> 6) & T2) | ((k.e >> 5) & T1), ((k.a8.y >> 6) & T2) | ((k.e8 >> 5) & T1), b[4], b[5]);
    mma_u8s8_k32(lo, k.e & L, k.e8 & L, (k.e >> 3) & L, (k.e8 >> 3) & L, b[6], b[7]);
  }
}

struct ScoreWarp {
  union {
    ExactWarp exact;
    struct {
      uint8_t qst[4 * QST_ROW];
      uint8_t pst[2][128];  // P bytes of a unit, coarse and full: [column][16 tokens]
    } s;
  };
};
struct ScoreFold {
  float2 stage[SCORE_WARPS][2][4];  // (m, l) of the first and the last virtual head of a warp's run
  int stage_vh[SCORE_WARPS][2];
  float2 window[SCORE_WARPS][4];    // a head's own CTAs: (m, l) of the warp's window sub-block
};
struct __align__(16) ScoreSmem {
  ScoreWarp w[SCORE_WARPS];
  ScoreFold fold;
  Table table;
};
struct __align__(16) HeadScoreSmem { ScoreWarp w[SCORE_WARPS]; ScoreFold fold; };

__device__ __forceinline__ float2 merge_mass(float2 x, float2 y) {  // (m, l) pairs; symmetric in its arguments up to the order of one sum
  const float m = fmaxf(x.x, y.x), by = m == -FBLA_INF ? 0.f : m;  // (nothing on either side: 2^-inf = 0)
  return make_float2(m, x.y * ex2(x.x - by) + y.y * ex2(y.x - by));
}

// lane l's pair becomes that of query l % QG over all lanes
template <int QG> __device__ __forceinline__ float2 merge_lanes(float2 acc, int lane) {
#pragma unroll
  for (int o = QG; o < 32; o <<= 1) {
    const float2 y = make_float2(__shfl_xor_sync(FULL, acc.x, o), __shfl_xor_sync(FULL, acc.y, o));
    acc = (lane & o) ? merge_mass(y, acc) : merge_mass(acc, y);
  }
  return acc;
}

// The CTA's share of the score pass: pieces of groups (units of NB sub-blocks) [first, first + count) and window chunk
// numbers [chunk, chunk + chunks); warp w of the CTA takes chunk number w and the run [lo, hi) of the pieces.
template <int QG>
__device__ __forceinline__ void score_item_units(int ctas, int cta, int total, int x_total, int run, int warp, int &chunk, int &lo, int &hi) {
  const int per = (total + ctas - 1) / ctas, first = min(total, cta * per), count = min(total, first + per) - first;
  const int chunks = (x_total + run - 1) / run, cper = (chunks + ctas - 1) / ctas, c0 = min(chunks, cta * cper), nc = min(chunks, c0 + cper) - c0;
  chunk = warp < nc ? c0 + warp : -1;
  // a chunk's cost in pieces; a warp with a chunk takes that many pieces fewer
  const int cost = run * window_cost<QG>();
  int with = 0, without = (count + SCORE_WARPS - 1) / SCORE_WARPS;
  if (nc > 0) {
    const int p = (cost * nc + count + SCORE_WARPS - 1) / SCORE_WARPS;
    if (p > cost) { with = p - cost; without = p; }
    else { with = nc == SCORE_WARPS ? (count + SCORE_WARPS - 1) / SCORE_WARPS : 0; without = nc < SCORE_WARPS ? (count + SCORE_WARPS - nc - 1) / (SCORE_WARPS - nc) : 0; }
  }
  const int at = warp < nc ? warp * with : nc * with + (warp - nc) * without;
  lo = first + min(count, at);
  hi = first + min(count, at + (warp < nc ? with : without));
}

// What the CTAs of one head hand on, in a plan's passes: through the scratch
template <int QG> struct ScratchVia {
  const fbla_k_decode &a;
  int ctas, vh, slot;
  __device__ __forceinline__ explicit ScratchVia(const fbla_k_decode &a_) : a(a_) { const Own own(a); ctas = own.ctas; vh = own.vh; slot = own.slot; }
  __device__ __forceinline__ ScratchVia(const fbla_k_decode &a_, int vh_) : a(a_), ctas(a_.head_ctas), vh(vh_), slot(0) {}
  __device__ __forceinline__ void ready() const {}
  __device__ __forceinline__ float *window(int x) const { return window_row(a, vh * SCORE_WARPS + x + vh); }  // the head's window sub-block x: [QG][PSTRIDE]
  // the CTA's (m, l) of query lane % QG
  __device__ __forceinline__ void put_mass(float2 mass, int lane) const { if (lane < QG) mass_pair(a, slot + vh)[lane] = mass; }
  __device__ __forceinline__ float2 mass(int cta, int q) const { return __ldcg(mass_pair(a, vh * ctas + cta + vh) + q); }
  // the CTA's sum of query q, channel ch (D: l), and that of CTA cta
  __device__ __forceinline__ void put(int q, int ch, float x) const { value_row(a, slot + vh)[q * PSTRIDE + ch] = x; }
  __device__ __forceinline__ float sum(int cta, int q, int ch) const { return __ldcg(value_row(a, vh * ctas + cta + vh) + q * PSTRIDE + ch); }
};
struct NoVia { __device__ __forceinline__ void ready() const {} };

// HEAD: every virtual head has CTAs of its own; else the work is dealt over all CTAs, `table` the batch's prefix sums
// (Via: how the parts of a head's own CTAs hand their results on)
template <int CB, int FB, int QG, bool HEAD, class Via>
__device__ __forceinline__ void score_units(const fbla_k_decode &a, ScoreWarp *ws, ScoreFold &fold, const Table *table, const Via &via) {
  constexpr int NB = 8 / QG, UPG = QG;  // sub-blocks per unit, units per group
  constexpr float HOFF = .5f * ((1 << FB) - 1);
  constexpr int RC = record_bytes(CB), RF = record_bytes(FB);
  const int lane = FBLA_POS::tid() & 31, warp = FBLA_POS::tid() >> 5, gid = lane >> 2, tig = lane & 3;
  const int hpr = HEAD ? (int)FBLA_POS::ny() : a.kv_heads * a.vg;
  int chunk, lo, hi, cta;
  Cursor c{0, 0, 0, 0};
  if constexpr (HEAD) {
    const Own own(a);
    cta = own.slot;
    score_item_units<QG>(own.ctas, own.rank, UPG * own.row.closed, own.row.exact, 1, warp, chunk, lo, hi);
    float2 mass = make_float2(-FBLA_INF, 0.f);
    if (chunk >= 0) {
      float *const row = via.window(chunk);
      exact_range<QG, false>(a, ws[warp].exact, lane, chunk, chunk + 1, Cursor{own.b, own.hir, chunk, own.row.exact}, [&](int) { return row; });
      __syncwarp();
      if (lane < QG) mass = make_float2(row[lane * PSTRIDE + D], row[lane * PSTRIDE + D + 1]);
    }
    if (lane < QG) fold.window[warp][lane] = mass;
    c = Cursor{own.b, own.hir, lo / UPG, own.row.closed};
  } else {
    cta = FBLA_POS::x();
    const int total = UPG * total_of<false>(a, table->closed, hpr), x_total = total_of<true>(a, table->exact, hpr), run = window_run(a, x_total);
    score_item_units<QG>(FBLA_POS::nx(), cta, total, x_total, run, warp, chunk, lo, hi);
    if (chunk >= 0) exact_range<QG, false>(a, ws[warp].exact, lane, chunk * run, min(x_total, (chunk + 1) * run), find<true>(a, table->exact, hpr, chunk * run),
                                             [&](int vh) { return window_row(a, chunk + vh); });
  }
  __syncwarp();
  uint8_t *const qst = ws[warp].s.qst;
  uint8_t (*const pst)[128] = ws[warp].s.pst;

  int first_vh = -1, cur_vh = -1;
  float m[2] = {-FBLA_INF, -FBLA_INF}, l[2] = {0.f, 0.f};  // of the thread's two columns
  // (m, l) of every query of the head into dst[0 .. QG): columns of one query are merged over the threads that hold them
  auto leave = [&](float2 *dst) {
    float2 v[2] = {make_float2(m[0], l[0]), make_float2(m[1], l[1])};
    if (QG == 1) v[0] = merge_mass(v[0], v[1]);
#pragma unroll
    for (int o = QG == 4 ? 2 : 1; o <= 2; o <<= 1)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float2 y = make_float2(__shfl_xor_sync(FULL, v[e].x, o), __shfl_xor_sync(FULL, v[e].y, o));
        v[e] = (lane & o) ? merge_mass(y, v[e]) : merge_mass(v[e], y);
      }
    if (gid == 0) {
      if (QG == 4) { if (tig < 2) { dst[2 * tig] = v[0]; dst[2 * tig + 1] = v[1]; } }
      else if (QG == 2) { if (tig == 0) { dst[0] = v[0]; dst[1] = v[1]; } }
      else if (tig == 0) dst[0] = v[0];
    }
  };
  if (lo < hi) {
    if constexpr (!HEAD) c = find<false>(a, table->closed, hpr, lo / UPG);
    int piece = lo % UPG;
    // Where the next unit's words lie, and the cells of the unit in work: pointers that run on, set anew with every head only.
    const uint8_t *kp, *fp, *mp;
    float *lp;
    uint32_t *wp;
    const size_t n_cells = cells_of(a);
    const long long k_skip = (long long)(a.gs - 1) * SBG * RC, f_skip = (long long)(a.gs - 1) * SBG * RF, m_step = (long long)a.gs * 1024;
    const int k_tail = KWords<3>::tail(tig);
    auto place_records = [&](const Cursor &x, int pc) {
      const size_t unit = (size_t)kv_of(a, x.b * hpr + x.hir) * a.hs + (size_t)group_of(a, x) * a.gs;
      kp = a.c.coarse + (unit * SBG + pc * NB) * RC + KWords<CB>::offset(gid, tig);
      fp = a.c.fine + (unit * SBG + pc * NB) * RF + KWords<FB>::offset(gid, tig);
      mp = reinterpret_cast<const uint8_t *>(a.c.meta) + unit * 1024 + 16 * lane;
    };
    place_records(c, piece);
    uint4 km = __ldg(reinterpret_cast<const uint4 *>(mp));
    KWords<CB> kw[NB];  // the next unit's words
    KWords<FB> kf[NB];
    auto load = [&] {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        kw[b].load(kp + b * RC, k_tail);
        kf[b].load(fp + b * RF, k_tail);
      }
      kp += NB * RC; fp += NB * RF;
    };
    load();
    uint2 q[QG];
    constexpr int SETS = QG == 4 ? 2 : 1;  // (with four queries the two sub-blocks' operands are kept, else formed per sub-block)
    uint32_t B[SETS][8];
    float2 c0 = make_float2(0.f, 0.f), sqc = c0, sqf = c0, qb2 = c0;
    bool fresh = true;  // the group's queries have not been quantised yet
    for (int u = lo; u < hi; ++u) {
      const int vh = c.b * hpr + c.hir;
      if (vh != cur_vh) {
        if (cur_vh >= 0) leave(cur_vh == first_vh ? fold.stage[warp][0] : mass_pair(a, cta + cur_vh));
        else first_vh = vh;
        cur_vh = vh;
        m[0] = m[1] = -FBLA_INF; l[0] = l[1] = 0.f;
        const size_t cell = ((size_t)vh * a.nblocks + (size_t)group_of(a, c) * SBG) * QG + 8 * piece;
        lp = a.lse + cell + 2 * tig;
        wp = weights_of(a) + cell * 4 + lane;
#pragma unroll
        for (int qi = 0; qi < QG; ++qi) q[qi] = __ldg(reinterpret_cast<const uint2 *>(a.q + (size_t)q_row(a, c.b, c.hir, qi) * D) + lane);
      }
      if (fresh) {
        fresh = false;
        __syncwarp();
        float am[QG], dot;
        quantize_group<QG>(km, q, qst, lane, am, dot);
        __syncwarp();
        uint32_t b[8], d[4];
        score_frag<CB>(qst, gid % QG, tig, b);
        // the sums of the codes of the thread's columns: products with an all-ones A
        mma_u8s8_k32_from(d, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, b[0], b[1], MAGIC);
#pragma unroll
        for (int i = 2; i < 8; i += 2) mma_u8s8_k32(d, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, b[i], b[i + 1]);
        const int qa = (2 * tig) % QG, qz = (2 * tig + 1) % QG;  // the columns' queries
        const float2 amax = make_float2(QG == 4 && (tig & 1) ? am[2 % QG] : am[0], QG == 4 && (tig & 1) ? am[3 % QG] : am[1 % QG]);
        sqf = __fmul2_rn(amax, splat(__fmul_rn(a.sl, 1.f / 127.f)));
        qb2 = __fmul2_rn(make_float2(__shfl_sync(FULL, dot, dot_lane<QG>(qa)), __shfl_sync(FULL, dot, dot_lane<QG>(qz))), splat(a.sl));
        sqc = __fmul2_rn(sqf, splat((float)(1 << FB)));
        c0 = __ffma2_rn(__fmul2_rn(sqf, splat(HOFF)), isum2(d[0], d[1]), qb2);
#pragma unroll
        for (int x = 0; x < SETS; ++x)
#pragma unroll
          for (int i = 0; i < 8; ++i) B[x][i] = SETS == 1 || gid / QG == x ? b[i] : 0u;
      }
      constexpr float UC = CB == 4 ? 1.f / 16 : 1.f / 8, UF = FB == 2 ? 1.f / 16 : 1.f / 8;
      uint32_t dl[4], dh[4], fl[4], fh[4];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        uint32_t mb[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) mb[i] = SETS == 2 ? B[b % SETS][i] : gid / QG == b ? B[0][i] : 0u;
        if (b == 0) score_products<CB, true>(kw[b], mb, tig, dl, dh); else score_products<CB, false>(kw[b], mb, tig, dl, dh);
        if (b == 0) score_products<FB, true>(kf[b], mb, tig, fl, fh); else score_products<FB, false>(kf[b], mb, tig, fl, fh);
      }
      // the next unit's words, and the next group's metadata with the group's first
      if (++piece == UPG) {
        piece = 0;
        fresh = true;
        if (u + 1 < hi) {
          if (c.i + 1 < c.n) {
            ++c.i;
            kp += k_skip; fp += f_skip; mp += m_step;
          } else {
            advance<false>(a, hpr, c);
            place_records(c, 0);
          }
          km = __ldg(reinterpret_cast<const uint4 *>(mp));
        }
      }
      if (u + 1 < hi) load();
      // code sums of tokens gid (x[0]), gid + 8 (x[1]) of the thread's columns, and from them scores, maxima, weights
      auto softmax = [&](float2 sA, float2 sB, float2 &mb, float2 &pA, float2 &pB, uint8_t *p) {
        mb = make_float2(fmaxf(sA.x, sB.x), fmaxf(sA.y, sB.y));
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) {
          mb.x = fmaxf(mb.x, __shfl_xor_sync(FULL, mb.x, o));
          mb.y = fmaxf(mb.y, __shfl_xor_sync(FULL, mb.y, o));
        }
        const float2 nm = make_float2(-mb.x, -mb.y), dA = __fadd2_rn(sA, nm), dB = __fadd2_rn(sB, nm);
        pA = __ffma2_rn(make_float2(ex2(dA.x), ex2(dA.y)), splat(255.f), splat(MAGICF));
        pB = __ffma2_rn(make_float2(ex2(dB.x), ex2(dB.y)), splat(255.f), splat(MAGICF));
        p += 32 * tig + gid;  // columns 2 tig, 2 tig + 1: 16 bytes apart
        p[0] = (uint8_t)__float_as_uint(pA.x); p[16] = (uint8_t)__float_as_uint(pA.y);
        p[8] = (uint8_t)__float_as_uint(pB.x); p[24] = (uint8_t)__float_as_uint(pB.y);
      };
      const float2 xA = __ffma2_rn(isum2(dh[0], dh[1]), splat(UC), isum2(dl[0], dl[1])), xB = __ffma2_rn(isum2(dh[2], dh[3]), splat(UC), isum2(dl[2], dl[3]));
      float2 mb, pA, pB;
      __syncwarp();  // (the previous unit's bytes have been read)
      softmax(__ffma2_rn(sqc, xA, c0), __ffma2_rn(sqc, xB, c0), mb, pA, pB, pst[0]);
      {
        const float2 fA = __ffma2_rn(isum2(fh[0], fh[1]), splat(UF), isum2(fl[0], fl[1])), fB = __ffma2_rn(isum2(fh[2], fh[3]), splat(UF), isum2(fl[2], fl[3]));
        float2 mf, qA, qB;
        softmax(__ffma2_rn(sqf, __ffma2_rn(splat((float)(1 << FB)), xA, fA), qb2), __ffma2_rn(sqf, __ffma2_rn(splat((float)(1 << FB)), xB, fB), qb2), mf, qA, qB, pst[1]);
        if (gid == 0) *reinterpret_cast<float2 *>(lp + 2 * n_cells) = mf;
      }
      // both columns' sums of p in one word (each below 2^13): low half column 0, high half column 1
      uint32_t ps = (__float_as_uint(pA.x) + __float_as_uint(pB.x)) + ((__float_as_uint(pA.y) + __float_as_uint(pB.y)) << 16) - 2u * MAGIC;
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) ps += __shfl_xor_sync(FULL, ps, o);
      const float2 sp = isum2((ps & 0xffffu) | MAGIC, (ps >> 16) | MAGIC);
      if (gid == 0) {
        *reinterpret_cast<float2 *>(lp) = make_float2(mb.x + lg2(sp.x), mb.y + lg2(sp.y));
        *reinterpret_cast<float2 *>(lp + n_cells) = mb;
      }
      // the running maximum moves only when a block exceeds it by more than 2^8
      if (mb.x > m[0] + 8.f) { l[0] *= ex2(m[0] - mb.x); m[0] = mb.x; }
      if (mb.y > m[1] + 8.f) { l[1] *= ex2(m[1] - mb.y); m[1] = mb.y; }
      l[0] = fmaf(sp.x, ex2(mb.x - m[0]), l[0]);
      l[1] = fmaf(sp.y, ex2(mb.y - m[1]), l[1]);
      __syncwarp();
      *wp = lds32(pst[0] + 4 * lane);
      wp[4 * n_cells] = lds32(pst[1] + 4 * lane);
      lp += 8; wp += 32;
    }
    leave(fold.stage[warp][cur_vh == first_vh ? 0 : 1]);
  }
  if (lane == 0) {
    fold.stage_vh[warp][0] = first_vh;
    fold.stage_vh[warp][1] = cur_vh != first_vh ? cur_vh : -1;
  }
  __syncthreads();
  via.ready();
  // the warps' pairs: a lane per (warp, query), merged by a butterfly (one after the other: 1 us)
  if constexpr (HEAD) {  // one head: its pairs of all warps, and of the CTA's window sub-blocks (a CTA without either leaves -inf)
    if (warp == 0) {
      float2 acc = make_float2(-FBLA_INF, 0.f);
#pragma unroll
      for (int e = lane; e < SCORE_WARPS * QG; e += 32) {
        if (fold.stage_vh[e / QG][0] >= 0) acc = merge_mass(acc, fold.stage[e / QG][0][e % QG]);
        acc = merge_mass(acc, fold.window[e / QG][e % QG]);
      }
      acc = merge_lanes<QG>(acc, lane);
      via.put_mass(acc, lane);
    }
  } else {  // rows of heads that may continue in neighbouring warps
    const Runs runs(fold.stage_vh, SCORE_WARPS, lane);
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
      if (!((r ? runs.mask1 : runs.mask0) >> warp & 1)) continue;
      const int v = fold.stage_vh[warp][r], n = runs.length(warp, r);
      float2 acc = make_float2(-FBLA_INF, 0.f);
#pragma unroll
      for (int e = lane; e < SCORE_WARPS * QG; e += 32)
        if (e / QG < n) acc = merge_mass(acc, fold.stage[warp + e / QG][e < QG ? r : 0][e % QG]);
      acc = merge_lanes<QG>(acc, lane);
      if (lane < QG) mass_pair(a, cta + v)[lane] = acc;
    }
  }
}

template <int CB, int FB, int QG, bool HEAD = false>
__device__ __forceinline__ void score_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  wait_previous_pass();  // (lengths, queries and the cache may come from the kernel before)
  allow_next_pass();     // (behind the wait: the value pass then finds everything before this call complete)
  if (FBLA_POS::x() == 0 && FBLA_POS::y() == 0 && FBLA_POS::z() == 0 && FBLA_POS::tid() == 0 && a.status) { a.status[0] = 0; a.status[1] = 0; }
  if constexpr (HEAD) {
    HeadScoreSmem &sm = *reinterpret_cast<HeadScoreSmem *>(smem_raw);
    score_units<CB, FB, QG, true>(a, sm.w, sm.fold, nullptr, ScratchVia<QG>(a));
  } else {
    ScoreSmem &sm = *reinterpret_cast<ScoreSmem *>(smem_raw);
    build_table(a, sm.table, 32 * SCORE_WARPS);
    if (FBLA_POS::x() == 0 && a.lstride)
      for (int i = FBLA_POS::tid(); i <= a.batch; i += 32 * SCORE_WARPS) { table_of(a)[i] = sm.table.closed[i]; table_of(a)[a.batch + 1 + i] = sm.table.exact[i]; }
    score_units<CB, FB, QG, false>(a, sm.w, sm.fold, &sm.table, NoVia());
  }
}

// ---- R of a virtual head: log2 of every query's mass --------------------------------------------------------------------------
// one warp; lane l returns that of query l % QG
struct Rows { int m0, m1, x0, x1, v0, v1; };  // slots of the head's (m, l) pairs, window rows and value rows (first, last; empty if last < first)
template <int QG>
__device__ __forceinline__ Rows rows_of(const fbla_k_decode &a, const int *closed, const int *exact, int hpr, int vh) {
  const int b = vh / hpr, hir = vh - b * hpr;
  Rows r{0, -1, 0, -1, 0, -1};
  const Span g = span_of<false>(a, closed, hpr, b, hir), x = span_of<true>(a, exact, hpr, b, hir);
  if (g.n > 0) {
    const int groups = total_of<false>(a, closed, hpr);
    const int per = (QG * groups + a.coarse_ctas - 1) / a.coarse_ctas, vper = (PAIRS * groups + a.coarse_ctas - 1) / a.coarse_ctas;
    r.m0 = QG * g.off / per; r.m1 = (QG * (g.off + g.n) - 1) / per;
    r.v0 = PAIRS * g.off / vper; r.v1 = (PAIRS * (g.off + g.n) - 1) / vper;
  }
  if (x.n > 0) {
    const int run = window_run(a, total_of<true>(a, exact, hpr));
    r.x0 = x.off / run; r.x1 = (x.off + x.n - 1) / run;
  }
  return r;
}
template <int QG>
__device__ __forceinline__ float row_mass(const fbla_k_decode &a, const Rows &r, int vh, int lane) {
  const int q = lane % QG, nm = r.m1 - r.m0 + 1, n = nm + r.x1 - r.x0 + 1;
  float2 acc = make_float2(-FBLA_INF, 0.f);
  for (int i0 = lane / QG; i0 < n; i0 += 4 * (32 / QG)) {
    float2 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = min(i0 + j * (32 / QG), n - 1);
      const float2 *const pair = mass_pair(a, r.m0 + i + vh) + q, *const window = reinterpret_cast<const float2 *>(window_row(a, r.x0 + i - nm + vh) + q * PSTRIDE + D);
      v[j] = __ldcg(i < nm ? pair : window);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + j * (32 / QG) < n) acc = merge_mass(acc, v[j]);
  }
  acc = merge_lanes<QG>(acc, lane);
  return acc.x + lg2(acc.y);  // (-inf for a shard that holds nothing of the row)
}
// the same where the head has CTAs of its own
template <int QG, class Via> __device__ __forceinline__ float head_mass(const Via &via, int ctas, int lane) {
  float2 acc = make_float2(-FBLA_INF, 0.f);
  for (int i = lane / QG; i < ctas; i += 32 / QG) acc = merge_mass(acc, via.mass(i, lane % QG));
  acc = merge_lanes<QG>(acc, lane);
  return acc.x + lg2(acc.y);
}
// the rows' masses into row_r: a shard's first phase, and a pass of its own under an executor. One warp per virtual head.
template <int QG>
__device__ __forceinline__ void mass_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  const int lane = FBLA_POS::tid() & 31, vh = FBLA_POS::x() * 8 + (FBLA_POS::tid() >> 5), hpr = a.kv_heads * a.vg;
  allow_next_pass();
  wait_previous_pass();
  if (vh >= a.batch * hpr) return;
  const int *t = table_of(a);
  const float R = a.head_ctas ? head_mass<QG>(ScratchVia<QG>(a, vh), a.head_ctas, lane) : row_mass<QG>(a, rows_of<QG>(a, t, t + a.batch + 1, hpr, vh), vh, lane);
  if (lane < QG) a.row_r[vh * QG + lane] = R;
}

// ---- value pass -------------------------------------------------------------------------------------------------------------------
// V words of a record: what thread (gid, tig) supplies to the products for record lanes 8 u + gid, u = 0..3, and its slots (as v_slots of
// fbla_frag.cuh). In registers; of 3 bits the record lanes' words W[4], W[5] lie in shared memory (`tail`: 8 bytes per record lane; the
// warp copies a record's 256 bytes there, 8 a lane): in registers they were two thirds of the words, each held by four threads, and the
// kernel spilled.
template <int BITS> struct VWords {
  uint32_t w[4][BITS == 4 ? 2 : 1];
  static __device__ __forceinline__ int offset(int gid, int tig) { return BITS == 4 ? 1024 + 512 * (tig >> 1) + 16 * gid + 8 * (tig & 1) : 512 + 16 * gid + 4 * tig; }
  __device__ __forceinline__ void load(const uint8_t *p) {  // p: the record + offset
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if constexpr (BITS == 4) {
        const uint2 y = __ldg(reinterpret_cast<const uint2 *>(p + 128 * u));
        w[u][0] = y.x; w[u][1] = y.y;
      } else {
        w[u][0] = __ldg(reinterpret_cast<const uint32_t *>(p + 128 * u));
      }
    }
  }
  __device__ __forceinline__ void slots(int u, int tig, const uint8_t *tail, uint32_t (&v)[4]) const {
    const uint32_t a = w[u][0];
    if constexpr (BITS == 4) {
      const uint32_t b = w[u][1];
      v[0] = a & 0x0f0f0f0fu; v[1] = b & 0x0f0f0f0fu; v[2] = a & 0xf0f0f0f0u; v[3] = b & 0xf0f0f0f0u;
    } else if constexpr (BITS == 2) {
      v[0] = a & 0x03030303u; v[1] = a & 0x0c0c0c0cu; v[2] = a & 0x30303030u; v[3] = a & 0xc0c0c0c0u;
    } else {  // W[4 + tig / 2]: the top bit of slot 12 + tig; W[4 + tig % 2]: slot 4 + tig for tig < 2, 10 + tig - 2 beyond
      v[0] = a & 0x07070707u;
      v[1] = a & 0x38383838u;
      v[2] = (lds32(tail + 64 * u + 4 * (tig & 1)) >> (3 * (tig >> 1))) & 0x07070707u;
      v[3] = ((a >> 6) & 0x03030303u) | ((lds32(tail + 64 * u + 4 * (tig >> 1)) >> (4 + (tig & 1))) & 0x04040404u);
    }
  }
};
constexpr int TAIL_BYTES = 256;               // of a record's V half
constexpr int TAILS_BYTES = 8 * TAIL_BYTES;   // of a warp: [coarse, fine][pair, alternating][sub-block of the pair]
struct __align__(16) ValueWarp {
  uint8_t meta[2][512];        // V's metadata of the group in work and of the next
  float stage[4][PSTRIDE];     // the row set of the first virtual head of the warp's run
  // The current head's sums (Sums, [word][lane]): in registers they would halve the warps that an SM holds. At the end: the last
  // head's row set.
  float2 run[17][32];
};
struct ValueSmem {
  ValueWarp w[VALUE_WARPS];
  uint8_t tails[VALUE_WARPS][TAILS_BYTES];
  int stage_vh[VALUE_WARPS][2];
  Table table;
};
struct __align__(16) HeadValueSmem { ValueWarp w[VALUE_WARPS]; };
struct __align__(16) HeadValueItemSmem { HeadValueSmem s; uint8_t tails[VALUE_WARPS][TAILS_BYTES]; };
static_assert(sizeof(ValueSmem) + 128 <= 227 * 1024, "one CTA's shared memory");

// the sums of one virtual head over the warp's pairs, in units of 2^-R: thread (gid, tig) holds channels 4 (8 u + gid) + cc of
// queries 2 (tig & 1) + e, summed over the sub-blocks of parity tig >> 1
struct Sums {
  float2 l, o[4][4];
};
template <int QG> __device__ __forceinline__ void write_sums(float *p, const Sums &s, int lane) {
  const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float le = e ? s.l.y : s.l.x, l = le + __shfl_xor_sync(FULL, le, 2);
    const int qe = 2 * tig + e;
    float *row = p + qe * PSTRIDE;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float v[4];
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        const float o = e ? s.o[u][cc].y : s.o[u][cc].x;
        v[cc] = o + __shfl_xor_sync(FULL, o, 2);
      }
      if (tig < 2 && qe < QG) *reinterpret_cast<float4 *>(row + 4 * (8 * u + gid)) = make_float4(v[0], v[1], v[2], v[3]);
    }
    if (tig < 2 && qe < QG && gid == 0) row[D] = l;
  }
}

// `wait` returns when the score pass's results may be read; what does not depend on them is asked for before. tails: the warp's.
template <int CB, int FB, int QG, bool HEAD, class Via, class Wait>
__device__ __forceinline__ void value_units(const fbla_k_decode &a, ValueWarp *ws, uint8_t *tails, int (*stage_vh)[2], const Table *table, const Via &via, Wait wait) {
  constexpr int RC = record_bytes(CB), RF = record_bytes(FB);
  constexpr float HOFF = .5f * ((1 << FB) - 1);
  const int lane = FBLA_POS::tid() & 31, warp = FBLA_POS::tid() >> 5, gid = lane >> 2, tig = lane & 3;
  const int hpr = HEAD ? (int)FBLA_POS::ny() : a.kv_heads * a.vg;
  ValueWarp &w = ws[warp];
  int cta, total, c_lo, c_n;
  Cursor c{0, 0, 0, 0};
  if constexpr (HEAD) {
    const Own own(a);
    cta = own.slot; total = PAIRS * own.row.closed;
    const int per = (QG * own.row.closed + own.ctas - 1) / own.ctas * (PAIRS / QG);  // the sub-blocks that the CTA has scored
    c_lo = min(total, own.rank * per); c_n = min(total, c_lo + per) - c_lo;
    c = Cursor{own.b, own.hir, 0, own.row.closed};
  } else {
    cta = FBLA_POS::x(); total = PAIRS * total_of<false>(a, table->closed, hpr);
    const int per = (total + (int)FBLA_POS::nx() - 1) / (int)FBLA_POS::nx();
    c_lo = min(total, cta * per); c_n = min(total, c_lo + per) - c_lo;
  }
  const int wper = (c_n + VALUE_WARPS - 1) / VALUE_WARPS, lo = c_lo + min(c_n, warp * wper), hi = c_lo + min(c_n, (warp + 1) * wper);
  float R = 0.f;  // lane l: of query l % QG of the current head
  // (HEAD: every warp asks for it, also one without pairs: the CTA's window sub-blocks need it)
  auto mass_of = [&](int vh) {
    if (a.mass_given) return __ldcg(a.row_r + vh * QG + lane % QG);
    if constexpr (HEAD) return head_mass<QG>(via, (int)FBLA_POS::nx(), lane);
    else return row_mass<QG>(a, rows_of<QG>(a, table->closed, table->exact, hpr, vh), vh, lane);
  };
  if (lo >= hi) {
    wait();
    if (HEAD) R = mass_of(c.b * hpr + c.hir);
  }
  int first_vh = -1, cur_vh = -1;
  if (lo < hi) {
    if constexpr (HEAD) c.i = lo / PAIRS;
    else c = find<false>(a, table->closed, hpr, lo / PAIRS);
    const int groups = (hi - 1) / PAIRS - lo / PAIRS + 1;
    int left = hi - lo;  // pairs
    // The sums of integer products are taken as they are: a nonnegative s32 below 2^23 read as FP32 is the subnormal s 2^-149, and a
    // weight times 2^75 brings the product back into range; the group's sums come out times 2^-74.
    constexpr float UP = 37778931862957161709568.f /* 2^75 */, BACK = 18889465931478580854784.f /* 2^74 */;
    // a group's place: its unit, and its first cell
    auto unit_of = [&](const Cursor &x) { return (size_t)kv_of(a, x.b * hpr + x.hir) * a.hs + (size_t)group_of(a, x) * a.gs; };
    auto cell_of = [&](const Cursor &x) { return ((size_t)(x.b * hpr + x.hir) * a.nblocks + (size_t)group_of(a, x) * SBG) * QG; };
    const size_t n_cells = cells_of(a);
    const int pcol = (gid >> 2) * QG + (gid & 3);  // the lane's column of a pair's P words: sub-block gid / 4, query gid % 4
    const bool has = (gid & 3) < QG;
    const uint32_t *const w0 = weights_of(a) + 4 * pcol + tig, *const w1 = w0 + 4 * n_cells;
    // what a group's cells hold, lane l: cell l = (sub-block l / QG, query l % QG)
    float lse_n, mc_n, mf_n = 0.f;
    size_t cell = cell_of(c), cell_n;
    auto ask = [&](size_t at) {
      lse_n = -FBLA_INF; mc_n = 0.f;
      if (lane < SBG * QG) { const float *p = a.lse + at + lane; lse_n = __ldcg(p); mc_n = __ldcg(p + n_cells); mf_n = __ldcg(p + 2 * n_cells); }
    };
    uint32_t pc = 0u, pf = 0u;  // the next pair's words
    auto ask_p = [&](size_t at, int J) {
      if (has) { pc = __ldcg(w0 + (at + 2 * QG * J) * 4); pf = __ldcg(w1 + (at + 2 * QG * J) * 4); }
    };
    size_t unit = unit_of(c);
    // Asynchronous copies, 3 bits (TAILS): they leave in the order of a pair's coarse tails, its fine tails, the next pair's coarse tails, ... -- a
    // group of copies each (empty where there is nothing to copy), the metadata of the next group of tokens with one of them -- so that
    // waiting for all but the last group is waiting for what the pair in work needs next. Else: the metadata alone.
    // AHEAD: both planes of a pair, one group of copies, a whole pair ahead instead of a plane half a pair ahead, in registers that the tails
    // do not take: 64 rows of 1K to 64K 811 -> 749 us (behind a flush of L2), 32 of 300 to 6 000 75.8 -> 72.9, 16 x 8 000 70.2 -> 66.7; but with
    // two queries 16 x 4 000 44.3 -> 45.6, and in the one kernel of a short decode, whose warps have a pair or two, 4K 11.5 -> 12.3.
    constexpr bool TAILS = CB == 3, AHEAD = TAILS && !HEAD && QG == 4;
    auto close_copies = [] { if (TAILS) asm volatile("cp.async.commit_group;" ::: "memory"); };
    auto arrived = [] {
      if (TAILS) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
      }
    };
    auto fetch_meta = [&](size_t un, int buf) {  // V's 512 bytes of metadata
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;"
                   ::"r"(smem_u32(w.meta[buf] + 16 * lane)), "l"(reinterpret_cast<const uint8_t *>(a.c.meta) + un * 1024 + 512 + 16 * lane) : "memory");
      if (!TAILS) asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int J = lo % PAIRS;
    fetch_meta(unit, 0);
    // where the words of the next pair (coarse) and of the pair in work (fine) lie: pointers that run on within a head
    const uint8_t *cp = a.c.coarse + (unit * SBG + 2 * J) * RC + VWords<CB>::offset(gid, tig), *fp = a.c.fine + (unit * SBG + 2 * J) * RF + VWords<FB>::offset(gid, tig);
    const long long c_skip = (long long)(a.gs - 1) * SBG * RC, f_skip = (long long)(a.gs - 1) * SBG * RF;
    VWords<CB> va, vb;
    VWords<FB> fa, fb;
    int turn = 0;  // the pair's place among the tails
    uint8_t *const ctail = tails + 8 * gid, *const ftail = ctail + 4 * TAIL_BYTES;
    auto fetch_tails = [&](const uint8_t *rec, int bytes, uint8_t *to) {  // rec: this thread's place in the first record
      if constexpr (TAILS) {
        const uint8_t *const from = rec - VWords<3>::offset(gid, tig) + 1280 + 8 * lane;
#pragma unroll
        for (int b = 0; b < 2; ++b)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(to - 8 * gid + 8 * lane + TAIL_BYTES * b)), "l"(from + bytes * b) : "memory");
      }
    };
    auto load_coarse = [&](VWords<CB> &x, VWords<CB> &y, int at) {
      x.load(cp);
      y.load(cp + RC);
      fetch_tails(cp, RC, ctail + 2 * TAIL_BYTES * at);
      cp += 2 * RC;
    };
    auto load_fine = [&](VWords<FB> &x, VWords<FB> &y, int at) {
      x.load(fp);
      y.load(fp + RF);
      fetch_tails(fp, RF, ftail + 2 * TAIL_BYTES * at);
      fp += 2 * RF;
    };
    load_coarse(va, vb, 0);
    if (!AHEAD) close_copies();
    if (HEAD || AHEAD) {  // (whether it is selected is not known yet; mostly it is)
      load_fine(fa, fb, 0);
      close_copies();
    }
    if constexpr (HEAD) {  // (the CTA's own cells: complete)
      ask(cell);
      ask_p(cell, J);
      wait();
    } else {
      wait();
      ask(cell);
      ask_p(cell, J);
    }
    auto sums = [&] {
      Sums r;
      r.l = w.run[16][lane];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) r.o[u][cc] = w.run[4 * u + cc][lane];
      return r;
    };
#pragma unroll 1
    for (int k = 0; k < groups; ++k) {
      const int vh = c.b * hpr + c.hir, j1 = min(PAIRS, J + left);
      if (vh != cur_vh) {
        if (cur_vh >= 0) write_sums<QG>(cur_vh == first_vh ? &w.stage[0][0] : value_row(a, cta + cur_vh), sums(), lane);
        else first_vh = vh;
        cur_vh = vh;
#pragma unroll
        for (int x = 0; x < 17; ++x) w.run[x][lane] = make_float2(0.f, 0.f);
        R = mass_of(vh);
        if (!HEAD && !a.mass_given && lane < QG) a.row_r[vh * QG + lane] = R;  // for the merge (every warp of the head writes the same)
      }
      const uint32_t mask = __ballot_sync(FULL, lse_n - R > a.log2_tau);  // bit cell: selected
      float wl = ex2(((mask >> lane) & 1 ? mf_n : mc_n) - R) * UP;          // lane: the weight of its cell
      if (lane >= SBG * QG) wl = 0.f;
      // the next group: its cells, its metadata
      Cursor n = c;
      size_t unit_n = unit;
      const bool more = k + 1 < groups, stay = c.i + 1 < c.n;  // stay: the next group is the head's next
      if (more) {
        if (stay) { ++n.i; unit_n += a.gs; cell_n = cell + SBG * QG; }
        else { advance<false>(a, hpr, n); unit_n = unit_of(n); cell_n = cell_of(n); }
        ask(cell_n);
        fetch_meta(unit_n, (k + 1) & 1);
      }
      float2 A[4][4], L = make_float2(0.f, 0.f), Hc = L;  // the group's sums in code units; sum w sum p, and its unselected part
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) A[u][cc] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (; J < j1; ++J, --left) {
        const uint32_t pm = (mask >> (2 * QG * J)) & ((1u << (2 * QG)) - 1u);  // the pair's selections
        const bool last = J + 1 >= PAIRS;
        auto move_on = [&] {  // from the group's last pair to the next group
          if (stay) { cp += c_skip; fp += f_skip; }
          else {
            cp = a.c.coarse + unit_n * SBG * RC + VWords<CB>::offset(gid, tig);
            fp = a.c.fine + unit_n * SBG * RF + VWords<FB>::offset(gid, tig);
          }
        };
        VWords<CB> na, nb;
        VWords<FB> ma, mb;
        if constexpr (AHEAD) {
          __syncwarp();  // (every lane has read the tails of the pair before: the next one's take their place)
          if (left > 1) {
            if (last) move_on();
            load_coarse(na, nb, turn ^ 1);
            if (last || ((mask >> (2 * QG * (J + 1))) & ((1u << (2 * QG)) - 1u))) load_fine(ma, mb, turn ^ 1);  // (the next group's selections are not known yet)
            else fp += 2 * RF;
          }
          close_copies();
        } else if constexpr (!HEAD) {
          if (pm) load_fine(fa, fb, turn);
          else fp += 2 * RF;
          close_copies();
        }
        arrived();  // the pair's coarse tails
        const uint8_t *const ct = ctail + 2 * TAIL_BYTES * turn, *const ft = ftail + 2 * TAIL_BYTES * turn;
        uint32_t pw = (pm >> pcol) & 1 ? pf : pc;
        if (!has) pw = 0u;
        if (left > 1) ask_p(last ? cell_n : cell, last ? 0 : J + 1);
        // the thread's two columns: sub-block tig >> 1, queries 2 (tig & 1) + e
        const int own = QG * (tig >> 1) + 2 * (tig & 1);
        float2 wt = make_float2(__shfl_sync(FULL, wl, 2 * QG * J + own), __shfl_sync(FULL, wl, (2 * QG * J + own + 1) & 31));
        if (QG < 4) { if (!query_valid<QG>(tig, 0)) wt.x = 0.f; if (!query_valid<QG>(tig, 1)) wt.y = 0.f; }
        const float2 ws = make_float2((pm >> own) & 1 ? wt.x : 0.f, (pm >> own) & 2 ? wt.y : 0.f);
        const uint32_t b0 = gid < 4 ? pw : 0u, b1 = gid < 4 ? 0u : pw;
        {
          uint32_t d[4];
          mma_u8u8_k32_zero(d, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, b0, b1);
          const float2 sp = tiny2(d[0], d[1]);
          L = __ffma2_rn(wt, sp, L);
          Hc = __ffma2_rn(__fadd2_rn(wt, make_float2(-ws.x, -ws.y)), sp, Hc);
        }
        // the weights times the planes' class factors: code units = 2^FB h + f
        auto add = [&](const uint32_t (&x)[4], const uint32_t (&y)[4], const float2 (&f)[4], float2 (&to)[4]) {
          uint32_t d01[4], d23[4];
          mma_u8u8_k32_zero(d01, x[0], x[1], y[0], y[1], b0, b1);
          mma_u8u8_k32_zero(d23, x[2], x[3], y[2], y[3], b0, b1);
          to[0] = __ffma2_rn(f[0], tiny2(d01[0], d01[1]), to[0]);
          to[1] = __ffma2_rn(f[1], tiny2(d01[2], d01[3]), to[1]);
          to[2] = __ffma2_rn(f[2], tiny2(d23[0], d23[1]), to[2]);
          to[3] = __ffma2_rn(f[3], tiny2(d23[2], d23[3]), to[3]);
        };
        {
          float2 f[4];
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) f[cc] = __fmul2_rn(wt, splat((float)(1 << FB) * v_unscale<CB>(cc)));
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t x[4], y[4];
            va.slots(u, tig, ct, x);
            vb.slots(u, tig, ct + TAIL_BYTES, y);
            add(x, y, f, A[u]);
          }
        }
        if constexpr (!AHEAD) {
          if (left > 1) {
            if (last) move_on();
            load_coarse(va, vb, turn ^ 1);
          }
          close_copies();
          arrived();  // the pair's fine tails
        }
        if (pm) {
          float2 f[4];
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) f[cc] = __fmul2_rn(ws, splat(v_unscale<FB>(cc)));
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t x[4], y[4];
            fa.slots(u, tig, ft, x);
            fb.slots(u, tig, ft + TAIL_BYTES, y);
            add(x, y, f, A[u]);
          }
        }
        if constexpr (AHEAD) {
          va = na; vb = nb; fa = ma; fb = mb;
        } else if constexpr (HEAD) {
          if (left > 1) load_fine(fa, fb, turn ^ 1);
          close_copies();
        }
        turn ^= 1;
      }
      J = 0;
      if (!TAILS) {  // (else the metadata has come with the tails)
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
      }
      const uint8_t *meta = w.meta[k & 1];
      L = __fmul2_rn(L, splat(BACK)); Hc = __fmul2_rn(Hc, splat(HOFF * BACK));
      w.run[16][lane] = __fadd2_rn(w.run[16][lane], L);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint4 vm = lds128(meta + 16 * (8 * u + gid));
        const float vbs[4] = {bf_lo(vm.x), bf_hi(vm.x), bf_lo(vm.y), bf_hi(vm.y)}, vs[4] = {bf_lo(vm.z), bf_hi(vm.z), bf_lo(vm.w), bf_hi(vm.w)};
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
          w.run[4 * u + cc][lane] = __fadd2_rn(w.run[4 * u + cc][lane], __ffma2_rn(splat(vs[cc]), __ffma2_rn(splat(BACK), A[u][cc], Hc), __fmul2_rn(splat(vbs[cc]), L)));
      }
      __syncwarp();  // (the metadata buffer has been read)
      c = n; unit = unit_n; cell = cell_n;
    }
    const Sums r = sums();
    __syncwarp();
    write_sums<QG>(cur_vh == first_vh ? &w.stage[0][0] : reinterpret_cast<float *>(w.run), r, lane);
  }
  if constexpr (HEAD) {
    // One head: a thread per (query, channel) adds the CTA's window sub-blocks, brought to units of 2^-R, and the warps' rows.
    const Own own(a);
    const int q = warp >> 2, ch = FBLA_POS::tid() & 127, x_per = (own.row.exact + own.ctas - 1) / own.ctas;
    const int x0 = min(own.row.exact, own.rank * x_per), x1 = min(own.row.exact, x0 + x_per), rows = wper ? (c_n + wper - 1) / wper : 0;
    const float Rq = __shfl_sync(FULL, R, q % QG);
    float o = 0.f, l = 0.f;
    if (q < QG)
      for (int x = x0; x < x1; ++x) {
        const float *const row = via.window(x) + q * PSTRIDE;
        const float e = ex2(row[D] - Rq);
        o = fmaf(e, row[ch], o);
        l = fmaf(e, row[D + 1], l);
      }
    __syncthreads();
    if (q < QG) {
#pragma unroll 4
      for (int x = 0; x < rows; ++x) o += ws[x].stage[q][ch];
      via.put(q, ch, o);
      if (ch == 0) {
#pragma unroll 4
        for (int x = 0; x < rows; ++x) l += ws[x].stage[q][D];
        via.put(q, D, l);
      }
    }
    return;
  }
  if (lane == 0) {
    stage_vh[warp][0] = first_vh;
    stage_vh[warp][1] = cur_vh != first_vh ? cur_vh : -1;
  }
  __syncthreads();
  // rows of heads that may continue in neighbouring warps, added in warp order (by the head's first warp alone: 8 x 16K 4+2 70.5 us, so 63.0)
  fold_heads(stage_vh, VALUE_WARPS, VALUE_WARPS / 4, [&](int x, int r, int n, int t) {
    add_sets<QG>(value_row(a, cta + stage_vh[x][r]), n, t,
                 [&](int y) { return y == 0 && r ? reinterpret_cast<const float *>(ws[x].run) : &ws[x + y].stage[0][0]; });
  });
}

template <int CB, int FB, int QG, bool HEAD = false>
__device__ __forceinline__ void value_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  allow_next_pass();
  if constexpr (HEAD) {  // (a plan's items only: the stream call's kernel is head_passes)
    HeadValueItemSmem &sm = *reinterpret_cast<HeadValueItemSmem *>(smem_raw);
    value_units<CB, FB, QG, true>(a, sm.s.w, sm.tails[FBLA_POS::tid() >> 5], nullptr, nullptr, ScratchVia<QG>(a), [] {});
  } else {
    ValueSmem &sm = *reinterpret_cast<ValueSmem *>(smem_raw);
    build_table(a, sm.table, 32 * VALUE_WARPS);
    if (a.phase != 0) wait_previous_pass();  // (a whole decode: the score pass let this one begin when all before the call was complete)
    value_units<CB, FB, QG, false>(a, sm.w, sm.tails[FBLA_POS::tid() >> 5], sm.stage_vh, &sm.table, NoVia(), [&] { if (a.phase == 0) wait_previous_pass(); });
  }
}

// ---- merge: out = (sum 2^(m_x - R) o_x + sum o_v) / (sum 2^(m_x - R) l_x + sum l_v), BF16 -----------------------------------
// Where the head has CTAs of its own: thread ch of 128 adds their sums(cta, channel or D for l), in order.
template <class Sum> __device__ __forceinline__ void write_row(const fbla_k_decode &a, int vh, int qi, int ch, int ctas, Sum sums) {
  float o = 0.f, l = 0.f;
#pragma unroll 4
  for (int i = 0; i < ctas; ++i) { o += sums(i, ch); l += sums(i, D); }
  a.out[((size_t)vh * a.qg + qi) * D + ch] = f32_to_bf16(__fdividef(o, l));  // (the row of query qi of virtual head vh)
}
// Else one CTA of four warps per output row: warp s sums rows s, s + 4, ... of the head's window and value rows, lane c channels
// 4 c .. 4 c + 3; the four sums are added in order.
template <int QG>
__device__ __forceinline__ void gather_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  __shared__ float4 so[4][32];
  __shared__ float sl[4];
  const int vh = FBLA_POS::x() / QG, qi = FBLA_POS::x() % QG, lane = FBLA_POS::tid() & 31, warp = FBLA_POS::tid() >> 5;
  allow_next_pass();
  wait_previous_pass();
  if (a.head_ctas) {
    const ScratchVia<QG> via(a, vh);
    write_row(a, vh, qi, FBLA_POS::tid(), a.head_ctas, [&](int cta, int ch) { return via.sum(cta, qi, ch); });
    return;
  }
  const int hpr = a.kv_heads * a.vg, b = vh / hpr, hir = vh - b * hpr;
  const int *t = table_of(a);
  const Rows r = rows_of<QG>(a, t, t + a.batch + 1, hpr, vh);
  // (a head without closed groups was nobody's in the value pass)
  const float R = a.mass_given || r.v1 >= r.v0 ? __ldcg(a.row_r + vh * QG + qi) : __shfl_sync(FULL, row_mass<QG>(a, r, vh, lane), qi);
  const int status = a.status ? __ldcg(a.status) : 0;
  const int nx = r.x1 - r.x0 + 1, n = nx + r.v1 - r.v0 + 1;
  float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
  float L = 0.f;
  constexpr int MJ = 5;
  for (int i0 = warp; i0 < n; i0 += 4 * MJ) {
    float m[MJ], l[MJ];
    float4 o[MJ];
#pragma unroll
    for (int j = 0; j < MJ; ++j) {
      const int i = min(i0 + 4 * j, n - 1);
      const float *p = (i < nx ? window_row(a, r.x0 + i + vh) : value_row(a, r.v0 + i - nx + vh)) + qi * PSTRIDE;
      o[j] = __ldcg(reinterpret_cast<const float4 *>(p) + lane);
      m[j] = __ldcg(p + D);
      l[j] = i < nx ? __ldcg(p + D + 1) : m[j];
    }
#pragma unroll
    for (int j = 0; j < MJ; ++j)
      if (i0 + 4 * j < n) {
        const float e = i0 + 4 * j >= nx ? 1.f : m[j] == -FBLA_INF ? 0.f : ex2(m[j] - R);
        L = fmaf(e, l[j], L);
        O.x = fmaf(e, o[j].x, O.x); O.y = fmaf(e, o[j].y, O.y); O.z = fmaf(e, o[j].z, O.z); O.w = fmaf(e, o[j].w, O.w);
      }
  }
  so[warp][lane] = O;
  if (lane == 0) sl[warp] = L;
  __syncthreads();
  const int ch = FBLA_POS::tid();
  const float *col = reinterpret_cast<const float *>(so) + ch;
  const float Os = (col[0] + col[D]) + (col[2 * D] + col[3 * D]), Ls = (sl[0] + sl[1]) + (sl[2] + sl[3]);
  const size_t row = (size_t)q_row(a, b, hir, qi);
  const bool failed = status != 0;  // (a wait gave up somewhere: not a plausible number)
  const float nan = __int_as_float(0x7fc00000);
  if (a.out_partial) {
    a.out_partial[row * PSTRIDE + ch] = failed ? nan : Os;
    if (ch == 0) a.out_partial[row * PSTRIDE + D] = failed ? nan : Ls;
  } else {
    a.out[row * D + ch] = failed ? (uint16_t)0x7fc0 : f32_to_bf16(__fdividef(Os, Ls));
  }
}
// ---- a short decode: all passes in one kernel -----------------------------------------------------------------------------------
// A cluster of a.head_ctas CTAs per virtual head does the head's scores, values and output rows: the same code as a plan's passes, hence the
// same bits, with the cluster's barrier in the place of a kernel boundary and masses and sums stored into the shared memory of the CTAs
// that read them.
struct __align__(16) HeadSmem {
  HeadScoreSmem s;
  HeadValueSmem v;  // (beside the scores': the first values are asked for before the cluster meets)
  float2 mass[16][4];  // [CTA][query]
  // in the scores' place once all CTAs have theirs: a window sub-block's row over its warp's V rows, the CTAs' sums over the queries
  __device__ __forceinline__ float *window(int warp) { return reinterpret_cast<float *>(&s.w[warp].exact.v[0][0]); }
  __device__ __forceinline__ uint8_t *tails(int warp) { return reinterpret_cast<uint8_t *>(window(warp) + 4 * PSTRIDE); }  // behind that row
  __device__ __forceinline__ float *sums(int slot) { return reinterpret_cast<float *>(&s.w[slot].exact.q[0][0]); }
};
static_assert(sizeof(HeadSmem) <= 227 * 1024, "one CTA's shared memory");
static_assert(SCORE_WARPS == 16 && VALUE_WARPS == 16, "one CTA runs both passes; at most sixteen CTAs of a head");
static_assert(sizeof(ExactWarp::v) >= 4 * PSTRIDE * sizeof(float) + TAILS_BYTES && sizeof(ExactWarp::q) >= PSTRIDE * sizeof(float) && sizeof(ExactWarp::q) >= sizeof(ScoreWarp::s),
              "a window sub-block's row and the tails beside the warp's later queries and P bytes");
template <int QG> struct ClusterVia {
  HeadSmem &sm;
  int ctas, rank, x0;  // x0: the first of the CTA's window sub-blocks
  __device__ __forceinline__ void ready() const { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }  // (every CTA has begun)
  __device__ __forceinline__ float *window(int x) const { return sm.window(x - x0); }
  __device__ __forceinline__ void put_mass(float2 mass, int lane) const {
    for (int i = lane / QG; i < ctas; i += 32 / QG) st_remote2(remote(&sm.mass[rank][lane % QG], i), mass);
  }
  __device__ __forceinline__ float2 mass(int cta, int q) const { return sm.mass[cta][q]; }
  // query q is CTA q % ctas's, its (q / ctas)-th
  __device__ __forceinline__ void put(int q, int ch, float x) const { st_remote1(remote(sm.sums(q / ctas * ctas + rank) + ch, q % ctas), x); }
};
template <int CB, int FB, int QG>
__device__ __forceinline__ void head_passes(const fbla_k_decode &a, uint8_t *smem_raw) {
  HeadSmem &sm = *reinterpret_cast<HeadSmem *>(smem_raw);
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  wait_previous_pass();
  allow_next_pass();
  if (FBLA_POS::x() == 0 && FBLA_POS::y() == 0 && FBLA_POS::z() == 0 && FBLA_POS::tid() == 0 && a.status) { a.status[0] = 0; a.status[1] = 0; }  // (no wait here gives up)
  const Own own(a);
  const int x_per = (own.row.exact + own.ctas - 1) / own.ctas;
  const ClusterVia<QG> via{sm, own.ctas, own.rank, min(own.row.exact, own.rank * x_per)};
  score_units<CB, FB, QG, true>(a, sm.s.w, sm.s.fold, nullptr, via);
  value_units<CB, FB, QG, true>(a, sm.v.w, sm.tails(FBLA_POS::tid() >> 5), nullptr, nullptr, via, [] { cluster_meet(); });
  cluster_meet();
  const int quad = FBLA_POS::tid() >> 7, qi = own.rank + own.ctas * quad;
  if (qi < QG) write_row(a, own.vh, qi, FBLA_POS::tid() & 127, own.ctas, [&](int cta, int ch) { return sm.sums(quad * own.ctas + cta)[ch]; });
}

}  // namespace dense
}  // namespace fbla
