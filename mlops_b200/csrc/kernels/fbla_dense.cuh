// FBLA compressed-KV decode for sm_100a where most sub-blocks are refined ("dense"): scores, then every block's value once.
//
// The decode of fbla_decode.cuh streams all coarse planes once and corrects the selected sub-blocks afterwards by
// full - coarse; where most are selected (contexts up to about 16 / tau tokens: the average 16-token block then holds more
// than tau of the mass) it computes their coarse scores and values twice and throws them away. Here
//   * the score pass reads only the K half of the coarse plane (straight into registers, no staging), forms every
//     sub-block's log2 mass and the rows' running (m, l), and serves the BF16 windows;
//   * the value pass knows every row's mass R before it starts, so it knows which (query, sub-block) pairs are selected: it
//     scores each sub-block again, with its fine bits where selected, and accumulates its values once, in units of 2^-R
//     -- no running maximum, no correction, no item list. Fine records nobody selected are not read.
// Both passes put the score columns of several sub-blocks into one product's eight columns (queries of sub-block b in
// columns b QG ..; its A fragments meet a B operand that is zero elsewhere, and all add into the same accumulators), so the
// softmax arithmetic runs once per eight (sub-block, query) columns on full warps. Semantics, formats and the definition of
// every number are fbla_decode.cuh's; only the order of the sums differs.
// Work is dealt in contiguous runs of the flattened (virtual head, group, piece of a group) list: first to CTAs, then to
// the CTA's warps, so that a head's partial rows are one per CTA, folded in warp order (reproducible bit for bit).
#pragma once
#include "fbla_decode.cuh"

namespace fbla {
namespace dense {

constexpr int SCORE_WARPS = 16, VALUE_WARPS = FBLA_K_DENSE_VALUE_WARPS;
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

// ---- scratch (inside the decode's `part` and `dpart` arrays) -----------------------------------------------------------------
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

// ---- quantisation of the virtual head's queries for one group (quantize_query_word), into QG rows of qst --------------------
// q: the queries in global memory; rows of qst are QST_ROW bytes apart. Per query the caller gets sq, qb, qsum through `take`.
template <int QG, class Take>
__device__ __forceinline__ void quantize_rows(uint4 km, const uint2 (&q)[QG], float sl, uint8_t *qst, int lane, Take take) {
#pragma unroll
  for (int qi = 0; qi < QG; ++qi) {
    float sq, qb, qsum;
    const float4 q4 = make_float4(bf_lo(q[qi].x), bf_hi(q[qi].x), bf_lo(q[qi].y), bf_hi(q[qi].y));
    reinterpret_cast<uint32_t *>(qst + QST_ROW * qi)[lane] = quantize_query_word(km, q4, sl, sq, qb, qsum);
    take(qi, sq, qb, qsum);
  }
}

// ---- score pass -----------------------------------------------------------------------------------------------------------------
// K words of one sub-block in registers: what thread (gid, tig) supplies to the products, for tokens gid and gid + 8.
// 4 bits: the thread takes the 16-byte piece `tig` of a token's four (words 0-3 / 4-7 of the two channel halves), whose four
// words serve two products; 3 bits: the words of qk_tile<3>.
template <int CB> struct KWords;
template <> struct KWords<4> {
  uint4 a, a8;
  __device__ __forceinline__ void load(const uint8_t *rec, int gid, int tig) {
    const uint8_t *p = rec + 512 * (tig & 1) + 256 * (tig >> 1) + 16 * gid;
    a = __ldg(reinterpret_cast<const uint4 *>(p));
    a8 = __ldg(reinterpret_cast<const uint4 *>(p + 128));
  }
};
template <> struct KWords<3> {
  uint32_t a, a8, c, c8, e, e8, f, f8;
  __device__ __forceinline__ void load(const uint8_t *rec, int gid, int tig) {
    const uint32_t *p = reinterpret_cast<const uint32_t *>(rec + 16 * gid + 4 * tig), *q = reinterpret_cast<const uint32_t *>(rec + 1024 + 16 * gid + 4 * (tig >> 1));
    a = __ldg(p); a8 = __ldg(p + 32); c = __ldg(p + 64); c8 = __ldg(p + 96);
    e = __ldg(q); e8 = __ldg(q + 32); f = __ldg(q + 2); f8 = __ldg(q + 34);
  }
};
// the qhat words matching KWords
template <int CB> __device__ __forceinline__ void score_frag(const uint8_t *qst, int row, int tig, uint32_t (&B)[8]) {
  if (CB == 4) {  // low nibbles: slots 4 (tig % 2) + i of half tig / 2; high nibbles: 8 further
    const uint8_t *p = qst + QST_ROW * row + 64 * (tig >> 1) + 16 * (tig & 1);
    const uint4 lo = lds128(p), hi = lds128(p + 32);
    B[0] = lo.x; B[1] = lo.y; B[2] = lo.z; B[3] = lo.w; B[4] = hi.x; B[5] = hi.y; B[6] = hi.z; B[7] = hi.w;
  } else {
    qhat_frag<3>(qst, row, tig, B);
  }
}
// adds the sub-block's products to the accumulators (low and high class); B is zero in other sub-blocks' columns
template <int CB> __device__ __forceinline__ void score_products(const KWords<CB> &k, const uint32_t (&B)[8], uint32_t mask, int tig, uint32_t (&lo)[4], uint32_t (&hi)[4]) {
  uint32_t b[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) b[i] = B[i] & mask;
  if constexpr (CB == 4) {
    constexpr uint32_t L = 0x0f0f0f0fu, H = 0xf0f0f0f0u;
    mma_u8s8_k32(lo, k.a.x & L, k.a8.x & L, k.a.y & L, k.a8.y & L, b[0], b[1]);
    mma_u8s8_k32(hi, k.a.x & H, k.a8.x & H, k.a.y & H, k.a8.y & H, b[4], b[5]);
    mma_u8s8_k32(lo, k.a.z & L, k.a8.z & L, k.a.w & L, k.a8.w & L, b[2], b[3]);
    mma_u8s8_k32(hi, k.a.z & H, k.a8.z & H, k.a.w & H, k.a8.w & H, b[6], b[7]);
  } else {
    const int sh = 4 + (tig & 1), se = 3 * (tig & 1);
    constexpr uint32_t L = 0x07070707u, M = 0x38383838u, T2 = 0x03030303u, T1 = 0x04040404u;
    mma_u8s8_k32(lo, k.a & L, k.a8 & L, k.c & L, k.c8 & L, b[0], b[1]);
    mma_u8s8_k32(hi, k.a & M, k.a8 & M, k.c & M, k.c8 & M, b[2], b[3]);
    mma_u8s8_k32(lo, ((k.a >> 6) & T2) | ((k.e >> sh) & T1), ((k.a8 >> 6) & T2) | ((k.e8 >> sh) & T1),
                 ((k.c >> 6) & T2) | ((k.f >> sh) & T1), ((k.c8 >> 6) & T2) | ((k.f8 >> sh) & T1), b[4], b[5]);
    mma_u8s8_k32(lo, (k.e >> se) & L, (k.e8 >> se) & L, (k.f >> se) & L, (k.f8 >> se) & L, b[6], b[7]);
  }
}

struct ScoreWarp {
  union {
    ExactWarp exact;
    uint8_t qst[4 * QST_ROW];
  };
};
struct __align__(16) ScoreSmem {
  ScoreWarp w[SCORE_WARPS];
  Table table;
  float2 stage[SCORE_WARPS][2][4];  // (m, l) of the first and the last virtual head of a warp's run
  int stage_vh[SCORE_WARPS][2];
};

__device__ __forceinline__ float2 merge_mass(float2 x, float2 y) {  // (m, l) pairs; symmetric in its arguments up to the order of one sum
  const float m = fmaxf(x.x, y.x);
  if (m == -FBLA_INF) return x;
  return make_float2(m, x.y * ex2(x.x - m) + y.y * ex2(y.x - m));
}

// The CTA's share of the score pass: pieces of groups (units of NB sub-blocks) [first, first + count) and window chunk
// numbers [chunk, chunk + chunks); warp w of the CTA takes chunk number w and the run [lo, hi) of the pieces.
template <int QG>
__device__ __forceinline__ void score_item_units(const fbla_k_decode &a, int total, int x_total, int run, int warp, int &chunk, int &lo, int &hi) {
  const int ctas = FBLA_POS::nx(), cta = FBLA_POS::x();
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

template <int CB, int FB, int QG>
__device__ __forceinline__ void score_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  constexpr int NB = 8 / QG, UPG = QG;  // sub-blocks per unit, units per group
  constexpr float HOFF = .5f * ((1 << FB) - 1);
  constexpr int RB = record_bytes(CB);
  ScoreSmem &sm = *reinterpret_cast<ScoreSmem *>(smem_raw);
  const int lane = FBLA_POS::tid() & 31, warp = FBLA_POS::tid() >> 5, gid = lane >> 2, tig = lane & 3;
  const int hpr = a.kv_heads * a.vg;
  wait_previous_pass();  // (lengths, queries and the cache may come from the kernel before)
  allow_next_pass();     // (behind the wait: the value pass then finds everything before this call complete)
  if (FBLA_POS::x() == 0 && FBLA_POS::tid() == 0 && a.status) { a.status[0] = 0; a.status[1] = 0; }
  build_table(a, sm.table, 32 * SCORE_WARPS);
  if (FBLA_POS::x() == 0 && a.lstride)
    for (int i = FBLA_POS::tid(); i <= a.batch; i += 32 * SCORE_WARPS) { table_of(a)[i] = sm.table.closed[i]; table_of(a)[a.batch + 1 + i] = sm.table.exact[i]; }
  const int total = UPG * total_of<false>(a, sm.table.closed, hpr), x_total = total_of<true>(a, sm.table.exact, hpr), run = window_run(a, x_total);
  int chunk, lo, hi;
  score_item_units<QG>(a, total, x_total, run, warp, chunk, lo, hi);
  if (chunk >= 0) exact_range<QG, false>(a, sm.w[warp].exact, lane, chunk * run, min(x_total, (chunk + 1) * run), find<true>(a, sm.table.exact, hpr, chunk * run), window_row(a, chunk));
  __syncwarp();
  uint8_t *const qst = sm.w[warp].qst;
  for (int i = lane; i < 4 * QST_ROW / 4; i += 32) reinterpret_cast<uint32_t *>(qst)[i] = 0u;
  __syncwarp();

  const int cta = FBLA_POS::x();
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
    Cursor c = find<false>(a, sm.table.closed, hpr, lo / UPG);
    int piece = lo % UPG;
    // the group a cursor stands on: its first record and its metadata
    auto records = [&](const Cursor &x, const uint8_t *&rec, const uint8_t *&meta) {
      const size_t unit = (size_t)((x.b * hpr + x.hir) / a.vg) * a.hs + (size_t)group_of(a, x) * a.gs;
      rec = a.c.coarse + unit * SBG * RB;
      meta = reinterpret_cast<const uint8_t *>(a.c.meta) + unit * 1024;
    };
    const uint8_t *rec, *meta;
    records(c, rec, meta);
    uint4 km = __ldg(reinterpret_cast<const uint4 *>(meta) + lane);
    KWords<CB> kw[NB];  // the next unit's words
#pragma unroll
    for (int b = 0; b < NB; ++b) kw[b].load(rec + (piece * NB + b) * RB, gid, tig);
    uint2 q[QG];
    uint32_t B[8];
    float c0[2] = {0.f, 0.f}, sqc[2] = {0.f, 0.f};
    bool fresh = true;  // the group's queries have not been quantised yet
    for (int u = lo; u < hi; ++u) {
      const int vh = c.b * hpr + c.hir;
      if (vh != cur_vh) {
        if (cur_vh >= 0) leave(cur_vh == first_vh ? sm.stage[warp][0] : mass_pair(a, cta + cur_vh));
        else first_vh = vh;
        cur_vh = vh;
        m[0] = m[1] = -FBLA_INF; l[0] = l[1] = 0.f;
#pragma unroll
        for (int qi = 0; qi < QG; ++qi) q[qi] = __ldg(reinterpret_cast<const uint2 *>(a.q + (size_t)q_row(a, c.b, c.hir, qi) * D) + lane);
      }
      if (fresh) {
        fresh = false;
        __syncwarp();
        quantize_rows<QG>(km, q, a.sl, qst, lane, [&](int qi, float sq, float qb, float qsum) {
          const float cc = fmaf(__fmul_rn(sq, HOFF), qsum, qb), s2 = __fmul_rn(sq, (float)(1 << FB));
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (qi == (2 * tig + e) % QG) { c0[e] = cc; sqc[e] = s2; }
        });
        __syncwarp();
        score_frag<CB>(qst, gid % QG, tig, B);
      }
      uint32_t dl[4] = {MAGIC, MAGIC, MAGIC, MAGIC}, dh[4] = {MAGIC, MAGIC, MAGIC, MAGIC};
#pragma unroll
      for (int b = 0; b < NB; ++b) score_products<CB>(kw[b], B, gid / QG == b ? FULL : 0u, tig, dl, dh);
      float *const lse = a.lse + ((size_t)vh * a.nblocks + (size_t)group_of(a, c) * SBG) * QG + 8 * piece + 2 * tig;
      // the next unit's words, and the next group's metadata with the group's first
      if (++piece == UPG) {
        piece = 0;
        fresh = true;
        if (u + 1 < hi) {
          advance<false>(a, hpr, c);
          records(c, rec, meta);
          km = __ldg(reinterpret_cast<const uint4 *>(meta) + lane);
        }
      }
      if (u + 1 < hi) {
#pragma unroll
        for (int b = 0; b < NB; ++b) kw[b].load(rec + (piece * NB + b) * RB, gid, tig);
      }
      constexpr float UN = CB == 4 ? 1.f / 16 : 1.f / 8;
      const float2 x01 = __ffma2_rn(isum2(dh[0], dh[1]), splat(UN), isum2(dl[0], dl[1])), x23 = __ffma2_rn(isum2(dh[2], dh[3]), splat(UN), isum2(dl[2], dl[3]));
      const float2 sq2 = make_float2(sqc[0], sqc[1]), cc2 = make_float2(c0[0], c0[1]);
      const float2 s01 = __ffma2_rn(sq2, x01, cc2), s23 = __ffma2_rn(sq2, x23, cc2);  // tokens gid, gid + 8 of the thread's columns
      float mb[2] = {fmaxf(s01.x, s23.x), fmaxf(s01.y, s23.y)};
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
        for (int e = 0; e < 2; ++e) mb[e] = fmaxf(mb[e], __shfl_xor_sync(FULL, mb[e], o));
      const float2 nm = make_float2(-mb[0], -mb[1]), d01 = __fadd2_rn(s01, nm), d23 = __fadd2_rn(s23, nm);
      const float2 p01 = __ffma2_rn(make_float2(ex2(d01.x), ex2(d01.y)), splat(255.f), splat(MAGICF));
      const float2 p23 = __ffma2_rn(make_float2(ex2(d23.x), ex2(d23.y)), splat(255.f), splat(MAGICF));
      // both columns' sums of p in one word (each below 2^13): low half column 0, high half column 1
      uint32_t ps = (__float_as_uint(p01.x) + __float_as_uint(p23.x)) + ((__float_as_uint(p01.y) + __float_as_uint(p23.y)) << 16) - 2u * MAGIC;
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) ps += __shfl_xor_sync(FULL, ps, o);
      const float2 sp = isum2((ps & 0xffffu) | MAGIC, (ps >> 16) | MAGIC);
      if (gid == 0) *reinterpret_cast<float2 *>(lse) = make_float2(mb[0] + lg2(sp.x), mb[1] + lg2(sp.y));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float mn = fmaxf(m[e], mb[e]);
        l[e] = fmaf(l[e], ex2(m[e] - mn), (e ? sp.y : sp.x) * ex2(mb[e] - mn));
        m[e] = mn;
      }
    }
    leave(sm.stage[warp][cur_vh == first_vh ? 0 : 1]);
  }
  if (lane == 0) {
    sm.stage_vh[warp][0] = first_vh;
    sm.stage_vh[warp][1] = cur_vh != first_vh ? cur_vh : -1;
  }
  __syncthreads();
  // rows of heads that may continue in neighbouring warps, in warp order (as coarse_item's fold)
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    const int v = sm.stage_vh[warp][r];
    if (v < 0) continue;
    if (r == 0 && warp > 0) {
      const int prev = sm.stage_vh[warp - 1][1] >= 0 ? sm.stage_vh[warp - 1][1] : sm.stage_vh[warp - 1][0];
      if (prev == v) continue;
    }
    if (lane < QG) {
      float2 acc = sm.stage[warp][r][lane];
      if (r == 1 || sm.stage_vh[warp][1] < 0)
        for (int x = warp + 1; x < SCORE_WARPS && sm.stage_vh[x][0] == v; ++x) {
          acc = merge_mass(acc, sm.stage[x][0][lane]);
          if (sm.stage_vh[x][1] >= 0) break;
        }
      mass_pair(a, cta + v)[lane] = acc;
    }
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
      const int i = i0 + j * (32 / QG);
      v[j] = make_float2(-FBLA_INF, 0.f);
      if (i < nm) v[j] = __ldcg(mass_pair(a, r.m0 + i + vh) + q);
      else if (i < n) v[j] = __ldcg(reinterpret_cast<const float2 *>(window_row(a, r.x0 + i - nm + vh) + q * PSTRIDE + D));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc = merge_mass(acc, v[j]);
  }
#pragma unroll
  for (int o = QG; o < 32; o <<= 1) {
    const float2 y = make_float2(__shfl_xor_sync(FULL, acc.x, o), __shfl_xor_sync(FULL, acc.y, o));
    acc = (lane & o) ? merge_mass(y, acc) : merge_mass(acc, y);
  }
  return acc.x + lg2(acc.y);  // (-inf for a shard that holds nothing of the row)
}
// the rows' masses into row_r: a shard's first phase, and a pass of its own under an executor. One warp per virtual head.
template <int QG>
__device__ __forceinline__ void mass_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  const int lane = FBLA_POS::tid() & 31, vh = FBLA_POS::x() * 8 + (FBLA_POS::tid() >> 5), hpr = a.kv_heads * a.vg;
  allow_next_pass();
  wait_previous_pass();
  if (vh >= a.batch * hpr) return;
  const int *t = table_of(a);
  const float R = row_mass<QG>(a, rows_of<QG>(a, t, t + a.batch + 1, hpr, vh), vh, lane);
  if (lane < QG) a.row_r[vh * QG + lane] = R;
}

// ---- value pass -------------------------------------------------------------------------------------------------------------------
template <int CB, int FB> struct __align__(128) ValueWarp {
  static constexpr int NST = 2;
  uint8_t pair[NST][2 * (record_bytes(CB) + record_bytes(FB))];  // two coarse records, two fine records
  uint8_t meta[2][1024];
  uint8_t qst[4 * QST_ROW];
  uint8_t pst[128];  // P bytes: [sub-block of the pair][query 0..3][16 tokens]
  float stage[4][PSTRIDE];  // the row set of the first virtual head of the warp's run (the last one's lies in `pair`)
  uint64_t bar[NST], bar_meta[2];
  int stage_vh[2];
};
template <int CB, int FB> struct ValueSmem {
  ValueWarp<CB, FB> w[VALUE_WARPS];
  Table table;
};
static_assert(sizeof(ValueSmem<3, 3>) + 128 <= 227 * 1024 && sizeof(ValueSmem<4, 2>) + 128 <= 227 * 1024, "one CTA's shared memory");

// scores of a record pair of a BITS plane: columns 0-3 the first record's queries, 4-7 the second's. Thread (gid, tig): tokens
// gid, gid + 8 of columns 2 tig, 2 tig + 1. m0 / m1: all ones in the threads whose B column belongs to the first / second record.
template <int BITS>
__device__ __forceinline__ void qk_pair(const uint8_t *ra, const uint8_t *rb, int gid, int tig, const uint32_t (&B)[8], uint32_t m0, uint32_t m1, float2 (&x)[2]) {
  constexpr int NC = BITS == 2 ? 4 : 2;
  uint32_t d[NC][4];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int i = 0; i < 4; ++i) d[c][i] = MAGIC;
#pragma unroll
  for (int par = 0; par < 2; ++par) {
    const uint8_t *rec = par ? rb : ra, *p0 = rec + 16 * gid + 4 * tig, *p1 = p0 + 128;
    const uint32_t m = par ? m1 : m0;
    uint32_t b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) b[i] = B[i] & m;
    if (BITS == 4) {
      const uint32_t a = lds32(p0), a8 = lds32(p1), bb = lds32(p0 + 512), bb8 = lds32(p1 + 512);
      const uint32_t c = lds32(p0 + 256), c8 = lds32(p1 + 256), e = lds32(p0 + 768), e8 = lds32(p1 + 768);
      constexpr uint32_t L = 0x0f0f0f0fu, H = 0xf0f0f0f0u;
      mma_u8s8_k32(d[0], a & L, a8 & L, bb & L, bb8 & L, b[0], b[1]);
      mma_u8s8_k32(d[1], a & H, a8 & H, bb & H, bb8 & H, b[2], b[3]);
      mma_u8s8_k32(d[0], c & L, c8 & L, e & L, e8 & L, b[4], b[5]);
      mma_u8s8_k32(d[1], c & H, c8 & H, e & H, e8 & H, b[6], b[7]);
    } else if (BITS == 2) {
      const uint32_t a = lds32(p0), a8 = lds32(p1), c = lds32(p0 + 256), c8 = lds32(p1 + 256);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t M = 0x03030303u << (2 * k);
        mma_u8s8_k32(d[k % NC], a & M, a8 & M, c & M, c8 & M, b[k], b[4 + k]);
      }
    } else {
      const int sh = 4 + (tig & 1), se = 3 * (tig & 1);
      const uint8_t *q0 = rec + 1024 + 16 * gid + 4 * (tig >> 1), *q1 = q0 + 128;
      const uint32_t a = lds32(p0), a8 = lds32(p1), c = lds32(p0 + 256), c8 = lds32(p1 + 256);
      const uint32_t e = lds32(q0), e8 = lds32(q1), f = lds32(q0 + 8), f8 = lds32(q1 + 8);
      constexpr uint32_t L = 0x07070707u, M = 0x38383838u, T2 = 0x03030303u, T1 = 0x04040404u;
      mma_u8s8_k32(d[0], a & L, a8 & L, c & L, c8 & L, b[0], b[1]);
      mma_u8s8_k32(d[1], a & M, a8 & M, c & M, c8 & M, b[2], b[3]);
      mma_u8s8_k32(d[0], ((a >> 6) & T2) | ((e >> sh) & T1), ((a8 >> 6) & T2) | ((e8 >> sh) & T1),
                   ((c >> 6) & T2) | ((f >> sh) & T1), ((c8 >> 6) & T2) | ((f8 >> sh) & T1), b[4], b[5]);
      mma_u8s8_k32(d[0], (e >> se) & L, (e8 >> se) & L, (f >> se) & L, (f8 >> se) & L, b[6], b[7]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (BITS == 2)
      x[i] = __ffma2_rn(isum2(d[3 % NC][2 * i], d[3 % NC][2 * i + 1]), splat(1.f / 64),
                        __ffma2_rn(isum2(d[2 % NC][2 * i], d[2 % NC][2 * i + 1]), splat(1.f / 16),
                                   __ffma2_rn(isum2(d[1][2 * i], d[1][2 * i + 1]), splat(1.f / 4), isum2(d[0][2 * i], d[0][2 * i + 1]))));
    else
      x[i] = __ffma2_rn(isum2(d[1][2 * i], d[1][2 * i + 1]), splat(BITS == 4 ? 1.f / 16 : 1.f / 8), isum2(d[0][2 * i], d[0][2 * i + 1]));
  }
}

// the sums of one virtual head over the warp's pairs, in units of 2^-R: thread (gid, tig) holds channels 4 (8 u + gid) + cc of
// queries 2 (tig & 1) + e, summed over the sub-blocks of parity tig >> 1
struct Sums {
  float2 l, o[4][4];
};
__device__ __forceinline__ void clear(Sums &s) {
  s.l = make_float2(0.f, 0.f);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) s.o[u][cc] = make_float2(0.f, 0.f);
}
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

template <int CB, int FB, int QG>
__device__ __forceinline__ void value_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  constexpr int RC = record_bytes(CB), RF = record_bytes(FB), NST = ValueWarp<CB, FB>::NST;
  constexpr float HOFF = .5f * ((1 << FB) - 1);
  smem_raw += (128u - (smem_u32(smem_raw) & 127u)) & 127u;
  ValueSmem<CB, FB> &sm = *reinterpret_cast<ValueSmem<CB, FB> *>(smem_raw);
  const int lane = FBLA_POS::tid() & 31, warp = FBLA_POS::tid() >> 5, gid = lane >> 2, tig = lane & 3;
  const int hpr = a.kv_heads * a.vg, cta = FBLA_POS::x();
  ValueWarp<CB, FB> &w = sm.w[warp];
  allow_next_pass();
  build_table(a, sm.table, 32 * VALUE_WARPS);
  const int total = PAIRS * total_of<false>(a, sm.table.closed, hpr), per = (total + (int)FBLA_POS::nx() - 1) / (int)FBLA_POS::nx();
  const int c_lo = min(total, cta * per), c_n = min(total, c_lo + per) - c_lo, wper = (c_n + VALUE_WARPS - 1) / VALUE_WARPS;
  const int lo = c_lo + min(c_n, warp * wper), hi = c_lo + min(c_n, (warp + 1) * wper);
  for (int i = lane; i < 4 * QST_ROW / 4; i += 32) reinterpret_cast<uint32_t *>(w.qst)[i] = 0u;
  reinterpret_cast<uint32_t *>(w.pst)[lane] = 0u;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NST; ++s) mbar_init(&w.bar[s], 1);
    mbar_init(&w.bar_meta[0], 1);
    mbar_init(&w.bar_meta[1], 1);
    mbar_init_fence();
  }
  __syncwarp();
  wait_previous_pass();
  int first_vh = -1, cur_vh = -1;
  bool ok = true;
  if (lo < hi) {
    // The stream of pairs. A cursor stands on a group; `mask` of a group: bit (sub-block QG + query) selected.
    Cursor c = find<false>(a, sm.table.closed, hpr, lo / PAIRS);
    const int J0 = lo % PAIRS;
    const int groups = (hi - 1) / PAIRS - lo / PAIRS + 1;
    float R = 0.f;  // lane l: of query l % QG of the head the issuing side stands on
    auto mass_of = [&](int vh) {
      if (a.mass_given) return __ldcg(a.row_r + vh * QG + lane % QG);
      const float r = row_mass<QG>(a, rows_of<QG>(a, sm.table.closed, sm.table.exact, hpr, vh), vh, lane);
      if (lane < QG) a.row_r[vh * QG + lane] = r;  // for the merge (every warp of the head writes the same)
      return r;
    };
    auto lse_of = [&](const Cursor &x) {  // lane l: (sub-block l / QG, query l % QG) of the group
      return lane < SBG * QG ? __ldcg(a.lse + ((size_t)(x.b * hpr + x.hir) * a.nblocks + (size_t)group_of(a, x) * SBG) * QG + lane) : -FBLA_INF;
    };
    auto issue = [&](const Cursor &x, uint32_t mask, int J, int s, bool with_meta, int ms) {  // lane 0
      const size_t unit = (size_t)((x.b * hpr + x.hir) / a.vg) * a.hs + (size_t)group_of(a, x) * a.gs;
      const bool fine = (mask >> (2 * QG * J)) & ((1u << (2 * QG)) - 1u);
      if (with_meta) {
        mbar_expect_tx(&w.bar_meta[ms], 1024);
        bulk_g2s(w.meta[ms], reinterpret_cast<const uint8_t *>(a.c.meta) + unit * 1024, 1024, &w.bar_meta[ms]);
      }
      mbar_expect_tx(&w.bar[s], 2 * RC + (fine ? 2 * RF : 0));
      bulk_g2s(w.pair[s], a.c.coarse + (unit * SBG + 2 * J) * RC, 2 * RC, &w.bar[s]);
      if (fine) bulk_g2s(w.pair[s] + 2 * RC, a.c.fine + (unit * SBG + 2 * J) * RF, 2 * RF, &w.bar[s]);
    };
    int r_vh = c.b * hpr + c.hir;  // the head R belongs to
    R = mass_of(r_vh);
    uint32_t mask = __ballot_sync(FULL, lse_of(c) - R > a.log2_tau), next_mask = 0;
    float Rc = R;        // R of the group in work
    Cursor n = c;        // the next group
    // group k covers pairs [k ? 0 : J0, ..); chunk number = pair number - lo
    int issued = 0;      // chunks issued
    const int chunks = hi - lo;
    // issues the next chunk; it belongs to group k or, from its pair `cross` on, to group k + 1
    auto issue_next = [&](int pair_in_group, const Cursor &x, uint32_t mk, int ms) {
      if (lane == 0) issue(x, mk, pair_in_group, issued % NST, issued == 0 || pair_in_group == 0, ms);
      ++issued;
    };
    Sums run;
    uint2 q[QG];
    float2 Rq = make_float2(0.f, 0.f);
    int done = 0;        // chunks consumed
    bool have_next = groups > 1;
    if (have_next) {
      advance<false>(a, hpr, n);
      const int nv = n.b * hpr + n.hir;
      if (nv != r_vh) { R = mass_of(nv); r_vh = nv; }
      next_mask = __ballot_sync(FULL, lse_of(n) - R > a.log2_tau);
    }
    // prologue: the first NST chunks
#pragma unroll
    for (int s = 0; s < NST; ++s)
      if (issued < chunks) {
        const int pg = J0 + issued;
        if (pg < PAIRS) issue_next(pg, c, mask, 0); else issue_next(pg - PAIRS, n, next_mask, 1);
      }
    for (int k = 0; k < groups && ok; ++k) {
      const int j0 = k ? 0 : J0, j1 = min(PAIRS, j0 + chunks - done);
      const int vh = c.b * hpr + c.hir;
      float Rn = R;      // R of the next group
      if (vh != cur_vh) {
        if (cur_vh >= 0) { if (cur_vh == first_vh) write_sums<QG>(&w.stage[0][0], run, lane); else write_sums<QG>(value_row(a, cta + cur_vh), run, lane); }
        else first_vh = vh;
        cur_vh = vh;
        clear(run);
        Rq = make_float2(__shfl_sync(FULL, Rc, (2 * (tig & 1)) % QG), __shfl_sync(FULL, Rc, (2 * (tig & 1) + 1) % QG));
#pragma unroll
        for (int qi = 0; qi < QG; ++qi) q[qi] = __ldg(reinterpret_cast<const uint2 *>(a.q + (size_t)q_row(a, c.b, c.hir, qi) * D) + lane);
      }
      // the group after the next: its masses are asked for now and looked at when its first chunk is issued
      Cursor nn = n;
      float nn_lse = -FBLA_INF;
      const bool have_nn = k + 2 < groups;
      if (have_nn) { advance<false>(a, hpr, nn); nn_lse = lse_of(nn); }
      if (!__all_sync(FULL, mbar_wait_bounded(&w.bar_meta[k & 1], (uint32_t)((k >> 1) & 1)))) { ok = false; break; }
      const uint8_t *meta = w.meta[k & 1];
      float2 sq2 = make_float2(0.f, 0.f), qb2 = sq2, c02 = sq2;
      __syncwarp();
      quantize_rows<QG>(lds128(meta + 16 * lane), q, a.sl, w.qst, lane, [&](int qi, float sq, float qb, float qsum) {
        const float cc = fmaf(__fmul_rn(sq, HOFF), qsum, qb);
        if (qi == 2 * (tig & 1)) { sq2.x = sq; qb2.x = qb; c02.x = cc; }
        if (qi == 2 * (tig & 1) + 1) { sq2.y = sq; qb2.y = qb; c02.y = cc; }
      });
      __syncwarp();
      uint32_t B[8];
      qhat_frag<CB>(w.qst, gid & 3, tig, B);
      const uint32_t m0 = gid < 4 ? FULL : 0u, m1 = ~m0;
      float2 A[4][4], L = make_float2(0.f, 0.f), Hc = L;  // the group's sums in code units; sum w sum p, and its unselected part
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) A[u][cc] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int J = j0; J < j1; ++J) {
        const int s = done % NST;
        if (!__all_sync(FULL, mbar_wait_bounded(&w.bar[s], (uint32_t)((done / NST) & 1)))) { ok = false; break; }
        ++done;
        const uint8_t *ra = w.pair[s], *rb = ra + RC, *fa = ra + 2 * RC, *fb = fa + RF;
        const uint32_t pm = (mask >> (2 * QG * J)) & ((1u << (2 * QG)) - 1u);  // the pair's selections
        const bool fine = pm != 0;
        // the thread's two columns: sub-block tig >> 1, queries 2 (tig & 1) + e
        const uint32_t mine = pm >> (QG * (tig >> 1) + 2 * (tig & 1));
        const float2 sel = make_float2(mine & 1u && query_valid<QG>(tig, 0) ? 1.f : 0.f, mine & 2u && query_valid<QG>(tig, 1) ? 1.f : 0.f);
        float2 x[2], y[2];
        qk_pair<CB>(ra, rb, gid, tig, B, m0, m1, x);
        float2 cst = c02;
        if (fine) {
          qk_pair<FB>(fa, fb, gid, tig, B, m0, m1, y);
          cst = make_float2(sel.x != 0.f ? qb2.x : c02.x, sel.y != 0.f ? qb2.y : c02.y);
#pragma unroll
          for (int i = 0; i < 2; ++i) x[i] = __ffma2_rn(splat((float)(1 << FB)), x[i], __fmul2_rn(sel, y[i]));  // whole numbers, exact
        } else {
#pragma unroll
          for (int i = 0; i < 2; ++i) x[i] = __fmul2_rn(splat((float)(1 << FB)), x[i]);
        }
        const float2 s0 = __ffma2_rn(sq2, x[0], cst), s1 = __ffma2_rn(sq2, x[1], cst);
        float mb[2] = {fmaxf(s0.x, s1.x), fmaxf(s0.y, s1.y)};
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
          for (int e = 0; e < 2; ++e) mb[e] = fmaxf(mb[e], __shfl_xor_sync(FULL, mb[e], o));
        const float2 nm = make_float2(-mb[0], -mb[1]), d0 = __fadd2_rn(s0, nm), d1 = __fadd2_rn(s1, nm);
        const float2 p0 = __ffma2_rn(make_float2(ex2(d0.x), ex2(d0.y)), splat(255.f), splat(MAGICF));
        const float2 p1 = __ffma2_rn(make_float2(ex2(d1.x), ex2(d1.y)), splat(255.f), splat(MAGICF));
        if (query_valid<QG>(tig, 0)) { w.pst[32 * tig + gid] = (uint8_t)__float_as_uint(p0.x); w.pst[32 * tig + gid + 8] = (uint8_t)__float_as_uint(p1.x); }
        if (query_valid<QG>(tig, 1)) { w.pst[32 * tig + 16 + gid] = (uint8_t)__float_as_uint(p0.y); w.pst[32 * tig + 16 + gid + 8] = (uint8_t)__float_as_uint(p1.y); }
        const float2 wt = make_float2(query_valid<QG>(tig, 0) ? ex2(mb[0] - Rq.x) : 0.f, query_valid<QG>(tig, 1) ? ex2(mb[1] - Rq.y) : 0.f);
        const float2 ws = __fmul2_rn(wt, sel);
        __syncwarp();
        const uint32_t pw = lds32(w.pst + 4 * lane), b0 = pw & m0, b1 = pw & m1;
        {
          uint32_t d[4];
          mma_u8u8_k32_from(d, 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u, b0, b1, MAGIC);
          const float2 sp = isum2(d[0], d[1]);
          L = __ffma2_rn(wt, sp, L);
          Hc = __ffma2_rn(__fadd2_rn(wt, make_float2(-ws.x, -ws.y)), sp, Hc);
        }
        // the weights times the planes' class factors: code units = 2^FB h + f
        float2 wc[4], wf[4];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          wc[cc] = __fmul2_rn(wt, splat((float)(1 << FB) * v_unscale<CB>(cc)));
          wf[cc] = __fmul2_rn(ws, splat(v_unscale<FB>(cc)));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint32_t va[4], vb[4], d01[4], d23[4];
          v_slots<CB>(ra, 8 * u + gid, tig, va);
          v_slots<CB>(rb, 8 * u + gid, tig, vb);
          mma_u8u8_k32_from(d01, va[0], va[1], vb[0], vb[1], b0, b1, MAGIC);
          mma_u8u8_k32_from(d23, va[2], va[3], vb[2], vb[3], b0, b1, MAGIC);
          A[u][0] = __ffma2_rn(wc[0], isum2(d01[0], d01[1]), A[u][0]);
          A[u][1] = __ffma2_rn(wc[1], isum2(d01[2], d01[3]), A[u][1]);
          A[u][2] = __ffma2_rn(wc[2], isum2(d23[0], d23[1]), A[u][2]);
          A[u][3] = __ffma2_rn(wc[3], isum2(d23[2], d23[3]), A[u][3]);
        }
        if (fine) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t va[4], vb[4], d01[4], d23[4];
            v_slots<FB>(fa, 8 * u + gid, tig, va);
            v_slots<FB>(fb, 8 * u + gid, tig, vb);
            mma_u8u8_k32_from(d01, va[0], va[1], vb[0], vb[1], b0, b1, MAGIC);
            mma_u8u8_k32_from(d23, va[2], va[3], vb[2], vb[3], b0, b1, MAGIC);
            A[u][0] = __ffma2_rn(wf[0], isum2(d01[0], d01[1]), A[u][0]);
            A[u][1] = __ffma2_rn(wf[1], isum2(d01[2], d01[3]), A[u][1]);
            A[u][2] = __ffma2_rn(wf[2], isum2(d23[0], d23[1]), A[u][2]);
            A[u][3] = __ffma2_rn(wf[3], isum2(d23[2], d23[3]), A[u][3]);
          }
        }
        __syncwarp();  // the slot and pst have been read
        if (issued < chunks) {
          const int pg = J + NST;
          if (pg < PAIRS) issue_next(pg, c, mask, k & 1); else issue_next(pg - PAIRS, n, next_mask, (k + 1) & 1);
        }
      }
      if (!ok) break;
      run.l = __fadd2_rn(run.l, L);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint4 vm = lds128(meta + 512 + 16 * (8 * u + gid));
        const float vb[4] = {bf_lo(vm.x), bf_hi(vm.x), bf_lo(vm.y), bf_hi(vm.y)}, vs[4] = {bf_lo(vm.z), bf_hi(vm.z), bf_lo(vm.w), bf_hi(vm.w)};
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
          run.o[u][cc] = __fadd2_rn(run.o[u][cc], __ffma2_rn(splat(vs[cc]), __ffma2_rn(splat(HOFF), Hc, A[u][cc]), __fmul2_rn(splat(vb[cc]), L)));
      }
      // on to the next group
      c = n; mask = next_mask; Rc = Rn;
      if (have_nn) {
        const int nv = nn.b * hpr + nn.hir;
        if (nv != r_vh) { R = mass_of(nv); r_vh = nv; }
        next_mask = __ballot_sync(FULL, nn_lse - R > a.log2_tau);
        n = nn;
      }
    }
    if (ok) {
      __syncwarp();
      write_sums<QG>(cur_vh == first_vh ? &w.stage[0][0] : reinterpret_cast<float *>(w.pair[0]), run, lane);
    } else if (lane == 0) report(a, 3);
  }
  __syncwarp();
  if (ok && lane == 0) {
#pragma unroll
    for (int s = 0; s < NST; ++s) mbar_inval(&w.bar[s]);
    mbar_inval(&w.bar_meta[0]);
    mbar_inval(&w.bar_meta[1]);
  }
  if (lane == 0) {
    w.stage_vh[0] = ok ? first_vh : -1;
    w.stage_vh[1] = ok && cur_vh != first_vh ? cur_vh : -1;
  }
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {  // rows of heads that may continue in neighbouring warps, added in warp order
    const int v = w.stage_vh[r];
    if (v < 0) continue;
    if (r == 0 && warp > 0) {
      const ValueWarp<CB, FB> &prev = sm.w[warp - 1];
      if ((prev.stage_vh[1] >= 0 ? prev.stage_vh[1] : prev.stage_vh[0]) == v) continue;
    }
    const bool open = r == 1 || w.stage_vh[1] < 0;
    const float *own = r ? reinterpret_cast<const float *>(w.pair[0]) : &w.stage[0][0];
    float *dst = value_row(a, cta + v);
    for (int i = lane; i < QG * (PSTRIDE / 4); i += 32) {
      float4 s = reinterpret_cast<const float4 *>(own)[i];
      if (open)
        for (int x = warp + 1; x < VALUE_WARPS && sm.w[x].stage_vh[0] == v; ++x) {
          const float4 y = reinterpret_cast<const float4 *>(&sm.w[x].stage[0][0])[i];
          s.x += y.x; s.y += y.y; s.z += y.z; s.w += y.w;
          if (sm.w[x].stage_vh[1] >= 0) break;
        }
      reinterpret_cast<float4 *>(dst)[i] = s;
    }
  }
}

// ---- merge: out = (sum 2^(m_x - R) o_x + sum o_v) / (sum 2^(m_x - R) l_x + sum l_v), BF16 -----------------------------------
// One CTA of four warps per output row: warp s sums rows s, s + 4, ... of the head's window and value rows, lane c channels
// 4 c .. 4 c + 3; the four sums are added in order.
template <int QG>
__device__ __forceinline__ void gather_item(const fbla_k_decode &a, uint8_t *smem_raw) {
  __shared__ float4 so[4][32];
  __shared__ float sl[4];
  const int vh = FBLA_POS::x() / QG, qi = FBLA_POS::x() % QG, lane = FBLA_POS::tid() & 31, warp = FBLA_POS::tid() >> 5;
  const int hpr = a.kv_heads * a.vg, b = vh / hpr, hir = vh - b * hpr;
  allow_next_pass();
  wait_previous_pass();
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

}  // namespace dense
}  // namespace fbla
