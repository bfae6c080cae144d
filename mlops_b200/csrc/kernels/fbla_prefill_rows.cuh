// Causal prefill attention of a few query rows over the compressed cache (chunks of fewer than 64 rows per KV head: drafted
// tokens, short continuations), sm_100a.
//
// Semantics (the reference's DP4A prefill, attention/fbla/src/fbla_prefill.cuh:389-705) -- the row at position p attends
// to 0..p: group 0 (sink) and its own group in BF16 from the windows / the chunk, closed groups 1..own-1 through their
// full 6-bit codes (coarse << FB | fine) with the per-(row, group) int8 qhat, 16-token integer P blocks everywhere.
//
// Eight rows of one KV head (a row tile) are the eight columns of the decode's integer tensor-core products, both planes joined
// to their codes on the way into the fragments (fbla_frag.cuh). A CTA's twelve warps are dealt to one to four row tiles, and a
// tile's closed groups, in pairs of sub-blocks, to its warps, each streaming its run through a private two-stage ring with a
// running (m, l, o); the BF16 blocks follow on BF16 products; the warps' rows are then merged in warp order. A long cache and
// few tiles would leave most SMs idle, so the pairs are also split into shares, one CTA of a thread-block cluster each, whose
// merged rows the cluster reads from each other's shared memory: no scratch, no second launch. Tiles and shares follow from the
// sizes alone (row_deal), and a CTA that has to do every share (an executor's item) takes them one after the other, so that
// both give the same bits.
// Bound by instruction latency: three warps per scheduler (the sums take the registers) issue about 0.5 instructions per cycle.
// 4 sequences x 5 drafted tokens at 12 345 tokens (32 / 8 heads): one warp per row walking the whole cache 1 670 us; a tile
// to a CTA and as many shares as even out the groups 120 (96 clusters of three: three waves); the deal 78; joined codes 65.
#pragma once
#include "fbla_decode.cuh"

namespace fbla {
namespace rows {

constexpr int WARPS = 12, COLS = 8, PAIRS = SBG / 2, NST = 2;
constexpr int MAX_SHARES = FBLA_K_ROW_SHARES, MAX_TILES = 4;
constexpr int SET = COLS * FBLA_K_PSTRIDE;  // floats of a tile's row set: per row o[128], m, l

// How the rows of `heads` KV heads are dealt: `tiles` row tiles to a CTA, `shares` CTAs (a cluster) to those tiles' groups.
struct RowDeal { int tiles, shares; };
// The deal whose longest SM has least to do: waves of CTAs x (a CTA's fixed cost + pairs of a warp). The fixed cost -- queries,
// BF16 blocks, merges -- measured as that of five pairs. SMs: a B200's 148, whatever the device, so that the choice is one of
// the sizes alone; clusters: what fits GPCs of 16, as every GPC has at least that many (96 clusters of three took three waves).
// No more shares than give a CTA twelve groups, so that a launch whose length is on the device need not make larger clusters
// than the cache's room asks for.
__host__ __device__ inline int deal_cost(int t, int c, int row_tiles, int heads, int groups) {  // (what is no deal: the largest cost)
  if (t > MAX_TILES || (t > 1 && t > row_tiles) || (c > 1 && WARPS * (c - 1) >= groups)) return (1 << 26) - 1;
  const int room = c == 1 ? 148 : 8 * (16 / c) * c, warps = WARPS / t * c;
  const long long cost = (long long)(((row_tiles + t - 1) / t * heads * c + room - 1) / room) * (5 + (PAIRS * groups + warps - 1) / warps);
  return cost < (1 << 26) - 2 ? (int)cost : (1 << 26) - 2;
}
__host__ __device__ inline RowDeal row_deal(int row_tiles, int heads, int groups) {
#ifdef __CUDA_ARCH__  // a lane per deal (every thread of the warp is here)
  static_assert(MAX_TILES * MAX_SHARES == 32, "a deal per lane");
  const unsigned lane = FBLA_POS::tid() & 31, n = __reduce_min_sync(FULL, (unsigned)deal_cost(1 + lane / MAX_SHARES, 1 + lane % MAX_SHARES, row_tiles, heads, groups) << 5 | lane) & 31;
#else
  int n = 0;
  for (int x = 0, least = 1 << 26; x < MAX_TILES * MAX_SHARES; ++x) {
    const int cost = deal_cost(1 + x / MAX_SHARES, 1 + x % MAX_SHARES, row_tiles, heads, groups);
    if (cost < least) { least = cost; n = x; }
  }
#endif
  RowDeal d;
  d.tiles = 1 + n / MAX_SHARES; d.shares = 1 + n % MAX_SHARES;
  return d;
}

template <int CB, int FB> struct __align__(128) RowWarp {
  uint8_t pair[NST][2 * (record_bytes(CB) + record_bytes(FB))];  // two coarse records, two fine records; later the warp's row set and BF16 staging
  uint8_t meta[2][1024];
  uint8_t qst[COLS * QST_ROW];
  uint8_t pst[128];  // P bytes of a sub-block: [row][16 tokens]
  uint64_t bar[NST], bar_meta[2];
};
struct __align__(16) RowStage {  // BF16 staging of a warp, in its ring
  uint16_t v[S][D + 8];
  uint16_t p[COLS][S];
};
template <int CB, int FB> struct RowSmem {
  RowWarp<CB, FB> w[WARPS];
  uint16_t q[MAX_TILES][COLS][D + 8];  // the tiles' queries, BF16 (rows past the end: zero)
  float share[MAX_TILES][SET];         // the merged row sets of the shares this CTA has done
  int failed;
};
static_assert(sizeof(RowSmem<3, 3>) + 128 <= 227 * 1024 && sizeof(RowSmem<4, 2>) + 128 <= 227 * 1024, "one CTA's shared memory");
static_assert(SET * sizeof(float) + sizeof(RowStage) <= sizeof(RowWarp<4, 2>::pair) && SET * sizeof(float) + sizeof(RowStage) <= sizeof(RowWarp<3, 3>::pair), "row set and staging fit the ring");

// the sums of a warp: rows 2 tig + e, e = 0, 1, in (.x, .y); channels 4 (8 u + gid) + cc
struct State { float m[2]; float2 l, o[4][4]; };

// ---- the warp's run of pairs [lo, hi) of the closed groups (pair p: sub-blocks 2 (p % 4), + 1 of group 1 + p / 4) ----------------
// own[e]: the group of row 2 tig + e (it attends to the closed groups before it). false: a bounded wait gave up.
template <int CB, int FB>
__device__ __forceinline__ bool closed_run(const fbla_k_prefill &a, RowWarp<CB, FB> &w, const uint16_t (&q)[COLS][D + 8], size_t head, int lo, int hi,
                                           const int (&own)[2], uint32_t &uses, State &st, int lane) {
  constexpr int RC = record_bytes(CB), RF = record_bytes(FB);
  // A group's integer sums are read as the FP32 subnormals of the same bits (2^-149 each); the weights carry 2^75, the group's end 2^74
  constexpr float UP = 37778931862957161709568.f /* 2^75 */, BACK = 18889465931478580854784.f /* 2^74 */;
  const int gid = lane >> 2, tig = lane & 3;
  const uint32_t base = uses;  // ring uses before this run (the barriers live through all of a CTA's shares)
  auto issue = [&](int p) {    // lane 0
    const int s = (base + (p - lo)) % NST, J = p % PAIRS, ms = (p / PAIRS) & 1;
    const size_t unit = head + (size_t)(1 + p / PAIRS) * a.gs;
    const bool meta = p == lo || J == 0;
    mbar_expect_tx(&w.bar[s], 2 * (RC + RF) + (meta ? 1024 : 0));
    bulk_g2s(w.pair[s], a.c.coarse + (unit * SBG + 2 * J) * RC, 2 * RC, &w.bar[s]);
    bulk_g2s(w.pair[s] + 2 * RC, a.c.fine + (unit * SBG + 2 * J) * RF, 2 * RF, &w.bar[s]);
    if (meta) bulk_g2s(w.meta[ms], reinterpret_cast<const uint8_t *>(a.c.meta) + unit * 1024, 1024, &w.bar[s]);
  };
  if (lane == 0) {
    fence_async_smem();  // (the ring may have held a row set)
#pragma unroll
    for (int s = 0; s < NST; ++s)
      if (lo + s < hi) issue(lo + s);
  }
  int p = lo;
  while (p < hi) {
    const int g = 1 + p / PAIRS, end = min(hi, (p / PAIRS + 1) * PAIRS);
    const uint8_t *meta = w.meta[(p / PAIRS) & 1];
    float2 sq2 = make_float2(0.f, 0.f), qb2 = sq2, A[4][4], L = sq2;
    uint32_t B[8];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) A[u][cc] = make_float2(0.f, 0.f);
    const bool on[2] = {g < own[0], g < own[1]};
    for (bool first = true; p < end; ++p, first = false) {
      const uint32_t use = base + (p - lo);
      if (!__all_sync(FULL, mbar_wait_bounded(&w.bar[use % NST], (use / NST) & 1))) return false;
      if (first) {  // the rows' qhat for this group
        const uint4 km = lds128(meta + 16 * lane);
#pragma unroll
        for (int r = 0; r < COLS; ++r) {
          const uint2 qw = *reinterpret_cast<const uint2 *>(&q[r][4 * lane]);
          float sq, qb, qsum;
          reinterpret_cast<uint32_t *>(w.qst + QST_ROW * r)[lane] = quantize_query_word(km, make_float4(bf_lo(qw.x), bf_hi(qw.x), bf_lo(qw.y), bf_hi(qw.y)), a.sl, sq, qb, qsum);
          if (r == 2 * tig) { sq2.x = sq; qb2.x = qb; }
          if (r == 2 * tig + 1) { sq2.y = sq; qb2.y = qb; }
        }
        __syncwarp();
        qhat_frag<CB>(w.qst, gid, tig, B);
      }
#pragma unroll 1
      for (int par = 0; par < 2; ++par) {
        const uint8_t *crec = w.pair[use % NST] + par * RC, *frec = w.pair[use % NST] + 2 * RC + par * RF;
        float2 x[2];
        qk_full<CB, FB>(crec, frec, gid, tig, B, x);
        const float2 s0 = __ffma2_rn(sq2, x[0], qb2), s1 = __ffma2_rn(sq2, x[1], qb2);
        float mb[2] = {fmaxf(s0.x, s1.x), fmaxf(s0.y, s1.y)};
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
          for (int e = 0; e < 2; ++e) mb[e] = fmaxf(mb[e], __shfl_xor_sync(FULL, mb[e], o));
        // the running maximum moves only when a block exceeds it by more than 2^8
        const bool grow0 = on[0] && mb[0] > st.m[0] + 8.f, grow1 = on[1] && mb[1] > st.m[1] + 8.f;
        if (__any_sync(FULL, grow0 || grow1)) {
          const float al0 = grow0 ? ex2(st.m[0] - mb[0]) : 1.f, al1 = grow1 ? ex2(st.m[1] - mb[1]) : 1.f;
          if (grow0) st.m[0] = mb[0];
          if (grow1) st.m[1] = mb[1];
          const float2 al = make_float2(al0, al1);
          st.l = __fmul2_rn(st.l, al);
          L = __fmul2_rn(L, al);
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) { st.o[u][cc] = __fmul2_rn(st.o[u][cc], al); A[u][cc] = __fmul2_rn(A[u][cc], al); }
        }
        const float2 nm = make_float2(-mb[0], -mb[1]), d0 = __fadd2_rn(s0, nm), d1 = __fadd2_rn(s1, nm);
        const float2 p0 = __ffma2_rn(make_float2(ex2(d0.x), ex2(d0.y)), splat(255.f), splat(MAGICF));
        const float2 p1 = __ffma2_rn(make_float2(ex2(d1.x), ex2(d1.y)), splat(255.f), splat(MAGICF));
        w.pst[32 * tig + gid] = (uint8_t)__float_as_uint(p0.x); w.pst[32 * tig + gid + 8] = (uint8_t)__float_as_uint(p1.x);
        w.pst[32 * tig + 16 + gid] = (uint8_t)__float_as_uint(p0.y); w.pst[32 * tig + 16 + gid + 8] = (uint8_t)__float_as_uint(p1.y);
        const float2 wt = make_float2(on[0] ? ex2(mb[0] - st.m[0]) : 0.f, on[1] ? ex2(mb[1] - st.m[1]) : 0.f);
        __syncwarp();
        const uint32_t b0 = lds32(w.pst + 4 * lane);  // row gid, tokens 4 tig ..
        const float2 w0 = __fmul2_rn(wt, splat(UP)), w1 = __fmul2_rn(wt, splat(UP * v_full_unscale<CB>(1)));
        {
          uint32_t d[4];
          mma_u8u8_k16_zero(d, 0x01010101u, 0x01010101u, b0);
          L = __ffma2_rn(w0, tiny2(d[0], d[1]), L);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint32_t v[4], d01[4], d23[4];
          v_full<CB, FB>(crec, frec, 8 * u + gid, tig, v);
          mma_u8u8_k16_zero(d01, v[0], v[1], b0);
          mma_u8u8_k16_zero(d23, v[2], v[3], b0);
          A[u][0] = __ffma2_rn(w0, tiny2(d01[0], d01[1]), A[u][0]);
          A[u][1] = __ffma2_rn(w1, tiny2(d01[2], d01[3]), A[u][1]);
          A[u][2] = __ffma2_rn(w1, tiny2(d23[0], d23[1]), A[u][2]);
          A[u][3] = __ffma2_rn(w1, tiny2(d23[2], d23[3]), A[u][3]);
        }
        __syncwarp();  // pst -- and behind the second sub-block the slot -- has been read
      }
      if (lane == 0 && p + NST < hi) issue(p + NST);
    }
    L = __fmul2_rn(L, splat(BACK));
    st.l = __fadd2_rn(st.l, L);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint4 vm = lds128(meta + 512 + 16 * (8 * u + gid));
      const float vb[4] = {bf_lo(vm.x), bf_hi(vm.x), bf_lo(vm.y), bf_hi(vm.y)}, vs[4] = {bf_lo(vm.z), bf_hi(vm.z), bf_lo(vm.w), bf_hi(vm.w)};
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) st.o[u][cc] = __ffma2_rn(splat(vs[cc]), __fmul2_rn(splat(BACK), A[u][cc]), __ffma2_rn(splat(vb[cc]), L, st.o[u][cc]));
    }
    __syncwarp();
  }
  uses = base + (uint32_t)max(hi - lo, 0);
  return true;
}

// the warp's row set in shared memory: per row o[128], m, l
__device__ __forceinline__ void write_state(float *set, const State &st, int lane) {
  const int gid = lane >> 2, tig = lane & 3;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    float *row = set + (2 * tig + e) * FBLA_K_PSTRIDE;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      *reinterpret_cast<float4 *>(row + 4 * (8 * u + gid)) = e ? make_float4(st.o[u][0].y, st.o[u][1].y, st.o[u][2].y, st.o[u][3].y)
                                                                : make_float4(st.o[u][0].x, st.o[u][1].x, st.o[u][2].x, st.o[u][3].x);
    if (gid == 0) { row[D] = st.m[e]; row[D + 1] = e ? st.l.y : st.l.x; }
  }
}

// BF16 sub-blocks first, first + step, ... < total of the tile's list, added to the warp's row set. Block n < sink: n-th of group
// 0; else (n - sink) % 8 of group own_lo + (n - sink) / 8. Row 2 tig + e stands at pos[e] (-1: no such row) in group own[e].
template <class RowOf>
__device__ __forceinline__ void exact_blocks(const fbla_k_prefill &a, const uint16_t (&q)[COLS][D + 8], RowStage &sm, float *set, int first, int step, int total,
                                             int sink, int own_lo, int n1, const int (&pos)[2], const int (&own)[2], int lane, RowOf row_of) {
  if (first >= total) return;
  const int gid = lane >> 2, tig = lane & 3;
  float m[2] = {-FBLA_INF, -FBLA_INF}, l[2] = {0.f, 0.f}, o[8][4];
#pragma unroll
  for (int mt = 0; mt < 8; ++mt) o[mt][0] = o[mt][1] = o[mt][2] = o[mt][3] = 0.f;
#pragma unroll 1
  for (int n = first; n < total; n += step) {
    const int g = n < sink ? 0 : own_lo + (n - sink) / SBG, t0 = g * G + S * (n < sink ? n : (n - sink) % SBG);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // V rows
      const int r = 2 * i + (lane >> 4);
      const uint4 v = t0 + r < n1 ? __ldcg(reinterpret_cast<const uint4 *>(row_of(t0 + r, 1)) + (lane & 15)) : make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4 *>(&sm.v[r][8 * (lane & 15)]) = v;
    }
    float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r4 = 0; r4 < 4; ++r4) {  // channels 32 r4 + 8 tig .. of tokens gid, gid + 8
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      const uint4 ka = t0 + gid < n1 ? __ldcg(reinterpret_cast<const uint4 *>(row_of(t0 + gid, 0) + 32 * r4 + 8 * tig)) : zero;
      const uint4 kb = t0 + gid + 8 < n1 ? __ldcg(reinterpret_cast<const uint4 *>(row_of(t0 + gid + 8, 0) + 32 * r4 + 8 * tig)) : zero;
      const uint4 qq = *reinterpret_cast<const uint4 *>(&q[gid][32 * r4 + 8 * tig]);
      mma_bf16_k16(x, ka.x, kb.x, ka.y, kb.y, qq.x, qq.y);
      mma_bf16_k16(x, ka.z, kb.z, ka.w, kb.w, qq.z, qq.w);
    }
    float al[2], wt[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool here = g == 0 || own[e] == g;
      const float s0 = here && t0 + gid <= pos[e] ? __fmul_rn(x[e], a.sl) : -FBLA_INF, s1 = here && t0 + gid + 8 <= pos[e] ? __fmul_rn(x[2 + e], a.sl) : -FBLA_INF;
      float mb = fmaxf(s0, s1);
#pragma unroll
      for (int off = 4; off <= 16; off <<= 1) mb = fmaxf(mb, __shfl_xor_sync(FULL, mb, off));
      const bool any = mb > -FBLA_INF;  // (a row that attends to nothing here keeps its sums)
      const float mn = any ? fmaxf(m[e], mb) : m[e], mr = any ? mb : 0.f;
      al[e] = any ? ex2(m[e] - mn) : 1.f;
      wt[e] = any ? ex2(mb - mn) : 0.f;
      m[e] = mn;
      const float p0 = fmaf(ex2(s0 - mr), 255.f, MAGICF) - MAGICF, p1 = fmaf(ex2(s1 - mr), 255.f, MAGICF) - MAGICF;
      sm.p[2 * tig + e][gid] = (uint16_t)(__float_as_uint(p0) >> 16);
      sm.p[2 * tig + e][gid + 8] = (uint16_t)(__float_as_uint(p1) >> 16);
      float sp = p0 + p1;
#pragma unroll
      for (int off = 4; off <= 16; off <<= 1) sp += __shfl_xor_sync(FULL, sp, off);
      l[e] = fmaf(al[e], l[e], wt[e] * sp);
    }
    __syncwarp();
    const uint32_t pb0 = *reinterpret_cast<const uint32_t *>(&sm.p[gid][2 * tig]), pb1 = *reinterpret_cast<const uint32_t *>(&sm.p[gid][2 * tig + 8]);
#pragma unroll
    for (int mt = 0; mt < 8; ++mt) {
      uint32_t va[4];
      ldmatrix_x4_trans(va, &sm.v[8 * (lane >> 4) + (lane & 7)][16 * mt + 8 * ((lane >> 3) & 1)]);
      float y[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16_k16(y, va[0], va[1], va[2], va[3], pb0, pb1);
      o[mt][0] = fmaf(al[0], o[mt][0], wt[0] * y[0]); o[mt][1] = fmaf(al[1], o[mt][1], wt[1] * y[1]);
      o[mt][2] = fmaf(al[0], o[mt][2], wt[0] * y[2]); o[mt][3] = fmaf(al[1], o[mt][3], wt[1] * y[3]);
    }
  }
  // into the row set
  float sa[2], sb[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    float *row = set + (2 * tig + e) * FBLA_K_PSTRIDE;
    const float ms = row[D], ls = row[D + 1], mn = fmaxf(ms, m[e]);
    sa[e] = ms == -FBLA_INF ? 0.f : ex2(ms - mn);
    sb[e] = m[e] == -FBLA_INF ? 0.f : ex2(m[e] - mn);
#pragma unroll
    for (int mt = 0; mt < 8; ++mt) {
      row[16 * mt + gid] = fmaf(sa[e], row[16 * mt + gid], sb[e] * o[mt][e]);
      row[16 * mt + gid + 8] = fmaf(sa[e], row[16 * mt + gid + 8], sb[e] * o[mt][2 + e]);
    }
    __syncwarp();
    if (gid == 0) { row[D] = mn; row[D + 1] = fmaf(sa[e], ls, sb[e] * l[e]); }
  }
}
// another share's sums (m, l, y) added to the sums (M, L, o) of the shares before it
__device__ __forceinline__ void add_share(float &M, float &L, float4 &o, float m, float l, float4 y) {
  const float mn = fmaxf(M, m), sa = M == -FBLA_INF ? 0.f : ex2(M - mn), sb = m == -FBLA_INF ? 0.f : ex2(m - mn);
  M = mn;
  L = fmaf(sa, L, sb * l);
  o.x = fmaf(sa, o.x, sb * y.x); o.y = fmaf(sa, o.y, sb * y.y); o.z = fmaf(sa, o.z, sb * y.z); o.w = fmaf(sa, o.w, sb * y.w);
}
}  // namespace rows

// CTA x of head y: bundle x / cluster of the deal's tiles, share x % cluster (cluster 1: every share of the bundle, one after the other)
template <int CB, int FB>
__device__ __forceinline__ void attend_rows_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  using namespace rows;
  smem_raw += (128u - (smem_u32(smem_raw) & 127u)) & 127u;
  RowSmem<CB, FB> &sm = *reinterpret_cast<RowSmem<CB, FB> *>(smem_raw);
  const int tid = FBLA_POS::tid(), lane = tid & 31, warp = tid >> 5, tig = lane & 3;
  const int bh = FBLA_POS::y(), b = bh / a.kv_heads, kh = bh - b * a.kv_heads, qg = a.q_heads / a.kv_heads;
  const int n0 = (a.length ? FBLA_POS::ro(a.length + (a.lstride ? b : 0)) : 0) + a.n0;
  const int count = a.dcount ? FBLA_POS::ro(a.dcount) : a.count, n1 = n0 + count, rows = count * qg;
  const int cluster = a.cluster, rank = FBLA_POS::x() % cluster;
  if (a.tc_min_rows && rows >= a.tc_min_rows) return;  // (a long device count is the tensor-core pass's work)
  const RowDeal deal = row_deal((rows + COLS - 1) / COLS, a.batch * a.kv_heads, (n1 - 1) / G);
  const int shares = deal.shares, first_row = FBLA_POS::x() / cluster * deal.tiles * COLS, held = deal.tiles * COLS;
  if (first_row >= rows) return;  // (cluster-uniform)
  // the warp's tile, and its place among the tile's warps
  const int per_tile = WARPS / deal.tiles, tile = min(warp / per_tile, deal.tiles - 1), place = warp - tile * per_tile;
  const int r0 = first_row + tile * COLS;
  const bool live = r0 < rows && place < per_tile;
  const int last = min(r0 + COLS, rows) - 1, max_pos = n0 + last / qg, own_min = (n0 + r0 / qg) / G, own_max = max_pos / G;
  const int pairs = live ? PAIRS * max(own_max - 1, 0) : 0;
  // the BF16 blocks: group 0, then the rows' own groups
  const int sink = min(SBG, max_pos / S + 1), own_lo = max(own_min, 1);
  const int exact = live ? sink + (own_max >= own_lo ? SBG * (own_max - own_lo) + (max_pos - own_max * G) / S + 1 : 0) : 0;
  int pos[2], own[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = r0 + 2 * tig + e;
    pos[e] = r < rows ? n0 + r / qg : -1;
    own[e] = r < rows ? pos[e] / G : 0;
  }
  const size_t eh = (size_t)bh * G * D, ih = (size_t)bh * a.count * D;
  // the BF16 row of position tp: the chunk, the sink window, or the window of the group that was open before the chunk
  auto token_row = [&](int tp, int x) -> const uint16_t * {
    return tp >= n0 ? (x ? a.v : a.k) + ih + (size_t)(tp - n0) * D : tp < G ? (x ? a.c.sink_v : a.c.sink_k) + eh + (size_t)tp * D
                                                                         : (x ? a.c.open_v : a.c.open_k) + eh + (size_t)(tp - (n0 - 1) / G * G) * D;
  };
  if (tid == 0) sm.failed = 0;
  for (int e = tid; e < held * (D / 8); e += 32 * WARPS) {
    const int c = e / (D / 8), r = first_row + c, i = r / qg;
    *reinterpret_cast<uint4 *>(&sm.q[0][c][8 * (e % (D / 8))]) =
        r < rows ? __ldg(reinterpret_cast<const uint4 *>(a.q + ((size_t)(b * a.q_heads + kh * qg + (r - i * qg)) * a.count + i) * D) + e % (D / 8)) : make_uint4(0u, 0u, 0u, 0u);
  }
  RowWarp<CB, FB> &w = sm.w[warp];
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NST; ++s) mbar_init(&w.bar[s], 1);
    mbar_init_fence();
  }
  __syncthreads();
  uint32_t uses = 0;
  bool ok = true;
  for (int s = cluster == 1 ? 0 : rank; s < shares; s += cluster) {
    const int p0 = (int)((long long)pairs * s / shares), p1 = (int)((long long)pairs * (s + 1) / shares), per = (p1 - p0 + per_tile - 1) / per_tile;
    State st;
    st.m[0] = st.m[1] = -FBLA_INF;
    st.l = make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) st.o[u][cc] = make_float2(0.f, 0.f);
    const int lo = min(p1, p0 + place * per), hi = min(p1, lo + per);
    if (ok && lo < hi) ok = closed_run<CB, FB>(a, w, sm.q[tile], (size_t)bh * a.hs, lo, hi, own, uses, st, lane);
    float *const set = reinterpret_cast<float *>(w.pair[0]);
    if (ok) {
      write_state(set, st, lane);
      __syncwarp();
      exact_blocks(a, sm.q[tile], *reinterpret_cast<RowStage *>(w.pair[0] + SET * sizeof(float)), set, s * per_tile + place, per_tile * shares, exact, sink, own_lo, n1, pos, own, lane, token_row);
    } else if (lane == 0) {
      sm.failed = 1;
    }
    __syncthreads();
    for (int c = warp; c < held && !sm.failed; c += WARPS) {  // row c over its tile's warps, in their order, then behind the earlier shares
      const RowWarp<CB, FB> *tw = sm.w + c / COLS * per_tile;
      const int at = c % COLS * FBLA_K_PSTRIDE;
      float M = -FBLA_INF;
      for (int x = 0; x < per_tile; ++x) M = fmaxf(M, reinterpret_cast<const float *>(tw[x].pair[0])[at + D]);
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
      float l = 0.f;
      for (int x = 0; x < per_tile; ++x) {
        const float *row = reinterpret_cast<const float *>(tw[x].pair[0]) + at;
        const float e = row[D] == -FBLA_INF ? 0.f : ex2(row[D] - M);
        const float4 y = *reinterpret_cast<const float4 *>(row + 4 * lane);
        l = fmaf(e, row[D + 1], l);
        o.x = fmaf(e, y.x, o.x); o.y = fmaf(e, y.y, o.y); o.z = fmaf(e, y.z, o.z); o.w = fmaf(e, y.w, o.w);
      }
      float *dst = sm.share[c / COLS] + at;
      if (cluster == 1 && s > 0) {
        float4 before = *reinterpret_cast<const float4 *>(dst + 4 * lane);
        float m0 = dst[D], l0 = dst[D + 1];
        __syncwarp();
        add_share(m0, l0, before, M, l, o);
        M = m0; l = l0; o = before;
      }
      *reinterpret_cast<float4 *>(dst + 4 * lane) = o;
      if (lane == 0) { dst[D] = M; dst[D + 1] = l; }
    }
    __syncthreads();
  }
  if (FBLA_STREAM_LAUNCH && cluster > 1) cluster_meet();
  // row c over the shares, in their order; a cluster's CTAs take rows rank, rank + cluster, ...
  for (int c = rank + warp * cluster; c < held && first_row + c < rows; c += WARPS * cluster) {
    bool failed = sm.failed != 0;
    const float *row = sm.share[c / COLS] + c % COLS * FBLA_K_PSTRIDE;
    float M = -FBLA_INF, l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (FBLA_STREAM_LAUNCH && cluster > 1) {
      for (int s = 0; s < shares; ++s) {
        const uint32_t p = remote(row, s);
        const float2 ml = ld_remote2(p + 4 * D);
        failed |= ld_remote1(remote(&sm.failed, s)) != 0;
        add_share(M, l, o, ml.x, ml.y, ld_remote4(p + 16 * lane));
      }
    } else {
      o = *reinterpret_cast<const float4 *>(row + 4 * lane);
      l = row[D + 1];
    }
    const float inv = failed ? __int_as_float(0x7fc00000) : 1.f / l;
    const int r = first_row + c, i = r / qg, hq = kh * qg + (r - i * qg);
    uint16_t *orow = a.out + (size_t)(b * a.q_heads + hq) * a.out_hs + (size_t)i * a.out_ts;
    const uint32_t w0 = f32_to_bf16(o.x * inv) | (uint32_t)f32_to_bf16(o.y * inv) << 16, w1 = f32_to_bf16(o.z * inv) | (uint32_t)f32_to_bf16(o.w * inv) << 16;
    reinterpret_cast<uint2 *>(orow)[lane] = make_uint2(w0, w1);
  }
  if (FBLA_STREAM_LAUNCH && cluster > 1) cluster_meet();  // (nobody leaves while its shared memory is being read)
  __syncthreads();
  if (ok && lane == 0) {
#pragma unroll
    for (int s = 0; s < NST; ++s) mbar_inval(&w.bar[s]);
  }
}

}  // namespace fbla
