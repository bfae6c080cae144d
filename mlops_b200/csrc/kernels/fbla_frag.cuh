// Register fragments of the integer tensor-core products, built straight from packed records in shared memory.
//
// A record (one plane, 16 tokens) is staged in shared memory byte for byte as it lies in the cache. The products run
// with TOKENS on the M axis for scores (S^T = K_codes x qhat^T) and CHANNELS on the M axis for values
// (O^T = V_codes^T x P^T), so a record's "slot" -- four codes in the four bytes of a 32-bit word -- is exactly one
// A-fragment register once it is masked; nothing is ever unpacked to bytes in memory. A mask leaves the codes times a
// fixed power of two ("class"); products of one class go to their own s32 accumulator (scores) or their own row
// (values) and the factor is folded into the FP32 epilogue.
//
// Thread T of a warp: gid = T / 4 (fragment row / column), tig = T % 4 (k block). Scores: thread (gid, tig) supplies,
// for tokens gid and gid + 8, the slots whose word index is tig. Values: it supplies token quad tig of the channels of
// record lanes 8 u + gid, u = 0..3.
#pragma once
#include "fbla_device.cuh"

namespace fbla {

__device__ __forceinline__ void mma_u8u8_k16_from(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, uint32_t c) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(c));
}
// D = A B; sums that are taken as FP32 subnormals (tiny2)
__device__ __forceinline__ void mma_u8u8_k16_zero(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "n"(0));
}

// ---- qhat fragments -------------------------------------------------------------------------------------------------
// qst: 8 rows (fragment columns: queries, rows >= QG zero) of 128 s8 codes in channel order, row stride QST_ROW bytes
// (36 words: 4 * gid + word is then conflict-free over a warp).
constexpr int QST_ROW = 144;
__device__ __forceinline__ uint32_t qword(const uint8_t *qst, int gid, int w) { return lds32(qst + QST_ROW * gid + 4 * w); }

// B[8]: the qhat words matching the A slots of kfrag<BITS> below (pairs: k blocks tig and 4 + tig of one product)
template <int BITS> __device__ __forceinline__ void qhat_frag(const uint8_t *qst, int gid, int tig, uint32_t (&B)[8]) {
  if (BITS == 3) {
    const int e = ((tig & 1) ? 10 : 4) + (tig >> 1);
    B[0] = qword(qst, gid, tig);      B[1] = qword(qst, gid, 16 + tig);       // slots tig (bits 0-2)
    B[2] = qword(qst, gid, 6 + tig);  B[3] = qword(qst, gid, 22 + tig);       // slots 6 + tig (bits 3-5, class x8)
    B[4] = qword(qst, gid, 12 + tig); B[5] = qword(qst, gid, 28 + tig);       // slots 12 + tig (split over two words)
    B[6] = qword(qst, gid, e);        B[7] = qword(qst, gid, 16 + e);         // slots 4, 5 (even tig) / 10, 11 (odd tig)
  } else {  // 4 and 2 bits: word 4 m + tig, m = 0..7 (m < 4: channels 0..63, m >= 4: 64..127)
#pragma unroll
    for (int m = 0; m < 8; ++m) B[m] = qword(qst, gid, 4 * m + tig);
  }
}

// ---- scores: x[i] = sum_c qhat[c] * plane_value[token][c], i = (gid, 2 tig), (gid, 2 tig + 1), (gid + 8, 2 tig), (gid + 8, 2 tig + 1)
template <int BITS> __device__ __forceinline__ void qk_tile(const uint8_t *rec, int gid, int tig, const uint32_t (&B)[8], float (&x)[4]) {
  const uint8_t *p0 = rec + 16 * gid + 4 * tig, *p1 = p0 + 128;  // tokens gid, gid + 8
  if (BITS == 4) {
    const uint32_t a = lds32(p0), a8 = lds32(p1), b = lds32(p0 + 512), b8 = lds32(p1 + 512);          // half 0: W[tig], W[4 + tig]
    const uint32_t c = lds32(p0 + 256), c8 = lds32(p1 + 256), d = lds32(p0 + 768), d8 = lds32(p1 + 768);  // half 1
    constexpr uint32_t L = 0x0f0f0f0fu, H = 0xf0f0f0f0u;
    uint32_t lo[4], hi[4];
    mma_u8s8_k32_from(lo, a & L, a8 & L, b & L, b8 & L, B[0], B[1], MAGIC);
    mma_u8s8_k32_from(hi, a & H, a8 & H, b & H, b8 & H, B[2], B[3], MAGIC);
    mma_u8s8_k32(lo, c & L, c8 & L, d & L, d8 & L, B[4], B[5]);
    mma_u8s8_k32(hi, c & H, c8 & H, d & H, d8 & H, B[6], B[7]);
    const float2 x01 = __ffma2_rn(isum2(hi[0], hi[1]), splat(1.f / 16), isum2(lo[0], lo[1]));
    const float2 x23 = __ffma2_rn(isum2(hi[2], hi[3]), splat(1.f / 16), isum2(lo[2], lo[3]));
    x[0] = x01.x; x[1] = x01.y; x[2] = x23.x; x[3] = x23.y;
  } else if (BITS == 2) {
    const uint32_t a = lds32(p0), a8 = lds32(p1), c = lds32(p0 + 256), c8 = lds32(p1 + 256);
    uint32_t acc[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint32_t M = 0x03030303u << (2 * m);
      mma_u8s8_k32_from(acc[m], a & M, a8 & M, c & M, c8 & M, B[m], B[4 + m], MAGIC);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      x[i] = fmaf(isum(acc[3][i]), 1.f / 64, fmaf(isum(acc[2][i]), 1.f / 16, fmaf(isum(acc[1][i]), 1.f / 4, isum(acc[0][i]))));
  } else {
    const int sh = 4 + (tig & 1), se = 3 * (tig & 1);
    const uint8_t *q0 = rec + 1024 + 16 * gid + 4 * (tig >> 1), *q1 = q0 + 128;  // W[4 + tig / 2]: half 0, half 1 at + 8
    const uint32_t a = lds32(p0), a8 = lds32(p1), c = lds32(p0 + 256), c8 = lds32(p1 + 256);
    const uint32_t e = lds32(q0), e8 = lds32(q1), f = lds32(q0 + 8), f8 = lds32(q1 + 8);
    constexpr uint32_t L = 0x07070707u, M = 0x38383838u, T2 = 0x03030303u, T1 = 0x04040404u;
    uint32_t lo[4], mid[4];
    mma_u8s8_k32_from(lo, a & L, a8 & L, c & L, c8 & L, B[0], B[1], MAGIC);
    mma_u8s8_k32_from(mid, a & M, a8 & M, c & M, c8 & M, B[2], B[3], MAGIC);
    mma_u8s8_k32(lo, ((a >> 6) & T2) | ((e >> sh) & T1), ((a8 >> 6) & T2) | ((e8 >> sh) & T1),
                 ((c >> 6) & T2) | ((f >> sh) & T1), ((c8 >> 6) & T2) | ((f8 >> sh) & T1), B[4], B[5]);
    mma_u8s8_k32(lo, (e >> se) & L, (e8 >> se) & L, (f >> se) & L, (f8 >> se) & L, B[6], B[7]);
    const float2 x01 = __ffma2_rn(isum2(mid[0], mid[1]), splat(1.f / 8), isum2(lo[0], lo[1]));
    const float2 x23 = __ffma2_rn(isum2(mid[2], mid[3]), splat(1.f / 8), isum2(lo[2], lo[3]));
    x[0] = x01.x; x[1] = x01.y; x[2] = x23.x; x[3] = x23.y;
  }
}

// The same scores of two sub-blocks at once, for at most four queries: columns 0-3 are the queries under sub-block 0 (k blocks
// 0-3 of every product), columns 4-7 under sub-block 1 (k blocks 4-7). As many products as two qk_tile, but no column multiplies
// zeros for nothing: half the results to convert, reduce and exponentiate. X: qhat_frag's words where gid < 4, else 0; Y: the
// words (of query gid - 4) where gid >= 4, else 0.
template <int BITS> __device__ __forceinline__ void qk_pair(const uint8_t *r0, const uint8_t *r1, int gid, int tig, const uint32_t (&X)[8], const uint32_t (&Y)[8], float2 (&x)[2]) {
  const uint8_t *p = r0 + 16 * gid + 4 * tig, *r = r1 + 16 * gid + 4 * tig;
  if (BITS == 4) {
    uint32_t lo[4], hi[4];
    constexpr uint32_t L = 0x0f0f0f0fu, H = 0xf0f0f0f0u;
#pragma unroll
    for (int w = 0; w < 4; ++w) {  // words W[tig], W[4 + tig] of half 0, then of half 1
      const int o = 512 * (w & 1) + 256 * (w >> 1), m = (w & 1) + 4 * (w >> 1);
      const uint32_t a = lds32(p + o), a8 = lds32(p + o + 128), b = lds32(r + o), b8 = lds32(r + o + 128);
      if (w == 0) {
        mma_u8s8_k32_from(lo, a & L, a8 & L, b & L, b8 & L, X[m], Y[m], MAGIC);
        mma_u8s8_k32_from(hi, a & H, a8 & H, b & H, b8 & H, X[m + 2], Y[m + 2], MAGIC);
      } else {
        mma_u8s8_k32(lo, a & L, a8 & L, b & L, b8 & L, X[m], Y[m]);
        mma_u8s8_k32(hi, a & H, a8 & H, b & H, b8 & H, X[m + 2], Y[m + 2]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) x[i] = __ffma2_rn(isum2(hi[2 * i], hi[2 * i + 1]), splat(1.f / 16), isum2(lo[2 * i], lo[2 * i + 1]));
  } else {
    static_assert(BITS == 3 || BITS == 4, "coarse planes");
    const int sh = 4 + (tig & 1), se = 3 * (tig & 1), t = 1024 + 16 * gid + 4 * (tig >> 1);
    constexpr uint32_t L = 0x07070707u, M = 0x38383838u, T2 = 0x03030303u, T1 = 0x04040404u;
    uint32_t lo[4], mid[4], ex[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // halves
      const uint32_t a = lds32(p + 256 * h), a8 = lds32(p + 256 * h + 128), b = lds32(r + 256 * h), b8 = lds32(r + 256 * h + 128);
      const uint32_t e = lds32(r0 + t + 8 * h), e8 = lds32(r0 + t + 8 * h + 128), f = lds32(r1 + t + 8 * h), f8 = lds32(r1 + t + 8 * h + 128);
      if (h == 0) {
        mma_u8s8_k32_from(lo, a & L, a8 & L, b & L, b8 & L, X[0], Y[0], MAGIC);
        mma_u8s8_k32_from(mid, a & M, a8 & M, b & M, b8 & M, X[2], Y[2], MAGIC);
        mma_u8s8_k32_from(ex, (e >> se) & L, (e8 >> se) & L, (f >> se) & L, (f8 >> se) & L, X[6], Y[6], MAGIC);
      } else {
        mma_u8s8_k32(lo, a & L, a8 & L, b & L, b8 & L, X[1], Y[1]);
        mma_u8s8_k32(mid, a & M, a8 & M, b & M, b8 & M, X[3], Y[3]);
        mma_u8s8_k32(ex, (e >> se) & L, (e8 >> se) & L, (f >> se) & L, (f8 >> se) & L, X[7], Y[7]);
      }
      mma_u8s8_k32(lo, ((a >> 6) & T2) | ((e >> sh) & T1), ((a8 >> 6) & T2) | ((e8 >> sh) & T1), ((b >> 6) & T2) | ((f >> sh) & T1),
                   ((b8 >> 6) & T2) | ((f8 >> sh) & T1), X[4 + h], Y[4 + h]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
      x[i] = __fadd2_rn(__ffma2_rn(isum2(mid[2 * i], mid[2 * i + 1]), splat(1.f / 8), isum2(lo[2 * i], lo[2 * i + 1])), isum2(ex[2 * i], ex[2 * i + 1]));
  }
}

// ---- values ---------------------------------------------------------------------------------------------------------
// The four masked slot words (channels 4 l + 0..3 of record lane l, token quad tig) of a BITS-plane record's V half.
// Channel cc carries the factor 1 / v_unscale<BITS>(cc).
template <int BITS> __device__ __forceinline__ void v_slots(const uint8_t *rec, int l, int tig, uint32_t (&v)[4]) {
  if (BITS == 4) {
    const uint2 y = lds64(rec + 1024 + 512 * (tig >> 1) + 16 * l + 8 * (tig & 1));
    v[0] = y.x & 0x0f0f0f0fu; v[1] = y.y & 0x0f0f0f0fu; v[2] = y.x & 0xf0f0f0f0u; v[3] = y.y & 0xf0f0f0f0u;
  } else if (BITS == 2) {
    const uint32_t w = lds32(rec + 512 + 16 * l + 4 * tig);
    v[0] = w & 0x03030303u; v[1] = w & 0x0c0c0c0cu; v[2] = w & 0x30303030u; v[3] = w & 0xc0c0c0c0u;
  } else {
    const uint32_t w = lds32(rec + 512 + 16 * l + 4 * tig);
    const uint2 y = lds64(rec + 1280 + 8 * l);
    const uint32_t wt = (tig >> 1) ? y.y : y.x;  // W[4 + tig / 2]: the top bit of slot 12 + tig
    const uint32_t ws = (tig & 1) ? y.y : y.x;   // W[4 + tig % 2]: slot 4 + tig (tig < 2) or 10 + tig - 2
    v[0] = w & 0x07070707u;
    v[1] = w & 0x38383838u;
    v[2] = (ws >> (3 * (tig >> 1))) & 0x07070707u;
    v[3] = ((w >> 6) & 0x03030303u) | ((wt >> (4 + (tig & 1))) & 0x04040404u);
  }
}
template <int BITS> __host__ __device__ constexpr float v_unscale(int cc) {
  return BITS == 4 ? (cc < 2 ? 1.f : 1.f / 16) : BITS == 2 ? (cc == 0 ? 1.f : cc == 1 ? 1.f / 4 : cc == 2 ? 1.f / 16 : 1.f / 64)
                                                            : (cc == 1 ? 1.f / 8 : 1.f);
}

// ---- full codes -------------------------------------------------------------------------------------------------------
// Both planes of a slot joined to its code 2^FB h + f, four of them in the bytes of a word, times a class factor of their own
// (4 + 2 bits: 4 but for the slots whose fine bits are the lowest; 3 + 3 bits: 1). One product and one sum then do for both
// planes: half the matrix instructions, and a quarter of the FP32 work behind them, for one shift more per slot.
__device__ __forceinline__ uint32_t join_4p2(int m, uint32_t h, uint32_t f) {  // m: place of the fine bits; h: the coarse word, low nibble m < 2, else high
  return m == 0   ? ((h << 2) & 0x3c3c3c3cu) | (f & 0x03030303u)
         : m == 1 ? ((h << 4) & 0xf0f0f0f0u) | (f & 0x0c0c0c0cu)
                  : (h & 0xf0f0f0f0u) | ((f >> (2 * m - 2)) & 0x0c0c0c0cu);
}
// 3 + 3 bits: bits 0-2, bits 3-5, bits 3 hi .. of the words, and the slot that is split over two words (its top bit is bit sh of e)
__device__ __forceinline__ uint32_t join_low(uint32_t h, uint32_t f) { return ((h << 3) & 0x38383838u) | (f & 0x07070707u); }
__device__ __forceinline__ uint32_t join_mid(uint32_t h, uint32_t f) { return (h & 0x38383838u) | ((f >> 3) & 0x07070707u); }
__device__ __forceinline__ uint32_t join_at(uint32_t h, uint32_t f, int hi) { return ((h << (3 - 3 * hi)) & 0x38383838u) | ((f >> (3 * hi)) & 0x07070707u); }
__device__ __forceinline__ uint32_t join_split(uint32_t h, uint32_t eh, uint32_t f, uint32_t ef, int sh) {
  return ((h >> 3) & 0x18181818u) | ((eh >> (sh - 3)) & 0x20202020u) | ((f >> 6) & 0x03030303u) | ((ef >> sh) & 0x04040404u);
}

// scores under the full codes: thread (gid, tig): tokens gid (x[0]) and gid + 8 (x[1]) of columns 2 tig, 2 tig + 1; B: qhat_frag<CB>
template <int CB, int FB>
__device__ __forceinline__ void qk_full(const uint8_t *crec, const uint8_t *frec, int gid, int tig, const uint32_t (&B)[8], float2 (&x)[2]) {
  const uint8_t *p = crec + 16 * gid + 4 * tig, *r = frec + 16 * gid + 4 * tig;
  uint32_t one[4], two[4];
  if (CB == 4) {
    const uint32_t a = lds32(p), a8 = lds32(p + 128), b = lds32(p + 512), b8 = lds32(p + 640);
    const uint32_t c = lds32(p + 256), c8 = lds32(p + 384), d = lds32(p + 768), d8 = lds32(p + 896);
    const uint32_t f = lds32(r), f8 = lds32(r + 128), g = lds32(r + 256), g8 = lds32(r + 384);
    mma_u8s8_k32_from(two, join_4p2(1, b, f), join_4p2(1, b8, f8), join_4p2(2, a, f), join_4p2(2, a8, f8), B[1], B[2], MAGIC);
    mma_u8s8_k32_from(one, join_4p2(0, a, f), join_4p2(0, a8, f8), join_4p2(0, c, g), join_4p2(0, c8, g8), B[0], B[4], MAGIC);
    mma_u8s8_k32(two, join_4p2(3, b, f), join_4p2(3, b8, f8), join_4p2(1, d, g), join_4p2(1, d8, g8), B[3], B[5]);
    mma_u8s8_k32(two, join_4p2(2, c, g), join_4p2(2, c8, g8), join_4p2(3, d, g), join_4p2(3, d8, g8), B[6], B[7]);
  } else {
    const int sh = 4 + (tig & 1), hi = tig & 1, t = 1024 + 16 * gid + 4 * (tig >> 1);
    const uint32_t a = lds32(p), a8 = lds32(p + 128), c = lds32(p + 256), c8 = lds32(p + 384);
    const uint32_t e = lds32(crec + t), e8 = lds32(crec + t + 128), g = lds32(crec + t + 8), g8 = lds32(crec + t + 136);
    const uint32_t fa = lds32(r), fa8 = lds32(r + 128), fc = lds32(r + 256), fc8 = lds32(r + 384);
    const uint32_t fe = lds32(frec + t), fe8 = lds32(frec + t + 128), fg = lds32(frec + t + 8), fg8 = lds32(frec + t + 136);
    mma_u8s8_k32_from(one, join_low(a, fa), join_low(a8, fa8), join_low(c, fc), join_low(c8, fc8), B[0], B[1], MAGIC);
    mma_u8s8_k32_from(two, join_mid(a, fa), join_mid(a8, fa8), join_mid(c, fc), join_mid(c8, fc8), B[2], B[3], MAGIC);
    mma_u8s8_k32(one, join_split(a, e, fa, fe, sh), join_split(a8, e8, fa8, fe8, sh), join_split(c, g, fc, fg, sh), join_split(c8, g8, fc8, fg8, sh), B[4], B[5]);
    mma_u8s8_k32(two, join_at(e, fe, hi), join_at(e8, fe8, hi), join_at(g, fg, hi), join_at(g8, fg8, hi), B[6], B[7]);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) x[i] = __ffma2_rn(isum2(two[2 * i], two[2 * i + 1]), splat(CB == 4 ? .25f : 1.f), isum2(one[2 * i], one[2 * i + 1]));
}

// the values' joined words, channels 4 l + 0..3 of record lane l, token quad tig; channel cc carries 1 / v_full_unscale<CB>(cc)
template <int CB, int FB> __device__ __forceinline__ void v_full(const uint8_t *crec, const uint8_t *frec, int l, int tig, uint32_t (&v)[4]) {
  const uint32_t f = lds32(frec + 512 + 16 * l + 4 * tig);
  if (CB == 4) {
    const uint2 h = lds64(crec + 1024 + 512 * (tig >> 1) + 16 * l + 8 * (tig & 1));
    v[0] = join_4p2(0, h.x, f); v[1] = join_4p2(1, h.y, f); v[2] = join_4p2(2, h.x, f); v[3] = join_4p2(3, h.y, f);
  } else {
    const uint32_t h = lds32(crec + 512 + 16 * l + 4 * tig);
    const uint2 y = lds64(crec + 1280 + 8 * l), z = lds64(frec + 1280 + 8 * l);
    v[0] = join_low(h, f);
    v[1] = join_mid(h, f);
    v[2] = join_at((tig & 1) ? y.y : y.x, (tig & 1) ? z.y : z.x, tig >> 1);
    v[3] = join_split(h, (tig >> 1) ? y.y : y.x, f, (tig >> 1) ? z.y : z.x, 4 + (tig & 1));
  }
}
template <int CB> __host__ __device__ constexpr float v_full_unscale(int cc) { return CB == 4 && cc > 0 ? .25f : 1.f; }

}  // namespace fbla
