// Causal prefill attention over the compressed cache on Blackwell tensor cores: tcgen05.mma with TMEM accumulators.
//
// Semantics: the reference's DP4A prefill (attention/fbla/src/fbla_prefill.cuh:389-705) -- the row at position p attends
// to 0..p: group 0 (sink) and its own group in BF16, closed groups 1..own-1 through their full 6-bit codes with the
// per-(row, group) int8 qhat, 16-token integer P blocks p = round(255 * 2^(s - max_block)) everywhere.
//
// One CTA = two tiles of 128 query rows of one KV head (row r = position r / qg, query r % qg) x a sequence of "passes",
// one per 128-token group the rows attend to. Per pass and tile, two tensor-core products with FP32 accumulators in
// tensor memory:
//   S[128 rows x 128 tokens]  = Qop[rows x 128 ch] . Kop[tokens x 128 ch]^T
//   O[128 rows x 128 ch]     += P'[rows x 128 tokens] . V'[ch x 128 tokens]^T
// Closed group: Qop = qhat (integers in [-127, 127]) and Kop = the 6-bit codes, both as FP16 -- products and the FP32
// sums (< 2^24) are exact, so S is the reference's integer dot product; BF16 group: Qop = q, Kop = k in BF16 (exact
// products, FP32 sums). P' = fp16(w_j p_t): the integer P block times its block weight 2^(m_j - m_row); V' =
// fp16(base + step * code) (closed) or fp16(v) (BF16), so O accumulates across ALL passes in tensor memory and is read
// once, at the end. The two FP16 roundings (relative 2^-11, zero mean) are the only deviations from the reference's
// arithmetic; they stay far inside the 2e-3 output tolerance.
//
// Warps 0-15 (softmax), 16-23 (quantiser), 24-27 (operands), 28 (issuer). Softmax: two threads per row (warps w and w + 8
// share a tensor-memory lane quadrant; warps 0-3, 8-11: tile 0). Quantiser: qhat of the next pass as soon as a tile's S
// product has read the current one, while that tile's rows are in their softmax: lane-per-channel-chunk over the tile's
// rows; the score biases of eight groups at a time are BF16 products on the side. Operand warps, shared by both tiles: they
// take the group's records from global memory straight into registers, one operand ahead, and unpack them into the Kop /
// V' tiles. Warp 28 allocates tensor memory; its lane 0 issues the products, which complete on mbarriers. Operand tiles are
// K-major with the 128-byte swizzle (8-row x 128-byte atoms, 16-byte chunk c of row r at c ^ (r % 8)).
// What bounds it: instruction issue of the CUDA cores -- per (row, group) the reference's semantics need 128 exp2 with
// integer rounding and the requantisation of the row's 128 query channels (about 17 000 warp instructions per pass at 0.6
// per cycle and scheduler); the tensor-core share of a pass is about as long as its exp2 share alone. Measured at batch 4 x
// 8192 (32 / 8 heads, 4+2): sixteen warps doing softmax and requantisation in turn 5.66 ms = 388 TFLOP/s; roles of their
// own 5.35; BF16 operands with all loads in flight 5.21; biases on tensor cores 4.75; a lane's eight rows requantised with one
// reduction, read twice, 4.60; four at a time, read once, 4.39 = 501 TFLOP/s. (64 registers per thread: 29 warps. Halving the softmax warps so that the tiles
// alternate, or one copy of the unpacking code for both records of an operand warp, measured slower.)
// Every wait is bounded: on a timeout the thread raises a flag, everybody drains, tensor memory is freed, the kernel
// returns and the host sees fbla_k_attend_tc_status() != 0.
#pragma once
#include "fbla_tc.cuh"
#include "fbla_decode.cuh"
#include "fbla_kernels.h"
#include <cuda_fp16.h>

namespace fbla {
namespace tc {

constexpr int ROWS = 128;                 // rows of a tile
constexpr int CTA_ROWS = 2 * ROWS;
constexpr int PRODUCERS = 4, PT = 32 * PRODUCERS;  // operand warps (two of a group's eight records each) and threads
constexpr int QUANT_WARP0 = 16, PRODUCER_WARP0 = 24, ISSUER_WARP = 24 + PRODUCERS;
constexpr int THREADS = (25 + PRODUCERS) * 32;
constexpr int SLAB = ROWS * 128;          // bytes of one K slab (128 rows x 128 bytes): 64 FP16 / BF16 of the K extent
constexpr int TILE = 2 * SLAB;            // a [128 x 128] 16-bit operand tile: 32 KiB
constexpr uint32_t WAIT_LIMIT = 1u << 18;

__device__ int g_status = 0;  // nonzero: a bounded wait gave up in some launch since the last read

struct __align__(1024) Smem {
  uint8_t q[2][TILE];   // Qop of BF16 passes: the rows' q, BF16
  uint8_t qp[2][TILE];  // Qop of closed passes: qhat as FP16 (at the very end: staging of the output rows)
  uint8_t k[TILE];      // Kop
  uint8_t v[TILE];      // V'
  float qscale[2][2][128];   // [pass parity][tile][row]: the pass's score scale (from the quantiser to the row's threads)
  float qbias[2][8][2][128];  // [eight passes, alternating][pass][tile][row]: the score bias sl q . base, formed for eight groups at once
  float ex2[2][128][2];  // exchange between the two threads of a row: pass maximum, final sum
  uint64_t bar_k, bar_v, bar_q[2], bar_s[2], bar_p[2], bar_o[2];
  float2 part[2 * ROWS];   // (m, l) of this CTA's share of every row
  uint32_t tmem_base;
  int abort;
};

static_assert(sizeof(Smem) + 1024 <= 232448, "operand tiles exceed the shared memory of an SM");

// ---- operand descriptors of this kernel's tiles ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t smem_desc(const void *tile_base, int slab, int kstep) { return smem_desc_at(tile_base, slab * SLAB + kstep * 32); }
__device__ __forceinline__ bool wait(Smem &sm, uint64_t *bar, uint32_t parity) {
  if (try_wait_hint(bar, parity)) return true;
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    if (*reinterpret_cast<volatile int *>(&sm.abort)) return false;
    if (try_wait_hint(bar, parity)) return true;
  }
  *reinterpret_cast<volatile int *>(&sm.abort) = 1;
  atomicExch(&g_status, 1);
  return false;
}

// ---- splitting a tile's passes over a thread-block cluster -----------------------------------------------------------------
// Few tiles over a long cache leave most SMs idle, and a CTA walks its groups one after the other. Then the passes of a tile
// are split into equal runs, one CTA of a cluster each, whose (m, l, O) are merged over distributed shared memory. As many
// as keep a run at twelve passes or more (the merge costs about three) while all clusters still fit the SMs at once -- 148,
// less what clusters of that size waste of them (a B200's number whatever the device: the runs decide the order of the sums, and
// with them the result's bits). 500 tokens at 30 000 (4 / 2 heads, 3+3): 999 -> 158 us.
// The number follows from the chunk's own size, wherever that lives: a launch for a count on the device serves the numbers
// (above, cluster], and of the launches for one chunk the count picks one; an executor's item does a tile's shares one after the
// other and merges them as the cluster does. So all of them give the same bits.
__host__ __device__ inline int tile_shares(long long tiles, int passes, int most) {
  int c = passes / 12;
  c = c > most ? most : c;
  while (c > 1 && tiles * c > 148 - 8 * (c - 1)) --c;
  return c < 1 ? 1 : c;
}

// V' tile row (= O column) of channel ch: 32 (ch % 4) + ch / 4, so that the 32 lanes of a record (4 channels each) write
// rows with all residues mod 8 -- conflict-free under the swizzle; the epilogue undoes it
__device__ __forceinline__ int vrow(int ch) { return 32 * (ch & 3) + (ch >> 2); }
// byte address of the 16-byte chunk holding K-extent element k0 (a multiple of 8) of tile row r
__device__ __forceinline__ uint8_t *chunk_at(uint8_t *tile, int r, int k0) {
  const int slab = k0 >> 6, c = (k0 & 63) >> 3;
  return tile + slab * SLAB + r * 128 + ((c ^ (r & 7)) << 4);
}

// ---- record unpacking (the slot maps of include/mlops_fbla.h) --------------------------------------------------------------
// one record lane's words of a tensor in a BITS plane, from global memory
template <int BITS> __device__ __forceinline__ void load_lane(const uint8_t *rec, int tensor, int lane, uint32_t (&W)[2 * BITS]) {
  const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(rec + word_offset(BITS, tensor, lane, 0)));
  W[0] = x.x; W[1] = x.y; W[2] = x.z; W[3] = x.w;
  if constexpr (BITS == 4) {
    const uint4 y = __ldcg(reinterpret_cast<const uint4 *>(rec + word_offset(BITS, tensor, lane, 4)));
    W[4] = y.x; W[5] = y.y; W[6] = y.z; W[7] = y.w;
  }
  if constexpr (BITS == 3) {
    const uint2 y = __ldcg(reinterpret_cast<const uint2 *>(rec + word_offset(BITS, tensor, lane, 4)));
    W[4] = y.x; W[5] = y.y;
  }
}
// four small unsigned integers (bytes of x, each < 1024) as two packed FP16 pairs: 0x6400 | b is 1024 + b
__device__ __forceinline__ uint2 bytes_to_half4(uint32_t x) {
  const uint32_t lo = __byte_perm(x, 0x64646464u, 0x7170), hi = __byte_perm(x, 0x64646464u, 0x7372);  // (b1 | 0x64 << 8) << 16 | b0 | 0x64 << 8
  const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0x6400));
  const __half2 a = __hsub2(*reinterpret_cast<const __half2 *>(&lo), bias), b = __hsub2(*reinterpret_cast<const __half2 *>(&hi), bias);
  return make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// FP16 pairs (code as FP16) * step + base, one rounding
__device__ __forceinline__ uint32_t hfma2_bits(uint32_t code2, __half2 step, __half2 base) {
  const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&code2), step, base);
  return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ float2 bf2(uint32_t w) { return make_float2(bf_lo(w), bf_hi(w)); }
// pairs of FP32 operations: the packed FP32x2 instructions of sm_100
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// ---- operands of the BF16 groups -------------------------------------------------------------------------------------------------
struct TokenRows {
  const uint16_t *chunk, *sink, *open;
  int n0;
  __device__ __forceinline__ const uint16_t *at(int tp) const {
    return tp >= n0 ? chunk + (size_t)(tp - n0) * D : tp < G ? sink + (size_t)tp * D : open + (size_t)(tp - (n0 - 1) / G * G) * D;
  }
};
// K rows of tokens t0 .. t0 + 127 as they are (zeros from n1 on), eight 16-byte pieces of the thread in flight
__device__ __forceinline__ void exact_k(uint8_t *tile, const TokenRows rows, int t0, int n1, int pt) {
#pragma unroll 1
  for (int e0 = pt; e0 < G * 16; e0 += 8 * PT) {
    uint4 w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + PT * i, tp = t0 + (e >> 4);
      w[i] = tp < n1 ? __ldcg(reinterpret_cast<const uint4 *>(rows.at(tp)) + (e & 15)) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4 *>(chunk_at(tile, (e0 + PT * i) >> 4, 8 * (e0 & 15))) = w[i];
  }
}
// V rows converted to FP16 and transposed (tokens along the K extent): a thread takes 8 channels of 8 tokens
__device__ __forceinline__ void exact_v(uint8_t *tile, const TokenRows rows, int t0, int n1, int pt) {
#pragma unroll 1
  for (int e = pt; e < G * 2; e += PT) {
    const int c = e & 15, t8 = 8 * (e >> 4);
    uint4 w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = t0 + t8 + i < n1 ? __ldcg(reinterpret_cast<const uint4 *>(rows.at(t0 + t8 + i)) + c) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      auto at = [&](int i) {
        const uint32_t v = x < 2 ? w[i].x : x < 4 ? w[i].y : x < 6 ? w[i].z : w[i].w;
        return (x & 1) ? bf_hi(v) : bf_lo(v);
      };
      *reinterpret_cast<uint4 *>(chunk_at(tile, vrow(8 * c + x), t8)) = make_uint4(pack_half2(at(0), at(1)), pack_half2(at(2), at(3)), pack_half2(at(4), at(5)), pack_half2(at(6), at(7)));
    }
  }
}

// How a CTA's two tiles are done: in one piece; as a share of a cluster; as one of the shares that an item does in turn. (One build
// per way: the loops of the first would carry the share's bounds in registers they lack, 9 % of the time at batch 4 x 8192.)
enum Way { WHOLE, CLUSTER, IN_TURN };
// IN_TURN: what the shares so far have left for the thread's row and columns
struct Kept { float m, l, o[64]; };
__device__ __forceinline__ int shares_of(const fbla_k_prefill &a, int rows, int n1) {
  return tile_shares((long long)((rows + CTA_ROWS - 1) / CTA_ROWS) * a.batch * a.kv_heads, (n1 - 1) / G + 1, FBLA_K_TILE_SHARES);
}

// whether a launch for a count on the device is the one that serves it (the same for every CTA of the grid)
__device__ __forceinline__ bool serves(const fbla_k_prefill &a) {
  const int count = FBLA_POS::ro(a.dcount), n1 = (a.length ? FBLA_POS::ro(a.length) : 0) + a.n0 + count, rows = count * (a.q_heads / a.kv_heads);
  const int shares = shares_of(a, rows, n1);
  return rows >= a.tc_min_rows && shares > a.above && shares <= a.cluster;
}

template <int CB, int FB, Way WAY>
__device__ __forceinline__ void attend_tiles(const fbla_k_prefill &a, uint8_t *smem_raw, int turn = 0, Kept *kept = nullptr) {
  constexpr bool SPLIT = WAY != WHOLE;
  smem_raw += (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;  // (an offset, not a rebuilt pointer: the address space stays known)
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  constexpr int RC = record_bytes(CB), RF = record_bytes(FB);
  const int tid = FBLA_POS::tid(), warp = tid >> 5, lane = tid & 31;
  const int bh = FBLA_POS::y(), b = bh / a.kv_heads, kh = bh - b * a.kv_heads, qg = a.q_heads / a.kv_heads;
  const int n0 = (a.length ? FBLA_POS::ro(a.length + (a.lstride ? b : 0)) : 0) + a.n0;
  const int count = a.dcount ? FBLA_POS::ro(a.dcount) : a.count, n1 = n0 + count;
  // the last tiles attend to the most groups: they are taken first, so that the grid's tail is made of short CTAs
  const int cluster = WAY == CLUSTER ? a.cluster : 1, rank = WAY == CLUSTER ? FBLA_POS::x() % cluster : turn;
  const int rows = count * qg, r0 = (FBLA_POS::nx() / cluster - 1 - FBLA_POS::x() / cluster) * CTA_ROWS;
  if (r0 >= rows || rows < a.tc_min_rows) return;  // (CTA-uniform; a short device count is the few-row pass's work)
  const int last_row = min(r0 + CTA_ROWS, rows) - 1;
  const int own_min = (n0 + r0 / qg) / G, own_max = (n0 + last_row / qg) / G;
  // passes: closed groups 1 .. own_max - 1, then the BF16 groups: 0 and the rows' own groups
  const int n_closed = max(own_max - 1, 0), own_lo = max(own_min, 1);
  const int n_pass = n_closed + 1 + max(own_max - own_lo + 1, 0);
  // this CTA's share of them: passes [p_lo, p_hi), of which [p_lo, c_hi) closed, [x_lo, p_hi) BF16
  const int shares = shares_of(a, rows, n1);
  // (of a cluster those leave that have no share: its barriers wait for threads that have not exited)
  if (WAY == CLUSTER ? shares <= a.above || shares > cluster || rank >= shares : WAY == WHOLE && shares > 1) return;
  const int p_lo = !SPLIT ? 0 : (int)((long long)n_pass * rank / shares);
  const int p_hi = !SPLIT ? n_pass : (int)((long long)n_pass * (rank + 1) / shares);
  const int c_hi = SPLIT ? min(n_closed, p_hi) : n_closed, x_lo = SPLIT ? max(n_closed, p_lo) : n_closed;
  auto pass_group = [&](int n, bool &closed) {
    closed = n < n_closed;
    return closed ? 1 + n : n == n_closed ? 0 : own_lo + (n - n_closed - 1);
  };

  if (tid == 0) {
    mbar_init(&sm.bar_k, PT); mbar_init(&sm.bar_v, PT);
    for (int x = 0; x < 2; ++x) { mbar_init(&sm.bar_q[x], 256); mbar_init(&sm.bar_s[x], 1); mbar_init(&sm.bar_p[x], 256); mbar_init(&sm.bar_o[x], 1); }
    sm.abort = 0;
    mbar_init_fence();
  }
  if (warp == ISSUER_WARP) {  // all 512 columns of tensor memory: S of tile x at 128 x, O at 256 + 128 x
    // (the allocation permit is kept: an executor may run further tensor-core items on this CTA, and a CTA that has given
    // its permit up may not allocate again)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)), "r"(512) : "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  const size_t head = (size_t)bh * a.hs, eh = (size_t)bh * G * D, ih = (size_t)bh * a.count * D;
  // the BF16 rows of K and of V: the chunk, the sink window, the window of the group that was open before the chunk
  const TokenRows rows_k{a.k + ih, a.c.sink_k + eh, a.c.open_k + eh, n0}, rows_v{a.v + ih, a.c.sink_v + eh, a.c.open_v + eh, n0};

  if (warp == ISSUER_WARP) {
    // ================= issuer: the products =================
    // Per pass S(n, 0), O(n - 1, 1), S(n, 1), O(n, 0): the order in which the half passes make their operands ready. Products
    // execute in the order they are issued, so S(n + 1, x) overwrites P'(n, x) only after O(n, x) has read it.
    if (lane == 0) {
      auto scores = [&](int n, int x) -> bool {
        if (!wait(sm, &sm.bar_q[x], (n - p_lo) & 1)) return false;
        tc_fence_after();
        const bool closed = n < n_closed;
        const uint8_t *qop = closed ? sm.qp[x] : sm.q[x];
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          mma_f16(tmem + 128 * x, smem_desc(qop, kk >> 2, kk & 3), smem_desc(sm.k, kk >> 2, kk & 3), closed ? IDESC_F16 : IDESC_BF16, kk > 0);
        mma_commit(&sm.bar_s[x]);
        return true;
      };
      auto values = [&](int n, int x) -> bool {
        if (!wait(sm, &sm.bar_p[x], (n - p_lo) & 1)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // P' of token block kk: eight columns inside the tile's S columns (see the softmax threads)
          mma_f16_ts(tmem + 256 + 128 * x, tmem + 128 * x + 64 * (kk >> 2) + 8 * (kk & 3), smem_desc(sm.v, kk >> 2, kk & 3), IDESC_F16, n > p_lo || kk > 0);
        mma_commit(&sm.bar_o[x]);
        return true;
      };
      bool ok = true;
      for (int n = p_lo; n < p_hi && ok; ++n)
        ok = wait(sm, &sm.bar_k, (n - p_lo) & 1) && scores(n, 0) && (n == p_lo || values(n - 1, 1)) && scores(n, 1) && wait(sm, &sm.bar_v, (n - p_lo) & 1) && values(n, 0);
      if (ok && (!SPLIT || p_lo < p_hi)) values(p_hi - 1, 1);
    }
  } else if (warp >= PRODUCER_WARP0) {
    // ================= operand producers =================
    const int pt = tid - 32 * PRODUCER_WARP0;  // 0 .. PT - 1
    const int l = pt & 31, j0 = pt >> 5;
    constexpr int NJ = SBG / PRODUCERS;        // records per warp
    uint32_t Wc[NJ][2 * CB], Wf[NJ][2 * FB];   // K's words of the next closed group, then V's of the current one
    auto load = [&](int g, int tensor) {
      const size_t unit = head + (size_t)g * a.gs;
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        load_lane<CB>(a.c.coarse + (unit * SBG + j0 + PRODUCERS * i) * RC, tensor, l, Wc[i]);
        load_lane<FB>(a.c.fine + (unit * SBG + j0 + PRODUCERS * i) * RF, tensor, l, Wf[i]);
      }
    };
    if (p_lo < c_hi) load(1 + p_lo, 0);
    bool ok = true;
    // Kop is free once both tiles' S of the previous pass are complete, V' once both tiles' O products are
    auto free_k = [&](int n) { return n == p_lo || (wait(sm, &sm.bar_s[0], (n - 1 - p_lo) & 1) && wait(sm, &sm.bar_s[1], (n - 1 - p_lo) & 1)); };
    auto free_v = [&](int n) { return n == p_lo || (wait(sm, &sm.bar_o[0], (n - 1 - p_lo) & 1) && wait(sm, &sm.bar_o[1], (n - 1 - p_lo) & 1)); };
    auto done = [&](uint64_t *bar) { fence_async_smem(); mbar_arrive(bar); };
#pragma unroll 1
    for (int n = p_lo; n < c_hi; ++n) {
      const int g = 1 + n;
      if (!(ok = free_k(n))) break;
      const uint4 vm = __ldcg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(a.c.meta) + (head + (size_t)g * a.gs) * 1024 + 512) + l);
      // (record j, lane l): token 16 j + l % 16, channels 64 (l / 16) + 4 s + byte: one 128-byte row of slab l / 16
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const int tok = 16 * (j0 + PRODUCERS * i) + (l & 15);
#pragma unroll
        for (int s2 = 0; s2 < 8; ++s2) {
          const uint2 x = bytes_to_half4((slot_value<CB>(Wc[i], 2 * s2) << FB) | slot_value<FB>(Wf[i], 2 * s2));
          const uint2 y = bytes_to_half4((slot_value<CB>(Wc[i], 2 * s2 + 1) << FB) | slot_value<FB>(Wf[i], 2 * s2 + 1));
          *reinterpret_cast<uint4 *>(chunk_at(sm.k, tok, 64 * (l >> 4) + 8 * s2)) = make_uint4(x.x, x.y, y.x, y.y);
        }
      }
      load(g, 1);
      done(&sm.bar_k);
      if (!(ok = free_v(n))) break;
      // (record j, lane l): channels 4 l + cc, tokens 16 j + 4 quad + byte, value base + step * code in FP16 arithmetic
      const __half2 vb[4] = {__float2half2_rn(bf_lo(vm.x)), __float2half2_rn(bf_hi(vm.x)), __float2half2_rn(bf_lo(vm.y)), __float2half2_rn(bf_hi(vm.y))};
      const __half2 vs[4] = {__float2half2_rn(bf_lo(vm.z)), __float2half2_rn(bf_hi(vm.z)), __float2half2_rn(bf_lo(vm.w)), __float2half2_rn(bf_hi(vm.w))};
#pragma unroll
      for (int i = 0; i < NJ; ++i) {
        const int j = j0 + PRODUCERS * i;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t h[8];
#pragma unroll
          for (int quad = 0; quad < 4; ++quad) {
            const uint2 c4 = bytes_to_half4((slot_value<CB>(Wc[i], v_slot_of(CB, cc, quad)) << FB) | slot_value<FB>(Wf[i], v_slot_of(FB, cc, quad)));
            h[2 * quad] = hfma2_bits(c4.x, vs[cc], vb[cc]);
            h[2 * quad + 1] = hfma2_bits(c4.y, vs[cc], vb[cc]);
          }
          *reinterpret_cast<uint4 *>(chunk_at(sm.v, 32 * cc + l, 16 * j)) = make_uint4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<uint4 *>(chunk_at(sm.v, 32 * cc + l, 16 * j + 8)) = make_uint4(h[4], h[5], h[6], h[7]);
        }
      }
      if (n + 1 < c_hi) load(g + 1, 0);
      done(&sm.bar_v);
    }
#pragma unroll 1
    for (int n = x_lo; n < p_hi && ok; ++n) {
      bool closed;
      const int t0 = pass_group(n, closed) * G;
      if (!(ok = free_k(n))) break;
      exact_k(sm.k, rows_k, t0, n1, pt);
      done(&sm.bar_k);
      if (!(ok = free_v(n))) break;
      exact_v(sm.v, rows_v, t0, n1, pt);
      done(&sm.bar_v);
    }
  } else if (warp >= QUANT_WARP0) {
    // ================= quantiser: Qop of every pass, tile 0 then tile 1 =================
    // A warp takes 16 rows of a tile, two rows at a time: lane (c = lane % 16, lane / 16) holds channels 8 c .. + 7 of one
    // row, with the group's steps of those channels in registers; max |z| is reduced over the 16 lanes of a row. The bias
    // dot products q . base of eight groups at a time are one BF16 tensor-core product per 16 rows (exact products, FP32 sums).
    const int qw = warp - QUANT_WARP0, qc = lane & 15, qrow0 = 16 * qw + (lane >> 4);  // (row % 8) of row qrow0 + 2 it = (2 it) | (qrow0 & 1)
    const uint32_t qoff = (qc >> 3) * SLAB + qrow0 * 128, qcx = (uint32_t)((qc & 7) ^ (qrow0 & 1)) << 4;
    // the rows' q into the BF16 Q tiles (rows past the end: zeros), by the same map
#pragma unroll
    for (int X = 0; X < 2; ++X)
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int Rq = r0 + ROWS * X + qrow0 + 2 * it;
        if (SPLIT && p_lo >= p_hi) continue;  // (a share without passes: the memory takes its row sums)
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (Rq < rows) {
          const int iq = Rq / qg;
          w = __ldg(reinterpret_cast<const uint4 *>(a.q + ((size_t)(b * a.q_heads + kh * qg + (Rq - iq * qg)) * a.count + iq) * D) + qc);
        }
        *reinterpret_cast<uint4 *>(sm.q[X] + qoff + 2 * it * 128 + (qcx ^ (((2 * it) & 7) << 4))) = w;
      }
    int tile_own[2];  // closed group g concerns the tile iff g < tile_own
#pragma unroll
    for (int X = 0; X < 2; ++X) {
      const int tile_last = min(r0 + ROWS * X + ROWS, rows) - 1;  // the tile's last row, if it has any
      tile_own[X] = tile_last >= r0 + ROWS * X ? (n0 + tile_last / qg) / G : -1;
    }
    const float2 mg = splat(MAGICF), ng = splat(-MAGICF);
    const float sl127 = __fmul_rn(a.sl, 1.f / 127.f);
    const uint8_t *const meta = reinterpret_cast<const uint8_t *>(a.c.meta) + head * 1024 + 32 * qc + 8;
    uint2 ma = make_uint2(0u, 0u), mb = ma;  // K's steps of channels 8 qc .. + 7 (the metadata: per four channels, four BF16 bases then four BF16 steps)
    auto load_meta = [&](int g) {
      ma = __ldcg(reinterpret_cast<const uint2 *>(meta + (size_t)g * a.gs * 1024));
      mb = __ldcg(reinterpret_cast<const uint2 *>(meta + (size_t)g * a.gs * 1024 + 16));
    };
    if (p_lo < c_hi) load_meta(1 + p_lo);
    __syncwarp();  // (the warp's own rows of the q tiles are in place)
#pragma unroll 1
    for (int n = p_lo; n < c_hi; ++n) {
      const int g = 1 + n, k = n - p_lo;
      if (!(k & 7)) {  // the biases of groups g .. g + 7 (those past the last: repeated, unused)
        const uint8_t *base = reinterpret_cast<const uint8_t *>(a.c.meta) + (head + (size_t)min(g + (lane >> 2), n_closed) * a.gs) * 1024 + 16 * ((lane & 3) >> 1) + 4 * (lane & 1);
#pragma unroll 1
        for (int X = 0; X < 2; ++X) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
          const int row = 16 * qw + (lane & 15);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {  // channels 16 kk ..
            uint32_t q4[4];
            ldmatrix_x4(q4, sm.q[X] + (kk >> 2) * SLAB + row * 128 + (((2 * (kk & 3) + (lane >> 4)) ^ (row & 7)) << 4));
            mma_bf16_k16(d, q4[0], q4[1], q4[2], q4[3], __ldcg(reinterpret_cast<const uint32_t *>(base + 64 * kk)), __ldcg(reinterpret_cast<const uint32_t *>(base + 64 * kk + 32)));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) sm.qbias[(k >> 3) & 1][2 * (lane & 3) + (i & 1)][X][16 * qw + (lane >> 2) + 8 * (i >> 1)] = __fmul_rn(d[i], a.sl);
        }
      }
      const float4 s0 = make_float4(bf_lo(ma.x), bf_hi(ma.x), bf_lo(ma.y), bf_hi(ma.y));
      const float4 s1 = make_float4(bf_lo(mb.x), bf_hi(mb.x), bf_lo(mb.y), bf_hi(mb.y));
      if (n + 1 < c_hi) load_meta(g + 1);
#pragma unroll 1
      for (int X = 0; X < 2; ++X) {
        // the tile's qhat buffer is free once the S product of the pass before is complete
        if (k > 0) wait(sm, &sm.bar_s[X], (k - 1) & 1);
        if (g < tile_own[X]) {
          // z = q * step_K, r = fl(127 / max|z|), rint(z r) written as FP16. The lane's shares of max |z|; a butterfly over a row's 16
          // lanes that hands half of the rows on in each of its first steps leaves one row in each group of lanes, which form its r once.
          auto place = [&](int it, int h) { return qoff + 1024 * h + 2 * it * 128 + (qcx ^ (((2 * it) & 7) << 4)); };  // of row it + 4 h of the lane's eight
          auto z_of = [&](int it, int h, float2 (&z)[4]) {
            const uint4 qv = *reinterpret_cast<const uint4 *>(sm.q[X] + place(it, h));
            z[0] = mul2(bf2(qv.x), make_float2(s0.x, s0.y)); z[1] = mul2(bf2(qv.y), make_float2(s0.z, s0.w));
            z[2] = mul2(bf2(qv.z), make_float2(s1.x, s1.y)); z[3] = mul2(bf2(qv.w), make_float2(s1.z, s1.w));
          };
          auto max_of = [](const float2 (&z)[4]) { return max3_abs(max3_abs(z[0].x, z[0].y, z[1].x), max3_abs(z[1].y, z[2].x, z[2].y), fmaxf(fabsf(z[3].x), fabsf(z[3].y))); };
          auto write = [&](int it, int h, const float2 (&z)[4], float r) {  // rint(z r) as the exact float (t - 1.5 * 2^23), then FP16 (an integer of magnitude <= 127: exact)
            const float2 rr2 = splat(r);
            const float2 t0 = add2(fma2(z[0], rr2, mg), ng), t1 = add2(fma2(z[1], rr2, mg), ng);
            const float2 t2 = add2(fma2(z[2], rr2, mg), ng), t3 = add2(fma2(z[3], rr2, mg), ng);
            *reinterpret_cast<uint4 *>(sm.qp[X] + place(it, h)) = make_uint4(pack_half2(t0.x, t0.y), pack_half2(t1.x, t1.y), pack_half2(t2.x, t2.y), pack_half2(t3.x, t3.y));
          };
          auto hand_on = [&](float (&amax)[4], int bit) {  // four rows to one: lane bits `bit` and bit / 2 decide which
#pragma unroll
            for (int w = 2; w; w >>= 1) {
              const int o = bit * w / 2;
              const bool up = lane & o;
#pragma unroll
              for (int i = 0; i < w; ++i) {
                const float keep = up ? amax[i + w] : amax[i], send = up ? amax[i] : amax[i + w];
                amax[i] = fmaxf(keep, __shfl_xor_sync(FULL, send, o));
              }
            }
          };
          // Whole tiles: four rows at a time, their z in registers (2 x 4 000 tokens 714 -> 677 us). A tile's shares, whose passes are no
          // faster so: all eight rows in one butterfly, q read twice (400 tokens behind 60 000, 32 / 8 heads 1 107 -> 1 021 us, 100 behind
          // 20 000 163 -> 155; 4+2: 1 088 -> 1 032, 159 -> 153).
          if constexpr (SPLIT) {  // (row 4 b3 + 2 b2 + b1 in the lanes with those bits)
            float amax[4] = {0.f, 0.f, 0.f, 0.f}, before[4];
#pragma unroll 1
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int it = 0; it < 4; ++it) {
                float2 z[4];
                z_of(it, h, z);
                before[it] = amax[it];
                amax[it] = max_of(z);
              }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const bool up = lane & 8;
              const float keep = up ? amax[i] : before[i], send = up ? before[i] : amax[i];
              amax[i] = fmaxf(keep, __shfl_xor_sync(FULL, send, 8));
            }
            hand_on(amax, 4);
            const float am = fmaxf(amax[0], __shfl_xor_sync(FULL, amax[0], 1));
            const float rq = quotient_127(am);
            if (!(lane & 1)) sm.qscale[k & 1][X][qrow0 + (lane & 14)] = __fmul_rn(am, sl127);  // (row qrow0 + 2 it)
#pragma unroll 1
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int it = 0; it < 4; ++it) {
                float2 z[4];
                z_of(it, h, z);
                write(it, h, z, __shfl_sync(FULL, rq, (lane & 16) | (8 * h + 2 * it)));
              }
          } else {  // (row 2 b3 + b2 in the lanes with those bits)
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              float2 z[4][4];
              float amax[4];
#pragma unroll
              for (int it = 0; it < 4; ++it) {
                z_of(it, h, z[it]);
                amax[it] = max_of(z[it]);
              }
              hand_on(amax, 8);
              float am = fmaxf(amax[0], __shfl_xor_sync(FULL, amax[0], 2));
              am = fmaxf(am, __shfl_xor_sync(FULL, am, 1));
              const float rq = quotient_127(am);
              if (!(lane & 3)) sm.qscale[k & 1][X][qrow0 + 8 * h + ((lane & 12) >> 1)] = __fmul_rn(am, sl127);  // (row qrow0 + 8 h + 2 it)
#pragma unroll
              for (int it = 0; it < 4; ++it) write(it, h, z[it], __shfl_sync(FULL, rq, (lane & 16) | (4 * it)));
            }
          }
        }
        fence_async_smem();
        mbar_arrive(&sm.bar_q[X]);
      }
    }
    if (p_lo >= c_hi) fence_async_smem();  // (the q tiles, otherwise covered by the first pass's)
#pragma unroll 1
    for (int n = x_lo; n < p_hi; ++n)  // BF16 passes take the q tiles as they are
      for (int X = 0; X < 2; ++X) {
        if (n > p_lo) wait(sm, &sm.bar_s[X], (n - 1 - p_lo) & 1);
        mbar_arrive(&sm.bar_q[X]);
      }
  } else {
    // ================= softmax, P', output: tile 0 then tile 1 of every pass =================
    // Two threads per row: warps w and w + 4 share a tensor-memory lane quadrant; thread hf owns tokens 64 hf .. + 63 of S and
    // P' and O columns 64 hf .. + 63; the pair meets on a named barrier to exchange the pass maximum. A thread never leaves
    // the pass loop early: after an abort every wait returns at once, so both threads of a pair still reach every named barrier.
    const int hf = warp >> 3, X = (warp >> 2) & 1, r = 32 * (warp & 3) + lane, pair_bar = 1 + (warp & 7);
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory"); };
    const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t tmem_s = tmem + 128 * X + 64 * hf + lane_base, tmem_o = tmem + 256 + 128 * X + 64 * hf + lane_base;
    float m_run = -FBLA_INF, l_run = 0.f;  // l_run: this thread's tokens only
    const int R = r0 + ROWS * X + r, pos = R < rows ? n0 + R / qg : -1, own = pos / G;  // pos -1: the tile has no such row
    bool ok = true;
    for (int n = p_lo; n < p_hi; ++n) {
      bool closed;
      const int g = pass_group(n, closed), k = n - p_lo;
      {
        const bool include = pos >= 0 && (closed ? g < own : (g == 0 || g == own));
        const bool any = __any_sync(FULL, include);
        // S(n) is complete, and with it every product issued before: O of the tile's pass n - 1 is stable
        ok &= __all_sync(FULL, wait(sm, &sm.bar_s[X], k & 1));
        tc_fence_after();
        // softmax of the row over the pass's 128 tokens, by 16-token blocks; P' = fp16(2^(m_block - m_row) p)
        const int lim = (include ? (closed ? G : pos - g * G) : -1) - 64 * hf;  // this thread's tokens 0 .. lim are attended
        const float mul1 = closed ? sm.qscale[k & 1][X][r] : a.sl, add1 = closed ? sm.qbias[(k >> 3) & 1][k & 7][X][r] : 0.f;  // score = mul x + add, monotonic in x (mul >= 0)
        // sweep 1: the block maxima, from the raw sums (each block's columns are asked for while the one before is worked on)
        float mbk[4];
        uint32_t xa[16], xb[16];
        if (any) {
          tmem_ld16(tmem_s, xa);
#pragma unroll
          for (int blk = 0; blk < 4; ++blk) {
            uint32_t (&x)[16] = blk & 1 ? xb : xa;
            tmem_ld_wait(x);
            if (blk < 3) tmem_ld16(tmem_s + 16 * (blk + 1), blk & 1 ? xa : xb);
            const int t0 = 16 * blk;
            float xm = -FBLA_INF;
            if (lim >= t0 + 15) {
              float y[4];
#pragma unroll
              for (int t = 0; t < 4; ++t) y[t] = max3(__uint_as_float(x[4 * t]), __uint_as_float(x[4 * t + 1]), __uint_as_float(x[4 * t + 2]));
              xm = max3(max3(y[0], y[1], __uint_as_float(x[3])), max3(y[2], y[3], __uint_as_float(x[7])), fmaxf(__uint_as_float(x[11]), __uint_as_float(x[15])));
            } else {
#pragma unroll
              for (int t = 0; t < 16; ++t) if (t0 + t <= lim) xm = fmaxf(xm, __uint_as_float(x[t]));
            }
            mbk[blk] = xm == -FBLA_INF ? -FBLA_INF : fmaf(mul1, xm, add1);  // -inf: a block without attended tokens
          }
          sm.ex2[X][r][hf] = fmaxf(fmaxf(mbk[0], mbk[1]), fmaxf(mbk[2], mbk[3]));
        }
        pair_sync();
        if (!any) {  // (warp-uniform, and the same in both warps of the pair) nothing to attend: P' = 0
          const uint32_t zero[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_st8(tmem_s + 8 * c, zero);
        } else {
          const float2 e = *reinterpret_cast<const float2 *>(&sm.ex2[X][r][0]);
          const float mp = fmaxf(e.x, e.y);
          // the row's running maximum moves only when a block exceeds it by more than 2^8 (rare): its sums and its O row in
          // tensor memory are rescaled. Tensor-memory accesses are warp-wide, so the whole warp takes part (rows that do
          // not move scale by 1); both threads of a row decide alike and each rescales its own 64 columns.
          const bool need = mp > m_run + 8.f;
          if (__any_sync(FULL, need)) {
            const float al = need ? ex2(m_run - mp) : 1.f;  // 0 on the row's first attended block
            if (k > 0) {
#pragma unroll 1
              for (int oc = 0; oc < 2; ++oc) {
                uint32_t o[32];
                tmem_ld32(tmem_o + 32 * oc, o);
#pragma unroll
                for (int z = 0; z < 32; ++z) o[z] = __float_as_uint(__uint_as_float(o[z]) * al);
                tmem_st32(tmem_o + 32 * oc, o);
              }
            }
            if (need) { l_run *= al; m_run = mp; }
          }
          // sweep 2: the integer P blocks times their weights. With a weight of 22 bits 1.5 * 2^23 w is a float, so that
          // (1.5 * 2^23 + p) w - 1.5 * 2^23 w is p w in one rounding (the integer p needs no instruction of its own).
          const float2 mul = splat(mul1), c255 = splat(255.f), mg = splat(MAGICF);
          float2 lacc = make_float2(0.f, 0.f);
          tmem_ld16(tmem_s, xa);
#pragma unroll
          for (int blk = 0; blk < 4; ++blk) {
            uint32_t (&x)[16] = blk & 1 ? xb : xa;
            tmem_ld_wait(x);
            if (blk < 3) tmem_ld16(tmem_s + 16 * (blk + 1), blk & 1 ? xa : xb);
            const int t0 = 16 * blk;
            const float mb = mbk[blk];
            // score - block maximum in one step: mul x + (add - m_block)
            const float w1 = mb == -FBLA_INF ? 0.f : __uint_as_float(__float_as_uint(ex2(mb - m_run)) & ~3u);
            const float2 addm = splat(mb == -FBLA_INF ? add1 : add1 - mb), w2 = splat(w1), mw = splat(-MAGICF * w1);
            float2 sc[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) sc[t] = fma2(make_float2(__uint_as_float(x[2 * t]), __uint_as_float(x[2 * t + 1])), mul, addm);
            if (lim < t0 + 15) {  // the causal edge (or a row that does not attend to this group)
#pragma unroll
              for (int t = 0; t < 8; ++t) {
                if (t0 + 2 * t > lim) sc[t].x = -FBLA_INF;
                if (t0 + 2 * t + 1 > lim) sc[t].y = -FBLA_INF;
              }
            }
            uint32_t h[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              const float2 pw = fma2(fma2(make_float2(ex2(sc[t].x), ex2(sc[t].y)), c255, mg), w2, mw);
              lacc = add2(lacc, pw);
              h[t] = pack_half2(pw.x, pw.y);
            }
            tmem_st8(tmem_s + 8 * blk, h);  // (over S columns this thread has already taken into registers)
          }
          l_run += lacc.x + lacc.y;
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&sm.bar_p[X]);
      }
    }
    {
      if (!SPLIT || p_lo < p_hi) ok &= __all_sync(FULL, wait(sm, &sm.bar_o[X], (p_hi - 1 - p_lo) & 1));
      tc_fence_after();
      pair_sync();  // (the partner has read the last pass's exchange)
      sm.ex2[X][r][hf] = l_run;
      pair_sync();
      const float l_row = sm.ex2[X][r][0] + sm.ex2[X][r][1];
      if (WAY == CLUSTER && shares > 1) {
        // This share's sums for the cluster: O as it lies in tensor memory, 16-byte piece c of row r at c ^ (r % 32), over the
        // query tiles (every product has read them: the O products were issued last); (m, l) beside them.
        float *const row = reinterpret_cast<float *>(sm.q[0]) + (size_t)(ROWS * X + r) * D;
        if (hf == 0) sm.part[ROWS * X + r] = make_float2(m_run, l_row);
#pragma unroll 1
        for (int cu = 0; cu < 2; ++cu) {
          uint32_t o[32];
          if (p_lo < p_hi) tmem_ld32(tmem_o + 32 * cu, o);
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4 *>(row + 4 * ((16 * hf + 8 * cu + c) ^ (r & 31))) =
                p_lo < p_hi ? make_uint4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (!ok) *reinterpret_cast<volatile int *>(&sm.abort) = 1;
      } else {
      float l_all = l_row;
      if constexpr (WAY == IN_TURN) {  // this share's sums onto those of the shares before, as the cluster's CTAs add them
        const float mn = fmaxf(kept->m, m_run), sa = kept->m == -FBLA_INF ? 0.f : ex2(kept->m - mn), sb = m_run == -FBLA_INF ? 0.f : ex2(m_run - mn);
        kept->m = mn;
        l_all = kept->l = fmaf(sa, kept->l, sb * l_row);
#pragma unroll 1
        for (int cu = 0; cu < 2; ++cu) {
          uint32_t o[32];
          if (p_lo < p_hi) tmem_ld32(tmem_o + 32 * cu, o);
#pragma unroll
          for (int z = 0; z < 32; ++z) kept->o[32 * cu + z] = fmaf(sa, kept->o[32 * cu + z], sb * (p_lo < p_hi ? __uint_as_float(o[z]) : 0.f));
        }
        if (!ok) kept->l = l_all = __int_as_float(0x7fc00000);
      }
      if (WAY != IN_TURN || rank == shares - 1) {
      // O column 32 cc + l is channel 4 l + cc: through the row's (now free) qhat row as BF16 in channel order, then out.
      // This thread: O columns 64 hf .. + 63 (cc = 2 hf, 2 hf + 1); then it copies chunks 8 hf .. + 7 of the row.
      const float inv = 1.f / l_all;
      uint16_t *stage = reinterpret_cast<uint16_t *>(sm.qp[X] + r * 256);  // 256 bytes per row, private to the pair
#pragma unroll 1
      for (int cu = 0; cu < 2; ++cu) {
        const int cc = 2 * hf + cu;
        uint32_t o[32];
        if constexpr (WAY == IN_TURN) {
#pragma unroll
          for (int l = 0; l < 32; ++l) o[l] = __float_as_uint(kept->o[32 * cu + l]);
        } else tmem_ld32(tmem + 256 + 128 * X + 64 * hf + lane_base + 32 * cu, o);
#pragma unroll
        for (int l = 0; l < 32; ++l)  // channel 4 l + cc: 16-byte chunk l / 2 of the row, stored at chunk (l / 2) ^ (r % 16)
          stage[8 * ((l >> 1) ^ (r & 15)) + 4 * (l & 1) + cc] = f32_to_bf16(__uint_as_float(o[l]) * inv);
      }
      pair_sync();
      if (R < rows) {  // (after a wait that gave up: NaN, so that the failure shows in the caller's data)
        const int i = R / qg, hq = kh * qg + (R - i * qg);
        uint16_t *orow = a.out + (size_t)(b * a.q_heads + hq) * a.out_hs + (size_t)i * a.out_ts;
        const uint4 nan4 = make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u);
#pragma unroll
        for (int c = 8 * hf; c < 8 * hf + 8; ++c) reinterpret_cast<uint4 *>(orow)[c] = ok ? reinterpret_cast<const uint4 *>(stage)[c ^ (r & 15)] : nan4;
      }
      }
    }
    }
  }
  if (WAY == CLUSTER && shares > 1) {
    // the cluster's CTAs merge the tiles' rows: this one rows rank, rank + shares, ... in 16-byte pieces of the output
    cluster_meet();
    {
      for (int e = tid; e < (2 * ROWS / shares + 1) * (D / 8); e += THREADS) {
        const int rr = rank + shares * (e / (D / 8)), c8 = e % (D / 8), R = r0 + rr;  // channels 8 c8 ..: columns 32 cc + 2 c8, + 1
        if (rr >= 2 * ROWS || R >= rows) continue;
        float M = -FBLA_INF, L = 0.f;
        float2 o[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // [cc]: channels 8 c8 + cc, + 4
        bool failed = false;
        for (int s = 0; s < shares; ++s) {
          const float2 ml = ld_remote2(remote(&sm.part[rr], s));
          const float mn = fmaxf(M, ml.x), sa = M == -FBLA_INF ? 0.f : ex2(M - mn), sb = ml.x == -FBLA_INF ? 0.f : ex2(ml.x - mn);
          M = mn;
          L = fmaf(sa, L, sb * ml.y);
          failed |= ld_remote1(remote(&sm.abort, s)) != 0;
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) {
            const int col = 32 * cc + 2 * c8;
            const float2 y = ld_remote2(remote(reinterpret_cast<float *>(sm.q[0]) + (size_t)rr * D + 4 * ((col >> 2) ^ (rr & 31)) + (col & 3), s));
            o[cc] = make_float2(fmaf(sa, o[cc].x, sb * y.x), fmaf(sa, o[cc].y, sb * y.y));
          }
        }
        const float inv = failed ? __int_as_float(0x7fc00000) : 1.f / L;
        const int i = R / qg, hq = kh * qg + (R - i * qg);
        auto pack = [&](float x, float y) { return f32_to_bf16(x * inv) | (uint32_t)f32_to_bf16(y * inv) << 16; };
        reinterpret_cast<uint4 *>(a.out + (size_t)(b * a.q_heads + hq) * a.out_hs + (size_t)i * a.out_ts)[c8] =
            make_uint4(pack(o[0].x, o[1].x), pack(o[2].x, o[3].x), pack(o[0].y, o[1].y), pack(o[2].y, o[3].y));
      }
    }
    cluster_meet();  // (nobody leaves while its shared memory is being read)
  }
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUER_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (tid == 0) {  // no live barrier object is left behind: an executor may run another item on this CTA next
    mbar_inval(&sm.bar_k); mbar_inval(&sm.bar_v);
    for (int x = 0; x < 2; ++x) { mbar_inval(&sm.bar_q[x]); mbar_inval(&sm.bar_s[x]); mbar_inval(&sm.bar_p[x]); mbar_inval(&sm.bar_o[x]); }
  }
}

// An executor's item: two tiles, in one piece or share after share.
template <int CB, int FB>
__device__ __forceinline__ void attend_tc_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  const int n0 = (a.length ? FBLA_POS::ro(a.length + (a.lstride ? FBLA_POS::y() / a.kv_heads : 0)) : 0) + a.n0;
  const int count = a.dcount ? FBLA_POS::ro(a.dcount) : a.count, shares = shares_of(a, count * (a.q_heads / a.kv_heads), n0 + count);
  if (shares == 1) {
    attend_tiles<CB, FB, WHOLE>(a, smem_raw);
    return;
  }
  Kept kept;
  kept.m = -FBLA_INF;
  kept.l = 0.f;
#pragma unroll 1
  for (int z = 0; z < 64; ++z) kept.o[z] = 0.f;
#pragma unroll 1
  for (int s = 0; s < shares; ++s) attend_tiles<CB, FB, IN_TURN>(a, smem_raw, s, &kept);
}

}  // namespace tc
}  // namespace fbla
