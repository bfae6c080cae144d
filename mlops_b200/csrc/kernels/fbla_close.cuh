// Quantize-on-write ("close") and the BF16 window update ("finish") of the FBLA cache, sm_100a.
//
// close: 512 threads per (group the chunk closes, KV head), 256 for K and 256 for V. Thread (r, c) of a tensor
// takes channels 8 c .. + 7 of tokens 8 r .. + 7 into registers with eight 128-bit loads (each token row comes from the
// chunk, the sink window or the old open window) and never reads them again: minima and maxima in packed BF16 over its
// eight tokens, over the warp and -- 512 bytes per warp -- over the tensor; a thread per channel then forms base (rounded
// down) and step (rounded up); the codes are formed from the registers and leave for shared memory as whole slot words
// (four codes: four channels of a token of K, four tokens of a channel of V); last, thread (tensor, sub-block, record
// lane) reads its lane's 16 slot words and packs both planes' words from them, stored 64 or 128 bits at a time.
// 64 KiB read, 25 KiB written per (head, group). A CTA per group, two per SM, idled HBM while both packed codes: 8 heads x 32 768 tokens 57.4
// us. A chunk without queries (write_chunk) is dealt over CTAs that stay, one tensor at a time (fewer threads at a barrier), the next unit
// on its way meanwhile, and the codes' bounds come with a saturating product: 43.9 us = 4.2 TB/s, now bound by the latency of its
// barriers and of shared memory (0.58 instructions issued per cycle and scheduler; stalls per issue: barrier 2.0, short scoreboard 1.9). Two
// threads per channel for base and step: 48.7 -> 50.0 (two tensors per CTA).
// A form with a thread per channel reading the 128 tokens of its channel from shared memory, and packing byte by byte from a
// byte-per-code tile, was bound by those single-byte accesses: 307 us.
// Replaces the reference's close_kernel / finish_kernel (attention/fbla/src/fbla_prefill.cuh:63-164); results are
// bit-identical by construction of the FP32 steps (no contraction: explicit round-to-nearest intrinsics).
#pragma once
#include "fbla_device.cuh"
#include "fbla_kernels.h"
#include <cuda_bf16.h>

namespace fbla {

// x rounded to BF16 toward -inf (up false) or +inf (up true)
__device__ __forceinline__ uint16_t bf16_directed(float x, bool up) {
  uint16_t u = f32_to_bf16(x);
  const float y = bf16_to_f32(u);
  if (up ? y < x : y > x) {
    if (y > 0.f) u = up ? u + 1 : u - 1;
    else if (y < 0.f) u = up ? u - 1 : u + 1;
    else u = up ? 0x0001 : 0x8001;
  }
  return u;
}

constexpr int CLOSE_THREADS = 512;

struct __align__(16) CloseSmem {  // of one tensor
  // The slot words of a sub-block, 16 per record lane (K: slot s; V: slot 4 cc + quad -- channel 4 l + cc, tokens 4 quad .. --, whatever the
  // plane's own order), at slot_at: a lane's four 16-byte pieces are read without conflicts, the words written two to a bank.
  uint32_t slot[SBG][32 * 16];
  uint32_t stat[8][2][D / 2];  // [warp][minimum, maximum][channel pair], BF16
  float base[D], inv[D];       // inv: 1 / step
  int odd;                     // a step outside the range that the short form of the codes takes
};
constexpr int TENSOR_THREADS = CLOSE_THREADS / 2;  // that close one tensor of a group
// in bytes: bit 3 ^ bit 4 of the lane on bit 0 of the lane, the lane's bits 1, 2 on the piece
__device__ __forceinline__ int slot_at(int l, int w) { return (64 * l + 4 * w) ^ (64 * (((l >> 3) ^ (l >> 4)) & 1)) ^ (16 * ((l >> 1) & 3)); }

__device__ __forceinline__ uint32_t bf16_min2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmin2(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
  return *reinterpret_cast<const uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t bf16_max2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
  return *reinterpret_cast<const uint32_t *>(&r);
}
// the low bytes of four words in one
__device__ __forceinline__ uint32_t low_bytes(float a, float b, float c, float d) {
  return __byte_perm(__byte_perm(__float_as_uint(a), __float_as_uint(b), 0x0040), __byte_perm(__float_as_uint(c), __float_as_uint(d), 0x0040), 0x5410);
}

// The plane's words of one (tensor, record lane) from its 16 slot words, and their stores. P(s): the plane's bits of slot s,
// one per byte.
template <int BITS, class P> __device__ __forceinline__ void store_plane(uint8_t *rec, int tensor, int l, P p) {
  uint32_t W[2 * BITS];
  if (BITS == 4) {
#pragma unroll
    for (int w = 0; w < 8; ++w) W[w] = p(w) | p(w + 8) << 4;
  } else if (BITS == 2) {
#pragma unroll
    for (int w = 0; w < 4; ++w) W[w] = p(w) | p(4 + w) << 2 | p(8 + w) << 4 | p(12 + w) << 6;
  } else {
#pragma unroll
    for (int w = 0; w < 4; ++w) W[w] = p(w) | p(w + 6) << 3 | (p(12 + w) & 0x03030303u) << 6;
#pragma unroll
    for (int w = 4; w < 6; ++w)
      W[w] = p(w) | p(w + 6) << 3 | ((p(12 + 2 * (w - 4)) >> 2) & 0x01010101u) << 6 | ((p(13 + 2 * (w - 4)) >> 2) & 0x01010101u) << 7;
  }
  *reinterpret_cast<uint4 *>(rec + word_offset(BITS, tensor, l, 0)) = make_uint4(W[0], W[1], W[2], W[3]);
  if (BITS == 4) *reinterpret_cast<uint4 *>(rec + word_offset(BITS, tensor, l, 4)) = make_uint4(W[4 % (2 * BITS)], W[5 % (2 * BITS)], W[6 % (2 * BITS)], W[7 % (2 * BITS)]);
  if (BITS == 3) *reinterpret_cast<uint2 *>(rec + word_offset(BITS, tensor, l, 4)) = make_uint2(W[4 % (2 * BITS)], W[5 % (2 * BITS)]);
}

// where a chunk stands in batch row b: its first position and its length
struct Chunk { int n0, count; };
__device__ __forceinline__ Chunk chunk_of(const fbla_k_prefill &a, int b) {
  return Chunk{(a.length ? FBLA_POS::ro(a.length + (a.lstride ? b : 0)) : 0) + a.n0, a.dcount ? FBLA_POS::ro(a.dcount) : a.count};
}

// the eight 16-byte pieces of thread t of 256 of tensor x (0: K, 1: V), group g of KV head bh: channels 8 c .. + 7 of tokens 8 r .. + 7, t = (r, c)
__device__ __forceinline__ void load_group(const fbla_k_prefill &a, int x, int t, int bh, int g, int n0, uint4 (&w)[8]) {
  const size_t eh = (size_t)bh * G * D, ih = (size_t)bh * a.count * D;
  const int r = t >> 4, c = t & 15;
  const uint16_t *in = x ? a.v : a.k;
  if (g * G >= n0) {  // all of it from the chunk
    const uint4 *const rows = reinterpret_cast<const uint4 *>(in + ih + (size_t)(g * G - n0 + 8 * r) * D) + c;
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = rows[i * (D / 8)];
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int pos = g * G + 8 * r + i;
    const uint16_t *row = pos >= n0 ? in + ih + (size_t)(pos - n0) * D
                        : pos < G   ? (x ? a.c.sink_v : a.c.sink_k) + eh + (size_t)pos * D
                                    : (x ? a.c.open_v : a.c.open_k) + eh + (size_t)(pos - (n0 - 1) / G * G) * D;
    w[i] = *(reinterpret_cast<const uint4 *>(row) + c);
  }
}

__device__ __forceinline__ float mul_sat(float a, float b) { float d; asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b)); return d; }  // to [0, 1]; not a number: 0

// The codes: rint of (value - base) / step held to [0, 63], not a number: 0. A step in the ordinary range: its reciprocal times 2^-6 is
// exact, the quotient at most 63 (1 + 2^-22), and the product's own saturation does for both bounds; the factor 64 goes with the rounding.
// ODD: some step of the tensor is outside it. Thread (r, c) of 256 of tensor x.
template <bool ODD> __device__ __forceinline__ void write_codes(CloseSmem &sm, int x, int r, int c, const uint4 (&w)[8]) {
  const int j = r >> 1;
  // -base and 1 / step of the thread's channel pair k, and 1.5 * 2^23 + code of two values
  auto numbers = [&](int k, float2 &nb, float2 &iv) {
    const float2 b2 = *reinterpret_cast<const float2 *>(&sm.base[8 * c + 2 * k]);
    nb = make_float2(-b2.x, -b2.y);
    iv = *reinterpret_cast<const float2 *>(&sm.inv[8 * c + 2 * k]);
    if (!ODD) iv = __fmul2_rn(iv, splat(1.f / 64));
  };
  auto code = [&](uint32_t e, float2 nb, float2 iv) {
    const float2 d = __fadd2_rn(make_float2(bf_lo(e), bf_hi(e)), nb);
    if constexpr (ODD) {
      const float2 v = __fmul2_rn(d, iv);
      return __fadd2_rn(make_float2(fminf(fmaxf(v.x, 0.f), 63.f), fminf(fmaxf(v.y, 0.f), 63.f)), splat(MAGICF));
    } else {
      return __ffma2_rn(make_float2(mul_sat(d.x, iv.x), mul_sat(d.y, iv.y)), splat(64.f), splat(MAGICF));
    }
  };
  uint8_t *const slots = reinterpret_cast<uint8_t *>(sm.slot[j]);
  if (x == 0) {  // a word: four channels of a token; record lane 8 (r % 2) + i + 16 (c / 8)
    const int at = slot_at(8 * (r & 1) + 16 * (c >> 3), 2 * (c & 7));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float2 nb[2], iv[2];
      numbers(2 * h, nb[0], iv[0]);
      numbers(2 * h + 1, nb[1], iv[1]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 p = code(h ? w[i].z : w[i].x, nb[0], iv[0]), q = code(h ? w[i].w : w[i].y, nb[1], iv[1]);
        *reinterpret_cast<uint32_t *>(slots + (at ^ (64 * (i & 1)) ^ (16 * (i >> 1))) + 128 * (i >> 1) + 4 * h) = low_bytes(p.x, p.y, q.x, q.y);
      }
    }
  } else {  // a word: four tokens of a channel; pair k, channels 8 c + 2 k, + 1: record lane 2 c + k / 2, cc = 2 (k % 2), + 1
    const int at = slot_at(2 * c, 2 * (r & 1));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 nb, iv;
      numbers(k, nb, iv);
      uint8_t *const s0 = slots + (at ^ (64 * (k >> 1)) ^ (32 * (k & 1))), *const s1 = slots + (at ^ (64 * (k >> 1)) ^ (32 * (k & 1)) ^ 16);
#pragma unroll
      for (int i4 = 0; i4 < 8; i4 += 4) {
        float2 f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 &y = w[i4 + i];
          f[i] = code(k == 0 ? y.x : k == 1 ? y.y : k == 2 ? y.z : y.w, nb, iv);
        }
        *reinterpret_cast<uint32_t *>(s0 + i4) = low_bytes(f[0].x, f[1].x, f[2].x, f[3].x);
        *reinterpret_cast<uint32_t *>(s1 + i4) = low_bytes(f[0].y, f[1].y, f[2].y, f[3].y);
      }
    }
  }
}

// Closes tensor x of group g of KV head bh from its rows in w: thread t of 256, which meet at sync(). `taken` runs once all have their rows.
template <int CB, int FB, class Sync, class Taken>
__device__ __forceinline__ void close_tensor(const fbla_k_prefill &a, CloseSmem &sm, int x, int t, int bh, int g, const uint4 (&w)[8], Sync sync, Taken taken) {
  const int r = t >> 4, c = t & 15, warp = t >> 5, lane = t & 31;
  uint32_t mn[4] = {0x7f807f80u, 0x7f807f80u, 0x7f807f80u, 0x7f807f80u}, mx[4] = {0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t e[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
    for (int k = 0; k < 4; ++k) { mn[k] = bf16_min2(mn[k], e[k]); mx[k] = bf16_max2(mx[k], e[k]); }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    mn[k] = bf16_min2(mn[k], __shfl_xor_sync(FULL, mn[k], 16));
    mx[k] = bf16_max2(mx[k], __shfl_xor_sync(FULL, mx[k], 16));
  }
  if (lane < 16) {
    *reinterpret_cast<uint4 *>(&sm.stat[warp][0][4 * c]) = make_uint4(mn[0], mn[1], mn[2], mn[3]);
    *reinterpret_cast<uint4 *>(&sm.stat[warp][1][4 * c]) = make_uint4(mx[0], mx[1], mx[2], mx[3]);
  }
  if (t == 0) sm.odd = 0;
  sync();
  taken();
  const size_t unit = (size_t)bh * a.hs + (size_t)g * a.gs;
  if (t < D) {
    const int ch = t;
    float lo = FBLA_INF, hi = -FBLA_INF;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      lo = fminf(lo, bf16_to_f32(reinterpret_cast<const uint16_t *>(sm.stat[v][0])[ch]));
      hi = fmaxf(hi, bf16_to_f32(reinterpret_cast<const uint16_t *>(sm.stat[v][1])[ch]));
    }
    const uint16_t ub = bf16_directed(lo, false);
    const float base = bf16_to_f32(ub);
    const uint16_t us = bf16_directed(__fmul_rn(__fsub_rn(hi, base), 1.f / 63.f), true);
    const float step = bf16_to_f32(us);
    sm.base[ch] = base;
    sm.inv[ch] = step > 0.f ? __frcp_rn(step) : 0.f;
    // (an infinite step has the reciprocal 0, with which every code is 0 in either form)
    if (step > 0.f && step < FBLA_INF && !(step >= 1.17549435e-38f /* 2^-126 */ && step <= 6.6461399e35f /* 2^119 */)) sm.odd = 1;
    uint16_t *meta = a.c.meta + unit * 512;
    meta[256 * x + 8 * (ch >> 2) + (ch & 3)] = ub;
    meta[256 * x + 8 * (ch >> 2) + 4 + (ch & 3)] = us;
  }
  sync();
  if (sm.odd) write_codes<true>(sm, x, r, c, w); else write_codes<false>(sm, x, r, c, w);
  sync();
  {
    const int j = warp, l = lane;  // record lane l of sub-block j
    uint32_t W[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4 *>(&W[4 * k]) = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(sm.slot[j]) + (slot_at(l, 0) ^ (16 * k)));
    uint8_t *const rc = a.c.coarse + (unit * SBG + j) * record_bytes(CB), *const rf = a.c.fine + (unit * SBG + j) * record_bytes(FB);
    constexpr uint32_t MC = 0x01010101u * ((1 << CB) - 1), MF = 0x01010101u * ((1 << FB) - 1);
    if (x == 0) {
      store_plane<CB>(rc, 0, l, [&](int s) { return (W[s] >> FB) & MC; });
      store_plane<FB>(rf, 0, l, [&](int s) { return W[s] & MF; });
    } else {
      store_plane<CB>(rc, 1, l, [&](int s) { return (W[4 * v_chan(CB, s) + v_quad(CB, s)] >> FB) & MC; });
      store_plane<FB>(rf, 1, l, [&](int s) { return W[4 * v_chan(FB, s) + v_quad(FB, s)] & MF; });
    }
  }
}

// all 512 threads: both tensors of a group
template <int CB, int FB>
__device__ __forceinline__ void close_group(const fbla_k_prefill &a, CloseSmem (&sm)[2], int bh, int g, int n0) {
  const int x = FBLA_POS::tid() / TENSOR_THREADS, t = FBLA_POS::tid() % TENSOR_THREADS;
  uint4 w[8];
  load_group(a, x, t, bh, g, n0, w);
  close_tensor<CB, FB>(a, sm[x], x, t, bh, g, w, [] { __syncthreads(); }, [] {});
}

// the group that CTA x of the pass may close, -1 if the chunk does not close it
__device__ __forceinline__ int closing_group(const Chunk &ch, int x) {
  const int g = (ch.n0 == 0 ? 0 : (ch.n0 - 1) / G) + x;
  return g < (ch.n0 + ch.count - 1) / G ? g : -1;
}

// finish: the sink window takes the chunk's positions < 128, the open window the tokens of the newest group; a fresh
// open group's unused rows are cleared. Tensor x of KV head bh by THREADS threads, PER 16-byte pieces per thread in flight.
template <int THREADS, int PER>
__device__ __forceinline__ void finish_tensor(const fbla_k_prefill &a, int x, int thread, int bh, const Chunk &ch) {
  const int n0 = ch.n0, n1 = n0 + ch.count, gl = (n1 - 1) / G;
  const bool fresh = n0 == 0 || (n0 - 1) / G != gl;
  const size_t eh = (size_t)bh * G * D, ih = (size_t)bh * a.count * D;
  const uint4 *in = reinterpret_cast<const uint4 *>((x ? a.v : a.k) + ih);
  uint4 *open = reinterpret_cast<uint4 *>((x ? a.c.open_v : a.c.open_k) + eh);
  uint4 *sink = reinterpret_cast<uint4 *>((x ? a.c.sink_v : a.c.sink_k) + eh);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int e0 = thread; e0 < G * 16; e0 += THREADS * PER) {
    uint4 o[PER], s[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = e0 + THREADS * i, t = e >> 4, pos = gl * G + t;
      o[i] = pos >= n0 && pos < n1 ? in[(size_t)(pos - n0) * 16 + (e & 15)] : zero;
      s[i] = t >= n0 && t < n1 ? in[(size_t)(t - n0) * 16 + (e & 15)] : zero;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = e0 + THREADS * i, t = e >> 4, pos = gl * G + t;
      if (pos >= n0 && (pos < n1 || fresh)) open[e] = o[i];
      if (t >= n0 && (t < n1 || a.clear_groups)) sink[e] = s[i];
    }
  }
}
// one CTA of 512 threads per KV head
__device__ __forceinline__ void finish_windows(const fbla_k_prefill &a, int bh, const Chunk &ch) {
#pragma unroll
  for (int x = 0; x < 2; ++x) finish_tensor<CLOSE_THREADS, 4>(a, x, FBLA_POS::tid(), bh, ch);
}
template <int CB, int FB>
__device__ __forceinline__ void close_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  const int bh = FBLA_POS::y();
  const Chunk ch = chunk_of(a, bh / a.kv_heads);
  const int g = closing_group(ch, FBLA_POS::x());
  if (g >= 0) close_group<CB, FB>(a, *reinterpret_cast<CloseSmem (*)[2]>(smem_raw), bh, g, ch.n0);
  if (a.early && ch.n0 == 0 && FBLA_POS::x() == 0) finish_windows(a, bh, ch);
}
__device__ __forceinline__ void finish_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  const Chunk ch = chunk_of(a, FBLA_POS::x() / a.kv_heads);
  if (!a.early || ch.n0 > 0) finish_windows(a, FBLA_POS::x(), ch);
}

// A chunk without queries in one launch. The (KV head, group, tensor) units, `blocks` possible groups per head, are dealt over the CTAs of a
// grid that the SMs hold at once, four of 256 threads each. A CTA's first unit comes straight into registers; while it works on one, the
// next one's 32 KiB are on their way into shared memory (a bulk copy), so that HBM does not idle while codes are packed. The CTA of a head's
// first possible group also updates the tensor's windows -- that group is the only one that may take rows from them, and has them in
// registers by then. a.clear_groups (a cache without initial contents, the chunk starting it): the units of the groups that stay open or
// unused are zeroed.
struct __align__(128) WriteSmem {
  uint8_t in[G * D * 2];  // the CTA's next unit
  CloseSmem s;
  uint64_t bar;
  int failed;  // a wait for a copy gave up: no more of them, the rows are loaded directly
};
template <int CB, int FB>
__device__ __forceinline__ void write_chunk(const fbla_k_prefill &a, uint8_t *smem_raw, int blocks) {
  WriteSmem &sm = *reinterpret_cast<WriteSmem *>(smem_raw);
  const int heads = a.batch * a.kv_heads, total = 2 * blocks * heads, tid = FBLA_POS::tid(), step = FBLA_POS::nx();
  int it = FBLA_POS::x();
  // asks for unit `at`, if there is one that lies in the chunk (the same answer in every thread; the first one asks)
  auto ask = [&](int at) {
    if (at >= total) return false;
    const int bh = (at >> 1) / blocks;
    const Chunk ch = chunk_of(a, bh / a.kv_heads);
    const int g = closing_group(ch, (at >> 1) - bh * blocks);
    if (g < 0 || g * G < ch.n0) return false;
    if (tid == 0 && !sm.failed) {
      fence_async_smem();  // (the buffer's rows have been read, behind a barrier)
      mbar_expect_tx(&sm.bar, sizeof sm.in);
      bulk_g2s(sm.in, ((at & 1) ? a.v : a.k) + (size_t)bh * a.count * D + (size_t)(g * G - ch.n0) * D, sizeof sm.in, &sm.bar);
    }
    return true;
  };
  if (tid == 0) {
    mbar_init(&sm.bar, 1);
    mbar_init_fence();
    sm.failed = 0;
  }
  __syncthreads();
  bool first = true, mine = false, next = ask(it + step);  // the unit in work comes through shared memory; the next one does
  uint32_t parity = 0;
#pragma unroll 1
  for (; it < total; it += step) {
    const int x = it & 1, bh = (it >> 1) / blocks, gi = (it >> 1) - bh * blocks;
    const Chunk ch = chunk_of(a, bh / a.kv_heads);
    const int g = closing_group(ch, gi);
    if (g >= 0) {
      uint4 w[8];
      bool direct = !mine || *reinterpret_cast<volatile int *>(&sm.failed);
      if (!direct && !mbar_wait_bounded(&sm.bar, parity)) {
        *reinterpret_cast<volatile int *>(&sm.failed) = 1;
        direct = true;
      }
      if (direct) {
        load_group(a, x, tid, bh, g, ch.n0, w);
      } else {
        const uint4 *const rows = reinterpret_cast<const uint4 *>(sm.in + 8 * (tid >> 4) * (D * 2)) + (tid & 15);
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = rows[i * (D / 8)];
      }
      if (mine) parity ^= 1;
      close_tensor<CB, FB>(a, sm.s, x, tid, bh, g, w, [] { __syncthreads(); }, [&] { if (!first) next = ask(it + step); });  // (the buffer is free then)
    } else if (!first) {
      next = ask(it + step);
    }
    mine = next;
    first = false;
    if (gi == 0) finish_tensor<TENSOR_THREADS, 4>(a, x, tid, bh, ch);
  }
  if (a.clear_groups) {  // (a chunk of host numbers at position 0)
    const int from = (a.count - 1) / G, units = a.clear_groups - from;
    for (int i = FBLA_POS::x(); i < units * heads; i += step) {
      const int bh = i / units;
      const size_t unit = (size_t)bh * a.hs + (size_t)(from + i - bh * units) * a.gs;
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      constexpr int NC = SBG * record_bytes(CB) / 16, NF = SBG * record_bytes(FB) / 16;
      for (int e = tid; e < NC; e += TENSOR_THREADS) reinterpret_cast<uint4 *>(a.c.coarse + unit * SBG * record_bytes(CB))[e] = zero;
      for (int e = tid; e < NF; e += TENSOR_THREADS) reinterpret_cast<uint4 *>(a.c.fine + unit * SBG * record_bytes(FB))[e] = zero;
      if (tid < 64) reinterpret_cast<uint4 *>(a.c.meta + unit * 512)[tid] = zero;
    }
  }
}

}  // namespace fbla
