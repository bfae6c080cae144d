// Quantize-on-write ("close") and the BF16 window update ("finish") of the FBLA cache, sm_100a.
//
// close: one CTA of 512 threads per (group the chunk closes, KV head), 256 for K and 256 for V. Thread (r, c) of a tensor
// takes channels 8 c .. + 7 of tokens 8 r .. + 7 into registers with eight 128-bit loads (each token row comes from the
// chunk, the sink window or the old open window) and never reads them again: minima and maxima in packed BF16 over its
// eight tokens, over the warp and -- 512 bytes per warp -- over the tensor; a thread per channel then forms base (rounded
// down) and step (rounded up); the codes are formed from the registers and leave for shared memory as whole slot words
// (four codes: four channels of a token of K, four tokens of a channel of V); last, thread (tensor, sub-block, record
// lane) reads its lane's 16 slot words and packs both planes' words from them, stored 64 or 128 bits at a time.
// Bound by HBM: 64 KiB read, 25 KiB written per (head, group); two CTAs per SM overlap one's loads with the other's
// packing. A form with a thread per channel reading the 128 tokens of its channel from shared memory, and packing byte by
// byte from a byte-per-code tile, was bound by those single-byte accesses: 8 heads x 32 768 tokens 307 us (0.6 TB/s).
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
constexpr int SLOT_ROW = 20;  // words per record lane: 16 slots and padding that keeps 128-bit reads of neighbouring lanes conflict-free

struct CloseSmem {
  // K: slot s of the record lane; V: slot 4 cc + quad (channel 4 l + cc, tokens 4 quad ..), whatever the plane's own order
  uint32_t slot[2][SBG][32][SLOT_ROW];
  uint32_t stat[2][8][2][D / 2];  // [tensor][warp][minimum, maximum][channel pair], BF16
  float base[2][D], inv[2][D];
};

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

// the group g of KV head bh (closed by the chunk)
template <int CB, int FB>
__device__ __forceinline__ void close_group(const fbla_k_prefill &a, CloseSmem &sm, int bh, int g, int n0) {
  const size_t eh = (size_t)bh * G * D, ih = (size_t)bh * a.count * D;
  const int tid = FBLA_POS::tid(), x = tid >> 8, r = (tid >> 4) & 15, c = tid & 15, warp = (tid >> 5) & 7, lane = tid & 31;
  const uint16_t *in = x ? a.v : a.k;
  uint4 w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int pos = g * G + 8 * r + i;
    const uint16_t *row = pos >= n0 ? in + ih + (size_t)(pos - n0) * D
                        : pos < G   ? (x ? a.c.sink_v : a.c.sink_k) + eh + (size_t)pos * D
                                    : (x ? a.c.open_v : a.c.open_k) + eh + (size_t)(pos - (n0 - 1) / G * G) * D;
    w[i] = *(reinterpret_cast<const uint4 *>(row) + c);
  }
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
    *reinterpret_cast<uint4 *>(&sm.stat[x][warp][0][4 * c]) = make_uint4(mn[0], mn[1], mn[2], mn[3]);
    *reinterpret_cast<uint4 *>(&sm.stat[x][warp][1][4 * c]) = make_uint4(mx[0], mx[1], mx[2], mx[3]);
  }
  __syncthreads();
  const size_t unit = (size_t)bh * a.hs + (size_t)g * a.gs;
  if ((tid & 255) < D) {
    const int ch = tid & 127;
    float lo = FBLA_INF, hi = -FBLA_INF;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      lo = fminf(lo, bf16_to_f32(reinterpret_cast<const uint16_t *>(sm.stat[x][v][0])[ch]));
      hi = fmaxf(hi, bf16_to_f32(reinterpret_cast<const uint16_t *>(sm.stat[x][v][1])[ch]));
    }
    const uint16_t ub = bf16_directed(lo, false);
    const float base = bf16_to_f32(ub);
    const uint16_t us = bf16_directed(__fmul_rn(__fsub_rn(hi, base), 1.f / 63.f), true);
    const float step = bf16_to_f32(us);
    sm.base[x][ch] = base;
    sm.inv[x][ch] = step > 0.f ? __frcp_rn(step) : 0.f;
    uint16_t *meta = a.c.meta + unit * 512;
    meta[256 * x + 8 * (ch >> 2) + (ch & 3)] = ub;
    meta[256 * x + 8 * (ch >> 2) + 4 + (ch & 3)] = us;
  }
  __syncthreads();
  {
    float2 nb[4], iv[4];  // -base and 1 / step of the thread's channel pairs
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 b2 = *reinterpret_cast<const float2 *>(&sm.base[x][8 * c + 2 * k]);
      nb[k] = make_float2(-b2.x, -b2.y);
      iv[k] = *reinterpret_cast<const float2 *>(&sm.inv[x][8 * c + 2 * k]);
    }
    const float2 mg = splat(MAGICF);
#pragma unroll
    for (int i4 = 0; i4 < 8; i4 += 4) {  // four tokens at a time
      float2 f[4][4];                     // [token][channel pair]: 1.5 * 2^23 + code
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t e[4] = {w[i4 + i].x, w[i4 + i].y, w[i4 + i].z, w[i4 + i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 v = __fmul2_rn(__fadd2_rn(make_float2(bf_lo(e[k]), bf_hi(e[k])), nb[k]), iv[k]);
          f[i][k] = __fadd2_rn(make_float2(fminf(fmaxf(v.x, 0.f), 63.f), fminf(fmaxf(v.y, 0.f), 63.f)), mg);  // (not a number: 0)
        }
      }
      const int j = r >> 1;
      if (x == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int l = (8 * (r & 1) + i4 + i) + 16 * (c >> 3);
          *reinterpret_cast<uint2 *>(&sm.slot[0][j][l][2 * (c & 7)]) =
              make_uint2(low_bytes(f[i][0].x, f[i][0].y, f[i][1].x, f[i][1].y), low_bytes(f[i][2].x, f[i][2].y, f[i][3].x, f[i][3].y));
        }
      } else {
        const int quad = 2 * (r & 1) + (i4 >> 2);
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // channels 8 c + 2 k, + 1: record lane 2 c + k / 2, cc = 2 (k % 2), + 1
          uint32_t *s = &sm.slot[1][j][2 * c + (k >> 1)][8 * (k & 1) + quad];
          s[0] = low_bytes(f[0][k].x, f[1][k].x, f[2][k].x, f[3][k].x);
          s[4] = low_bytes(f[0][k].y, f[1][k].y, f[2][k].y, f[3][k].y);
        }
      }
    }
  }
  __syncthreads();
  {
    const int j = warp, l = lane;  // record lane l of sub-block j
    uint32_t W[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4 *>(&W[4 * k]) = *reinterpret_cast<const uint4 *>(&sm.slot[x][j][l][4 * k]);
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

// the group that CTA x of the pass may close, -1 if the chunk does not close it
__device__ __forceinline__ int closing_group(const Chunk &ch, int x) {
  const int g = (ch.n0 == 0 ? 0 : (ch.n0 - 1) / G) + x;
  return g < (ch.n0 + ch.count - 1) / G ? g : -1;
}

// finish: the sink window takes the chunk's positions < 128, the open window the tokens of the newest group; a fresh
// open group's unused rows are cleared. One CTA of 512 threads per KV head, four 16-byte pieces per thread in flight.
__device__ __forceinline__ void finish_windows(const fbla_k_prefill &a, int bh, const Chunk &ch) {
  const int n0 = ch.n0, n1 = n0 + ch.count, gl = (n1 - 1) / G;
  const bool fresh = n0 == 0 || (n0 - 1) / G != gl;
  const size_t eh = (size_t)bh * G * D, ih = (size_t)bh * a.count * D;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const uint4 *in = reinterpret_cast<const uint4 *>((x ? a.v : a.k) + ih);
    uint4 *open = reinterpret_cast<uint4 *>((x ? a.c.open_v : a.c.open_k) + eh);
    uint4 *sink = reinterpret_cast<uint4 *>((x ? a.c.sink_v : a.c.sink_k) + eh);
    constexpr int PER = G * 16 / CLOSE_THREADS;
    uint4 o[PER], s[PER];
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = FBLA_POS::tid() + CLOSE_THREADS * i, t = e >> 4, pos = gl * G + t;
      o[i] = pos >= n0 && pos < n1 ? in[(size_t)(pos - n0) * 16 + (e & 15)] : zero;
      s[i] = t >= n0 && t < n1 ? in[(size_t)(t - n0) * 16 + (e & 15)] : zero;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = FBLA_POS::tid() + CLOSE_THREADS * i, t = e >> 4, pos = gl * G + t;
      if (pos >= n0 && (pos < n1 || fresh)) open[e] = o[i];
      if (t >= n0 && (t < n1 || a.clear_groups)) sink[e] = s[i];
    }
  }
}
template <int CB, int FB>
__device__ __forceinline__ void close_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  const int bh = FBLA_POS::y();
  const Chunk ch = chunk_of(a, bh / a.kv_heads);
  const int g = closing_group(ch, FBLA_POS::x());
  if (g >= 0) close_group<CB, FB>(a, *reinterpret_cast<CloseSmem *>(smem_raw), bh, g, ch.n0);
  if (a.early && ch.n0 == 0 && FBLA_POS::x() == 0) finish_windows(a, bh, ch);
}
__device__ __forceinline__ void finish_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  const Chunk ch = chunk_of(a, FBLA_POS::x() / a.kv_heads);
  if (!a.early || ch.n0 > 0) finish_windows(a, FBLA_POS::x(), ch);
}

// A chunk without queries in one launch: CTA (x, bh) closes its group; CTA (0, bh) also updates the windows -- it is the
// only one whose group takes rows from them, and has them in registers by then. a.clear_groups (a cache without initial
// contents, the chunk starting it): the units of the groups that stay open or unused are zeroed, dealt over the head's CTAs.
template <int CB, int FB>
__device__ __forceinline__ void write_item(const fbla_k_prefill &a, uint8_t *smem_raw) {
  const int bh = FBLA_POS::y(), x = FBLA_POS::x();
  const Chunk ch = chunk_of(a, bh / a.kv_heads);
  const int g = closing_group(ch, x);
  if (g >= 0) close_group<CB, FB>(a, *reinterpret_cast<CloseSmem *>(smem_raw), bh, g, ch.n0);
  if (x == 0) finish_windows(a, bh, ch);
  for (int e = (ch.n0 + ch.count - 1) / G + x; e < a.clear_groups; e += FBLA_POS::nx()) {
    const size_t unit = (size_t)bh * a.hs + (size_t)e * a.gs;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    constexpr int NC = SBG * record_bytes(CB) / 16, NF = SBG * record_bytes(FB) / 16;
    for (int i = FBLA_POS::tid(); i < NC; i += CLOSE_THREADS) reinterpret_cast<uint4 *>(a.c.coarse + unit * SBG * record_bytes(CB))[i] = zero;
    for (int i = FBLA_POS::tid(); i < NF; i += CLOSE_THREADS) reinterpret_cast<uint4 *>(a.c.fine + unit * SBG * record_bytes(FB))[i] = zero;
    if (FBLA_POS::tid() < 64) reinterpret_cast<uint4 *>(a.c.meta + unit * 512)[FBLA_POS::tid()] = zero;
  }
}

}  // namespace fbla
