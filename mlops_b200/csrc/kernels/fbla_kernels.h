// The thin C ABI between the C++ host layer (validation, geometry, dispatch) and the CUDA kernels: plain structs of
// pointers and sizes, one launcher per pass. The host layer fills these; nothing here validates.
#pragma once
#include "fbla_device.cuh"  /* fixed-width integers; under run-time compilation no host header is available */
#ifndef __CUDACC_RTC__
#include <stddef.h>
#define FBLA_HOST_API(decl) decl
#else
#define FBLA_HOST_API(decl)  /* launchers exist only in the library */
#endif

#ifdef __cplusplus
extern "C" {
#endif

typedef struct {
  uint8_t *coarse, *fine;
  uint16_t *meta, *sink_k, *sink_v, *open_k, *open_v;
} fbla_k_cache;

// ---- decode -------------------------------------------------------------------------------------------------------
// Virtual heads: a KV head with r = q_heads / kv_heads queries is served as vg = r / qg virtual heads of qg in {1, 2, 4}
// queries each (virtual head vh = kv_head_linear * vg + j owns queries j * qg .. j * qg + qg - 1 of its KV head).
// Scratch arrays (all written before they are read; no initial contents needed):
//   lse    [VH][nblocks][qg]  float  log2 mass of every closed sub-block under the coarse scores (two sweeps: then the weights, fbla_dense.cuh)
//   part   [2 TW + 2 VH][qg][132] float  (o[128], m, l) partials: slot w + vh for streaming warp (or, folded, CTA) w,
//          coarse_ctas * coarse_warps + VH + x + vh for window warp x; TW = coarse_ctas * coarse_warps
//   dpart  [RW + VH][qg][132] float  (do[128], dl) corrections of refine warp (or, folded, CTA) w at slot w + vh; before that pass its first
//          words are the coarse CTAs' reports (nonzero: a bounded wait gave up)
//   row_r  [VH][qg]           float  log2 of the row's total coarse mass
//   counts [VH][nslices]      int    selected sub-blocks per slice of 1024 sub-blocks
//   items  [VH][nslices][1024] int   (sub-block << 4) | query mask, in sub-block order
//   item_off [VH * nslices + 1] int  exclusive prefix of counts (written by the refine pass for the merge)
//   status [4]                int    0 ok; nonzero: a bounded wait gave up (which pass, which CTA)
typedef struct {
  fbla_k_cache c;
  const uint16_t *q;
  uint16_t *out;
  float *lse, *part, *dpart, *row_r;
  int *counts, *items, *item_off, *status;
  const int *length;  // NULL, or device lengths: tokens of batch row b = length[b * lstride] + tokens
  int lstride;
  int batch, q_heads, kv_heads, tokens;
  int nblocks, nslices;  // layout of lse / items: sub-blocks and slices per head at the capacity
  int hs, gs;            // units between KV heads and between groups
  int qg, vg;            // queries per virtual head, virtual heads per KV head
  int cb, fb;            // plane bits
  int coarse_ctas, coarse_warps;  // persistent coarse CTAs and their warps: how the work is dealt to them is `deal`
  int refine_ctas, refine_warps;  // RW = refine_ctas * refine_warps
  float sl, log2_tau;
  // Sequence shards (one GPU's part of a long context); shard_on 0: the whole cache. A shard processes the closed groups
  // [sh_first, sh_first + sh_count) of its local cache, the BF16 sink window if sh_windows & 1, the open window if & 2.
  // phase 0: a whole decode. phase 1: coarse pass, then only the rows' local log2 mass into row_r. phase 2: select with
  // the given (global) row_r, refine, and the rows' unnormalised sums (o[128], l, relative to row_r) into out_partial.
  int sh_first, sh_count;
  short shard_on, sh_windows, phase;
  short mass_given;    // dense: the rows' masses are in row_r (a pass before, or a shard's caller) instead of formed by the value pass
  float *out_partial;  // [rows][FBLA_K_PSTRIDE] floats (phase 2)
  short refine_fold;   // 1: the refine pass leaves one row of corrections per (CTA, virtual head) instead of one per (warp, virtual head)
  char fold;           // 1: the coarse pass leaves one partial row per (CTA, virtual head) instead of one per (warp, virtual head)
  char deep;           // the coarse pass's shape: 1: few warps with a whole group in flight each; 0: more warps (fbla_decode.cuh)
  char dense;          // 1: two sweeps, weights kept between them (fbla_dense.cuh); 0: coarse sums, then corrections (fbla_decode.cuh)
  char head_ctas;      // two sweeps: n > 0: every virtual head has n CTAs of its own (coarse_ctas in all), in a stream call a cluster of one kernel; 0: the work is dealt over all CTAs
  short deal;          // how the coarse pass's warps share the work, FBLA_K_DEAL_*
} fbla_k_decode;
#define FBLA_K_DEAL_LENGTHS 0 /* a CTA's warps are split between windows and groups by the rows' lengths (short contexts) */
#define FBLA_K_DEAL_FIXED 1   /* the last warps of a CTA (one at least) serve windows, the others stream groups */
#define FBLA_K_DEAL_COST 2    /* every warp takes an equal cost share of windows and groups (long contexts) */

#define FBLA_K_DENSE_MAX_BATCH 1024  /* batch rows of a dense decode: their prefix sums lie in shared memory */
#define FBLA_K_TWO_SCORE_WARPS 16
#define FBLA_K_TWO_VALUE_WARPS 16
#define FBLA_K_PSTRIDE 132 /* floats of one partial row: o[128], then (m, l) or (dl) and padding */
#define FBLA_K_SLICE 1024  /* sub-blocks per select slice */

FBLA_HOST_API(cudaError_t fbla_k_decode_launch(const fbla_k_decode *a, cudaStream_t stream);)
// One pass of a decode alone (0 coarse, 1 select, 2 refine, 3 merge) as an ordinary launch, for timing the passes one by
// one; `a` as fbla_k_decode_launch takes it (e.g. the argument blob of a decode plan). Valid after one whole decode has
// run on the device.
FBLA_HOST_API(cudaError_t fbla_k_decode_pass_launch(const fbla_k_decode *a, int pass, cudaStream_t stream);)
// chooses the split of the coarse CTAs' warps for rows of about `tokens` tokens (after fbla_k_decode_shape; the scratch layout holds either)
FBLA_HOST_API(void fbla_k_decode_split(fbla_k_decode *a, long long tokens);)
// (virtual head, sub-block, query) cells of a decode, padded to 256 bytes of floats. The `lse` array of a decode in two sweeps is
// followed by 2 x cells block maxima and 2 x cells x 16 bytes of weights: FBLA_K_TWO_FLOATS floats per cell in all.
static inline __host__ __device__ size_t fbla_k_two_cells(size_t vheads, int nblocks, int qg) { return (vheads * nblocks * qg + 63) / 64 * 64; }
#define FBLA_K_TWO_FLOATS 11
// whether a decode of rows of about `tokens` tokens with selection threshold tau runs in two sweeps (vheads: virtual heads of the call, qg queries each)
FBLA_HOST_API(int fbla_k_two_sweeps(int batch, int vheads, int qg, long long tokens, float tau);)
// CTAs per virtual head of a decode in two sweeps that may run as one kernel; 0: it runs as three (pure host arithmetic)
FBLA_HOST_API(int fbla_k_head_ctas(int vheads, long long tokens);)
// whether it does, for heads of qg queries and rows of one length or of lengths of their own, where held(a, ctas) clusters of that many CTAs are at
// work at once: its CTAs per head, or 0
FBLA_HOST_API(int fbla_k_head_choice(const fbla_k_decode *a, int vheads, int qg, int own_lengths, long long tokens, int (*held)(const fbla_k_decode *a, int ctas));)
// `held` of the current device
FBLA_HOST_API(int fbla_k_head_clusters(const fbla_k_decode *a, int ctas);)
// the dense passes (0 scores, 1 rows' masses, 2 values, 3 merge): a whole decode or shard phase; one pass (of a decode in one kernel: 0 all of it)
FBLA_HOST_API(cudaError_t fbla_k_dense_launch(const fbla_k_decode *a, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_dense_pass_launch(const fbla_k_decode *a, int pass, cudaStream_t stream);)
// the same choice for a shape given by its numbers (pure host arithmetic: no device is touched): deal and fold as fbla_k_decode_split sets them
FBLA_HOST_API(void fbla_k_decode_split_of(int cb, int batch, int kv_heads, int vg, long long tokens, int *deal, int *fold);)
// and its shape for qg queries per virtual head
FBLA_HOST_API(int fbla_k_decode_deep_of(int batch, int kv_heads, int vg, int qg, long long tokens);)
// out[row][ch] = bf16(partial[row][ch] / partial[row][128]) for rows rows of FBLA_K_PSTRIDE floats
// total[i] = log2 sum over shards of 2^mass[s][i]
FBLA_HOST_API(cudaError_t fbla_k_total_mass_launch(const float *mass, float *total, int shards, int rows, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_combine_launch(const float *partial, uint16_t *out, int rows, cudaStream_t stream);)
// the most (virtual head, slice) entries one decode may have: the refine pass keeps their prefix sums in shared memory
// (fold: with room for the row sets of refine_fold)
FBLA_HOST_API(long long fbla_k_refine_entry_limit(int cb, int fold);)
// occupancy-derived launch shape for the current device; fills coarse_ctas .. refine_warps from cb / qg
FBLA_HOST_API(cudaError_t fbla_k_decode_shape(fbla_k_decode *a);)

// ---- the exchanges of a sequence-sharded decode as stores into the peers' memory (kernels/fbla_link.cu) -------------------
#define FBLA_K_MAX_RANKS 8
typedef struct {
  void *peer[FBLA_K_MAX_RANKS];  // the base of every rank's mailbox, as this rank addresses it (peer[rank]: its own)
  int rank, world, rows;         // rows = batch * q_heads
  unsigned spin_limit;           // polls (64 ns apart) before a wait for a peer gives up
} fbla_k_link;
// Byte offsets inside a mailbox (the same on every rank). epoch: the step counter; status: 0, or which wait gave up
// (1 masses, 2 sums, + 16 * the silent rank); *_flag[s], *_in[s]: the stamp and the data rank s stored here.
typedef struct {
  size_t epoch, status, mass_flag, part_flag, mass_in, local_mass, total, part_in, local_part, bytes;
} fbla_k_mailbox;
static inline __host__ __device__ fbla_k_mailbox fbla_k_mailbox_of(int world, int rows) {
  fbla_k_mailbox m;
  size_t at = 0;
  m.epoch = at; at += 16;
  m.status = at; at += 240;
  m.mass_flag = at; at += 256;
  m.part_flag = at; at += 256;
  m.mass_in = at; at += ((size_t)world * rows * 4 + 255) / 256 * 256;
  m.local_mass = at; at += ((size_t)rows * 4 + 255) / 256 * 256;
  m.total = at; at += ((size_t)rows * 4 + 255) / 256 * 256;
  m.part_in = at; at += ((size_t)world * rows * FBLA_K_PSTRIDE * 4 + 255) / 256 * 256;
  m.local_part = at; at += ((size_t)rows * FBLA_K_PSTRIDE * 4 + 255) / 256 * 256;
  m.bytes = at;
  return m;
}
FBLA_HOST_API(cudaError_t fbla_k_link_push_mass(const fbla_k_link *L, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_link_gather_mass(const fbla_k_link *L, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_link_push_partial(const fbla_k_link *L, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_link_combine(const fbla_k_link *L, uint16_t *out, cudaStream_t stream);)

// ---- prefill: close the chunk's groups, attention, update the BF16 windows --------------------------------------------
typedef struct {
  fbla_k_cache c;
  const uint16_t *q, *k, *v;  // q NULL: append only
  uint16_t *out;
  int64_t out_hs;             // elements between q heads of out
  int out_ts;                 // elements between positions of out
  const int *length;          // NULL, or the chunk starts at length[row * lstride] + n0
  const int *dcount;          // NULL, or the chunk's token count on the device (count is then its ceiling)
  int lstride;
  int batch, q_heads, kv_heads, n0, count;
  int hs, gs;
  int cb, fb;
  float sl;
  // 0: the attention pass serves every count. > 0 (a chunk whose count lives on the device): the attention is two
  // passes and the count decides on the device which of them works -- the tensor-core pass when count * queries per KV
  // head >= tc_min_rows, the few-row pass below that -- so that a device-count call takes the kernel the host-count
  // call of the same chunk takes and the two stay bit-identical.
  int tc_min_rows;
  // > 0 (a chunk that starts a cache whose arrays have no initial contents): the groups per KV head that the layout has
  // room for; what the chunk does not write of their units and of the sink window is zeroed (fbla_k_write_launch)
  int clear_groups;
  int early;    // 1: the close pass also updates the windows of a chunk that starts its cache (nothing reads them then), the finish pass leaves that to it
  int room;     // tokens the cache is laid out for
  int cluster;  // attention passes: CTAs of a tile's cluster, one per share of its groups (1: one CTA does the tile)
  int above;    // tensor-core pass: this launch works where the chunk's tiles have more than `above` and at most `cluster` shares
} fbla_k_prefill;

// close_blocks: grid x of the close pass (groups the chunk can close); 0 skips it
FBLA_HOST_API(cudaError_t fbla_k_close_launch(const fbla_k_prefill *a, int close_blocks, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_finish_launch(const fbla_k_prefill *a, cudaStream_t stream);)
// close and finish of a chunk without queries as one launch
FBLA_HOST_API(cudaError_t fbla_k_write_launch(const fbla_k_prefill *a, int close_blocks, cudaStream_t stream);)
// Attention of the chunk's rows: the tensor-core kernel (tcgen05, 128 rows per CTA), or -- for chunks of fewer than
// FBLA_K_TC_MIN_ROWS rows, or when the environment variable MLOPS_FBLA_PREFILL=rows asks for it -- the few-row kernel.
// fbla_k_attend_plan splits a chunk's attention into its one or two passes (two when the count is on the device and
// its ceiling reaches the tensor-core kernel, see tc_min_rows): args[i] / tensor[i] for pass i; returns their number.
FBLA_HOST_API(int fbla_k_attend_plan(const fbla_k_prefill *a, fbla_k_prefill args[2], int tensor[2]);)
FBLA_HOST_API(cudaError_t fbla_k_attend_launch(const fbla_k_prefill *a, cudaStream_t stream);)  // every pass of the plan
FBLA_HOST_API(cudaError_t fbla_k_attend_rows_launch(const fbla_k_prefill *a, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_attend_tc_launch(const fbla_k_prefill *a, cudaStream_t stream);)
// How the tensor-core pass of `tiles` pairs of row tiles per KV head over `passes` groups is launched (pure host arithmetic): one launch
// for a count on the host, one or two for a count on the device with that ceiling, of which the count picks one. Returns their number.
typedef struct { int cluster, above, tiles; } fbla_k_tc_deal;
FBLA_HOST_API(int fbla_k_attend_tc_deal(int heads, int tiles, int passes, int device_count, fbla_k_tc_deal deal[2]);)
// 1 if a bounded wait of the tensor-core kernel gave up since the last call (and clears it), 0 if not, -1 on a CUDA
// error. A CTA whose wait gave up also writes NaN to every output row it owns, so the failure shows in the data.
FBLA_HOST_API(int fbla_k_attend_tc_status(void);)
#define FBLA_K_TC_MIN_ROWS 64
#define FBLA_K_TILE_SHARES 8  /* CTAs of a tensor-core tile's cluster at most */
#define FBLA_K_ROW_SHARES 8  /* CTAs of a few-row tile's cluster at most */

// ---- fused QKV step: RMSNorm + rotary embedding of new tokens (+ the window stores of the one-token step) ------------------
typedef struct {
  fbla_k_cache c;                 // token step only
  const uint16_t *q, *k, *v;      // the projection's output
  int64_t batch_stride, q_group_stride, kv_group_stride;  // elements; batch_stride is the row stride of a chunk
  const uint16_t *q_norm, *k_norm;  // both or neither
  const float *freq;              // 64 x (fh, fl, gh, gl)
  float eps, att;
  const int *length, *dcount;
  int lstride, n0, max_count;
  int batch, q_heads, kv_heads;
  uint16_t *q_out, *k_out, *v_out;
} fbla_k_token;
// the one-token step: the group the position closes, then the token, in one launch
FBLA_HOST_API(cudaError_t fbla_k_qkv_step_launch(const fbla_k_prefill *closing, const fbla_k_token *a, cudaStream_t stream);)
FBLA_HOST_API(cudaError_t fbla_k_qkv_chunk_launch(const fbla_k_token *a, cudaStream_t stream);)

// ---- what an executor needs to run a pass from kernels of its own (include/mlops_fbla_items.h) ---------------------------
typedef struct {
  int gx, gy, gz;    // the grid of the equivalent launch: one item per CTA
  int threads;       // the exact CTA size
  int smem_bytes;    // shared memory to hand the entry (includes the slack entries use to re-align a 16-byte aligned pointer)
  int regs;          // registers per thread of this library's kernel
  char entry[96];    // the device function (kernels/*.cuh), called as entry(args, shared memory)
} fbla_k_pass;
FBLA_HOST_API(cudaError_t fbla_k_decode_passes(const fbla_k_decode *a, fbla_k_pass info[4]);)  // coarse, select, refine, merge
FBLA_HOST_API(cudaError_t fbla_k_dense_passes(const fbla_k_decode *a, fbla_k_pass info[4]);)
FBLA_HOST_API(cudaError_t fbla_k_close_pass(const fbla_k_prefill *a, int close_blocks, fbla_k_pass *info);)
FBLA_HOST_API(cudaError_t fbla_k_finish_pass(const fbla_k_prefill *a, fbla_k_pass *info);)
FBLA_HOST_API(cudaError_t fbla_k_attend_rows_pass(fbla_k_prefill *a, fbla_k_pass *info);)  // (sets a->cluster)
FBLA_HOST_API(cudaError_t fbla_k_attend_tc_pass(fbla_k_prefill *a, fbla_k_pass *info);)    // (sets a->cluster)
FBLA_HOST_API(cudaError_t fbla_k_qkv_token_pass(const fbla_k_token *a, fbla_k_pass *info);)
FBLA_HOST_API(cudaError_t fbla_k_qkv_chunk_pass(const fbla_k_token *a, fbla_k_pass *info);)

#ifdef __cplusplus
}
#endif
