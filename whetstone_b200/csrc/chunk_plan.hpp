/* Where a chunk's attention goes and how its KV range is cut, from sizes alone: host arithmetic of
 * attention_api.cu and attn_prefill.cu, apart so that it can be checked without a GPU. */
#pragma once

namespace wst {

constexpr int kKvTile = 128;       /* positions per KV tile of the tcgen05 kernels */
constexpr int kMaxChunkSlices = 64;

/* A query tile is up to 128 rows, whole tokens with all the heads of a KV head's group. */
inline long long query_tiles(int n, int gqa) {
  const int tokens = 128 / gqa;
  return (static_cast<long long>(n) + tokens - 1) / tokens;
}

/* KV tiles of a slice when `len` positions are cut into `slices` runs; the last may be shorter. */
inline int slice_tiles(int len, int slices) {
  const int tiles = (len + kKvTile - 1) / kKvTile;
  return (tiles + slices - 1) / slices;
}

/* Slices of the KV range for a chunk launch of `tiles` (unit, query tile) pairs against `len`
 * positions: none when the tiles fill the GPU by themselves or the prefix is short; else enough to
 * fill it, in runs of at least two KV tiles.  Up to sixteen tiles, full or not, leave so many SMs
 * idle that runs of one pay, behind 256 rows already (384 from nine tiles on: 64 tokens of 28 heads over
 * 4 behind 257 rows 14.5 us unsplit, 16.5 in three slices; append and attention, caches from HBM: 5 tokens of
 * 28 heads over 4 of 128 behind 500 rows 10.6 us in four slices, 11.7 in two, 12.5 unsplit; 24
 * behind 1000 rows 16.0 in eight and 16.7 in four; 73 of 14 over 2 of 64 behind 1024 12.3 and 13.3;
 * in the mean over three shapes and prefixes to 32,768 at most 1.5 % behind the best cut, runs of two
 * 6 % at four tiles, 3 to 6 at eight, 1 to 2 at sixteen; 256 tokens of 28 heads over 4 behind none or
 * 256: 17.1 us unsplit, 19.6 split).
 * `exact`: every query tile sees about `len`.  Where it is only the capacity of the caches a short
 * prefix pays for every slice that finds nothing: 16 tokens behind 200 rows in a cache of 2048 take
 * 11.3 us in sixteen slices and 10.5 in eight, and behind 1000 rows the two are level. */
inline int chunk_slices(int sm_count, long long tiles, int hd, int len, bool exact) {
  const bool ones = exact && tiles <= 16;
  const int least = !ones ? 512 : tiles > 8 ? 384 : 256;
  if (tiles <= 0 || tiles * 2 > sm_count || len <= least) return 1;
  long long s = sm_count / tiles;
  const int kv_tiles = (len + kKvTile - 1) / kKvTile;
  const int most = kv_tiles / (ones ? 1 : 2);
  if (s > most) s = most;
  if (s > kMaxChunkSlices) s = kMaxChunkSlices;
  if (s < 2) return 1;
  if (!exact) return static_cast<int>(s); /* the kernel cuts each prefix as it finds it */
  int each = slice_tiles(len, static_cast<int>(s));
  /* where runs of one would take nearly every SM the merge and the next launch find none free: 5
   * tokens of 28 heads over 4 of 128 behind 4103 rows 13.7 us in 33 slices, 12.1 in 17.  (Tiles of 64
   * columns take half as long: 24 of 14 over 2 of 64 11.2 and 11.9.) */
  if (hd == 128 && each == 1 && kv_tiles * tiles * 8 > sm_count * 7LL) each = 2;
  return (kv_tiles + each - 1) / each; /* no slice without a tile */
}

/* Does a chunk of fewer than 64 query rows per KV head (`rows` = tokens x heads of the group) go to
 * the 128-row tcgen05 tiles, cut along the prefix, or to the mma.sync row-block kernel, 16 rows per
 * block?  What a block costs goes with rows x head_dim, a tile costs the same however empty it is.
 * Append and attention, caches from HBM, tiles against row blocks:
 *   one block of 128 columns or two of 64: 1 token of 28 heads over 4 of 128 behind 300, 2000 and
 *     16384 rows 8.1, 8.1 and 13.8 us against 5.9, 7.2 and 13.4; 4 of 14 over 2 of 64 behind 2000
 *     10.1 and 8.6.  Behind a single KV tile, which needs no merge, 3 tokens of 64 columns 6.9 and 7.4;
 *   up to twice that: 4 of 28 over 4 behind 300, 2000 and 4103 rows 10.6, 11.4 and 11.7 against
 *     10.2, 10.8 and 12.7; behind 128 rows 8.2 and 9.4;
 *   more (head_dim 128): 5 of 28 over 4 behind 300, 2000 and 16384 rows 10.9, 11.8 and 17.7 against
 *     12.3, 13.0 and 27.0. */
inline bool chunk_in_tiles(int rows, int hd, int len) {
  const int cells = rows * hd;
  if (cells <= 16 * 128) return rows > 16 && len <= kKvTile;
  if (cells <= 32 * 128) return len <= 2 * kKvTile || len > 2048;
  return true;
}

/* Ragged paged batches with prompts of more than one query tile per KV head: the persistent tcgen05
 * kernel pays three KV tiles' time for each (sequence, KV head, query tile) and a merge of partial
 * rows, the row-block kernel reads K and V once per 64 rows.  Known here: the longest context and the
 * mean of query rows per (sequence, KV head).  Layer with the append, 410 batches of up to 24
 * sequences with 1 to 6 prompts of 16 to 512 rows, head_dim 64 and 128: below the line the row blocks
 * take 0.80 of the time in the mean (0.59 to 1.16; 24 sequences of 211 to 633 rows, three prompts of
 * 22: 24 and 31 us); above it the items take 0.77 in the mean (10 of 387 to 3096, four prompts of 483:
 * 198 and 434 us) and 22 of 192 batches are 1.05 to 1.38 times as fast with row blocks. */
inline bool prompts_in_items(int max_len, long long mean_rows) { return 5LL * max_len + mean_rows > 4500; }

}  // namespace wst
