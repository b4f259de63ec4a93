/* CPU-only checks of the arithmetic that cuts a chunk's KV range and picks its kernel
 * (whetstone_b200/csrc/chunk_plan.hpp). */
#include <cstdio>
#include <initializer_list>

#include "chunk_plan.hpp"

using namespace wst;

static int failures = 0;
#define CHECK(cond, ...)                                          \
  do {                                                            \
    if (!(cond)) {                                                \
      std::printf("FAILED %s:%d: %s  ", __FILE__, __LINE__, #cond); \
      std::printf(__VA_ARGS__);                                   \
      std::printf("\n");                                          \
      ++failures;                                                 \
    }                                                             \
  } while (0)

constexpr int kSms = 148;
static int up(int a, int b) { return (a + b - 1) / b; }

/* heads of a group, KV heads, tokens, positions: every tile in one slice, no slice without one,
 * no launch of more CTAs than SMs */
static void slices_cover_the_prefix_and_none_is_empty() {
  for (int gqa : {1, 4, 7, 8, 64})
    for (int n_kv : {1, 2, 4, 8, 32})
      for (int n : {1, 2, 5, 9, 18, 19, 64, 73, 128, 256, 512})
        for (int len = n; len <= 40000; len = len < 1100 ? len + 1 : len + 61) {
          const int hd = len % 2 ? 64 : 128;
          const long long tiles = query_tiles(n, gqa) * n_kv;
          const int s = chunk_slices(kSms, tiles, hd, len, true);
          if (s == 1) continue;
          const int kv = up(len, kKvTile), each = slice_tiles(len, s);
          CHECK(s <= kMaxChunkSlices && s * tiles <= kSms, "%d slices of %lld tiles", s, tiles);
          CHECK(s * each >= kv && (s - 1) * each < kv, "%d slices of %d for %d tiles, len %d", s, each, kv, len);
        }
}

/* either side of a KV tile's end the same prefix is cut the same way */
static void a_prefix_that_ends_with_a_tile_is_cut_like_its_neighbours() {
  for (int tiles : {1, 2, 4, 8})
    for (int len = 512; len <= 4096; len += 128) {
      const int hd = len % 256 ? 128 : 64;
      const int s = chunk_slices(kSms, tiles, hd, len, true);
      CHECK(s == chunk_slices(kSms, tiles, hd, len - 1, true), "len %d", len);
      CHECK(slice_tiles(len, s) == slice_tiles(len - 1, s), "len %d", len);
    }
  /* 28 heads over 4, 5 tokens, 4096 positions: 32 KV tiles in 32 slices */
  const int s = chunk_slices(kSms, query_tiles(5, 7) * 4, 128, 4096, true);
  CHECK(s == 32 && slice_tiles(4096, s) == 1, "%d slices of %d", s, slice_tiles(4096, s));
}

/* tiles hold whole tokens: 18 of seven heads, not 128 rows */
static void query_tiles_are_the_kernels_own() {
  CHECK(query_tiles(73, 7) == 5, "%lld", query_tiles(73, 7));
  CHECK(query_tiles(18, 7) == 1 && query_tiles(19, 7) == 2, "18 tokens fill one");
  CHECK(query_tiles(32, 4) == 1 && query_tiles(33, 4) == 2, "32 tokens fill one");
  CHECK(query_tiles(3, 64) == 2, "two tokens fill one");
}

/* the capacity of a cache says little about the prefix: no runs of single tiles */
static void a_capacity_is_cut_into_runs_of_two_tiles_at_least() {
  for (int tiles : {1, 2, 4, 8, 16, 32, 74})
    for (int cap : {128, 512, 513, 2048, 8192, 32768})
      CHECK(chunk_slices(kSms, tiles, 128, cap, false) == 1 || chunk_slices(kSms, tiles, 128, cap, false) * 2 <= up(cap, kKvTile),
            "%d tiles, %d rows", tiles, cap);
}

/* few query rows: the row blocks keep what they stream faster */
static void few_rows_go_where_they_are_faster() {
  for (int len : {2, 128, 300, 2000, 4103, 32768}) {
    CHECK(!chunk_in_tiles(7, 128, len) && !chunk_in_tiles(16, 128, len), "one block, len %d", len);
    CHECK(chunk_in_tiles(35, 128, len) && chunk_in_tiles(63, 128, len), "three and four blocks, len %d", len);
    CHECK(!chunk_in_tiles(14, 64, len) && chunk_in_tiles(28, 64, len) == (len <= 128), "64 columns, len %d", len);
    CHECK(chunk_in_tiles(28, 128, len) == (len <= 256 || len > 2048), "two blocks, len %d", len);
    CHECK(chunk_in_tiles(56, 64, len) == (len <= 256 || len > 2048), "four of 64 columns, len %d", len);
  }
  CHECK(!prompts_in_items(633, 25) && !prompts_in_items(890, 50) && prompts_in_items(891, 50), "short contexts");
  CHECK(prompts_in_items(768, 700) && !prompts_in_items(600, 1500) && prompts_in_items(600, 1501), "long prompts");
}

int main() {
  slices_cover_the_prefix_and_none_is_empty();
  a_prefix_that_ends_with_a_tile_is_cut_like_its_neighbours();
  query_tiles_are_the_kernels_own();
  a_capacity_is_cut_into_runs_of_two_tiles_at_least();
  few_rows_go_where_they_are_faster();
  std::printf(failures ? "%d failures\n" : "chunk plan ok\n", failures);
  return failures != 0;
}
