/* Hierarchical int4 weights on their way into a tensor-core operand tile (cuda/hier.cuh:8-13
 * of the engine, the arithmetic of cuda/chunk_gemm.cu:121-132): a warp that fetches the packed
 * words and scale bytes of 128 columns of some rows into a slot of shared memory, and warps
 * that unpack a slot into two 64-column slabs of the swizzled operand layout.  The fetch is
 * asynchronous and a warp's own because the unpacking warps' fence towards the async proxy
 * would wait for any load from global memory that they have in flight. */
#pragma once

#include "wst_ptx.cuh"

namespace wst {

/* A slot: 64 bytes of packed words per row, then 4 scale bytes per row. */
constexpr int slot_bytes(int rows) { return rows * 68; }

/* The fetching warp's view of rows n0 .. n0 + ROWS - 1 (a whole warp works on it).  A stage costs
 * it a request and a few copies per lane; what does not change from stage to stage is worked out
 * once, or the single warp is what bounds the narrower tiles. */
template <int ROWS>
struct PackedRows {
  static constexpr int N = ROWS / 32;
  const uint8_t *at[N]; /* scale bytes of rows n0 + lane + 32 i */
  uint32_t take[N];     /* 4, or 0 past the last row: zeros */
  const CUtensorMap *map;
  int groups, n0;
  bool quads; /* four scale bytes of a row and stage in one asynchronous copy where they lie aligned */

  __device__ __forceinline__ PackedRows(const CUtensorMap *map_, const uint8_t *si, int groups_, int out_f,
                                        int n0_, int lane)
      : map(map_), groups(groups_), n0(n0_) {
    quads = groups % 4 == 0 && (reinterpret_cast<uintptr_t>(si) & 3) == 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int row = n0 + lane + 32 * i;
      take[i] = row < out_f ? 4 : 0;
      at[i] = si + static_cast<size_t>(row < out_f ? row : 0) * groups;
    }
  }
  /* Fills `slot` with columns 128 kb .. + 127; `full` counts one arrival of the words' request
   * and 32 of the lanes' scale bytes. */
  __device__ __forceinline__ void fetch(uint32_t slot, uint32_t full, int kb, int lane) const {
    using namespace ptx;
    if (lane == 0) {
      mbar_arrive_expect_tx(full, ROWS * 64);
      tma_load_3d(slot, map, full, kb * 32, n0, 0);
    }
    const uint32_t dst = slot + ROWS * 64 + 4 * lane;
    if (quads) {
#pragma unroll
      for (int i = 0; i < N; ++i)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 128 * i), "l"(at[i] + 4 * kb),
                     "r"(take[i])
                     : "memory");
      asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(full) : "memory");
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        uint32_t v = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (take[i] && 4 * kb + j < groups)
            v |= static_cast<uint32_t>(__ldg(at[i] + 4 * kb + j)) << (8 * j);
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + 128 * i), "r"(v) : "memory");
      }
      mbar_arrive(full);
    }
  }
};
/* before the fetching warp leaves: its own copies have landed */
__device__ __forceinline__ void fetch_packed_drain() { asm volatile("cp.async.wait_all;" ::: "memory"); }

/* A nibble q dropped into byte 2 of 0x3F000000 is the float 0.5 + q / 256, one byte permute
 * per weight; then w = q s - dmin lm = (256 s) f - (128 s + dmin lm) with s = d * ls is ONE fp32
 * fma per weight, and the result is rounded to fp16 once -- the only difference from the exact
 * weight, random in sign.  (In half2 arithmetic the rounded offset is common to the 32 weights
 * of a group and adds up along it: 9.7e-3 from the exact product on the engine's test case
 * where this form has 1.3e-3.) */
struct GroupScale {
  float mul, add; /* 256 s, -(128 s + dmin lm) */
};
__device__ __forceinline__ GroupScale group_scale(float2 dd, unsigned idx) {
  const float s1 = dd.x * static_cast<float>(idx & 0xFu); /* d * ls */
  return {256.0f * s1, fmaf(-128.0f, s1, -dd.y * static_cast<float>(idx >> 4))};
}
/* the eight weights of a word, 2i (low nibble of byte i) and 2i + 1 as one half2 */
__device__ __forceinline__ void unpack_word(uint32_t word, GroupScale g, uint32_t (&o)[4]) {
  const uint32_t even = word & 0x0F0F0F0Fu, odd = (word >> 4) & 0x0F0F0F0Fu;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float f0 = __uint_as_float(__byte_perm(even, 0x3F000000u, 0x7044u | (i << 8)));
    const float f1 = __uint_as_float(__byte_perm(odd, 0x3F000000u, 0x7044u | (i << 8)));
    o[i] = ptx::pack_half2(fmaf(f0, g.mul, g.add), fmaf(f1, g.mul, g.add));
  }
}

/* Group j (32 columns) of `row` of a ROWS-row slot -> fp16 weights in the operand tile of two
 * 64-column slabs at `tile`.  Eight rows x four groups per warp: lane = 4 (row % 8) + j.
 * Columns past in_f came as zeros and meet zeros of x. */
template <int ROWS>
__device__ __forceinline__ void unpack_group(const uint8_t *slot, uint8_t *tile, int row, int j, float2 dd) {
  using namespace ptx;
  const uint4 w = *reinterpret_cast<const uint4 *>(slot + row * 64 + j * 16);
  const unsigned idx = slot[ROWS * 64 + row * 4 + j];
  uint8_t *slab = tile + (j >> 1) * ROWS * 128;
  const GroupScale scale = group_scale(dd, idx);
  /* the two slabs' lanes take their words in different order: the eight 16-byte stores of a
   * phase, two rows x four groups, then fall on eight different bank groups */
  const bool swap = j >= 2;
  const uint32_t words[4] = {swap ? w.z : w.x, swap ? w.w : w.y, swap ? w.x : w.z, swap ? w.y : w.w};
#pragma unroll
  for (int wi = 0; wi < 4; ++wi) { /* 8 weights = one 16-byte chunk per word */
    uint32_t o[4];
    unpack_word(words[wi], scale, o);
    const int chunk = (j & 1) * 4 + (swap ? wi ^ 2 : wi);
    *reinterpret_cast<uint4 *>(slab + swz128(row, chunk)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace wst
