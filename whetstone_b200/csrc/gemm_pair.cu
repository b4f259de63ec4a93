/* The projections of a real chunk (more than 128 tokens): two SMs on one tile.
 *
 *     y[j][r] (+)= sum_c x[j][c] * w[r][c] + bias[r]        j < n tokens, r < out_f
 *
 * What bounds it is the tensor pipe, once the operands reach it: a 128 x 256 tile on one SM
 * brings 48 KB into shared memory and reads 48 KB out of it for every 512 clocks of
 * tcgen05.mma, more than the 128 bytes a clock that shared memory moves.  So a cluster of
 * two CTAs takes one 256-token x BN-feature tile with cta_group::2 MMAs: each CTA holds its
 * 128 token rows and HALF of the weight tile, both accumulate 128 x BN in their own tensor
 * memory, and a k-step moves two thirds of the bytes.  Two accumulators, so the epilogue of
 * one tile runs under the main loop of the next; persistent clusters walk the tiles
 * token-tile fastest, the clusters that run together share weight tiles in L2.  fp16, 2048
 * tokens of 4096 -> 4096: 53 us (1300 TFLOP/s), 70 with one SM per 128 x 256 tile.
 *
 * int4 weights (INT4): sixteen warps of each CTA unpack its half of the weight tile into the
 * operand layout, half the work per SM that a tile of one SM would need.  The packed words
 * come through a ring of their own (TMA; one warp copies the scale bytes): an unpacking warp
 * has no load from global memory of its own in flight, because its fence towards the async
 * proxy would wait for it.  1527 tokens of 4096 -> 4096, accumulating: 54 us, 317 with every
 * tile unpacked by one SM from loads of its own.
 *
 * The fused qkv form (ROPE) normalises, rotates and stores whole heads from the accumulator.
 *
 * Products are exact in fp32 and accumulated in fp32. */

#include "gemm_pair.cuh"
#include "int4_tile.cuh"
#include "tensor_map.cuh"
#include "wst_ptx.cuh"

namespace wst {
namespace {

using namespace ptx;

constexpr int kUnpackWarps = 16;

/* BN features per tile of the pair; a stage is 128 columns of K: two 64-column slabs of
 * this CTA's 128 token rows and BN / 2 weight rows. */
template <int BN, bool INT4>
struct PairCfg {
  static constexpr int BM = 128, KS = 2, BK = 64 * KS, BH = BN / 2;
  static constexpr int A_SLAB = BM * 128, B_SLAB = BH * 128;
  static constexpr int A_BYTES = KS * A_SLAB, B_BYTES = KS * B_SLAB;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int NSTAGE = (192 * 1024) / STAGE_BYTES;
  /* packed words and scale bytes of one stage */
  static constexpr int SLOT_BYTES = slot_bytes(BH);
  static constexpr int NSLOT = !INT4 ? 0 : 26112 / SLOT_BYTES < 8 ? 26112 / SLOT_BYTES : 8;
  static constexpr int OFF_PACK = NSTAGE * STAGE_BYTES;
  static constexpr int EC = INT4 ? 16 : 32; /* columns that the epilogue stages at a time */
  static constexpr int EPI_WARP = 32 * EC * 4;
  static constexpr int OFF_EPI = OFF_PACK + NSLOT * SLOT_BYTES;
  static constexpr int OFF_BAR = OFF_EPI + 4 * EPI_WARP;
  static constexpr int NBAR = 2 * NSTAGE + 4 + 2 * NSLOT;
  static constexpr int OFF_BOX = (OFF_BAR + NBAR * 8 + 4 + 15) / 16 * 16;
  static constexpr int SMEM_BYTES = OFF_BOX + 16 + 1024;
  static constexpr int TMEM_COLS = 2 * BN;
  /* Unpacking warps on one stage, each with UNITS times eight rows, and sets of them that take
   * the stages in turn: with all sixteen on one stage (BN = 256, one unit each) they waited,
   * unpacked and fenced in step, 1600 clocks a stage of which 600 were instructions. */
  static constexpr int UNITS = BN >= 256 ? 2 : 1;
  static constexpr int STAGE_WARPS = BH / (8 * UNITS);
  static constexpr int SETS = kUnpackWarps / STAGE_WARPS;
  static_assert(SMEM_BYTES <= 227 * 1024 && TMEM_COLS <= 512, "does not fit");
  static_assert(SLOT_BYTES % 128 == 0 && SETS >= 1, "slot geometry");
};

struct PairArgs {
  PairGemm g;
  int m_tiles, n_tiles;
  unsigned int *err_word;
};

/* ---- two-CTA forms of the tcgen05 and mbarrier instructions */

/* Tells the pair's first CTA, by 16 bytes that its barrier counts, that what this thread has seen
 * happen in its own CTA has happened: the copy is issued behind that, and its completion is a
 * release at cluster scope.  (An arrival with such a release is as sound but makes the arriving
 * thread wait for the SM's memory traffic, 0.5 to 0.9 us each: 256 tokens of 3584 -> 4608, int4
 * weights, 15.5 us with messages, 28 with one arrival a stage, 15.0 with arrivals that order nothing.) */
constexpr int kMessage = 16;
__device__ __forceinline__ void tell_leader(uint32_t mailbox, uint32_t src, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(in_cta(mailbox, 0)), "r"(src), "n"(kMessage), "r"(in_cta(bar, 0))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
/* mbar_wait for what the other CTA announces */
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, unsigned int *err_word,
                                                  unsigned int code) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait_cluster(bar, parity)) {
    if (clock64() - t0 > kWaitCycleLimit) {
      if (err_word) atomicCAS(err_word, 0u, code);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void pair_tmem_alloc(uint32_t dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
               : "memory");
}
/* this CTA's half of an operand tile; the bytes are counted on `bar`, in either CTA */
__device__ __forceinline__ void pair_tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                                 int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void pair_umma_ss_f16(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo,
                                                 uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
/* arrives on the barrier at this offset in both CTAs once the MMAs issued so far are done */
__device__ __forceinline__ void pair_umma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"(static_cast<uint16_t>(3))
      : "memory");
}
/* y += v on four floats, 16-byte aligned; no other thread adds to them.  The reduction adds where
 * the numbers lie, without the latency of reading them, but takes numbers below 2^-126 for zeros,
 * in y and in the sum.  With |v| >= 2^-100 that changes nothing -- such a y is below half of v's
 * last place, and a sum that cancels is a multiple of 2^-124 -- and below it a sum of products of
 * fp16 numbers is zero: those are added in registers.  (Read ahead by a pass, y cost 1000 tokens of 4096 -> 4096
 * with int4 weights 50 us instead of 33, 2048 with fp16 ones 56 instead of 54.) */
__device__ __forceinline__ void add_v4(float *y, float4 v) {
  constexpr float kSmall = 0x1p-100f;
  if (fminf(fminf(fabsf(v.x), fabsf(v.y)), fminf(fabsf(v.z), fabsf(v.w))) >= kSmall) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(y), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
  } else {
    float4 old = *reinterpret_cast<const float4 *>(y);
    old.x += v.x; old.y += v.y; old.z += v.z; old.w += v.w;
    *reinterpret_cast<float4 *>(y) = old;
  }
}

/* Epilogue of the fused form for one head of one token: HD accumulator columns from tensor
 * memory (+ bias) -> per-head RMS norm with fp16 gains (q and k heads, if gains are given) ->
 * half-rotation RoPE at the token's position -> fp16, to the q buffer or to the token's cache
 * row; v heads are narrowed and stored as they are.  The arithmetic is that of
 * rope_append_kernel (norm before rotation, x * inv * gain, cuda/decode.cu:112-178 and
 * cuda/chunk_ops.cu:101-150 of the engine).  The head is read twice, once for the norm and
 * then sixteen column pairs at a time: 736 threads leave 80 registers. */
template <int HD>
__device__ __forceinline__ void rope_head_epilogue(const PairGemm &g, uint32_t tmem_head, int head,
                                                   int tpos, long long kv_row, int tok, bool valid) {
  constexpr int HALF = HD / 2;
  const bool is_q = head < g.n_q, is_k = !is_q && head < g.n_q + g.n_kv;
  const bool rotate = is_q || is_k;
  const __half *gain = is_q ? g.q_gain : is_k ? g.k_gain : nullptr;
  const __half *bias = g.bias && valid ? g.bias + head * HD : nullptr;
  auto with_bias = [bias](uint32_t (&v)[16], int c0, float (&f)[16]) {
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      f[e] = __uint_as_float(v[e]);
      f[e + 1] = __uint_as_float(v[e + 1]);
      if (bias) {
        const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(bias + c0 + e));
        f[e] += b.x;
        f[e + 1] += b.y;
      }
    }
  };
  float inv = 1.f;
  if (gain) {
    float ss = 0.f;
#pragma unroll
    for (int c0 = 0; c0 < HALF; c0 += 16) {
      uint32_t lo[16], hi[16];
      tmem_ld_32x16(tmem_head + c0, lo);
      tmem_ld_32x16(tmem_head + HALF + c0, hi);
      tmem_ld_wait();
      float a[16], b[16];
      with_bias(lo, c0, a);
      with_bias(hi, HALF + c0, b);
#pragma unroll
      for (int e = 0; e < 16; ++e) ss = fmaf(a[e], a[e], fmaf(b[e], b[e], ss));
    }
    inv = rsqrtf(ss / static_cast<float>(HD) + g.eps);
  }
  __half *dst;
  if (is_q) {
    dst = g.q_out + (static_cast<long long>(tok) * g.n_q + head) * HD;
  } else {
    const int kvh = is_k ? head - g.n_q : head - g.n_q - g.n_kv;
    dst = (is_k ? g.k_cache : g.v_cache) + kv_row + static_cast<long long>(kvh) * g.max_seq * HD;
  }
  const float4 *ct = reinterpret_cast<const float4 *>(g.cos_tab + static_cast<long long>(tpos) * HALF);
  const float4 *st = reinterpret_cast<const float4 *>(g.sin_tab + static_cast<long long>(tpos) * HALF);
#pragma unroll 1
  for (int c0 = 0; c0 < HALF; c0 += 16) {
    uint32_t lo[16], hi[16];
    __syncwarp(); /* the lanes without a token skipped the stores of the step before */
    tmem_ld_32x16(tmem_head + c0, lo);
    tmem_ld_32x16(tmem_head + HALF + c0, hi);
    tmem_ld_wait();
    if (!valid) continue;
    float a[16], b[16];
    with_bias(lo, c0, a);
    with_bias(hi, HALF + c0, b);
    if (gain) {
#pragma unroll
      for (int e = 0; e < 16; e += 2) {
        const float2 ga = __half22float2(*reinterpret_cast<const __half2 *>(gain + c0 + e));
        const float2 gb = __half22float2(*reinterpret_cast<const __half2 *>(gain + HALF + c0 + e));
        a[e] = a[e] * inv * ga.x;
        a[e + 1] = a[e + 1] * inv * ga.y;
        b[e] = b[e] * inv * gb.x;
        b[e + 1] = b[e + 1] * inv * gb.y;
      }
    }
    if (rotate) {
#pragma unroll
      for (int e = 0; e < 16; e += 4) {
        const float4 c = __ldg(ct + (c0 + e) / 4), s = __ldg(st + (c0 + e) / 4);
        const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float x1 = a[e + k], x2 = b[e + k];
          a[e + k] = x1 * cc[k] - x2 * ss[k];
          b[e + k] = x2 * cc[k] + x1 * ss[k];
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 16; e += 8) {
      *reinterpret_cast<uint4 *>(dst + c0 + e) =
          make_uint4(pack_half2(a[e], a[e + 1]), pack_half2(a[e + 2], a[e + 3]),
                     pack_half2(a[e + 4], a[e + 5]), pack_half2(a[e + 6], a[e + 7]));
      *reinterpret_cast<uint4 *>(dst + HALF + c0 + e) =
          make_uint4(pack_half2(b[e], b[e + 1]), pack_half2(b[e + 2], b[e + 3]),
                     pack_half2(b[e + 4], b[e + 5]), pack_half2(b[e + 6], b[e + 7]));
    }
  }
}

/* Threads of a CTA: 4 epilogue warps, the MMA warp, the TMA warp, and for the int4 form the
 * warp that fetches packed weights and those that unpack them into shared memory. */
constexpr int pair_threads(bool int4) { return 32 * (int4 ? 7 + kUnpackWarps : 6); }

template <int BN, bool ROPE, bool INT4>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_threads(INT4), 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                 const __grid_constant__ PairArgs a) {
  using C = PairCfg<BN, INT4>;
  constexpr int NSTAGE = C::NSTAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto bar = [bar0](int i) { return bar0 + 8u * i; };
  /* EMPTY and ACC_FULL: the leader's MMAs announce them in each CTA.  FULL and ACC_EMPTY: what a
   * CTA's own threads have done for its half of a tile is counted in that CTA; the second CTA's
   * idle MMA warp waits there and tells the leader's barrier. */
  constexpr int FULL = 0, EMPTY = NSTAGE, ACC_FULL = 2 * NSTAGE, ACC_EMPTY = ACC_FULL + 2;
  constexpr int P_FULL = ACC_EMPTY + 2, P_EMPTY = P_FULL + C::NSLOT;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::OFF_BAR + C::NBAR * 8);
  const uint32_t mailbox = sbase + C::OFF_BOX; /* of messages: nobody reads it */
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const PairGemm &g = a.g;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NSTAGE; ++i) {
      /* leader: the announcement of the bytes; either: its own unpacking warps */
      mbar_init(bar(FULL + i), !INT4 ? 1 : rank == 0 ? 1 + C::STAGE_WARPS : C::STAGE_WARPS);
      mbar_init(bar(EMPTY + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(ACC_FULL + i), 1);
      mbar_init(bar(ACC_EMPTY + i), 4);
    }
    for (int i = 0; i < C::NSLOT; ++i) {
      mbar_init(bar(P_FULL + i), 1 + 32); /* the words' request, each lane's scale bytes */
      mbar_init(bar(P_EMPTY + i), C::STAGE_WARPS);
    }
    mbar_init_fence();
    tma_prefetch_desc(&xmap);
    tma_prefetch_desc(&wmap);
  }
  __syncwarp();
  if (warp == 4) pair_tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync(); /* both CTAs' barriers exist before either is arrived on */
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  grid_dependency_wait();

  const int n_tiles_total = a.m_tiles * a.n_tiles;
  const int k_blocks = (g.in_f + C::BK - 1) / C::BK;
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int my_tiles =
      first_tile < n_tiles_total ? (n_tiles_total - 1 - first_tile) / tile_step + 1 : 0;

  if (warp == 5) {
    /* ------------------------------------------------------ TMA producer, one per CTA */
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_step) {
        const int m0 = (tile % a.m_tiles) * 256 + rank * 128;
        const int n0 = (tile / a.m_tiles) * BN + rank * C::BH;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int st = it % NSTAGE;
          if (it >= NSTAGE &&
              !mbar_wait(bar(EMPTY + st), ((it / NSTAGE) - 1) & 1, a.err_word, 0x901u)) {
            ok = false;
            break;
          }
          /* the leader's barrier counts the bytes of both CTAs, and the message that the second
           * CTA's weights are unpacked */
          if (rank == 0)
            mbar_arrive_expect_tx(bar(FULL + st), INT4 ? 2 * C::A_BYTES + kMessage : 2 * C::STAGE_BYTES);
          const uint32_t full = in_cta(bar(FULL + st), 0);
          const uint32_t dst = sbase + st * C::STAGE_BYTES;
#pragma unroll
          for (int s = 0; s < C::KS; ++s) {
            pair_tma_load_3d(dst + s * C::A_SLAB, &xmap, full, kb * C::BK + 64 * s, m0, 0);
            if constexpr (!INT4)
              pair_tma_load_3d(dst + C::A_BYTES + s * C::B_SLAB, &wmap, full, kb * C::BK + 64 * s, n0, 0);
          }
        }
      }
      /* the last uses' commits arrive here, from the leader's MMAs: not after this CTA is gone */
      for (int u = it > NSTAGE ? it - NSTAGE : 0; ok && u < it; ++u)
        ok = mbar_wait(bar(EMPTY + u % NSTAGE), (u / NSTAGE) & 1, a.err_word, 0x909u);
    }
  } else if (INT4 && warp == 6) {
    /* -------------------------------- packed words and scale bytes of this CTA's rows */
    if constexpr (INT4) {
      int it = 0;
      bool ok = true;
      for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_step) {
        const PackedRows<C::BH> packed(&wmap, g.si, g.in_f / 32, g.out_f,
                                       (tile / a.m_tiles) * BN + rank * C::BH, lane);
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int sl = it % C::NSLOT;
          if (it >= C::NSLOT) {
            const bool free = mbar_wait(bar(P_EMPTY + sl), ((it / C::NSLOT) - 1) & 1, a.err_word, 0x907u);
            if (!__all_sync(0xffffffffu, free)) { ok = false; break; }
          }
          packed.fetch(sbase + C::OFF_PACK + sl * C::SLOT_BYTES, bar(P_FULL + sl), kb, lane);
        }
      }
      fetch_packed_drain();
    }
  } else if (warp > 6) {
    /* ---------------------- int4 weights -> this CTA's half of the fp16 tile.  A warp takes
     * UNITS times 8 rows x 4 groups of 32 weights = its rows' 128 columns of the stage. */
    if constexpr (INT4) {
      const int uw = warp - 7;
      const int row0 = (uw % C::STAGE_WARPS) * 8 * C::UNITS + (lane >> 2), j = lane & 3;
      const int set = uw / C::STAGE_WARPS; /* this warp's stages: set, set + SETS, ... */
      const int total = my_tiles * k_blocks;
      int kb = set, tile = first_tile;
      float2 dd[C::UNITS]; /* (d, dmin) of the rows row0 + 8 u; zeros past the last row */
      auto row_scales = [&]() {
#pragma unroll
        for (int u = 0; u < C::UNITS; ++u) {
          const int grow = (tile / a.m_tiles) * BN + rank * C::BH + row0 + 8 * u;
          dd[u] = grow < g.out_f ? __half22float2(__ldg(g.sb + grow)) : make_float2(0.f, 0.f);
        }
      };
      if (set < total) {
        while (kb >= k_blocks) kb -= k_blocks, tile += tile_step;
        row_scales();
      }
      bool ok = true;
      for (int it = set; ok && it < total; it += C::SETS) {
        const int st = it % NSTAGE, sl = it % C::NSLOT;
        ok = mbar_wait(bar(P_FULL + sl), (it / C::NSLOT) & 1, a.err_word, 0x908u) &&
             (it < NSTAGE || mbar_wait(bar(EMPTY + st), ((it / NSTAGE) - 1) & 1, a.err_word, 0x905u));
        if (!__all_sync(0xffffffffu, ok)) break;
        const uint8_t *slot = smem + C::OFF_PACK + sl * C::SLOT_BYTES;
#pragma unroll
        for (int u = 0; u < C::UNITS; ++u)
          unpack_group<C::BH>(slot, smem + st * C::STAGE_BYTES + C::A_BYTES, row0 + 8 * u, j, dd[u]);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(FULL + st));
          mbar_arrive(bar(P_EMPTY + sl));
        }
        kb += C::SETS;
        if (kb >= k_blocks && it + C::SETS < total) {
          while (kb >= k_blocks) kb -= k_blocks, tile += tile_step;
          row_scales();
        }
      }
    }
  } else if (warp == 4) {
    /* ------------------------------------------------ MMA issuer, in the leader */
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc(256, BN, 0);
      int it = 0, local = 0;
      bool ok = true;
      for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_step, ++local) {
        const int buf = local & 1;
        /* both CTAs' epilogues of the tile two back have emptied this accumulator */
        if (local >= 2 &&
            !mbar_wait_cluster(bar(ACC_EMPTY + buf), ((local >> 1) - 1) & 1, a.err_word, 0x902u)) break;
        tc_fence_after_sync();
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int st = it % NSTAGE;
          if (!mbar_wait_cluster(bar(FULL + st), (it / NSTAGE) & 1, a.err_word, 0x903u)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t a_lo = umma_desc_lo(sbase + st * C::STAGE_BYTES, 16);
          const uint32_t b_lo = umma_desc_lo(sbase + st * C::STAGE_BYTES + C::A_BYTES, 16);
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < C::BK / 16; ++ks) {
              const uint32_t a_off = ((ks >> 2) * C::A_SLAB + (ks & 3) * 32) >> 4;
              const uint32_t b_off = ((ks >> 2) * C::B_SLAB + (ks & 3) * 32) >> 4;
              pair_umma_ss_f16(tmem + buf * BN, a_lo + a_off, b_lo + b_off, kDescHi, idesc,
                               (kb > 0 || ks > 0) ? 1u : 0u);
            }
            pair_umma_commit(bar(EMPTY + st));
            if (kb == k_blocks - 1) pair_umma_commit(bar(ACC_FULL + buf));
          }
          __syncwarp();
        }
      }
    } else if (lane == 0) {
      /* ------------ the second CTA: passes its accumulators and weight tiles on, in the order in
       * which the leader waits for them */
      int it = 0, local = 0;
      bool ok = true;
      for (int tile = first_tile; ok && tile < n_tiles_total; tile += tile_step, ++local) {
        const int buf = local & 1;
        if (local >= 2) {
          if (!mbar_wait(bar(ACC_EMPTY + buf), ((local >> 1) - 1) & 1, a.err_word, 0x90Au)) break;
          tc_fence_after_sync();
          tc_fence_before_sync();
          tell_leader(mailbox, mailbox, bar(ACC_EMPTY + buf));
        }
        if constexpr (INT4) {
          for (int kb = 0; kb < k_blocks; ++kb, ++it) {
            const int st = it % NSTAGE;
            if (!mbar_wait(bar(FULL + st), (it / NSTAGE) & 1, a.err_word, 0x90Bu)) { ok = false; break; }
            tell_leader(mailbox, sbase + st * C::STAGE_BYTES + C::A_BYTES, bar(FULL + st));
          }
        }
      }
    }
  } else {
    /* ------------------------------ epilogue: warp w holds token rows 32 w .. 32 w + 31 */
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const bool vec = (g.out_f & 3) == 0;
    uint8_t *stage = smem + C::OFF_EPI + warp * C::EPI_WARP;
    int local = 0;
    for (int tile = first_tile; tile < n_tiles_total; tile += tile_step, ++local) {
      const int buf = local & 1;
      const int m0 = (tile % a.m_tiles) * 256 + rank * 128, n0 = (tile / a.m_tiles) * BN;
      if (!mbar_wait_idle(bar(ACC_FULL + buf), (local >> 1) & 1, a.err_word, 0x904u)) break;
      tc_fence_after_sync();
      const uint32_t acc = tmem + lane_base + buf * BN;
      if constexpr (ROPE) {
        /* the token's sequence, cache position (clamped, never trusted) and cache row */
        const int row = m0 + warp * 32 + lane;
        const bool valid = row < g.n;
        const int sq = valid ? row / g.n_per_seq : 0;
        int pos = valid ? g.seq_pos0[sq] + (row - sq * g.n_per_seq) : 0;
        pos = pos < 0 ? 0 : pos;
        pos = pos < g.max_seq - 1 ? pos : g.max_seq - 1;
        const int tpos = pos < g.table_len - 1 ? pos : g.table_len - 1;
        const long long kv_row =
            (static_cast<long long>(sq) * g.n_kv * g.max_seq + pos) * static_cast<long long>(g.hd);
        if (g.hd == 128) {
#pragma unroll 1
          for (int h = 0; h < BN / 128; ++h) {
            const int head = n0 / 128 + h;
            rope_head_epilogue<128>(g, acc + h * 128, head, tpos, kv_row, row,
                                    valid && head * 128 < g.out_f);
          }
        } else {
#pragma unroll 1
          for (int h = 0; h < BN / 64; ++h) {
            const int head = n0 / 64 + h;
            rope_head_epilogue<64>(g, acc + h * 64, head, tpos, kv_row, row,
                                   valid && head * 64 < g.out_f);
          }
        }
      } else {
        /* EC columns at a time through shared memory: a thread's row of the accumulator goes
         * in, runs of EC floats of several rows at once come out */
        constexpr int EC = C::EC, Q = EC / 4; /* Q lanes per row, Q passes of 32 / Q rows */
        auto at = [](int row, int chunk) { /* 16-byte chunk of a row, bank conflicts spread */
          return EC == 32 ? swz128(row, chunk) : static_cast<uint32_t>(row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4));
        };
        const int row0 = m0 + warp * 32;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += EC) {
          const int col0 = n0 + c0;
          if (row0 >= g.n || col0 >= g.out_f) break;
          uint32_t v[EC];
          if constexpr (EC == 32) tmem_ld_32x32(acc + c0, v);
          else tmem_ld_32x16(acc + c0, v);
          if (vec && col0 + EC <= g.out_f) {
            const int chunk = lane % Q, sub = lane / Q; /* columns 4 chunk .. + 3 of rows sub + 32 / Q i */
            float *dst = g.y + static_cast<long long>(row0 + sub) * g.out_f + col0 + 4 * chunk;
            const long long step = static_cast<long long>(32 / Q) * g.out_f;
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (g.bias) {
              const uint2 h = __ldg(reinterpret_cast<const uint2 *>(g.bias + col0 + 4 * chunk));
              const float2 b0 = __half22float2(*reinterpret_cast<const __half2 *>(&h.x));
              const float2 b1 = __half22float2(*reinterpret_cast<const __half2 *>(&h.y));
              b = make_float4(b0.x, b0.y, b1.x, b1.y);
            }
            tmem_ld_wait();
            __syncwarp(); /* the columns before have left the staging rows */
#pragma unroll
            for (int e = 0; e < Q; ++e)
              *reinterpret_cast<uint4 *>(stage + at(lane, e)) =
                  make_uint4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < Q; ++i) {
              float4 o = *reinterpret_cast<const float4 *>(stage + at(sub + 32 / Q * i, chunk));
              o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
              if (row0 + sub + 32 / Q * i < g.n) {
                if (g.accum) add_v4(dst + i * step, o);
                else *reinterpret_cast<float4 *>(dst + i * step) = o;
              }
            }
          } else {
            tmem_ld_wait();
            const int row = row0 + lane;
            float *yrow = g.y + static_cast<long long>(row) * g.out_f;
#pragma unroll
            for (int e = 0; e < EC; ++e) {
              if (row < g.n && col0 + e < g.out_f) {
                float o = __uint_as_float(v[e]);
                if (g.bias) o += __half2float(g.bias[col0 + e]);
                if (g.accum) o += yrow[col0 + e];
                yrow[col0 + e] = o;
              }
            }
            __syncwarp();
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (rank == 0 && warp == 0) mbar_arrive_expect_tx(bar(ACC_EMPTY + buf), kMessage);
        else mbar_arrive(bar(ACC_EMPTY + buf));
      }
    }
    grid_launch_dependents();
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_sync(); /* nothing of the other CTA arrives here any more */
  if (warp == 4) {
    tc_fence_after_sync();
    pair_tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

template <int BN, bool ROPE, bool INT4>
wst_status_t launch_tile(const PairGemm &g, int sm_count) {
  using C = PairCfg<BN, INT4>;
  auto kern = gemm_pair_kernel<BN, ROPE, INT4>;
  CUtensorMap xmap, wmap;
  wst_status_t st = rows_map(&xmap, g.x, g.in_f, g.n, C::BM);
  if (st != WST_OK) return st;
  /* packed rows are in_f / 2 bytes: in_f / 4 elements of the maps' two bytes */
  st = INT4 ? packed_map(&wmap, g.qw, g.in_f / 4, g.out_f, C::BH)
            : rows_map(&wmap, g.w, g.in_f, g.out_f, C::BH);
  if (st != WST_OK) return st;
  PairArgs a{};
  a.g = g;
  a.m_tiles = (g.n + 255) / 256;
  a.n_tiles = (g.out_f + BN - 1) / BN;
  a.err_word = device_error_word();
  if (!a.err_word) return WST_ERR_CUDA;

  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(pair_threads(INT4));
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = current_stream();
  /* clusters that the device holds at once: an odd number of SMs in a GPC leaves one out */
  static thread_local int configured_dev = -1, clusters = 0;
  int dev = 0;
  WST_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    WST_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    cfg.gridDim = dim3(2);
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      clusters = sm_count / 2;
    }
    if (clusters > sm_count / 2) clusters = sm_count / 2;
    configured_dev = dev;
  }
  const long long tiles = static_cast<long long>(a.m_tiles) * a.n_tiles;
  cfg.gridDim = dim3(2u * static_cast<unsigned>(tiles < clusters ? tiles : clusters));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, xmap, wmap, a);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess)
    return fail(WST_ERR_CUDA, "%s (launch): %s (%s)", g.name, cudaGetErrorString(e), cudaGetErrorName(e));
  return WST_OK;
}

template <bool ROPE, bool INT4>
wst_status_t launch_form(const PairGemm &g, int sm_count) {
  /* The feature tile by waves x clocks of 64 columns of K (measured, K = 4096, one to seven
   * waves): 256 features are bound by the tensor pipe, the narrower ones by what a tile brings
   * in from L2, the packed ones by unpacking too.  Narrow tiles win where 256 leave clusters
   * idle: 256 tokens of 4096 -> 4096 take 27, 18 and 16 us with 256, 128 and 64 features, 2048
   * tokens 53, 59 and 82. */
  static const int tile[3] = {256, 128, 64};
  static const int clocks[2][3] = {{530, 290, 240}, {690, 440, 270}};
  const long long pairs = sm_count / 2, m_tiles = (g.n + 255) / 256;
  int best = 0;
  long long best_cost = -1;

  for (int i = 0; i < 3; ++i) {
    if (ROPE && tile[i] < g.hd) continue; /* whole heads */
    const long long tiles = m_tiles * ((g.out_f + tile[i] - 1) / tile[i]);
    const long long cost = (tiles + pairs - 1) / pairs * clocks[INT4][i];
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = tile[i]; }
  }
  switch (best) {
    case 256: return launch_tile<256, ROPE, INT4>(g, sm_count);
    case 128: return launch_tile<128, ROPE, INT4>(g, sm_count);
    default: return launch_tile<64, ROPE, INT4>(g, sm_count);
  }
}

}  // namespace

wst_status_t launch_gemm_pair(const PairGemm &g, int sm_count) {
  const bool int4 = g.qw != nullptr;
  if (g.q_out) return int4 ? launch_form<true, true>(g, sm_count) : launch_form<true, false>(g, sm_count);
  return int4 ? launch_form<false, true>(g, sm_count) : launch_form<false, false>(g, sm_count);
}

}  // namespace wst
