/* int4-hier projections of 17 to 128 tokens:
 *
 *     y[j][r] (+)= sum_c x[j][c] * w[r][c] + bias[r]        j < n tokens, r < out_f
 *
 * The launch is a stream of packed weights (8.8 MB for 3584 -> 4608, 1.4 us of HBM), and what
 * bounds it is unpacking them: every SM has to have its share, once, and start early.  A CTA
 * owns 128 (or 64) weight rows -- the M side of tcgen05.mma, the tokens are N -- and a slice
 * of K; the CTAs of a cluster split K, lay their accumulators down in shared memory and each
 * adds up a share of the tokens from all of them (DSMEM), always in the same order.  The
 * packed words of up to eight stages are on their way at once; they are asked towards L2
 * before the grid dependency resolves (a prefetch has no architectural effect, whatever the
 * launch ahead writes).  80 tokens, a launch in a graph: 3584 -> 4608 35 us with 72 CTAs that
 * walked all of K, 14 now; 4096 -> 4096 33 and 13.
 *
 * Products are exact in fp32 and accumulated in fp32. */

#include "gemm_pair.cuh"
#include "int4_tile.cuh"
#include "tensor_map.cuh"
#include "wst_ptx.cuh"

namespace wst {
namespace {

using namespace ptx;

constexpr int kNarrowUnpackWarps = 16;
constexpr int kMaxCluster = 8;


/* ROWS = 64 or 128 weight rows per CTA, 128 columns of K per stage.  The MMA is always M = 128:
 * with 64 rows it reads whatever follows them in shared memory, and those accumulator rows are
 * not used. */
template <int ROWS>
struct NarrowCfg {
  static constexpr int KS = 2, BK = 64 * KS;
  static constexpr int A_SLAB = ROWS * 128, A_BYTES = KS * A_SLAB;
  static constexpr int MAX_STAGES = 3, MAX_SLOTS = 8;
  static constexpr int SLOT_BYTES = slot_bytes(ROWS);
  static constexpr int UNITS = ROWS == 128 ? 2 : 1;
  static constexpr int STAGE_WARPS = ROWS / (8 * UNITS), SETS = kNarrowUnpackWarps / STAGE_WARPS;
  static constexpr int NBAR = 2 * MAX_STAGES + 1 + 2 * MAX_SLOTS;
  static constexpr int THREADS = 32 * (7 + kNarrowUnpackWarps);
  static constexpr int SMEM_BYTES = 226 * 1024; /* one CTA per SM */
  /* for stages and slots; beyond the last stage's 64 rows the MMA may read up to 128 of them */
  static constexpr int ROOM = SMEM_BYTES - NBAR * 8 - 16 - 1024 - (ROWS < 128 ? 8192 : 0);
  static_assert(SETS >= 1 && ROOM >= 2 * (A_BYTES + KS * 128 * 128) + 3 * SLOT_BYTES, "does not fit");
};

struct NarrowArgs {
  PairGemm g;
  int cols, stages;      /* tokens rounded up to 16: N of the MMA; ring depth */
  int slots;             /* of packed words */
  int k_blocks, kb_cta;  /* stages' worth of K in all and per CTA of a cluster */
  unsigned int *err_word;
};

__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap *map, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
template <int ROWS>
__global__ void __launch_bounds__(NarrowCfg<ROWS>::THREADS, 1)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                   const __grid_constant__ NarrowArgs a) {
  using C = NarrowCfg<ROWS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sbase = smem_u32(smem);
  const PairGemm &g = a.g;
  const int b_slab = a.cols * 128, stage_bytes = C::A_BYTES + C::KS * b_slab;
  const int nstage = a.stages;
  const int off_pack = nstage * stage_bytes;
  const int nslot = a.slots;
  const int off_bar = off_pack + nslot * C::SLOT_BYTES;
  const uint32_t bar0 = sbase + off_bar;
  auto bar = [bar0](int i) { return bar0 + 8u * i; };
  constexpr int FULL = 0, EMPTY = C::MAX_STAGES, ACC_FULL = 2 * C::MAX_STAGES;
  constexpr int P_FULL = ACC_FULL + 1, P_EMPTY = P_FULL + C::MAX_SLOTS;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + off_bar + C::NBAR * 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  int csize;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
  const int rank = static_cast<int>(cluster_rank());
  const int row0 = static_cast<int>(blockIdx.x / csize) * ROWS;
  const int kb0 = rank * a.kb_cta;
  const int nkb = min(a.kb_cta, a.k_blocks - kb0); /* the last CTA of a cluster may have fewer */

  if (threadIdx.x == 0) {
    for (int i = 0; i < nstage; ++i) {
      mbar_init(bar(FULL + i), 1 + C::STAGE_WARPS);
      mbar_init(bar(EMPTY + i), 1);
    }
    mbar_init(bar(ACC_FULL), 1);
    for (int i = 0; i < nslot; ++i) {
      mbar_init(bar(P_FULL + i), 1 + 32);
      mbar_init(bar(P_EMPTY + i), C::STAGE_WARPS);
    }
    mbar_init_fence();
    tma_prefetch_desc(&xmap);
    tma_prefetch_desc(&wmap);
  }
  __syncwarp();
  if (warp == 4) {
    tmem_alloc(smem_u32(tmem_slot), 128);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  grid_launch_dependents();
  if (warp == 5 && lane == 0) /* this CTA's share of the packed words towards L2 */
    for (int i = 0; i < nkb; ++i) tma_prefetch_3d(&wmap, (kb0 + i) * (C::BK / 4), row0, 0);

  grid_dependency_wait();

  if (warp == 5) {
    /* ------------------------------------------------------ TMA producer */
    if (lane == 0) {
      for (int i = 0; i < nkb; ++i) {
        const int st = i % nstage, k0 = (kb0 + i) * C::BK;
        if (i >= nstage && !mbar_wait(bar(EMPTY + st), ((i / nstage) - 1) & 1, a.err_word, 0x801u)) break;
        mbar_arrive_expect_tx(bar(FULL + st), C::KS * b_slab);
        const uint32_t dst = sbase + st * stage_bytes;
#pragma unroll
        for (int s = 0; s < C::KS; ++s)
          tma_load_3d(dst + C::A_BYTES + s * b_slab, &xmap, bar(FULL + st), k0 + 64 * s, 0, 0);
      }
    }
  } else if (warp == 4) {
    /* -------------------------------------------------------- MMA issuer */
    const uint32_t idesc = umma_idesc(128, 0, 0) | (static_cast<uint32_t>(a.cols >> 3) << 17);
    for (int i = 0; i < nkb; ++i) {
      const int st = i % nstage;
      if (!mbar_wait(bar(FULL + st), (i / nstage) & 1, a.err_word, 0x803u)) break;
      tc_fence_after_sync();
      const uint32_t a_lo = umma_desc_lo(sbase + st * stage_bytes, 16);
      const uint32_t b_lo = umma_desc_lo(sbase + st * stage_bytes + C::A_BYTES, 16);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < C::BK / 16; ++ks) {
          const uint32_t a_off = ((ks >> 2) * C::A_SLAB + (ks & 3) * 32) >> 4;
          const uint32_t b_off = ((ks >> 2) * b_slab + (ks & 3) * 32) >> 4;
          umma_ss_f16_lohi(tmem, a_lo + a_off, b_lo + b_off, kDescHi, idesc, (i > 0 || ks > 0) ? 1u : 0u);
        }
        umma_commit(bar(EMPTY + st));
        if (i == nkb - 1) umma_commit(bar(ACC_FULL));
      }
      __syncwarp();
    }
  } else if (warp == 6) {
    /* ------------------------------------------ packed words and scale bytes */
    const PackedRows<ROWS> packed(&wmap, g.si, g.in_f / 32, g.out_f, row0, lane);
    for (int i = 0; i < nkb; ++i) {
      const int sl = i % nslot;
      if (i >= nslot) {
        const bool free = mbar_wait(bar(P_EMPTY + sl), ((i / nslot) - 1) & 1, a.err_word, 0x807u);
        if (!__all_sync(0xffffffffu, free)) break;
      }
      packed.fetch(sbase + off_pack + sl * C::SLOT_BYTES, bar(P_FULL + sl), kb0 + i, lane);
    }
    fetch_packed_drain();
  } else if (warp > 6) {
    /* ------------------------------------------ unpacked into the weight side of the stage */
    const int uw = warp - 7;
    const int r0 = (uw % C::STAGE_WARPS) * 8 * C::UNITS + (lane >> 2), j = lane & 3;
    float2 dd[C::UNITS]; /* (d, dmin) of the rows r0 + 8 u; zeros past the last row */
#pragma unroll
    for (int u = 0; u < C::UNITS; ++u) {
      const int row = row0 + r0 + 8 * u;
      dd[u] = row < g.out_f ? __half22float2(__ldg(g.sb + row)) : make_float2(0.f, 0.f);
    }
    for (int i = uw / C::STAGE_WARPS; i < nkb; i += C::SETS) {
      const int st = i % nstage, sl = i % nslot;
      const bool ok =
          mbar_wait(bar(P_FULL + sl), (i / nslot) & 1, a.err_word, 0x808u) &&
          (i < nstage || mbar_wait(bar(EMPTY + st), ((i / nstage) - 1) & 1, a.err_word, 0x805u));
      if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
      for (int u = 0; u < C::UNITS; ++u)
        unpack_group<ROWS>(smem + off_pack + sl * C::SLOT_BYTES, smem + st * stage_bytes, r0 + 8 * u, j,
                           dd[u]);
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar(FULL + st));
        mbar_arrive(bar(P_EMPTY + sl));
      }
    }
  } else {
    /* ---- accumulator -> shared memory, [token][rows] floats over the ring, which is idle
     * once the last MMA is done: thread r of the four warps holds weight row r */
    const uint32_t acc = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    float *part = reinterpret_cast<float *>(smem) + warp * 32 + lane;
    const bool used = warp * 32 + lane < ROWS;
    const bool ok = mbar_wait(bar(ACC_FULL), 0, a.err_word, 0x804u);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after_sync();
#pragma unroll 1
      for (int c0 = 0; c0 < a.cols; c0 += 16) {
        uint32_t v[16];
        tmem_ld_32x16(acc + c0, v);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (used) part[(c0 + e) * ROWS] = __uint_as_float(v[e]);
        __syncwarp();
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  cluster_sync(); /* every CTA's part is there */
  {
    /* this CTA's share of the tokens, a warp per token, four weight rows per lane */
    const int per = (g.n + csize - 1) / csize, tok1 = min(g.n, (rank + 1) * per);
    const int r = row0 + 4 * lane, end = min(g.out_f, row0 + ROWS);
    const bool vec = (g.out_f & 3) == 0;
    uint32_t from[kMaxCluster];
#pragma unroll
    for (int p = 0; p < kMaxCluster; ++p) from[p] = in_cta(sbase + 16 * lane, p < csize ? p : 0);
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (g.bias && r + e < end) bias[e] = __half2float(g.bias[r + e]);
    for (int tok = rank * per + warp; tok < tok1 && r < end; tok += C::THREADS / 32) {
      float *dst = g.y + static_cast<long long>(tok) * g.out_f + r;
      float4 old = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g.accum && vec) old = *reinterpret_cast<const float4 *>(dst);
      float4 part[kMaxCluster];
#pragma unroll
      for (int p = 0; p < kMaxCluster; ++p)
        if (p < csize) part[p] = ld_cluster_f32x4(from[p] + tok * (ROWS * 4));
      float4 o = part[0];
#pragma unroll
      for (int p = 1; p < kMaxCluster; ++p)
        if (p < csize) {
          o.x += part[p].x; o.y += part[p].y; o.z += part[p].z; o.w += part[p].w;
        }
      o.x += bias[0]; o.y += bias[1]; o.z += bias[2]; o.w += bias[3];
      if (vec) {
        if (g.accum) { o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w; }
        *reinterpret_cast<float4 *>(dst) = o;
      } else {
        const float f[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (r + e < end) dst[e] = g.accum ? dst[e] + f[e] : f[e];
      }
    }
  }
  cluster_sync(); /* nobody reads this CTA's part any more */
  if (warp == 4) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 128);
  }
}

/* Clusters of `size` CTAs that the device holds at once: a cluster does not cross a GPC, so 33 of
 * four and not 37.  0 = not known. */
template <int ROWS>
int resident_clusters(int size) {
  using C = NarrowCfg<ROWS>;
  static thread_local int dev_of = -1, known[kMaxCluster + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev_of != dev) {
    if (cudaFuncSetAttribute(gemm_narrow_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             C::SMEM_BYTES) != cudaSuccess)
      return 0;
    for (int s = 1; s <= kMaxCluster; ++s) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(static_cast<unsigned>(s));
      cfg.blockDim = dim3(C::THREADS);
      cfg.dynamicSmemBytes = C::SMEM_BYTES;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = static_cast<unsigned>(s);
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&known[s], gemm_narrow_kernel<ROWS>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        known[s] = 0;
      }
    }
    dev_of = dev;
  }
  return known[size];
}

/* How a projection is cut: rows per CTA, CTAs per cluster. */
struct Cut {
  int rows = 128, split = 1;
  long long cost = -1;
};

/* Waves of clusters x (what a launch costs anyway + the stages of a CTA), in 10 ns: fitted to
 * 24, 80 and 128 tokens of five shapes at every cut.  Where one more CTA per cluster starts a
 * second wave it is lost: 48 tiles of 6144 rows take 18 us with two and 27 with three. */
template <int ROWS>
Cut best_cut(int k_blocks, int out_f) {
  const long long tiles = (static_cast<long long>(out_f) + ROWS - 1) / ROWS;
  Cut best;
  for (int s = 1; s <= kMaxCluster && s <= k_blocks; ++s) {
    const int hold = resident_clusters<ROWS>(s);
    if (hold < 1) continue;
    const long long waves = (tiles + hold - 1) / hold;
    const long long cost = waves * (600 + 12 * s + (k_blocks + s - 1) / s * (ROWS == 128 ? 73 : 60));
    if (best.cost < 0 || cost < best.cost) best = Cut{ROWS, s, cost};
  }
  return best;
}

template <int ROWS>
wst_status_t launch_cut(const PairGemm &g, int split) {
  using C = NarrowCfg<ROWS>;
  NarrowArgs a{};
  a.g = g;
  a.cols = (g.n + 15) / 16 * 16;
  a.k_blocks = (g.in_f + C::BK - 1) / C::BK;
  a.kb_cta = (a.k_blocks + split - 1) / split;
  split = (a.k_blocks + a.kb_cta - 1) / a.kb_cta; /* no CTA without a part of K */
  a.err_word = device_error_word();
  if (!a.err_word) return WST_ERR_CUDA;
  /* three stages if they fit beside as many slots, else two; the rest holds packed words */
  const int stage_bytes = C::A_BYTES + C::KS * a.cols * 128;
  a.stages = 3 * (stage_bytes + C::SLOT_BYTES) <= C::ROOM ? 3 : 2;
  a.slots = (C::ROOM - a.stages * stage_bytes) / C::SLOT_BYTES;
  if (a.slots > C::MAX_SLOTS) a.slots = C::MAX_SLOTS;
  CUtensorMap xmap, wmap;
  wst_status_t st = rows_map(&xmap, g.x, g.in_f, g.n, a.cols);
  if (st != WST_OK) return st;
  /* packed rows are in_f / 2 bytes: in_f / 4 elements of the maps' two bytes */
  st = packed_map(&wmap, g.qw, g.in_f / 4, g.out_f, ROWS);
  if (st != WST_OK) return st;
  const long long ctas = (static_cast<long long>(g.out_f) + ROWS - 1) / ROWS * split;
  if (ctas > 0x7fffffffLL) return fail(WST_ERR_SHAPE, "%s: too many output features", g.name);

  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = current_stream();
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(split);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_narrow_kernel<ROWS>, xmap, wmap, a);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess)
    return fail(WST_ERR_CUDA, "%s (launch): %s (%s)", g.name, cudaGetErrorString(e), cudaGetErrorName(e));
  return WST_OK;
}

}  // namespace

wst_status_t launch_gemm_narrow(const PairGemm &g) {
  const int k_blocks = (g.in_f + 127) / 128;
  const Cut wide = best_cut<128>(k_blocks, g.out_f), slim = best_cut<64>(k_blocks, g.out_f);
  if (wide.cost < 0 && slim.cost < 0)
    return fail(WST_ERR_CUDA, "%s: the device holds no cluster of this kernel", g.name);
  return wide.cost < 0 || (slim.cost >= 0 && slim.cost < wide.cost) ? launch_cut<64>(g, slim.split)
                                                                     : launch_cut<128>(g, wide.split);
}

}  // namespace wst
