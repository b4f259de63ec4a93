/* wst_gemm_int4_hier for a handful of tokens (decode-side chunks, speculative
 * verification of one sequence): y[j][r] (+)= sum_c x[j][c] * w[r][c] + bias[r] with the
 * weights in the hierarchical int4 format (cuda/hier.cuh:8-13 of the engine,
 * cuda/chunk_gemm.cu:61-176).
 *
 * What bounds it: the packed weights are read once (8.8 MB for 3584 -> 4608: 1.4 us of
 * HBM), and unpacking them costs about three instructions per weight (the same again over
 * 148 SMs).  With operand tiles in shared memory a handful of tokens pay a barrier round trip
 * per k-block for nothing: no token shares another's.  Here nothing goes through shared memory
 * and nothing waits for another warp before the last step:
 *
 *   - a CTA owns 16 * MT weight rows, its warps take interleaved 128-column slabs of K, so
 *     every SM pulls on HBM at once and a warp walks two to four slabs;
 *   - the order of K inside a slab is free as long as both operands agree on it: lane t of
 *     a quad takes the slab's t-th group of 32 weights of its rows -- one 16-byte load, the
 *     quad's four loads one 64-byte run -- unpacks it in registers and feeds
 *     mma.sync m16n8k16 steps of four weights per lane; its x fragments are the same
 *     group's columns, 16 bytes per step pair straight from L2;
 *   - the packed words a CTA will need are prefetched towards L2 before the grid dependency
 *     resolves (a prefetch has no architectural effect, whatever the launch ahead writes).
 * Measured, a launch in a graph, 5 tokens of 3584 -> 4608: 6.1 us; operand tiles and
 * tensor memory took 38.
 *
 * Per weight the arithmetic is that of int4_tile.cuh: w = q (d ls) - dmin lm in one fp32 fma,
 * rounded to fp16 once; products and sums fp32. */

#include "gemm_int4_few.cuh"
#include "int4_tile.cuh"
#include "wst_ptx.cuh"

namespace wst {
namespace {

using namespace ptx;

struct FewArgs {
  const uint4 *qw;    /* [out_f][in_f / 32] words of 32 nibbles */
  const uint8_t *si;  /* [out_f][in_f / 32]: ls | lm << 4 */
  const __half2 *sb;  /* [out_f]: (d, dmin) */
  const __half *x;    /* [n][in_f] */
  const __half *bias; /* [out_f] or null */
  float *y;           /* [n][out_f] */
  int in_f, out_f, n, accum;
};

/* One slab of a lane: its group of each of its 2 * MT rows. */
template <int MT>
struct Slab {
  uint4 w[2 * MT];
  uint8_t idx[2 * MT];
};

/* WARPS on a CTA: sixteen on an SM in one or two CTAs */
template <int MT, int NT, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS) gemm_int4_few_kernel(const FewArgs a) {
  constexpr int R = 16 * MT, RI = 2 * MT;
  constexpr int LD = R + 4; /* a warp's stores fall into 32 different banks */
  __shared__ float red[WARPS][8 * NT][LD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int row0 = blockIdx.x * R;
  const int groups = a.in_f / 32;
  const int slabs = (groups + 3) / 4;

  grid_launch_dependents();
  int row[RI]; /* past the last row: the last one again, its sums are not stored */
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = row0 + 8 * i + g;
    row[i] = r < a.out_f ? r : a.out_f - 1;
  }
  for (int s = warp; s < slabs; s += WARPS)
    if (t == 0)
#pragma unroll
      for (int i = 0; i < RI; ++i)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.qw + static_cast<size_t>(row[i]) * groups + 4 * s));
  grid_dependency_wait();

  float2 dd[RI];
#pragma unroll
  for (int i = 0; i < RI; ++i) dd[i] = __half22float2(__ldg(a.sb + row[i]));
  const __half *xrow[NT]; /* past the last token: the last one again */
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int tok = 8 * nt + g;
    xrow[nt] = a.x + static_cast<size_t>(tok < a.n ? tok : a.n - 1) * a.in_f;
  }

  float acc[MT][NT][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[mt][nt][c] = 0.f;

  auto fetch = [&](int s, Slab<MT> &d) {
    const int grp = 4 * s + t;
    const bool in = grp < groups; /* past the last group: zero weights times zeros */
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const size_t at = static_cast<size_t>(row[i]) * groups + grp;
      d.w[i] = in ? __ldg(a.qw + at) : make_uint4(0u, 0u, 0u, 0u);
      d.idx[i] = in ? __ldg(a.si + at) : 0;
    }
  };
  /* the x columns under word `wi` of slab s, eight per lane and token tile */
  auto fetch_x = [&](int s, int wi, uint4 (&d)[NT]) {
    const int grp = 4 * s + t;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      d[nt] = grp < groups ? reinterpret_cast<const uint4 *>(xrow[nt] + grp * 32)[wi]
                           : make_uint4(0u, 0u, 0u, 0u);
  };
  /* word `wi` of the rows' groups: unpacked, multiplied */
  auto multiply = [&](const Slab<MT> &d, const GroupScale (&sc)[RI], int wi, const uint4 (&x)[NT]) {
    uint32_t o[RI][4]; /* the word's weights 2i, 2i + 1 as fp16 */
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const uint32_t word = wi == 0 ? d.w[i].x : wi == 1 ? d.w[i].y : wi == 2 ? d.w[i].z : d.w[i].w;
      unpack_word(word, sc[i], o[i]);
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const uint32_t a0[4] = {o[2 * mt][0], o[2 * mt + 1][0], o[2 * mt][1], o[2 * mt + 1][1]};
      const uint32_t a1[4] = {o[2 * mt][2], o[2 * mt + 1][2], o[2 * mt][3], o[2 * mt + 1][3]};
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        mma_16816(acc[mt][nt], a0, x[nt].x, x[nt].y);
        mma_16816(acc[mt][nt], a1, x[nt].z, x[nt].w);
      }
    }
  };

  /* the next slab's words and the next RING words' x columns are on their way while one
   * word is multiplied: as many as 32 registers hold */
  constexpr int RING = 8 / NT;
  Slab<MT> buf[2];
  uint4 xb[RING][NT];
  if (warp < slabs) fetch(warp, buf[0]);
#pragma unroll
  for (int p = 0; p < RING; ++p) fetch_x(warp + (p >> 2) * WARPS, p & 3, xb[p]);
  for (int s = warp; s < slabs; s += 2 * WARPS) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (s + h * WARPS >= slabs) break;
      fetch(s + (h + 1) * WARPS, buf[h ^ 1]);
      const Slab<MT> &d = buf[h];
      GroupScale sc[RI];
#pragma unroll
      for (int i = 0; i < RI; ++i) sc[i] = group_scale(dd[i], d.idx[i]);
#pragma unroll
      for (int wi = 0; wi < 4; ++wi) {
        const int p = 4 * h + wi, next = p + RING;
        multiply(d, sc, wi, xb[p % RING]);
        fetch_x(s + (next >> 2) * WARPS, next & 3, xb[p % RING]);
      }
    }
  }

#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        red[warp][8 * nt + 2 * t + (c & 1)][16 * mt + g + 8 * (c >> 1)] = acc[mt][nt][c];
  __syncthreads();
  for (int i = threadIdx.x; i < 8 * NT * R; i += 32 * WARPS) {
    const int tok = i / R, r = i % R;
    if (tok >= a.n || row0 + r >= a.out_f) continue;
    float sum = a.bias ? __half2float(a.bias[row0 + r]) : 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) sum += red[w][tok][r];
    float *dst = a.y + static_cast<size_t>(tok) * a.out_f + row0 + r;
    *dst = a.accum ? *dst + sum : sum;
  }
}

template <int MT, int NT, int WARPS>
wst_status_t launch_few(const FewArgs &a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((a.out_f + 16 * MT - 1) / (16 * MT)));
  cfg.blockDim = dim3(32 * WARPS);
  cfg.stream = current_stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_int4_few_kernel<MT, NT, WARPS>, a);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail("wst_gemm_int4_hier (launch)", e);
  return WST_OK;
}

}  // namespace

wst_status_t launch_gemm_int4_few(const void *qw, const void *si, const void *sb, const void *x,
                                  const void *bias, void *y, int in_f, int out_f, int n, int accum,
                                  int sm_count) {
  FewArgs a{};
  a.qw = static_cast<const uint4 *>(qw);
  a.si = static_cast<const uint8_t *>(si);
  a.sb = static_cast<const __half2 *>(sb);
  a.x = static_cast<const __half *>(x);
  a.bias = static_cast<const __half *>(bias);
  a.y = static_cast<float *>(y);
  a.in_f = in_f;
  a.out_f = out_f;
  a.n = n;
  a.accum = accum;
  /* Sixteen warps per SM that each walk little of K: with eight (32 rows per CTA, one CTA per SM)
   * 5 tokens of 3584 -> 4608 took 9.7 us, with two CTAs of 16 rows 6.1; 4096 -> 6144 11.3 and
   * 9.9.  From 9 tokens on 32 rows in one CTA of sixteen warps halve the x traffic where one
   * wave takes them all: 16 tokens 12.2 -> 7.4 us, 8.1 with 16 rows; 4096 -> 6144 15.0 and 13.9
   * before.  Few rows: sixteen warps on one CTA of 16 (896 -> 1152 2.4 -> 2.0). */
  const bool narrow = static_cast<long long>(out_f) < 16ll * sm_count;
  const bool one_wave = static_cast<long long>(out_f) <= 32ll * sm_count;
  if (n <= 8) return narrow ? launch_few<1, 1, 16>(a) : launch_few<1, 1, 8>(a);
  if (n <= 16)
    return narrow ? launch_few<1, 2, 16>(a) : one_wave ? launch_few<2, 2, 16>(a) : launch_few<2, 2, 8>(a);
  return narrow ? launch_few<1, 4, 8>(a) : launch_few<2, 4, 8>(a);
}

}  // namespace wst
