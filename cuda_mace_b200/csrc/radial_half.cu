// Hidden layers of the radial perceptrons with their derivative (what radial_tangent.cu computes), float32, on the
// tensor cores' fp16 rate: 3-term split  x = hi + lo  of both operands into fp16,  Ahi*Bhi + Ahi*Blo + Alo*Bhi  with the
// float32 accumulator in tensor memory.  fp16 and TF32 have the same 11-bit significand, so the split carries the same
// 22 bits as the TF32 one at half the instructions and half the operand bytes; what fp16 lacks is exponent range.  The
// range is settled when the model is laid out: the basis and its derivative are bounded functions of one variable, so
// bounds of every layer's values follow from the weights, and powers of two (RadialScales) put each operand below
// 2^15.  A model whose bounds leave less than that takes the TF32 kernel instead (the caller decides).
//
// Both operands of an activation live in tensor memory (the elementwise phase writes its lane with tcgen05.st; nothing
// passes shared memory, no proxy fence), and the MMAs read only the 2 KB weight slices from shared memory: a
// tcgen05.mma with its A operand in shared memory is bound by reading 4 KB of it, 48 cycles at N = 64 instead of 32.
// Tensor memory per group of eight warps, for values and derivatives each: 64 accumulator columns, 32 + 32 of hi and lo.
//
// A pair of edges shares a row (EdgeRows): 322 -> 182 us at 16 000 atoms, 1 375 -> 745 at 64 000, 79 -> 52 at 3 000, 30 -> 22 at
// 400, the look-up of the other edges' rows included.
//
// Output rows: HALF: [E][hi 64 | lo 64] fp16 of the value times a power of two, what the products and sums of the step
// read; otherwise [E, 64] float32.
#include "common.cuh"
#include "step_common.cuh"
#include "tc_ptx.cuh"

namespace cmace {

constexpr int RQ_TILE = 128;
constexpr int RQ_GROUP_THREADS = 256;
constexpr int RQ_THREADS = 2 * RQ_GROUP_THREADS;
constexpr int RQ_IMAGE = 64 * 128;            // one weight image: 64 rows of 64 fp16
constexpr int RQ_OUT = 2 * RQ_TILE * 128;     // staging of one output tile: two images of 128 rows x 128 bytes

struct RadialHalfArgs {
  const float *basis;           // [E, 2 nb]
  const void *w[2][3];          // per layer: hi image, lo image (128-byte swizzle), zero rows beyond nb in the first
  RadialScales s[2];
  EdgeRows rows;
  int32_t *status;
  int64_t E;
  int nb, nper;
  int half_out[2];
};
struct RadialHalfMaps {
  CUtensorMap h[2], dh[2];
};

__device__ __forceinline__ float rq_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rq_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void __launch_bounds__(RQ_THREADS, 1)
    radial_half_kernel(const RadialHalfArgs g, const __grid_constant__ RadialHalfMaps maps) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[5];   // weights; done[group][operand]
  __shared__ uint32_t tmem_base_slot;
  __shared__ int32_t edge_s[RQ_THREADS];      // a thread's own: the edge of its next row

  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int group = warp >> 3, gw = warp & 7, gtid = tid & (RQ_GROUP_THREADS - 1);
  const bool second = (blockIdx.x % (unsigned)g.nper) != 0;
  const uint32_t wbar = smem_u32(&bars[0]);
  const uint32_t done0 = wbar + 8u * (1 + 2 * group);
  const uint32_t sOut = smem_base + 6u * RQ_IMAGE + (uint32_t)(2 * group) * RQ_OUT;   // + operand * RQ_OUT

  if (tid == 0) {
    for (int i = 0; i < 5; i++) mbar_init(wbar + 8u * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem0 = (uint32_t)uniform((int)tmem_base_slot) + (uint32_t)group * 256u;   // operand o: + 128 o; hi at + 64, lo at + 96

  if (warp == 0 && elect_one()) {
    mbar_arrive_expect_tx(wbar, 6u * RQ_IMAGE);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const unsigned char *src = static_cast<const unsigned char *>(second ? g.w[1][i] : g.w[0][i]);
      bulk_copy_g2s(smem_base + 2u * i * RQ_IMAGE, src, RQ_IMAGE, wbar);
      bulk_copy_g2s(smem_base + (2u * i + 1u) * RQ_IMAGE, src + RQ_IMAGE, RQ_IMAGE, wbar);
    }
  }
  grid_wait();
  grid_release();   // after the allocation
  bool ok = warp_wait(wbar, 0, lane);
  if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 31);

  resolve_rows(g.rows, g.E, (int64_t)blockIdx.x * RQ_THREADS + tid, (int64_t)gridDim.x * RQ_THREADS);
  const int64_t nrows = count_rows(g.rows, g.E), ntiles = (nrows + RQ_TILE - 1) / RQ_TILE;
  const int64_t step = (int64_t)(gridDim.x / (unsigned)g.nper) * 2;
  const int64_t first = (int64_t)(blockIdx.x / (unsigned)g.nper) * 2 + group;
  const int q = gw & 3, h = gw >> 2;      // lane quarter; column half (first operand: 0 values, 1 derivatives)
  const int r = q * 32 + lane;            // edge of the tile this thread owns
  const uint32_t lane_field = (uint32_t)(q * 32) << 16;
  const bool half_out = (second ? g.half_out[1] : g.half_out[0]) != 0;
  uint32_t phase = 0;

  float4 pre[4];
  // whose basis this thread's row of tile t has, brought by an asynchronous copy (a register more is one too many: it would be
  // spilled, and the spill would wait for the load)
  auto load_edge = [&](int64_t t) {
    const int64_t k = t * RQ_TILE + r;
    if (g.rows.count && k < nrows)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(edge_s + tid)), "l"(g.rows.leaders + k) : "memory");
  };
  auto load_basis = [&](int64_t t) {
    const int64_t k = t * RQ_TILE + r;
    int64_t e = k;
    if (g.rows.count) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      e = k < nrows ? *static_cast<volatile int32_t *>(edge_s + tid) : 0;
    }
    const float4 *b = reinterpret_cast<const float4 *>(g.basis + e * 2 * g.nb + h * g.nb);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      pre[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (4 * i < g.nb && k < nrows) pre[i] = __ldg(b + i);
    }
    load_edge(t + step);
  };
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(RQ_GROUP_THREADS) : "memory"); };
  auto issue = [&](int o, int layer) {
    const uint32_t idesc = umma_idesc_f16(RQ_TILE, 64);
    const uint32_t acc = tmem0 + 128u * (uint32_t)o, a_hi = acc + 64u, a_lo = acc + 96u;
    const uint64_t b_hi = umma_desc_sw128(smem_base + 2u * (uint32_t)layer * RQ_IMAGE);
    const uint64_t b_lo = umma_desc_sw128(smem_base + (2u * (uint32_t)layer + 1u) * RQ_IMAGE);
    const int ksteps = layer == 0 ? 1 : 4;
    for (int j = 0; j < ksteps; j++) {
      umma_f16_ts(acc, a_hi + 8u * j, b_hi + (uint64_t)(2 * j), idesc, j != 0);
      umma_f16_ts(acc, a_hi + 8u * j, b_lo + (uint64_t)(2 * j), idesc, 1);
      umma_f16_ts(acc, a_lo + 8u * j, b_hi + (uint64_t)(2 * j), idesc, 1);
    }
    umma_commit(done0 + 8u * (uint32_t)o);
  };
  // the group has written operand o and read its accumulator
  auto hand_over = [&](int o, int layer) {
    tmem_st_wait();
    tc_fence_before();
    group_sync();
    if (gw == 0 && elect_one()) {
      tc_fence_after();
      issue(o, layer);
    }
  };
  // this thread's 32 columns of operand o: the next operand in tensor memory, or (last layer) the output tile
  auto put = [&](int o, const unsigned long long (&a)[16], bool last) {
    if (last && !half_out) {   // [128 rows x 32 columns] float32 images, one per column half
      const uint32_t row = sOut + (uint32_t)o * RQ_OUT + (uint32_t)h * (RQ_OUT / 2);
#pragma unroll
      for (int c = 0; c < 8; c++)
        asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(row + (uint32_t)sw128_offset(r, c)), "l"(a[2 * c]), "l"(a[2 * c + 1])
                     : "memory");
      return;
    }
    uint32_t hi[16], lo[16];
#pragma unroll
    for (int k = 0; k < 16; k++) split_half2(a[k], hi[k], lo[k]);
    if (last) {                // [128 rows x 64 columns] fp16 images, hi and lo
      const uint32_t row = sOut + (uint32_t)o * RQ_OUT;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const uint32_t off = (uint32_t)sw128_offset(r, 4 * h + c);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + off), "r"(hi[4 * c]), "r"(hi[4 * c + 1]),
                     "r"(hi[4 * c + 2]), "r"(hi[4 * c + 3])
                     : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + RQ_OUT / 2 + off), "r"(lo[4 * c]),
                     "r"(lo[4 * c + 1]), "r"(lo[4 * c + 2]), "r"(lo[4 * c + 3])
                     : "memory");
      }
      return;
    }
    const uint32_t t = tmem0 + 128u * (uint32_t)o + lane_field + 16u * (uint32_t)h;
    tmem_st16(t + 64u, hi);
    tmem_st16(t + 96u, lo);
  };
  auto finish = [&](int o, int layer, int64_t tile) {
    if (layer < 2) {
      hand_over(o, layer + 1);
      return;
    }
    tc_fence_before();
    fence_proxy_async();
    group_sync();
    if (gw == 0 && elect_one()) {   // rows past the end of the array are clipped
      const uint32_t sT = sOut + (uint32_t)o * RQ_OUT;
      const CUtensorMap *map = o == 0 ? (second ? &maps.h[1] : &maps.h[0]) : (second ? &maps.dh[1] : &maps.dh[0]);
      tma_store_2d(map, 0, (int)(tile * RQ_TILE), sT);
      tma_store_2d(map, half_out ? 64 : 32, (int)(tile * RQ_TILE), sT + RQ_OUT / 2);
    }
  };

  load_edge(first);
  load_basis(first);
  for (int64_t tile = first; ok && tile < ntiles; tile += step) {
    {
      const float sc = h == 0 ? (second ? g.s[1].in_v : g.s[0].in_v) : (second ? g.s[1].in_t : g.s[0].in_t);
      const unsigned long long sc2 = pack2(sc, sc);
      uint32_t hi[8], lo[8];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        split_half2(mul2(pack2(pre[i].x, pre[i].y), sc2), hi[2 * i], lo[2 * i]);
        split_half2(mul2(pack2(pre[i].z, pre[i].w), sc2), hi[2 * i + 1], lo[2 * i + 1]);
      }
      const uint32_t t = tmem0 + 128u * (uint32_t)h + lane_field;
      tmem_st8(t + 64u, hi);
      tmem_st8(t + 96u, lo);
      tmem_st_wait();
      tc_fence_before();
      if (tile != first && gw == 0 && elect_one()) tma_store_wait_read();   // the staging buffers are written again at layer 3
      group_sync();
      if (gw == 0 && elect_one()) {
        tc_fence_after();
        issue(0, 0);
        issue(1, 0);
      }
    }
    load_basis(tile + step);
#pragma unroll
    for (int layer = 0; layer < 3; layer++) {
      const float zi = second ? g.s[1].z[layer] : g.s[0].z[layer];
      const float av = second ? g.s[1].a[layer] : g.s[0].a[layer];
      const float tv = second ? g.s[1].t[layer] : g.s[0].t[layer];
      unsigned long long d[16];   // silu'(z) times the derivatives' factor, 32 columns
      if (!warp_wait(done0, phase, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 32);
        ok = false;
        break;
      }
      tc_fence_after();
      {
        unsigned long long a[16];
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          uint32_t v[16];
          tmem_ld16_nowait(tmem0 + lane_field + 32u * h + 16u * hh, v);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const unsigned long long one2 = pack2(1.0f, 1.0f);
            const unsigned long long D = pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
            const unsigned long long z2 = mul2(D, pack2(zi, zi));
            float t0, t1, n0, n1;
            unpack2(mul2(z2, pack2(-1.4426950408889634f, -1.4426950408889634f)), t0, t1);
            unpack2(add2(pack2(rq_ex2(t0), rq_ex2(t1)), one2), n0, n1);
            const unsigned long long s2 = pack2(rq_rcp(n0), rq_rcp(n1));
            a[8 * hh + k] = mul2(mul2(D, pack2(av, av)), s2);
            d[8 * hh + k] = mul2(mul2(s2, pack2(tv, tv)), fma2(z2, fma2(s2, pack2(-1.0f, -1.0f), one2), one2));
          }
        }
        put(0, a, layer == 2);
      }
      finish(0, layer, tile);
      if (!warp_wait(done0 + 8u, phase, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 33);
        ok = false;
        break;
      }
      tc_fence_after();
      {
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          uint32_t v[16];
          tmem_ld16_nowait(tmem0 + 128u + lane_field + 32u * h + 16u * hh, v);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 8; k++)
            d[8 * hh + k] = mul2(d[8 * hh + k], pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])));
        }
        put(1, d, layer == 2);
      }
      finish(1, layer, tile);
      phase ^= 1;
    }
  }
  if (gw == 0 && elect_one()) tma_store_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base_slot, 512);
}

// [rows, 128] fp16 as boxes of 128 rows x 64 columns with the 128-byte swizzle
int encode_half_rows_tensor_map(CUtensorMap *tmap, const void *base, int64_t rows, int box_rows, const char *what);

int radial_half(const float *basis, int nb, const void *const (*w)[3], const RadialScales *scales, const int *half_out,
                int nper, const EdgeRows &rows, int64_t nedges, void *const *h, void *const *dh, int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(radial)";
  if (nedges == 0) return CMACE_OK;
  if (nb != 8 && nb != 16) return fail(CMACE_ERR_UNSUPPORTED, "%s: the basis size must be 8 or 16", what);
  RadialHalfArgs g{};
  RadialHalfMaps maps;
  g.basis = basis; g.rows = rows; g.status = status; g.E = nedges; g.nb = nb; g.nper = nper;
  for (int i = 0; i < nper; i++) {
    for (int k = 0; k < 3; k++) g.w[i][k] = w[i][k];
    g.s[i] = scales[i];
    g.half_out[i] = half_out[i];
    for (int o = 0; o < 2; o++) {
      CUtensorMap *m = o ? &maps.dh[i] : &maps.h[i];
      void *p = o ? dh[i] : h[i];
      const int rc = half_out[i] ? encode_half_rows_tensor_map(m, p, nedges, RQ_TILE, what)
                                 : encode_rows_tensor_map(m, static_cast<const float *>(p), nedges, ST_H, what);
      if (rc) return rc;
    }
  }
  const size_t smem = 6 * RQ_IMAGE + 4 * (size_t)RQ_OUT + 1024;
  const int64_t ntiles = (nedges + RQ_TILE - 1) / RQ_TILE;
  if (ntiles * RQ_TILE > 0x7fffffffLL) return fail(CMACE_ERR_UNSUPPORTED, "%s: too many edges", what);
  int64_t blocks = (ntiles + 1) / 2;
  if (blocks > 148 / nper) blocks = 148 / nper;
  cudaError_t e = cudaFuncSetAttribute(radial_half_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  launch_chained(radial_half_kernel, (unsigned)(blocks * nper), RQ_THREADS, smem, st, g, maps);
  return check_launch(what);
}

}  // namespace cmace
