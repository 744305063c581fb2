// Hidden layers of the radial perceptron with their derivative along the edge length, both layers' perceptrons of a
// model in one launch:
//
//   h = silu(silu(silu(B(r) W1) W2) W3),   h' = dh/dr:   z_k = a_{k-1} W_k,  z'_k = a'_{k-1} W_k,  a_k = silu(z_k),
//   a'_k = silu'(z_k) z'_k,  a_0 = B(r), a'_0 = dB/dr.
//
// A perceptron of one variable has one derivative: carrying it along costs a second row per edge in every product and
// replaces the whole backward (three products, three saved [E, 64] derivative arrays written and read): per edge and
// perceptron 64 + 512 bytes move instead of 32 + 1024 and 1056 more in the backward.
//
// float32: the machinery of radial_mlp.cu (3-term TF32 split, raw images in shared memory, residual images in tensor
// memory).  A tile is 128 edges, its values and its derivatives are two operands with the same rows, so a thread finds
// z and z' of an (edge, unit) in its own lane.  Each of the two groups of eight warps has one tile in flight: the
// values' products of the next layer run while the derivatives' elementwise phase does, and the groups overlap each
// other.  Tensor memory holds per group 64 accumulator + 64 residual columns for each operand: all 512.
#include "common.cuh"
#include "sigmoid64.cuh"
#include "step_common.cuh"
#include "tc_ptx.cuh"

namespace cmace {

constexpr int RT_TILE = 128;
constexpr int RT_GROUP_THREADS = 256;
constexpr int RT_THREADS = 2 * RT_GROUP_THREADS;
constexpr int RT_SLAB = RT_TILE * 128;        // one image of 128 rows x 32 columns
constexpr int RT_BUF = 2 * RT_SLAB;           // an operand's 64 columns (first layer: raw and residual image of the basis)
constexpr int RT_W_SMALL = 2 * 64 * 128;      // packed [nb <= 32, 64]
constexpr int RT_W_BIG = 2 * RT_W_SMALL;      // packed [64, 64]
constexpr int RT_TMEM_OP = 128;               // columns of one operand: 64 accumulator + 64 residual

struct RadialPairArgs {
  const float *basis;        // [E, 2 nb]: values then derivatives
  const float *w[2][3];      // packed weights of the two perceptrons
  int32_t *status;
  int64_t E;
  int nb, nper;              // perceptrons: block b works for perceptron b % nper
};
struct RadialPairMaps {
  CUtensorMap h[2], dh[2];   // [E, 64] outputs as 128-row x 32-column boxes
};

__device__ __forceinline__ float rt_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rt_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// silu(z) = z s, silu'(z) = s (1 + z (1 - s)), s = 1 / (1 + 2^(-z log2 e)), two values at once
__device__ __forceinline__ void rt_silu2(unsigned long long z2, unsigned long long &a2, unsigned long long &d2) {
  const unsigned long long one2 = pack2(1.0f, 1.0f);
  float t0, t1, n0, n1;
  unpack2(mul2(z2, pack2(-1.4426950408889634f, -1.4426950408889634f)), t0, t1);
  unpack2(add2(pack2(rt_ex2(t0), rt_ex2(t1)), one2), n0, n1);
  const unsigned long long s2 = pack2(rt_rcp(n0), rt_rcp(n1));
  a2 = mul2(z2, s2);
  d2 = mul2(s2, fma2(z2, fma2(s2, pack2(-1.0f, -1.0f), one2), one2));
}

// products of one layer for one operand into its 64 accumulator columns
__device__ __forceinline__ void rt_issue(uint32_t acc, uint32_t sA, uint32_t sB, bool first, int nb) {
  const uint32_t idesc = umma_idesc_tf32(RT_TILE, 64);
  constexpr uint32_t image = 64u * 128u;
  if (first) {
    const uint64_t a_hi = umma_desc_sw128(sA), a_lo = umma_desc_sw128(sA + RT_SLAB);
    const uint64_t b_hi = umma_desc_sw128(sB), b_lo = umma_desc_sw128(sB + image);
    for (int j = 0; j < nb / 8; j++) {
      umma_tf32(acc, a_hi + (uint64_t)(2 * j), b_hi + (uint64_t)(2 * j), idesc, j != 0);
      umma_tf32_acc(acc, a_hi + (uint64_t)(2 * j), b_lo + (uint64_t)(2 * j), idesc);
      umma_tf32_acc(acc, a_lo + (uint64_t)(2 * j), b_hi + (uint64_t)(2 * j), idesc);
    }
    return;
  }
#pragma unroll
  for (int kb = 0; kb < 2; kb++) {
    const uint64_t a_hi = umma_desc_sw128(sA + kb * RT_SLAB);
    const uint64_t b_hi = umma_desc_sw128(sB + kb * 2 * image), b_lo = umma_desc_sw128(sB + kb * 2 * image + image);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      umma_tf32(acc, a_hi + (uint64_t)(2 * j), b_hi + (uint64_t)(2 * j), idesc, (kb | j) != 0);
      umma_tf32_acc(acc, a_hi + (uint64_t)(2 * j), b_lo + (uint64_t)(2 * j), idesc);
      umma_tf32_ts_acc(acc, acc + 64u + 32u * kb + 8u * j, b_hi + (uint64_t)(2 * j), idesc);
    }
  }
}

__device__ __forceinline__ void rt_store_split(uint32_t s_hi, float4 a) {
  float4 lo;
  lo.x = to_tf32(a.x - __uint_as_float(__float_as_uint(a.x) & 0xFFFFE000u));
  lo.y = to_tf32(a.y - __uint_as_float(__float_as_uint(a.y) & 0xFFFFE000u));
  lo.z = to_tf32(a.z - __uint_as_float(__float_as_uint(a.z) & 0xFFFFE000u));
  lo.w = to_tf32(a.w - __uint_as_float(__float_as_uint(a.w) & 0xFFFFE000u));
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(s_hi), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w) : "memory");
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(s_hi + RT_SLAB), "f"(lo.x), "f"(lo.y), "f"(lo.z), "f"(lo.w)
               : "memory");
}

// NI: 16-byte chunks of the basis a thread carries per tile (nb / 4: values and derivatives of 128 edges, 256 threads)
template <int NI>
__global__ void __launch_bounds__(RT_THREADS, 1)
    radial_pair_kernel(const RadialPairArgs g, const __grid_constant__ RadialPairMaps maps) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[5];   // weights; done[group][operand]
  __shared__ uint32_t tmem_base_slot;

  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int group = warp >> 3, gw = warp & 7, gtid = tid & (RT_GROUP_THREADS - 1);
  const int per = (int)(blockIdx.x % (unsigned)g.nper);
  const uint32_t wbar = smem_u32(&bars[0]);
  const uint32_t done0 = wbar + 8u * (1 + 2 * group);

  const uint32_t w_bytes[3] = {(uint32_t)RT_W_SMALL, (uint32_t)RT_W_BIG, (uint32_t)RT_W_BIG};
  const uint32_t sW[3] = {smem_base, smem_base + w_bytes[0], smem_base + w_bytes[0] + w_bytes[1]};
  const uint32_t sA0 = smem_base + w_bytes[0] + w_bytes[1] + w_bytes[2] + (uint32_t)(2 * group) * RT_BUF;

  if (tid == 0) {
    for (int i = 0; i < 5; i++) mbar_init(wbar + 8u * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_wait();
  if (warp == 0) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_release();   // after the allocation
  const uint32_t tmem0 = (uint32_t)uniform((int)tmem_base_slot) + (uint32_t)(2 * group) * RT_TMEM_OP;   // + operand * RT_TMEM_OP

  if (warp == 0 && elect_one()) {
    mbar_arrive_expect_tx(wbar, w_bytes[0] + w_bytes[1] + w_bytes[2]);
#pragma unroll
    for (int i = 0; i < 3; i++)
      for (uint32_t off = 0; off < w_bytes[i]; off += 8192u)
        bulk_copy_g2s(sW[i] + off, reinterpret_cast<const unsigned char *>(per ? g.w[1][i] : g.w[0][i]) + off, 8192u, wbar);
  }
  bool ok = warp_wait(wbar, 0, lane);
  if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 21);

  const int64_t ntiles = (g.E + RT_TILE - 1) / RT_TILE;
  const int64_t step = (int64_t)(gridDim.x / (unsigned)g.nper) * 2;
  const int64_t first = (int64_t)(blockIdx.x / (unsigned)g.nper) * 2 + group;
  const int q = gw & 3, h = gw >> 2;      // tensor-memory lane quarter, column half (= K block of the next layer)
  const int r = q * 32 + lane;            // edge of the tile this thread owns in the elementwise phases
  const uint32_t lane_field = (uint32_t)(q * 32) << 16;
  const int half_chunks = g.nb / 4;       // 16-byte chunks of the values; as many of the derivatives follow
  uint32_t phase = 0;

  float4 pre[NI];
  auto load_basis = [&](int64_t t) {
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int idx = gtid + RT_GROUP_THREADS * i;
      const int rr = idx / (2 * half_chunks), c = idx - rr * (2 * half_chunks);
      const int64_t e = t * RT_TILE + rr;
      pre[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < ntiles && e < g.E) pre[i] = __ldg(reinterpret_cast<const float4 *>(g.basis + e * 2 * g.nb) + c);
    }
  };
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(RT_GROUP_THREADS) : "memory"); };
  // operand o (0 values, 1 derivatives) of the next layer is written: the group's first thread issues its products
  auto hand_over = [&](int o, int layer) {
    fence_proxy_async();
    group_sync();
    if (gw == 0 && elect_one()) {
      tc_fence_after();
      rt_issue(tmem0 + (uint32_t)o * RT_TMEM_OP, sA0 + (uint32_t)o * RT_BUF, layer == 1 ? sW[1] : sW[2], false, g.nb);
      umma_commit(done0 + 8u * o);
    }
  };
  // 16 columns of an operand: raw values into the swizzled image, residual into tensor memory
  auto put16 = [&](int o, int hh, const unsigned long long (&a)[8], bool residual) {
    const uint32_t a_row = sA0 + (uint32_t)o * RT_BUF + (uint32_t)h * RT_SLAB;
#pragma unroll
    for (int c = 0; c < 4; c++)
      asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a_row + (uint32_t)sw128_offset(r, 4 * hh + c)), "l"(a[2 * c]),
                   "l"(a[2 * c + 1])
                   : "memory");
    if (!residual) return;
    uint32_t lo[16];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const unsigned long long l2 = sub2(a[k], a[k] & 0xFFFFE000FFFFE000ull);
      asm("mov.b64 {%0, %1}, %2;" : "=r"(lo[2 * k]), "=r"(lo[2 * k + 1]) : "l"(l2));
    }
    tmem_st16(tmem0 + (uint32_t)o * RT_TMEM_OP + lane_field + 64u + 32u * h + 16u * hh, lo);
  };
  auto finish_operand = [&](int o, int layer, int64_t tile) {
    if (layer < 2) {
      tmem_st_wait();
      tc_fence_before();
      hand_over(o, layer + 1);
    } else {
      // the swizzled images of the last layer are what the tile stores read; rows past the end are clipped
      tc_fence_before();
      fence_proxy_async();
      group_sync();
      if (gw == 0 && elect_one()) {
        const uint32_t sT = sA0 + (uint32_t)o * RT_BUF;
        const CUtensorMap *map = o == 0 ? (per ? &maps.h[1] : &maps.h[0]) : (per ? &maps.dh[1] : &maps.dh[0]);
        tma_store_2d(map, 0, (int)(tile * RT_TILE), sT);
        tma_store_2d(map, 32, (int)(tile * RT_TILE), sT + RT_SLAB);
      }
    }
  };

  load_basis(first);
  for (int64_t tile = first; ok && tile < ntiles; tile += step) {
    if (tile != first) {
      if (gw == 0 && elect_one()) tma_store_wait_read();   // the previous tile's stores read the buffers that are written next
      group_sync();
    }
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int idx = gtid + RT_GROUP_THREADS * i;
      const int rr = idx / (2 * half_chunks), c = idx - rr * (2 * half_chunks);
      const int o = c >= half_chunks ? 1 : 0;
      rt_store_split(sA0 + (uint32_t)o * RT_BUF + (uint32_t)sw128_offset(rr, c - o * half_chunks), pre[i]);
    }
    tc_fence_before();
    fence_proxy_async();
    group_sync();
    if (gw == 0 && elect_one()) {
      tc_fence_after();
#pragma unroll
      for (int o = 0; o < 2; o++) {
        rt_issue(tmem0 + (uint32_t)o * RT_TMEM_OP, sA0 + (uint32_t)o * RT_BUF, sW[0], true, g.nb);
        umma_commit(done0 + 8u * o);
      }
    }
    load_basis(tile + step);
    for (int layer = 0; ok && layer < 3; layer++) {
      unsigned long long d[16];   // silu'(z) of this thread's 32 columns
      if (!warp_wait(done0, phase, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 22);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int hh = 0; hh < 2; hh++) {
        uint32_t v[16];
        tmem_ld16_nowait(tmem0 + lane_field + 32u * h + 16u * hh, v);
        tmem_ld_wait();
        unsigned long long a[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
          rt_silu2(pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])), a[k], d[8 * hh + k]);
        put16(0, hh, a, layer < 2);
      }
      finish_operand(0, layer, tile);
      if (!warp_wait(done0 + 8u, phase, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 23);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int hh = 0; hh < 2; hh++) {
        uint32_t v[16];
        tmem_ld16_nowait(tmem0 + RT_TMEM_OP + lane_field + 32u * h + 16u * hh, v);
        tmem_ld_wait();
        unsigned long long a[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
          a[k] = mul2(d[8 * hh + k], pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])));
        put16(1, hh, a, layer < 2);
      }
      finish_operand(1, layer, tile);
      phase ^= 1;
    }
  }
  if (gw == 0 && elect_one()) tma_store_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base_slot, 512);
}

// ---- float64 on the FP64 tensor cores ------------------------------------------------------------------------------
// 16 warps per CTA, tile of 128 edges; a warp owns the values and the derivatives of eight edges through all layers
// (no block barrier), so one B fragment feeds two mma.m8n8k4 and the elementwise phase pairs z and z' in registers.
// Row strides of 68 doubles make the fragment loads of both operands conflict-free.  A pair of edges shares a row (EdgeRows):
// 1 178 -> 646 us at 8 000 atoms, of which the products are 392 at the instruction's rate and the sigmoids about 110; 67 -> 35 at 192.
constexpr int RD_WARPS = 16, RD_LD = 68;

struct RadialPairArgs64 {
  const double *basis;
  const double *w[2][3];   // [nb, 64], [64, 64], [64, 64]
  double *h[2], *dh[2];
  EdgeRows rows;
  int64_t E;
  int nb, nper;
};

__global__ void __launch_bounds__(RD_WARPS * 32, 1) radial_pair_f64_kernel(const RadialPairArgs64 g) {
  extern __shared__ __align__(16) double rd_smem[];
  __shared__ double etab[32];   // 2^(j/32)
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int per = (int)(blockIdx.x % (unsigned)g.nper);
  if (tid < 32) etab[tid] = exp2((double)tid / 32.0);
  double *const sW1 = rd_smem, *const sW2 = sW1 + 16 * RD_LD, *const sW3 = sW2 + 64 * RD_LD;
  double *const act = sW3 + 64 * RD_LD + warp * (16 * RD_LD);   // 8 rows of values, 8 of derivatives
  for (int i = tid; i < g.nb * 64; i += RD_WARPS * 32) sW1[(i >> 6) * RD_LD + (i & 63)] = (per ? g.w[1][0] : g.w[0][0])[i];
  for (int i = tid; i < 64 * 64; i += RD_WARPS * 32) {
    sW2[(i >> 6) * RD_LD + (i & 63)] = (per ? g.w[1][1] : g.w[0][1])[i];
    sW3[(i >> 6) * RD_LD + (i & 63)] = (per ? g.w[1][2] : g.w[0][2])[i];
  }
  __syncthreads();
  grid_begin();
  const int fr = lane >> 2, fk = lane & 3;
  double *const h_out = per ? g.h[1] : g.h[0], *const dh_out = per ? g.dh[1] : g.dh[0];
  resolve_rows(g.rows, g.E, (int64_t)blockIdx.x * (RD_WARPS * 32) + tid, (int64_t)gridDim.x * (RD_WARPS * 32));
  const int64_t nrows = count_rows(g.rows, g.E), groups = (nrows + 7) / 8;
  const int64_t stride = (int64_t)(gridDim.x / (unsigned)g.nper) * RD_WARPS;
  for (int64_t t = (int64_t)(blockIdx.x / (unsigned)g.nper) * RD_WARPS + warp; t < groups; t += stride) {
    const int64_t e0 = t * 8, mine = e0 + (lane & 7);
    const int edge = mine < nrows ? (g.rows.count ? g.rows.leaders[mine] : (int)mine) : -1;
    for (int i = lane; i < 16 * g.nb; i += 32) {   // a multiple of 32
      const int row = i / (2 * g.nb), c = i - row * 2 * g.nb;
      const int from = __shfl_sync(0xffffffffu, edge, row);
      const double v = from >= 0 ? g.basis[(int64_t)from * 2 * g.nb + c] : 0.0;
      const int o = c >= g.nb ? 1 : 0;
      act[(8 * o + row) * RD_LD + c - o * g.nb] = v;
    }
    __syncwarp();
    double acc[2][8][2];
#pragma unroll 1
    for (int layer = 0; layer < 3; layer++) {
      const double *W = layer == 0 ? sW1 : (layer == 1 ? sW2 : sW3);
      const int K = layer == 0 ? g.nb : 64;
#pragma unroll
      for (int n = 0; n < 8; n++) acc[0][n][0] = acc[0][n][1] = acc[1][n][0] = acc[1][n][1] = 0.0;
#pragma unroll 2
      for (int k = 0; k < K; k += 4) {
        const double av = act[fr * RD_LD + k + fk], at = act[(8 + fr) * RD_LD + k + fk];
#pragma unroll
        for (int n = 0; n < 8; n++) {
          const double b = W[(k + fk) * RD_LD + 8 * n + fr];
          dmma(acc[0][n], av, b);
          dmma(acc[1][n], at, b);
        }
      }
      __syncwarp();
#pragma unroll
      for (int n = 0; n < 8; n++) {
        double a[2], da[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const double z = acc[0][n][u], s = table_sigmoid(z, etab);
          a[u] = z * s;
          da[u] = s * (1.0 + z * (1.0 - s)) * acc[1][n][u];
        }
        const int col = 8 * n + 2 * fk;
        if (layer < 2) {
          *reinterpret_cast<double2 *>(act + fr * RD_LD + col) = make_double2(a[0], a[1]);
          *reinterpret_cast<double2 *>(act + (8 + fr) * RD_LD + col) = make_double2(da[0], da[1]);
        } else if (e0 + fr < nrows) {
          *reinterpret_cast<double2 *>(h_out + (e0 + fr) * ST_H + col) = make_double2(a[0], a[1]);
          *reinterpret_cast<double2 *>(dh_out + (e0 + fr) * ST_H + col) = make_double2(da[0], da[1]);
        }
      }
      __syncwarp();
    }
  }
}

// Both perceptrons share the grid: even blocks work for the first, odd ones for the second.
int radial_pair_f32(const float *basis, int nb, const float *const (*w)[3], int nper, int64_t nedges, float *const *h,
                    float *const *dh, int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(radial)";
  if (nedges == 0) return CMACE_OK;
  if (nb != 8 && nb != 16) return fail(CMACE_ERR_UNSUPPORTED, "%s: the basis size must be 8 or 16", what);
  RadialPairArgs g{};
  RadialPairMaps maps;
  g.basis = basis; g.status = status; g.E = nedges; g.nb = nb; g.nper = nper;
  for (int i = 0; i < nper; i++) {
    for (int k = 0; k < 3; k++) g.w[i][k] = w[i][k];
    if (int rc = encode_rows_tensor_map(&maps.h[i], h[i], nedges, ST_H, what)) return rc;
    if (int rc = encode_rows_tensor_map(&maps.dh[i], dh[i], nedges, ST_H, what)) return rc;
  }
  const size_t smem = RT_W_SMALL + 2 * RT_W_BIG + 4 * (size_t)RT_BUF + 1024;
  const int64_t ntiles = (nedges + RT_TILE - 1) / RT_TILE;
  if (ntiles * RT_TILE > 0x7fffffffLL) return fail(CMACE_ERR_UNSUPPORTED, "%s: too many edges", what);
  int64_t blocks = (ntiles + 1) / 2;
  if (blocks > 148 / nper) blocks = 148 / nper;
  auto kern = nb == 8 ? radial_pair_kernel<2> : radial_pair_kernel<4>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  launch_chained(kern, (unsigned)(blocks * nper), RT_THREADS, smem, st, g, maps);
  return check_launch(what);
}

int radial_pair_f64(const double *basis, int nb, const double *const (*w)[3], int nper, const EdgeRows &rows, int64_t nedges,
                    double *const *h, double *const *dh, cudaStream_t st) {
  const char *what = "cmace_step(radial)";
  if (nedges == 0) return CMACE_OK;
  if (nb != 8 && nb != 16) return fail(CMACE_ERR_UNSUPPORTED, "%s: the basis size must be 8 or 16", what);
  RadialPairArgs64 g{};
  g.rows = rows;
  g.basis = basis; g.E = nedges; g.nb = nb; g.nper = nper;
  for (int i = 0; i < nper; i++) {
    for (int k = 0; k < 3; k++) g.w[i][k] = w[i][k];
    g.h[i] = h[i];
    g.dh[i] = dh[i];
  }
  const size_t smem = (size_t)(16 + 2 * 64 + 16 * RD_WARPS) * RD_LD * sizeof(double);
  int64_t blocks = (nedges + 8 * RD_WARPS - 1) / (8 * RD_WARPS);
  if (blocks > 148 / nper) blocks = 148 / nper;
  cudaError_t e = cudaFuncSetAttribute(radial_pair_f64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  launch_chained(radial_pair_f64_kernel, (unsigned)(blocks * nper), RD_WARPS * 32, smem, st, g);
  return check_launch(what);
}

}  // namespace cmace
