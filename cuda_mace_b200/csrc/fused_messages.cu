// Second layer's message passing with the radial weights formed where they are used (float32, 128 channels), forward
// and backward:
//
//   m[i, lm, c] = sum_{e -> i} Y[lm, e] X[s(e), c] R_l[e, c],   R_l[e, c] = sum_k h[e, k] W[k, l, c].
//
// The unfused form writes R [E, 512] (2 KB an edge) with a product and reads it in the scatter and in its backward.  Here
// R^T is the accumulator of a tcgen05.mma: rows of W^T are the tensor-memory lanes, a tile's edges its columns.  Both
// images of W^T (hi, lo) are the A operand and stay in tensor memory for the whole kernel: 4 blocks of 128 rows x (32 +
// 32) columns; the accumulators of two independent sets of warps take the other 2 x 128 columns.  With A in tensor
// memory an MMA reads only 1 KB of h from shared memory, where the consumers need the bandwidth (with A in shared memory
// its 4 KB are what a narrow MMA waits for).
//
// What bounds the consumers is the shared-memory pipe: a value that a whole warp reads (Y) still costs a wavefront, and
// so does a shuffle.  A warp reaches 32 of the 128 lanes, and which (l, channel) rows those are is free: lane quarters 0
// and 1 hold l = 3 and l = 0, quarters 2 and 3 hold l = 1 and l = 2, two channels a lane, blocks (l, even), (l, odd),
// (l', even), (l', odd).  Every quarter then works for eight components of two channels a lane: an edge costs 32 + 2
// wavefronts of Y instead of 64, and its sums over channels 8 values a warp instead of 16.
#include "common.cuh"
#include "step_common.cuh"
#include "tc_ptx.cuh"

namespace cmace {

constexpr int FM_C = 128;
constexpr int FM_SETS = 2;                        // independent pipelines of a CTA
constexpr int FM_THREADS = FM_SETS * 6 * 32;      // per set: four consumer warps, an MMA warp, a loader warp

// first node whose edges start at or after e
__device__ __forceinline__ int64_t first_node_at(const int32_t *__restrict__ row_ptr, int64_t nnodes, int64_t e) {
  int64_t lo = 0, hi = nnodes;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (row_ptr[mid] >= e) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ float lds1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// W^T [512 rows][hi 64 | lo 64] fp16 into tensor memory: block j at columns 64 j (hi) and 64 j + 32 (lo); four warps
__device__ __forceinline__ void load_w_tmem(const uint4 *__restrict__ W, uint32_t tmem, int q, int lane) {
  const uint4 *w = W + (int64_t)(32 * q + lane) * 16;
#pragma unroll 1
  for (int j = 0; j < 4; j++)
#pragma unroll 1
    for (int im = 0; im < 2; im++) {
      uint32_t v[32];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint4 u = __ldg(w + (int64_t)j * 128 * 16 + 8 * im + i);
        v[4 * i] = u.x;
        v[4 * i + 1] = u.y;
        v[4 * i + 2] = u.z;
        v[4 * i + 3] = u.w;
      }
      tmem_st32(tmem + ((uint32_t)(32 * q) << 16) + 64u * j + 32u * im, v);
    }
  tmem_st_wait();
}

// the 48 products of a tile: D block j [128 x 32] = W block j (hi, lo) times the 32 rows of the B images
__device__ __forceinline__ void issue_tile(uint32_t tmem, uint32_t acc, uint32_t sB, uint32_t image_bytes) {
  const uint32_t idesc = umma_idesc_f16(128, 32);
  const uint64_t b_hi = umma_desc_sw128(sB), b_lo = umma_desc_sw128(sB + image_bytes);
#pragma unroll 1
  for (int j = 0; j < 4; j++) {
    const uint32_t d = acc + 32u * j, a = tmem + 64u * j;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      umma_f16_ts(d, a + 8u * k, b_hi + (uint64_t)(2 * k), idesc, k != 0);
      umma_f16_ts(d, a + 8u * k, b_lo + (uint64_t)(2 * k), idesc, 1);
      umma_f16_ts(d, a + 32u + 8u * k, b_hi + (uint64_t)(2 * k), idesc, 1);
    }
  }
}

// a row of X (512 bytes) for every lane's sender index s, rows i = 0 .. N - 1: one 16-byte asynchronous copy a lane each;
// the 32 lanes' arrivals on bar follow their copies
template <int N>
__device__ __forceinline__ void copy_sender_rows(const float *__restrict__ X, int s, uint32_t dst, uint32_t bar, int lane) {
#pragma unroll 8
  for (int i = 0; i < N; i++) {
    const int64_t row = __shfl_sync(0xffffffffu, s, i);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)i * 512u + 16u * lane),
                 "l"(X + row * FM_C + 4 * lane)
                 : "memory");
  }
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- forward --------------------------------------------------------------------------------------------------------
// A set owns a contiguous range of receivers, so no sum is split and none is atomic; its warps keep 16 sums a lane.
constexpr int FF_TILE = 32;                       // edges of a tile
constexpr int FF_STAGES = 3;
constexpr int FF_X_BYTES = FF_TILE * FM_C * 4;    // sender rows
constexpr int FF_H_BYTES = 2 * FF_TILE * 128;     // hi and lo image of h
constexpr int FF_Y_BYTES = FF_TILE * 64;
constexpr int FF_STAGE_BYTES = FF_X_BYTES + FF_H_BYTES + FF_Y_BYTES;

struct FusedMessagesArgs {
  const float *X, *Y;            // [Ns, 128], [E, 16]
  const uint4 *W;                // permuted W^T
  const int32_t *sender, *receiver, *row_ptr;
  int32_t *status;
  int64_t nnodes, nedges;
  float factor;                  // undoes the powers of two of h and W
  float *out;                    // [nnodes, 16, 128]
};

// Y of an edge for one kind of quarter: HIGH components 9 .. 15 (l = 3; l = 0 has Y = 1), otherwise 1 .. 8
template <bool HIGH>
__device__ __forceinline__ void load_y(float (&y)[8], uint32_t ya) {
  const float4 u = lds4(ya + (HIGH ? 32u : 0u)), v = lds4(ya + (HIGH ? 48u : 16u));
  y[0] = u.y; y[1] = u.z; y[2] = u.w; y[3] = v.x; y[4] = v.y; y[5] = v.z; y[6] = v.w;
  y[7] = HIGH ? 1.f : lds1(ya + 32u);
}

// one edge into the 16 sums of a lane (components in pairs of channels)
template <bool HIGH>
__device__ __forceinline__ void add_edge(float (&acc)[16], const float (&y)[8], float2 x, uint32_t ra, uint32_t rb, uint32_t rc,
                                         uint32_t rd) {
  const float pa = x.x * __uint_as_float(ra), pb = x.y * __uint_as_float(rb);
  const float qa = x.x * __uint_as_float(rc), qb = x.y * __uint_as_float(rd);
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const bool first = HIGH ? m < 7 : m < 3;
    if (HIGH && m == 7) {
      acc[14] += qa;
      acc[15] += qb;
    } else {
      acc[2 * m] = fmaf(y[m], first ? pa : qa, acc[2 * m]);
      acc[2 * m + 1] = fmaf(y[m], first ? pb : qb, acc[2 * m + 1]);
    }
  }
}

// What a set's consumers do with one tile; HIGH: quarters 0, 1 (l = 3, 0), otherwise l = 1, 2.  Eight edges at a time;
// without a receiver's last edge among them there is no branch, so that the loads of several edges are on their way
// before the first sum (with a branch per edge: 1.85 ms at 64 000 atoms instead of 1.55).
template <bool HIGH>
__device__ __forceinline__ void forward_tile(float (&acc)[16], uint32_t ta, uint32_t sX, uint32_t sY, int nvalid,
                                             uint32_t last, const int32_t *recv, float factor, float *out) {
#pragma unroll 1
  for (int i0 = 0; i0 < nvalid; i0 += 8) {
    uint32_t r[4][8];
#pragma unroll
    for (int j = 0; j < 4; j++) tmem_ld8_nowait(ta + 32u * j + (uint32_t)i0, r[j]);
    float2 x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = lds2(sX + 512u * (uint32_t)(i0 + i));
    const uint32_t ya = sY + 64u * (uint32_t)i0;
    if (nvalid - i0 >= 8 && ((last >> i0) & 0xffu) == 0) {
      float y[4][8];
#pragma unroll
      for (int i = 0; i < 4; i++) load_y<HIGH>(y[i], ya + 64u * i);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; i++) {
        add_edge<HIGH>(acc, y[i], x[i], r[0][i], r[1][i], r[2][i], r[3][i]);
        load_y<HIGH>(y[i], ya + 64u * (4 + i));
      }
#pragma unroll
      for (int i = 0; i < 4; i++) add_edge<HIGH>(acc, y[i], x[4 + i], r[0][4 + i], r[1][4 + i], r[2][4 + i], r[3][4 + i]);
    } else {
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (i0 + i < nvalid) {
          float y[8];
          load_y<HIGH>(y, ya + 64u * i);
          add_edge<HIGH>(acc, y, x[i], r[0][i], r[1][i], r[2][i], r[3][i]);
          if ((last >> (i0 + i)) & 1u) {
            float *o = out + (int64_t)recv[i0 + i] * (16 * FM_C);
#pragma unroll
            for (int m = 0; m < 8; m++) {
              const int lm = HIGH ? (m < 7 ? 9 + m : 0) : 1 + m;
              *reinterpret_cast<float2 *>(o + lm * FM_C) = make_float2(acc[2 * m] * factor, acc[2 * m + 1] * factor);
              acc[2 * m] = acc[2 * m + 1] = 0.f;
            }
          }
        }
      }
    }
  }
}

__global__ void __launch_bounds__(FM_THREADS, 1)
    fused_messages_kernel(const FusedMessagesArgs g, const __grid_constant__ CUtensorMap h_map) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[FM_SETS][3 * FF_STAGES + 2];   // h landed, X / Y landed, stage free; acc full, free
  __shared__ int32_t recv_s[FM_SETS][FF_STAGES][FF_TILE];
  __shared__ uint32_t last_s[FM_SETS][FF_STAGES];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int64_t range_s[FM_SETS + 1];

  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // warps 0-3, 4-7: consumers of sets 0, 1; 8, 9: their MMA warps; 10, 11: their loaders
  const int set = warp < 8 ? warp >> 2 : warp & 1;
  const uint32_t h_full = smem_u32(&bars[set][0]), x_full = h_full + 8u * FF_STAGES, st_free = x_full + 8u * FF_STAGES;
  const uint32_t acc_full = st_free + 8u * FF_STAGES, acc_free = acc_full + 8u;
  const uint32_t stages = smem_base + (uint32_t)(set * FF_STAGES) * FF_STAGE_BYTES;

  if (tid == 0) {
    for (int k = 0; k < FM_SETS; k++) {
      const uint32_t b = smem_u32(&bars[k][0]);
      for (int s = 0; s < FF_STAGES; s++) {
        mbar_init(b + 8u * s, 1);
        mbar_init(b + 8u * (FF_STAGES + s), 33);       // the loader's 32 lanes and its expect_tx
        mbar_init(b + 8u * (2 * FF_STAGES + s), 4);
      }
      mbar_init(b + 8u * (3 * FF_STAGES), 1);
      mbar_init(b + 8u * (3 * FF_STAGES + 1), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid <= FM_SETS) {
    const int64_t pieces = (int64_t)gridDim.x * FM_SETS, b = (int64_t)blockIdx.x * FM_SETS + tid;
    const int64_t per = (g.nedges + pieces - 1) / pieces;
    range_s[tid] = b >= pieces ? g.nnodes : (b == 0 ? 0 : first_node_at(g.row_ptr, g.nnodes, b * per));
  }
  if (warp == 8) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot, acc_t = tmem + 256u + 128u * (uint32_t)set;
  if (warp < 4) load_w_tmem(g.W, tmem, warp, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const int64_t n0 = range_s[set], n1 = range_s[set + 1];
  const int64_t e0 = n0 < n1 ? g.row_ptr[n0] : 0, e1 = n0 < n1 ? g.row_ptr[n1] : 0;
  const int64_t ntiles = (e1 - e0 + FF_TILE - 1) / FF_TILE;
  int stage = 0;
  uint32_t phase = 0;
  auto advance = [&]() {
    if (++stage == FF_STAGES) {
      stage = 0;
      phase ^= 1;
    }
  };

  if (warp >= 10) {
    // ---- loader: h rows by TMA, Y rows as one bulk copy, sender rows by asynchronous copies
    for (int64_t t = 0; t < ntiles; t++) {
      if (!warp_wait(st_free + 8u * stage, phase ^ 1, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 41);
        break;
      }
      const int64_t base = e0 + t * FF_TILE, e = base + lane < e1 ? base + lane : e1 - 1;
      const uint32_t sX = stages + (uint32_t)stage * FF_STAGE_BYTES, sH = sX + FF_X_BYTES, sY = sH + FF_H_BYTES;
      if (lane == 0) {
        mbar_arrive_expect_tx(h_full + 8u * stage, FF_H_BYTES);
        tma_load_2d(sH, &h_map, 0, (int)base, h_full + 8u * stage);
        tma_load_2d(sH + FF_H_BYTES / 2, &h_map, 64, (int)base, h_full + 8u * stage);
      }
      const int s = g.sender[e], r = g.receiver[e];
      const int rn = base + lane + 1 < e1 ? g.receiver[base + lane + 1] : -1;
      const unsigned last = __ballot_sync(0xffffffffu, base + lane < e1 && rn != r);
      recv_s[set][stage][lane] = r;
      if (lane == 0) last_s[set][stage] = last;
      __syncwarp();
      if (lane == 0) {
        const uint32_t bytes = (uint32_t)(e1 - base < FF_TILE ? e1 - base : FF_TILE) * 64u;
        mbar_arrive_expect_tx(x_full + 8u * stage, bytes);
        bulk_copy_g2s(sY, g.Y + base * 16, bytes, x_full + 8u * stage);
      }
      copy_sender_rows<FF_TILE>(g.X, s, sX, x_full + 8u * stage, lane);
      advance();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= 8) {
    // ---- MMA issuer
    for (int64_t t = 0; t < ntiles; t++) {
      if (!warp_wait(acc_free, ((uint32_t)t & 1u) ^ 1u, lane) || !warp_wait(h_full + 8u * stage, phase, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 42);
        break;
      }
      if (lane == 0) {
        tc_fence_after();
        issue_tile(tmem, acc_t, stages + (uint32_t)stage * FF_STAGE_BYTES + FF_X_BYTES, FF_H_BYTES / 2);
        umma_commit(acc_full);
      }
      __syncwarp();
      advance();
    }
  } else {
    // ---- consumers
    const int q = warp & 3;
    const bool high = q < 2;
    const int c = 64 * (q & 1) + 2 * lane;
    const uint32_t ta = acc_t + ((uint32_t)(32 * q) << 16);
    // receivers of this range without edges: their rows are zero
    for (int64_t n = n0; n < n1; n++)
      if (g.row_ptr[n] == g.row_ptr[n + 1])
        for (int m = 0; m < 8; m++) {
          const int lm = high ? (m < 7 ? 9 + m : 0) : 1 + m;
          *reinterpret_cast<float2 *>(g.out + n * (16 * FM_C) + lm * FM_C + c) = make_float2(0.f, 0.f);
        }
    float acc[16];
#pragma unroll
    for (int m = 0; m < 16; m++) acc[m] = 0.f;
    for (int64_t t = 0; t < ntiles; t++) {
      if (!warp_wait(x_full + 8u * stage, phase, lane) || !warp_wait(acc_full, (uint32_t)t & 1u, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 43);
        break;
      }
      tc_fence_after();
      const uint32_t sX = stages + (uint32_t)stage * FF_STAGE_BYTES, sY = sX + FF_X_BYTES + FF_H_BYTES;
      const int64_t left = e1 - (e0 + t * FF_TILE);
      const int nvalid = (int)(left < FF_TILE ? left : FF_TILE);
      if (high) forward_tile<true>(acc, ta, sX + 4u * c, sY, nvalid, last_s[set][stage], recv_s[set][stage], g.factor, g.out + c);
      else forward_tile<false>(acc, ta, sX + 4u * c, sY, nvalid, last_s[set][stage], recv_s[set][stage], g.factor, g.out + c);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(acc_free);
        mbar_arrive(st_free + 8u * stage);
      }
      advance();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, 512);
}

int encode_half_rows_tensor_map(CUtensorMap *tmap, const void *base, int64_t rows, int box_rows, const char *what);

int fused_messages(const float *X, const float *Y, const void *h, const void *W, float factor, const int32_t *sender,
                   const int32_t *receiver, const int32_t *row_ptr, int64_t nnodes, int64_t nedges, float *out,
                   int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(messages)";
  if (nnodes == 0) return CMACE_OK;
  if (nedges == 0) {
    cudaError_t e = cudaMemsetAsync(out, 0, (size_t)nnodes * 16 * FM_C * sizeof(float), st);
    return e == cudaSuccess ? CMACE_OK : fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  }
  FusedMessagesArgs g{X, Y, static_cast<const uint4 *>(W), sender, receiver, row_ptr, status, nnodes, nedges, factor, out};
  CUtensorMap map;
  if (int rc = encode_half_rows_tensor_map(&map, h, nedges, FF_TILE, what)) return rc;
  const size_t smem = (size_t)FM_SETS * FF_STAGES * FF_STAGE_BYTES + 1024;
  cudaError_t e = cudaFuncSetAttribute(fused_messages_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  int64_t blocks = (nnodes + FM_SETS - 1) / FM_SETS;
  if (blocks > 148) blocks = 148;
  fused_messages_kernel<<<(unsigned)blocks, FM_THREADS, smem, st>>>(g, map);
  return check_launch(what);
}

// ---- backward -------------------------------------------------------------------------------------------------------
// With u_l[e, c] = sum_m Y[lm, e] G[i, lm, c] (G the gradient of the messages) an edge's results are
//
//   T[e, c] = sum_l R_l u_l,   grad Y[lm, e] = sum_c X R_l G[lm],   dE/dr = sum_c X sum_l R'_l u_l,   R' = h' W,
//
// so neither R nor the gradient of R nor that of h exists in memory.  A tile is 16 edges: rows of the B images are 16 rows
// of h followed by 16 of h', and one set of products gives R and R'.  The quarters with l = 1, 2 pass their part of T and
// of sum_l R'_l u_l through shared memory to the quarters with l = 3, 0 of the same channels.  Sums over channels: four
// edges' eight values a lane are 32 values for the 32 lanes (31 shuffles); two quarters' results are added in the end.
// dE/dr takes the place of component 0, whose gradient nobody needs (Y_00 is constant).
constexpr int FB_TILE = 16;
constexpr int FB_STAGES = 4;
constexpr int FB_X_BYTES = FB_TILE * FM_C * 4;
constexpr int FB_H_BYTES = 2 * 2 * FB_TILE * 128;     // hi image (h, h'), lo image (h, h')
constexpr int FB_Y_BYTES = FB_TILE * 64;
constexpr int FB_STAGE_BYTES = FB_X_BYTES + FB_H_BYTES + FB_Y_BYTES;
constexpr int FB_EX_BYTES = 2 * FB_TILE * 512;        // exchange of a set: [pair][edge][lane] float4
constexpr int FB_PART_FLOATS = 4 * FB_TILE * 8;       // sums of a set: [quarter][edge][8], two buffers
constexpr int FB_SET_BYTES = FB_STAGES * FB_STAGE_BYTES + FB_EX_BYTES + 2 * FB_PART_FLOATS * 4;

struct FusedBackArgs {
  const float *X, *Y, *G;        // [Ns, 128], [E, 16], [nnodes, 16, 128]
  const uint4 *W;
  const int32_t *sender, *receiver;
  int32_t *status;
  int64_t nnodes, nedges, tiles_per_block;
  float factor_v, factor_t;      // undo the powers of two of h W and h' W
  float *T, *gY;                 // [E, 128], [E, 16]
};

// v[i][m] (edge i of four, value m of eight) summed over the lanes: lane L ends with edge L >> 3, value L & 7
__device__ __forceinline__ float reduce_4x8(float (&v)[4][8], int lane) {
  float a[2][8], b[8], c[4], d[2];
  bool up = lane & 16;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int m = 0; m < 8; m++)
      a[i][m] = (up ? v[i + 2][m] : v[i][m]) + __shfl_xor_sync(0xffffffffu, up ? v[i][m] : v[i + 2][m], 16);
  up = lane & 8;
#pragma unroll
  for (int m = 0; m < 8; m++) b[m] = (up ? a[1][m] : a[0][m]) + __shfl_xor_sync(0xffffffffu, up ? a[0][m] : a[1][m], 8);
  up = lane & 4;
#pragma unroll
  for (int m = 0; m < 4; m++) c[m] = (up ? b[m + 4] : b[m]) + __shfl_xor_sync(0xffffffffu, up ? b[m] : b[m + 4], 4);
  up = lane & 2;
#pragma unroll
  for (int m = 0; m < 2; m++) d[m] = (up ? c[m + 2] : c[m]) + __shfl_xor_sync(0xffffffffu, up ? c[m] : c[m + 2], 2);
  up = lane & 1;
  return (up ? d[1] : d[0]) + __shfl_xor_sync(0xffffffffu, up ? d[0] : d[1], 1);
}

// G of a receiver: the eight components of this quarter, two channels
template <bool HIGH>
__device__ __forceinline__ void load_g(float2 (&g)[8], const float *__restrict__ G, int64_t node) {
#pragma unroll
  for (int m = 0; m < 8; m++) {
    const int lm = HIGH ? (m < 7 ? 9 + m : 0) : 1 + m;
    g[m] = __ldg(reinterpret_cast<const float2 *>(G + node * (16 * FM_C) + lm * FM_C));
  }
}

// grad Y of edges s0 .. s1 - 1 of the tile (one receiver) into part [edge][8]
template <bool HIGH>
__device__ __forceinline__ void back_grad_y(const float2 (&g)[8], uint32_t ta, uint32_t sX, int s0, int s1, float factor,
                                            float *part, int lane) {
#pragma unroll 1
  for (int at = s0 & ~3; at < s1; at += 4) {   // aligned groups of four edges, those outside the segment count as zero
    uint32_t r[4][4];
#pragma unroll
    for (int j = 0; j < (HIGH ? 2 : 4); j++) tmem_ld4_nowait(ta + 32u * j + (uint32_t)at, r[j]);
    float2 x[4];
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = lds2(sX + 512u * (uint32_t)(at + i));
    tmem_ld_wait();
    float v[4][8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const bool in = at + i >= s0 && at + i < s1;
      const float xa = in ? x[i].x : 0.f, xb = in ? x[i].y : 0.f;
      const float pa = xa * __uint_as_float(r[0][i]), pb = xb * __uint_as_float(r[1][i]);
      if (HIGH) {
#pragma unroll
        for (int m = 0; m < 7; m++) v[i][m] = fmaf(pa, g[m].x, pb * g[m].y);
        v[i][7] = 0.f;
      } else {
        const float qa = xa * __uint_as_float(r[2][i]), qb = xb * __uint_as_float(r[3][i]);
#pragma unroll
        for (int m = 0; m < 8; m++) v[i][m] = m < 3 ? fmaf(pa, g[m].x, pb * g[m].y) : fmaf(qa, g[m].x, qb * g[m].y);
      }
    }
    const float sum = reduce_4x8(v, lane) * factor;
    const int e = at + (lane >> 3);
    if (e >= s0 && e < s1 && !(HIGH && (lane & 7) == 7)) part[e * 8 + (lane & 7)] = sum;
  }
}

// this quarter's part of T and of sum_l R'_l u_l, edges s0 .. s1 - 1.  l = 1, 2: into the exchange; l = 3, 0: added to
// the partner's, T stored, and the channels' sum of X times the other into slot 7 of part
template <bool HIGH>
__device__ __forceinline__ void back_products(const float2 (&g)[8], uint32_t ta, uint32_t sX, uint32_t sY, uint32_t ex,
                                              int s0, int s1, float factor_v, float factor_t, float *T, float *part,
                                              int lane) {
#pragma unroll 1
  for (int at = s0 & ~3; at < s1; at += 4) {
    uint32_t r[4][4], d[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      tmem_ld4_nowait(ta + 32u * j + (uint32_t)at, r[j]);
      tmem_ld4_nowait(ta + 32u * j + 16u + (uint32_t)at, d[j]);
    }
    tmem_ld_wait();
    float dr[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      dr[i] = 0.f;
      if (at + i >= s0 && at + i < s1) {
        const uint32_t ya = sY + 64u * (uint32_t)(at + i);
        float y[8];
        float ua, ub, wa, wb;   // u of the first two blocks' degree and of the other two's
        if (HIGH) {
          const float4 u = lds4(ya + 32u), v = lds4(ya + 48u);
          y[0] = u.y; y[1] = u.z; y[2] = u.w; y[3] = v.x; y[4] = v.y; y[5] = v.z; y[6] = v.w;
          ua = y[0] * g[0].x;
          ub = y[0] * g[0].y;
#pragma unroll
          for (int m = 1; m < 7; m++) {
            ua = fmaf(y[m], g[m].x, ua);
            ub = fmaf(y[m], g[m].y, ub);
          }
          wa = g[7].x;
          wb = g[7].y;
        } else {
          const float4 u = lds4(ya), v = lds4(ya + 16u);
          y[0] = u.y; y[1] = u.z; y[2] = u.w; y[3] = v.x; y[4] = v.y; y[5] = v.z; y[6] = v.w;
          y[7] = lds1(ya + 32u);
          ua = y[0] * g[0].x;
          ub = y[0] * g[0].y;
          wa = y[3] * g[3].x;
          wb = y[3] * g[3].y;
#pragma unroll
          for (int m = 1; m < 3; m++) {
            ua = fmaf(y[m], g[m].x, ua);
            ub = fmaf(y[m], g[m].y, ub);
          }
#pragma unroll
          for (int m = 4; m < 8; m++) {
            wa = fmaf(y[m], g[m].x, wa);
            wb = fmaf(y[m], g[m].y, wb);
          }
        }
        const float t0 = fmaf(__uint_as_float(r[0][i]), ua, __uint_as_float(r[2][i]) * wa);
        const float t1 = fmaf(__uint_as_float(r[1][i]), ub, __uint_as_float(r[3][i]) * wb);
        const float v0 = fmaf(__uint_as_float(d[0][i]), ua, __uint_as_float(d[2][i]) * wa);
        const float v1 = fmaf(__uint_as_float(d[1][i]), ub, __uint_as_float(d[3][i]) * wb);
        const uint32_t xa = ex + 512u * (uint32_t)(at + i) + 16u * lane;
        if (HIGH) {
          const float4 o = lds4(xa);
          const float2 x = lds2(sX + 512u * (uint32_t)(at + i));
          *reinterpret_cast<float2 *>(T + (int64_t)(at + i) * FM_C) = make_float2((t0 + o.x) * factor_v, (t1 + o.y) * factor_v);
          dr[i] = fmaf(x.x, v0 + o.z, x.y * (v1 + o.w));
        } else {
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(xa), "f"(t0), "f"(t1), "f"(v0), "f"(v1) : "memory");
        }
      }
    }
    if (HIGH) {   // four sums over the lanes: lane 8 k ends with edge k's
      bool up = lane & 16;
      const float a0 = (up ? dr[2] : dr[0]) + __shfl_xor_sync(0xffffffffu, up ? dr[0] : dr[2], 16);
      const float a1 = (up ? dr[3] : dr[1]) + __shfl_xor_sync(0xffffffffu, up ? dr[1] : dr[3], 16);
      up = lane & 8;
      float b = (up ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up ? a0 : a1, 8);
      b += __shfl_xor_sync(0xffffffffu, b, 4);
      b += __shfl_xor_sync(0xffffffffu, b, 2);
      b += __shfl_xor_sync(0xffffffffu, b, 1);
      const int e = at + (lane >> 3);
      if ((lane & 7) == 0 && e >= s0 && e < s1) part[e * 8 + 7] = b * factor_t;
    }
  }
}

// barrier of a set's 128 consumer threads; true when `ok` holds for all of them
__device__ __forceinline__ bool set_barrier(int set, bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"(ok ? 1u : 0u), "r"(5 + set)
      : "memory");
  return all != 0;
}

// the quarters' sums of a tile to grad Y [16 edges][16]: component 0 is dE/dr (slot 7 of quarters 0 and 1), 1 .. 8 come
// from quarters 2 and 3, 9 .. 15 from 0 and 1
__device__ __forceinline__ void back_combine(const float *pt, float *__restrict__ gY, int nvalid, int thread) {
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int i = thread * 2 + u, e = i >> 4, lm = i & 15;
    const int from = lm >= 1 && lm <= 8 ? 2 : 0, slot = lm == 0 ? 7 : (lm <= 8 ? lm - 1 : lm - 9);
    const float v = pt[from * (FB_TILE * 8) + e * 8 + slot] + pt[(from + 1) * (FB_TILE * 8) + e * 8 + slot];
    if (e < nvalid) gY[i] = v;
  }
}

struct BackBars {
  uint32_t x_full, st_free, acc_full, acc_free;
};

template <bool HIGH>
__device__ __forceinline__ void back_consume(const FusedBackArgs &g, int64_t tile0, int64_t tile1, int set, int q, int lane,
                                             uint32_t stages, uint32_t ex, float *part, uint32_t acc_t, const BackBars &bar,
                                             const int32_t (*recv_s)[FB_TILE]) {
  const int c = 64 * (q & 1) + 2 * lane;
  const uint32_t ta = acc_t + ((uint32_t)(32 * q) << 16);
  float2 gr[8], gn[8];            // this receiver's and (expected) next receiver's G
#pragma unroll
  for (int m = 0; m < 8; m++) gr[m] = gn[m] = make_float2(0.f, 0.f);
  int64_t node = -1, next = -1;
  int stage = 0;
  uint32_t phase = 0;
  int64_t k = 0, last_base = 0;
  for (int64_t t = tile0 + set; t < tile1; t += FM_SETS, k++) {
    const bool ok = warp_wait(bar.x_full + 8u * stage, phase, lane) && warp_wait(bar.acc_full, (uint32_t)k & 1u, lane);
    if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 53);
    // one barrier a tile: the four quarters go on, or give up, together; and the previous tile's sums are complete
    if (!set_barrier(set, ok)) return;
    if (k > 0)
      back_combine(part + ((k - 1) & 1) * FB_PART_FLOATS, g.gY + (t - FM_SETS) * (FB_TILE * 16), FB_TILE, q * 32 + lane);
    tc_fence_after();
    const int64_t base = t * FB_TILE;
    const int nvalid = (int)(g.nedges - base < FB_TILE ? g.nedges - base : FB_TILE);
    const uint32_t sX = stages + (uint32_t)stage * FB_STAGE_BYTES + 4u * c;
    const uint32_t sY = stages + (uint32_t)stage * FB_STAGE_BYTES + FB_X_BYTES + FB_H_BYTES;
    const uint32_t exq = ex + (uint32_t)(q & 1) * (FB_EX_BYTES / 2);
    // two buffers: the barrier keeps the writers of one a tile behind its readers
    float *pt = part + (k & 1) * FB_PART_FLOATS + q * (FB_TILE * 8);
    const int mine = recv_s[stage][lane & (FB_TILE - 1)];   // receiver of edge `lane`
    float *T = g.T + base * FM_C + c;
    for (int s0 = 0; s0 < nvalid;) {
      // edges of one receiver: s0 .. s1 - 1 (the list is sorted)
      const int r = __shfl_sync(0xffffffffu, mine, s0);
      const unsigned same = __ballot_sync(0xffffffffu, lane >= s0 && lane < nvalid && mine == r);
      int s1 = 32 - __clz(same);
      s1 = s1 > s0 ? s1 : s0 + 1;
      if (r != node) {
        if (r == next) {
#pragma unroll
          for (int m = 0; m < 8; m++) gr[m] = gn[m];
        } else {
          load_g<HIGH>(gr, g.G + c, r);
        }
        node = r;
        next = r + 1 < g.nnodes ? r + 1 : -1;
        if (next >= 0) load_g<HIGH>(gn, g.G + c, next);
      }
      // the two quarters of a channel range meet once a segment
      if (HIGH) {
        back_grad_y<true>(gr, ta, sX, s0, s1, g.factor_v, pt, lane);
        asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * set + (q & 1)) : "memory");
        back_products<true>(gr, ta, sX, sY, exq, s0, s1, g.factor_v, g.factor_t, T, pt, lane);
      } else {
        back_products<false>(gr, ta, sX, sY, exq, s0, s1, g.factor_v, g.factor_t, T, pt, lane);
        asm volatile("bar.sync %0, 64;" ::"r"(1 + 2 * set + (q & 1)) : "memory");
        back_grad_y<false>(gr, ta, sX, s0, s1, g.factor_v, pt, lane);
      }
      s0 = s1;
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(bar.acc_free);
      mbar_arrive(bar.st_free + 8u * stage);
    }
    last_base = base;
    if (++stage == FB_STAGES) {
      stage = 0;
      phase ^= 1;
    }
  }
  if (k > 0) {
    set_barrier(set, true);
    const int64_t left = g.nedges - last_base;
    back_combine(part + ((k - 1) & 1) * FB_PART_FLOATS, g.gY + last_base * 16, (int)(left < FB_TILE ? left : FB_TILE),
                 q * 32 + lane);
  }
}

__global__ void __launch_bounds__(FM_THREADS, 1)
    fused_messages_back_kernel(const FusedBackArgs g, const __grid_constant__ CUtensorMap h_map,
                               const __grid_constant__ CUtensorMap dh_map) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[FM_SETS][3 * FB_STAGES + 2];
  __shared__ int32_t recv_s[FM_SETS][FB_STAGES][FB_TILE];
  __shared__ uint32_t tmem_base_slot;

  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int set = warp < 8 ? warp >> 2 : warp & 1;
  const uint32_t h_full = smem_u32(&bars[set][0]);
  const BackBars bar{h_full + 8u * FB_STAGES, h_full + 16u * FB_STAGES, h_full + 24u * FB_STAGES, h_full + 24u * FB_STAGES + 8u};
  const uint32_t stages = smem_base + (uint32_t)set * (FB_STAGES * FB_STAGE_BYTES);
  const uint32_t ex = smem_base + FM_SETS * FB_STAGES * FB_STAGE_BYTES + (uint32_t)set * FB_EX_BYTES;
  float *part = reinterpret_cast<float *>(smem + (smem_base - smem_u32(smem)) + FM_SETS * FB_STAGES * FB_STAGE_BYTES +
                                          FM_SETS * FB_EX_BYTES) +
                set * 2 * FB_PART_FLOATS;

  if (tid == 0) {
    for (int k = 0; k < FM_SETS; k++) {
      const uint32_t b = smem_u32(&bars[k][0]);
      for (int s = 0; s < FB_STAGES; s++) {
        mbar_init(b + 8u * s, 1);
        mbar_init(b + 8u * (FB_STAGES + s), 33);
        mbar_init(b + 8u * (2 * FB_STAGES + s), 4);
      }
      mbar_init(b + 8u * (3 * FB_STAGES), 1);
      mbar_init(b + 8u * (3 * FB_STAGES + 1), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot, acc_t = tmem + 256u + 128u * (uint32_t)set;
  if (warp < 4) load_w_tmem(g.W, tmem, warp, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const int64_t ntiles = (g.nedges + FB_TILE - 1) / FB_TILE;
  const int64_t tile0 = (int64_t)blockIdx.x * g.tiles_per_block;
  const int64_t tile1 = tile0 + g.tiles_per_block < ntiles ? tile0 + g.tiles_per_block : ntiles;
  int stage = 0;
  uint32_t phase = 0;
  auto advance = [&]() {
    if (++stage == FB_STAGES) {
      stage = 0;
      phase ^= 1;
    }
  };

  if (warp >= 10) {
    // ---- loader
    for (int64_t t = tile0 + set; t < tile1; t += FM_SETS) {
      if (!warp_wait(bar.st_free + 8u * stage, phase ^ 1, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 51);
        break;
      }
      const int64_t base = t * FB_TILE;
      const int l16 = lane & 15;
      const int64_t e = base + l16 < g.nedges ? base + l16 : g.nedges - 1;
      const uint32_t sX = stages + (uint32_t)stage * FB_STAGE_BYTES, sH = sX + FB_X_BYTES, sY = sH + FB_H_BYTES;
      if (lane == 0) {
        mbar_arrive_expect_tx(h_full + 8u * stage, FB_H_BYTES);
        tma_load_2d(sH, &h_map, 0, (int)base, h_full + 8u * stage);
        tma_load_2d(sH + FB_TILE * 128, &dh_map, 0, (int)base, h_full + 8u * stage);
        tma_load_2d(sH + FB_H_BYTES / 2, &h_map, 64, (int)base, h_full + 8u * stage);
        tma_load_2d(sH + FB_H_BYTES / 2 + FB_TILE * 128, &dh_map, 64, (int)base, h_full + 8u * stage);
      }
      const int s = g.sender[e];
      if (lane < FB_TILE) recv_s[set][stage][lane] = g.receiver[e];
      __syncwarp();
      if (lane == 0) {
        const uint32_t bytes = (uint32_t)(g.nedges - base < FB_TILE ? g.nedges - base : FB_TILE) * 64u;
        mbar_arrive_expect_tx(bar.x_full + 8u * stage, bytes);
        bulk_copy_g2s(sY, g.Y + base * 16, bytes, bar.x_full + 8u * stage);
      }
      copy_sender_rows<FB_TILE>(g.X, s, sX, bar.x_full + 8u * stage, lane);
      advance();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= 8) {
    // ---- MMA issuer
    uint32_t k = 0;
    for (int64_t t = tile0 + set; t < tile1; t += FM_SETS, k++) {
      if (!warp_wait(bar.acc_free, (k & 1u) ^ 1u, lane) || !warp_wait(h_full + 8u * stage, phase, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 52);
        break;
      }
      if (lane == 0) {
        tc_fence_after();
        issue_tile(tmem, acc_t, stages + (uint32_t)stage * FB_STAGE_BYTES + FB_X_BYTES, FB_H_BYTES / 2);
        umma_commit(bar.acc_full);
      }
      __syncwarp();
      advance();
    }
  } else if ((warp & 3) < 2) {
    back_consume<true>(g, tile0, tile1, set, warp & 3, lane, stages, ex, part, acc_t, bar, recv_s[set]);
  } else {
    back_consume<false>(g, tile0, tile1, set, warp & 3, lane, stages, ex, part, acc_t, bar, recv_s[set]);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, 512);
}

int fused_messages_back(const float *X, const float *Y, const float *G, const void *h, const void *dh, const void *W,
                        float factor_v, float factor_t, const int32_t *sender, const int32_t *receiver, int64_t nnodes,
                        int64_t nedges, float *T, float *gY, int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(edges_back)";
  if (nedges == 0) return CMACE_OK;
  const int64_t ntiles = (nedges + FB_TILE - 1) / FB_TILE;
  if (ntiles * FB_TILE > 0x7fffffffLL) return fail(CMACE_ERR_UNSUPPORTED, "%s: too many edges", what);
  FusedBackArgs g{X, Y, G, static_cast<const uint4 *>(W), sender, receiver, status, nnodes, nedges, (ntiles + 147) / 148,
                  factor_v, factor_t, T, gY};
  CUtensorMap h_map, dh_map;
  if (int rc = encode_half_rows_tensor_map(&h_map, h, nedges, FB_TILE, what)) return rc;
  if (int rc = encode_half_rows_tensor_map(&dh_map, dh, nedges, FB_TILE, what)) return rc;
  const size_t smem = (size_t)FM_SETS * FB_SET_BYTES + 1024;
  cudaError_t e = cudaFuncSetAttribute(fused_messages_back_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  const int64_t blocks = (ntiles + g.tiles_per_block - 1) / g.tiles_per_block;
  fused_messages_back_kernel<<<(unsigned)blocks, FM_THREADS, smem, st>>>(g, h_map, dh_map);
  return check_launch(what);
}

}  // namespace cmace
