// Second layer's message passing with the radial weights formed where they are used (float32, 128 channels; backward in
// fused_messages_back.cu):
//
//   m[i, lm, c] = sum_{e -> i} Y[lm, e] X[s(e), c] R_l[e, c],   R_l[e, c] = sum_k h[e, k] W[k, l, c].
//
// The unfused form writes R [E, 512] (2 KB an edge) with a product and reads it in the scatter.  Here
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
// wavefronts of Y instead of 64.
//
// A set's loader has to keep up with four consumer warps: its part of the list is in registers a tile ahead, a lane's rows are
// its own (a shuffle per row: 112 cycles a copy instead of about 30), and the MMAs come from one thread that asks its barriers
// itself.  317 -> 254 us at 16 000 atoms (833 000 edges), 1 320 -> 1 046 at 64 000, 80 -> 66 at 3 000, 264 -> 240 for 412 000
// edges of 4 a receiver, 294 -> 300 of 3 (events around the kernel, both in one run).  One copy instruction writes 64 bytes of
// eight rows, all on the same 16 banks, eight wavefronts instead of four; without that conflict (128 bytes of four rows) the
// kernel takes the same at 16 000 atoms, with the 64 bytes rotated by the row 259 us.
//
// What bounds it now: a set's products and sums take turns on one accumulator buffer.  Of 254 us at 16 000 atoms 182 remain
// without the products, 125 without the sums, 86 without both; of 1 046 at 64 000 744, 500 and 297.
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
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
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
  grid_wait();
  if (tid <= FM_SETS) {
    const int64_t pieces = (int64_t)gridDim.x * FM_SETS, b = (int64_t)blockIdx.x * FM_SETS + tid;
    const int64_t per = (g.nedges + pieces - 1) / pieces;
    range_s[tid] = b >= pieces ? g.nnodes : (b == 0 ? 0 : first_node_at(g.row_ptr, g.nnodes, b * per));
  }
  if (warp == 8) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_release();   // after the allocation
  const uint32_t tmem = (uint32_t)uniform((int)tmem_base_slot), acc_t = tmem + 256u + 128u * (uint32_t)set;
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
    // ---- loader: h rows by TMA, Y rows as one bulk copy, sender rows by asynchronous copies (lane: rows lane / 4 + 8 i, of
    // every 64 bytes the 16 at lane % 4); the next tile's part of the list is on its way meanwhile
    const int rr = lane >> 2;
    int send[4], r = 0, rn = 0;
    auto load_list = [&](int64_t t) {
      const int64_t base = e0 + t * FF_TILE;
      auto at = [&](int64_t e) { return e < e1 ? e : e1 - 1; };
#pragma unroll
      for (int i = 0; i < 4; i++) send[i] = __ldg(g.sender + at(base + rr + 8 * i));
      r = __ldg(g.receiver + at(base + lane));
      rn = base + lane + 1 < e1 ? __ldg(g.receiver + base + lane + 1) : -1;
    };
    if (ntiles > 0) load_list(0);
    for (int64_t t = 0; t < ntiles; t++) {
      const int64_t base = e0 + t * FF_TILE;
      const unsigned last = __ballot_sync(0xffffffffu, base + lane < e1 && rn != r);
      const int receiver = r;
      const float *src[4];
#pragma unroll
      for (int i = 0; i < 4; i++) src[i] = g.X + (int64_t)send[i] * FM_C + 4 * (lane & 3);
      if (t + 1 < ntiles) load_list(t + 1);
      if (!warp_wait_all(st_free + 8u * stage, phase ^ 1, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 41);
        break;
      }
      const uint32_t sX = stages + (uint32_t)stage * FF_STAGE_BYTES, sH = sX + FF_X_BYTES, sY = sH + FF_H_BYTES;
      if (elect_one()) {
        mbar_arrive_expect_tx(h_full + 8u * stage, FF_H_BYTES);
        tma_load_2d(sH, &h_map, 0, (int)base, h_full + 8u * stage);
        tma_load_2d(sH + FF_H_BYTES / 2, &h_map, 64, (int)base, h_full + 8u * stage);
      }
      recv_s[set][stage][lane] = receiver;
      if (lane == 0) last_s[set][stage] = last;
      __syncwarp();
      if (elect_one()) {
        const uint32_t bytes = (uint32_t)(e1 - base < FF_TILE ? e1 - base : FF_TILE) * 64u;
        mbar_arrive_expect_tx(x_full + 8u * stage, bytes);
        bulk_copy_g2s(sY, g.Y + base * 16, bytes, x_full + 8u * stage);
      }
      const uint32_t dst = sX + 512u * (uint32_t)rr + 16u * (uint32_t)(lane & 3);
#pragma unroll
      for (int k = 0; k < 8; k++)
#pragma unroll
        for (int i = 0; i < 4; i++)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4096u * i + 64u * k), "l"(src[i] + 16 * k) : "memory");
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(x_full + 8u * stage) : "memory");
      advance();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= 8) {
    // ---- MMA issuer, one thread
    if (elect_one()) {
      bool ok = true;
      for (int64_t t = 0; t < ntiles; t++) {
        ok = mbar_wait(h_full + 8u * stage, phase) && mbar_wait(acc_free, ((uint32_t)t & 1u) ^ 1u);
        if (!ok) break;
        tc_fence_after();
        issue_tile(tmem, acc_t, stages + (uint32_t)stage * FF_STAGE_BYTES + FF_X_BYTES, FF_H_BYTES / 2);
        umma_commit(acc_full);
        advance();
      }
      if (!ok && g.status) atomicCAS(g.status, 0, 42);
    }
    __syncwarp();
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
      if (!warp_wait_all(x_full + 8u * stage, phase, lane) || !warp_wait_all(acc_full, (uint32_t)t & 1u, lane)) {
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
  launch_chained(fused_messages_kernel, (unsigned)blocks, FM_THREADS, smem, st, g, map);
  return check_launch(what);
}

}  // namespace cmace
