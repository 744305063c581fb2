// Second layer's message passing with the radial weights formed where they are used (float32; backward in
// fused_messages_back.cu):
//
//   m[i, lm, c] = sum_{e -> i} Y[lm, e] X[s(e), c] R_l[e, c],   R_l[e, c] = sum_k h[e, k] W[k, l, c].
//
// The unfused form writes R [E, 4 C] (2 KB an edge at 128 channels) with a product and reads it in the scatter.  Here
// R^T is the accumulator of a tcgen05.mma: rows of W^T are the tensor-memory lanes, a tile's edges its columns.  Both
// images of W^T (hi, lo) are the A operand and stay in tensor memory for the whole kernel: at 128 channels 4 blocks of 128
// rows x (32 + 32) columns; the accumulators of two independent sets of warps take the other 2 x 128 columns.  With A in tensor
// memory an MMA reads only 1 KB of h from shared memory, where the consumers need the bandwidth (with A in shared memory
// its 4 KB are what a narrow MMA waits for).
//
// What bounds the consumers is the shared-memory pipe: a value that a whole warp reads (Y) still costs a wavefront, and
// so does a shuffle.  A warp reaches 32 of the 128 lanes, and which (l, channel) rows those are is free: lane quarters 0
// and 1 hold l = 3 and l = 0, quarters 2 and 3 hold l = 1 and l = 2, two channels a lane, blocks (l, even), (l, odd),
// (l', even), (l', odd).  Every quarter then works for eight components of two channels a lane: an edge costs 32 + 2
// wavefronts of Y instead of 64.
//
// h and W are pairs of fp16 with a power of two each, also for narrow models, whose rows were float32 while their weights were written:
// a row is rounded by 4e-8 instead of 2.5e-8 (more for the small rows near the cutoff), and the error of forces and node energies
// against float64 stays what it was, 0.9997 +- 0.0003 of it over 48 systems at each of 32, 64 and 96 channels.
//
// Rows of h that two edges share (EdgeRows) come by the loader's asynchronous copies into the swizzled images, as fast as boxes
// of consecutive rows (256 and 254 us at 16 000 atoms; four rows an instruction by TMA, from a warp of its own, 281; at 32 channels
// 177 against 113).  The lanes' copies and the tensor core's reads are ordered by a proxy fence of the thread that issues the MMAs.
//
// A set's loader has to keep up with four consumer warps: its part of the list is in registers a tile ahead, a lane's rows are
// its own (a shuffle per row: 112 cycles a copy instead of about 30), and the MMAs come from one thread that asks its barriers
// itself.  317 -> 254 us at 16 000 atoms (833 000 edges), 1 320 -> 1 046 at 64 000, 80 -> 66 at 3 000, 264 -> 240 for 412 000
// edges of 4 a receiver, 294 -> 300 of 3 (events around the kernel, both in one run).  One copy instruction writes 64 bytes of
// eight rows, all on the same 16 banks, eight wavefronts instead of four; without that conflict (128 bytes of four rows) the
// kernel takes the same at 16 000 atoms, with the 64 bytes rotated by the row 259 us.
//
// What bounds it now, at 128 channels: a set's products and sums take turns on one accumulator buffer.  Of 254 us at 16 000 atoms
// 182 remain without the products, 125 without the sums, 86 without both; of 1 046 at 64 000 744, 500 and 297.
//
// Fewer channels leave tensor memory for more: at 64 a lane has one channel and W^T two blocks, so that three sets fit with two
// accumulator buffers each; at 32 W^T is one block of a degree a quarter, three sets on tiles of 64 edges.  An edge's Y costs as
// many wavefronts as at 128 channels, which bounds both.  Product, written weights and scatter together -> this kernel, us at
// 16 000 atoms of 52 edges: 261 -> 103 at 32 channels, 410 -> 133 at 64, 720 -> 282 at 96; 3 000 atoms: 67 -> 33, 96 -> 40,
// 139 -> 70.  Other shapes of the same, us at 16 000 atoms (sets, edges a tile, stages, accumulator buffers): 64 channels 3, 64, 2,
// 1: 139; 2, 32, 5, 3: 146; 2, 64, 3, 1: 162; 32 channels 3, 64, 2, 2: 105; 3, 32, 4, 2: 110; 2, 64, 3, 1: 125; 96 channels with
// three stages for four: 285.
#include "common.cuh"
#include "step_common.cuh"
#include "tc_ptx.cuh"

namespace cmace {

// Blocks of 128 rows of W^T and what a lane of them has.  128 and 96 channels: two channels a lane (rows beyond 96 are zero
// and their lanes store nothing).  64: one channel a lane, blocks l and l'.  32: one block, quarter q holds l = 3 - q.
// A set is a pipeline of its own: four consumer warps, an MMA warp, a loader warp.
template <int C>
struct FusedShape {
  static constexpr int BLOCKS = C == 32 ? 1 : (C == 64 ? 2 : 4);
  static constexpr int PER = C <= 64 ? 1 : 2;                   // channels of a lane
  static constexpr int SETS = C <= 64 ? 3 : 2;
  static constexpr int TILE = C == 32 ? 64 : 32;                // edges of a tile
  static constexpr int STAGES = C == 64 ? 4 : (C == 32 ? 2 : (C == 96 ? 4 : 3));
  static constexpr int ACCS = C == 64 ? 2 : 1;                  // accumulator buffers of a set
  static constexpr int THREADS = SETS * 6 * 32;
  static constexpr int X_BYTES = TILE * C * 4;                  // sender rows
  static constexpr int H_BYTES = 2 * TILE * 128;                // hi and lo image of h
  static constexpr int Y_BYTES = TILE * 64;
  static constexpr int STAGE_BYTES = X_BYTES + H_BYTES + Y_BYTES;
  static constexpr int SMEM = SETS * STAGES * STAGE_BYTES + 1024;
  static_assert(TILE == 32 || TILE == 64, "a tile's last edges are one or two words");
  static_assert(64 * BLOCKS + SETS * ACCS * BLOCKS * TILE <= 512, "tensor memory");
  static_assert(SMEM <= 225 * 1024, "shared memory");
  static_assert(STAGE_BYTES % 1024 == 0 && X_BYTES % 1024 == 0, "swizzled images start on 1024 bytes");
};

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

// W^T [BLOCKS * 128 rows][hi 64 | lo 64] fp16 into tensor memory: block j at columns 64 j (hi) and 64 j + 32 (lo); four warps
template <int BLOCKS>
__device__ __forceinline__ void load_w_tmem(const uint4 *__restrict__ W, uint32_t tmem, int q, int lane) {
  const uint4 *w = W + (int64_t)(32 * q + lane) * 16;
#pragma unroll 1
  for (int j = 0; j < BLOCKS; j++)
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

// the 12 products of a block and tile: D block j [128 x TILE] = W block j (hi, lo) times the TILE rows of the B images
template <int BLOCKS, int TILE>
__device__ __forceinline__ void issue_tile(uint32_t tmem, uint32_t acc, uint32_t sB) {
  const uint32_t idesc = umma_idesc_f16(128, TILE);
  const uint64_t b_hi = umma_desc_sw128(sB), b_lo = umma_desc_sw128(sB + TILE * 128);
#pragma unroll 1
  for (int j = 0; j < BLOCKS; j++) {
    const uint32_t d = acc + (uint32_t)(TILE * j), a = tmem + 64u * j;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      umma_f16_ts(d, a + 8u * k, b_hi + (uint64_t)(2 * k), idesc, k != 0);
      umma_f16_ts(d, a + 8u * k, b_lo + (uint64_t)(2 * k), idesc, 1);
      umma_f16_ts(d, a + 32u + 8u * k, b_hi + (uint64_t)(2 * k), idesc, 1);
    }
  }
}

// ---- forward --------------------------------------------------------------------------------------------------------
// A set owns a contiguous range of receivers, so no sum is split and none is atomic; its warps keep up to 16 sums a lane.
struct FusedMessagesArgs {
  const float *X, *Y;            // [Ns, C], [E, 16]
  const char *h;                 // rows of [hi 64 | lo 64] fp16
  const uint4 *W;                // permuted W^T
  const int32_t *sender, *receiver, *row_ptr, *row_of;   // row_of: an edge's row of h; null: its own
  int32_t *status;
  int64_t nnodes, nedges;
  float factor;                  // undoes the powers of two of h and W
  float *out;                    // [nnodes, 16, C]
};

// A lane's components: degree L0 from the first PER blocks, then degree L1 (or none) from the others
template <int L0, int L1>
struct Degrees {
  static constexpr int N0 = 2 * L0 + 1, N = N0 + (L1 < 0 ? 0 : 2 * L1 + 1);
  static __device__ __forceinline__ int lm(int m) { return m < N0 ? L0 * L0 + m : L1 * L1 + m - N0; }
};

// Y of an edge for a lane's components: of l = 3 and 0 components 9 .. 15 (Y_00 = 1), of l = 1 and 2 1 .. 8
template <int L0, int L1>
__device__ __forceinline__ void load_y(float (&y)[Degrees<L0, L1>::N], uint32_t ya) {
  if constexpr (L0 == 3) {
    const float4 u = lds4(ya + 32u), v = lds4(ya + 48u);
    y[0] = u.y; y[1] = u.z; y[2] = u.w; y[3] = v.x; y[4] = v.y; y[5] = v.z; y[6] = v.w;
    if constexpr (L1 == 0) y[7] = 1.f;
  } else if constexpr (L0 == 2) {
    const float4 v = lds4(ya + 16u);
    y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
    y[4] = lds1(ya + 32u);
  } else if constexpr (L0 == 1) {
    const float4 u = lds4(ya);
    y[0] = u.y; y[1] = u.z; y[2] = u.w;
    if constexpr (L1 == 2) {
      const float4 v = lds4(ya + 16u);
      y[3] = v.x; y[4] = v.y; y[5] = v.z; y[6] = v.w;
      y[7] = lds1(ya + 32u);
    }
  } else {
    y[0] = 1.f;
  }
}

// one edge into the sums of a lane (PER channels a component); r: its accumulators, degree L0 first
template <int L0, int L1, int PER>
__device__ __forceinline__ void add_edge(float (&acc)[Degrees<L0, L1>::N * PER], const float (&y)[Degrees<L0, L1>::N],
                                         const float (&x)[PER], const float (&r)[(L1 < 0 ? 1 : 2) * PER]) {
  using D = Degrees<L0, L1>;
  float p[2][PER];
#pragma unroll
  for (int c = 0; c < PER; c++) {
    p[0][c] = x[c] * r[c];
    if constexpr (L1 >= 0) p[1][c] = x[c] * r[PER + c];
  }
#pragma unroll
  for (int m = 0; m < D::N; m++)
#pragma unroll
    for (int c = 0; c < PER; c++) {
      const float v = p[m < D::N0 ? 0 : 1][c];
      if (D::lm(m) == 0) acc[m * PER + c] += v;
      else acc[m * PER + c] = fmaf(y[m], v, acc[m * PER + c]);
    }
}

// What a set's consumers do with one tile.  Eight edges at a time; without a receiver's last edge among them there is no
// branch, so that the loads of several edges are on their way before the first sum (with a branch per edge: 1.85 ms at
// 64 000 atoms and 128 channels instead of 1.55).  stores: whether the lane's channels exist.
template <int C, int L0, int L1>
__device__ __forceinline__ void forward_tile(float (&acc)[Degrees<L0, L1>::N * FusedShape<C>::PER], uint32_t ta, uint32_t sX,
                                             uint32_t sY, int nvalid, const uint32_t (&words)[FusedShape<C>::TILE / 32],
                                             const int32_t *recv, float factor,
                                             float *out, bool stores) {
  using S = FusedShape<C>;
  using D = Degrees<L0, L1>;
  constexpr int PER = S::PER, NB = (L1 < 0 ? 1 : 2) * PER;
#pragma unroll 1
  for (int i0 = 0; i0 < nvalid; i0 += 8) {
    const uint32_t last = (S::TILE == 32 || i0 < 32 ? words[0] : words[S::TILE / 32 - 1]) >> (i0 & 31);
    uint32_t r[NB][8];
#pragma unroll
    for (int j = 0; j < NB; j++) tmem_ld8_nowait(ta + (uint32_t)(S::TILE * j + i0), r[j]);
    float x[8][PER];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if constexpr (PER == 2) {
        const float2 v = lds2(sX + (uint32_t)(4 * C * (i0 + i)));
        x[i][0] = v.x;
        x[i][1] = v.y;
      } else {
        x[i][0] = lds1(sX + (uint32_t)(4 * C * (i0 + i)));
      }
    }
    auto add = [&](const float (&y)[D::N], int i) {
      float rr[NB];
#pragma unroll
      for (int j = 0; j < NB; j++) rr[j] = __uint_as_float(r[j][i]);
      add_edge<L0, L1, PER>(acc, y, x[i], rr);
    };
    const uint32_t ya = sY + 64u * (uint32_t)i0;
    if (nvalid - i0 >= 8 && (last & 0xffu) == 0) {
      float y[4][D::N];
#pragma unroll
      for (int i = 0; i < 4; i++) load_y<L0, L1>(y[i], ya + 64u * i);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; i++) {
        add(y[i], i);
        load_y<L0, L1>(y[i], ya + 64u * (4 + i));
      }
#pragma unroll
      for (int i = 0; i < 4; i++) add(y[i], 4 + i);
    } else {
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (i0 + i < nvalid) {
          float y[D::N];
          load_y<L0, L1>(y, ya + 64u * i);
          add(y, i);
          if ((last >> i) & 1u) {
            float *o = out + (int64_t)recv[i0 + i] * (16 * C);
#pragma unroll
            for (int m = 0; m < D::N; m++) {
              if constexpr (PER == 2) {
                if (C == 128 || stores)
                  *reinterpret_cast<float2 *>(o + D::lm(m) * C) = make_float2(acc[2 * m] * factor, acc[2 * m + 1] * factor);
                acc[2 * m] = acc[2 * m + 1] = 0.f;
              } else {
                o[D::lm(m) * C] = acc[m] * factor;
                acc[m] = 0.f;
              }
            }
          }
        }
      }
    }
  }
}

template <int C>
__global__ void __launch_bounds__(FusedShape<C>::THREADS, 1)
    fused_messages_kernel(const FusedMessagesArgs g, const __grid_constant__ CUtensorMap h_map) {
  using S = FusedShape<C>;
  constexpr int SETS = S::SETS, STAGES = S::STAGES, TILE = S::TILE, ACCS = S::ACCS;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[SETS][3 * STAGES + 2 * ACCS];   // h landed, X / Y landed, stage free; acc full, free
  __shared__ int32_t recv_s[SETS][STAGES][TILE];
  __shared__ uint32_t last_s[SETS][STAGES][TILE / 32];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int64_t range_s[SETS + 1];

  const uint32_t smem_base = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  // warps 0-3, 4-7, ..: consumers of sets 0, 1, ..; then the sets' MMA warps, then their loaders
  constexpr int MMA0 = 4 * SETS, LOADER0 = 5 * SETS;
  const int set = warp < MMA0 ? warp >> 2 : (warp - MMA0) % SETS;
  const uint32_t h_full = smem_u32(&bars[set][0]), x_full = h_full + 8u * STAGES, st_free = x_full + 8u * STAGES;
  const uint32_t acc_full = st_free + 8u * STAGES, acc_free = acc_full + 8u * ACCS;
  const uint32_t stages = smem_base + (uint32_t)(set * STAGES) * S::STAGE_BYTES;

  if (tid == 0) {
    for (int k = 0; k < SETS; k++) {
      const uint32_t b = smem_u32(&bars[k][0]);
      for (int s = 0; s < STAGES; s++) {
        mbar_init(b + 8u * s, g.row_of ? 32 : 1);      // h: the loader's lanes, or its expect_tx
        mbar_init(b + 8u * (STAGES + s), 33);          // the loader's 32 lanes and its expect_tx
        mbar_init(b + 8u * (2 * STAGES + s), 4);
      }
      for (int a = 0; a < ACCS; a++) {
        mbar_init(b + 8u * (3 * STAGES + a), 1);
        mbar_init(b + 8u * (3 * STAGES + ACCS + a), 4);
      }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid <= SETS) {
    const int64_t pieces = (int64_t)gridDim.x * SETS, b = (int64_t)blockIdx.x * SETS + tid;
    const int64_t per = (g.nedges + pieces - 1) / pieces;
    range_s[tid] = b >= pieces ? g.nnodes : (b == 0 ? 0 : first_node_at(g.row_ptr, g.nnodes, b * per));
  }
  if (warp == MMA0) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)uniform((int)tmem_base_slot), acc_t = tmem + 64u * S::BLOCKS + (uint32_t)(set * ACCS * S::BLOCKS * TILE);
  if (warp < 4) load_w_tmem<S::BLOCKS>(g.W, tmem, warp, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_wait();      // the list and the weights are older than the kernel before
  grid_release();   // after the allocation

  const int64_t n0 = range_s[set], n1 = range_s[set + 1];
  const int64_t e0 = n0 < n1 ? g.row_ptr[n0] : 0, e1 = n0 < n1 ? g.row_ptr[n1] : 0;
  const int64_t ntiles = (e1 - e0 + TILE - 1) / TILE;
  int stage = 0, at_acc = 0;
  uint32_t phase = 0, acc_phase = 0;
  auto advance = [&]() {
    if (++stage == STAGES) {
      stage = 0;
      phase ^= 1;
    }
    if (++at_acc == ACCS) {
      at_acc = 0;
      acc_phase ^= 1;
    }
  };

  if (warp >= LOADER0) {
    // ---- loader: Y rows as one bulk copy, sender rows by asynchronous copies (lane: rows lane / 4 + 8 i, of every 64 bytes
    // the 16 at lane % 4); rows of h the same way into the swizzled images, or as two boxes where an edge has a row of its own;
    // the next tile's part of the list is on its way meanwhile
    const int rr = lane >> 2;
    constexpr int ROWS = TILE / 8, WORDS = TILE / 32;
    int send[ROWS], hrow[ROWS], r[WORDS], rn[WORDS];
    auto load_list = [&](int64_t t) {
      const int64_t base = e0 + t * TILE;
      auto at = [&](int64_t e) { return e < e1 ? e : e1 - 1; };
#pragma unroll
      for (int i = 0; i < ROWS; i++) send[i] = __ldg(g.sender + at(base + rr + 8 * i));
      if (g.row_of) {
#pragma unroll
        for (int i = 0; i < ROWS; i++) hrow[i] = __ldg(g.row_of + at(base + rr + 8 * i));
      }
#pragma unroll
      for (int k = 0; k < WORDS; k++) {
        const int64_t e = base + 32 * k + lane;
        r[k] = __ldg(g.receiver + at(e));
        rn[k] = e + 1 < e1 ? __ldg(g.receiver + e + 1) : -1;
      }
    };
    if (ntiles > 0) load_list(0);
    for (int64_t t = 0; t < ntiles; t++) {
      const int64_t base = e0 + t * TILE;
      unsigned last[WORDS];
      int receiver[WORDS];
#pragma unroll
      for (int k = 0; k < WORDS; k++) {
        last[k] = __ballot_sync(0xffffffffu, base + 32 * k + lane < e1 && rn[k] != r[k]);
        receiver[k] = r[k];
      }
      const float *src[ROWS];
      const char *hsrc[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; i++) {
        src[i] = g.X + (int64_t)send[i] * C + 4 * (lane & 3);
        hsrc[i] = g.h + (int64_t)hrow[i] * 256 + 16 * (lane & 3);
      }
      if (t + 1 < ntiles) load_list(t + 1);
      if (!warp_wait_all(st_free + 8u * stage, phase ^ 1, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 41);
        break;
      }
      const uint32_t sX = stages + (uint32_t)stage * S::STAGE_BYTES, sH = sX + S::X_BYTES, sY = sH + S::H_BYTES;
      if (g.row_of) {
#pragma unroll
        for (int k = 0; k < 4; k++)   // 64 bytes of hi, 64 more, the same of lo
#pragma unroll
          for (int i = 0; i < ROWS; i++)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sH + (k >> 1) * (S::H_BYTES / 2) +
                                                                          (uint32_t)sw128_offset(rr + 8 * i, (lane & 3) + 4 * (k & 1))),
                         "l"(hsrc[i] + 64 * k)
                         : "memory");
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(h_full + 8u * stage) : "memory");
      } else if (elect_one()) {
        mbar_arrive_expect_tx(h_full + 8u * stage, S::H_BYTES);
        tma_load_2d(sH, &h_map, 0, (int)base, h_full + 8u * stage);
        tma_load_2d(sH + S::H_BYTES / 2, &h_map, 64, (int)base, h_full + 8u * stage);
      }
#pragma unroll
      for (int k = 0; k < WORDS; k++) {
        recv_s[set][stage][32 * k + lane] = receiver[k];
        if (lane == 0) last_s[set][stage][k] = last[k];
      }
      __syncwarp();
      if (elect_one()) {
        const uint32_t bytes = (uint32_t)(e1 - base < TILE ? e1 - base : TILE) * 64u;
        mbar_arrive_expect_tx(x_full + 8u * stage, bytes);
        bulk_copy_g2s(sY, g.Y + base * 16, bytes, x_full + 8u * stage);
      }
      const uint32_t dst = sX + (uint32_t)(4 * C * rr) + 16u * (uint32_t)(lane & 3);
#pragma unroll
      for (int k = 0; k < C / 16; k++)
#pragma unroll
        for (int i = 0; i < ROWS; i++)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 32u * C * i + 64u * k), "l"(src[i] + 16 * k) : "memory");
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(x_full + 8u * stage) : "memory");
      advance();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= MMA0) {
    // ---- MMA issuer, one thread
    if (elect_one()) {
      bool ok = true;
      for (int64_t t = 0; t < ntiles; t++) {
        ok = mbar_wait(h_full + 8u * stage, phase);
        if (g.row_of) fence_proxy_async();   // rows copied by the loader's lanes, read by the tensor core
        ok = ok && mbar_wait(acc_free + 8u * at_acc, acc_phase ^ 1u);
        if (!ok) break;
        tc_fence_after();
        issue_tile<S::BLOCKS, TILE>(tmem, acc_t + (uint32_t)(at_acc * S::BLOCKS * TILE),
                                    stages + (uint32_t)stage * S::STAGE_BYTES + S::X_BYTES);
        umma_commit(acc_full + 8u * at_acc);
        advance();
      }
      if (!ok && g.status) atomicCAS(g.status, 0, 42);
    }
    __syncwarp();
  } else {
    // ---- consumers
    const int q = warp & 3;
    const int c = C == 32 ? lane : (C == 64 ? 32 * (q & 1) + lane : 64 * (q & 1) + 2 * lane);
    const bool stores = c < C;
    const uint32_t sc = 4u * (uint32_t)(stores ? c : 0);
    auto consume = [&](auto first, auto second) {
      constexpr int L0 = decltype(first)::value, L1 = decltype(second)::value;
      using D = Degrees<L0, L1>;
      // receivers of this range without edges: their rows are zero
      for (int64_t n = n0; n < n1; n++)
        if (g.row_ptr[n] == g.row_ptr[n + 1])
          for (int m = 0; m < D::N; m++)
            if (stores)
#pragma unroll
              for (int v = 0; v < S::PER; v++) g.out[n * (16 * C) + D::lm(m) * C + c + v] = 0.f;
      float acc[D::N * S::PER];
#pragma unroll
      for (int m = 0; m < D::N * S::PER; m++) acc[m] = 0.f;
      for (int64_t t = 0; t < ntiles; t++) {
        if (!warp_wait_all(x_full + 8u * stage, phase, lane) || !warp_wait_all(acc_full + 8u * at_acc, acc_phase, lane)) {
          if (lane == 0 && g.status) atomicCAS(g.status, 0, 43);
          break;
        }
        tc_fence_after();
        const uint32_t sX = stages + (uint32_t)stage * S::STAGE_BYTES, sY = sX + S::X_BYTES + S::H_BYTES;
        uint32_t last[TILE / 32];
#pragma unroll
        for (int k = 0; k < TILE / 32; k++) last[k] = last_s[set][stage][k];
        const int64_t left = e1 - (e0 + t * TILE);
        const int nvalid = (int)(left < TILE ? left : TILE);
        forward_tile<C, L0, L1>(acc, acc_t + ((uint32_t)(32 * q) << 16) + (uint32_t)(at_acc * S::BLOCKS * TILE), sX + sc, sY, nvalid,
                                last, recv_s[set][stage], g.factor, g.out + c, stores);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(acc_free + 8u * at_acc);
          mbar_arrive(st_free + 8u * stage);
        }
        advance();
      }
    };
    using std::integral_constant;
    if constexpr (C == 32) {
      if (q == 0) consume(integral_constant<int, 3>{}, integral_constant<int, -1>{});
      else if (q == 1) consume(integral_constant<int, 2>{}, integral_constant<int, -1>{});
      else if (q == 2) consume(integral_constant<int, 1>{}, integral_constant<int, -1>{});
      else consume(integral_constant<int, 0>{}, integral_constant<int, -1>{});
    } else {
      if (q < 2) consume(integral_constant<int, 3>{}, integral_constant<int, 0>{});
      else consume(integral_constant<int, 1>{}, integral_constant<int, 2>{});
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA0) tmem_dealloc(tmem, 512);
}

int encode_half_rows_tensor_map(CUtensorMap *tmap, const void *base, int64_t rows, int box_rows, const char *what);

template <int C>
static int launch_fused_messages(const FusedMessagesArgs &g, const char *what, cudaStream_t st) {
  using S = FusedShape<C>;
  CUtensorMap map;
  if (int rc = encode_half_rows_tensor_map(&map, g.h, g.nedges, S::TILE, what)) return rc;
  cudaError_t e = cudaFuncSetAttribute(fused_messages_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  int64_t blocks = (g.nnodes + S::SETS - 1) / S::SETS;
  if (blocks > 148) blocks = 148;
  launch_chained(fused_messages_kernel<C>, (unsigned)blocks, S::THREADS, S::SMEM, st, g, map);
  return check_launch(what);
}

int fused_messages(const float *X, const float *Y, const void *h, const void *W, float factor, const int32_t *sender,
                   const int32_t *receiver, const int32_t *row_ptr, const int32_t *row_of, int64_t nnodes, int64_t nedges, int C,
                   float *out, int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(messages)";
  if (nnodes == 0) return CMACE_OK;
  if (nedges == 0) {
    cudaError_t e = cudaMemsetAsync(out, 0, (size_t)nnodes * 16 * C * sizeof(float), st);
    return e == cudaSuccess ? CMACE_OK : fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  }
  const FusedMessagesArgs g{X, Y, static_cast<const char *>(h), static_cast<const uint4 *>(W), sender, receiver, row_ptr, row_of,
                            status, nnodes, nedges, factor, out};
  switch (C) {
    case 32: return launch_fused_messages<32>(g, what, st);
    case 64: return launch_fused_messages<64>(g, what, st);
    case 96: return launch_fused_messages<96>(g, what, st);
    case 128: return launch_fused_messages<128>(g, what, st);
  }
  return fail(CMACE_ERR_UNSUPPORTED, "%s: no kernel for %d channels", what, C);
}

}  // namespace cmace
