// Backward of the second layer's message passing with the radial weights formed where they are used (float32, 128
// channels; forward in fused_messages.cu).  With u_l[e, c] = sum_m Y[lm, e] G[i, lm, c] (G the gradient of the messages,
// i the receiver of edge e) an edge's results are
//
//   T[e, c] = sum_l R_l u_l,   grad Y[lm, e] = sum_c X R_l G[lm],   dE/dr = sum_c X sum_l R'_l u_l,
//   R = h W,  R' = h' W,
//
// so neither R nor the gradients of R and h exist in memory.  Edges are the tensor-memory lanes: a thread owns an edge,
// every sum above runs over that thread's own values, no shuffles.  (With channels on the lanes, as in the forward, the
// sums over channels cost 31 shuffles per four edges and warp, and the kernel took 5.0 ms at 64 000 atoms.)
//
// Tile = 128 edges, taken 16 channels at a time by two sets of four consumer warps in turn, in steps of 8 channels: an
// accumulator buffer holds 32 (R, four l) + 32 (R') columns, two buffers a set, so that the products of a set's next step
// run while it works (with one buffer of 16 channels a set it waited for them: 2.35 against 2.13 ms at 64 000 atoms).
// A operand: h and h' (hi, lo fp16), 128 columns of tensor memory, two buffers; the consumers bring the next tile's rows
// over in quarters during a tile's first four steps.  B operand: 8 KB of W per step, streamed from L2 (every CTA reads the same
// 128 KB).  With A in tensor memory a narrow MMA runs at its own rate (16 cycles at N = 32).
//
//   warps 0-3, 4-7  the two sets of consumers; warp w reaches the rows 32 (w % 4) .. of the tile
//   warp 8          issues the MMAs
//   warp 9          W blocks and the G rows of the next tile's receivers (contiguous: the list is sorted), bulk copies
//   warp 10         sender rows X, 64 bytes of 128 rows per block, asynchronous copies
//
// What bounds it: the bytes that shared memory delivers to registers: a thread needs G[lm, c] of its receiver, 2048 words
// an edge, as warp-wide broadcasts (64 wavefronts an edge), next to the B operand (24), X, T and W (24).
#include "common.cuh"
#include "step_common.cuh"
#include "tc_ptx.cuh"

namespace cmace {

constexpr int EB_TILE = 128;
constexpr int EB_C = 128;
constexpr int EB_BLK = 16;                        // channels of a block
constexpr int EB_NBLK = EB_C / EB_BLK;
constexpr int EB_THREADS = 384;
constexpr int EB_STEP = 8;                        // channels of a step
constexpr int EB_NSTEP = EB_C / EB_STEP;
constexpr int EB_W_BYTES = 2 * 32 * 128;          // hi and lo image of a step's W: 32 rows (l, channel)
constexpr int EB_W_SLOTS = 6;
constexpr int EB_X_BYTES = EB_TILE * EB_BLK * 4;
constexpr int EB_X_SLOTS = 5;
// Receivers staged per tile; a warp with a further one reads G from global memory.  Five hold a tile of a condensed system: 0.57
// ns an edge at 52 edges a receiver, 0.68 at 31, 0.96 at 21, 1.07 at 10 (832 000 edges).  Two buffers of more do not fit.
constexpr int EB_G_RECV = 5;
constexpr int EB_G_BYTES = EB_G_RECV * 16 * EB_C * 4;
constexpr int EB_PIECE = 2048;                    // 32 rows x 64 bytes
constexpr int EB_PART = EB_TILE * 17;             // floats of a buffer of partial sums
constexpr int EB_OFF_W = 0;
constexpr int EB_OFF_X = EB_OFF_W + EB_W_SLOTS * EB_W_BYTES;
constexpr int EB_OFF_G = EB_OFF_X + EB_X_SLOTS * EB_X_BYTES;
constexpr int EB_OFF_T = EB_OFF_G + 2 * EB_G_BYTES;        // eight pieces: T of a warp on its way out
constexpr int EB_OFF_H = EB_OFF_T + 8 * EB_PIECE;          // eight pieces: h of the next tile on its way in
constexpr int EB_OFF_P = EB_OFF_H + 8 * EB_PIECE;
constexpr int EB_SMEM = EB_OFF_P + 2 * EB_PART * 4 + 1024;

struct EdgeBackArgs {
  const float *X, *Y, *G;        // [Ns, 128], [E, 16], [nnodes, 16, 128]
  const char *h, *dh;            // [E rounded up to a tile][hi 64 | lo 64] fp16
  const char *W;                 // [16 steps][hi, lo][32 rows x 128 B, swizzled]
  const int32_t *sender, *receiver;
  int32_t *status;
  int64_t nedges;
  float factor_v, factor_t;      // undo the powers of two of h W and h' W
  float *gY;                     // [E, 16]; component 0 is dE/dr (Y_00 is constant)
};

__device__ __forceinline__ void eb_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// the loads' registers go through the wait, so that nothing that reads them can be placed before it
__device__ __forceinline__ void eb_ld_wait(uint32_t (&r)[8], uint32_t (&d)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(d[0]),
                 "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7])::"memory");
}
__device__ __forceinline__ void eb_lds(uint32_t a, unsigned long long &x, unsigned long long &y) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ void eb_cp16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// eight channels of one edge: sums into gy2 (pairs of channels per component), dr2; returns T in t2
template <bool STAGED>
__device__ __forceinline__ void eb_half(uint32_t ta, uint32_t gs, const float *gg, const unsigned long long (&x2)[4],
                                        const float (&y)[16], unsigned long long (&gy2)[16], unsigned long long &dr2,
                                        unsigned long long (&t2)[4]) {
  unsigned long long v2[4];
  uint32_t r[2][8], d[2][8];
  eb_ld8(ta, r[0]);
  eb_ld8(ta + 32u, d[0]);
#pragma unroll
  for (int l = 0; l < 4; l++) {
    eb_ld_wait(r[l & 1], d[l & 1]);
    if (l < 3) {   // the next degree's accumulators are on their way meanwhile
      eb_ld8(ta + 8u * (l + 1), r[(l + 1) & 1]);
      eb_ld8(ta + 32u + 8u * (l + 1), d[(l + 1) & 1]);
    }
    unsigned long long u2[4], p2[4], r2[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      r2[c] = pack2(__uint_as_float(r[l & 1][2 * c]), __uint_as_float(r[l & 1][2 * c + 1]));
      if (l > 0) p2[c] = mul2(r2[c], x2[c]);
    }
#pragma unroll
    for (int m = l * l; m < (l + 1) * (l + 1); m++) {
      unsigned long long g2[4];
      if (STAGED) {
        eb_lds(gs + (uint32_t)(m * EB_C * 4), g2[0], g2[1]);
        eb_lds(gs + (uint32_t)(m * EB_C * 4) + 16u, g2[2], g2[3]);
      } else {
        const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2 *>(gg + m * EB_C));
        const ulonglong2 b = __ldg(reinterpret_cast<const ulonglong2 *>(gg + m * EB_C) + 1);
        g2[0] = a.x; g2[1] = a.y; g2[2] = b.x; g2[3] = b.y;
      }
      const unsigned long long yy = pack2(y[m], y[m]);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (l == 0) u2[c] = g2[c];                       // Y_00 = 1
        else u2[c] = m == l * l ? mul2(yy, g2[c]) : fma2(yy, g2[c], u2[c]);
        if (l > 0) gy2[m] = fma2(p2[c], g2[c], gy2[m]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const unsigned long long d2 = pack2(__uint_as_float(d[l & 1][2 * c]), __uint_as_float(d[l & 1][2 * c + 1]));
      t2[c] = l == 0 ? mul2(r2[c], u2[c]) : fma2(r2[c], u2[c], t2[c]);
      v2[c] = l == 0 ? mul2(d2, u2[c]) : fma2(d2, u2[c], v2[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < 4; c++) dr2 = fma2(x2[c], v2[c], dr2);
}

__global__ void __launch_bounds__(EB_THREADS, 1)
    edge_back_kernel(const EdgeBackArgs g, const __grid_constant__ CUtensorMap t_map) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[2 * EB_W_SLOTS + 2 * EB_X_SLOTS + 18];
  __shared__ uint32_t tmem_base_slot;

  const uint32_t base_s = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const uint32_t w_full = smem_u32(&bars[0]), w_free = w_full + 8u * EB_W_SLOTS;
  const uint32_t x_full = w_free + 8u * EB_W_SLOTS, x_free = x_full + 8u * EB_X_SLOTS;
  const uint32_t g_full = x_free + 8u * EB_X_SLOTS, g_free = g_full + 16u, h_full = g_free + 16u;
  const uint32_t acc_full = h_full + 16u, acc_free = acc_full + 32u, part_full = acc_free + 32u;

  if (tid == 0) {
    for (int s = 0; s < EB_W_SLOTS; s++) {
      mbar_init(w_full + 8u * s, 1);
      mbar_init(w_free + 8u * s, 1);     // the commit of the MMAs that read the slot
    }
    for (int s = 0; s < EB_X_SLOTS; s++) {
      mbar_init(x_full + 8u * s, 32);
      mbar_init(x_free + 8u * s, 4);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(g_full + 8u * b, 1);
      mbar_init(g_free + 8u * b, 8);
      mbar_init(h_full + 8u * b, 8);
    }
    for (int b = 0; b < 4; b++) {
      mbar_init(acc_full + 8u * b, 1);
      mbar_init(acc_free + 8u * b, 4);
      mbar_init(part_full + 8u * b, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_wait();
  if (warp == 8) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_release();   // after the allocation
  const uint32_t tmem = (uint32_t)uniform((int)tmem_base_slot);   // h buffer b at 128 b: h hi, h lo, h' hi, h' lo (32 each); acc b at 256 + 64 b
  const int64_t ntiles = (g.nedges + EB_TILE - 1) / EB_TILE;

  if (warp < 8) {
    // ---- consumers
    const int q = warp & 3, set = warp >> 2;
    const int row = 32 * q + lane;
    const uint32_t lanes = (uint32_t)(32 * q) << 16;
    const uint32_t sT = base_s + EB_OFF_T + (uint32_t)warp * EB_PIECE, sH = base_s + EB_OFF_H + (uint32_t)warp * EB_PIECE;
    float *part0 = reinterpret_cast<float *>(smem + (base_s - smem_u32(smem)) + EB_OFF_P) + row * 17;
    const char *hlane = (set == 0 ? g.h : g.dh) + (32 * q + (lane >> 2)) * 256 + 16 * (lane & 3);
    const uint32_t hdst = sH + (uint32_t)sw64_offset(lane >> 2, lane & 3);
    bool ok = true;

    // 64 bytes (32 k of hi or lo) of this warp's 32 rows of a tile: started here, finished by h_put
    auto h_start = [&](int64_t tile, int piece) {
      const char *src = hlane + tile * (EB_TILE * 256) + 64 * piece;
#pragma unroll
      for (int i = 0; i < 4; i++) eb_cp16(hdst + 512u * i, src + 8 * 256 * i);   // sw64_offset(r + 8, c) = sw64_offset(r, c) + 512
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto h_put = [&](int buf, int piece) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      uint32_t v[16];
#pragma unroll
      for (int c = 0; c < 4; c++)
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[4 * c]), "=r"(v[4 * c + 1]), "=r"(v[4 * c + 2]), "=r"(v[4 * c + 3])
                     : "r"(sH + (uint32_t)sw64_offset(lane, c))
                     : "memory");
      tmem_st16(tmem + lanes + 128u * (uint32_t)buf + 64u * (uint32_t)set + 16u * (uint32_t)piece, v);
      if (piece == 3) {
        tmem_st_wait();
        tc_fence_before();
      }
      __syncwarp();
    };

    if (blockIdx.x < ntiles)
      for (int p = 0; p < 4; p++) {
        h_start(blockIdx.x, p);
        h_put(0, p);
      }
    if (lane == 0) mbar_arrive(h_full);

    uint32_t k = 0;   // tiles done
    int xs = set;     // X slot of this set's next block: blocks are numbered through the tiles, this set takes every other
    uint32_t xphase = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int64_t base = tile * EB_TILE, e = base + row;
      const bool in = e < g.nedges;
      const int64_t ec = in ? e : g.nedges - 1;
      const int r_first = __ldg(g.receiver + base);
      const int my = __ldg(g.receiver + ec);
      float y[16];
      {
        const float4 *yp = reinterpret_cast<const float4 *>(g.Y + ec * 16);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float4 v = __ldg(yp + i);
          y[4 * i] = v.x; y[4 * i + 1] = v.y; y[4 * i + 2] = v.z; y[4 * i + 3] = v.w;
        }
      }
      const bool staged = __all_sync(0xffffffffu, my - r_first < EB_G_RECV);
      const uint32_t gs = base_s + EB_OFF_G + (k & 1u) * EB_G_BYTES + (uint32_t)(my - r_first) * (16 * EB_C * 4);
      const float *gg = g.G + (int64_t)my * (16 * EB_C);
      if (ok && !warp_wait(g_full + 8u * (k & 1u), (k >> 1) & 1u, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 61);
        ok = false;
      }
      const bool more = tile + gridDim.x < ntiles;
      unsigned long long gy2[16], dr2 = 0ull;
#pragma unroll
      for (int m = 0; m < 16; m++) gy2[m] = 0ull;
#pragma unroll 1
      for (int j = 0; ok && j < EB_NBLK / 2; j++) {
        const int blk = 2 * j + set;
        if (more && j == 2) {   // what the next tile starts with
          const int64_t en = e + (int64_t)gridDim.x * EB_TILE < g.nedges ? e + (int64_t)gridDim.x * EB_TILE : g.nedges - 1;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(g.Y + en * 16));
          if (lane == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(g.receiver + en));
        }
        const uint32_t use = 4u * k + (uint32_t)j;   // uses of each of this set's accumulator buffers
        if (!(ok = warp_wait(x_full + 8u * xs, xphase, lane))) break;
        const uint32_t sX = base_s + EB_OFF_X + (uint32_t)xs * EB_X_BYTES;
#pragma unroll 1
        for (int hf = 0; hf < 2; hf++) {
          const uint32_t buf = 2u * (uint32_t)set + (uint32_t)hf;
          const int piece = 2 * j + hf;            // of the next tile's h, in this tile's first four steps
          if (more && piece < 4) h_start(tile + gridDim.x, piece);
          if (!(ok = warp_wait(acc_full + 8u * buf, use & 1u, lane))) break;
          tc_fence_after();
          unsigned long long x2[4], t2[4];
          eb_lds(sX + (uint32_t)sw64_offset(row, 2 * hf), x2[0], x2[1]);
          eb_lds(sX + (uint32_t)sw64_offset(row, 2 * hf + 1), x2[2], x2[3]);
          const uint32_t ta = tmem + lanes + 256u + 64u * buf;
          const uint32_t coff = (uint32_t)(EB_BLK * blk + 8 * hf);
          if (staged) eb_half<true>(ta, gs + 4u * coff, gg, x2, y, gy2, dr2, t2);
          else eb_half<false>(ta, gs, gg + coff, x2, y, gy2, dr2, t2);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_free + 8u * buf);
          if (more && piece < 4) {
            h_put((int)((k + 1) & 1u), piece);
            if (piece == 3 && lane == 0) mbar_arrive(h_full + 8u * ((k + 1) & 1u));
          }
          if (hf == 0) {
            if (elect_one()) tma_store_wait_read();   // the previous block's T has left the piece
            __syncwarp();
          }
          const unsigned long long f2 = pack2(g.factor_v, g.factor_v);
#pragma unroll
          for (int c = 0; c < 2; c++)
            asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(sT + (uint32_t)sw64_offset(lane, 2 * hf + c)),
                         "l"(mul2(t2[2 * c], f2)), "l"(mul2(t2[2 * c + 1], f2))
                         : "memory");
        }
        if (!ok) break;
        fence_proxy_async();
        __syncwarp();
        if (elect_one()) {
          mbar_arrive(x_free + 8u * xs);
          if (base + 32 * q < g.nedges) tma_store_2d(&t_map, EB_BLK * blk, (int)base + 32 * q, sT);
        }
        xs += 2;
        if (xs >= EB_X_SLOTS) {
          xs -= EB_X_SLOTS;
          xphase ^= 1;
        }
      }
      if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 62);
      __syncwarp();
      if (lane == 0) mbar_arrive(g_free + 8u * (k & 1u));
      // The two sets' sums of an edge meet through shared memory.  Set 0 is the one ahead: it leaves its sums and goes on,
      // set 1 adds them.  (Two buffers: the MMAs come in step order, so set 0 cannot finish a tile before set 1 has left
      // the previous one.)
      float v[16], lo, hi;
      unpack2(dr2, lo, hi);
      v[0] = (lo + hi) * g.factor_t;
#pragma unroll
      for (int m = 1; m < 16; m++) {
        unpack2(gy2[m], lo, hi);
        v[m] = (lo + hi) * g.factor_v;
      }
      float *part = part0 + (k & 1u) * EB_PART;
      if (set == 0) {
#pragma unroll
        for (int m = 0; m < 16; m++) part[m] = v[m];
        __syncwarp();
        if (lane == 0) mbar_arrive(part_full + 8u * q);
      } else {
        if (ok && !warp_wait(part_full + 8u * q, k & 1u, lane)) {
          if (lane == 0 && g.status) atomicCAS(g.status, 0, 66);
          ok = false;
        }
        if (in && ok) {
#pragma unroll
          for (int m = 0; m < 16; m++) v[m] += part[m];
          float4 *o = reinterpret_cast<float4 *>(g.gY + e * 16);
#pragma unroll
          for (int i = 0; i < 4; i++) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (elect_one()) tma_store_wait_all();
  } else if (warp == 8) {
    // ---- MMA issuer
    const uint32_t idesc = umma_idesc_f16(128, 32);
    int slot = 0;
    uint32_t wphase = 0, k = 0;
    bool ok = true;
    for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, k++) {
      ok = warp_wait(h_full + 8u * (k & 1u), (k >> 1) & 1u, lane);
      for (int n = 0; ok && n < EB_NSTEP; n++) {
        const uint32_t b = (uint32_t)n & 3u, use = 4u * k + (uint32_t)(n >> 2);   // buffers 0, 1 are set 0's, 2, 3 set 1's
        ok = warp_wait(acc_free + 8u * b, (use & 1u) ^ 1u, lane) && warp_wait(w_full + 8u * slot, wphase, lane);
        if (!ok) break;
        if (elect_one()) {
          tc_fence_after();
          const uint32_t sW = base_s + EB_OFF_W + (uint32_t)slot * EB_W_BYTES;
          const uint64_t b_hi = umma_desc_sw128(sW), b_lo = umma_desc_sw128(sW + EB_W_BYTES / 2);
          const uint32_t d = tmem + 256u + 64u * b, a = tmem + 128u * (k & 1u);
#pragma unroll
          for (int j = 0; j < 4; j++) {   // R and R'
            umma_f16_ts(d, a + 8u * j, b_hi + (uint64_t)(2 * j), idesc, j != 0);
            umma_f16_ts(d + 32u, a + 64u + 8u * j, b_hi + (uint64_t)(2 * j), idesc, j != 0);
            umma_f16_ts(d, a + 8u * j, b_lo + (uint64_t)(2 * j), idesc, 1);
            umma_f16_ts(d + 32u, a + 64u + 8u * j, b_lo + (uint64_t)(2 * j), idesc, 1);
            umma_f16_ts(d, a + 32u + 8u * j, b_hi + (uint64_t)(2 * j), idesc, 1);
            umma_f16_ts(d + 32u, a + 96u + 8u * j, b_hi + (uint64_t)(2 * j), idesc, 1);
          }
          umma_commit(w_free + 8u * slot);
          umma_commit(acc_full + 8u * b);
        }
        __syncwarp();
        if (++slot == EB_W_SLOTS) {
          slot = 0;
          wphase ^= 1;
        }
      }
    }
    if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 63);
  } else if (warp == 9) {
    // ---- W blocks and G rows; one thread
    if (elect_one()) {
      int slot = 0;
      uint32_t wphase = 0, k = 0;
      bool ok = true;
      auto load_g = [&](int64_t tile, uint32_t n) -> bool {   // n: how many tiles of this CTA came before
        const int64_t base = tile * EB_TILE, last = base + EB_TILE - 1 < g.nedges ? base + EB_TILE - 1 : g.nedges - 1;
        const int r0 = __ldg(g.receiver + base);
        int count = __ldg(g.receiver + last) - r0 + 1;
        count = count < EB_G_RECV ? count : EB_G_RECV;
        if (!mbar_wait(g_free + 8u * (n & 1u), ((n >> 1) & 1u) ^ 1u)) return false;
        const uint32_t bar = g_full + 8u * (n & 1u), dst = base_s + EB_OFF_G + (n & 1u) * EB_G_BYTES;
        mbar_arrive_expect_tx(bar, (uint32_t)count * (16 * EB_C * 4));
        for (int i = 0; i < count; i++)
          bulk_copy_g2s(dst + (uint32_t)i * (16 * EB_C * 4), g.G + (int64_t)(r0 + i) * (16 * EB_C), 16 * EB_C * 4, bar);
        return true;
      };
      if (blockIdx.x < ntiles) ok = load_g(blockIdx.x, 0);
      for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, k++)
        for (int n = 0; ok && n < EB_NSTEP; n++) {
          ok = mbar_wait(w_free + 8u * slot, wphase ^ 1);
          if (!ok) break;
          mbar_arrive_expect_tx(w_full + 8u * slot, EB_W_BYTES);
          bulk_copy_g2s(base_s + EB_OFF_W + (uint32_t)slot * EB_W_BYTES, g.W + (int64_t)n * EB_W_BYTES, EB_W_BYTES,
                        w_full + 8u * slot);
          if (++slot == EB_W_SLOTS) {
            slot = 0;
            wphase ^= 1;
          }
          // the buffer was last read by the tile before this one, which the consumers have left by step 8
          if (n == 8 && tile + gridDim.x < ntiles) ok = load_g(tile + gridDim.x, k + 1);
        }
      if (!ok && g.status) atomicCAS(g.status, 0, 64);
    }
    __syncwarp();
  } else if (warp == 10) {
    // ---- sender rows
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
      int s[16];
#pragma unroll
      for (int i = 0; i < 16; i++) {
        int64_t e = tile * EB_TILE + 8 * i + (lane >> 2);
        e = e < g.nedges ? e : g.nedges - 1;
        s[i] = __ldg(g.sender + e);
      }
#pragma unroll 1
      for (int blk = 0; blk < EB_NBLK; blk++) {
        ok = warp_wait(x_free + 8u * slot, phase ^ 1, lane);
        if (!ok) break;
        const uint32_t dst = base_s + EB_OFF_X + (uint32_t)slot * EB_X_BYTES;
        const float *src = g.X + EB_BLK * blk + 4 * (lane & 3);
#pragma unroll
        for (int i = 0; i < 16; i++)
          eb_cp16(dst + (uint32_t)sw64_offset(8 * i + (lane >> 2), lane & 3), src + (int64_t)s[i] * EB_C);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(x_full + 8u * slot) : "memory");
        if (++slot == EB_X_SLOTS) {
          slot = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 65);
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, 512);
}

// [rows, 128] float32 as boxes of 32 rows x 16 columns with the 64-byte swizzle
int encode_piece_tensor_map(CUtensorMap *tmap, float *base, int64_t rows, int cols, const char *what);

int fused_messages_back(const float *X, const float *Y, const float *G, const void *h, const void *dh, const void *W,
                        float factor_v, float factor_t, const int32_t *sender, const int32_t *receiver, int64_t nedges,
                        float *T, float *gY, int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(edges_back)";
  if (nedges == 0) return CMACE_OK;
  const int64_t ntiles = (nedges + EB_TILE - 1) / EB_TILE;
  if (ntiles * EB_TILE > 0x7fffffffLL) return fail(CMACE_ERR_UNSUPPORTED, "%s: too many edges", what);
  const EdgeBackArgs g{X, Y, G, static_cast<const char *>(h), static_cast<const char *>(dh), static_cast<const char *>(W),
                       sender, receiver, status, nedges, factor_v, factor_t, gY};
  CUtensorMap map;
  if (int rc = encode_piece_tensor_map(&map, T, nedges, EB_C, what)) return rc;
  cudaError_t e = cudaFuncSetAttribute(edge_back_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, EB_SMEM);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  launch_chained(edge_back_kernel, (unsigned)(ntiles < 148 ? ntiles : 148), EB_THREADS, EB_SMEM, st, g, map);
  return check_launch(what);
}

}  // namespace cmace
