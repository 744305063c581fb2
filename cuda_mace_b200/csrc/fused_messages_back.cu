// Backward of the second layer's message passing with the radial weights formed where they are used (float32; forward in
// fused_messages.cu).  With u_l[e, c] = sum_m Y[lm, e] G[i, lm, c] (G the gradient of the messages,
// i the receiver of edge e) an edge's results are
//
//   T[e, c] = sum_l R_l u_l,   grad Y[lm, e] = sum_c X R_l G[lm],   dE/dr = sum_c X sum_l R'_l u_l,
//   R = h W,  R' = h' W,
//
// so neither R nor the gradients of R and h exist in memory.  Edges are the tensor-memory lanes: a thread owns an edge,
// every sum above runs over that thread's own values, no shuffles.  (With channels on the lanes, as in the forward, the
// sums over channels cost 31 shuffles per four edges and warp, and the kernel took 5.0 ms at 64 000 atoms.)
//
// Tile = 128 edges in steps of 16 channels.  A operand: h and h' (hi, lo fp16), 128 columns of tensor memory, two buffers.
// B operand: 16 KB of W per step, streamed from L2 (every CTA reads the same C KB).  An accumulator buffer holds 64 (R,
// four l) + 64 (R') columns; two buffers, so that the next step's products run while a step is worked on.
//
// A consumer warp has 16 edges and all channels: lane (g, t) holds two edges and four channels of a step, which is what
// tcgen05.ld.16x256b hands out (column 8 j + 2 t + i of a degree is channel 4 t + 2 j + i of the step).  Every word of G
// that a lane reads serves two edges; with an edge a lane and eight channels a step the same sums read twice the words, 2 048 an
// edge (128 bytes a cycle: 64 of the 158 cycles an edge took).
//
//   warps 0-7    consumers: warp w the rows 32 (w % 4) + 16 (w / 4) .. of the tile
//   warp 8       issues the MMAs
//   warp 9       W blocks, bulk copies
//   warps 10, 11 sender rows X, 64 bytes of 64 rows per step each, asynchronous copies
//   warps 12-15  the next tile: Y and receivers to shared memory, h and h' through shared memory to tensor memory, and the
//                G rows of its receivers (contiguous: the list is sorted), bulk copies by warp 12
//
// The consumers' 184 registers leave the other eight warps 72 (setmaxnreg); with 168 or 192 one side spills, 420 -> 465 us.
//
// What the consumers do besides the sums is kept short, since two warps a scheduler hide little of it: h, h', Y and G are
// brought by other warps (consumers doing it themselves: 150 of 890 thousand cycles at 16 000 atoms), T goes out in 64-byte
// pieces from registers instead of through shared memory, a step's barriers are asked for while the step before it is worked
// on, the MMA issuer is one thread that does the same.  With the words of G halved 16 000 atoms (833 000 edges) take 471 -> 411 us,
// 64 000 2 000 -> 1 700, 3 000 107 -> 92 (events around the kernel, both in one run).  What bounds it: instruction issue (59 %) and
// the latency of a step's chain, accumulators to registers, G, sums, with two warps a scheduler; of 417 us 312 are left without
// the sums, 257 without the products as well.
//
// Fewer channels are fewer steps a tile.  Edge pass on written weights and the product for dE/dr together -> this kernel, us at
// 16 000 atoms: 564 -> 199 at 32 channels, 722 -> 244 at 64, 1 446 -> 330 at 96; 3 000 atoms: 148 -> 46, 178 -> 58, 315 -> 74.
#include <atomic>

#include "common.cuh"
#include "register_split.hpp"
#include "step_common.cuh"
#include "tc_ptx.cuh"

namespace cmace {

constexpr int EB_TILE = 128;
constexpr int EB_STEP = 16;                       // channels of a step
constexpr int EB_THREADS = 512;
constexpr int EB_REGS = 184, EB_REGS_OTHER = 72;
// 128 registers are the most that 512 threads can have, and what ptxas gives a kernel with these bounds and setmaxnreg (also
// without optimisation and under -maxrregcount); the launch asks, since a block that started with fewer would wait for good
static_assert(register_split_fits(65536 / EB_THREADS, EB_THREADS, EB_REGS, EB_REGS_OTHER), "register split");
constexpr int EB_W_BYTES = 2 * 64 * 128;          // hi and lo image of a step's W: 64 rows (l, channel)
constexpr int EB_W_SLOTS = 3;
constexpr int EB_X_BYTES = EB_TILE * EB_STEP * 4;
constexpr int EB_X_SLOTS = 5;
constexpr int EB_PIECE = 2048;                    // 32 rows x 64 bytes
constexpr int EB_SMEM_MOST = 226 * 1024;          // a block's 227 KB less its static part

template <int C>
struct EdgeBackShape {
  static constexpr int NSTEP = C / EB_STEP;
  static constexpr int G_ROW = 16 * C * 4;        // gradient of a receiver's messages
  static constexpr int OFF_W = 0;
  static constexpr int OFF_X = OFF_W + EB_W_SLOTS * EB_W_BYTES;
  static constexpr int OFF_H = OFF_X + EB_X_SLOTS * EB_X_BYTES;   // eight pieces: h of the next tile on its way in, two a warp
  static constexpr int OFF_Y = OFF_H + 8 * EB_PIECE;              // Y of the next tile, then its receivers
  static constexpr int OFF_G = OFF_Y + EB_TILE * 64 + EB_TILE * 4;
  // Receivers staged per tile, as many as two buffers hold; a warp with a further one reads G from global memory.  Nanoseconds
  // an edge with seven and six, 413 000 edges, 128 channels: 0.55 and 0.55 at 52 edges a receiver, 0.52 and 0.52 at 31, 0.70 and
  // 0.89 at 21, 0.96 and 0.96 at 10, 1.05 and 1.05 at 5.
  static constexpr int RECV = (EB_SMEM_MOST - 1024 - OFF_G) / (2 * G_ROW);
  static constexpr int G_BYTES = RECV * G_ROW;
  static constexpr int SMEM = OFF_G + 2 * G_BYTES + 1024;
  static_assert(SMEM <= EB_SMEM_MOST && RECV >= 7, "receivers staged: as many as fit");
  static_assert(OFF_G % 16 == 0, "bulk copies");
};

// Which edge of the tile a row of tensor memory and shared memory holds: rows r and r + 8 of 16 are two edges in a row, so
// that few lanes have edges of two receivers (8 of 52 places for a receiver's end in a condensed system, 15 otherwise).
__device__ __forceinline__ int eb_edge(int row) { return (row & ~15) + 2 * (row & 7) + ((row >> 3) & 1); }

struct EdgeBackArgs {
  const float *X, *Y, *G;        // [Ns, C], [E, 16], [nnodes, 16, C]
  const char *h, *dh;            // rows of [hi 64 | lo 64] fp16
  const char *W;                 // [C / 16 steps][hi, lo][64 rows x 128 B, swizzled]
  const int32_t *sender, *receiver, *row_of;   // row_of: an edge's row of h and h'; null: its own
  int32_t *status;
  int64_t nedges;
  float factor_v, factor_t;      // undo the powers of two of h W and h' W
  float *T;                      // [E, C]
  float *gY;                     // [E, 16]; component 0 is dE/dr (Y_00 is constant)
};

// 16 lanes x 16 columns: thread (g, t) gets, for j = 0, 1, r[4 j], r[4 j + 1] = lane g, columns 8 j + 2 t, + 1 and r[4 j + 2],
// r[4 j + 3] = lane g + 8, the same columns
__device__ __forceinline__ void eb_ld(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
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
__device__ __forceinline__ void eb_lds(uint32_t a, unsigned long long (&x)[2]) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x[0]), "=l"(x[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void eb_cp16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void eb_cp4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void eb_cp_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Four channels (two pairs) of two edges: sums into gy (per edge and component) and dr2; T in t2.
// SAME: both edges have the same receiver.  The accumulators are given back as soon as the last of them is in registers;
// ready says whether the next step's accumulators and sender rows were there at that time.
template <int C, bool STAGED, bool SAME>
__device__ __forceinline__ void eb_step(uint32_t ta, uint32_t acc_free, uint32_t next_acc, uint32_t next_acc_phase,
                                        uint32_t next_x, uint32_t next_x_phase, bool &ready, int lane, const uint32_t (&gs)[2],
                                        const float *const (&gg)[2], const unsigned long long (&x2)[2][2],
                                        const float (&y)[2][16], float (&gy)[2][16],
                                        unsigned long long (&dr2)[2], unsigned long long (&t2)[2][2]) {
  unsigned long long v2[2][2];
  uint32_t r[2][8], d[2][8];
  eb_ld(ta, r[0]);
  eb_ld(ta + 64u, d[0]);
#pragma unroll
  for (int l = 0; l < 4; l++) {
    eb_ld_wait(r[l & 1], d[l & 1]);
    if (l < 3) {   // the next degree's accumulators are on their way meanwhile
      eb_ld(ta + 16u * (l + 1), r[(l + 1) & 1]);
      eb_ld(ta + 64u + 16u * (l + 1), d[(l + 1) & 1]);
    } else {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
      ready = mbar_test(next_acc, next_acc_phase) && mbar_test(next_x, next_x_phase);
    }
    unsigned long long r2[2][2], u2[2][2];
    float p[2][4], u[2][4];
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        r2[e][c] = pack2(__uint_as_float(r[l & 1][4 * c + 2 * e]), __uint_as_float(r[l & 1][4 * c + 2 * e + 1]));
        if (l > 0) unpack2(mul2(r2[e][c], x2[e][c]), p[e][2 * c], p[e][2 * c + 1]);
      }
#pragma unroll
    for (int m = l * l; m < (l + 1) * (l + 1); m++) {
      unsigned long long w[2][2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        if (e == 1 && SAME) {
          w[1][0] = w[0][0];
          w[1][1] = w[0][1];
        } else if (STAGED) {
          eb_lds(gs[e] + (uint32_t)(m * C * 4), w[e]);
        } else {
          const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2 *>(gg[e] + m * C));
          w[e][0] = q.x;
          w[e][1] = q.y;
        }
      }
#pragma unroll
      for (int e = 0; e < 2; e++)
#pragma unroll
          for (int c = 0; c < 2; c++) {
            float wa, wb;
            unpack2(w[e][c], wa, wb);
            if (l == 0) {                       // Y_00 = 1
              u[e][2 * c] = wa;
              u[e][2 * c + 1] = wb;
            } else {
              u[e][2 * c] = m == l * l ? y[e][m] * wa : fmaf(y[e][m], wa, u[e][2 * c]);
              u[e][2 * c + 1] = m == l * l ? y[e][m] * wb : fmaf(y[e][m], wb, u[e][2 * c + 1]);
              gy[e][m] = fmaf(p[e][2 * c + 1], wb, fmaf(p[e][2 * c], wa, gy[e][m]));
            }
          }
    }
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        u2[e][c] = pack2(u[e][2 * c], u[e][2 * c + 1]);
        const unsigned long long d2 = pack2(__uint_as_float(d[l & 1][4 * c + 2 * e]), __uint_as_float(d[l & 1][4 * c + 2 * e + 1]));
        t2[e][c] = l == 0 ? mul2(r2[e][c], u2[e][c]) : fma2(r2[e][c], u2[e][c], t2[e][c]);
        v2[e][c] = l == 0 ? mul2(d2, u2[e][c]) : fma2(d2, u2[e][c], v2[e][c]);
      }
  }
#pragma unroll
  for (int e = 0; e < 2; e++)
#pragma unroll
    for (int c = 0; c < 2; c++) dr2[e] = fma2(x2[e][c], v2[e][c], dr2[e]);
}

template <int C>
__global__ void __launch_bounds__(EB_THREADS, 1)
    edge_back_kernel(const EdgeBackArgs g) {
  using S = EdgeBackShape<C>;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[2 * EB_W_SLOTS + 2 * EB_X_SLOTS + 10];
  __shared__ uint32_t tmem_base_slot;

  const uint32_t base_s = (smem_u32(smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const uint32_t w_full = smem_u32(&bars[0]), w_free = w_full + 8u * EB_W_SLOTS;
  const uint32_t x_full = w_free + 8u * EB_W_SLOTS, x_free = x_full + 8u * EB_X_SLOTS;
  const uint32_t g_full = x_free + 8u * EB_X_SLOTS, h_full = g_full + 16u, acc_full = h_full + 16u, acc_free = acc_full + 16u;
  const uint32_t y_full = acc_free + 16u, y_free = y_full + 8u;

  if (tid == 0) {
    for (int s = 0; s < EB_W_SLOTS; s++) {
      mbar_init(w_full + 8u * s, 1);
      mbar_init(w_free + 8u * s, 1);     // the commit of the MMAs that read the slot
    }
    for (int s = 0; s < EB_X_SLOTS; s++) {
      mbar_init(x_full + 8u * s, 64);
      mbar_init(x_free + 8u * s, 8);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(g_full + 8u * b, 1);
      mbar_init(h_full + 8u * b, 4);
      mbar_init(acc_full + 8u * b, 1);
      mbar_init(acc_free + 8u * b, 8);
    }
    mbar_init(y_full, 128);
    mbar_init(y_free, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) tmem_alloc(smem_u32(&tmem_base_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Of all that the block reads only G is the kernel before's: warp 12 waits for it and holds everybody else up with g_full.
  // h buffer b at 128 b: h, h', hi and lo 32 each; acc b at 256 + 128 b
  const uint32_t tmem = (uint32_t)uniform((int)tmem_base_slot);
  const int64_t ntiles = (g.nedges + EB_TILE - 1) / EB_TILE;

  if (warp < 8) {
    // ---- consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EB_REGS));   // by whole warpgroups
    const int row0 = 32 * (warp & 3) + 16 * (warp >> 2), rg = row0 + (lane >> 2), t = lane & 3;   // rows rg, rg + 8 of the tile
    const uint32_t sY = base_s + S::OFF_Y;
    const uint32_t acc0 = tmem + ((uint32_t)row0 << 16) + 256u;
    bool ok = true;
    uint32_t k = 0;   // tiles done
    int xs = 0;
    uint32_t xphase = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, k++) {
      const int64_t e0 = tile * EB_TILE + row0 + 2 * (lane >> 2), e1 = e0 + 1;   // eb_edge()
      if (ok && !warp_wait_all(y_full, k & 1u, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 61);
        ok = false;
      }
      float y[2][16];
      int my[2], r_first;
#pragma unroll
      for (int e = 0; e < 2; e++) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(y[e][4 * i]), "=f"(y[e][4 * i + 1]), "=f"(y[e][4 * i + 2]), "=f"(y[e][4 * i + 3])
                       : "r"(sY + (uint32_t)sw64_offset(rg + 8 * e, i))
                       : "memory");
        }
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(my[e]) : "r"(sY + EB_TILE * 64 + 4u * (uint32_t)(rg + 8 * e)) : "memory");
      }
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(r_first) : "r"(sY + EB_TILE * 64) : "memory");
      __syncwarp();
      // Y is in registers, and this warp has left the tile before: its G and h buffers are free
      if (lane == 0) mbar_arrive(y_free);
      const bool same = __all_sync(0xffffffffu, my[0] == my[1]);
      const bool staged = __all_sync(0xffffffffu, my[1] - r_first < S::RECV);   // the list is sorted
      if (ok && !warp_wait_all(g_full + 8u * (k & 1u), (k >> 1) & 1u, lane)) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 62);
        ok = false;
      }
      const uint32_t sG = base_s + S::OFF_G + (k & 1u) * S::G_BYTES + 16u * t;
      float gy[2][16];
      unsigned long long dr2[2] = {0ull, 0ull};
#pragma unroll
      for (int m = 0; m < 16; m++) gy[0][m] = gy[1][m] = 0.f;
      bool ready = false;
#pragma unroll 1
      for (int n = 0; ok && n < S::NSTEP; n++) {
        // use number k NSTEP / 2 + n / 2 of accumulator buffer b
        const uint32_t use = k * (S::NSTEP / 2), b = (uint32_t)n & 1u, next_phase = (use + ((uint32_t)(n + 1) >> 1)) & 1u;
        if (!__all_sync(0xffffffffu, ready)) {
          ok = warp_wait(x_full + 8u * xs, xphase, lane) && warp_wait(acc_full + 8u * b, (use + ((uint32_t)n >> 1)) & 1u, lane);
          if (!ok) break;
        }
        tc_fence_after();
        const uint32_t sX = base_s + S::OFF_X + (uint32_t)xs * EB_X_BYTES, x_done = x_free + 8u * xs;
        unsigned long long x2[2][2], t2[2][2];
        eb_lds(sX + (uint32_t)sw64_offset(rg, t), x2[0]);
        eb_lds(sX + (uint32_t)sw64_offset(rg + 8, t), x2[1]);
        if (++xs == EB_X_SLOTS) {
          xs = 0;
          xphase ^= 1;
        }
        const int c0 = EB_STEP * n + 4 * t;
        const uint32_t gs[2] = {sG + (uint32_t)(my[0] - r_first) * S::G_ROW + 4u * EB_STEP * (uint32_t)n,
                                sG + (uint32_t)(my[1] - r_first) * S::G_ROW + 4u * EB_STEP * (uint32_t)n};
        const float *const gg[2] = {g.G + (int64_t)my[0] * (16 * C) + c0, g.G + (int64_t)my[1] * (16 * C) + c0};
        auto step = [&](auto in_smem, auto one) {
          eb_step<C, decltype(in_smem)::value, decltype(one)::value>(
              acc0 + 128u * b, acc_free + 8u * b, acc_full + 8u * (b ^ 1u), next_phase, x_full + 8u * xs, xphase, ready, lane,
              gs, gg, x2, y, gy, dr2, t2);
        };
        if (staged && same) step(std::true_type{}, std::true_type{});
        else if (staged) step(std::true_type{}, std::false_type{});
        else step(std::false_type{}, std::false_type{});
        if (lane == 0) mbar_arrive(x_done);   // the accumulators went back after every lane had read its X
        const unsigned long long f2 = pack2(g.factor_v, g.factor_v);
        ulonglong2 *out = reinterpret_cast<ulonglong2 *>(g.T + e0 * C + c0);
        if (e0 < g.nedges) out[0] = make_ulonglong2(mul2(t2[0][0], f2), mul2(t2[0][1], f2));
        if (e1 < g.nedges) out[C / 4] = make_ulonglong2(mul2(t2[1][0], f2), mul2(t2[1][1], f2));
      }
      if (!ok) {
        if (lane == 0 && g.status) atomicCAS(g.status, 0, 66);
        break;
      }
      // the four lanes of an edge hold its sums over their channels; lane t ends up with the components 4 t .. 4 t + 3
#pragma unroll
      for (int e = 0; e < 2; e++) {
        float h8[8], o[4], lo, hi;
        unpack2(dr2[e], lo, hi);
        gy[e][0] = lo + hi;
        const bool up = (t & 2) != 0, odd = (t & 1) != 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float send = up ? gy[e][i] : gy[e][i + 8], keep = up ? gy[e][i + 8] : gy[e][i];
          h8[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float send = odd ? h8[i] : h8[i + 4], keep = odd ? h8[i + 4] : h8[i];
          o[i] = (keep + __shfl_xor_sync(0xffffffffu, send, 1)) * (i == 0 && t == 0 ? g.factor_t : g.factor_v);
        }
        const int64_t ee = e ? e1 : e0;
        if (ee < g.nedges) *reinterpret_cast<float4 *>(g.gY + ee * 16 + 4 * t) = make_float4(o[0], o[1], o[2], o[3]);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(EB_REGS_OTHER));
    if (warp == 8) {
      // ---- MMA issuer, one thread: what a step waits for is asked for while the step before it is still being issued
      if (elect_one()) {
        const uint32_t idesc = umma_idesc_f16(128, 64);
        int slot = 0;
        uint32_t wphase = 0, k = 0;
        bool ok = true;
        for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, k++) {
          ok = mbar_wait(h_full + 8u * (k & 1u), (k >> 1) & 1u);
          bool ready = false;
          const uint32_t use = k * (S::NSTEP / 2);
          for (int n = 0; ok && n < S::NSTEP; n++) {
            const uint32_t b = (uint32_t)n & 1u;
            if (!ready) ok = mbar_wait(acc_free + 8u * b, ((use + ((uint32_t)n >> 1)) & 1u) ^ 1u) && mbar_wait(w_full + 8u * slot, wphase);
            if (!ok) break;
            tc_fence_after();
            const uint32_t sW = base_s + S::OFF_W + (uint32_t)slot * EB_W_BYTES;
            const uint64_t b_hi = umma_desc_sw128(sW), b_lo = umma_desc_sw128(sW + EB_W_BYTES / 2);
            const uint32_t d = tmem + 256u + 128u * b, a = tmem + 128u * (k & 1u);
            const uint32_t done = w_free + 8u * slot;
            if (++slot == EB_W_SLOTS) {
              slot = 0;
              wphase ^= 1;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {   // R and R'
              if (j == 3)
                ready = n + 1 < S::NSTEP && mbar_test(acc_free + 8u * (b ^ 1u), ((use + ((uint32_t)(n + 1) >> 1)) & 1u) ^ 1u) &&
                        mbar_test(w_full + 8u * slot, wphase);
              umma_f16_ts(d, a + 8u * j, b_hi + (uint64_t)(2 * j), idesc, j != 0);
              umma_f16_ts(d + 64u, a + 64u + 8u * j, b_hi + (uint64_t)(2 * j), idesc, j != 0);
              umma_f16_ts(d, a + 8u * j, b_lo + (uint64_t)(2 * j), idesc, 1);
              umma_f16_ts(d + 64u, a + 64u + 8u * j, b_lo + (uint64_t)(2 * j), idesc, 1);
              umma_f16_ts(d, a + 32u + 8u * j, b_hi + (uint64_t)(2 * j), idesc, 1);
              umma_f16_ts(d + 64u, a + 96u + 8u * j, b_hi + (uint64_t)(2 * j), idesc, 1);
            }
            umma_commit(done);
            umma_commit(acc_full + 8u * b);
          }
        }
        if (!ok && g.status) atomicCAS(g.status, 0, 63);
      }
      __syncwarp();
    } else if (warp == 9) {
      // ---- W blocks; one thread
      if (elect_one()) {
        int slot = 0;
        uint32_t wphase = 0;
        bool ok = true;
        for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x)
          for (int n = 0; ok && n < S::NSTEP; n++) {
            ok = mbar_wait(w_free + 8u * slot, wphase ^ 1);
            if (!ok) break;
            mbar_arrive_expect_tx(w_full + 8u * slot, EB_W_BYTES);
            bulk_copy_g2s(base_s + S::OFF_W + (uint32_t)slot * EB_W_BYTES, g.W + (int64_t)n * EB_W_BYTES, EB_W_BYTES,
                          w_full + 8u * slot);
            if (++slot == EB_W_SLOTS) {
              slot = 0;
              wphase ^= 1;
            }
          }
        if (!ok && g.status) atomicCAS(g.status, 0, 64);
      }
      __syncwarp();
    } else if (warp < 12) {
      // ---- sender rows: warp 10 the first 64 of a tile, warp 11 the others
      const int r0 = 64 * (warp - 10) + (lane >> 2);
      int slot = 0;
      uint32_t phase = 0;
      bool ok = true;
      int next[8];
      auto load_senders = [&](int64_t tile) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int64_t e = tile * EB_TILE + eb_edge(8 * i + r0);
          next[i] = __ldg(g.sender + (e < g.nedges ? e : g.nedges - 1));
        }
      };
      if (blockIdx.x < ntiles) load_senders(blockIdx.x);
      for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
        const float *src[8];
#pragma unroll
        for (int i = 0; i < 8; i++) src[i] = g.X + (int64_t)next[i] * C + 4 * (lane & 3);
        if (tile + gridDim.x < ntiles) load_senders(tile + gridDim.x);
#pragma unroll 1
        for (int n = 0; n < S::NSTEP; n++) {
          ok = warp_wait_all(x_free + 8u * slot, phase ^ 1, lane);
          if (!ok) break;
          const uint32_t dst = base_s + S::OFF_X + (uint32_t)slot * EB_X_BYTES;
#pragma unroll
          for (int i = 0; i < 8; i++) eb_cp16(dst + (uint32_t)sw64_offset(8 * i + r0, lane & 3), src[i] + EB_STEP * n);
          eb_cp_arrive(x_full + 8u * slot);
          if (++slot == EB_X_SLOTS) {
            slot = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok && lane == 0 && g.status) atomicCAS(g.status, 0, 65);
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
      // ---- the next tile's rows; warp 12 + q the rows 32 q ..
      const int q = warp & 3;
      const uint32_t sH = base_s + S::OFF_H + (uint32_t)(2 * q) * EB_PIECE, sY = base_s + S::OFF_Y;
      const uint32_t lanes = (uint32_t)(32 * q) << 16;
      const int r0 = 32 * q + (lane >> 2);
      const uint32_t hdst = sH + (uint32_t)sw64_offset(lane >> 2, lane & 3);
      bool ok = true;
      uint32_t k = 0;
      if (warp == 12 && blockIdx.x >= ntiles) {   // nothing to do, but the block has to wait
        grid_wait();
        grid_release();
      }
      int next[4];   // rows of h of this lane's edges in the next tile
      auto load_rows = [&](int64_t tile) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int64_t e = tile * EB_TILE + eb_edge(r0 + 8 * i), c = e < g.nedges ? e : g.nedges - 1;
          next[i] = g.row_of ? __ldcg(g.row_of + c) : (int)c;
        }
      };
      if (blockIdx.x < ntiles) load_rows(blockIdx.x);
      for (int64_t tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, k++) {
        const int64_t base = tile * EB_TILE;
        int row[4];
#pragma unroll
        for (int i = 0; i < 4; i++) row[i] = next[i];
        if (tile + gridDim.x < ntiles) load_rows(tile + gridDim.x);
        if (k && !warp_wait_all(y_free, (k & 1u) ^ 1u, lane)) {   // the consumers have begun the tile before this one
          if (lane == 0 && g.status) atomicCAS(g.status, 0, 67);
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int64_t r = base + eb_edge(r0 + 8 * i), e = r < g.nedges ? r : g.nedges - 1;
          eb_cp16(sY + (uint32_t)sw64_offset(r0 + 8 * i, lane & 3), g.Y + e * 16 + 4 * (lane & 3));
        }
        const int64_t rr = base + eb_edge(32 * q + lane), er = rr < g.nedges ? rr : g.nedges - 1;
        eb_cp4(sY + EB_TILE * 64 + 4u * (uint32_t)(32 * q + lane), g.receiver + er);
        eb_cp_arrive(y_full);
        // 64 bytes (32 k of hi or lo) of 32 rows: pieces 0-3 of h, 4-7 of h'
        auto start = [&](int piece) {
          if (piece < 8) {
            const char *src = (piece < 4 ? g.h : g.dh) + 64 * (piece & 3) + 16 * (lane & 3);
#pragma unroll
            for (int i = 0; i < 4; i++)   // sw64_offset(r + 8, c) = sw64_offset(r, c) + 512
              eb_cp16(hdst + (uint32_t)((piece & 1) * EB_PIECE) + 512u * i, src + (int64_t)row[i] * 256);
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
        };
        start(0);
        start(1);
        if (warp == 12 && k == 0) {
          grid_wait();
          grid_release();   // after the allocation
        }
        if (warp == 12 && elect_one()) {
          const int64_t last = base + EB_TILE - 1 < g.nedges ? base + EB_TILE - 1 : g.nedges - 1;
          const int first = __ldg(g.receiver + base);
          int count = __ldg(g.receiver + last) - first + 1;
          count = count < S::RECV ? count : S::RECV;
          const uint32_t bar = g_full + 8u * (k & 1u), dst = base_s + S::OFF_G + (k & 1u) * S::G_BYTES;
          mbar_arrive_expect_tx(bar, (uint32_t)count * S::G_ROW);
          for (int i = 0; i < count; i++)
            bulk_copy_g2s(dst + (uint32_t)i * S::G_ROW, g.G + (int64_t)(first + i) * (16 * C), S::G_ROW, bar);
        }
        __syncwarp();
#pragma unroll 1
        for (int piece = 0; piece < 8; piece++) {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          __syncwarp();
          uint32_t v[16];
#pragma unroll
          for (int c = 0; c < 4; c++)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v[4 * c]), "=r"(v[4 * c + 1]), "=r"(v[4 * c + 2]), "=r"(v[4 * c + 3])
                         : "r"(sH + (uint32_t)((piece & 1) * EB_PIECE) + (uint32_t)sw64_offset(lane, c))
                         : "memory");
          tmem_st16(tmem + lanes + 128u * (k & 1u) + 16u * (uint32_t)piece, v);
          __syncwarp();
          start(piece + 2);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(h_full + 8u * (k & 1u));
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, 512);
}

template <int C>
static int launch_edge_back(const EdgeBackArgs &g, const char *what, cudaStream_t st) {
  using S = EdgeBackShape<C>;
  static std::atomic<int> compiled_regs{0};   // a property of the binary
  int regs = compiled_regs.load(std::memory_order_relaxed);
  cudaError_t e = cudaSuccess;
  if (regs == 0) {
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, edge_back_kernel<C>);
    if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    compiled_regs.store(regs = attr.numRegs, std::memory_order_relaxed);
  }
  if (!register_split_fits(regs, EB_THREADS, EB_REGS, EB_REGS_OTHER))
    return fail(CMACE_ERR_UNSUPPORTED, "%s: compiled with %d registers a thread, too few for its register split", what, regs);
  e = cudaFuncSetAttribute(edge_back_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  const int64_t ntiles = (g.nedges + EB_TILE - 1) / EB_TILE;
  launch_chained(edge_back_kernel<C>, (unsigned)(ntiles < 148 ? ntiles : 148), EB_THREADS, S::SMEM, st, g);
  return check_launch(what);
}

int fused_messages_back(const float *X, const float *Y, const float *G, const void *h, const void *dh, const void *W,
                        float factor_v, float factor_t, const int32_t *sender, const int32_t *receiver, const int32_t *row_of,
                        int64_t nedges, int C, float *T, float *gY, int32_t *status, cudaStream_t st) {
  const char *what = "cmace_step(edges_back)";
  if (nedges == 0) return CMACE_OK;
  const int64_t ntiles = (nedges + EB_TILE - 1) / EB_TILE;
  if (ntiles * EB_TILE > 0x7fffffffLL) return fail(CMACE_ERR_UNSUPPORTED, "%s: too many edges", what);
  const EdgeBackArgs g{X, Y, G, static_cast<const char *>(h), static_cast<const char *>(dh), static_cast<const char *>(W),
                       sender, receiver, row_of, status, nedges, factor_v, factor_t, T, gY};
  switch (C) {
    case 32: return launch_edge_back<32>(g, what, st);
    case 64: return launch_edge_back<64>(g, what, st);
    case 96: return launch_edge_back<96>(g, what, st);
    case 128: return launch_edge_back<128>(g, what, st);
  }
  return fail(CMACE_ERR_UNSUPPORTED, "%s: no kernel for %d channels", what, C);
}

}  // namespace cmace
