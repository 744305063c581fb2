// Invariant message passing: receiver-sorted gather * product * segmented sum, and its backward.
//
//   out[i, lm, c] = sum_{e in row(i)} X[sender[e], c] * Y[lm, e] * R[e, l(lm), c]
//
// Work split: one warp owns one receiver row and a chunk of 32*VEC channels (lane <-> VEC
// consecutive channels, 16-byte loads).  The warp walks the receiver's contiguous edge range,
// keeps all 16 (l,m) accumulators of its channels in registers and writes each output once:
// no atomics, a fixed summation order, and R (the dominant HBM stream, E*4*C scalars) is read
// exactly once with full 128-byte lines.  Y [16, E] is component-major, so the 16 values of an
// edge are fetched by 16 lanes (two edges per 32-lane load) and broadcast with shuffles.
//
// Backward, edge pass (same mapping, G[i] = d loss / d out[i] held in registers):
//   u[l, c]      = sum_{m in l} Y[m, e] * G[i, m, c]
//   gradR[e,l,c] = X[s, c] * u[l, c]
//   T[e, c]      = sum_l u[l, c] * R[e, l, c]                (sender contribution of edge e)
//   gradY[m, e]  = sum_c G[i, m, c] * R[e, l, c] * X[s, c]   (16-value warp transpose-reduce)
// Backward, node pass: gradX[s, c] = sum over the edges sent by s of T[e, c], walking the
// sender-grouped edge permutation; again one warp per node, no atomics.
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "step_common.cuh"

namespace cmace {

constexpr int kWarpsPerBlock = 4;

// SPLIT = 1: as described above.  SPLIT = 8: a block owns one receiver (and channel chunk), its eight warps take every
// eighth pair of edges and add up through shared memory in a fixed order: with fewer receivers than the chip holds warps
// the walk over one receiver's edges, about 1.6 us a pair, is all there is (192 receivers, 52 edges: 43 us with one warp
// each).
// ROWS: edge e reads row row_of[e] of R, which another edge may read as well; rows and senders are looked up a pair ahead (420 ->
// 338 us at 8 000 atoms in float64, the same as from a row of its own).
template <typename T, int VEC, int SPLIT, bool ROWS = false>
__global__ void __launch_bounds__(SPLIT == 1 ? kWarpsPerBlock * 32 : SPLIT * 32, SPLIT == 1 && sizeof(T) == 4 ? 4 : 1)
    imp_fwd_kernel(const T *__restrict__ X, const T *__restrict__ Y, const T *__restrict__ R,
                   const int32_t *__restrict__ row_of, const int32_t *__restrict__ sender, const int32_t *__restrict__ row_ptr,
                   int64_t nnodes, ImpLayout ys, int C, T *__restrict__ out) {
  grid_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t node = SPLIT == 1 ? (int64_t)blockIdx.x * kWarpsPerBlock + warp : blockIdx.x;
  if (node >= nnodes) return;
  const int c0 = blockIdx.y * (32 * VEC) + lane * VEC;
  const int64_t e0 = row_ptr[node], e1 = row_ptr[node + 1];

  T acc[16][VEC];
#pragma unroll
  for (int m = 0; m < 16; m++)
#pragma unroll
    for (int v = 0; v < VEC; v++) acc[m][v] = T(0);

  __shared__ __align__(16) PairHarmonics<T, SPLIT == 1 ? kWarpsPerBlock : SPLIT> harmonics;
  constexpr bool BRANCH = sizeof(T) == 8 || SPLIT > 1;
  int turn = 0;
  const int ylm = lane & 15, yedge = lane >> 4;
  int32_t next[4];   // ROWS: senders and rows of the next pair, or the row of R would wait for its number
  auto look_up = [&](int64_t e) {
    const int64_t a = e < e1 ? e : e1 - 1, b = e + 1 < e1 ? e + 1 : e1 - 1;
    next[0] = __ldg(sender + a), next[1] = __ldg(sender + b), next[2] = __ldg(row_of + a), next[3] = __ldg(row_of + b);
  };
  if (ROWS && e0 < e1) look_up(e0 + (SPLIT > 1 ? 2 * warp : 0));
  for (int64_t e = e0 + (SPLIT > 1 ? 2 * warp : 0); e < e1; e += 2 * SPLIT, turn ^= 1) {
    // second edge of the pair: clamp to a valid edge, what it would add is zeroed below.  Zero harmonics alone would not do, the last
    // edge's weights may be infinite.  us at 8 192 receivers of 30 edges, 128 channels: 106.1 -> 106.6 by selects, 131 in a branch
    // (registers), 132 with a row of zeros, 107 with the last edge behind the loop; float64 223.3 -> 223.8 in a branch, 225.8 by
    // selects, 280 with a row of zeros or behind the loop; eight warps a receiver, 800 of 52: 28.8 -> 28.8 in a branch, 30.8 by
    // selects.
    const bool second = e + 1 < e1;
    const int64_t eb = second ? e + 1 : e;
    const int64_t ey = yedge ? eb : e;
    T yv = __ldg(Y + ylm * ys.m + ey * ys.e);
    if (yedge && !second) yv = T(0);
    const int64_t sa = ROWS ? next[0] : sender[e], sb = ROWS ? next[1] : sender[eb];
    const int64_t ea = ROWS ? next[2] : e, ec = ROWS ? next[3] : eb;
    if (ROWS) look_up(e + 2 * SPLIT);
    T xa[VEC], xb[VEC], ra[4][VEC], rb[4][VEC];
    load_vec<T, VEC>(xa, X + sa * C + c0);
    load_vec<T, VEC>(xb, X + sb * C + c0);
#pragma unroll
    for (int l = 0; l < 4; l++) {
      if constexpr (ROWS) {
        load_vec<T, VEC>(ra[l], R + (ea * 4 + l) * C + c0);
        load_vec<T, VEC>(rb[l], R + (ec * 4 + l) * C + c0);
      } else {
        load_vec_stream<T, VEC>(ra[l], R + (ea * 4 + l) * C + c0);
        load_vec_stream<T, VEC>(rb[l], R + (ec * 4 + l) * C + c0);
      }
    }
#pragma unroll
    for (int l = 0; l < 4; l++)
#pragma unroll
      for (int v = 0; v < VEC; v++) {
        ra[l][v] *= xa[v];
        rb[l][v] *= xb[v];
        if (!BRANCH && !second) rb[l][v] = T(0);
      }
    if (BRANCH && !second) {   // volatile: it stays a branch
#pragma unroll
      for (int l = 0; l < 4; l++)
#pragma unroll
        for (int v = 0; v < VEC; v++) {
          if constexpr (sizeof(T) == 8) asm volatile("mov.f64 %0, 0d0000000000000000;" : "=d"(rb[l][v]));
          else asm volatile("mov.f32 %0, 0f00000000;" : "=f"(rb[l][v]));
        }
    }
    T *yp = harmonics.v[warp][turn];
    yp[lane] = yv;
    __syncwarp();
    T y[16];
    take16<T>(y, yp);
#pragma unroll
    for (int m = 0; m < 16; m++)
#pragma unroll
      for (int v = 0; v < VEC; v++) acc[m][v] = fma(y[m], ra[l_of_lm(m)][v], acc[m][v]);
    take16<T>(y, yp + 16);
#pragma unroll
    for (int m = 0; m < 16; m++)
#pragma unroll
      for (int v = 0; v < VEC; v++) acc[m][v] = fma(y[m], rb[l_of_lm(m)][v], acc[m][v]);
  }
  T *o = out + node * 16 * C + c0;
  if constexpr (SPLIT > 1) {
    extern __shared__ __align__(16) unsigned char imp_smem[];
    T *part = reinterpret_cast<T *>(imp_smem);   // [SPLIT][16][32 VEC]
#pragma unroll
    for (int m = 0; m < 16; m++) store_vec<T, VEC>(part + ((warp * 16 + m) * 32 + lane) * VEC, acc[m]);
    __syncthreads();
    for (int m = warp; m < 16; m += SPLIT) {     // every warp sums two components
      T sum[VEC];
#pragma unroll
      for (int v = 0; v < VEC; v++) sum[v] = T(0);
#pragma unroll
      for (int w = 0; w < SPLIT; w++)
#pragma unroll
        for (int v = 0; v < VEC; v++) sum[v] += part[((w * 16 + m) * 32 + lane) * VEC + v];
      store_vec<T, VEC>(o + m * C, sum);
    }
    return;
  }
#pragma unroll
  for (int m = 0; m < 16; m++) store_vec<T, VEC>(o + m * C, acc[m]);
}

// JOIN: a block's warps have the chunks from `chunk` on of one receiver and slice, and their shares of gradY are added up in shared
// memory in order, from the second launch on to what the launch before has left; otherwise a warp has a receiver and slice.
template <typename T, int VEC, bool JOIN = false>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
    imp_bwd_edge_kernel(const T *__restrict__ X, const T *__restrict__ Y, const T *__restrict__ R,
                        const T *__restrict__ G, const int32_t *__restrict__ sender,
                        const int32_t *__restrict__ row_ptr, int64_t nnodes, int64_t nedges, ImpLayout ys, int C,
                        int slices, int chunk, T *__restrict__ gradR, T *__restrict__ gradY_out, T *__restrict__ Tout) {
  grid_begin();
  const int lane = threadIdx.x & 31;
  // everything written is per edge: `slices` warps share a receiver, each takes every slices-th pair of its edges
  const int64_t item = JOIN ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  const int64_t node = slices == 1 ? item : item / slices;
  const int slice = slices == 1 ? 0 : (int)(item - node * slices);
  if (node >= nnodes) return;
  const int c0 = (JOIN ? chunk + (int)(threadIdx.x >> 5) : (int)blockIdx.y) * (32 * VEC) + lane * VEC;
  const int64_t e0 = row_ptr[node], e1 = row_ptr[node + 1];
  if (e0 >= e1) return;
  // with several channel chunks each chunk writes its own [16, E] partial of gradY
  T *gy = gradY_out + (int64_t)blockIdx.y * 16 * nedges;

  T g[16][VEC];
#pragma unroll
  for (int m = 0; m < 16; m++) load_vec<T, VEC>(g[m], G + (node * 16 + m) * C + c0);

  __shared__ __align__(16) PairHarmonics<T, kWarpsPerBlock> harmonics;
  __shared__ T shares[JOIN ? 2 : 1][JOIN ? kWarpsPerBlock : 1][32];   // of a pair of edges
  int turn = 0;
  const int ylm = lane & 15, yedge = lane >> 4;
  for (int64_t e = e0 + 2 * slice; e < e1; e += 2 * slices, turn ^= 1) {
    const int64_t eb = (e + 1 < e1) ? e + 1 : e;
    const T yv = __ldg(Y + ylm * ys.m + (yedge ? eb : e) * ys.e);
    T *yp = harmonics.v[threadIdx.x >> 5][turn];
    // loads of both edges of the pair are issued before either is consumed
    const int64_t s2[2] = {sender[e], sender[eb]};
    T xx[2][VEC], rr[2][4][VEC];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      load_vec<T, VEC>(xx[h], X + s2[h] * C + c0);
#pragma unroll
      for (int l = 0; l < 4; l++) load_vec_stream<T, VEC>(rr[h][l], R + ((h ? eb : e) * 4 + l) * C + c0);
    }
    yp[lane] = yv;
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t ee = h ? eb : e;
      if (h && e + 1 >= e1) break;  // warp-uniform
      T(&x)[VEC] = xx[h];
      T(&r)[4][VEC] = rr[h];
      T u[4][VEC], p[16], yy[16];
      take16<T>(yy, yp + 16 * h);
#pragma unroll
      for (int l = 0; l < 4; l++)
#pragma unroll
        for (int v = 0; v < VEC; v++) u[l][v] = T(0);
#pragma unroll
      for (int m = 0; m < 16; m++) {
        const T y = yy[m];
        T pm = T(0);
#pragma unroll
        for (int v = 0; v < VEC; v++) {
          u[l_of_lm(m)][v] = fma(y, g[m][v], u[l_of_lm(m)][v]);
          pm = fma(g[m][v], r[l_of_lm(m)][v] * x[v], pm);
        }
        p[m] = pm;
      }
      T t[VEC];
#pragma unroll
      for (int v = 0; v < VEC; v++) t[v] = T(0);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        T gr[VEC];
#pragma unroll
        for (int v = 0; v < VEC; v++) {
          t[v] = fma(u[l][v], r[l][v], t[v]);
          gr[v] = x[v] * u[l][v];
        }
        if (gradR != nullptr) store_vec_stream<T, VEC>(gradR + (ee * 4 + l) * C + c0, gr);
      }
      if (Tout != nullptr) store_vec<T, VEC>(Tout + ee * C + c0, t);
      const T tot = warp_reduce16(p, lane);
      if ((lane & 1) == 0) {
        if (JOIN) shares[turn][threadIdx.x >> 5][16 * h + (lane >> 1)] = tot;
        else gy[(lane >> 1) * ys.m + ee * ys.e] = tot;
      }
    }
    if constexpr (JOIN) {
      __syncthreads();   // the buffer of the pair before has been read by then
      const int warps = blockDim.x >> 5;
      if ((int)(threadIdx.x >> 5) == turn % warps && (!yedge || e + 1 < e1)) {
        T *dst = gy + ylm * ys.m + (yedge ? eb : e) * ys.e, sum = chunk ? *dst : T(0);
        for (int w = 0; w < warps; w++) sum += shares[turn][w][lane];
        *dst = sum;
      }
    }
  }
}

// The edge pass of a float64 step, with dE/dr from the radial weights' derivative instead of a gradient of the weights that a
// product would read again:  T and grad Y as above, dE/dr = sum_c X sum_l R'_l u_l in the place of grad Y_00 (Y_00 is constant).
// Edge e reads rows row_of[e] (null: e) of R and R', whose numbers are asked for a pair of edges ahead.  Each channel chunk has its
// own gY [E, 16].  Bound by bytes, as the pass that wrote the gradient: 848 -> 678 us at 8 000 atoms and 128 channels (805 with
// 220 registers, two blocks an SM), 406 -> 363 at 64.
template <int VEC>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, 3)
    imp_bwd_edge_pair_kernel(const double *__restrict__ X, const double *__restrict__ Y, const double *__restrict__ R,
                             const double *__restrict__ dR, const int32_t *__restrict__ row_of, const double *__restrict__ G,
                             const int32_t *__restrict__ sender, const int32_t *__restrict__ row_ptr, int64_t nnodes,
                             int64_t nedges, int C, int slices, double *__restrict__ gY, double *__restrict__ Tout) {
  grid_begin();
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  const int64_t node = slices == 1 ? item : item / slices;
  const int slice = slices == 1 ? 0 : (int)(item - node * slices);
  if (node >= nnodes) return;
  const int c0 = blockIdx.y * (32 * VEC) + lane * VEC;
  const int64_t e0 = row_ptr[node], e1 = row_ptr[node + 1];
  if (e0 + 2 * slice >= e1) return;
  double *gy = gY + (int64_t)blockIdx.y * 16 * nedges;
  double g[16][VEC];
#pragma unroll
  for (int m = 0; m < 16; m++) load_vec<double, VEC>(g[m], G + (node * 16 + m) * C + c0);
  __shared__ __align__(16) PairHarmonics<double, kWarpsPerBlock> harmonics;
  int turn = 0;
  const int ylm = lane & 15, yedge = lane >> 4;
  int32_t next[4];   // senders and rows of the next pair of edges
  auto look_up = [&](int64_t e) {
    const int64_t a = e < e1 ? e : e1 - 1, b = e + 1 < e1 ? e + 1 : e1 - 1;
    next[0] = __ldg(sender + a), next[1] = __ldg(sender + b);
    next[2] = row_of ? __ldg(row_of + a) : (int32_t)a, next[3] = row_of ? __ldg(row_of + b) : (int32_t)b;
  };
  look_up(e0 + 2 * slice);
  for (int64_t e = e0 + 2 * slice; e < e1; e += 2 * slices, turn ^= 1) {
    const int64_t eb = e + 1 < e1 ? e + 1 : e;
    const double yv = __ldg(Y + ylm + (yedge ? eb : e) * 16);
    double *yp = harmonics.v[threadIdx.x >> 5][turn];
    const int64_t s2[2] = {next[0], next[1]}, row[2] = {next[2], next[3]};
    look_up(e + 2 * slices);
    double xx[2][VEC], rr[2][4][VEC], dd[2][4][VEC];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      load_vec<double, VEC>(xx[h], X + s2[h] * C + c0);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        load_vec<double, VEC>(rr[h][l], R + (row[h] * 4 + l) * C + c0);
        load_vec<double, VEC>(dd[h][l], dR + (row[h] * 4 + l) * C + c0);
      }
    }
    yp[lane] = yv;
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t ee = h ? eb : e;
      if (h && e + 1 >= e1) break;  // warp-uniform
      double(&x)[VEC] = xx[h], p[16], yy[16], t[VEC], v[VEC];
      take16<double>(yy, yp + 16 * h);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        double u[VEC], rx[VEC];
#pragma unroll
        for (int c = 0; c < VEC; c++) rx[c] = rr[h][l][c] * x[c];
#pragma unroll
        for (int m = l * l; m < (l + 1) * (l + 1); m++) {
          double pm = 0.0;
#pragma unroll
          for (int c = 0; c < VEC; c++) {
            u[c] = m == l * l ? yy[m] * g[m][c] : fma(yy[m], g[m][c], u[c]);
            pm = fma(g[m][c], rx[c], pm);
          }
          p[m] = pm;
        }
#pragma unroll
        for (int c = 0; c < VEC; c++) {
          t[c] = l == 0 ? u[c] * rr[h][l][c] : fma(u[c], rr[h][l][c], t[c]);
          v[c] = l == 0 ? u[c] * dd[h][l][c] : fma(u[c], dd[h][l][c], v[c]);
        }
      }
      p[0] = 0.0;
#pragma unroll
      for (int c = 0; c < VEC; c++) p[0] = fma(x[c], v[c], p[0]);
      store_vec<double, VEC>(Tout + ee * C + c0, t);
      const double tot = warp_reduce16(p, lane);
      if ((lane & 1) == 0) gy[(lane >> 1) + ee * 16] = tot;
    }
  }
}

// ---- narrow rows: several edges a warp -----------------------------------------------------------------------------
// With 32 or 64 channels a row does not fill a warp with 16-byte pieces, and what an edge costs beside its channels (harmonics
// handed out, sums over channels, addresses) is what binds: 32 channels took 0.8 of 64 channels' time.  Here LANES lanes own an
// edge, EPW = 32 / LANES edges are worked on side by side and AT of those one after the other, all of one receiver.  96 channels:
// three a lane, 32 apart, in one pass instead of three chunks with a share of grad Y each.  us at 8 192 nodes of 30 edges, forward and
// edge pass, before -> now: float32 50 -> 37 and 116 -> 72 with 32 channels, 71 -> 70 and 145 -> 125 with 64, 129 -> 83 and 352 -> 203
// with 96; float64 86 -> 64 and 170 -> 139 with 32, 233 -> 167 and 538 -> 388 with 96 (64 channels fill a warp with 16-byte pieces).
// In a float64 step of 8 000 atoms 138 -> 108 and 273 -> 216 with 32 channels, 366 -> 276 and 731 -> 631 with 96.
template <typename T, int VEC>
__device__ __forceinline__ void load_lane(T (&d)[VEC], const T *row, int sub, bool stream) {
  if constexpr (VEC == 3) {
#pragma unroll
    for (int v = 0; v < 3; v++) d[v] = stream ? __ldcs(row + sub + 32 * v) : __ldg(row + sub + 32 * v);
  } else {
    if (stream) load_vec_stream<T, VEC>(d, row + sub * VEC);
    else load_vec<T, VEC>(d, row + sub * VEC);
  }
}
template <typename T, int VEC>
__device__ __forceinline__ void store_lane(T *row, int sub, const T (&d)[VEC], bool stream) {
  if constexpr (VEC == 3) {
#pragma unroll
    for (int v = 0; v < 3; v++) {
      if (stream) __stcs(row + sub + 32 * v, d[v]);
      else row[sub + 32 * v] = d[v];
    }
  } else {
    if (stream) store_vec_stream<T, VEC>(row + sub * VEC, d);
    else store_vec<T, VEC>(row + sub * VEC, d);
  }
}

template <typename T, int EDGES>
struct SlotHarmonics {
  static constexpr int LD = 16 + 16 / (int)sizeof(T);   // an edge's 16 values; a piece more keeps eight edges in different banks
  static constexpr int PER = (EDGES * 16 + 31) / 32;    // values a lane
  // component and edge of a lane's value i, consecutive in memory for neighbouring lanes
  static __device__ __forceinline__ bool at(int i, int lane, const ImpLayout &ys, int &edge, int &m) {
    const int k = 32 * i + lane;
    edge = ys.m == 1 ? k >> 4 : k % EDGES;
    m = ys.m == 1 ? k & 15 : k / EDGES;
    return k < EDGES * 16;
  }
};

// Blocks an SM, as measured: float32 37 us with three at 32 channels (44 with four), 70 with four at 64 (81 with three); float64 of 32
// channels 64 with three (76 with four), but 108 with four (166 with three) where rows are looked up.  A block's 128 threads then have
// 96 (five), 128 (four) or 168 registers each (three), 202 to 204 with two; none spills but 64 channels of float32 (16 bytes).
template <typename T, int VEC, int LANES, bool ROWS>
constexpr int fwd_slots_blocks() {
  if (VEC == 3) return sizeof(T) == 4 ? 5 : 2;
  return (sizeof(T) == 4 ? LANES == 16 : ROWS) ? 4 : 3;
}
template <typename T, int VEC, int LANES, int SPLIT, bool ROWS>
__global__ void __launch_bounds__(SPLIT == 1 ? kWarpsPerBlock * 32 : SPLIT * 32, SPLIT > 1 ? 1 : fwd_slots_blocks<T, VEC, LANES, ROWS>())
    imp_fwd_slots_kernel(const T *__restrict__ X, const T *__restrict__ Y, const T *__restrict__ R, const int32_t *__restrict__ row_of,
                         const int32_t *__restrict__ sender, const int32_t *__restrict__ row_ptr, int64_t nnodes, ImpLayout ys,
                         T *__restrict__ out) {
  grid_begin();
  constexpr int EPW = 32 / LANES, AT = 2, EDGES = AT * EPW, C = VEC * LANES, KEPT = 16 / EPW;
  using H = SlotHarmonics<T, EDGES>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LANES, slot = lane / LANES;
  const int64_t node = SPLIT == 1 ? (int64_t)blockIdx.x * kWarpsPerBlock + warp : blockIdx.x;
  if (node >= nnodes) return;
  const int64_t e0 = row_ptr[node], e1 = row_ptr[node + 1], begin = e0 + (SPLIT > 1 ? EDGES * warp : 0);
  T acc[16][VEC];
#pragma unroll
  for (int m = 0; m < 16; m++)
#pragma unroll
    for (int v = 0; v < VEC; v++) acc[m][v] = T(0);
  __shared__ __align__(16) T harmonics[SPLIT == 1 ? kWarpsPerBlock : SPLIT][2][EDGES * H::LD];
  int turn = 0;
  int32_t next[AT][2];   // senders and rows of this slot's next edges
  auto look_up = [&](int64_t e) {
#pragma unroll
    for (int a = 0; a < AT; a++) {
      const int64_t i = e + a * EPW + slot < e1 ? e + a * EPW + slot : e1 - 1;
      next[a][0] = __ldg(sender + i);
      next[a][1] = ROWS ? __ldg(row_of + i) : (int32_t)i;
    }
  };
  if (begin < e1) look_up(begin);
  for (int64_t e = begin; e < e1; e += EDGES * SPLIT, turn ^= 1) {
    T yv[H::PER];
#pragma unroll
    for (int i = 0; i < H::PER; i++) {
      int edge, m;
      yv[i] = T(0);
      if (H::at(i, lane, ys, edge, m) && e + edge < e1) yv[i] = __ldg(Y + m * ys.m + (e + edge) * ys.e);
    }
    T x[AT][VEC], r[AT][4][VEC];
#pragma unroll
    for (int a = 0; a < AT; a++) {
      const bool there = e + a * EPW + slot < e1;   // beyond the receiver's edges: nothing is read or added
#pragma unroll
      for (int v = 0; v < VEC; v++) x[a][v] = r[a][0][v] = r[a][1][v] = r[a][2][v] = r[a][3][v] = T(0);
      if (there) {
        load_lane<T, VEC>(x[a], X + (int64_t)next[a][0] * C, sub, false);
#pragma unroll
        for (int l = 0; l < 4; l++) load_lane<T, VEC>(r[a][l], R + ((int64_t)next[a][1] * 4 + l) * C, sub, !ROWS);
      }
    }
    look_up(e + EDGES * SPLIT);
#pragma unroll
    for (int a = 0; a < AT; a++)
#pragma unroll
      for (int l = 0; l < 4; l++)
#pragma unroll
        for (int v = 0; v < VEC; v++) r[a][l][v] *= x[a][v];
    T *yp = harmonics[warp][turn];
#pragma unroll
    for (int i = 0; i < H::PER; i++) {
      int edge, m;
      if (H::at(i, lane, ys, edge, m)) yp[edge * H::LD + m] = yv[i];
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < AT; a++) {
      T y[16];
      take16<T>(y, yp + (a * EPW + slot) * H::LD);
#pragma unroll
      for (int m = 0; m < 16; m++)
#pragma unroll
        for (int v = 0; v < VEC; v++) acc[m][v] = fma(y[m], r[a][l_of_lm(m)][v], acc[m][v]);
    }
  }
  // the slots' sums: every slot ends up with KEPT components of all of them
  if constexpr (EPW >= 2) {
    const bool up = lane & 16;
#pragma unroll
    for (int m = 0; m < 8; m++)
#pragma unroll
      for (int v = 0; v < VEC; v++) {
        const T send = up ? acc[m][v] : acc[m + 8][v], keep = up ? acc[m + 8][v] : acc[m][v];
        acc[m][v] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
      }
  }
  if constexpr (EPW == 4) {
    const bool up = lane & 8;
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
      for (int v = 0; v < VEC; v++) {
        const T send = up ? acc[m][v] : acc[m + 4][v], keep = up ? acc[m + 4][v] : acc[m][v];
        acc[m][v] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
      }
  }
  T *o = out + node * 16 * C;
  if constexpr (SPLIT > 1) {
    extern __shared__ __align__(16) unsigned char imp_smem[];
    T *part = reinterpret_cast<T *>(imp_smem);   // [SPLIT][16][C]
#pragma unroll
    for (int m = 0; m < KEPT; m++) store_lane<T, VEC>(part + (warp * 16 + slot * KEPT + m) * C, sub, acc[m], false);
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * C; i += SPLIT * 32) {
      T sum = T(0);
#pragma unroll
      for (int w = 0; w < SPLIT; w++) sum += part[w * 16 * C + i];
      o[i] = sum;
    }
  } else {
#pragma unroll
    for (int m = 0; m < KEPT; m++) store_lane<T, VEC>(o + (slot * KEPT + m) * C, sub, acc[m], false);
  }
}

// Sums of p[m] over a slot's lanes: lane `sub` gets the components of `own` values from sub * own on (one of two lanes of 32 its
// own: the other holds the same).
template <typename T, int LANES>
__device__ __forceinline__ void slot_reduce16(T (&p)[16], int lane) {
  if constexpr (LANES == 32) {
    p[0] = warp_reduce16(p, lane);
  } else {
    constexpr int STEPS = LANES == 16 ? 4 : 3;
    int n = 16, off = LANES / 2;
#pragma unroll
    for (int k = 0; k < STEPS; k++, off >>= 1) {
      n >>= 1;
      const bool up = lane & off;
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (i < n) {
          const T send = up ? p[i] : p[i + n], keep = up ? p[i + n] : p[i];
          p[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
  }
}

// PAIR: as imp_bwd_edge_pair_kernel (rows of R and R' by row_of, dE/dr in the place of grad Y_00); otherwise as imp_bwd_edge_kernel
template <typename T, int VEC, int LANES, bool PAIR>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, VEC != 3 ? 3 : (sizeof(T) == 4 ? 4 : 2))
    imp_bwd_edge_slots_kernel(const T *__restrict__ X, const T *__restrict__ Y, const T *__restrict__ R, const T *__restrict__ dR,
                              const int32_t *__restrict__ row_of, const T *__restrict__ G, const int32_t *__restrict__ sender,
                              const int32_t *__restrict__ row_ptr, int64_t nnodes, ImpLayout ys, int slices, T *__restrict__ gradR,
                              T *__restrict__ gradY, T *__restrict__ Tout) {
  grid_begin();
  constexpr int EPW = 32 / LANES, AT = PAIR && VEC == 3 ? 1 : 2, EDGES = AT * EPW, C = VEC * LANES;
  using H = SlotHarmonics<T, EDGES>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LANES, slot = lane / LANES;
  const int64_t item = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  const int64_t node = slices == 1 ? item : item / slices;
  const int slice = slices == 1 ? 0 : (int)(item - node * slices);
  if (node >= nnodes) return;
  const int64_t e1 = row_ptr[node + 1], begin = row_ptr[node] + EDGES * slice;
  if (begin >= e1) return;
  T g[16][VEC];
#pragma unroll
  for (int m = 0; m < 16; m++) load_lane<T, VEC>(g[m], G + (node * 16 + m) * C, sub, false);
  __shared__ __align__(16) T harmonics[kWarpsPerBlock][2][EDGES * H::LD], sums[kWarpsPerBlock][EDGES * H::LD];
  int turn = 0;
  int32_t next[AT][2];
  auto look_up = [&](int64_t e) {
#pragma unroll
    for (int a = 0; a < AT; a++) {
      const int64_t i = e + a * EPW + slot < e1 ? e + a * EPW + slot : e1 - 1;
      next[a][0] = __ldg(sender + i);
      next[a][1] = PAIR && row_of ? __ldg(row_of + i) : (int32_t)i;
    }
  };
  look_up(begin);
  for (int64_t e = begin; e < e1; e += EDGES * slices, turn ^= 1) {
    T yv[H::PER];
#pragma unroll
    for (int i = 0; i < H::PER; i++) {
      int edge, m;
      yv[i] = T(0);
      if (H::at(i, lane, ys, edge, m) && e + edge < e1) yv[i] = __ldg(Y + m * ys.m + (e + edge) * ys.e);
    }
    T x[AT][VEC], r[AT][4][VEC], d[PAIR ? AT : 1][4][VEC];
#pragma unroll
    for (int a = 0; a < AT; a++) {   // an edge beyond the receiver's last is that one; it is not stored
      load_lane<T, VEC>(x[a], X + (int64_t)next[a][0] * C, sub, false);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        load_lane<T, VEC>(r[a][l], R + ((int64_t)next[a][1] * 4 + l) * C, sub, !PAIR);
        if constexpr (PAIR) load_lane<T, VEC>(d[a][l], dR + ((int64_t)next[a][1] * 4 + l) * C, sub, false);
      }
    }
    look_up(e + EDGES * slices);
    T *yp = harmonics[warp][turn];
#pragma unroll
    for (int i = 0; i < H::PER; i++) {
      int edge, m;
      if (H::at(i, lane, ys, edge, m)) yp[edge * H::LD + m] = yv[i];
    }
    __syncwarp();   // and everybody has read the sums of the edges before
#pragma unroll
    for (int a = 0; a < AT; a++) {
      const int64_t ee = e + a * EPW + slot;
      const bool there = ee < e1;
      T y[16], p[16], t[VEC], w[VEC];
      take16<T>(y, yp + (a * EPW + slot) * H::LD);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        T u[VEC], rx[VEC];
#pragma unroll
        for (int v = 0; v < VEC; v++) rx[v] = r[a][l][v] * x[a][v];
#pragma unroll
        for (int m = l * l; m < (l + 1) * (l + 1); m++) {
          T pm = T(0);
#pragma unroll
          for (int v = 0; v < VEC; v++) {
            u[v] = m == l * l ? y[m] * g[m][v] : fma(y[m], g[m][v], u[v]);
            pm = fma(g[m][v], rx[v], pm);
          }
          p[m] = pm;
        }
        T gr[VEC];
#pragma unroll
        for (int v = 0; v < VEC; v++) {
          t[v] = l == 0 ? u[v] * r[a][l][v] : fma(u[v], r[a][l][v], t[v]);
          if constexpr (PAIR) w[v] = l == 0 ? u[v] * d[a][l][v] : fma(u[v], d[a][l][v], w[v]);
          else gr[v] = x[a][v] * u[v];
        }
        if constexpr (!PAIR)
          if (gradR != nullptr && there) store_lane<T, VEC>(gradR + (ee * 4 + l) * C, sub, gr, true);
      }
      if constexpr (PAIR) {
        p[0] = T(0);
#pragma unroll
        for (int v = 0; v < VEC; v++) p[0] = fma(x[a][v], w[v], p[0]);
      }
      if (Tout != nullptr && there) store_lane<T, VEC>(Tout + ee * C, sub, t, false);
      slot_reduce16<T, LANES>(p, lane);
      T *q = sums[warp] + (a * EPW + slot) * H::LD;
      if constexpr (LANES == 32) {
        if ((lane & 1) == 0) q[lane >> 1] = p[0];
      } else if constexpr (LANES == 16) {
        q[sub] = p[0];
      } else {
        q[2 * sub] = p[0];
        q[2 * sub + 1] = p[1];
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < H::PER; i++) {
      int edge, m;
      if (H::at(i, lane, ys, edge, m) && e + edge < e1) gradY[m * ys.m + (e + edge) * ys.e] = sums[warp][edge * H::LD + m];
    }
  }
}

// ---- edge pass with the R rows staged through shared memory (float32, 128 channels) -------------------------
// The kernel above keeps the loads of one pair of edges in flight per warp, and the register budget allows 12
// warps per SM: about 48 KB in flight, not enough to cover HBM latency at full bandwidth.  Here every warp owns a
// ring of BS_SLOTS shared-memory slots; one lane starts, BS_SLOTS edges ahead of where the warp computes, a bulk
// copy of the edge's four R rows (2 KB, contiguous) and of its sender's feature row (512 B) that completes on the
// slot's mbarrier.  160 KB per SM are then on their way from HBM at any time, independent of registers.
// The arithmetic per edge is that of imp_bwd_edge_kernel.  Everything this pass writes is per edge (gradY, T, gradR),
// so the edge list is cut into equal contiguous pieces, one per warp of a persistent grid, wherever the receiver
// boundaries fall (a warp reloads G when its edges move on to the next receiver): the warps finish together
// whatever the degrees are, which matters most for small systems (3 000 atoms: 2 368 warps, 0.139 -> 0.10 ms).
// Every wait is bounded and sets *stalled when it gives up.  Measured at 64 000 atoms: 3.36 ms with
// the register-prefetch kernel, 3.38 ms with 8 warps x 8 slots (two warps per scheduler cannot hide the latency of
// their own instruction chains), 3.06 ms with 16 warps x 4 slots, 3.22 ms with 16 x 5 (the modulo by 5).
constexpr int BS_WARPS = 16;
constexpr int BS_SLOTS = 4;
constexpr int BS_C = 128;
constexpr int BS_R_BYTES = 4 * BS_C * 4;
constexpr int BS_SLOT_BYTES = BS_R_BYTES + BS_C * 4;
constexpr long long BS_TIMEOUT_CYCLES = 400000000LL;   // bound of every wait, about 0.2 s

// position in a warp's piece [e, end) of the receiver-sorted edge list: edge e belongs to receiver `node`, whose
// edges end at e1; e = -1 when the piece is exhausted
struct EdgeCursor {
  int64_t node, e, e1, end;
};

// first = first edge of the piece: the receiver is found by bisection in row_ptr [nnodes + 1]
__device__ __forceinline__ void cursor_start(EdgeCursor &c, const int32_t *__restrict__ row_ptr, int64_t nnodes,
                                             int64_t first, int64_t end) {
  c.end = end;
  if (first >= end) {
    c.e = c.e1 = -1;
    c.node = 0;
    return;
  }
  int64_t lo = 0, hi = nnodes;   // invariant: row_ptr[lo] <= first < row_ptr[hi]
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (row_ptr[mid] <= first) lo = mid;
    else hi = mid;
  }
  c.node = lo;
  c.e = first;
  c.e1 = row_ptr[lo + 1];
}
__device__ __forceinline__ void cursor_next(EdgeCursor &c, const int32_t *__restrict__ row_ptr) {
  if (++c.e >= c.end) {
    c.e = -1;
    return;
  }
  while (c.e >= c.e1) c.e1 = row_ptr[++c.node + 1];   // receivers without edges are stepped over
}

// WANT_T / WANT_GR: whether T [E,C] and gradR [E,4,C] are written.  With neither (the first layer of a model whose
// radial gradient is formed inside the GEMM) u[l,c] is not needed at all, and Y is not read: gradY does not depend
// on it.
template <bool WANT_T, bool WANT_GR>
__global__ void __launch_bounds__(BS_WARPS * 32, 1)
    imp_bwd_edge_staged_kernel(const float *__restrict__ X, const float *__restrict__ Y, const float *__restrict__ R,
                               const float *__restrict__ G, const int32_t *__restrict__ sender,
                               const int32_t *__restrict__ row_ptr, int64_t nnodes, int64_t nedges, ImpLayout ys,
                               float *__restrict__ gradR, float *__restrict__ gy, float *__restrict__ Tout,
                               int *__restrict__ stalled) {
  grid_begin();
  extern __shared__ __align__(128) unsigned char bs_smem[];
  __shared__ __align__(8) uint64_t bs_bars[BS_WARPS][BS_SLOTS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(bs_smem) + (uint32_t)w * BS_SLOTS * BS_SLOT_BYTES;
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(&bs_bars[w][0]);
  if (lane == 0) {
    for (int s = 0; s < BS_SLOTS; s++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8 * s), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();

  const int64_t nwarps = (int64_t)gridDim.x * BS_WARPS, wid = (int64_t)blockIdx.x * BS_WARPS + w;
  const int64_t per = (nedges + nwarps - 1) / nwarps;
  const int64_t e_first = wid * per, e_end = e_first + per < nedges ? e_first + per : nedges;
  EdgeCursor ic, cc;   // where copies are issued, where the warp computes
  cursor_start(ic, row_ptr, nnodes, e_first, e_end);
  cc = ic;
  int64_t chunk_base = -64;
  int snd = 0;
  uint32_t icount = 0, ccount = 0;

  auto issue_one = [&]() {
    if (ic.e < 0) return;
    // sender indices of the issue stream, 32 at a time
    if (ic.e >= chunk_base + 32) {
      chunk_base = ic.e;
      snd = (ic.e + lane < ic.end) ? sender[ic.e + lane] : 0;
    }
    const int s = __shfl_sync(0xffffffffu, snd, (int)(ic.e - chunk_base));
    if (elect_one()) {
      const uint32_t slot = ring + (icount % BS_SLOTS) * BS_SLOT_BYTES, bar = bar0 + 8 * (icount % BS_SLOTS);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(BS_SLOT_BYTES) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(slot),
                   "l"(R + ic.e * (4 * BS_C)), "r"(BS_R_BYTES), "r"(bar)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       slot + BS_R_BYTES),
                   "l"(X + (int64_t)s * BS_C), "r"(BS_C * 4), "r"(bar)
                   : "memory");
    }
    icount++;
    cursor_next(ic, row_ptr);
  };
  for (int i = 0; i < BS_SLOTS; i++) issue_one();

  const int c0 = lane * 4;
  const int ylm = lane & 15;
  constexpr bool WANT_U = WANT_T || WANT_GR;
  unsigned long long g2[16][2];   // G[node, m, c0 .. c0 + 3] as two register pairs
  int64_t g_node = -1;
  float yv_next = (WANT_U && cc.e >= 0) ? __ldg(Y + ylm * ys.m + cc.e * ys.e) : 0.f;
  while (cc.e >= 0) {
    const int64_t e = cc.e, node = cc.node;
    EdgeCursor nc = cc;
    cursor_next(nc, row_ptr);
    const float yv = yv_next;
    if (WANT_U && nc.e >= 0) yv_next = __ldg(Y + ylm * ys.m + nc.e * ys.e);
    if (node != g_node) {
      g_node = node;
    #pragma unroll
      for (int m = 0; m < 16; m++) {
        const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(G + (node * 16 + m) * BS_C + c0));
        g2[m][0] = v.x;
        g2[m][1] = v.y;
      }
    }
    // wait for the edge's slot
    const uint32_t slot = ring + (ccount % BS_SLOTS) * BS_SLOT_BYTES, bar = bar0 + 8 * (ccount % BS_SLOTS);
    const uint32_t parity = (ccount / BS_SLOTS) & 1u;
    {
      uint32_t ok = 0;
      const long long t0 = clock64();
      for (;;) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok || clock64() - t0 > BS_TIMEOUT_CYCLES) break;
      }
      if (!__all_sync(0xffffffffu, ok != 0)) {
        // Give up on this warp's receivers, but not before the copies it still has in flight have landed: they
        // target this CTA's shared memory, which must stay allocated until they complete.  Slots ccount + 1 ..
        // icount - 1 are outstanding; each gets one more bounded wait.
        if (lane == 0 && stalled) atomicExch(stalled, 1);
        for (uint32_t k = ccount + 1; k < icount; k++) {
          const uint32_t kbar = bar0 + 8 * (k % BS_SLOTS), kpar = (k / BS_SLOTS) & 1u;
          uint32_t done = 0;
          const long long t1 = clock64();
          do {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(kbar), "r"(kpar)
                : "memory");
          } while (!done && clock64() - t1 < BS_TIMEOUT_CYCLES);
        }
        break;
      }
    }
    unsigned long long x2[2], r2[4][2], rx2[4][2];
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x2[0]), "=l"(x2[1]) : "r"(slot + BS_R_BYTES + lane * 16));
#pragma unroll
    for (int l = 0; l < 4; l++) {
      asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];"
                   : "=l"(r2[l][0]), "=l"(r2[l][1])
                   : "r"(slot + l * (BS_C * 4) + lane * 16));
      rx2[l][0] = mul2(r2[l][0], x2[0]);
      rx2[l][1] = mul2(r2[l][1], x2[1]);
    }
    unsigned long long u2[4][2];
    float p[16];
#pragma unroll
    for (int l = 0; l < 4; l++) u2[l][0] = u2[l][1] = 0ull;
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const int l = l_of_lm(m);
      if (WANT_U) {
        const float y = __shfl_sync(0xffffffffu, yv, m);
        const unsigned long long yy = pack2(y, y);
        u2[l][0] = fma2(yy, g2[m][0], u2[l][0]);
        u2[l][1] = fma2(yy, g2[m][1], u2[l][1]);
      }
      const unsigned long long pm = fma2(g2[m][1], rx2[l][1], mul2(g2[m][0], rx2[l][0]));
      float pa, pb;
      unpack2(pm, pa, pb);
      p[m] = pa + pb;
    }
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    if (WANT_T) {
      unsigned long long t2[2] = {0ull, 0ull};
#pragma unroll
      for (int l = 0; l < 4; l++) {
        t2[0] = fma2(u2[l][0], r2[l][0], t2[0]);
        t2[1] = fma2(u2[l][1], r2[l][1], t2[1]);
      }
      unpack2(t2[0], t[0], t[1]);
      unpack2(t2[1], t[2], t[3]);
    }
    if (WANT_GR) {
#pragma unroll
      for (int l = 0; l < 4; l++) {
        float gr[4];
        unpack2(mul2(x2[0], u2[l][0]), gr[0], gr[1]);
        unpack2(mul2(x2[1], u2[l][1]), gr[2], gr[3]);
        store_vec_stream<float, 4>(gradR + (e * 4 + l) * BS_C + c0, gr);
      }
    }
    // every value read from the slot has been consumed by now: the next copy may go into it
    __syncwarp();
    ccount++;
    issue_one();
    if (WANT_T) store_vec<float, 4>(Tout + e * BS_C + c0, t);
    const float tot = warp_reduce16(p, lane);
    if ((lane & 1) == 0) gy[(lane >> 1) * ys.m + e * ys.e] = tot;
    cc = nc;
  }
}

// gradY[m, e] = sum over chunks of partial[chunk, m, e]
template <typename T>
__global__ void sum_partials_kernel(const T *__restrict__ partial, int nchunks, int64_t n,
                                    T *__restrict__ out) {
  grid_begin();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  T s = T(0);
  for (int k = 0; k < nchunks; k++) s += partial[(int64_t)k * n + i];
  out[i] = s;
}

// Gathers rows of T by the sender's list: bound by the latency of a row and the warps there are to wait.  What the compiler keeps in
// flight follows the registers that it believes it has, so every width says for how many blocks an SM it is compiled (0: nothing said).
// SPLIT warps a sender (few senders), five blocks, three doubles a lane four (48 registers would spill); with nothing said 29 -> 25 us
// at 3 000 atoms of 128 channels in float32, 68 -> 58 at 8 000, 47 -> 37 in float64 at 3 000, 25 -> 21 with 96 channels.  (Six blocks:
// 29 and 64; eight rows at a time instead of four: 31 and 68; two rows, eight blocks: 25 and 54, but 23 with 96 channels.) One warp a
// sender, float32, at 16 000 atoms: 32 channels ten blocks 52 -> 44 (one 60, sixteen 64), 64 channels eight 70 -> 58 (one 60, ten 60,
// twelve 80; 209 -> 183 at 64 000), 128 channels one 95 -> 88 (eight 91, ten 117; 330 -> 301 at 64 000), 96 channels nothing said and
// the list's lines prefetched 81 (109 without the prefetch, which is no help to the others; one, six to nine 88, twelve 130); float64
// with 96 channels one 84 -> 76 at 8 000.  Registers that come of it: 48 of 256 threads (64 with three doubles a lane); of 128 threads
// in float32 48, 62, 48, 74 for one to four values a lane, in float64 64 or 80.  A compiler that arrives at others: measure again.
template <typename T, int VEC, int SPLIT>
constexpr int node_blocks_an_sm() {
  if (SPLIT > 1) return sizeof(T) * VEC <= 16 ? 5 : 4;
  if (sizeof(T) == 8) return 1;
  return VEC == 1 ? 10 : VEC == 2 ? 8 : VEC == 3 ? 0 : 1;
}

template <typename T, int VEC, int SPLIT>
__global__ void __launch_bounds__(SPLIT == 1 ? kWarpsPerBlock * 32 : SPLIT * 32, node_blocks_an_sm<T, VEC, SPLIT>())
    imp_bwd_node_kernel(const T *__restrict__ Tin, const int32_t *__restrict__ perm,
                        const int32_t *__restrict__ send_ptr, int64_t nnodes, int C,
                        T *__restrict__ gradX) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t node = SPLIT == 1 ? (int64_t)blockIdx.x * kWarpsPerBlock + warp : blockIdx.x;
  if (node >= nnodes) {
    grid_begin();
    return;
  }
  const int chunk = blockIdx.y * (32 * VEC);
  const int64_t k0 = send_ptr[node] + (SPLIT > 1 ? warp : 0), k1 = send_ptr[node + 1];
  if (VEC == 3 && k0 + 32 * lane < k1) asm volatile("prefetch.global.L1 [%0];" ::"l"(perm + k0 + 32 * lane));
  grid_begin();
  // 32 edges' indices in one load, then four rows in flight at a time
  constexpr int AHEAD = 4;
  T acc[2][VEC];
#pragma unroll
  for (int v = 0; v < VEC; v++) acc[0][v] = acc[1][v] = T(0);
  for (int64_t k = k0; k < k1; k += 32 * SPLIT) {
    const int64_t mine = k + (int64_t)SPLIT * lane;
    const int32_t e = mine < k1 ? perm[mine] : 0;
    const int n = (int)((k1 - k + SPLIT - 1) / SPLIT < 32 ? (k1 - k + SPLIT - 1) / SPLIT : 32);
    for (int j = 0; j < n; j += AHEAD) {
      T a[AHEAD][VEC];
#pragma unroll
      for (int u = 0; u < AHEAD; u++) {
        const int64_t row = __shfl_sync(0xffffffffu, e, (j + u) & 31);
        if (j + u < n) load_lane<T, VEC>(a[u], Tin + row * C + chunk, lane, false);
      }
#pragma unroll
      for (int u = 0; u < AHEAD; u++)
        if (j + u < n) {
#pragma unroll
          for (int v = 0; v < VEC; v++) acc[u & 1][v] += a[u][v];
        }
    }
  }
#pragma unroll
  for (int v = 0; v < VEC; v++) acc[0][v] += acc[1][v];
  if constexpr (SPLIT > 1) {
    __shared__ __align__(16) T part[SPLIT][32 * VEC];
#pragma unroll
    for (int v = 0; v < VEC; v++) part[warp][lane * VEC + v] = acc[0][v];
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int w = 1; w < SPLIT; w++)
#pragma unroll
      for (int v = 0; v < VEC; v++) acc[0][v] += part[w][lane * VEC + v];
  }
  store_lane<T, VEC>(gradX + node * C + chunk, lane, acc[0], false);
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
template <typename T>
static int check_common(const void *a, const void *b, const void *c, int64_t nnodes, int64_t nedges,
                        int C, const char *what) {
  if (nnodes < 0 || nedges < 0) return fail(CMACE_ERR_ARG, "%s: negative size", what);
  if (C <= 0 || C % 32 != 0)
    return fail(CMACE_ERR_UNSUPPORTED, "%s: channels must be a positive multiple of 32, got %d", what, C);
  if (nnodes > 0x7fffffffLL / kWarpsPerBlock * kWarpsPerBlock)
    return fail(CMACE_ERR_UNSUPPORTED, "%s: too many nodes", what);
  if (!aligned16(a) || !aligned16(b) || !aligned16(c))
    return fail(CMACE_ERR_ARG, "%s: pointers must be 16-byte aligned", what);
  return CMACE_OK;
}

// Warps per receiver when there are few (receiver, channel chunk) pairs: up to eight pairs an SM the eight-fold split
// is one wave of blocks and takes a quarter of the time; beyond that one warp a pair fills the chip by itself.
constexpr int kSplit = 8;
static bool few_nodes(int64_t pairs) { return pairs <= 148 * 8; }

template <typename T, int VEC, bool ROWS = false>
static void launch_fwd(const T *X, const T *Y, const T *R, const int32_t *row_of, const int32_t *sender,
                       const int32_t *row_ptr, int64_t nnodes, ImpLayout ys, int C, T *out,
                       cudaStream_t st) {
  const int chunks = C / (32 * VEC);
  if (few_nodes(nnodes * chunks)) {
    constexpr int smem = kSplit * 16 * 32 * VEC * (int)sizeof(T);
    cudaFuncSetAttribute(imp_fwd_kernel<T, VEC, kSplit, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    launch_chained(imp_fwd_kernel<T, VEC, kSplit, ROWS>, dim3((unsigned)nnodes, chunks), kSplit * 32, smem, st, X, Y, R, row_of, sender,
                   row_ptr, nnodes, ys, C, out);
    return;
  }
  dim3 grid((unsigned)((nnodes + kWarpsPerBlock - 1) / kWarpsPerBlock), chunks);
  launch_chained(imp_fwd_kernel<T, VEC, 1, ROWS>, grid, kWarpsPerBlock * 32, 0, st, X, Y, R, row_of, sender, row_ptr, nnodes, ys, C,
                 out);
}

// whether rows of C channels go several edges (or 96 channels) to a warp
template <typename T>
static bool takes_slots(int C) {
  return C == 32 || C == 96 || (sizeof(T) == 4 && C == 64);
}
template <typename T, int VEC, int LANES, bool ROWS>
static void launch_fwd_slots(const T *X, const T *Y, const T *R, const int32_t *row_of, const int32_t *sender, const int32_t *row_ptr,
                             int64_t nnodes, ImpLayout ys, T *out, cudaStream_t st) {
  // Warps a receiver while there are few: with 168 registers and more a thread an SM holds one or two blocks of eight warps.  us with
  // one, two, four and eight (and of the kernel for whole warps), float32: 64 channels, 52 edges a receiver 14.4, 7.3, 6.2, 6.2 (6.2)
  // at 64 receivers, 16.5, 8.3, 6.2, 9.4 (8.3) at 300, 19.7, 10.3, 10.6, 14.4 (12.1) at 600, 23.6, 16.5, 16.4, 22.8 (16.7) at 1 150; 30
  // edges 14.6, 12.4, 12.4, 18.5 (13.3) at 1 150; 32 channels 8.3, 8.4, 10.2, 14.4 (10.4); 96 channels, 52 edges, float32 28.7, 16.4,
  // 14.4, 14.5 (22.5) at 600, float64 29.1, 19.7, 14.4, 15.5 (22.6) at 300, 42.5, 40.2, 41.0, 47.7 (57.4) at 1 150.
  auto split = [&](auto warps) {
    constexpr int SPLIT = decltype(warps)::value, smem = SPLIT * 16 * VEC * LANES * (int)sizeof(T);
    auto kernel = imp_fwd_slots_kernel<T, VEC, LANES, SPLIT, ROWS>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    launch_chained(kernel, (unsigned)nnodes, SPLIT * 32, smem, st, X, Y, R, row_of, sender, row_ptr, nnodes, ys, out);
  };
  if (nnodes <= (VEC == 3 ? 222 : 148)) return split(std::integral_constant<int, 8>{});
  if (nnodes <= (VEC == 3 && sizeof(T) == 4 ? 800 : 444)) return split(std::integral_constant<int, 4>{});
  if (few_nodes(nnodes)) return split(std::integral_constant<int, 2>{});
  launch_chained(imp_fwd_slots_kernel<T, VEC, LANES, 1, ROWS>, (unsigned)((nnodes + kWarpsPerBlock - 1) / kWarpsPerBlock),
                 kWarpsPerBlock * 32, 0, st, X, Y, R, row_of, sender, row_ptr, nnodes, ys, out);
}
template <typename T, bool ROWS>
static void fwd_slots(const T *X, const T *Y, const T *R, const int32_t *row_of, const int32_t *sender, const int32_t *row_ptr,
                      int64_t nnodes, ImpLayout ys, int C, T *out, cudaStream_t st) {
  if (C == 96) launch_fwd_slots<T, 3, 32, ROWS>(X, Y, R, row_of, sender, row_ptr, nnodes, ys, out, st);
  else if constexpr (sizeof(T) == 8) launch_fwd_slots<T, 2, 16, ROWS>(X, Y, R, row_of, sender, row_ptr, nnodes, ys, out, st);
  else if (C == 64) launch_fwd_slots<T, 4, 16, ROWS>(X, Y, R, row_of, sender, row_ptr, nnodes, ys, out, st);
  else launch_fwd_slots<T, 4, 8, ROWS>(X, Y, R, row_of, sender, row_ptr, nnodes, ys, out, st);
}
template <typename T, bool PAIR>
static void bwd_edge_slots(const T *X, const T *Y, const T *R, const T *dR, const int32_t *row_of, const T *G, const int32_t *sender,
                           const int32_t *row_ptr, int64_t nnodes, int64_t nedges, ImpLayout ys, int C, T *gradR, T *gY, T *Tout,
                           cudaStream_t st) {
  // Warps a receiver while there are few: 444 blocks of four run at a time, and a warp takes four or eight edges.  us with four and
  // eight, 52 edges a receiver, float32, 64 channels: 8.3, 6.2 at 64 receivers, 11.3, 12.4 at 300, 20.4, 18.5 at 600, 30.9, 30.8
  // at 1 150; 8 edges, 32 channels: 4.4, 6.2 at 300, 6.2, 6.3 at 600, 8.3, 10.0 at 1 150.  96 channels, two edges a warp, 52: 20.6,
  // 16.4 at 300.
  const int slices = !few_nodes(nnodes) ? 1 : (C == 96 || nnodes <= 222 || (nnodes <= 700 && nedges >= 16 * nnodes) ? 8 : 4);
  auto launch = [&](auto kernel) {
    launch_chained(kernel, (unsigned)((nnodes * slices + kWarpsPerBlock - 1) / kWarpsPerBlock), kWarpsPerBlock * 32, 0, st, X, Y, R, dR,
                   row_of, G, sender, row_ptr, nnodes, ys, slices, gradR, gY, Tout);
  };
  if (C == 96) launch(imp_bwd_edge_slots_kernel<T, 3, 32, PAIR>);
  else if constexpr (sizeof(T) == 8) launch(imp_bwd_edge_slots_kernel<T, 2, 16, PAIR>);
  else if (C == 64) launch(imp_bwd_edge_slots_kernel<T, 4, 16, PAIR>);
  else launch(imp_bwd_edge_slots_kernel<T, 4, 8, PAIR>);
}

template <typename T>
int imp_fwd(const T *X, const T *Y, const T *R, const int32_t *sender, const int32_t *row_ptr,
            int64_t nnodes, int64_t nedges, ImpLayout ys, int C, T *out, cmace_stream_t stream) {
  int rc = check_common<T>(X, R, out, nnodes, nedges, C, "cmace_imp_fwd");
  if (rc) return rc;
  if (nnodes == 0) return CMACE_OK;
  if (!out || !row_ptr || (nedges > 0 && (!X || !R || !Y || !sender)))
    return fail(CMACE_ERR_ARG, "cmace_imp_fwd: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  // Many receivers of few edges leave places of a warp empty, us of the two kernels, float32: 32 channels, 20 000 receivers of 2 edges
  // 22.6 against 16.5, of 4 26.7, 24.6, of 6 30.8, 30.7, of 8 35.0, 36.9; 64 channels, of 2 34.9, 31.1, of 8 63.6, 61.4, of 12 81.4,
  // 79.8, 8 000 of 20 45.1, 45.1, of 30 61.8, 63.6.  At 1 300 receivers the places cost nothing; 96 channels and float64 gain at any
  // number of edges.
  const bool sparse = sizeof(T) == 4 && C <= 64 && nnodes >= 2000 && nedges < (C == 32 ? 6 : 20) * nnodes;
  if (takes_slots<T>(C) && !sparse) {
    fwd_slots<T, false>(X, Y, R, nullptr, sender, row_ptr, nnodes, ys, C, out, st);
    return check_launch("cmace_imp_fwd");
  }
  switch (pick_vec<T>(C)) {
    case 4:
      if constexpr (sizeof(T) == 4) launch_fwd<T, 4>(X, Y, R, nullptr, sender, row_ptr, nnodes, ys, C, out, st);
      break;
    case 2: launch_fwd<T, 2>(X, Y, R, nullptr, sender, row_ptr, nnodes, ys, C, out, st); break;
    default: launch_fwd<T, 1>(X, Y, R, nullptr, sender, row_ptr, nnodes, ys, C, out, st); break;
  }
  return check_launch("cmace_imp_fwd");
}

template <typename T, int VEC>
static void launch_bwd_edge(const T *X, const T *Y, const T *R, const T *G, const int32_t *sender,
                            const int32_t *row_ptr, int64_t nnodes, int64_t nedges, ImpLayout ys, int C, T *gradR,
                            T *gy, T *Tout, cudaStream_t st) {
  const int slices = few_nodes(nnodes * (C / (32 * VEC))) ? kSplit : 1;
  dim3 grid((unsigned)((nnodes * slices + kWarpsPerBlock - 1) / kWarpsPerBlock), C / (32 * VEC));
  launch_chained(imp_bwd_edge_kernel<T, VEC>, grid, kWarpsPerBlock * 32, 0, st, X, Y, R, G, sender, row_ptr,
                                                                     nnodes, nedges, ys, C, slices, 0, gradR, gy, Tout);
}
// the same without partials (no edge is left undefined: gradY starts from zero)
template <typename T, int VEC>
static int launch_bwd_edge_joined(const T *X, const T *Y, const T *R, const T *G, const int32_t *sender, const int32_t *row_ptr,
                                  int64_t nnodes, int64_t nedges, ImpLayout ys, int C, T *gradR, T *gradY, T *Tout,
                                  const char *what, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(gradY, 0, (size_t)(16 * nedges) * sizeof(T), st);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  // us with 1, 2, 4 and 8 slices at 128 channels: 300 receivers of 200 edges 222, 215, 178, 159; 800 of 80 194, 159, 163, 163; 2 000 of
  // 30 158, 150, 156, 169; 6 000 of 10 156, 167, 194, 240 (partials in memory and a pass that sums them: 134, 146, 149, 146)
  const int chunks = C / (32 * VEC), slices = few_nodes(2 * nnodes) ? 8 : (nnodes <= 4 * 148 * 8 ? 2 : 1);
  if (nnodes * slices > 0x7fffffffLL) return fail(CMACE_ERR_UNSUPPORTED, "%s: too many nodes", what);
  for (int chunk = 0; chunk < chunks; chunk += kWarpsPerBlock) {
    const int warps = chunks - chunk < kWarpsPerBlock ? chunks - chunk : kWarpsPerBlock;
    launch_chained(imp_bwd_edge_kernel<T, VEC, true>, (unsigned)(nnodes * slices), warps * 32, 0, st, X, Y, R, G, sender, row_ptr,
                   nnodes, nedges, ys, C, slices, chunk, gradR, gradY, Tout);
  }
  return check_launch(what);
}

int imp_bwd_edge_pair_f64(const double *X, const double *Y, const double *R, const double *dR, const int32_t *row_of,
                          const double *G, const int32_t *sender, const int32_t *row_ptr, int64_t nnodes, int64_t nedges, int C,
                          double *gY, double *T, cudaStream_t st) {
  if (nnodes == 0 || nedges == 0) return CMACE_OK;
  if (takes_slots<double>(C)) {
    bwd_edge_slots<double, true>(X, Y, R, dR, row_of, G, sender, row_ptr, nnodes, nedges, ImpLayout{1, 16}, C, nullptr, gY, T, st);
    return check_launch("cmace_step(edges_back)");
  }
  auto launch = [&](auto kernel, int chunks) {
    const int slices = few_nodes(nnodes * chunks) ? kSplit : 1;
    const dim3 grid((unsigned)((nnodes * slices + kWarpsPerBlock - 1) / kWarpsPerBlock), (unsigned)chunks);
    launch_chained(kernel, grid, kWarpsPerBlock * 32, 0, st, X, Y, R, dR, row_of, G, sender, row_ptr, nnodes, nedges, C, slices, gY, T);
  };
  launch(imp_bwd_edge_pair_kernel<2>, C / 64);
  return check_launch("cmace_step(edges_back)");
}
int imp_fwd_rows_f64(const double *X, const double *Y, const double *R, const int32_t *row_of, const int32_t *sender,
                     const int32_t *row_ptr, int64_t nnodes, int64_t nedges, int C, double *out, cudaStream_t st) {
  if (nnodes == 0) return CMACE_OK;
  const ImpLayout ys{1, 16};
  if (takes_slots<double>(C)) fwd_slots<double, true>(X, Y, R, row_of, sender, row_ptr, nnodes, ys, C, out, st);
  else launch_fwd<double, 2, true>(X, Y, R, row_of, sender, row_ptr, nnodes, ys, C, out, st);
  return check_launch("cmace_step(messages)");
}

static __device__ int g_staged_stall;   // set when a bounded wait of the staged edge pass gave up
int *staged_stall_flag() {
  static std::atomic<int *> per_device[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  int *p = per_device[dev].load(std::memory_order_relaxed);
  if (p == nullptr && cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_staged_stall) == cudaSuccess)
    per_device[dev].store(p, std::memory_order_relaxed);   // several threads: the same address
  return p;
}

template <typename T>
static int check_bwd_edge(const T *X, const T *Y, const T *R, const T *G, const int32_t *sender, const int32_t *row_ptr,
                          int64_t nnodes, int64_t nedges, int C, const T *gradR, const T *gradY, const T *Tout) {
  int rc = check_common<T>(X, R, G, nnodes, nedges, C, "cmace_imp_bwd_edge");
  if (rc || nnodes == 0 || nedges == 0) return rc;
  if (!X || !Y || !R || !G || !sender || !row_ptr || !gradY)
    return fail(CMACE_ERR_ARG, "cmace_imp_bwd_edge: null pointer");
  if ((gradR && !aligned16(gradR)) || (Tout && !aligned16(Tout)))
    return fail(CMACE_ERR_ARG, "cmace_imp_bwd_edge: outputs must be 16-byte aligned");
  return CMACE_OK;
}

template <typename T>
int imp_bwd_edge(const T *X, const T *Y, const T *R, const T *G, const int32_t *sender,
                        const int32_t *row_ptr, int64_t nnodes, int64_t nedges, ImpLayout ys, int C, T *gradR,
                        T *gradY, T *Tout, T *partial, cmace_stream_t stream) {
  int rc = check_bwd_edge<T>(X, Y, R, G, sender, row_ptr, nnodes, nedges, C, gradR, gradY, Tout);
  if (rc || nnodes == 0 || nedges == 0) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  // as in the forward, us of the two kernels: 20 000 receivers of 1 edge 28.7 against 20.5 (32 channels), 31.2, 25.7 (64), 36.9, 28.7
  // (32 in float64), of 2 edges 32.8, 28.7, 47.1, 44.9, 49.2, 46.7, of 3 39.0, 41.0, 55.3, 55.2, 61.3, 62.9; 3 000 of 1 edge 8.3, 6.2,
  // of 2 8.3, 8.3
  const bool sparse = C <= 64 && nnodes >= 2000 && 2 * nedges < (nnodes >= 6000 ? 6 : 3) * nnodes;
  if (takes_slots<T>(C) && !sparse) {   // a whole row at a time: no partials
    bwd_edge_slots<T, false>(X, Y, R, nullptr, nullptr, G, sender, row_ptr, nnodes, nedges, ys, C, gradR, gradY, Tout, st);
    return check_launch("cmace_imp_bwd_edge");
  }
  const int vec = pick_vec<T>(C);
  const int nchunks = C / (32 * vec);
  if (nchunks > 1 && !partial)
    return fail(CMACE_ERR_ARG, "cmace_imp_bwd_edge: gradY_partial scratch required for %d chunks", nchunks);
  T *gy = nchunks > 1 ? partial : gradY;
  if constexpr (sizeof(T) == 4) {
    if (C == BS_C && aligned16(R) && aligned16(X) && aligned16(G)) {
      static int num_sms = 0;
      if (num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (num_sms <= 0) num_sms = 148;
      }
      const size_t smem = (size_t)BS_WARPS * BS_SLOTS * BS_SLOT_BYTES;
      int64_t blocks = (nedges + BS_WARPS * 8 - 1) / (BS_WARPS * 8);   // at least a few edges a warp
      blocks = blocks < num_sms ? blocks : num_sms;
      auto launch = [&](auto kernel) -> int {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "cmace_imp_bwd_edge: %s", cudaGetErrorString(e));
        launch_chained(kernel, (unsigned)blocks, BS_WARPS * 32, smem, st, X, Y, R, G, sender, row_ptr, nnodes, nedges, ys, gradR, gy,
                                                              Tout, staged_stall_flag());
        return check_launch("cmace_imp_bwd_edge");
      };
      if (Tout && gradR) return launch(imp_bwd_edge_staged_kernel<true, true>);
      if (Tout) return launch(imp_bwd_edge_staged_kernel<true, false>);
      if (gradR) return launch(imp_bwd_edge_staged_kernel<false, true>);
      return launch(imp_bwd_edge_staged_kernel<false, false>);
    }
  }
  switch (vec) {
    case 4:
      if constexpr (sizeof(T) == 4)
        launch_bwd_edge<T, 4>(X, Y, R, G, sender, row_ptr, nnodes, nedges, ys, C, gradR, gy, Tout, st);
      break;
    case 2: launch_bwd_edge<T, 2>(X, Y, R, G, sender, row_ptr, nnodes, nedges, ys, C, gradR, gy, Tout, st); break;
    default: launch_bwd_edge<T, 1>(X, Y, R, G, sender, row_ptr, nnodes, nedges, ys, C, gradR, gy, Tout, st); break;
  }
  rc = check_launch("cmace_imp_bwd_edge");
  if (rc) return rc;
  if (nchunks > 1) {
    const int64_t n = 16 * nedges;
    launch_chained(sum_partials_kernel<T>, (unsigned)((n + 255) / 256), 256, 0, st, partial, nchunks, n, gradY);
    rc = check_launch("cmace_imp_bwd_edge(sum)");
  }
  return rc;
}

template <typename T, int VEC>
static void launch_bwd_node(const T *Tin, const int32_t *perm, const int32_t *send_ptr, int64_t nnodes, int64_t nedges,
                            int C, T *gradX, cudaStream_t st) {
  const int chunks = C / (32 * VEC);
  // float32: eight warps a sender (one; eight), us at 128 channels: 36.9; 23.4 at 3 000 nodes of 52 edges, 53.3; 47.1 at
  // 8 192 of 40, 69.6; 62.3 at 9 500 of 52, but 45.2; 43.0 at 8 192 of 32, 30.6; 32.9 of 20 and 16.0; 27.0 of 8: a warp
  // with fewer than four rows has its loads' latency and the sum through shared memory to pay for.  98.3; 96.3 at 16 000 of
  // 52 and 170.0; 176.3 at 32 000: one warp a sender fills the chip.  float64: 84 against 130 at 8 000 of 52.
  const bool dense = nedges < 0 || nedges >= 36 * nnodes;   // unknown: as in a condensed system
  if (sizeof(T) == 4 ? dense && nnodes * chunks <= 148 * 64 : few_nodes(nnodes * chunks)) {
    launch_chained(imp_bwd_node_kernel<T, VEC, kSplit>, dim3((unsigned)nnodes, chunks), kSplit * 32, 0, st, Tin, perm, send_ptr, nnodes, C,
                                                                                              gradX);
    return;
  }
  dim3 grid((unsigned)((nnodes + kWarpsPerBlock - 1) / kWarpsPerBlock), chunks);
  launch_chained(imp_bwd_node_kernel<T, VEC, 1>, grid, kWarpsPerBlock * 32, 0, st, Tin, perm, send_ptr, nnodes, C, gradX);
}

template <typename T>
int imp_bwd_node(const T *Tin, const int32_t *perm, const int32_t *send_ptr, int64_t nnodes, int64_t nedges, int C,
                 T *gradX, cmace_stream_t stream) {
  int rc = check_common<T>(Tin, gradX, gradX, nnodes, 0, C, "cmace_imp_bwd_node");
  if (rc) return rc;
  if (nnodes == 0) return CMACE_OK;
  if (!send_ptr || !gradX) return fail(CMACE_ERR_ARG, "cmace_imp_bwd_node: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (C == 96) {   // one pass over the rows instead of three
    launch_bwd_node<T, 3>(Tin, perm, send_ptr, nnodes, nedges, C, gradX, st);
    return check_launch("cmace_imp_bwd_node");
  }
  switch (pick_vec<T>(C)) {
    case 4:
      if constexpr (sizeof(T) == 4) launch_bwd_node<T, 4>(Tin, perm, send_ptr, nnodes, nedges, C, gradX, st);
      break;
    case 2: launch_bwd_node<T, 2>(Tin, perm, send_ptr, nnodes, nedges, C, gradX, st); break;
    default: launch_bwd_node<T, 1>(Tin, perm, send_ptr, nnodes, nedges, C, gradX, st); break;
  }
  return check_launch("cmace_imp_bwd_node");
}

#define CMACE_IMP_LAUNCHERS(T)                                                                                        \
  template int imp_fwd<T>(const T *, const T *, const T *, const int32_t *, const int32_t *, int64_t, int64_t, ImpLayout, \
                          int, T *, cmace_stream_t);                                                                   \
  template int imp_bwd_edge<T>(const T *, const T *, const T *, const T *, const int32_t *, const int32_t *, int64_t,  \
                               int64_t, ImpLayout, int, T *, T *, T *, T *, cmace_stream_t);                           \
  template int imp_bwd_node<T>(const T *, const int32_t *, const int32_t *, int64_t, int64_t, int, T *, cmace_stream_t);
CMACE_IMP_LAUNCHERS(float)
CMACE_IMP_LAUNCHERS(double)

// ---- variant without caller scratch -------------------------------------------------------------
// Some callers cannot hand over scratch memory because they cannot allocate on the device at the point
// of the call: a plugin running inside another framework's memory pool that is already sized, or a
// host thread that must not call into an allocator while the device is busy.  For those, the float64
// edge backward adds up the channel chunks' shares of gradY in its blocks; nothing is shared between calls.
constexpr int64_t kNoallocElems = 2 * 1024 * 1024;  // scratch doubles a call would need otherwise, e.g. 65 536 edges at C = 128

}  // namespace cmace

using namespace cmace;

extern "C" {

int cmace_imp_staged_stalled(void) {
  int *flag = staged_stall_flag();
  int v = 0;
  if (flag == nullptr) return 0;
  if (cudaMemcpy(&v, flag, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v != 0) cudaMemset(flag, 0, sizeof(int));
  return v;
}

int cmace_imp_fwd_f32(const float *X, const float *Y, const float *R, const int32_t *sender,
                      const int32_t *row_ptr, int64_t nnodes, int64_t nedges, int channels, float *out,
                      cmace_stream_t stream) {
  return imp_fwd<float>(X, Y, R, sender, row_ptr, nnodes, nedges, ImpLayout{nedges, 1}, channels, out, stream);
}
int cmace_imp_fwd_f64(const double *X, const double *Y, const double *R, const int32_t *sender,
                      const int32_t *row_ptr, int64_t nnodes, int64_t nedges, int channels, double *out,
                      cmace_stream_t stream) {
  return imp_fwd<double>(X, Y, R, sender, row_ptr, nnodes, nedges, ImpLayout{nedges, 1}, channels, out, stream);
}
int64_t cmace_imp_bwd_scratch_elems(int64_t nedges, int channels, int is_f64) {
  if (channels <= 0 || channels % 32 != 0) return 0;
  const int vec = is_f64 ? pick_vec<double>(channels) : pick_vec<float>(channels);
  const int nchunks = channels / (32 * vec);
  return nchunks > 1 ? (int64_t)nchunks * 16 * nedges : 0;
}
int cmace_imp_bwd_edge_f32(const float *X, const float *Y, const float *R, const float *G,
                           const int32_t *sender, const int32_t *row_ptr, int64_t nnodes, int64_t nedges,
                           int channels, float *gradR, float *gradY, float *T, float *gradY_partial,
                           cmace_stream_t stream) {
  return imp_bwd_edge<float>(X, Y, R, G, sender, row_ptr, nnodes, nedges, ImpLayout{nedges, 1}, channels, gradR, gradY, T,
                             gradY_partial, stream);
}
int cmace_imp_bwd_edge_f64(const double *X, const double *Y, const double *R, const double *G,
                           const int32_t *sender, const int32_t *row_ptr, int64_t nnodes, int64_t nedges,
                           int channels, double *gradR, double *gradY, double *T, double *gradY_partial,
                           cmace_stream_t stream) {
  return imp_bwd_edge<double>(X, Y, R, G, sender, row_ptr, nnodes, nedges, ImpLayout{nedges, 1}, channels, gradR, gradY, T,
                              gradY_partial, stream);
}
int64_t cmace_imp_bwd_edge_f64_noalloc_max_elems(void) { return kNoallocElems; }

int cmace_imp_bwd_edge_f64_noalloc(const double *X, const double *Y, const double *R, const double *G,
                                   const int32_t *sender, const int32_t *row_ptr, int64_t nnodes, int64_t nedges,
                                   int channels, double *gradR, double *gradY, double *T, cmace_stream_t stream) {
  const int64_t need = cmace_imp_bwd_scratch_elems(nedges, channels, 1);
  const ImpLayout ys{nedges, 1};
  if (need > kNoallocElems)
    return fail(CMACE_ERR_UNSUPPORTED,
                "cmace_imp_bwd_edge_f64_noalloc: %lld scratch elements needed, calls are limited to the %lld of its former "
                "built-in array (reduce the number of edges per call or use cmace_imp_bwd_edge_f64 with your own scratch)",
                (long long)need, (long long)kNoallocElems);
  if (need == 0 || takes_slots<double>(channels))
    return imp_bwd_edge<double>(X, Y, R, G, sender, row_ptr, nnodes, nedges, ys, channels, gradR, gradY, T, nullptr, stream);
  const int rc = check_bwd_edge<double>(X, Y, R, G, sender, row_ptr, nnodes, nedges, channels, gradR, gradY, T);
  if (rc || nnodes == 0 || nedges == 0) return rc;
  auto run = [&](auto launch) {
    return launch(X, Y, R, G, sender, row_ptr, nnodes, nedges, ys, channels, gradR, gradY, T, "cmace_imp_bwd_edge_f64_noalloc",
                  (cudaStream_t)stream);
  };
  return pick_vec<double>(channels) == 2 ? run(launch_bwd_edge_joined<double, 2>) : run(launch_bwd_edge_joined<double, 1>);
}

int cmace_imp_bwd_node_f32(const float *T, const int32_t *perm, const int32_t *send_ptr, int64_t nnodes,
                           int channels, float *gradX, cmace_stream_t stream) {
  return imp_bwd_node<float>(T, perm, send_ptr, nnodes, -1, channels, gradX, stream);
}
int cmace_imp_bwd_node_f64(const double *T, const int32_t *perm, const int32_t *send_ptr, int64_t nnodes,
                           int channels, double *gradX, cmace_stream_t stream) {
  return imp_bwd_node<double>(T, perm, send_ptr, nnodes, -1, channels, gradX, stream);
}
int cmace_imp_bwd_node_edges(int is_f64, const void *T, const int32_t *perm, const int32_t *send_ptr, int64_t nnodes,
                             int64_t nedges, int channels, void *gradX, cmace_stream_t stream) {
  if (is_f64)
    return imp_bwd_node<double>(static_cast<const double *>(T), perm, send_ptr, nnodes, nedges, channels,
                                static_cast<double *>(gradX), stream);
  return imp_bwd_node<float>(static_cast<const float *>(T), perm, send_ptr, nnodes, nedges, channels,
                             static_cast<float *>(gradX), stream);
}
}
