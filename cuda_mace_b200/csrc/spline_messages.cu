// Messages of a step with tabulated radial weights: the spline is evaluated where the message is formed, and its
// derivative where the edge's gradient is, so that no [E, 4, C] array of weights or of their gradients exists.
//
//   forward    out[i, lm, c] = sum_{e in row(i)} X[s, c] Y[e, lm] R_l(r_e)[c]
//   backward   T[e, c]  = sum_l u_l R_l,  u_l = sum_{m in l} Y[e, lm] G[i, lm, c]
//              gY[e, lm] = sum_c G[i, lm, c] R_l X[s, c]
//              dr[e]    = sum_{l, c} R'_l X[s, c] u_l
//
// Work split as in message_passing.cu: a warp owns a receiver (or every SPLIT-th pair of its edges) and 32 VEC channels, a
// lane VEC of them; every pair of edges has its 2 x 16 coefficient loads in flight while the lengths, harmonics and rows
// of the next pair are fetched.  The table costs four coefficients per (edge, l, channel), 8 KB an edge at 128 channels,
// mostly from L2; what bounds it is the instructions around them and the latency that 16 warps an SM leave (0.5 issued
// a cycle and scheduler), so C is a template parameter (every offset an immediate: 282 -> 180 instructions per edge and
// 64 channels forward) and the interval is looked up once per edge (SplinePoint).  At 157 000 edges, C = 128, float32, a
// layer: evaluating R, storing it, reading it for the messages, and in the backward reading R, storing its gradient and
// reading that against the derivative took 78 + 75 us and 141 + 89 us; these take 88 us and 163 us.
#include "step_common.cuh"

namespace cmace {

template <typename T, int VEC, int C>
__device__ __forceinline__ void load_coeffs(T (&cf)[4][4][VEC], const SplineTable<T> &t, bool inside, int idx, int c0) {
  const T *p = t.coeffs + (int64_t)idx * 16 * C + c0;
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int l = 0; l < 4; l++) {
      if (inside) {
        load_vec<T, VEC>(cf[q][l], p + (q * 4 + l) * C);
      } else {
#pragma unroll
        for (int v = 0; v < VEC; v++) cf[q][l][v] = T(0);
      }
    }
}

constexpr int SM_WARPS = 4, SM_SPLIT = 8;

template <typename T, int VEC, int C, int SPLIT>
__global__ void __launch_bounds__(SPLIT == 1 ? SM_WARPS * 32 : SPLIT * 32)
    spline_messages_kernel(const T *__restrict__ X, const int32_t *__restrict__ row_of, const T *__restrict__ Y,
                           const SplinePoint<T> *__restrict__ r, const SplineTable<T> table, const int32_t *__restrict__ sender,
                           const int32_t *__restrict__ row_ptr, int64_t nnodes, const int32_t *__restrict__ out_row,
                           T *__restrict__ out) {
  grid_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t node = SPLIT == 1 ? (int64_t)blockIdx.x * SM_WARPS + warp : blockIdx.x;
  if (node >= nnodes) return;
  const int c0 = blockIdx.y * (32 * VEC) + lane * VEC;
  const int64_t e0 = row_ptr[node] + (SPLIT > 1 ? 2 * warp : 0), e1 = row_ptr[node + 1];
  T acc[16][VEC];
#pragma unroll
  for (int m = 0; m < 16; m++)
#pragma unroll
    for (int v = 0; v < VEC; v++) acc[m][v] = T(0);
  // lengths, harmonics and rows of the next pair are on their way while a pair is worked on
  SplinePoint<T> rn[2];
  T yn = T(0);   // lanes 0 .. 15: the first edge's harmonics, 16 .. 31: the second's
  int32_t sn[2] = {0, 0};
  auto fetch = [&](int64_t e) {
    yn = Y[(lane < 16 || e + 1 >= e1 ? e : e + 1) * 16 + (lane & 15)];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t ee = e + h < e1 ? e + h : e;
      rn[h] = r[ee];
      const int32_t s = sender[ee];
      sn[h] = row_of ? row_of[s] : s;
    }
  };
  __shared__ __align__(16) PairHarmonics<T, SPLIT == 1 ? SM_WARPS : SPLIT> harmonics;
  int turn = 0;
  if (e0 < e1) fetch(e0);
  for (int64_t e = e0; e < e1; e += 2 * SPLIT, turn ^= 1) {
    T cf[2][4][4][VEC], xx[2][VEC], x[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      x[h] = rn[h].x;
      load_coeffs<T, VEC, C>(cf[h], table, rn[h].interval >= 0 && e + h < e1, (int)rn[h].interval, c0);
      load_vec<T, VEC>(xx[h], X + (int64_t)sn[h] * C + c0);
    }
    T *yp = harmonics.v[warp][turn];
    yp[lane] = yn;
    if (e + 2 * SPLIT < e1) fetch(e + 2 * SPLIT);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      T R[4][VEC];   // a missing second edge has zero weights
#pragma unroll
      for (int l = 0; l < 4; l++)
#pragma unroll
        for (int v = 0; v < VEC; v++)
          R[l][v] = (cf[h][0][l][v] + x[h] * (cf[h][1][l][v] + x[h] * (cf[h][2][l][v] + x[h] * cf[h][3][l][v]))) * xx[h][v];
      T y[16];
      take16<T>(y, yp + 16 * h);
#pragma unroll
      for (int m = 0; m < 16; m++)
#pragma unroll
        for (int v = 0; v < VEC; v++) acc[m][v] = fma(y[m], R[l_of_lm(m)][v], acc[m][v]);
    }
  }
  T *o = out + (out_row ? (int64_t)out_row[node] : node) * 16 * C + c0;
  if constexpr (SPLIT > 1) {
    extern __shared__ __align__(16) unsigned char sm_smem[];
    T *part = reinterpret_cast<T *>(sm_smem);   // [SPLIT][16][32 VEC]
#pragma unroll
    for (int m = 0; m < 16; m++) store_vec<T, VEC>(part + ((warp * 16 + m) * 32 + lane) * VEC, acc[m]);
    __syncthreads();
    for (int m = warp; m < 16; m += SPLIT) {
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

// Every channel chunk writes its own share of gY [chunks, E, 16] and dr [chunks, E]; the pass that turns them into the
// gradient of the edge's vector adds them up.
template <typename T, int VEC, int C>
__global__ void __launch_bounds__(SM_WARPS * 32, sizeof(T) == 4 ? 4 : 3)
    spline_edges_back_kernel(const T *__restrict__ X, const int32_t *__restrict__ row_of, const T *__restrict__ Y,
                             const SplinePoint<T> *__restrict__ r, const SplineTable<T> table, const T *__restrict__ G,
                             const int32_t *__restrict__ g_row, const int32_t *__restrict__ sender,
                             const int32_t *__restrict__ row_ptr, int64_t nnodes, int64_t nedges, int slices,
                             T *__restrict__ Tout, T *__restrict__ gY, T *__restrict__ dr) {
  grid_begin();
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * SM_WARPS + (threadIdx.x >> 5);
  const int64_t node = slices == 1 ? item : item / slices;
  const int slice = slices == 1 ? 0 : (int)(item - node * slices);
  if (node >= nnodes) return;
  const int c0 = blockIdx.y * (32 * VEC) + lane * VEC;
  const int64_t e0 = row_ptr[node] + 2 * slice, e1 = row_ptr[node + 1];
  if (e0 >= e1) return;
  gY += (int64_t)blockIdx.y * 16 * nedges;
  dr += (int64_t)blockIdx.y * nedges;
  T g[16][VEC];
  const int64_t grow = g_row ? (int64_t)g_row[node] : node;
#pragma unroll
  for (int m = 0; m < 16; m++) load_vec<T, VEC>(g[m], G + (grow * 16 + m) * C + c0);
  SplinePoint<T> rn[2];
  T yn;
  int32_t sn[2];
  auto fetch = [&](int64_t e) {
    yn = Y[(lane < 16 || e + 1 >= e1 ? e : e + 1) * 16 + (lane & 15)];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t ee = e + h < e1 ? e + h : e;
      rn[h] = r[ee];
      const int32_t s = sender[ee];
      sn[h] = row_of ? row_of[s] : s;
    }
  };
  __shared__ __align__(16) PairHarmonics<T, SM_WARPS> harmonics;
  int turn = 0;
  fetch(e0);
  for (int64_t e = e0; e < e1; e += 2 * slices, turn ^= 1) {
    T cf[2][4][4][VEC], xx[2][VEC], x[2], d[2] = {T(0), T(0)};
#pragma unroll
    for (int h = 0; h < 2; h++) {
      x[h] = rn[h].x;
      load_coeffs<T, VEC, C>(cf[h], table, rn[h].interval >= 0 && e + h < e1, (int)rn[h].interval, c0);
      load_vec<T, VEC>(xx[h], X + (int64_t)sn[h] * C + c0);
    }
    T *yp = harmonics.v[threadIdx.x >> 5][turn];
    yp[lane] = yn;
    if (e + 2 * slices < e1) fetch(e + 2 * slices);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (h && e + 1 >= e1) break;   // warp-uniform
      const int64_t ee = e + h;
      T y[16], p[16], t[VEC];
      take16<T>(y, yp + 16 * h);
#pragma unroll
      for (int v = 0; v < VEC; v++) t[v] = T(0);
#pragma unroll
      for (int l = 0; l < 4; l++) {
        T rx[VEC], u[VEC];
#pragma unroll
        for (int v = 0; v < VEC; v++) {
          const T a = cf[h][0][l][v], b = cf[h][1][l][v], c = cf[h][2][l][v], q = cf[h][3][l][v];
          u[v] = T(0);
#pragma unroll
          for (int m = l * l; m < (l + 1) * (l + 1); m++) u[v] = fma(y[m], g[m][v], u[v]);
          const T R = a + x[h] * (b + x[h] * (c + x[h] * q));
          t[v] = fma(u[v], R, t[v]);
          rx[v] = R * xx[h][v];
          d[h] = fma((b + x[h] * (T(2) * c + T(3) * x[h] * q)) * xx[h][v], u[v], d[h]);
        }
#pragma unroll
        for (int m = l * l; m < (l + 1) * (l + 1); m++) {
          T pm = T(0);
#pragma unroll
          for (int v = 0; v < VEC; v++) pm = fma(g[m][v], rx[v], pm);
          p[m] = pm;
        }
      }
      if (Tout != nullptr) store_vec<T, VEC>(Tout + ee * C + c0, t);
      const T tot = warp_reduce16(p, lane);
      if ((lane & 1) == 0) gY[ee * 16 + (lane >> 1)] = tot;
    }
    // dE/dr of both edges in one reduction: the lower half of the warp ends up with the first edge's
    const bool up = lane & 16;
    T s = (up ? d[1] : d[0]) + __shfl_xor_sync(0xffffffffu, up ? d[0] : d[1], 16);
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((lane & 15) == 0 && (!up || e + 1 < e1)) dr[e + (up ? 1 : 0)] = s;
  }
}

// two channels a lane (float32, whole chunks of 64) keep two edges' coefficients in 64 registers
template <typename T>
static constexpr int channels_per_lane(int C) { return sizeof(T) == 4 && C % 64 == 0 ? 2 : 1; }

template <typename T>
int spline_chunks(int C) { return C / (32 * channels_per_lane<T>(C)); }

// as in message_passing.cu: eight warps a receiver while that is one wave of blocks
static bool few_nodes(int64_t pairs) { return pairs <= 148 * 8; }

template <typename T, int C>
static void launch_messages(const T *X, const int32_t *row_of, const T *Y, const SplinePoint<T> *r, const SplineTable<T> &table,
                            const int32_t *sender, const int32_t *row_ptr, int64_t n, const int32_t *out_row, T *out,
                            cudaStream_t st) {
  constexpr int VEC = channels_per_lane<T>(C), chunks = C / (32 * VEC);
  if (few_nodes(n * chunks)) {
    constexpr int smem = SM_SPLIT * 16 * 32 * VEC * (int)sizeof(T);
    cudaFuncSetAttribute(spline_messages_kernel<T, VEC, C, SM_SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    launch_chained(spline_messages_kernel<T, VEC, C, SM_SPLIT>, dim3((unsigned)n, chunks), SM_SPLIT * 32, smem, st, X, row_of,
                   Y, r, table, sender, row_ptr, n, out_row, out);
    return;
  }
  launch_chained(spline_messages_kernel<T, VEC, C, 1>, dim3((unsigned)((n + SM_WARPS - 1) / SM_WARPS), chunks), SM_WARPS * 32,
                 0, st, X, row_of, Y, r, table, sender, row_ptr, n, out_row, out);
}

template <typename T>
int spline_messages(const T *X, const int32_t *row_of, const T *Y, const SplinePoint<T> *r, const SplineTable<T> &table,
                    const int32_t *sender, const int32_t *row_ptr, int64_t n, const int32_t *out_row, int C, T *out,
                    cudaStream_t st) {
  switch (C) {
    case 32: launch_messages<T, 32>(X, row_of, Y, r, table, sender, row_ptr, n, out_row, out, st); break;
    case 64: launch_messages<T, 64>(X, row_of, Y, r, table, sender, row_ptr, n, out_row, out, st); break;
    case 96: launch_messages<T, 96>(X, row_of, Y, r, table, sender, row_ptr, n, out_row, out, st); break;
    default: launch_messages<T, 128>(X, row_of, Y, r, table, sender, row_ptr, n, out_row, out, st); break;
  }
  return check_launch("cmace_step(messages)");
}

template <typename T, int C>
static void launch_back(const T *X, const int32_t *row_of, const T *Y, const SplinePoint<T> *r, const SplineTable<T> &table, const T *G,
                        const int32_t *g_row, const int32_t *sender, const int32_t *row_ptr, int64_t n, int64_t E, T *Tout,
                        T *gY, T *dr, cudaStream_t st) {
  constexpr int VEC = channels_per_lane<T>(C), chunks = C / (32 * VEC);
  const int slices = few_nodes(n * chunks) ? SM_SPLIT : 1;
  launch_chained(spline_edges_back_kernel<T, VEC, C>, dim3((unsigned)((n * slices + SM_WARPS - 1) / SM_WARPS), chunks),
                 SM_WARPS * 32, 0, st, X, row_of, Y, r, table, G, g_row, sender, row_ptr, n, E, slices, Tout, gY, dr);
}

template <typename T>
int spline_edges_back(const T *X, const int32_t *row_of, const T *Y, const SplinePoint<T> *r, const SplineTable<T> &table, const T *G,
                      const int32_t *g_row, const int32_t *sender, const int32_t *row_ptr, int64_t n, int64_t E, int C,
                      T *Tout, T *gY, T *dr, cudaStream_t st) {
  switch (C) {
    case 32: launch_back<T, 32>(X, row_of, Y, r, table, G, g_row, sender, row_ptr, n, E, Tout, gY, dr, st); break;
    case 64: launch_back<T, 64>(X, row_of, Y, r, table, G, g_row, sender, row_ptr, n, E, Tout, gY, dr, st); break;
    case 96: launch_back<T, 96>(X, row_of, Y, r, table, G, g_row, sender, row_ptr, n, E, Tout, gY, dr, st); break;
    default: launch_back<T, 128>(X, row_of, Y, r, table, G, g_row, sender, row_ptr, n, E, Tout, gY, dr, st); break;
  }
  return check_launch("cmace_step(edges_back)");
}

#define CMACE_SPLINE_MESSAGES(T)                                                                                         \
  template int spline_chunks<T>(int);                                                                                    \
  template int spline_messages<T>(const T *, const int32_t *, const T *, const SplinePoint<T> *, const SplineTable<T> &,              \
                                  const int32_t *, const int32_t *, int64_t, const int32_t *, int, T *, cudaStream_t);   \
  template int spline_edges_back<T>(const T *, const int32_t *, const T *, const SplinePoint<T> *, const SplineTable<T> &, const T *, \
                                    const int32_t *, const int32_t *, const int32_t *, int64_t, int64_t, int, T *, T *,  \
                                    T *, cudaStream_t);
CMACE_SPLINE_MESSAGES(float)
CMACE_SPLINE_MESSAGES(double)

}  // namespace cmace
