// Kernels of the energy+force step that walk edges.
//
// The first layer's sender features depend on the sender's element alone, x[s, c] = x_z[c], and the radial weights
// are R[e, l, c] = sum_k h[e, k] W[k, l c].  The message therefore factors,
//
//   m[i, lm, c] = sum_z sum_k ( sum_{e in (i, z)} Y[lm, e] h[e, k] ) x_z[c] W[k, l c],
//
// and the edges only have to form A[i, lm, z, k] = sum_{e in (i, z)} Y[lm, e] h[e, k]: 16 x 64 sums per (receiver,
// element) instead of 4 C radial weights per edge.  The rest is an element-dependent Linear of width 64 Z whose weight
// also absorbs the layer's own Linear.  The backward is the mirror image: with P = grad A[i, :, z, :]
//
//   grad Y[lm, e] = sum_k P[lm, k] h[e, k],   d E / d r_e += sum_k h'[e, k] sum_lm Y[lm, e] P[lm, k],
//
// where h' = dh/dr came with the forward, so no gradient passes back through the perceptron.
#include "edge_math.cuh"
#include "step_common.cuh"

namespace cmace {

// ---- edge geometry, basis and node grouping ----------------------------------------------------------------------
constexpr int EP_THREADS = 256;
constexpr int EP_MAX_NB = 16;

// Block 0 resolves the species and groups the owned nodes by element (stable): thread t counts and then places the
// nodes of its own consecutive piece, so equal elements keep their order.  It runs beside the edge blocks.
template <typename OH>
__device__ int first_max(const OH *row, int n) {
  int best = 0;
  OH v = row[0];
  for (int k = 1; k < n; k++)
    if (row[k] > v) {
      v = row[k];
      best = k;
    }
  return best;
}

__device__ void group_nodes(const int32_t *species_in, const void *one_hot, int one_hot_f64, int64_t n_local,
                            int64_t n_owned, int elements, int32_t *species, int32_t *slot_of, int32_t *node_of,
                            int32_t *slot_type, int32_t *elem_start) {
  __shared__ int count[ST_MAX_Z][EP_THREADS + 1];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int64_t per = (n_owned + EP_THREADS - 1) / EP_THREADS;
  const int64_t lo = t * per < n_owned ? t * per : n_owned, hi = lo + per < n_owned ? lo + per : n_owned;
  for (int z = 0; z < elements; z++) count[z][t] = 0;
  // coalesced pass over the species first: the counting pass then reads what this block wrote
  for (int64_t i = t; i < n_local; i += EP_THREADS) {
    int z;
    if (species_in) z = species_in[i];
    else if (one_hot_f64) z = first_max(static_cast<const double *>(one_hot) + i * elements, elements);
    else z = first_max(static_cast<const float *>(one_hot) + i * elements, elements);
    species[i] = z < 0 ? 0 : (z >= elements ? elements - 1 : z);
  }
  __syncthreads();
  for (int64_t i = lo; i < hi; i++) count[species[i]][t]++;
  __syncthreads();
  // exclusive prefix over (element, thread): warp w scans elements w, w + 8, ...
  __shared__ int total[ST_MAX_Z];
  for (int z = w; z < elements; z += EP_THREADS / 32) {
    int run = 0;
    for (int b = 0; b < EP_THREADS; b += 32) {
      const int v = count[z][b + lane];
      int inc = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += o;
      }
      count[z][b + lane] = run + inc - v;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) total[z] = run;
  }
  __syncthreads();
  if (t == 0) {
    int acc = 0;
    for (int z = 0; z < elements; z++) {
      elem_start[z] = acc;
      const int c = total[z];
      total[z] = acc;
      acc += c;
    }
    elem_start[elements] = acc;
  }
  __syncthreads();
  for (int64_t i = lo; i < hi; i++) {
    const int z = species[i];
    const int s = total[z] + count[z][t]++;
    slot_of[i] = s;
    node_of[s] = (int32_t)i;
    slot_type[s] = z;
  }
}

// One thread per edge: vector in float64, then unit vector and 1/r, basis and its derivative [E, 2 nb], Y [E, 16].
template <typename T>
__global__ void __launch_bounds__(EP_THREADS)
    edge_prep_kernel(const double *__restrict__ pos, const int32_t *__restrict__ sender,
                     const int32_t *__restrict__ receiver, const double *__restrict__ shifts, int64_t nedges, T r_max,
                     int nb, int p, Quad<T> *__restrict__ geo, T *__restrict__ basis, T *__restrict__ Y,
                     const int32_t *species_in, const void *one_hot, int one_hot_f64, int64_t n_local, int64_t n_owned,
                     int elements, int32_t *species, int32_t *slot_of, int32_t *node_of, int32_t *slot_type,
                     int32_t *elem_start) {
  if (blockIdx.x == 0) {
    group_nodes(species_in, one_hot, one_hot_f64, n_local, n_owned, elements, species, slot_of, node_of, slot_type,
                elem_start);
    return;
  }
  const int64_t e = (int64_t)(blockIdx.x - 1) * EP_THREADS + threadIdx.x;
  if (e >= nedges) return;
  const int64_t s = sender[e], r = receiver[e];
  T v[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    double d = __dsub_rn(pos[s * 3 + c], pos[r * 3 + c]);
    if (shifts) d = __dadd_rn(d, shifts[e * 3 + c]);
    v[c] = (T)d;
  }
  const T r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
  const T ir = inv_sqrt(r2);
  const T ux = v[0] * ir, uy = v[1] * ir, uz = v[2] * ir;
  T y[16];
  sph_l3<T>(uz, ux, uy, y);
  geo[e] = Quad<T>{ux, uy, uz, ir};
  Quad<T> *yo = reinterpret_cast<Quad<T> *>(Y + e * 16);
#pragma unroll
  for (int i = 0; i < 4; i++) yo[i] = Quad<T>{y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]};
  if (basis != nullptr) {
    T b[EP_MAX_NB], db[EP_MAX_NB];
    bessel_cutoff<T>(r2 * ir, r_max, nb, p, b, db);
    T *bo = basis + e * 2 * nb;
    for (int n = 0; n < nb; n++) {
      bo[n] = b[n];
      bo[nb + n] = db[n];
    }
  }
}

template <typename T>
int StepKernels<T>::edge_prep(const double *pos, const int32_t *sender, const int32_t *receiver, const double *shifts,
                              int64_t nedges, double r_max, int nb, int p, Quad<T> *geo, T *basis, T *Y,
                              const int32_t *species_in, const void *one_hot, int one_hot_f64, int64_t n_local,
                              int64_t n_owned, int elements, int32_t *species, int32_t *slot_of, int32_t *node_of,
                              int32_t *slot_type, int32_t *elem_start, cudaStream_t st) {
  const int64_t blocks = 1 + (nedges + EP_THREADS - 1) / EP_THREADS;
  edge_prep_kernel<T><<<(unsigned)blocks, EP_THREADS, 0, st>>>(
      pos, sender, receiver, shifts, nedges, (T)r_max, nb, p, geo, basis, Y, species_in, one_hot, one_hot_f64, n_local,
      n_owned, elements, species, slot_of, node_of, slot_type, elem_start);
  return check_launch("cmace_step(edge_prep)");
}

// ---- the edges of one (receiver, element) pair -------------------------------------------------------------------
// A warp owns the pair.  It lists the edges whose sender has the element, 32 candidates at a time (ballot), into a
// per-warp buffer and calls body(list, n) whenever the buffer is full and at the end; edges come in list order.
constexpr int SU_WARPS = 4;
constexpr int SU_LIST = 64;

template <typename Body>
__device__ __forceinline__ void for_edges_of_element(const int32_t *__restrict__ sender,
                                                     const int32_t *__restrict__ species, int64_t e0, int64_t e1, int z,
                                                     int32_t *list, int lane, Body body) {
  int n = 0;
  for (int64_t eb = e0; eb < e1; eb += 32) {
    const int64_t e = eb + lane;
    const bool hit = e < e1 && species[sender[e]] == z;
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (hit) list[n + __popc(m & ((1u << lane) - 1u))] = (int32_t)e;
    n += __popc(m);
    if (n > SU_LIST - 32) {
      __syncwarp();
      body(n);
      __syncwarp();
      n = 0;
    }
  }
  __syncwarp();
  if (n > 0) body(n);
}

// sums over k0 = 2 lane, 2 lane + 1; float: accumulators paired over lm, so that Y pairs come straight from memory
template <typename T>
struct SumAcc {
  T a[16][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int m = 0; m < 16; m++) a[m][0] = a[m][1] = T(0);
  }
  __device__ __forceinline__ void add(const T *__restrict__ y, T h0, T h1) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const double2 v = __ldg(reinterpret_cast<const double2 *>(y) + i);
      a[2 * i][0] = fma(v.x, h0, a[2 * i][0]);
      a[2 * i][1] = fma(v.x, h1, a[2 * i][1]);
      a[2 * i + 1][0] = fma(v.y, h0, a[2 * i + 1][0]);
      a[2 * i + 1][1] = fma(v.y, h1, a[2 * i + 1][1]);
    }
  }
  __device__ __forceinline__ void get(int m, T &x0, T &x1) const { x0 = a[m][0]; x1 = a[m][1]; }
};
template <>
struct SumAcc<float> {
  unsigned long long a[8][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int m = 0; m < 8; m++) a[m][0] = a[m][1] = 0ull;
  }
  __device__ __forceinline__ void add(const float *__restrict__ y, float h0, float h1) {
    const unsigned long long h00 = pack2(h0, h0), h11 = pack2(h1, h1);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(y) + i);
      a[2 * i][0] = fma2(v.x, h00, a[2 * i][0]);
      a[2 * i][1] = fma2(v.x, h11, a[2 * i][1]);
      a[2 * i + 1][0] = fma2(v.y, h00, a[2 * i + 1][0]);
      a[2 * i + 1][1] = fma2(v.y, h11, a[2 * i + 1][1]);
    }
  }
  __device__ __forceinline__ void get(int m, float &x0, float &x1) const {
    float lo, hi;
    unpack2(a[m >> 1][0], lo, hi);
    x0 = (m & 1) ? hi : lo;
    unpack2(a[m >> 1][1], lo, hi);
    x1 = (m & 1) ? hi : lo;
  }
};

template <typename T>
__global__ void __launch_bounds__(SU_WARPS * 32)
    sums_kernel(const T *__restrict__ h, const T *__restrict__ Y, const int32_t *__restrict__ sender,
                const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ species,
                const int32_t *__restrict__ slot_of, int64_t nnodes, int elements, T *__restrict__ A) {
  __shared__ int32_t lists[SU_WARPS][SU_LIST];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (pair >= nnodes * elements) return;
  const int64_t node = pair / elements;
  const int z = (int)(pair - node * elements);
  int32_t *list = lists[w];
  SumAcc<T> acc;
  acc.zero();
  using V2 = typename Vec<T, 2>::type;
  for_edges_of_element(sender, species, row_ptr[node], row_ptr[node + 1], z, list, lane, [&](int n) {
    int j = 0;
    for (; j + 3 < n; j += 4) {   // four edges' rows on their way before the first is used
      int64_t e[4];
      V2 v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        e[u] = list[j + u];
        v[u] = __ldg(reinterpret_cast<const V2 *>(h + e[u] * ST_H) + lane);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) acc.add(Y + e[u] * 16, v[u].x, v[u].y);
    }
    for (; j < n; j++) {
      const int64_t e = list[j];
      const V2 v = __ldg(reinterpret_cast<const V2 *>(h + e * ST_H) + lane);
      acc.add(Y + e * 16, v.x, v.y);
    }
  });
  const int width = elements * ST_H;
  T *o = A + (int64_t)slot_of[node] * 16 * width + z * ST_H + 2 * lane;
#pragma unroll
  for (int m = 0; m < 16; m++) {
    V2 v;
    acc.get(m, v.x, v.y);
    *reinterpret_cast<V2 *>(o + (int64_t)m * width) = v;
  }
}

template <typename T>
int StepKernels<T>::sums(const T *h, const T *Y, const int32_t *sender, const int32_t *row_ptr, const int32_t *species,
                         const int32_t *slot_of, int64_t nnodes, int elements, T *A, cudaStream_t st) {
  const int64_t blocks = (nnodes * elements + SU_WARPS - 1) / SU_WARPS;
  if (blocks > 0) sums_kernel<T><<<(unsigned)blocks, SU_WARPS * 32, 0, st>>>(h, Y, sender, row_ptr, species, slot_of, nnodes, elements, A);
  return check_launch("cmace_step(sums)");
}

// ---- backward over the edges of a (receiver, element) pair, down to the gradient of the edge vector ---------------
// The warp holds P = grad A[i, :, z, 2 lane .. 2 lane + 1]; per edge 16 + 1 sums over k (warp transpose-reduce), which
// wait in shared memory until 32 edges (or the list's end) are there: then lane j turns edge j's numbers, plus the
// second layer's grad Y and dE/dr, into the gradient of its vector.
template <typename T>
__device__ __forceinline__ T reduce16(T (&p)[16], int lane) {
  T q8[8], q4[4], q2[2];
  bool up = lane & 16;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const T send = up ? p[i] : p[i + 8], keep = up ? p[i + 8] : p[i];
    q8[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  up = lane & 8;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const T send = up ? q8[i] : q8[i + 4], keep = up ? q8[i + 4] : q8[i];
    q4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  up = lane & 4;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const T send = up ? q4[i] : q4[i + 2], keep = up ? q4[i + 2] : q4[i];
    q2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  up = lane & 2;
  const T send = up ? q2[0] : q2[1], keep = up ? q2[1] : q2[0];
  T r = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);   // component lane >> 1
}

template <typename T>
struct PairGrad {   // P, as the accumulators above hold it
  T p[16][2];
  __device__ __forceinline__ void set(int m, T x0, T x1) { p[m][0] = x0; p[m][1] = x1; }
  // g[lm] = sum over this lane's k of P h; returns sum_k h'_k sum_lm Y P of this lane
  __device__ __forceinline__ T edge(const T *__restrict__ y, T h0, T h1, T d0, T d1, T (&g)[16]) const {
    T s0 = T(0), s1 = T(0);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const double2 v = __ldg(reinterpret_cast<const double2 *>(y) + i);
      s0 = fma(v.x, p[2 * i][0], s0);
      s1 = fma(v.x, p[2 * i][1], s1);
      s0 = fma(v.y, p[2 * i + 1][0], s0);
      s1 = fma(v.y, p[2 * i + 1][1], s1);
    }
#pragma unroll
    for (int m = 0; m < 16; m++) g[m] = fma(p[m][1], h1, p[m][0] * h0);
    return fma(s1, d1, s0 * d0);
  }
};
template <>
struct PairGrad<float> {
  unsigned long long p[8][2];
  __device__ __forceinline__ void set(int m, float x0, float x1) {
    float lo, hi;
    unpack2(p[m >> 1][0], lo, hi);
    p[m >> 1][0] = (m & 1) ? pack2(lo, x0) : pack2(x0, hi);
    unpack2(p[m >> 1][1], lo, hi);
    p[m >> 1][1] = (m & 1) ? pack2(lo, x1) : pack2(x1, hi);
  }
  __device__ __forceinline__ float edge(const float *__restrict__ y, float h0, float h1, float d0, float d1,
                                        float (&g)[16]) const {
    const unsigned long long h00 = pack2(h0, h0), h11 = pack2(h1, h1);
    unsigned long long s0 = 0ull, s1 = 0ull;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(y) + i);
      s0 = fma2(v.x, p[2 * i][0], s0);
      s1 = fma2(v.x, p[2 * i][1], s1);
      s0 = fma2(v.y, p[2 * i + 1][0], s0);
      s1 = fma2(v.y, p[2 * i + 1][1], s1);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) unpack2(fma2(p[i][1], h11, mul2(p[i][0], h00)), g[2 * i], g[2 * i + 1]);
    float a, b, c, d;
    unpack2(s0, a, b);
    unpack2(s1, c, d);
    return fmaf(c + d, d1, (a + b) * d0);
  }
};

template <typename T>
__global__ void __launch_bounds__(SU_WARPS * 32)
    sums_bwd_kernel(const T *__restrict__ gA, const T *__restrict__ h, const T *__restrict__ dh,
                    const T *__restrict__ Y, const int32_t *__restrict__ sender, const int32_t *__restrict__ row_ptr,
                    const int32_t *__restrict__ species, const int32_t *__restrict__ slot_of,
                    const T *__restrict__ gY1, const T *__restrict__ dr1, const Quad<T> *__restrict__ geo,
                    int64_t nnodes, int elements, T *__restrict__ gvec) {
  __shared__ int32_t lists[SU_WARPS][SU_LIST];
  __shared__ T stage[SU_WARPS][32 * 17];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (pair >= nnodes * elements) return;
  const int64_t node = pair / elements;
  const int z = (int)(pair - node * elements);
  int32_t *list = lists[w];
  T *st = stage[w];
  using V2 = typename Vec<T, 2>::type;
  PairGrad<T> P;
  {
    const int b = z >> 1, width = sums_block_width(elements, b);
    const T *g = gA + (int64_t)b * nnodes * (16 * 128) + (int64_t)slot_of[node] * 16 * width + (z & 1) * ST_H + 2 * lane;
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const V2 v = __ldg(reinterpret_cast<const V2 *>(g + m * width));
      P.set(m, v.x, v.y);
    }
  }
  for_edges_of_element(sender, species, row_ptr[node], row_ptr[node + 1], z, list, lane, [&](int n) {
    for (int j0 = 0; j0 < n; j0 += 32) {
      const int nj = n - j0 < 32 ? n - j0 : 32;
      V2 hv = V2{}, dv = V2{};
      if (nj > 0) {
        const int64_t e = list[j0];
        hv = __ldg(reinterpret_cast<const V2 *>(h + e * ST_H) + lane);
        dv = __ldg(reinterpret_cast<const V2 *>(dh + e * ST_H) + lane);
      }
      for (int j = 0; j < nj; j++) {
        const int64_t e = list[j0 + j];
        const V2 hc = hv, dc = dv;
        if (j + 1 < nj) {   // the next edge's rows
          const int64_t en = list[j0 + j + 1];
          hv = __ldg(reinterpret_cast<const V2 *>(h + en * ST_H) + lane);
          dv = __ldg(reinterpret_cast<const V2 *>(dh + en * ST_H) + lane);
        }
        T g[16];
        T r = P.edge(Y + e * 16, hc.x, hc.y, dc.x, dc.y, g);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
        const T tot = reduce16(g, lane);
        if ((lane & 1) == 0) st[j * 17 + (lane >> 1)] = tot;
        if (lane == 1) st[j * 17 + 16] = r;
      }
      __syncwarp();
      if (lane < nj) {
        const int64_t e = list[j0 + lane];
        T g[16];
        const Quad<T> *gy = reinterpret_cast<const Quad<T> *>(gY1 + e * 16);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const Quad<T> q = gy[i];
          g[4 * i] = st[lane * 17 + 4 * i] + q.x;
          g[4 * i + 1] = st[lane * 17 + 4 * i + 1] + q.y;
          g[4 * i + 2] = st[lane * 17 + 4 * i + 2] + q.z;
          g[4 * i + 3] = st[lane * 17 + 4 * i + 3] + q.w;
        }
        const T dr = st[lane * 17 + 16] + dr1[e];
        const Quad<T> q = geo[e];   // unit vector in the input's component order: harmonic axes are (z, x, y)
        T GX, GY, GZ;
        sph_l3_vjp<T>(q.z, q.x, q.y, g, GX, GY, GZ);
        gvec[e * 3] = GY * q.w + dr * q.x;
        gvec[e * 3 + 1] = GZ * q.w + dr * q.y;
        gvec[e * 3 + 2] = GX * q.w + dr * q.z;
      }
      __syncwarp();
    }
  });
}

template <typename T>
int StepKernels<T>::sums_bwd(const T *gA, const T *h, const T *dh, const T *Y, const int32_t *sender,
                             const int32_t *row_ptr, const int32_t *species, const int32_t *slot_of, const T *gY1,
                             const T *dr1, const Quad<T> *geo, int64_t nnodes, int elements, T *gvec, cudaStream_t st) {
  const int64_t blocks = (nnodes * elements + SU_WARPS - 1) / SU_WARPS;
  if (blocks > 0)
    sums_bwd_kernel<T><<<(unsigned)blocks, SU_WARPS * 32, 0, st>>>(gA, h, dh, Y, sender, row_ptr, species, slot_of, gY1,
                                                                   dr1, geo, nnodes, elements, gvec);
  return check_launch("cmace_step(sums_bwd)");
}

// ---- forces and energies ------------------------------------------------------------------------------------------
// One warp per atom sums its edges' gradients from both groupings (float64, fixed order, no atomics); block 0 adds up
// the energies meanwhile: sums[0] over node_energy, sums[1] over the interaction energies.
template <typename T>
__global__ void __launch_bounds__(256)
    forces_kernel(const T *__restrict__ g, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ perm,
                  const int32_t *__restrict__ send_ptr, int64_t nrecv, int64_t nsend, double sign,
                  double *__restrict__ out, const double *__restrict__ inter, const double *__restrict__ node_energy,
                  double *__restrict__ sums) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.x == 0) {
    __shared__ double part[2][8];
    double a = 0.0, b = 0.0;
    for (int64_t i = threadIdx.x; i < nrecv; i += 256) {
      a += node_energy[i];
      b += inter[i];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, off);
      b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    if (lane == 0) {
      part[0][w] = a;
      part[1][w] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      double s = 0.0;
      for (int k = 0; k < 8; k++) s += part[threadIdx.x][k];
      sums[threadIdx.x] = s;
    }
    return;
  }
  const int64_t n = (int64_t)(blockIdx.x - 1) * 8 + w;
  if (n >= nsend) return;
  double ax = 0.0, ay = 0.0, az = 0.0;
  for (int k = send_ptr[n] + lane; k < send_ptr[n + 1]; k += 32) {
    const int64_t e = perm[k];
    ax += (double)g[e * 3];
    ay += (double)g[e * 3 + 1];
    az += (double)g[e * 3 + 2];
  }
  if (n < nrecv) {
    for (int64_t e = row_ptr[n] + lane; e < row_ptr[n + 1]; e += 32) {
      ax -= (double)g[e * 3];
      ay -= (double)g[e * 3 + 1];
      az -= (double)g[e * 3 + 2];
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, off);
    ay += __shfl_xor_sync(0xffffffffu, ay, off);
    az += __shfl_xor_sync(0xffffffffu, az, off);
  }
  if (lane < 3) out[n * 3 + lane] = sign * (lane == 0 ? ax : (lane == 1 ? ay : az));
}

template <typename T>
int StepKernels<T>::forces(const T *gvec, const int32_t *row_ptr, const int32_t *perm, const int32_t *send_ptr,
                           int64_t nrecv, int64_t nsend, double sign, double *out, const double *inter,
                           const double *node_energy, double *sums, cudaStream_t st) {
  const int64_t blocks = 1 + (nsend + 7) / 8;
  forces_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(gvec, row_ptr, perm, send_ptr, nrecv, nsend, sign, out, inter,
                                                     node_energy, sums);
  return check_launch("cmace_step(forces)");
}

#define CMACE_STEP_EDGES(T)                                                                                         \
  template int StepKernels<T>::edge_prep(const double *, const int32_t *, const int32_t *, const double *, int64_t, \
                                         double, int, int, Quad<T> *, T *, T *, const int32_t *, const void *, int, \
                                         int64_t, int64_t, int, int32_t *, int32_t *, int32_t *, int32_t *,         \
                                         int32_t *, cudaStream_t);                                                  \
  template int StepKernels<T>::sums(const T *, const T *, const int32_t *, const int32_t *, const int32_t *,        \
                                    const int32_t *, int64_t, int, T *, cudaStream_t);                              \
  template int StepKernels<T>::sums_bwd(const T *, const T *, const T *, const T *, const int32_t *,                \
                                        const int32_t *, const int32_t *, const int32_t *, const T *, const T *,    \
                                        const Quad<T> *, int64_t, int, T *, cudaStream_t);                          \
  template int StepKernels<T>::forces(const T *, const int32_t *, const int32_t *, const int32_t *, int64_t,        \
                                      int64_t, double, double *, const double *, const double *, double *,          \
                                      cudaStream_t);
CMACE_STEP_EDGES(float)
CMACE_STEP_EDGES(double)

}  // namespace cmace
