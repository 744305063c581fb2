// Kernels of the energy+force step that walk nodes: the symmetric contraction (generated program, one thread per
// channel), fused in the second layer with the readout and its own gradient, and the products between the layers.
//
// All weights between the first contraction's output b0 [n, C] and what the rest of the model reads from it are
// folded when the model is laid out: up1 = b0 Wu (product and linear_up of the two layers), q0 = b0 Wsc[z] (product,
// skip connection and first readout layer: the skip term only ever enters the second readout) and e0 = b0 . w0.
#include "step_common.cuh"
#include "symcon_canonical.inc"

namespace cmace {

static_assert(ST_NW == canon::NCLASS3 + canon::NCLASS2 + 1, "effective weights per channel");

// effective weights of one (element, channel), weff [Z][13][C]
template <typename T>
__device__ __forceinline__ void load_weff(const T *__restrict__ weff, int z, int C, int c, T (&w3)[canon::NCLASS3],
                                          T (&w2)[canon::NCLASS2], T &w1) {
  const T *w = weff + (int64_t)z * ST_NW * C + c;
#pragma unroll
  for (int q = 0; q < canon::NCLASS3; q++) w3[q] = __ldg(w + q * C);
#pragma unroll
  for (int q = 0; q < canon::NCLASS2; q++) w2[q] = __ldg(w + (canon::NCLASS3 + q) * C);
  w1 = __ldg(w + (ST_NW - 1) * C);
}

template <typename T, bool BWD>
__global__ void __launch_bounds__(128)
    step_contract_kernel(const T *__restrict__ X, const int32_t *__restrict__ types, const T *__restrict__ weff,
                         const T *__restrict__ gb, int64_t nnodes, int C, T *__restrict__ out) {
  const int c = threadIdx.x;
  for (int64_t node = blockIdx.x; node < nnodes; node += gridDim.x) {
    T x[16], g[16], w3[canon::NCLASS3], w2[canon::NCLASS2], w1, value;
    const T *xr = X + node * 16 * C + c;
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = __ldcs(xr + i * C);
    load_weff(weff, types[node], C, c, w3, w2, w1);
    const T go = BWD ? gb[node * C + c] : T(0);
    canon::eval<T>(x, w3, w2, w1, g, value);
    if (BWD) {
      T *o = out + node * 16 * C + c;
#pragma unroll
      for (int i = 0; i < 16; i++) __stcs(o + i * C, go * g[i]);
    } else {
      out[node * C + c] = value;
    }
  }
}

static int64_t node_blocks(int64_t n, int per_sm) {
  const int64_t cap = (int64_t)148 * per_sm;
  return n < cap ? n : cap;
}

template <typename T>
int StepKernels<T>::contract_fwd(const T *X, const int32_t *types, const T *weff, int64_t n, int C, T *b,
                                 cudaStream_t st) {
  if (n > 0) step_contract_kernel<T, false><<<(unsigned)node_blocks(n, 12), C, 0, st>>>(X, types, weff, nullptr, n, C, b);
  return check_launch("cmace_step(contract_fwd)");
}
template <typename T>
int StepKernels<T>::contract_bwd(const T *X, const int32_t *types, const T *weff, const T *gb, int64_t n, int C, T *gX,
                                 cudaStream_t st) {
  if (n > 0) step_contract_kernel<T, true><<<(unsigned)node_blocks(n, 12), C, 0, st>>>(X, types, weff, gb, n, C, gX);
  return check_launch("cmace_step(contract_bwd)");
}

// Second layer: value b and gradient factors from one evaluation; q = q0 + b Wp1 (float64), the readout
// e1 = sum_j silu(q_j) w2_j, and back: grad b = Wp1 (silu'(q) w2), grad X = grad b * dB/dx.  w2 carries the
// activation's normalisation.  C threads per node; the 16 sums over channels go through two barriers.
template <typename T>
__global__ void __launch_bounds__(128)
    contract_readout_kernel(const T *__restrict__ X, const int32_t *__restrict__ types, const T *__restrict__ weff,
                            const double *__restrict__ wp1, const double *__restrict__ w2ro,
                            const double *__restrict__ q0, const double *__restrict__ e0,
                            const double *__restrict__ atomic_e, double scale, double shift, int64_t nnodes, int C,
                            T *__restrict__ gX, double *__restrict__ dq_out, double *__restrict__ inter,
                            double *__restrict__ node_energy) {
  __shared__ double part[4][ST_RO];
  __shared__ double dq_s[ST_RO];
  const int c = threadIdx.x, lane = c & 31, w = c >> 5, nw = C >> 5;
  double wp[ST_RO];
#pragma unroll
  for (int j = 0; j < ST_RO; j++) wp[j] = wp1[c * ST_RO + j];
  for (int64_t node = blockIdx.x; node < nnodes; node += gridDim.x) {
    T x[16], g[16], w3[canon::NCLASS3], w2[canon::NCLASS2], w1, value;
    const T *xr = X + node * 16 * C + c;
    const int z = types[node];
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = __ldcs(xr + i * C);
    load_weff(weff, z, C, c, w3, w2, w1);
    canon::eval<T>(x, w3, w2, w1, g, value);
    double p[ST_RO];
#pragma unroll
    for (int j = 0; j < ST_RO; j++) p[j] = (double)value * wp[j];
    // 16 sums over the warp's lanes at once: every lane ends with component lane >> 1
    {
      double q8[8], q4[4], q2[2];
      bool up = lane & 16;
#pragma unroll
      for (int i = 0; i < 8; i++) q8[i] = (up ? p[i + 8] : p[i]) + __shfl_xor_sync(0xffffffffu, up ? p[i] : p[i + 8], 16);
      up = lane & 8;
#pragma unroll
      for (int i = 0; i < 4; i++) q4[i] = (up ? q8[i + 4] : q8[i]) + __shfl_xor_sync(0xffffffffu, up ? q8[i] : q8[i + 4], 8);
      up = lane & 4;
#pragma unroll
      for (int i = 0; i < 2; i++) q2[i] = (up ? q4[i + 2] : q4[i]) + __shfl_xor_sync(0xffffffffu, up ? q4[i] : q4[i + 2], 4);
      up = lane & 2;
      double r = (up ? q2[1] : q2[0]) + __shfl_xor_sync(0xffffffffu, up ? q2[0] : q2[1], 2);
      r += __shfl_xor_sync(0xffffffffu, r, 1);
      if ((lane & 1) == 0) part[w][lane >> 1] = r;
    }
    __syncthreads();
    if (c < 32) {
      double e1 = 0.0;
      if (c < ST_RO) {
        double q = q0[node * ST_RO + c];
        for (int k = 0; k < nw; k++) q += part[k][c];
        const double s = 1.0 / (1.0 + exp(-q));
        const double wj = w2ro[c];
        e1 = q * s * wj;
        const double d = scale * wj * s * (1.0 + q * (1.0 - s));
        dq_s[c] = d;
        dq_out[node * ST_RO + c] = d;
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) e1 += __shfl_xor_sync(0xffffffffu, e1, off);
      if (c == 0) {
        const double v = scale * (e0[node] + e1) + shift;
        inter[node] = v;
        node_energy[node] = atomic_e[z] + v;
      }
    }
    __syncthreads();
    double gbd = 0.0;
#pragma unroll
    for (int j = 0; j < ST_RO; j++) gbd = fma(dq_s[j], wp[j], gbd);
    const T go = (T)gbd;
    T *o = gX + node * 16 * C + c;
#pragma unroll
    for (int i = 0; i < 16; i++) __stcs(o + i * C, go * g[i]);
  }
}

template <typename T>
int StepKernels<T>::contract_readout(const T *X, const int32_t *types, const T *weff, const double *wp1,
                                     const double *w2, const double *q0, const double *e0, const double *atomic_e,
                                     double scale, double shift, int64_t n, int C, T *gX, double *dq, double *inter,
                                     double *node_energy, cudaStream_t st) {
  if (n > 0)
    contract_readout_kernel<T><<<(unsigned)node_blocks(n, 8), C, 0, st>>>(X, types, weff, wp1, w2, q0, e0, atomic_e, scale,
                                                                         shift, n, C, gX, dq, inter, node_energy);
  return check_launch("cmace_step(contract_readout)");
}

// ---- between the layers --------------------------------------------------------------------------------------------
// One block per MID_NODES consecutive nodes, their input rows in shared memory.  Thread t owns output column t mod C of
// every MID_GROUPS-th node; a weight is loaded once (coalesced, L1 / L2) for all of the thread's nodes and multiplies
// values that the whole warp reads from one shared-memory address.  The float64 parts (q0, e0) are 17 short dot
// products a node.
constexpr int MID_THREADS = 256;

template <typename T, int NODES>
__global__ void __launch_bounds__(MID_THREADS)
    mid_fwd_kernel(const T *__restrict__ b, const int32_t *__restrict__ slot_of, const int32_t *__restrict__ species,
                   const T *__restrict__ wu, const double *__restrict__ wsc, const double *__restrict__ w0, int64_t n,
                   int C, T *__restrict__ up, double *__restrict__ q0, double *__restrict__ e0) {
  __shared__ __align__(16) T rows[NODES][128];
  const int64_t first = (int64_t)blockIdx.x * NODES;
  const int nn = n - first < NODES ? (int)(n - first) : NODES;
  const int tid = threadIdx.x;
  for (int i = tid; i < NODES * C; i += MID_THREADS) {
    const int j = i / C, c = i - j * C;
    rows[j][c] = j < nn ? b[(int64_t)slot_of[first + j] * C + c] : T(0);
  }
  __syncthreads();
  const int groups = MID_THREADS / C;   // threads beyond groups * C (C = 96) only help with the dot products
  const int c = tid % C, gidx = tid / C;
  if (gidx < groups) {
    constexpr int MAXN = NODES / 2;     // C = 128: two groups
    for (int j0 = gidx * MAXN; j0 < NODES; j0 += groups * MAXN) {
      T acc[MAXN];
#pragma unroll
      for (int j = 0; j < MAXN; j++) acc[j] = T(0);
      for (int k = 0; k < C; k += 4) {
        T w[4];
#pragma unroll
        for (int u = 0; u < 4; u++) w[u] = __ldg(wu + (k + u) * C + c);
#pragma unroll
        for (int j = 0; j < MAXN; j++) {
          const Quad<T> v = *reinterpret_cast<const Quad<T> *>(&rows[j0 + j][k]);
          acc[j] = fma(v.x, w[0], acc[j]);
          acc[j] = fma(v.y, w[1], acc[j]);
          acc[j] = fma(v.z, w[2], acc[j]);
          acc[j] = fma(v.w, w[3], acc[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < MAXN; j++)
        if (j0 + j < nn) up[(first + j0 + j) * C + c] = acc[j];
    }
  }
  for (int i = tid; i < nn * ST_RO; i += MID_THREADS) {
    const int j = i / ST_RO, col = i - j * ST_RO;
    const double *w = wsc + ((int64_t)species[first + j] * C) * ST_RO + col;
    double a0 = 0.0, a1 = 0.0;
    for (int k = 0; k < C; k += 2) {
      a0 = fma((double)rows[j][k], __ldg(w + k * ST_RO), a0);
      a1 = fma((double)rows[j][k + 1], __ldg(w + (k + 1) * ST_RO), a1);
    }
    q0[(first + j) * ST_RO + col] = a0 + a1;
  }
  const int lane = tid & 31;
  for (int j = tid >> 5; j < nn; j += MID_THREADS / 32) {
    double a = 0.0;
    for (int k = lane; k < C; k += 32) a = fma((double)rows[j][k], __ldg(w0 + k), a);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if (lane == 0) e0[first + j] = a;
  }
}

// grad b0 [slot order] = grad up1 Wu^T + dq Wsc[z]^T + scale w0  (dq already carries the scale)
template <typename T, int NODES>
__global__ void __launch_bounds__(MID_THREADS)
    mid_bwd_kernel(const T *__restrict__ gup, const int32_t *__restrict__ slot_of, const int32_t *__restrict__ species,
                   const double *__restrict__ dq, const T *__restrict__ wu_t, const double *__restrict__ wsc,
                   const double *__restrict__ w0, double scale, int64_t n, int C, T *__restrict__ gb) {
  __shared__ __align__(16) T rows[NODES][128];
  __shared__ double dqs[NODES][ST_RO];
  const int64_t first = (int64_t)blockIdx.x * NODES;
  const int nn = n - first < NODES ? (int)(n - first) : NODES;
  const int tid = threadIdx.x;
  for (int i = tid; i < NODES * C; i += MID_THREADS) {
    const int j = i / C, c = i - j * C;
    rows[j][c] = j < nn ? gup[(first + j) * C + c] : T(0);
  }
  for (int i = tid; i < nn * ST_RO; i += MID_THREADS) dqs[i / ST_RO][i % ST_RO] = dq[first * ST_RO + i];
  __syncthreads();
  const int groups = MID_THREADS / C;
  const int c = tid % C, gidx = tid / C;
  if (gidx >= groups) return;
  constexpr int MAXN = NODES / 2;
  for (int j0 = gidx * MAXN; j0 < NODES; j0 += groups * MAXN) {
    T acc[MAXN];
#pragma unroll
    for (int j = 0; j < MAXN; j++) acc[j] = T(0);
    for (int k = 0; k < C; k += 4) {
      T w[4];
#pragma unroll
      for (int u = 0; u < 4; u++) w[u] = __ldg(wu_t + (k + u) * C + c);
#pragma unroll
      for (int j = 0; j < MAXN; j++) {
        const Quad<T> v = *reinterpret_cast<const Quad<T> *>(&rows[j0 + j][k]);
        acc[j] = fma(v.x, w[0], acc[j]);
        acc[j] = fma(v.y, w[1], acc[j]);
        acc[j] = fma(v.z, w[2], acc[j]);
        acc[j] = fma(v.w, w[3], acc[j]);
      }
    }
    const double base = scale * __ldg(w0 + c);
#pragma unroll
    for (int j = 0; j < MAXN; j++) {
      if (j0 + j >= nn) break;
      const int64_t node = first + j0 + j;
      const double *w = wsc + ((int64_t)species[node] * C + c) * ST_RO;
      double s = base;
#pragma unroll
      for (int k = 0; k < ST_RO; k++) s = fma(dqs[j0 + j][k], __ldg(w + k), s);
      gb[(int64_t)slot_of[node] * C + c] = (T)(s + (double)acc[j]);
    }
  }
}

// 16 nodes a block until that gives every SM two blocks, then 32 (twice the reuse of a weight)
template <typename T>
int StepKernels<T>::mid_fwd(const T *b, const int32_t *slot_of, const int32_t *species, const T *wu, const double *wsc,
                            const double *w0, int64_t n, int C, T *up, double *q0, double *e0, cudaStream_t st) {
  if (n > 0) {
    if (n < 32 * 148 * 2)
      mid_fwd_kernel<T, 16><<<(unsigned)((n + 15) / 16), MID_THREADS, 0, st>>>(b, slot_of, species, wu, wsc, w0, n, C, up, q0, e0);
    else
      mid_fwd_kernel<T, 32><<<(unsigned)((n + 31) / 32), MID_THREADS, 0, st>>>(b, slot_of, species, wu, wsc, w0, n, C, up, q0, e0);
  }
  return check_launch("cmace_step(mid_fwd)");
}
template <typename T>
int StepKernels<T>::mid_bwd(const T *gup, const int32_t *slot_of, const int32_t *species, const double *dq,
                            const T *wu_t, const double *wsc, const double *w0, double scale, int64_t n, int C, T *gb,
                            cudaStream_t st) {
  if (n > 0) {
    if (n < 32 * 148 * 2)
      mid_bwd_kernel<T, 16><<<(unsigned)((n + 15) / 16), MID_THREADS, 0, st>>>(gup, slot_of, species, dq, wu_t, wsc, w0, scale, n, C, gb);
    else
      mid_bwd_kernel<T, 32><<<(unsigned)((n + 31) / 32), MID_THREADS, 0, st>>>(gup, slot_of, species, dq, wu_t, wsc, w0, scale, n, C, gb);
  }
  return check_launch("cmace_step(mid_bwd)");
}

#define CMACE_STEP_NODES(T)                                                                                          \
  template int StepKernels<T>::contract_fwd(const T *, const int32_t *, const T *, int64_t, int, T *, cudaStream_t); \
  template int StepKernels<T>::contract_bwd(const T *, const int32_t *, const T *, const T *, int64_t, int, T *,     \
                                            cudaStream_t);                                                           \
  template int StepKernels<T>::contract_readout(const T *, const int32_t *, const T *, const double *,               \
                                                const double *, const double *, const double *, const double *,      \
                                                double, double, int64_t, int, T *, double *, double *, double *,     \
                                                cudaStream_t);                                                       \
  template int StepKernels<T>::mid_fwd(const T *, const int32_t *, const int32_t *, const T *, const double *,       \
                                       const double *, int64_t, int, T *, double *, double *, cudaStream_t);         \
  template int StepKernels<T>::mid_bwd(const T *, const int32_t *, const int32_t *, const double *, const T *,       \
                                       const double *, const double *, double, int64_t, int, T *, cudaStream_t);
CMACE_STEP_NODES(float)
CMACE_STEP_NODES(double)

}  // namespace cmace
