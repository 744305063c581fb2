// Kernels of the energy+force step that walk nodes: the symmetric contraction (generated program, one thread per
// channel), fused in the second layer with the readout and its own gradient, and the products between the layers.
//
// All weights between the first contraction's output b0 [n, C] and what the rest of the model reads from it are
// folded when the model is laid out: up = b0 Wu (product and linear_up of the two layers) and q0 = b0 Wsc[z] [17]: product,
// skip connection and first readout matrix (the skip term only ever enters the second readout), and the first readout.
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
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 5 : 3)
    step_contract_kernel(const T *__restrict__ X, const int32_t *__restrict__ types, const T *__restrict__ weff,
                         const T *__restrict__ gb, int64_t nnodes, int C, T *__restrict__ out) {
  grid_begin();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
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

// threads a node: its channels, or the widest block of at most 128 that divides them
static int channel_block(int C) {
  if (C <= 128) return C;
  for (int ch = 128; ch > 32; ch -= 32)
    if (C % ch == 0) return ch;
  return 32;
}

static int64_t node_blocks(int64_t n, int per_sm) {
  const int64_t cap = (int64_t)148 * per_sm;
  return n < cap ? n : cap;
}

template <typename T>
int StepKernels<T>::contract_fwd(const T *X, const int32_t *types, const T *weff, int64_t n, int C, T *b,
                                 cudaStream_t st) {
  const int ch = channel_block(C);
  if (n > 0)
    launch_chained(step_contract_kernel<T, false>, dim3((unsigned)node_blocks(n, 12), C / ch), ch, 0, st, X, types, weff, nullptr, n, C, b);
  return check_launch("cmace_step(contract_fwd)");
}
template <typename T>
int StepKernels<T>::contract_bwd(const T *X, const int32_t *types, const T *weff, const T *gb, int64_t n, int C, T *gX,
                                 cudaStream_t st) {
  const int ch = channel_block(C);
  if (n > 0)
    launch_chained(step_contract_kernel<T, true>, dim3((unsigned)node_blocks(n, 12), C / ch), ch, 0, st, X, types, weff, gb, n, C, gX);
  return check_launch("cmace_step(contract_bwd)");
}

// Second layer: value b and gradient factors from one evaluation; q = q0 + b Wp1, the readout e1 = sum_j silu(q_j) w2_j
// (float64 from the sums over a warp's channels on), and back: grad b = Wp1 (silu'(q) w2), grad X = grad b * dB/dx.
// w2 carries the activation's normalisation.  C threads per node; the 16 sums over channels go through two barriers.
// q0 [n][17]: 16 of the hidden layer, then the first readout.
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 5 : 3)
    contract_readout_kernel(const T *__restrict__ X, const int32_t *__restrict__ types, const T *__restrict__ weff,
                            const T *__restrict__ wp1, const double *__restrict__ w2ro, const T *__restrict__ q0,
                            const double *__restrict__ atomic_e, double scale, double shift, int64_t nnodes, int C,
                            T *__restrict__ gX, T *__restrict__ dq_out, double *__restrict__ inter,
                            double *__restrict__ node_energy) {
  grid_begin();
  __shared__ T part[4][ST_RO];
  __shared__ T dq_s[ST_RO];
  const int c = threadIdx.x, lane = c & 31, w = c >> 5, nw = C >> 5;
  T wp[ST_RO];
#pragma unroll
  for (int j = 0; j < ST_RO; j++) wp[j] = __ldg(wp1 + j * C + c);
  for (int64_t node = blockIdx.x; node < nnodes; node += gridDim.x) {
    T x[16], g[16], w3[canon::NCLASS3], w2[canon::NCLASS2], w1, value;
    const T *xr = X + node * 16 * C + c;
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = __ldcs(xr + i * C);
    const int z = types[node];
    load_weff(weff, z, C, c, w3, w2, w1);
    double qd = 0.0, e0 = 0.0;
    if (c < ST_RO) qd = (double)q0[node * (ST_RO + 1) + c];
    if (c == 0) e0 = (double)q0[node * (ST_RO + 1) + ST_RO];
    canon::eval<T>(x, w3, w2, w1, g, value);
    T p[ST_RO];
#pragma unroll
    for (int j = 0; j < ST_RO; j++) p[j] = value * wp[j];
    // 16 sums over the warp's lanes at once: every lane ends with component lane >> 1
    {
      T q8[8], q4[4], q2[2];
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
      T r = (up ? q2[1] : q2[0]) + __shfl_xor_sync(0xffffffffu, up ? q2[0] : q2[1], 2);
      r += __shfl_xor_sync(0xffffffffu, r, 1);
      if ((lane & 1) == 0) part[w][lane >> 1] = r;
    }
    __syncthreads();
    if (c < 32) {
      double e1 = 0.0;
      if (c < ST_RO) {
        double q = qd;
        for (int k = 0; k < nw; k++) q += (double)part[k][c];
        const double s = 1.0 / (1.0 + exp(-q));
        const double wj = w2ro[c];
        e1 = q * s * wj;
        const T d = (T)(scale * wj * s * (1.0 + q * (1.0 - s)));
        dq_s[c] = d;
        dq_out[node * ST_RO + c] = d;
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) e1 += __shfl_xor_sync(0xffffffffu, e1, off);
      if (c == 0) {
        const double v = scale * (e0 + e1) + shift;
        inter[node] = v;
        node_energy[node] = atomic_e[z] + v;
      }
    }
    __syncthreads();
    T go = T(0);
#pragma unroll
    for (int j = 0; j < ST_RO; j++) go = fma(dq_s[j], wp[j], go);
    T *o = gX + node * 16 * C + c;
#pragma unroll
    for (int i = 0; i < 16; i++) __stcs(o + i * C, go * g[i]);
  }
}

template <typename T>
int StepKernels<T>::contract_readout(const T *X, const int32_t *types, const T *weff, const T *wp1, const double *w2,
                                     const T *q0, const double *atomic_e, double scale, double shift, int64_t n, int C,
                                     T *gX, T *dq, double *inter, double *node_energy, cudaStream_t st) {
  if (n > 0)
    launch_chained(contract_readout_kernel<T>, (unsigned)node_blocks(n, 10), C, 0, st, X, types, weff, wp1, w2, q0, atomic_e, scale,
                                                                          shift, n, C, gX, dq, inter, node_energy);
  return check_launch("cmace_step(contract_readout)");
}

// ---- between the layers --------------------------------------------------------------------------------------------
// Products with a [C, C] matrix that stays in shared memory (64 KB float32, 128 KB float64: one fill per block, blocks
// are persistent), plus 17 columns that depend on the element: 16 of the second readout's hidden layer and the first
// readout.  Nodes are taken in slot order, so the nodes of a tile nearly always share the element.  2 C threads: a
// thread owns 4 columns of NODES / 8 nodes; what bounds it is the shared-memory pipe (four 16-byte loads of weights
// and NODES / 8 of rows per 4 k).
constexpr int MID_EXTRA = ST_RO + 1;

template <typename T>
__device__ __forceinline__ void mid_fill(T *sW, const T *__restrict__ W, int C, int tid, int nthreads) {
  for (int i = tid; i < C * C / (16 / (int)sizeof(T)); i += nthreads) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(sW) + 16u * (uint32_t)i;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(reinterpret_cast<const char *>(W) + 16 * (int64_t)i) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// acc[i][u] = sum_k rows[j0 + i][k] W[k][4 tx + u]
template <typename T, int PER>
__device__ __forceinline__ void mid_product(const T *rows, const T *sW, int C, int j0, int tx, T (&acc)[PER][4]) {
#pragma unroll
  for (int i = 0; i < PER; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = T(0);
#pragma unroll 2
  for (int k = 0; k < C; k += 4) {
    Quad<T> r[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) r[i] = *reinterpret_cast<const Quad<T> *>(rows + (j0 + i) * C + k);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const Quad<T> w = *reinterpret_cast<const Quad<T> *>(sW + (k + u) * C + 4 * tx);
#pragma unroll
      for (int i = 0; i < PER; i++) {
        const T v = u == 0 ? r[i].x : (u == 1 ? r[i].y : (u == 2 ? r[i].z : r[i].w));
        acc[i][0] = fma(v, w.x, acc[i][0]);
        acc[i][1] = fma(v, w.y, acc[i][1]);
        acc[i][2] = fma(v, w.z, acc[i][2]);
        acc[i][3] = fma(v, w.w, acc[i][3]);
      }
    }
  }
}

// extra: [Z][C/4][17][4]
template <typename T, int NODES>
__global__ void __launch_bounds__(256)
    mid_fwd_kernel(const T *__restrict__ b, const int32_t *__restrict__ node_of, const int32_t *__restrict__ slot_type,
                   const T *__restrict__ wu, const T *__restrict__ extra, int64_t n, int C, T *__restrict__ up,
                   T *__restrict__ q0) {
  grid_begin();
  extern __shared__ __align__(32) unsigned char mid_smem[];
  T *sW = reinterpret_cast<T *>(mid_smem), *rows = sW + C * C;
  constexpr int PER = NODES / 8;
  const int tid = threadIdx.x, nt = 2 * C, tx = tid % (C / 4), ty = tid / (C / 4);
  mid_fill(sW, wu, C, tid, nt);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int64_t first = (int64_t)blockIdx.x * NODES; first < n; first += (int64_t)gridDim.x * NODES) {
    const int nn = n - first < NODES ? (int)(n - first) : NODES;
    __syncthreads();
    for (int i = tid; i < NODES * C; i += nt) rows[i] = i < nn * C ? b[first * C + i] : T(0);
    __syncthreads();
    T acc[PER][4];
    mid_product<T, PER>(rows, sW, C, ty * PER, tx, acc);
#pragma unroll
    for (int i = 0; i < PER; i++)
      if (ty * PER + i < nn)
        *reinterpret_cast<Quad<T> *>(up + (int64_t)node_of[first + ty * PER + i] * C + 4 * tx) =
            Quad<T>{acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
    for (int i = tid; i < nn * MID_EXTRA; i += nt) {
      const int j = i / MID_EXTRA, col = i - j * MID_EXTRA;
      const Quad<T> *w = reinterpret_cast<const Quad<T> *>(extra) + (int64_t)slot_type[first + j] * (C / 4) * MID_EXTRA + col;
      T a = T(0), a2 = T(0);
#pragma unroll 8
      for (int k = 0; k < C / 4; k++) {
        const Quad<T> x = w[k * MID_EXTRA], r = *reinterpret_cast<const Quad<T> *>(rows + j * C + 4 * k);
        a = fma(r.x, x.x, a);
        a2 = fma(r.y, x.y, a2);
        a = fma(r.z, x.z, a);
        a2 = fma(r.w, x.w, a2);
      }
      q0[(int64_t)node_of[first + j] * MID_EXTRA + col] = a + a2;
    }
  }
}

// grad b0 [slot order] = grad up Wu^T + (dq, scale) [17] extra_t[z] [17, C]
template <typename T, int NODES>
__global__ void __launch_bounds__(256)
    mid_bwd_kernel(const T *__restrict__ gup, const int32_t *__restrict__ node_of, const int32_t *__restrict__ slot_type,
                   const T *__restrict__ dq, const T *__restrict__ wu_t, const T *__restrict__ extra_t, T scale,
                   int64_t n, int C, T *__restrict__ gb) {
  grid_begin();
  extern __shared__ __align__(32) unsigned char mid_smem[];
  T *sW = reinterpret_cast<T *>(mid_smem), *rows = sW + C * C, *sdq = rows + NODES * C;
  constexpr int PER = NODES / 8;
  const int tid = threadIdx.x, nt = 2 * C, tx = tid % (C / 4), ty = tid / (C / 4);
  mid_fill(sW, wu_t, C, tid, nt);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int64_t first = (int64_t)blockIdx.x * NODES; first < n; first += (int64_t)gridDim.x * NODES) {
    const int nn = n - first < NODES ? (int)(n - first) : NODES;
    __syncthreads();
    for (int i = tid; i < NODES * C; i += nt) {
      const int j = i / C;
      rows[i] = j < nn ? gup[(int64_t)node_of[first + j] * C + (i - j * C)] : T(0);
    }
    for (int i = tid; i < nn * ST_RO; i += nt) sdq[i] = dq[(int64_t)node_of[first + i / ST_RO] * ST_RO + i % ST_RO];
    __syncthreads();
    T acc[PER][4];
    mid_product<T, PER>(rows, sW, C, ty * PER, tx, acc);
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int j = ty * PER + i;
      if (j < nn) {
        const Quad<T> *w = reinterpret_cast<const Quad<T> *>(extra_t + (int64_t)slot_type[first + j] * MID_EXTRA * C) + tx;
#pragma unroll
        for (int k = 0; k < MID_EXTRA; k++) {
          const Quad<T> x = w[k * (C / 4)];
          const T d = k < ST_RO ? sdq[j * ST_RO + k] : scale;
          acc[i][0] = fma(d, x.x, acc[i][0]);
          acc[i][1] = fma(d, x.y, acc[i][1]);
          acc[i][2] = fma(d, x.z, acc[i][2]);
          acc[i][3] = fma(d, x.w, acc[i][3]);
        }
        *reinterpret_cast<Quad<T> *>(gb + (first + j) * C + 4 * tx) = Quad<T>{acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
      }
    }
  }
}

// 8 nodes a tile while that leaves SMs idle, else 32 (four times the reuse of a weight); two blocks an SM in float32
template <typename T, typename Kernel8, typename Kernel32, typename... Args>
static int launch_mid(const char *what, int64_t n, int C, Kernel8 k8, Kernel32 k32, cudaStream_t st, Args... args) {
  if (n == 0) return CMACE_OK;
  const bool small = n < 32 * 148;
  const int nodes = small ? 8 : 32;
  const size_t smem = sizeof(T) * ((size_t)C * C + (size_t)nodes * (C + ST_RO));
  int64_t blocks = (n + nodes - 1) / nodes;
  const int64_t cap = 148 * (sizeof(T) == 4 ? 2 : 1);
  if (blocks > cap) blocks = cap;
  cudaError_t e = small ? cudaFuncSetAttribute(k8, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                        : cudaFuncSetAttribute(k32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  if (small) launch_chained(k8, (unsigned)blocks, 2 * C, smem, st, args...);
  else launch_chained(k32, (unsigned)blocks, 2 * C, smem, st, args...);
  return check_launch(what);
}
template <typename T>
int StepKernels<T>::mid_fwd(const T *b, const int32_t *node_of, const int32_t *slot_type, const T *wu, const T *extra,
                            int64_t n, int C, T *up, T *q0, cudaStream_t st) {
  return launch_mid<T>("cmace_step(mid_fwd)", n, C, mid_fwd_kernel<T, 8>, mid_fwd_kernel<T, 32>, st, b, node_of, slot_type,
                       wu, extra, n, C, up, q0);
}
template <typename T>
int StepKernels<T>::mid_bwd(const T *gup, const int32_t *node_of, const int32_t *slot_type, const T *dq, const T *wu_t,
                            const T *extra_t, double scale, int64_t n, int C, T *gb, cudaStream_t st) {
  return launch_mid<T>("cmace_step(mid_bwd)", n, C, mid_bwd_kernel<T, 8>, mid_bwd_kernel<T, 32>, st, gup, node_of, slot_type,
                       dq, wu_t, extra_t, (T)scale, n, C, gb);
}

#define CMACE_STEP_NODES(T)                                                                                          \
  template int StepKernels<T>::contract_fwd(const T *, const int32_t *, const T *, int64_t, int, T *, cudaStream_t); \
  template int StepKernels<T>::contract_bwd(const T *, const int32_t *, const T *, const T *, int64_t, int, T *,     \
                                            cudaStream_t);                                                           \
  template int StepKernels<T>::contract_readout(const T *, const int32_t *, const T *, const T *, const double *,    \
                                                const T *, const double *, double, double, int64_t, int, T *, T *,   \
                                                double *, double *, cudaStream_t);                                   \
  template int StepKernels<T>::mid_fwd(const T *, const int32_t *, const int32_t *, const T *, const T *, int64_t,   \
                                       int, T *, T *, cudaStream_t);                                                 \
  template int StepKernels<T>::mid_bwd(const T *, const int32_t *, const int32_t *, const T *, const T *, const T *, \
                                       double, int64_t, int, T *, cudaStream_t);
CMACE_STEP_NODES(float)
CMACE_STEP_NODES(double)

}  // namespace cmace

using namespace cmace;

extern "C" {
int cmace_symcon_apply(int is_f64, const void *X, const int32_t *atom_types, const void *weff, const void *gout,
                       int64_t nnodes, int channels, void *out, cmace_stream_t stream) {
  if (nnodes < 0) return fail(CMACE_ERR_ARG, "cmace_symcon_apply: bad size");
  if (channels <= 0 || channels % 32 != 0)
    return fail(CMACE_ERR_UNSUPPORTED, "cmace_symcon_apply: channels must be a multiple of 32");
  if (nnodes == 0) return CMACE_OK;
  if (!X || !atom_types || !weff || !out) return fail(CMACE_ERR_ARG, "cmace_symcon_apply: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (is_f64) {
    const double *x = static_cast<const double *>(X), *w = static_cast<const double *>(weff);
    double *o = static_cast<double *>(out);
    return gout ? StepKernels<double>::contract_bwd(x, atom_types, w, static_cast<const double *>(gout), nnodes, channels, o, st)
                : StepKernels<double>::contract_fwd(x, atom_types, w, nnodes, channels, o, st);
  }
  const float *x = static_cast<const float *>(X), *w = static_cast<const float *>(weff);
  float *o = static_cast<float *>(out);
  return gout ? StepKernels<float>::contract_bwd(x, atom_types, w, static_cast<const float *>(gout), nnodes, channels, o, st)
              : StepKernels<float>::contract_fwd(x, atom_types, w, nnodes, channels, o, st);
}
}
