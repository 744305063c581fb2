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

// Before grid_wait(): the weights of a block's node to L1, a row of the warp's channels a lane.  Where a block has more than one
// node it costs more than it gives (66 -> 72 us at 16 000 nodes).
template <typename T>
__device__ __forceinline__ void prefetch_weff(const T *__restrict__ weff, int z, int C, int c) {
  const int lane = threadIdx.x & 31;
  if (lane < ST_NW) asm volatile("prefetch.global.L1 [%0];" ::"l"(weff + ((int64_t)z * ST_NW + lane) * C + (c & ~31)));
}

// A block's next node on its way to L1, the lines of the warp's channels: the loads at the head of a node stall every warp of a block that
// has little else resident.  us at 64 000 and 16 000 atoms of 128 channels: contract0 137 -> 130 and 37 -> 35, contract1 357 -> 349 and
// 87 -> 84, contract0_back 261 -> 229 and 64 -> 58.  (The next node's element kept in a register as well: 146, 349, 251.)
template <typename T>
__device__ __forceinline__ void prefetch_node(const T *__restrict__ X, int64_t node, int64_t nnodes, int C, int c) {
  constexpr int LINES = (int)sizeof(T) / 4;   // of 128 bytes, of a row of 32 channels
  const int lane = threadIdx.x & 31;
  if (node < nnodes && lane < 16 * LINES)
    asm volatile("prefetch.global.L1 [%0];" ::"l"(X + (node * 16 + lane / LINES) * C + (c & ~31) + lane % LINES * 16));
}

// The value alone needs a third of the gradient's work (canon::value) and half its registers: forward 95 -> 58 us at 32 000 nodes of
// 128 channels (278 MB: 43 us), 52 -> 35 at 16 000 in a step, 45 -> 29 in float64 at 8 000.  The backward is bound by its
// arithmetic (about 500 instructions a node and channel: 114 us of its 229 at 64 000 nodes by issue alone).
//
// early: whether types and weights are older than the kernel before (not where that kernel has laid the weights out)
template <typename T, bool BWD>
__global__ void __launch_bounds__(128, BWD ? (sizeof(T) == 4 ? 5 : 3) : (sizeof(T) == 4 ? 10 : 6))
    step_contract_kernel(const T *__restrict__ X, const int32_t *__restrict__ types, const T *__restrict__ weff,
                         const T *__restrict__ gb, int64_t nnodes, int C, bool early, T *__restrict__ out) {
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (early && nnodes <= gridDim.x) prefetch_weff(weff, __ldcg(types + blockIdx.x), C, c);
  grid_begin();
  for (int64_t node = blockIdx.x; node < nnodes; node += gridDim.x) {
    T x[16], w3[canon::NCLASS3], w2[canon::NCLASS2], w1;
    const T *xr = X + node * 16 * C + c;
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = __ldcs(xr + i * C);
    load_weff(weff, types[node], C, c, w3, w2, w1);
    prefetch_node(X, node + gridDim.x, nnodes, C, c);
    if constexpr (BWD) {
      T g[16], value;
      const T go = gb[node * C + c];
      canon::eval<T>(x, w3, w2, w1, g, value);
      T *o = out + node * 16 * C + c;
#pragma unroll
      for (int i = 0; i < 16; i++) __stcs(o + i * C, go * g[i]);
    } else {
      out[node * C + c] = canon::value<T>(x, w3, w2, w1);
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

// blocks of ch threads: per_sm an SM of 128 threads, more of fewer
static int64_t node_blocks(int64_t n, int per_sm, int ch) {
  const int64_t cap = (int64_t)148 * per_sm * (128 / ch);
  return n < cap ? n : cap;
}

template <typename T>
int StepKernels<T>::contract_fwd(const T *X, const int32_t *types, const T *weff, int64_t n, int C, bool early, T *b,
                                 cudaStream_t st) {
  const int ch = channel_block(C);
  if (n > 0)
    launch_chained(step_contract_kernel<T, false>, dim3((unsigned)node_blocks(n, 16, ch), C / ch), ch, 0, st, X, types, weff, nullptr, n,
                   C, early, b);
  return check_launch("cmace_step(contract_fwd)");
}
template <typename T>
int StepKernels<T>::contract_bwd(const T *X, const int32_t *types, const T *weff, const T *gb, int64_t n, int C, bool early, T *gX,
                                 cudaStream_t st) {
  const int ch = channel_block(C);
  if (n > 0)
    launch_chained(step_contract_kernel<T, true>, dim3((unsigned)node_blocks(n, 12, ch), C / ch), ch, 0, st, X, types, weff, gb, n, C,
                   early, gX);
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
  __shared__ T part[4][ST_RO];
  __shared__ T dq_s[ST_RO];
  const int c = threadIdx.x, lane = c & 31, w = c >> 5, nw = C >> 5;
  T wp[ST_RO];
#pragma unroll
  for (int j = 0; j < ST_RO; j++) wp[j] = __ldg(wp1 + j * C + c);
  if (nnodes <= gridDim.x) prefetch_weff(weff, __ldcg(types + blockIdx.x), C, c);
  grid_begin();
  for (int64_t node = blockIdx.x; node < nnodes; node += gridDim.x) {
    T x[16], g[16], w3[canon::NCLASS3], w2[canon::NCLASS2], w1, value;
    const T *xr = X + node * 16 * C + c;
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = __ldcs(xr + i * C);
    const int z = types[node];
    load_weff(weff, z, C, c, w3, w2, w1);
    prefetch_node(X, node + gridDim.x, nnodes, C, c);
    double qd = 0.0, e0 = 0.0;
    if (c < ST_RO) qd = (double)q0[node * (ST_RO + 1) + c];
    if (c == 0) e0 = (double)q0[node * (ST_RO + 1) + ST_RO];
    canon::eval<T>(x, w3, w2, w1, g, value);
    T p[ST_RO];
#pragma unroll
    for (int j = 0; j < ST_RO; j++) p[j] = value * wp[j];
    const T r = warp_reduce16(p, lane);
    if ((lane & 1) == 0) part[w][lane >> 1] = r;
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
    launch_chained(contract_readout_kernel<T>, (unsigned)node_blocks(n, 10, C), C, 0, st, X, types, weff, wp1, w2, q0, atomic_e, scale,
                                                                          shift, n, C, gX, dq, inter, node_energy);
  return check_launch("cmace_step(contract_readout)");
}

// ---- between the layers --------------------------------------------------------------------------------------------
// Products with a [C, C] matrix that stays in shared memory (64 KB float32, 128 KB float64: one fill per block, blocks
// are persistent), plus 17 columns (padded to 20) that depend on the element: 16 of the second readout's hidden layer and
// the first readout.  Nodes are taken in slot order, so the nodes of a tile nearly always share the element, whose part
// of the matrix is kept beside the other (a tile where the element changes takes one after the other).  The
// next tile's rows are copied while a tile is worked on.  2 C threads: a thread owns 4 columns of NODES / 8 nodes; what
// bounds it then is the shared-memory pipe (four 16-byte loads of weights and NODES / 8 of rows per 4 k).  With rows
// loaded at the head of a tile and the element's columns read from memory, forward and backward took 150 + 170 us at
// 64 000 nodes, 22 + 20 us at 3 000; now 92 + 79 and 14 + 12.
constexpr int MID_EXTRA = ST_RO + 1, MID_PAD = 20;

__device__ __forceinline__ void copy16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// count values, a multiple of 16 bytes
template <typename T>
__device__ __forceinline__ void mid_fill(T *dst, const T *__restrict__ src, int count, int tid, int nthreads) {
  constexpr int V = 16 / (int)sizeof(T);
  for (int i = tid; i < count / V; i += nthreads) copy16(dst + i * V, src + (int64_t)i * V);
}

// acc[i][u] += sum_k rows[j0 + i STRIDE][k] W[k][4 tx + u], k < K (a multiple of 4)
template <typename T, int PER, int STRIDE = 1>
__device__ __forceinline__ void mid_product(const T *rows, int ld, const T *W, int ldw, int K, int j0, int tx, T (&acc)[PER][4]) {
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    Quad<T> r[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) r[i] = *reinterpret_cast<const Quad<T> *>(rows + (j0 + i * STRIDE) * ld + k);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const Quad<T> w = *reinterpret_cast<const Quad<T> *>(W + (k + u) * ldw + 4 * tx);
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
template <typename T, int PER>
__device__ __forceinline__ void mid_zero(T (&acc)[PER][4]) {
#pragma unroll
  for (int i = 0; i < PER; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = T(0);
}

// The elements of a tile in turn: body(z) with z's part of the matrix in sE.  type: of the tile's node `lane`, -1 past the
// end; held: the element whose part is there.  Called by all threads of the block.
template <typename T, typename Body>
__device__ __forceinline__ void for_elements_of_tile(int type, int nn, T *sE, const T *__restrict__ extra, int count, int tid,
                                                     int nthreads, int &held, Body body) {
  int z = __shfl_sync(0xffffffffu, type, 0);
  const int last = __shfl_sync(0xffffffffu, type, nn - 1);
  while (true) {
    if (z != held) {
      __syncthreads();   // the part that is there has been read
      mid_fill(sE, extra + (int64_t)z * count, count, tid, nthreads);
      copies_commit();
      copies_wait();
      __syncthreads();
      held = z;
    }
    body(z);
    if (z == last) break;
    const unsigned later = __ballot_sync(0xffffffffu, type > z);   // sorted: the next element's first node
    z = __shfl_sync(0xffffffffu, type, __ffs(later) - 1);
  }
}

// extra: [Z][C][20].  The block's last 64 threads own the extra columns: 5 groups of 4 times 8 groups of nodes,
// every eighth node each; rows are 4 values longer than C, so that the 8 nodes lie in different banks.
template <typename T, int NODES>
__global__ void __launch_bounds__(320)
    mid_fwd_kernel(const T *__restrict__ b, const int32_t *__restrict__ node_of, const int32_t *__restrict__ slot_type,
                   const T *__restrict__ wu, const T *__restrict__ extra, int64_t n, int C, T *__restrict__ up,
                   T *__restrict__ q0) {
  extern __shared__ __align__(32) unsigned char mid_smem[];
  T *sW = reinterpret_cast<T *>(mid_smem), *sE = sW + C * C, *buf = sE + C * MID_PAD;
  constexpr int PER = NODES / 8, V = 16 / (int)sizeof(T);
  const int tid = threadIdx.x, nt = 2 * C, x = tid - nt;
  const int ld = C + 4;
  const int tx = x < 0 ? tid % (C / 4) : x % (MID_PAD / 4), ty = x < 0 ? tid / (C / 4) : x / (MID_PAD / 4);
  mid_fill(sW, wu, C * C, tid, nt + 64);
  grid_begin();
  auto fetch = [&](int64_t first, T *rows) {   // rows past the end: the last one
    for (int i = tid; i < NODES * C / V; i += nt + 64) {
      const int j = i / (C / V), c = (i - j * (C / V)) * V;
      const int64_t s = first + j < n ? first + j : n - 1;
      copy16(rows + j * ld + c, b + s * C + c);
    }
  };
  int64_t first = (int64_t)blockIdx.x * NODES;
  fetch(first, buf);
  int held = first < n ? slot_type[first] : -1;
  if (held >= 0) mid_fill(sE, extra + (int64_t)held * C * MID_PAD, C * MID_PAD, tid, nt + 64);
  copies_commit();
  for (int turn = 0; first < n; first += (int64_t)gridDim.x * NODES, turn ^= 1) {
    T *rows = buf + turn * NODES * ld;
    const int nn = n - first < NODES ? (int)(n - first) : NODES;
    const int type = (tid & 31) < nn ? slot_type[first + (tid & 31)] : -1;
    int32_t node[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int j = x < 0 ? ty * PER + i : ty + 8 * i;
      node[i] = ty < 8 && j < nn ? node_of[first + j] : 0;
    }
    copies_wait();
    __syncthreads();
    if (first + (int64_t)gridDim.x * NODES < n) {
      fetch(first + (int64_t)gridDim.x * NODES, buf + (turn ^ 1) * NODES * ld);
      copies_commit();
    }
    T acc[PER][4];
    for_elements_of_tile<T>(type, nn, sE, extra, C * MID_PAD, tid, nt + 64, held, [&](int z) {
      if (x < 0 || ty >= 8) return;
      mid_zero<T, PER>(acc);
      mid_product<T, PER, 8>(rows, ld, sE, MID_PAD, C, ty, tx, acc);
#pragma unroll
      for (int i = 0; i < PER; i++)
        if (ty + 8 * i < nn && slot_type[first + ty + 8 * i] == z)
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (4 * tx + u < MID_EXTRA) q0[(int64_t)node[i] * MID_EXTRA + 4 * tx + u] = acc[i][u];
    });
    if (x >= 0) continue;
    mid_zero<T, PER>(acc);
    mid_product<T, PER>(rows, ld, sW, C, C, ty * PER, tx, acc);
#pragma unroll
    for (int i = 0; i < PER; i++)
      if (ty * PER + i < nn)
        *reinterpret_cast<Quad<T> *>(up + (int64_t)node[i] * C + 4 * tx) = Quad<T>{acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
  }
}

// grad b0 [slot order] = grad up Wu^T + (dq, scale, 0) [20] extra_t[z] [20, C]
template <typename T, int NODES>
__global__ void __launch_bounds__(256)
    mid_bwd_kernel(const T *__restrict__ gup, const int32_t *__restrict__ node_of, const int32_t *__restrict__ slot_type,
                   const T *__restrict__ dq, const T *__restrict__ wu_t, const T *__restrict__ extra_t, T scale,
                   int64_t n, int C, T *__restrict__ gb) {
  extern __shared__ __align__(32) unsigned char mid_smem[];
  T *sW = reinterpret_cast<T *>(mid_smem), *sE = sW + C * C, *buf = sE + C * MID_PAD;
  constexpr int PER = NODES / 8, V = 16 / (int)sizeof(T);
  T *const sdq = buf + 2 * NODES * C;
  const int tid = threadIdx.x, nt = 2 * C, tx = tid % (C / 4), ty = tid / (C / 4);
  mid_fill(sW, wu_t, C * C, tid, nt);
  for (int i = tid; i < 2 * NODES; i += nt)
#pragma unroll
    for (int u = ST_RO; u < MID_PAD; u++) sdq[i * MID_PAD + u] = u == ST_RO ? scale : T(0);
  grid_begin();
  // a thread copies NODES sizeof(T) / 32 pieces of rows; the atoms they belong to are looked up a tile ahead
  constexpr int PIECES = NODES * (int)sizeof(T) / 32;
  constexpr int DQ = NODES * ST_RO / V, DQ_MOST = (DQ + 63) / 64;   // pieces of dq; at most so many a thread (C = 32)
  int32_t at[PIECES], at_dq[DQ_MOST];
  auto look_up = [&](int64_t first) {
#pragma unroll
    for (int p = 0; p < PIECES; p++) {
      const int64_t s = first + (tid + p * nt) / (C / V);
      at[p] = node_of[s < n ? s : n - 1];
    }
#pragma unroll
    for (int p = 0; p < DQ_MOST; p++) {
      const int64_t s = first + (tid + p * nt) / (ST_RO / V);
      at_dq[p] = node_of[s < n ? s : n - 1];
    }
  };
  auto fetch = [&](int turn) {
#pragma unroll
    for (int p = 0; p < PIECES; p++) {
      const int i = tid + p * nt, j = i / (C / V), c = (i - j * (C / V)) * V;
      copy16(buf + (turn * NODES + j) * C + c, gup + (int64_t)at[p] * C + c);
    }
#pragma unroll
    for (int p = 0; p < DQ_MOST; p++) {
      const int i = tid + p * nt, j = i / (ST_RO / V), c = (i - j * (ST_RO / V)) * V;
      if (i < DQ) copy16(sdq + (turn * NODES + j) * MID_PAD + c, dq + (int64_t)at_dq[p] * ST_RO + c);
    }
    copies_commit();
  };
  const int64_t step = (int64_t)gridDim.x * NODES;
  int64_t first = (int64_t)blockIdx.x * NODES;
  look_up(first);
  int held = first < n ? slot_type[first] : -1;
  if (held >= 0) mid_fill(sE, extra_t + (int64_t)held * C * MID_PAD, C * MID_PAD, tid, nt);
  fetch(0);
  if (first + step < n) look_up(first + step);
  for (int turn = 0; first < n; first += step, turn ^= 1) {
    const T *rows = buf + turn * NODES * C, *sd = sdq + turn * NODES * MID_PAD;
    const int nn = n - first < NODES ? (int)(n - first) : NODES;
    const int type = (tid & 31) < nn ? slot_type[first + (tid & 31)] : -1;
    copies_wait();
    __syncthreads();
    if (first + step < n) {
      fetch(turn ^ 1);
      if (first + 2 * step < n) look_up(first + 2 * step);
    }
    T acc[PER][4];
    mid_zero<T, PER>(acc);
    mid_product<T, PER>(rows, C, sW, C, C, ty * PER, tx, acc);
    for_elements_of_tile<T>(type, nn, sE, extra_t, C * MID_PAD, tid, nt, held, [&](int z) {
      T more[PER][4];
      mid_zero<T, PER>(more);
      mid_product<T, PER>(sd, MID_PAD, sE, C, MID_PAD, ty * PER, tx, more);
#pragma unroll
      for (int i = 0; i < PER; i++)
        if (ty * PER + i < nn && slot_type[first + ty * PER + i] == z)
#pragma unroll
          for (int u = 0; u < 4; u++) acc[i][u] += more[i][u];
    });
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int j = ty * PER + i;
      if (j < nn)
        *reinterpret_cast<Quad<T> *>(gb + (first + j) * C + 4 * tx) = Quad<T>{acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
    }
  }
}

// 8 nodes a tile while that leaves SMs idle, 16 while every block has one tile, else 32 (four times the reuse of a weight); two blocks
// an SM in float32.  16 against 32, us forward and back, 128 channels: 1 500 nodes 14.6 + 12.7 against 16.8 + 14.8 (float64 25.6 + 23.0
// against 29.1 + 25.0), 3 000 16.4 + 14.8 against 16.9 + 14.8 (float64, two tiles a block, 33.2 + 31.2 against 29.1 + 25.0), 6 000
// 21.0 + 18.9 against 18.9 + 17.9; 32 channels, 3 000: 9.2 + 8.7 against 10.6 + 10.6.
template <typename T, typename Kernel, typename... Args>
static int launch_mid(const char *what, int64_t n, int C, int threads, Kernel k8, Kernel k16, Kernel k32, cudaStream_t st, Args... args) {
  if (n == 0) return CMACE_OK;
  const int64_t cap = 148 * (sizeof(T) == 4 ? 2 : 1);
  const int nodes = n <= 8 * 148 ? 8 : (n <= 16 * cap ? 16 : 32);
  const Kernel kernel = nodes == 8 ? k8 : (nodes == 16 ? k16 : k32);
  const size_t smem = sizeof(T) * ((size_t)C * (C + MID_PAD) + 2 * (size_t)nodes * (C + MID_PAD));   // forward: C + 4 a row
  int64_t blocks = (n + nodes - 1) / nodes;
  if (blocks > cap) blocks = cap;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  launch_chained(kernel, (unsigned)blocks, threads, smem, st, args...);
  return check_launch(what);
}
template <typename T>
int StepKernels<T>::mid_fwd(const T *b, const int32_t *node_of, const int32_t *slot_type, const T *wu, const T *extra,
                            int64_t n, int C, T *up, T *q0, cudaStream_t st) {
  return launch_mid<T>("cmace_step(mid_fwd)", n, C, 2 * C + 64, mid_fwd_kernel<T, 8>, mid_fwd_kernel<T, 16>, mid_fwd_kernel<T, 32>, st,
                       b, node_of, slot_type, wu, extra, n, C, up, q0);
}
template <typename T>
int StepKernels<T>::mid_bwd(const T *gup, const int32_t *node_of, const int32_t *slot_type, const T *dq, const T *wu_t,
                            const T *extra_t, double scale, int64_t n, int C, T *gb, cudaStream_t st) {
  return launch_mid<T>("cmace_step(mid_bwd)", n, C, 2 * C, mid_bwd_kernel<T, 8>, mid_bwd_kernel<T, 16>, mid_bwd_kernel<T, 32>, st, gup,
                       node_of, slot_type, dq, wu_t, extra_t, (T)scale, n, C, gb);
}

#define CMACE_STEP_NODES(T)                                                                                          \
  template int StepKernels<T>::contract_fwd(const T *, const int32_t *, const T *, int64_t, int, bool, T *,          \
                                            cudaStream_t);                                                           \
  template int StepKernels<T>::contract_bwd(const T *, const int32_t *, const T *, const T *, int64_t, int, bool,    \
                                            T *, cudaStream_t);                                                      \
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
  const ChainScope chained;
  if (is_f64) {
    const double *x = static_cast<const double *>(X), *w = static_cast<const double *>(weff);
    double *o = static_cast<double *>(out);
    return gout ? StepKernels<double>::contract_bwd(x, atom_types, w, static_cast<const double *>(gout), nnodes, channels, false, o, st)
                : StepKernels<double>::contract_fwd(x, atom_types, w, nnodes, channels, false, o, st);
  }
  const float *x = static_cast<const float *>(X), *w = static_cast<const float *>(weff);
  float *o = static_cast<float *>(out);
  return gout ? StepKernels<float>::contract_bwd(x, atom_types, w, static_cast<const float *>(gout), nnodes, channels, false, o, st)
              : StepKernels<float>::contract_fwd(x, atom_types, w, nnodes, channels, false, o, st);
}
}
