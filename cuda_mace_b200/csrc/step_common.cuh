// Shapes and array layouts shared by the kernels of the whole energy+force step (step.cu holds the sequence).
#pragma once
#include <type_traits>

#include "common.cuh"

namespace cmace {

constexpr int ST_H = 64;          // hidden width of the radial perceptron
constexpr int ST_RO = 16;         // hidden width of the second layer's readout
constexpr int ST_MAX_Z = 16;      // elements the step's kernels are laid out for
constexpr int ST_NW = 13;         // effective contraction weights per (element, channel): 8 cubic, 4 quadratic, 1 linear

template <typename T>
struct alignas(4 * sizeof(T)) Quad {
  T x, y, z, w;
};

// Gradients of the first layer's sums leave the element-dependent product in blocks of at most two elements:
// block b is a [nodes, 16, width(b)] array, width = 64 times the elements it holds.
__host__ __device__ inline int sums_block_width(int elements, int b) { return elements - 2 * b >= 2 ? 128 : 64; }

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Powers of two of the fp16 radial kernel.  in_v, in_t: factors of the basis and its derivative; per layer k: z scales
// the accumulator to the pre-activation, a to the scaled activation (before the sigmoid factor), t to the scaled
// derivative.  Activations of layer 3 leave with out_v = 1 / h and out_t = 1 / h' of the stored value.
struct RadialScales {
  float in_v, in_t, z[3], a[3], t[3], out_v, out_t;
};

// tabulated radial weights: coefficients [intervals, 4 powers, 4 C], knots of width apart, zero beyond r_max
template <typename T>
struct SplineTable {
  const T *coeffs, *knots;
  T width, r_max;
  int intervals;
};
// where in the table an edge's length lies: distance from the interval's knot; interval -1 beyond r_max
template <typename T>
struct alignas(2 * sizeof(T)) SplinePoint {
  T x;
  typename std::conditional<sizeof(T) == 8, int64_t, int32_t>::type interval;
};
// spline_messages.cu; gY [spline_chunks, E, 16] and dr [spline_chunks, E] are shares to be added up
template <typename T>
int spline_chunks(int C);
template <typename T>
int spline_messages(const T *X, const int32_t *row_of, const T *Y, const SplinePoint<T> *r, const SplineTable<T> &table,
                    const int32_t *sender, const int32_t *row_ptr, int64_t n, const int32_t *out_row, int C, T *out,
                    cudaStream_t st);
template <typename T>
int spline_edges_back(const T *X, const int32_t *row_of, const T *Y, const SplinePoint<T> *r, const SplineTable<T> &table, const T *G,
                      const int32_t *g_row, const int32_t *sender, const int32_t *row_ptr, int64_t n, int64_t E, int C,
                      T *Tout, T *gY, T *dr, cudaStream_t st);

// Rows of the perceptrons' h and h' shared by edges of one length (step_edges.cu): count of them on the device, the edge that
// row k belongs to, an edge's row; all null: an edge has a row of its own.  Radial kernels go through the rows and look up
// what find_pairs left open.
struct EdgeRows {
  int32_t *row_of, *leaders, *count;
};
#ifdef __CUDACC__
__device__ __forceinline__ int64_t count_rows(const EdgeRows &rows, int64_t nedges) { return rows.count ? (int64_t)*rows.count : nedges; }
// the row of the other edge of a pair, in place of its leader; a share of the edges a thread
__device__ __forceinline__ void resolve_rows(const EdgeRows &rows, int64_t nedges, int64_t thread, int64_t nthreads) {
  if (!rows.count) return;
  for (int64_t e = thread; e < nedges; e += nthreads) {
    const int32_t r = rows.row_of[e];
    if (r < 0) rows.row_of[e] = rows.row_of[~r];   // a leader's row, which nobody writes here
  }
}
#endif

// radial_out64.cu: R = h W, dR = dh W, float64, for the rows of EdgeRows; W [64, N]
int radial_out_f64(const double *h, const double *dh, const double *W, const EdgeRows &rows, int64_t nedges, int N, double *R,
                   double *dR, cudaStream_t st);
// message_passing.cu: the edge pass with dE/dr from R' in component 0 of gY [chunks, E, 16]; R, dR rows by row_of (or null)
int imp_bwd_edge_pair_f64(const double *X, const double *Y, const double *R, const double *dR, const int32_t *row_of,
                          const double *G, const int32_t *sender, const int32_t *row_ptr, int64_t nnodes, int64_t nedges, int C,
                          double *gY, double *T, cudaStream_t st);
int imp_fwd_rows_f64(const double *X, const double *Y, const double *R, const int32_t *row_of, const int32_t *sender,
                     const int32_t *row_ptr, int64_t nnodes, int64_t nedges, int C, double *out, cudaStream_t st);

// status words of inputs that only a kernel sees; what such an input enters comes out as NaN
constexpr int32_t CMACE_STEP_BAD_SHIFT = 90;     // a row of the shift table that does not exist
constexpr int32_t CMACE_STEP_BAD_ELEMENT = 91;   // an element index outside 0 .. elements - 1

int *staged_stall_flag();   // message_passing.cu: device word of the staged edge pass, or null

constexpr int GN_NODES = 2048;   // nodes a block of edge_prep resolves; several such blocks take a second launch
constexpr int64_t node_blocks(int64_t n_local) { return (n_local + GN_NODES - 1) / GN_NODES; }

// launchers (one per kernel; every one checks its launch)
template <typename T>
struct StepKernels {
  static int edge_prep(const double *pos, const int32_t *sender, const int32_t *receiver, const double *shifts,
                       const uint8_t *shift_index, const double *shift_table, int64_t shift_rows, int32_t *status,
                       int64_t nedges, double r_max, int nb, int p, const SplineTable<T> &spline, Quad<T> *geo, T *basis,
                       T *Y,
                       const int32_t *species_in, const void *one_hot, int one_hot_f64, int64_t n_local, int64_t n_owned,
                       int elements, int32_t *species, int32_t *counts, int32_t *slot_of, int32_t *node_of,
                       int32_t *slot_type, int32_t *elem_start, const int32_t *row_ptr, const EdgeRows &rows, cudaStream_t st);
  static int sums(const T *h, const T *Y, const int32_t *sender, const int32_t *row_ptr, const int32_t *species,
                  const int32_t *slot_of, const int32_t *row_of, int64_t nnodes, int elements, T *A, cudaStream_t st);
  static int contract_fwd(const T *X, const int32_t *types, const T *weff, int64_t n, int C, bool early, T *b, cudaStream_t st);
  static int contract_bwd(const T *X, const int32_t *types, const T *weff, const T *gb, int64_t n, int C, bool early, T *gX,
                          cudaStream_t st);
  static int contract_readout(const T *X, const int32_t *types, const T *weff, const T *wp1, const double *w2,
                              const T *q0, const double *atomic_e, double scale, double shift, int64_t n, int C, T *gX,
                              T *dq, double *inter, double *node_energy, cudaStream_t st);
  static int mid_fwd(const T *b, const int32_t *node_of, const int32_t *slot_type, const T *wu, const T *extra,
                     int64_t n, int C, T *up, T *q0, cudaStream_t st);
  static int mid_bwd(const T *gup, const int32_t *node_of, const int32_t *slot_type, const T *dq, const T *wu_t,
                     const T *extra_t, double scale, int64_t n, int C, T *gb, cudaStream_t st);
  static int sums_bwd(const T *gA, const T *h, const T *dh, const T *Y, const int32_t *sender, const int32_t *row_ptr,
                      const int32_t *species, const int32_t *slot_of, const int32_t *row_of, const T *gY1, int shares, const T *dr1,
                      const Quad<T> *geo, int64_t nnodes, int64_t nedges, int elements, T *gvec, cudaStream_t st);
  static int forces(const T *gvec, const int32_t *row_ptr, const int32_t *perm, const int32_t *send_ptr, int64_t nrecv,
                    int64_t nsend, double sign, double *out, const int32_t *species_in, int elements, double *inter,
                    double *node_energy, const int32_t *status, const int *stalled, double *sums, cudaStream_t st);
};

}  // namespace cmace
