// The whole energy+force step of a two-layer invariant model as one sequence of launches (cmace_step_run).
//
//   edge_prep     unit vectors, Y [E, 16], basis and its derivative; nodes grouped by element beside it
//   radial        both perceptrons' hidden layers h and h' = dh/dr                        (radial_tangent.cu)
//   sums          first layer: A[i, lm, (z, k)] = sum_{e in (i, z)} Y h                   (step_edges.cu)
//   fold          A times the element-dependent matrices that hold everything up to the layer's Linear
//   contract0     b0
//   mid_fwd       up = b0 Wu, q0 = b0 Wsc[z] [n, 17]                                      (step_nodes.cu)
//       -- a decomposed system fills the ghost rows of `up` here --
//   radial_out    second layer: R = h W4 [E, 4C]  (not in float32 with fp16 pairs: `messages` and `edges_back` form R and
//                 R' = h' W4 themselves, fused_messages.cu, and `radial_back` is part of `edges_back`)
//   messages, linear, contract1 (value, readout, energy and gradient in one kernel), linear_back
//   edges_back    T [E, C] and grad Y of the second layer; radial_back: dE/dr of the second layer (float64: part of edges_back,
//                 from R' = h' W4 that radial_out forms beside R, a row a pair of edges)
//   senders       grad up = sum of T over a sender's edges
//       -- and returns the gradients of the ghost rows here --
//   mid_back, contract0_back, fold_back
//   sums_back     grad Y and dE/dr of the first layer, plus the second layer's: gradient of every edge vector
//   forces        position gradient and energies
//
// With tabulated radial weights (cubic splines) the first layer has no perceptron to sum against: `sums` is the
// message passing on the element's constant feature row, with the table evaluated there (spline_messages.cu), `fold` the
// layer's element-dependent Linear, and the backward mirrors that.
//
// Nodes of the first layer are kept in element order (slots) between `sums` and `mid_fwd` and on the way back, so the
// element-dependent products see consecutive rows whatever the caller's order is.
#include <cstring>

#include "step_common.cuh"

namespace cmace {

int radial_pair_f32(const float *basis, int nb, const float *const (*w)[3], int nper, int64_t nedges, float *const *h,
                    float *const *dh, int32_t *status, cudaStream_t st);
int radial_half(const float *basis, int nb, const void *const (*w)[3], const RadialScales *scales, const int *half_out,
                int nper, const EdgeRows &rows, int64_t nedges, void *const *h, void *const *dh, int32_t *status,
                cudaStream_t st);
int step_sums_half(const void *h, const float *Y, const int32_t *sender, const int32_t *row_ptr, const int32_t *species,
                   const int32_t *slot_of, const int32_t *row_of, int64_t nnodes, int elements, float out_v, float *A,
                   cudaStream_t st);
int step_sums_bwd_half(const float *gA, const void *h, const void *dh, const float *Y, const int32_t *sender,
                       const int32_t *row_ptr, const int32_t *species, const int32_t *slot_of, const int32_t *row_of,
                       const float *gY1, const float *dr1, const Quad<float> *geo, int64_t nnodes, int elements, float out_v,
                       float out_t, float *gvec, cudaStream_t st);
int fused_messages(const float *X, const float *Y, const void *h, const void *W, float factor, const int32_t *sender,
                   const int32_t *receiver, const int32_t *row_ptr, const int32_t *row_of, int64_t nnodes, int64_t nedges, int C,
                   float *out, int32_t *status, cudaStream_t st);
int fused_messages_back(const float *X, const float *Y, const float *G, const void *h, const void *dh, const void *W,
                        float factor_v, float factor_t, const int32_t *sender, const int32_t *receiver, const int32_t *row_of,
                        int64_t nedges, int C, float *T, float *gY, int32_t *status, cudaStream_t st);
template <typename T>
int step_edge_finish(const T *gY0, const T *dr0, const T *gY1, const T *dr1, const Quad<T> *geo, int64_t nedges, int shares, T *gvec,
                     cudaStream_t st);
int radial_pair_f64(const double *basis, int nb, const double *const (*w)[3], int nper, const EdgeRows &rows, int64_t nedges,
                    double *const *h, double *const *dh, cudaStream_t st);

enum StepId {
  S_EDGE_PREP, S_RADIAL, S_SUMS, S_FOLD, S_CONTRACT0, S_MID_FWD,
  S_RADIAL_OUT, S_MESSAGES, S_LINEAR, S_CONTRACT1, S_LINEAR_BACK, S_EDGES_BACK, S_RADIAL_BACK, S_SENDERS,
  S_MID_BACK, S_CONTRACT0_BACK, S_FOLD_BACK, S_SUMS_BACK, S_FORCES, S_COUNT
};
static const char *const kStepNames[S_COUNT] = {
    "edge_prep", "radial", "sums", "fold", "contract0", "mid_fwd",
    "radial_out", "messages", "linear", "contract1", "linear_back", "edges_back", "radial_back", "senders",
    "mid_back", "contract0_back", "fold_back", "sums_back", "forces"};

static bool is_spline(const cmace_step_model &m) { return m.spline[0] != nullptr; }
// second layer with the radial weights formed inside its kernels: fp16 pairs of h (fused_messages.cu)
static bool is_fused(const cmace_step_model &m) {
  return !is_spline(m) && !m.is_f64 && m.fused_w != nullptr &&
         m.fused_layout == (m.channels == 128 ? CMACE_FUSED_LAYOUT : CMACE_FUSED_LAYOUT_NARROW);
}

// Whether the edges of a pair share a row of h and h' (find_pairs): once the radial kernel needs more than one round of its warps
// (float64: eight edges each) or groups (float32: 128 edges) without it.  The search takes 8 us there, the second round 30 and 10:
// float32, 64 channels, 127 -> 125 us a step at 20 900 edges, 136 -> 132 at 26 200, 150 -> 145 at 36 700, 226 -> 211 at 73 000; at
// 15 500, in one round, 112 -> 121.
constexpr int64_t kPairEdges64 = 74 * 16 * 8, kPairEdges32 = 74 * 2 * 128;
static bool has_pairs(const cmace_step_model &m, int64_t edges) {
  return m.is_f64 ? !is_spline(m) && edges > kPairEdges64 : is_fused(m) && edges > kPairEdges32;
}

template <typename T>
struct Workspace {
  int32_t *species, *counts, *slot_of, *node_of, *slot_type, *elem_start;
  EdgeRows rows;
  Quad<T> *geo;
  T *basis, *Y, *h[2], *dh[2], *A, *m0, *b0, *up, *R, *m1, *l1, *gX1, *gm1, *T_, *gY1, *dr1, *gup, *gb0, *gX0, *gA,
      *gvec, *dR, *q0, *dq, *gY0, *dr0;
  int64_t bytes;
  int shares;   // of grad Y of the second layer, to be added up

  Workspace(void *base, const cmace_step_model &m, int64_t n, int64_t nl, int64_t E) {
    char *p = static_cast<char *>(base);
    bytes = 0;
    auto take = [&](auto *&ptr, int64_t count) {
      using U = typename std::remove_reference<decltype(*ptr)>::type;
      ptr = reinterpret_cast<U *>(p + bytes);
      bytes += (count * (int64_t)sizeof(U) + 255) / 256 * 256;
    };
    const int64_t C = m.channels, Z = m.elements;
    take(species, nl);
    take(counts, node_blocks(nl) * ST_MAX_Z);
    take(slot_of, n);
    take(node_of, n);
    take(slot_type, n);
    take(elem_start, Z + 1);
    take(geo, E);
    const bool sp = is_spline(m);
    take(basis, E * 2 * (sp ? 1 : m.nbessel));   // with tables: a SplinePoint an edge
    const bool f64 = sizeof(T) == 8, pairs = has_pairs(m, E);
    take(rows.row_of, pairs ? E : 0);
    take(rows.leaders, pairs ? E : 0);
    take(rows.count, pairs ? 1 : 0);
    if (!pairs) rows = EdgeRows{};
    shares = sp ? spline_chunks<T>((int)C) : (f64 && C == 128 ? 2 : 1);   // float64: imp_bwd_edge_pair_f64's channel chunks
    take(gY0, sp ? shares * E * 16 : 0);
    take(dr0, sp ? shares * E : 0);
    take(Y, E * 16);
    for (int i = 0; i < 2; i++) {
      take(h[i], sp ? 0 : (E + 127) / 128 * 128 * ST_H);   // whole tiles of the kernels that read them
      take(dh[i], sp ? 0 : (E + 127) / 128 * 128 * ST_H);
    }
    take(A, n * 16 * (sp ? C : ST_H * Z));
    take(m0, n * 16 * C);
    take(b0, n * C);
    take(up, n * C);
    take(q0, n * (ST_RO + 1));
    take(R, is_fused(m) || sp ? 0 : E * 4 * C);
    take(m1, n * 16 * C);
    take(l1, n * 16 * C);
    take(gX1, n * 16 * C);
    take(dq, n * ST_RO);
    take(T_, E * C);
    take(gY1, shares * E * 16);
    take(dr1, f64 && !sp ? 0 : shares * E);   // float64: in component 0 of gY1
    take(gup, nl * C);
    take(gb0, n * C);
    take(gX0, n * 16 * C);
    take(gvec, E * 4);
    take(dR, f64 && !sp ? E * 4 * C : 0);
    gm1 = m1;   // the messages are not read again after the Linear
    gA = A;     // nor the sums after their product
  }
};

int linear_tc(const float *X, const float *packed, const int32_t *node_order, const int32_t *elem_start, int nelements,
              int nblocks, int64_t nnodes, int K, int Nout, double scale, float *out, int32_t *status, cudaStream_t stream);

static int linear_any(const float *X, const void *W, const int32_t *start, int nel, int64_t n, int K, int N, float *out,
                      int32_t *status, cmace_stream_t st) {
  return cmace_linear_tc_f32(X, static_cast<const float *>(W), nullptr, start, nel, n, K, N, 1.0, out, status, st);
}
static int linear_any(const double *X, const void *W, const int32_t *start, int nel, int64_t n, int K, int N, double *out,
                      int32_t *, cmace_stream_t st) {
  return cmace_linear_f64(X, static_cast<const double *>(W), nullptr, start, nel, n, K, N, 1.0, out, st);
}

// the steps that tabulated radial weights do differently; -1 for the others
template <typename T>
static int run_spline_step(const cmace_step_model &m, cmace_step_io &io, const Workspace<T> &w, int step, const T *up,
                           cudaStream_t st) {
  const int64_t n = io.n_owned, E = io.nedges;
  const int C = m.channels, Z = m.elements;
  const int32_t *start = Z > 1 ? w.elem_start : nullptr;
  const T *senders = static_cast<const T *>(m.sender_table);
  auto table = [&](int layer) {
    return SplineTable<T>{static_cast<const T *>(m.spline[layer]), static_cast<const T *>(m.spline_knots), (T)m.spline_width,
                          (T)m.spline_rmax, m.spline_intervals};
  };
  const SplinePoint<T> *at = reinterpret_cast<const SplinePoint<T> *>(w.basis);
  switch (step) {
    case S_EDGE_PREP:
      return StepKernels<T>::edge_prep(io.positions, io.sender, io.receiver, io.shifts, io.shift_index, io.shift_table,
                                       io.shift_rows, io.status, E, m.r_max, 0, m.cutoff_p, table(0), w.geo,
                                       w.basis, w.Y, io.species, io.one_hot, io.one_hot_is_f64, io.n_local, n, Z, w.species,
                                       w.counts, w.slot_of, w.node_of, w.slot_type, w.elem_start, io.row_ptr, w.rows, st);
    case S_SUMS:
      return spline_messages<T>(senders, w.species, w.Y, at, table(0), io.sender, io.row_ptr, n, w.slot_of, C, w.A, st);
    case S_FOLD: return linear_any(w.A, m.fold, start, Z, n, C, C, w.m0, io.status, st);
    case S_RADIAL:
    case S_RADIAL_OUT:
    case S_RADIAL_BACK: io.launches--; return CMACE_OK;
    case S_MESSAGES:
      return spline_messages<T>(up, nullptr, w.Y, at, table(1), io.sender, io.row_ptr, n, nullptr, C, w.m1, st);
    case S_EDGES_BACK:
      return spline_edges_back<T>(up, nullptr, w.Y, at, table(1), w.gm1, nullptr, io.sender, io.row_ptr, n, E, C, w.T_,
                                  w.gY1, w.dr1, st);
    case S_FOLD_BACK: return linear_any(w.gX0, m.fold_back[0], start, Z, n, C, C, w.gA, io.status, st);
    case S_SUMS_BACK:
      io.launches++;
      if (int rc = spline_edges_back<T>(senders, w.species, w.Y, at, table(0), w.gA, w.slot_of, io.sender, io.row_ptr, n, E,
                                        C, nullptr, w.gY0, w.dr0, st))
        return rc;
      return step_edge_finish<T>(w.gY0, w.dr0, w.gY1, w.dr1, w.geo, E, spline_chunks<T>(C), w.gvec, st);
  }
  return -1;
}

template <typename T>
static int run_step(const cmace_step_model &m, cmace_step_io &io, const Workspace<T> &w, int step, cudaStream_t st) {
  using K = StepKernels<T>;
  const int64_t n = io.n_owned, nl = io.n_local, E = io.nedges;
  const int C = m.channels, Z = m.elements;
  const T *up = io.up_local ? static_cast<const T *>(io.up_local) : w.up;
  T *gup = io.gup_local ? static_cast<T *>(io.gup_local) : w.gup;
  const T *gup_owned = io.gup_owned ? static_cast<const T *>(io.gup_owned) : gup;
  const ImpLayout ys{1, 16};
  const int32_t *start = Z > 1 ? w.elem_start : nullptr;
  constexpr bool f64 = sizeof(T) == 8;
  // float32 with radial layers whose values are bounded inside fp16's range: h and h' of the first layer are fp16 pairs
  static_assert(sizeof(RadialScales) == sizeof(m.half_scales[0]), "RadialScales is the header's array");
  const bool half = !f64 && m.radial_half[0][0] != nullptr;
  const bool fused = is_fused(m);
  RadialScales scales[2];
  memcpy(scales, m.half_scales, sizeof(scales));
  if (!fused) {   // the second layer's h and h' leave as float32, without the scale of the pairs
    RadialScales &s = scales[1];
    s.a[2] *= s.out_v;
    s.t[2] *= s.out_t;
    s.out_v = s.out_t = 1.f;
  }
  if (fused && (step == S_RADIAL_OUT || step == S_RADIAL_BACK)) return CMACE_OK;
  if (f64 && !is_spline(m) && step == S_RADIAL_BACK) return CMACE_OK;   // part of edges_back
  io.launches++;
  if (step == S_EDGE_PREP && (node_blocks(io.n_local) > 1 || w.rows.count)) io.launches++;
  if (is_spline(m)) {
    const int rc = run_spline_step<T>(m, io, w, step, up, st);
    if (rc >= 0) return rc;
  }
  switch (step) {
    case S_EDGE_PREP:
      return K::edge_prep(io.positions, io.sender, io.receiver, io.shifts, io.shift_index, io.shift_table,
                                       io.shift_rows, io.status, E, m.r_max, m.nbessel, m.cutoff_p, SplineTable<T>{}, w.geo,
                          w.basis, w.Y, io.species, io.one_hot, io.one_hot_is_f64, nl, n, Z, w.species, w.counts,
                          w.slot_of, w.node_of, w.slot_type, w.elem_start, io.row_ptr, w.rows, st);
    case S_RADIAL: {
      const T *rw[2][3];
      for (int i = 0; i < 2; i++)
        for (int k = 0; k < 3; k++) rw[i][k] = static_cast<const T *>(m.radial[i][k]);
      if constexpr (f64) return radial_pair_f64(w.basis, m.nbessel, rw, 2, w.rows, E, w.h, w.dh, st);
      else if (half) {
        const int half_out[2] = {1, fused ? 1 : 0};
        void *const h[2] = {w.h[0], w.h[1]}, *const dh[2] = {w.dh[0], w.dh[1]};
        return radial_half(w.basis, m.nbessel, m.radial_half, scales, half_out, 2, w.rows, E, h, dh, io.status, st);
      } else return radial_pair_f32(w.basis, m.nbessel, rw, 2, E, w.h, w.dh, io.status, st);
    }
    case S_SUMS:
      if constexpr (!f64)
        if (half) return step_sums_half(w.h[0], w.Y, io.sender, io.row_ptr, w.species, w.slot_of, w.rows.row_of, n, Z, scales[0].out_v, w.A,
                                        st);
      return K::sums(w.h[0], w.Y, io.sender, io.row_ptr, w.species, w.slot_of, w.rows.row_of, n, Z, w.A, st);
    case S_FOLD: return linear_any(w.A, m.fold, start, Z, n, ST_H * Z, C, w.m0, io.status, st);
    case S_CONTRACT0: return K::contract_fwd(w.m0, w.slot_type, static_cast<const T *>(m.weff[0]), n, C, true, w.b0, st);
    case S_MID_FWD:
      return K::mid_fwd(w.b0, w.node_of, w.slot_type, static_cast<const T *>(m.up), static_cast<const T *>(m.extra), n, C,
                        io.up_local ? static_cast<T *>(io.up_local) : w.up, w.q0, st);
    case S_RADIAL_OUT:
      if constexpr (f64)
        return radial_out_f64(w.h[1], w.dh[1], static_cast<const double *>(m.radial[1][3]), w.rows, E, 4 * C, w.R, w.dR, st);
      else return cmace_gemm3x_f32(w.h[1], static_cast<const float *>(m.radial[1][3]), E, ST_H, 4 * C, 1.0, w.R, io.status, st);
    case S_MESSAGES:
      if constexpr (!f64)
        if (fused)
          return fused_messages(up, w.Y, w.h[1], m.fused_w, scales[1].out_v * m.fused_scale, io.sender, io.receiver,
                                io.row_ptr, w.rows.row_of, n, E, C, w.m1, io.status, st);
      if constexpr (f64)
        if (w.rows.count) return imp_fwd_rows_f64(up, w.Y, w.R, w.rows.row_of, io.sender, io.row_ptr, n, E, C, w.m1, st);
      return imp_fwd<T>(up, w.Y, w.R, io.sender, io.row_ptr, n, E, ys, C, w.m1, st);
    case S_LINEAR: return linear_any(w.m1, m.linear[0], nullptr, 1, n, C, C, w.l1, io.status, st);
    case S_CONTRACT1:
      return K::contract_readout(w.l1, w.species, static_cast<const T *>(m.weff[1]), static_cast<const T *>(m.readout1),
                                 m.readout2, w.q0, m.atomic_energies, m.scale, m.shift, n, C, w.gX1, w.dq, io.interaction,
                                 io.node_energy, st);
    case S_LINEAR_BACK: return linear_any(w.gX1, m.linear[1], nullptr, 1, n, C, C, w.gm1, io.status, st);
    case S_EDGES_BACK:
      if constexpr (!f64)
        if (fused)
          return fused_messages_back(up, w.Y, w.gm1, w.h[1], w.dh[1], m.fused_w_back, scales[1].out_v * m.fused_scale,
                                     scales[1].out_t * m.fused_scale, io.sender, io.receiver, w.rows.row_of, E, C, w.T_, w.gY1,
                                     io.status, st);
      if constexpr (f64)
        return imp_bwd_edge_pair_f64(up, w.Y, w.R, w.dR, w.rows.row_of, w.gm1, io.sender, io.row_ptr, n, E, C, w.gY1, w.T_, st);
      else
        return imp_bwd_edge<T>(up, w.Y, w.R, w.gm1, io.sender, io.row_ptr, n, E, ys, C, nullptr, w.gY1, w.T_, nullptr, st);
    case S_RADIAL_BACK:
      if constexpr (!f64)
        return gemm3x_gradr(up, w.gm1, w.Y, ys, io.sender, io.receiver, static_cast<const float *>(m.radial_back), E, C,
                            ST_H, w.dh[1], w.dr1, io.status, st);
      break;
    case S_SENDERS:
      return imp_bwd_node<T>(w.T_, io.perm, io.send_ptr, nl, E, C, gup, st);
    case S_MID_BACK:
      return K::mid_bwd(gup_owned, w.node_of, w.slot_type, w.dq, static_cast<const T *>(m.up_back),
                        static_cast<const T *>(m.extra_back), m.scale, n, C, w.gb0, st);
    case S_CONTRACT0_BACK:
      return K::contract_bwd(w.m0, w.slot_type, static_cast<const T *>(m.weff[0]), w.gb0, n, C, true, w.gX0, st);
    case S_FOLD_BACK:
      // float32: the blocks of two elements in one launch, which reads the rows from memory once
      if constexpr (!f64) {
        if (Z >= 4) {
          if (int rc = linear_tc(w.gX0, static_cast<const float *>(m.fold_back[0]), nullptr, start, Z, Z / 2, n, C, 128, 1.0, w.gA,
                                 io.status, st))
            return rc;
          if (Z % 2 == 0) return CMACE_OK;
        }
      }
      for (int b = !f64 && Z >= 4 ? Z / 2 : 0; 2 * b < Z; b++) {
        if (int rc = linear_any(w.gX0, m.fold_back[b], start, Z, n, C, sums_block_width(Z, b),
                                w.gA + (int64_t)b * n * (16 * 128), io.status, st))
          return rc;
        if (b) io.launches++;
      }
      return CMACE_OK;
    case S_SUMS_BACK:
      if constexpr (!f64)
        if (half)
          return step_sums_bwd_half(w.gA, w.h[0], w.dh[0], w.Y, io.sender, io.row_ptr, w.species, w.slot_of, w.rows.row_of, w.gY1,
                                    fused ? nullptr : w.dr1, w.geo, n, Z, scales[0].out_v, scales[0].out_t, w.gvec, st);
      return K::sums_bwd(w.gA, w.h[0], w.dh[0], w.Y, io.sender, io.row_ptr, w.species, w.slot_of, w.rows.row_of, w.gY1, w.shares,
                         f64 ? nullptr : w.dr1, w.geo, n, E, Z, w.gvec, st);
    case S_FORCES:
      return K::forces(w.gvec, io.row_ptr, io.perm, io.send_ptr, n, nl, io.gradient_sign, io.gradient, io.species, Z,
                       io.interaction, io.node_energy, io.status, f64 ? nullptr : staged_stall_flag(), io.sums, st);
  }
  return fail(CMACE_ERR_ARG, "cmace_step: no step %d", step);
}

// Programmatic launches while launch latency shows between the kernels, us a float32 step of 128 channels without and with them:
// 250 -> 199 at 52 000 edges, 347 -> 306 at 104 000, 454 -> 418 at 156 000, 756 -> 732 at 312 000, 952 -> 961 at 416 000, 1 793 -> 1 859
// at 832 000 (64 channels: 692 -> 678 at 416 000, 1 233 -> 1 255 at 832 000).  A recorded step has smaller gaps: 324 -> 311 at
// 104 000, 429 -> 424 at 156 000, the same at 208 000, 727 -> 740 at 312 000.  float64, whose kernels are long by then: 804 -> 779 at
// 104 000 edges of 64 channels, 1 071 -> 1 123 at 156 000, 1 167 -> 1 211 at 104 000 of 128; recorded 437 -> 433 at 52 000, 775 -> 788
// at 104 000: chained kernels keep their predecessor's split between shared memory and L1.  Tabulated radial weights live on L1:
// half the edges (521 -> 501 us at 104 000, 720 -> 709 at 156 000, 911 -> 914 at 208 000; recorded 187 -> 183 at 26 000, 309 -> 313
// at 52 000).
constexpr int64_t kChainEdges = 98304, kChainEdgesRecorded = 196608, kChainEdgesLive = 393216;

static bool chain_for(const cmace_step_model &m, int64_t edges, cudaStream_t st) {
  const int64_t e = is_spline(m) ? 2 * edges : edges;
  if (e <= kChainEdges) return true;
  if (m.is_f64 || e > kChainEdgesLive) return false;
  if (!is_spline(m) && e <= kChainEdgesRecorded) return true;
  cudaStreamCaptureStatus status;
  return cudaStreamIsCapturing(st, &status) == cudaSuccess && status == cudaStreamCaptureStatusNone;
}

template <typename T>
static int run_steps(const cmace_step_model &m, cmace_step_io &io, int first, int last, cudaStream_t st) {
  const Workspace<T> w(io.workspace, m, io.n_owned, io.n_local, io.nedges);
  if (io.workspace_bytes < w.bytes)
    return fail(CMACE_ERR_ARG, "cmace_step: workspace of %lld bytes, %lld needed", (long long)io.workspace_bytes, (long long)w.bytes);
  // The first kernel of a range beyond step 0 is not chained: its beginning may read the list or an exchanged row before its
  // wait, and the caller may have put the kernel that makes them right before this call.  Step 0 begins with its wait.
  chain_launches() = !chain_for(m, io.nedges, st) ? Chain::off : first > 0 ? Chain::from_second : Chain::on;
  int rc = CMACE_OK;
  for (int s = first; s < last && rc == CMACE_OK; s++) rc = run_step<T>(m, io, w, s, st);
  chain_launches() = Chain::off;
  return rc;
}

}  // namespace cmace

using namespace cmace;

extern "C" {

int64_t cmace_step_workspace_bytes(const cmace_step_model *m, int64_t n_owned, int64_t n_local, int64_t nedges) {
  if (!m || n_owned < 0 || n_local < n_owned || nedges < 0) return 0;
  return m->is_f64 ? Workspace<double>(nullptr, *m, n_owned, n_local, nedges).bytes
                   : Workspace<float>(nullptr, *m, n_owned, n_local, nedges).bytes;
}
int cmace_step_count(void) { return S_COUNT; }
int cmace_step_struct_bytes(int which) { return which == 0 ? (int)sizeof(cmace_step_model) : (int)sizeof(cmace_step_io); }
const char *cmace_step_name(int step) { return step >= 0 && step < S_COUNT ? kStepNames[step] : ""; }

int cmace_step_run(const cmace_step_model *m, cmace_step_io *io, int first, int last, cmace_stream_t stream) {
  if (!m || !io || first < 0 || last > S_COUNT || first > last) return fail(CMACE_ERR_ARG, "cmace_step: bad argument");
  if (m->channels % 32 != 0 || m->channels < 32 || m->channels > 128 || m->elements < 1 || m->elements > ST_MAX_Z ||
      (!is_spline(*m) && m->nbessel != 8 && m->nbessel != 16))
    return fail(CMACE_ERR_UNSUPPORTED, "cmace_step: 32, 64, 96 or 128 channels, 1..%d elements, 8 or 16 basis functions", ST_MAX_Z);
  if (io->n_owned < 1 || io->n_local < io->n_owned || io->nedges < 0 || io->nedges > 0x7fffff00LL)
    return fail(CMACE_ERR_ARG, "cmace_step: bad size");
  if (!io->positions || (!io->species && !io->one_hot) || !io->row_ptr || !io->send_ptr || !io->workspace ||
      !io->node_energy || !io->interaction || !io->sums || !io->gradient ||
      (io->nedges > 0 && (!io->sender || !io->receiver || !io->perm)) ||
      (io->shift_index && (!io->shift_table || !io->status)))
    return fail(CMACE_ERR_ARG, "cmace_step: null pointer");
  if (io->n_local != io->n_owned && (!io->up_local || !io->gup_local || !io->gup_owned))
    return fail(CMACE_ERR_ARG, "cmace_step: ghost rows need the caller's node feature arrays");
  cudaStream_t st = (cudaStream_t)stream;
  return m->is_f64 ? run_steps<double>(*m, *io, first, last, st) : run_steps<float>(*m, *io, first, last, st);
}
}
