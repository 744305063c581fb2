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
#include "tc_ptx.cuh"

namespace cmace {

// ---- edge geometry, basis and node grouping ----------------------------------------------------------------------
constexpr int EP_THREADS = 256;

// The first blocks resolve the species, GN_NODES nodes each, beside the edge blocks.  One block (the usual number in the
// systems that are bound by launches) also groups the owned nodes by element, stable; several leave their counts per element to
// group_nodes_kernel.  One block for all nodes was the kernel's whole time: 325 us at 64 000 nodes, 50 us at 8 000, where
// the edges take 110 and 15; now 123 and 18.
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

__device__ void resolve_nodes(const int32_t *__restrict__ species_in, const void *__restrict__ one_hot, int one_hot_f64,
                              int64_t lo, int64_t hi, int elements, int32_t *__restrict__ species, int32_t *status) {
  constexpr int PER = GN_NODES / EP_THREADS;
  int z[PER];
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const int64_t i = lo + u * EP_THREADS + threadIdx.x;
    z[u] = 0;
    if (i >= hi) continue;
    if (species_in) z[u] = species_in[i];
    else if (one_hot_f64) z[u] = first_max(static_cast<const double *>(one_hot) + i * elements, elements);
    else z[u] = first_max(static_cast<const float *>(one_hot) + i * elements, elements);
  }
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const int64_t i = lo + u * EP_THREADS + threadIdx.x;
    if (i >= hi) continue;
    const bool known = z[u] >= 0 && z[u] < elements;
    species[i] = known ? z[u] : 0;   // the tables are read with it; forces_kernel takes such a node's energy away
    if (!known && status) *status = CMACE_STEP_BAD_ELEMENT;
  }
  __syncthreads();
}

// Groups the nodes [first, end) of one block, or counts them.  A warp takes a consecutive piece, four nodes a lane, and
// ranks them by ballot, so that loads and stores are coalesced.  counts: [blocks, ST_MAX_Z]; with one block the start of
// every element follows from its own counts.
__device__ void group_nodes(int64_t first, int64_t end, int blocks, int block, bool count_only, int elements,
                            const int32_t *species, int32_t *counts, int32_t *slot_of, int32_t *node_of, int32_t *slot_type,
                            int32_t *elem_start) {
  constexpr int WARPS = EP_THREADS / 32, PIECE = GN_NODES / WARPS;
  __shared__ int count[WARPS][ST_MAX_Z];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t lo = first + w * PIECE < end ? first + w * PIECE : end, hi = lo + PIECE < end ? lo + PIECE : end;
  const unsigned below = (1u << lane) - 1u;
  int run = 0;   // lane z: first its number of nodes, then the slot of the next one
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
#pragma unroll 1
    for (int64_t b = lo; b < hi; b += 128) {
      const int64_t i = b + 4 * lane;
      int4 z = make_int4(-1, -1, -1, -1);
      if (i < hi) z = *reinterpret_cast<const int4 *>(species + i);   // the array ends on a 256-byte boundary
      if (i + 1 >= hi) z.y = -1;
      if (i + 2 >= hi) z.z = -1;
      if (i + 3 >= hi) z.w = -1;
      int4 slot = make_int4(0, 0, 0, 0);
#pragma unroll 1
      for (int k = 0; k < elements; k++) {
        const unsigned m0 = __ballot_sync(0xffffffffu, z.x == k), m1 = __ballot_sync(0xffffffffu, z.y == k);
        const unsigned m2 = __ballot_sync(0xffffffffu, z.z == k), m3 = __ballot_sync(0xffffffffu, z.w == k);
        int at = __shfl_sync(0xffffffffu, run, k) + __popc(m0 & below) + __popc(m1 & below) + __popc(m2 & below) + __popc(m3 & below);
        if (z.x == k) slot.x = at++;
        if (z.y == k) slot.y = at++;
        if (z.z == k) slot.z = at++;
        if (z.w == k) slot.w = at++;
        if (lane == k) run += __popc(m0) + __popc(m1) + __popc(m2) + __popc(m3);
      }
      if (pass == 0) continue;
      auto place = [&](int64_t node, int s, int zz) {
        if (zz < 0) return;
        slot_of[node] = s;
        node_of[s] = (int32_t)node;
        slot_type[s] = zz;
      };
      place(i, slot.x, z.x);
      place(i + 1, slot.y, z.y);
      place(i + 2, slot.z, z.z);
      place(i + 3, slot.w, z.w);
    }
    if (pass == 1) break;
    if (lane < ST_MAX_Z) count[w][lane] = run;
    __syncthreads();
    int before = 0, total = 0;   // lane z: nodes of element z before this warp's piece, and in all
    if (lane < elements) {
      for (int v = 0; v < WARPS; v++) {
        before += v < w ? count[v][lane] : 0;
        total += count[v][lane];
      }
      if (count_only) {
        if (w == 0) counts[block * ST_MAX_Z + lane] = total;
      } else if (blocks > 1) {
        total = 0;
#pragma unroll 4
        for (int v = 0; v < blocks; v++) {
          const int c = counts[v * ST_MAX_Z + lane];
          before += v < block ? c : 0;
          total += c;
        }
      }
    }
    if (count_only) return;
    int inc = total;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += o;
    }
    if (w == 0 && block == 0 && lane <= elements) elem_start[lane] = inc - total;   // lane `elements` has none: the end
    run = inc - total + before;
  }
}

// ---- edges that share a length ------------------------------------------------------------------------------------
// The vectors of an edge j -> i and its reverse i -> j are exact negatives, so their lengths and both perceptrons' rows h and h' are
// the same: they are formed once a pair.  In a complete list that is half of the radial work; an edge whose reverse is missing (an
// incomplete list, a ghost sender) keeps a row of its own.  What is compared are the rounded unit vectors and 1/r of this call:
// two edges between the same atoms that agree in these have the same length but for its rounding.
//
// Of a pair the edge with the lower receiver leads; the other looks for it in its sender's row of the list: a warp asks the rows
// of eight of its edges at a time, lanes beside one another, the first edge that matches is the leader.  Leaders are numbered as
// they come, a block at a time (rows do not depend on one another, so their places need not be the same in every call):
// leaders[k] is the edge of row k, row_of[e] the row of a leader, and ~leader for the other edge of a pair until the radial kernel
// looks its row up (resolve_rows).  The search is a chain of four dependent loads in short lists and instruction issue in long ones:
// 8 us for 9 900 edges, 14 for 416 000 in float64, 22 for 833 000 and 100 for 3.3 million in float32 (a quarter of the blocks'
// additions to the counter: the same); with the vectors compared for four edges one after the other 20 and 39 in float64.  A list
// without reverses pays the search for nothing, us of a step: 3 to 4 for 20 600 edges, 7 for 42 000, 16 for 416 000, 60 for 1.7 million
// where every edge looks (senders below their receivers), 3, 4, 4 and 18 where none does.  In a complete list the float32 radial kernel
// alone saves 8 for 20 900 edges, 27 for 156 000, 140 for 833 000, 630 for 3.3 million.
template <typename T>
__device__ __forceinline__ void find_pairs(int64_t first, const int32_t *__restrict__ sender, const int32_t *__restrict__ receiver,
                                           const int32_t *__restrict__ row_ptr, const Quad<T> *__restrict__ geo, int64_t nedges,
                                           int32_t *__restrict__ row_of, int32_t *__restrict__ leaders, int32_t *count) {
  __shared__ int32_t found[EP_THREADS / 32], start;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t e = first + threadIdx.x;
  const bool valid = e < nedges;
  int s = 0, r = 0, k0 = 0, k1 = 0, leader = -1;
  Quad<T> q{};
  if (valid) {
    s = sender[e];
    r = receiver[e];
    q = geo[e];
  }
  const bool looks = valid && s < r;   // then the sender receives too
  if (looks) {
    k0 = row_ptr[s];
    k1 = row_ptr[s + 1];
  }
  unsigned open = __ballot_sync(0xffffffffu, looks);
  for (int at = 0; open != 0; at += 64) {
    unsigned hits[2] = {0, 0};   // candidates at .. at + 63 with the right sender, of this lane's edge
    for (unsigned todo = open; todo != 0;) {
      constexpr int AT = 8;      // rows on their way together
      int src[AT], cand[AT][2];
#pragma unroll
      for (int u = 0; u < AT; u++) {
        src[u] = todo ? __ffs(todo) - 1 : -1;
        todo &= todo - 1;
        const int c = __shfl_sync(0xffffffffu, k0, src[u] & 31) + at + lane, hi = __shfl_sync(0xffffffffu, k1, src[u] & 31);
        cand[u][0] = src[u] >= 0 && c < hi ? __ldg(sender + c) : -1;
        cand[u][1] = src[u] >= 0 && c + 32 < hi ? __ldg(sender + c + 32) : -1;
      }
#pragma unroll
      for (int u = 0; u < AT; u++) {
        if (src[u] < 0) break;
        const int want = __shfl_sync(0xffffffffu, r, src[u]);
        const unsigned m0 = __ballot_sync(0xffffffffu, cand[u][0] == want), m1 = __ballot_sync(0xffffffffu, cand[u][1] == want);
        if (lane == src[u]) {
          hits[0] = m0;
          hits[1] = m1;
        }
      }
    }
    // every lane for itself: nearly always one candidate, several where images of an atom are neighbours
#pragma unroll
    for (int h = 0; h < 2; h++)
      while (leader < 0 && hits[h] != 0) {
        const int c = k0 + at + 32 * h + __ffs(hits[h]) - 1;
        hits[h] &= hits[h] - 1;
        const Quad<T> v = geo[c];
        if (v.x == -q.x && v.y == -q.y && v.z == -q.z && v.w == q.w) leader = c;
      }
    __syncwarp();
    open = __ballot_sync(0xffffffffu, looks && leader < 0 && k0 + at + 64 < k1);
  }
  const bool leads = valid && leader < 0;
  const unsigned mine = __ballot_sync(0xffffffffu, leads);
  if (lane == 0) found[w] = __popc(mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = 0;
    for (int k = 0; k < EP_THREADS / 32; k++) n += found[k];
    start = atomicAdd(count, n);
  }
  __syncthreads();
  int row = start + __popc(mine & ((1u << lane) - 1u));
  for (int k = 0; k < w; k++) row += found[k];
  if (leads) leaders[row] = (int32_t)e;
  if (valid) row_of[e] = leads ? row : ~leader;
}

// What has to wait for edge_prep's counts and vectors: with several node blocks the grouping of the nodes, and the pairs
template <typename T>
__global__ void __launch_bounds__(EP_THREADS)
    group_kernel(int64_t n_owned, int grouping, int elements, const int32_t *species, int32_t *counts, int32_t *slot_of,
                 int32_t *node_of, int32_t *slot_type, int32_t *elem_start, const int32_t *sender, const int32_t *receiver,
                 const int32_t *row_ptr, const Quad<T> *geo, int64_t nedges, int32_t *row_of, int32_t *leaders, int32_t *count) {
  grid_begin();
  if ((int)blockIdx.x < grouping) {
    const int64_t first = (int64_t)blockIdx.x * GN_NODES;
    group_nodes(first, first + GN_NODES < n_owned ? first + GN_NODES : n_owned, grouping, (int)blockIdx.x, false, elements,
                species, counts, slot_of, node_of, slot_type, elem_start);
    return;
  }
  find_pairs<T>(((int64_t)blockIdx.x - grouping) * EP_THREADS, sender, receiver, row_ptr, geo, nedges, row_of, leaders, count);
}

// A warp's 32 rows of N values each, one row per lane, to consecutive memory: through shared memory, so that a store
// instruction covers consecutive 16-byte pieces (row stride of one piece more than the row: no bank conflicts).
template <typename T, int N>
__device__ __forceinline__ void store_rows(uint4 *buf, const T (&v)[N], T *__restrict__ out, int rows, int lane) {
  constexpr int PIECES = N * (int)sizeof(T) / 16, PER = 16 / (int)sizeof(T);
#pragma unroll
  for (int i = 0; i < PIECES; i++) {
    uint4 q;
    T *t = reinterpret_cast<T *>(&q);
#pragma unroll
    for (int u = 0; u < PER; u++) t[u] = v[i * PER + u];
    buf[lane * (PIECES + 1) + i] = q;
  }
  __syncwarp();
  uint4 *o = reinterpret_cast<uint4 *>(out);
#pragma unroll
  for (int i = 0; i < PIECES; i++) {
    const int k = i * 32 + lane, row = k / PIECES;
    if (row < rows) o[k] = buf[row * (PIECES + 1) + (k - row * PIECES)];
  }
  __syncwarp();
}

// One thread per edge: vector in float64, then unit vector and 1/r, basis and its derivative [E, 2 NB], Y [E, 16].
template <typename T, int NB>
__global__ void __launch_bounds__(EP_THREADS, sizeof(T) == 4 ? 5 : 3)
    edge_prep_kernel(const double *__restrict__ pos, const int32_t *__restrict__ sender,
                     const int32_t *__restrict__ receiver, const double *__restrict__ shifts,
                     const uint8_t *__restrict__ shift_index, const double *__restrict__ shift_table, int shift_rows,
                     int32_t *status, int64_t nedges, T r_max,
                     int p, const SplineTable<T> spline, Quad<T> *__restrict__ geo, T *__restrict__ basis, T *__restrict__ Y,
                     const int32_t *species_in, const void *one_hot, int one_hot_f64, int64_t n_local, int64_t n_owned,
                     int elements, int32_t *species, int32_t *counts, int32_t *slot_of, int32_t *node_of,
                     int32_t *slot_type, int32_t *elem_start, int32_t *pair_count) {
  grid_begin();
  if (pair_count && blockIdx.x == 0 && threadIdx.x == 0) *pair_count = 0;
  const int nblocks = (int)node_blocks(n_local);
  if ((int)blockIdx.x < nblocks) {
    const int64_t first = (int64_t)blockIdx.x * GN_NODES, end = first + GN_NODES;
    resolve_nodes(species_in, one_hot, one_hot_f64, first, end < n_local ? end : n_local, elements, species, status);
    group_nodes(first, end < n_owned ? end : n_owned, 1, (int)blockIdx.x, nblocks > 1, elements, species, counts, slot_of,
                node_of, slot_type, elem_start);
    return;
  }
  extern __shared__ uint4 ep_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int MOST = 2 * NB > 16 ? 2 * NB : 16;
  uint4 *buf = ep_smem + w * 32 * (MOST * (int)sizeof(T) / 16 + 1);
  const int64_t base = ((int64_t)blockIdx.x - nblocks) * EP_THREADS + w * 32;
  if (base >= nedges) return;
  const int rows = nedges - base < 32 ? (int)(nedges - base) : 32;
  const int64_t e = base + (lane < rows ? lane : rows - 1);
  const int64_t s = sender[e], r = receiver[e];
  const double *sh = shifts ? shifts + e * 3 : nullptr;
  bool known = true;
  if (shift_index) {
    const int k = shift_index[e];
    known = k < shift_rows;
    if (known) sh = shift_table + 3 * k;
    else *status = CMACE_STEP_BAD_SHIFT;
  }
  T v[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    double d = __dsub_rn(pos[s * 3 + c], pos[r * 3 + c]);
    if (sh) d = __dadd_rn(d, sh[c]);
    v[c] = known ? (T)d : (T)CUDART_NAN;
  }
  const T r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
  const T ir = inv_sqrt(r2);
  const T ux = v[0] * ir, uy = v[1] * ir, uz = v[2] * ir;
  T y[16];
  sph_l3<T>(uz, ux, uy, y);
  if (lane < rows) geo[e] = Quad<T>{ux, uy, uz, ir};
  store_rows<T, 16>(buf, y, Y + base * 16, rows, lane);
  if constexpr (NB == 0) {   // tabulated radial weights: where the length lies in the table
    const T len = r2 * ir;
    SplinePoint<T> at;
    at.x = T(0);
    at.interval = -1;
    if (!(len > spline.r_max)) {
      const int k = (int)(len / spline.width);
      at.interval = k < 0 ? 0 : (k >= spline.intervals ? spline.intervals - 1 : k);
      at.x = len - spline.knots[at.interval];
    }
    if (lane < rows) reinterpret_cast<SplinePoint<T> *>(basis)[e] = at;
  } else {
    T b[2 * NB];
    bessel_cutoff<T>(r2 * ir, r_max, NB, p, b, b + NB);
    store_rows<T, 2 * NB>(buf, b, basis + base * 2 * NB, rows, lane);
  }
}

template <typename T>
int StepKernels<T>::edge_prep(const double *pos, const int32_t *sender, const int32_t *receiver, const double *shifts,
                              const uint8_t *shift_index, const double *shift_table, int64_t shift_rows, int32_t *status,
                              int64_t nedges, double r_max, int nb, int p, const SplineTable<T> &spline, Quad<T> *geo,
                              T *basis, T *Y,
                              const int32_t *species_in, const void *one_hot, int one_hot_f64, int64_t n_local,
                              int64_t n_owned, int elements, int32_t *species, int32_t *counts, int32_t *slot_of, int32_t *node_of,
                              int32_t *slot_type, int32_t *elem_start, const int32_t *row_ptr, const EdgeRows &rows,
                              cudaStream_t st) {
  const int64_t blocks = node_blocks(n_local) + (nedges + EP_THREADS - 1) / EP_THREADS;
  const size_t smem = (size_t)EP_THREADS * ((nb == 16 ? 32 : 16) * sizeof(T) + 16);
  auto kern = nb == 16 ? edge_prep_kernel<T, 16> : (nb == 8 ? edge_prep_kernel<T, 8> : edge_prep_kernel<T, 0>);
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return fail(CMACE_ERR_CUDA, "cmace_step(edge_prep): %s", cudaGetErrorString(err));
  launch_chained(kern, (unsigned)blocks, EP_THREADS, smem, st, pos, sender, receiver, shifts, shift_index, shift_table,
                 (int)(shift_rows < 256 ? shift_rows : 256), status, nedges, (T)r_max, p, spline, geo, basis, Y, species_in, one_hot,
                 one_hot_f64, n_local, n_owned, elements, species, counts, slot_of, node_of, slot_type,
                 elem_start, rows.count);
  const int64_t grouping = node_blocks(n_local) > 1 ? node_blocks(n_owned) : 0;
  const int64_t pairs = rows.count ? (nedges + EP_THREADS - 1) / EP_THREADS : 0;
  if (grouping + pairs > 0)
    launch_chained(group_kernel<T>, (unsigned)(grouping + pairs), EP_THREADS, 0, st, n_owned, (int)grouping, elements, species, counts,
                   slot_of, node_of, slot_type, elem_start, sender, receiver, row_ptr, geo, nedges, rows.row_of, rows.leaders,
                   rows.count);
  return check_launch("cmace_step(edge_prep)");
}

// ---- the edges of one (receiver, element) pair -------------------------------------------------------------------
// A warp owns the pair.  It lists the edges whose sender has the element, 32 candidates at a time (ballot), into a
// per-warp buffer and calls body(list, n) whenever the buffer is full and at the end; edges come in list order.  The elements
// of the first 64 edges' senders are two dependent loads that the caller starts before it waits for anything else
// (SenderElements): a pair's life is a chain of such loads and little work.
constexpr int SU_WARPS = 4;
constexpr int SU_LIST = 64;

// Elements of a receiver that a warp takes one after the other (float32): its list, the senders' elements and the rows are looked up
// once, which is most of a pair's chain of loads; while that leaves the chip about 24 warps an SM, in equal parts.  us, sums and
// backward, one element a warp and this: 136, 183 -> 109, 166 at 16 000 atoms of 4 elements, 262, 289 -> 203, 264 of 10; 562, 735 ->
// 414, 629 at 64 000; 33, 46 -> 29, 43 at 3 000 of 4 (all four: 31, 48).  In float64 the registers of the loop cost a block an SM:
// 127, 260 -> 135, 260 at 8 000.
static int elements_per_warp(int64_t nnodes, int elements) {
  const int64_t fit = nnodes * elements / (148 * 24);
  const int most = fit < 1 ? 1 : (fit > elements ? elements : (int)fit), chunks = (elements + most - 1) / most;
  return (elements + chunks - 1) / chunks;
}

// In a chain of launches (EARLY) the list is read before grid_wait(), and while few warps ask (kSoonWarps) the senders' elements as well,
// from L2: 91.9 -> 91.2 us a step of 192 atoms of 4 elements, but 106 -> 113 at 300 of 10, whose 3 000 warps meet at the ten lines of the
// elements; those look them up behind the wait, through L1.  Otherwise the look-up stands behind the loads that it would hold up: with
// one order for both the sums of 16 000 atoms took 144 us instead of 135, their backward 191 instead of 183.
constexpr int64_t kSoonWarps = 148 * 8;
struct SenderElements {
  const int32_t *__restrict__ sender, *__restrict__ species;
  int64_t e0, e1;
  int32_t s[2];
  int lane;
  __device__ __forceinline__ SenderElements(const int32_t *__restrict__ sender_, const int32_t *__restrict__ species_,
                                            int64_t e0_, int64_t e1_, int lane_)
      : sender(sender_), species(species_), e0(e0_), e1(e1_), lane(lane_) {
#pragma unroll
    for (int c = 0; c < 2; c++) s[c] = e0 + 32 * c + lane < e1 ? __ldg(sender + e0 + 32 * c + lane) : -1;
  }
  template <bool EARLY = false>
  __device__ __forceinline__ void look_up() {   // the elements in place of the senders
#pragma unroll
    for (int c = 0; c < 2; c++) s[c] = s[c] >= 0 ? (EARLY ? __ldcg(species + s[c]) : __ldg(species + s[c])) : -1;
  }
};

// Rows of h and h' of a receiver's edges (EdgeRows; null: an edge's own), listed beside the edges.  Those of the first 64 wait in
// shared memory, where asynchronous copies bring them: in registers they cost these kernels a block an SM, from L1, prefetched, the
// sums of 16 000 atoms take 158 us instead of 137 in float32, of 8 000 156 instead of 127 in float64.
struct SharedRows {
  const int32_t *__restrict__ row_of;
  int32_t *first, *list;
  // early: before grid_wait(), from L2
  __device__ __forceinline__ SharedRows(const int32_t *__restrict__ row_of_, int32_t (&buf)[64 + SU_LIST], const SenderElements &from,
                                        bool early = false)
      : row_of(row_of_), first(buf), list(buf + 64) {
#pragma unroll
    for (int i = 0; i < 64; i += 32)
      if (from.e0 + i + from.lane < from.e1) {
        if (row_of && early)
          first[i + from.lane] = __ldcg(row_of + from.e0 + i + from.lane);
        else if (row_of)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(first + i + from.lane)),
                       "l"(row_of + from.e0 + i + from.lane)
                       : "memory");
        else
          first[i + from.lane] = (int32_t)from.e0 + i + from.lane;
      }
  }
  __device__ __forceinline__ void wait() const {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }
  __device__ __forceinline__ void put(int at, int64_t e, int64_t e0) {
    list[at] = e - e0 < 64 ? first[e - e0] : (row_of ? __ldg(row_of + e) : (int32_t)e);
  }
  __device__ __forceinline__ int64_t operator[](int i) const { return list[i]; }
};
struct OwnRows {
  __device__ __forceinline__ void put(int, int64_t, int64_t) {}
};

template <typename Rows, typename Body>
__device__ __forceinline__ void for_edges_of_element(const SenderElements &from, int z, int32_t *list, Rows &rows, Body body) {
  const int lane = from.lane;
  int n = 0;
  for (int64_t eb = from.e0; eb < from.e1; eb += 32) {
    const int64_t e = eb + lane;
    int of = -1;
    if (eb == from.e0) of = from.s[0];
    else if (eb == from.e0 + 32) of = from.s[1];
    else if (e < from.e1) of = __ldg(from.species + __ldg(from.sender + e));
    const bool hit = of == z;
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (hit) {
      const int at = n + __popc(m & ((1u << lane) - 1u));
      list[at] = (int32_t)e;
      rows.put(at, e, from.e0);
    }
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

// 32 bytes of one lane in one store.  The lanes of a result tile hold 64 bytes of a row each: in 16-byte stores every
// instruction half-fills 32 sectors, which L2 takes as 2.5 times the writes (10.2 million sectors for 131 MB).
__device__ __forceinline__ void store32(float *p, float a, float b, float c, float d, float e, float f, float g, float h) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d), "f"(e),
               "f"(f), "f"(g), "f"(h)
               : "memory");
}
__device__ __forceinline__ void store32(double *p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// and in one load; volatile, like the wait for the kernel before that wrote these rows, so that it stays behind it
__device__ __forceinline__ void load32(const float *p, float4 &a, float4 &b) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
               : "l"(p));
}
__device__ __forceinline__ void load_row16(const float *p, float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 2; i++) {
    float4 a, b;
    load32(p + 8 * i, a, b);
    v[8 * i] = a.x, v[8 * i + 1] = a.y, v[8 * i + 2] = a.z, v[8 * i + 3] = a.w;
    v[8 * i + 4] = b.x, v[8 * i + 5] = b.y, v[8 * i + 6] = b.z, v[8 * i + 7] = b.w;
  }
}
__device__ __forceinline__ void load_row16(const double *p, double (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; i++)
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[4 * i]), "=d"(v[4 * i + 1]), "=d"(v[4 * i + 2]), "=d"(v[4 * i + 3])
                 : "l"(p + 4 * i));
}
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ void store_quad(float *p, float a, float b, float c) {
  *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, 0.f);
}
__device__ __forceinline__ void store_quad(double *p, double a, double b, double c) { store32(p, a, b, c, 0.0); }

// 3-term TF32 split for mma.sync m16n8k8: x = hi + lo, hi by truncation, lo rounded
__device__ __forceinline__ void split_tf32(float x, uint32_t &hi, uint32_t &lo) {
  hi = __float_as_uint(x) & 0xFFFFE000u;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// float32: eight edges at a time on the warp-level tensor instruction.  The operands of a pair are tiny (16 x n times
// n x 64, n about 13) and come straight from memory into fragments, which is what mma.sync is for; a tcgen05 tile of
// 128 rows would be padding.  D = Y^T h: A fragment = Y of edges t, t + 4 (t = lane & 3) for lm = g, g + 8 (g = lane >> 2);
// column g of tile j is k = 8 g + j, so that a lane reads 32 consecutive bytes of an edge's row and the lanes of an edge
// its whole row, and so that what a lane holds in the end is 16 consecutive k of two rows of the sums.
__global__ void __launch_bounds__(SU_WARPS * 32)
    sums_tf32_kernel(const float *__restrict__ h, const float *__restrict__ Y, const int32_t *__restrict__ sender,
                     const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ species,
                     const int32_t *__restrict__ slot_of, int64_t nnodes, int elements, float *__restrict__ A) {
  grid_begin();
  __shared__ int32_t lists[SU_WARPS][SU_LIST];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (pair >= nnodes * elements) return;
  const int64_t node = pair / elements;
  const int z = (int)(pair - node * elements);
  SenderElements from(sender, species, row_ptr[node], row_ptr[node + 1], lane);
  int32_t *list = lists[w];
  float acc[8][4];
#pragma unroll
  for (int j = 0; j < 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  from.look_up();
  OwnRows rows;
  for_edges_of_element(from, z, list, rows, [&](int n) {
    float4 hv[2][2];
    float yv[4];
    auto load = [&](int j0) {   // edges j0 + t and j0 + t + 4; past the end: the last edge with Y = 0
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int j = j0 + t + 4 * u;
        const int64_t e = list[j < n ? j : n - 1];
        const float4 *hp = reinterpret_cast<const float4 *>(h + e * ST_H + 8 * g);
        hv[u][0] = __ldg(hp);
        hv[u][1] = __ldg(hp + 1);
        yv[2 * u] = j < n ? __ldg(Y + e * 16 + g) : 0.f;
        yv[2 * u + 1] = j < n ? __ldg(Y + e * 16 + g + 8) : 0.f;
      }
    };
    load(0);
    for (int j0 = 0; j0 < n; j0 += 8) {
      uint32_t ah[4], al[4], bh[2][8], bl[2][8];
#pragma unroll
      for (int i = 0; i < 4; i++) split_tf32(yv[i], ah[i], al[i]);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        split_tf32(hv[u][0].x, bh[u][0], bl[u][0]);
        split_tf32(hv[u][0].y, bh[u][1], bl[u][1]);
        split_tf32(hv[u][0].z, bh[u][2], bl[u][2]);
        split_tf32(hv[u][0].w, bh[u][3], bl[u][3]);
        split_tf32(hv[u][1].x, bh[u][4], bl[u][4]);
        split_tf32(hv[u][1].y, bh[u][5], bl[u][5]);
        split_tf32(hv[u][1].z, bh[u][6], bl[u][6]);
        split_tf32(hv[u][1].w, bh[u][7], bl[u][7]);
      }
      if (j0 + 8 < n) load(j0 + 8);
#pragma unroll
      for (int j = 0; j < 8; j++) mma_tf32(acc[j], ah, bh[0][j], bh[1][j]);
#pragma unroll
      for (int j = 0; j < 8; j++) mma_tf32(acc[j], ah, bl[0][j], bl[1][j]);
#pragma unroll
      for (int j = 0; j < 8; j++) mma_tf32(acc[j], al, bh[0][j], bh[1][j]);
    }
  });
  const int width = elements * ST_H;
  float *o = A + (int64_t)slot_of[node] * 16 * width + z * ST_H + 16 * t;
#pragma unroll
  for (int half = 0; half < 2; half++) {   // rows lm = g and g + 8
    float *row = o + (int64_t)(g + 8 * half) * width;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int c = 2 * half + u;
      store32(row + 8 * u, acc[0][c], acc[1][c], acc[2][c], acc[3][c], acc[4][c], acc[5][c], acc[6][c], acc[7][c]);
    }
  }
}

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The same with h as fp16 hi / lo rows ([E][hi 64 | lo 64], scaled): sixteen edges an instruction, nothing to split but
// Y (times 2^8: |Y| < 2.7).  Lane (g, t) reads 16 bytes of the hi and of the lo row of edges 2 t, 2 t + 1, 2 t + 8,
// 2 t + 9; a B fragment pairs the same column of two edges (one byte permute).
constexpr float SU_Y_SCALE = 256.f;

template <bool EARLY>
__global__ void __launch_bounds__(SU_WARPS * 32)
    sums_f16_kernel(const uint4 *__restrict__ h, const float *__restrict__ Y, const int32_t *__restrict__ sender,
                    const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ species,
                    const int32_t *__restrict__ slot_of, const int32_t *__restrict__ row_of, int64_t nnodes, int elements, int per,
                    float factor,
                    float *__restrict__ A) {
  __shared__ int32_t lists[SU_WARPS][SU_LIST], row_lists[SU_WARPS][64 + SU_LIST];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (!EARLY) grid_begin();
  const int chunks = (elements + per - 1) / per;
  if (pair >= nnodes * chunks) {
    if (EARLY) grid_begin();
    return;
  }
  const bool soon = nnodes * chunks <= kSoonWarps;
  const int64_t node = pair / chunks;
  const int z0 = (int)(pair - node * chunks) * per, z1 = z0 + per < elements ? z0 + per : elements;
  SenderElements from(sender, species, row_ptr[node], row_ptr[node + 1], lane);
  if (EARLY) {
    if (soon) from.look_up<true>();
    grid_begin();
    if (!soon) from.look_up();
  }
  SharedRows rows(row_of, row_lists[w], from);
  int32_t *list = lists[w];
  if (!EARLY) from.look_up();
  rows.wait();
#pragma unroll 1
  for (int z = z0; z < z1; z++) {
    __syncwarp();   // the list of the element before has been read
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    for_edges_of_element(from, z, list, rows, [&](int n) {
      for (int j0 = 0; j0 < n; j0 += 16) {
        uint4 hv[4], lv[4];
        uint32_t ah[4], al[4];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          float y[2][2];
#pragma unroll
          for (int v = 0; v < 2; v++) {   // past the end: the last edge with Y = 0
            const int j = j0 + 8 * u + 2 * t + v;
            const int64_t e = list[j < n ? j : n - 1];
            const int64_t row = rows[j < n ? j : n - 1];
            hv[2 * u + v] = __ldg(h + row * 16 + g);
            lv[2 * u + v] = __ldg(h + row * 16 + 8 + g);
            y[v][0] = j < n ? __ldg(Y + e * 16 + g) * SU_Y_SCALE : 0.f;
            y[v][1] = j < n ? __ldg(Y + e * 16 + g + 8) * SU_Y_SCALE : 0.f;
          }
          split_half2(pack2(y[0][0], y[1][0]), ah[2 * u], al[2 * u]);
          split_half2(pack2(y[0][1], y[1][1]), ah[2 * u + 1], al[2 * u + 1]);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          auto word = [&](const uint4 &x) { return (j >> 1) == 0 ? x.x : ((j >> 1) == 1 ? x.y : ((j >> 1) == 2 ? x.z : x.w)); };
          const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
          const uint32_t h0 = __byte_perm(word(hv[0]), word(hv[1]), sel), h1 = __byte_perm(word(hv[2]), word(hv[3]), sel);
          const uint32_t l0 = __byte_perm(word(lv[0]), word(lv[1]), sel), l1 = __byte_perm(word(lv[2]), word(lv[3]), sel);
          mma_f16(acc[j], ah, h0, h1);
          mma_f16(acc[j], ah, l0, l1);
          mma_f16(acc[j], al, h0, h1);
        }
      }
    });
    const int width = elements * ST_H;
    float *o = A + (int64_t)slot_of[node] * 16 * width + z * ST_H + 16 * t;
#pragma unroll
    for (int half = 0; half < 2; half++) {   // rows lm = g and g + 8
      float *row = o + (int64_t)(g + 8 * half) * width;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int c = 2 * half + u;
        store32(row + 8 * u, acc[0][c] * factor, acc[1][c] * factor, acc[2][c] * factor, acc[3][c] * factor, acc[4][c] * factor,
                acc[5][c] * factor, acc[6][c] * factor, acc[7][c] * factor);
      }
    }
  }
}

int step_sums_half(const void *h, const float *Y, const int32_t *sender, const int32_t *row_ptr, const int32_t *species,
                   const int32_t *slot_of, const int32_t *row_of, int64_t nnodes, int elements, float out_v, float *A,
                   cudaStream_t st) {
  const int per = elements_per_warp(nnodes, elements);
  const int64_t blocks = (nnodes * ((elements + per - 1) / per) + SU_WARPS - 1) / SU_WARPS;
  if (blocks > 0)
    launch_chained(chain_launches() == Chain::on ? sums_f16_kernel<true> : sums_f16_kernel<false>, (unsigned)blocks, SU_WARPS * 32, 0,
                   st, static_cast<const uint4 *>(h), Y, sender, row_ptr, species, slot_of, row_of, nnodes, elements, per,
                   out_v / SU_Y_SCALE, A);
  return check_launch("cmace_step(sums)");
}

// float64: four edges at a time on the float64 tensor instruction (m8n8k4), laid out as in sums_tf32_kernel: row g + 8 i of
// the sums, column g of tile j is k = 8 g + j.  With fma instructions a lane held two columns and all 16 rows, its edges
// went one after the other through eight loads of Y each: 262 us at 8 000 atoms and 23 us at 192, where the loads and the
// stores need 80 us at 8 000; now 179 and 10 us.
template <bool EARLY>
__global__ void __launch_bounds__(SU_WARPS * 32)
    sums_f64_kernel(const double *__restrict__ h, const double *__restrict__ Y, const int32_t *__restrict__ sender,
                const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ species,
                const int32_t *__restrict__ slot_of, const int32_t *__restrict__ row_of, int64_t nnodes, int elements,
                double *__restrict__ A) {
  __shared__ int32_t lists[SU_WARPS][SU_LIST], row_lists[SU_WARPS][64 + SU_LIST];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (!EARLY) grid_begin();
  if (pair >= nnodes * elements) {
    if (EARLY) grid_begin();
    return;
  }
  const bool soon = nnodes * elements <= kSoonWarps;
  const int64_t node = pair / elements;
  const int z = (int)(pair - node * elements);
  SenderElements from(sender, species, row_ptr[node], row_ptr[node + 1], lane);
  if (EARLY) {
    if (soon) from.look_up<true>();
    grid_begin();
    if (!soon) from.look_up();
  }
  SharedRows rows(row_of, row_lists[w], from);
  int32_t *list = lists[w];
  double acc[2][8][2];
#pragma unroll
  for (int j = 0; j < 8; j++) acc[0][j][0] = acc[0][j][1] = acc[1][j][0] = acc[1][j][1] = 0.0;
  if (!EARLY) from.look_up();
  rows.wait();
  for_edges_of_element(from, z, list, rows, [&](int n) {
    double2 hv[4];
    double yv[2];
    auto load = [&](int j0) {   // edge j0 + t; past the end: the last edge with Y = 0
      const int j = j0 + t;
      const int64_t e = list[j < n ? j : n - 1];
      const double2 *hp = reinterpret_cast<const double2 *>(h + rows[j < n ? j : n - 1] * ST_H + 8 * g);
#pragma unroll
      for (int u = 0; u < 4; u++) hv[u] = __ldg(hp + u);
      yv[0] = j < n ? __ldg(Y + e * 16 + g) : 0.0;
      yv[1] = j < n ? __ldg(Y + e * 16 + g + 8) : 0.0;
    };
    load(0);
    for (int j0 = 0; j0 < n; j0 += 4) {
      double b[8];
      const double y0 = yv[0], y1 = yv[1];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        b[2 * u] = hv[u].x;
        b[2 * u + 1] = hv[u].y;
      }
      if (j0 + 4 < n) load(j0 + 4);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        dmma(acc[0][j], y0, b[j]);
        dmma(acc[1][j], y1, b[j]);
      }
    }
  });
  const int width = elements * ST_H;
  double *o = A + (int64_t)slot_of[node] * 16 * width + z * ST_H + 16 * t;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    double *row = o + (int64_t)(g + 8 * i) * width;
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int j = 0; j < 2; j++)
        store32(row + 8 * u + 4 * j, acc[i][4 * j][u], acc[i][4 * j + 1][u], acc[i][4 * j + 2][u], acc[i][4 * j + 3][u]);
  }
}

template <typename T>
int StepKernels<T>::sums(const T *h, const T *Y, const int32_t *sender, const int32_t *row_ptr, const int32_t *species,
                         const int32_t *slot_of, const int32_t *row_of, int64_t nnodes, int elements, T *A, cudaStream_t st) {
  const int64_t blocks = (nnodes * elements + SU_WARPS - 1) / SU_WARPS;
  if (blocks > 0) {
    if constexpr (sizeof(T) == 4)
      launch_chained(sums_tf32_kernel, (unsigned)blocks, SU_WARPS * 32, 0, st, h, Y, sender, row_ptr, species, slot_of, nnodes,
                     elements, A);
    else
      launch_chained(chain_launches() == Chain::on ? sums_f64_kernel<true> : sums_f64_kernel<false>, (unsigned)blocks, SU_WARPS * 32,
                     0, st, h, Y, sender, row_ptr, species, slot_of, row_of, nnodes, elements, A);
  }
  return check_launch("cmace_step(sums)");
}

// ---- backward over the edges of a (receiver, element) pair, down to the gradient of the edge vector ---------------
// The warp holds P = grad A[i, :, z, :]; the 16 + 1 sums of an edge over k wait in shared memory until 32 edges (or the
// list's end) are there: then lane j turns edge j's numbers, plus the second layer's grad Y and dE/dr, into the
// gradient of its vector.
// lane j of the warp: edge list[j], its 16 + 1 sums in st[j * 17 ..], to the gradient of the edge's vector
template <typename T>
__device__ __forceinline__ void finish_edge(const T *st, int64_t e, const T *__restrict__ gY1, const T *__restrict__ dr1,
                                            const Quad<T> *__restrict__ geo, T *__restrict__ gvec, int shares = 1,
                                            int64_t nedges = 0) {
  T g[16];
  load_row16(gY1 + e * 16, g);
  for (int k = 1; k < shares; k++) {   // gY1 [shares, E, 16]
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const Quad<T> more = reinterpret_cast<const Quad<T> *>(gY1 + (k * nedges + e) * 16)[i];
      g[4 * i] += more.x, g[4 * i + 1] += more.y, g[4 * i + 2] += more.z, g[4 * i + 3] += more.w;
    }
  }
  // without an array of its own the second layer's dE/dr is component 0 of its grad Y (Y_00 is constant)
  const T dr = st[16] + (dr1 != nullptr ? dr1[e] : g[0]);
#pragma unroll
  for (int i = 0; i < 16; i++) g[i] += st[i];
  const Quad<T> q = geo[e];   // unit vector in the input's component order: harmonic axes are (z, x, y)
  T GX, GY, GZ;
  sph_l3_vjp<T>(q.z, q.x, q.y, g, GX, GY, GZ);
  store_quad(gvec + e * 4, GY * q.w + dr * q.x, GZ * q.w + dr * q.y, GX * q.w + dr * q.z);
}

// float32: eight edges at a time on the warp-level tensor instruction, D = P h^T and P h'^T.  P [16 x 64] stays in
// registers as A fragments (hi and lo); an edge's row is read as four 16-byte pieces per lane (lanes t of edge g cover
// 64 consecutive bytes each time), and the k order of the fragments follows: piece q holds k = 16 q + 4 t + 0 .. 3, its
// first two values are K step 2 q, the other two K step 2 q + 1.  No shuffles but for dE/dr (8 lanes hold its lm).
__global__ void __launch_bounds__(SU_WARPS * 32, 3)
    sums_bwd_tf32_kernel(const float *__restrict__ gA, const float *__restrict__ h, const float *__restrict__ dh,
                         const float *__restrict__ Y, const int32_t *__restrict__ sender,
                         const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ species,
                         const int32_t *__restrict__ slot_of, const float *__restrict__ gY1,
                         const float *__restrict__ dr1, const Quad<float> *__restrict__ geo, int64_t nnodes, int elements,
                         float *__restrict__ gvec) {
  grid_begin();
  __shared__ int32_t lists[SU_WARPS][SU_LIST];
  __shared__ float stage[SU_WARPS][32 * 17];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (pair >= nnodes * elements) return;
  const int64_t node = pair / elements;
  const int z = (int)(pair - node * elements);
  SenderElements from(sender, species, row_ptr[node], row_ptr[node + 1], lane);
  int32_t *list = lists[w];
  float *st = stage[w];
  uint32_t ph[8][4], pl[8][4];   // A fragments of the 8 K steps
  {
    const int b = z >> 1, width = sums_block_width(elements, b);
    const float *p = gA + (int64_t)b * nnodes * (16 * 128) + (int64_t)slot_of[node] * 16 * width + (z & 1) * ST_H + 4 * t;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float4 u = __ldg(reinterpret_cast<const float4 *>(p + g * width + 16 * q));
      const float4 v = __ldg(reinterpret_cast<const float4 *>(p + (g + 8) * width + 16 * q));
      split_tf32(u.x, ph[2 * q][0], pl[2 * q][0]);
      split_tf32(v.x, ph[2 * q][1], pl[2 * q][1]);
      split_tf32(u.y, ph[2 * q][2], pl[2 * q][2]);
      split_tf32(v.y, ph[2 * q][3], pl[2 * q][3]);
      split_tf32(u.z, ph[2 * q + 1][0], pl[2 * q + 1][0]);
      split_tf32(v.z, ph[2 * q + 1][1], pl[2 * q + 1][1]);
      split_tf32(u.w, ph[2 * q + 1][2], pl[2 * q + 1][2]);
      split_tf32(v.w, ph[2 * q + 1][3], pl[2 * q + 1][3]);
    }
  }
  from.look_up();
  OwnRows rows;
  for_edges_of_element(from, z, list, rows, [&](int n) {
    for (int j0 = 0; j0 < n; j0 += 32) {
      const int nj = n - j0 < 32 ? n - j0 : 32;
      if (lane < nj) {   // what finish_edge reads
        prefetch_l1(gY1 + (int64_t)list[j0 + lane] * 16);
        prefetch_l1(geo + list[j0 + lane]);
      }
      float4 hv[4], dv[4];
      auto load = [&](int j) {   // edge j0 + j + g, or the last one
        const int i = j0 + j + g;
        const int64_t e = list[i < n ? i : n - 1];
        const float4 *hp = reinterpret_cast<const float4 *>(h + e * ST_H + 4 * t);
        const float4 *dp = reinterpret_cast<const float4 *>(dh + e * ST_H + 4 * t);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          hv[q] = __ldg(hp + 4 * q);
          dv[q] = __ldg(dp + 4 * q);
        }
      };
      load(0);
      for (int j = 0; j < nj; j += 8) {
        float ch[4] = {0.f, 0.f, 0.f, 0.f}, cd[4] = {0.f, 0.f, 0.f, 0.f};
        const int i0 = j0 + j + 2 * t;   // this lane's result columns: edges 2 t and 2 t + 1 of the eight
        const int64_t e0 = list[i0 < n ? i0 : n - 1], e1 = list[i0 + 1 < n ? i0 + 1 : n - 1];
        const float y00 = __ldg(Y + e0 * 16 + g), y01 = __ldg(Y + e0 * 16 + g + 8);
        const float y10 = __ldg(Y + e1 * 16 + g), y11 = __ldg(Y + e1 * 16 + g + 8);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          uint32_t h0, l0, h1, l1, g0, m0, g1, m1;
          split_tf32(hv[q].x, h0, l0);
          split_tf32(hv[q].y, h1, l1);
          split_tf32(dv[q].x, g0, m0);
          split_tf32(dv[q].y, g1, m1);
          mma_tf32(ch, ph[2 * q], h0, h1);
          mma_tf32(cd, ph[2 * q], g0, g1);
          mma_tf32(ch, ph[2 * q], l0, l1);
          mma_tf32(cd, ph[2 * q], m0, m1);
          mma_tf32(ch, pl[2 * q], h0, h1);
          mma_tf32(cd, pl[2 * q], g0, g1);
          split_tf32(hv[q].z, h0, l0);
          split_tf32(hv[q].w, h1, l1);
          split_tf32(dv[q].z, g0, m0);
          split_tf32(dv[q].w, g1, m1);
          mma_tf32(ch, ph[2 * q + 1], h0, h1);
          mma_tf32(cd, ph[2 * q + 1], g0, g1);
          mma_tf32(ch, ph[2 * q + 1], l0, l1);
          mma_tf32(cd, ph[2 * q + 1], m0, m1);
          mma_tf32(ch, pl[2 * q + 1], h0, h1);
          mma_tf32(cd, pl[2 * q + 1], g0, g1);
        }
        if (j + 8 < nj) load(j + 8);
        float *s0 = st + (j + 2 * t) * 17, *s1 = s0 + 17;
        s0[g] = ch[0];
        s1[g] = ch[1];
        s0[g + 8] = ch[2];
        s1[g + 8] = ch[3];
        float r0 = fmaf(y00, cd[0], y01 * cd[2]), r1 = fmaf(y10, cd[1], y11 * cd[3]);
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
          r0 += __shfl_xor_sync(0xffffffffu, r0, off);
          r1 += __shfl_xor_sync(0xffffffffu, r1, off);
        }
        if (g == 0) {
          s0[16] = r0;
          s1[16] = r1;
        }
      }
      __syncwarp();
      if (lane < nj) finish_edge<float>(st + lane * 17, list[j0 + lane], gY1, dr1, geo, gvec);
      __syncwarp();
    }
  });
}

// The same with h and h' as fp16 hi / lo rows.  P is scaled by the power of two that puts its largest entry of the
// pair just below 2^14 (its magnitude is the caller's gradient's), so its split loses nothing either.  A lane reads
// pieces t and t + 4 of an edge's 128-byte hi or lo row: piece i holds k = 8 (t + 4 i) .. + 7 of K steps 2 i and 2 i + 1.
template <bool EARLY>
__global__ void __launch_bounds__(SU_WARPS * 32, 4)
    sums_bwd_f16_kernel(const float *__restrict__ gA, const uint4 *__restrict__ h, const uint4 *__restrict__ dh,
                        const float *__restrict__ Y, const int32_t *__restrict__ sender,
                        const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ species,
                        const int32_t *__restrict__ slot_of, const int32_t *__restrict__ row_of, const float *__restrict__ gY1,
                        const float *__restrict__ dr1, const Quad<float> *__restrict__ geo, int64_t nnodes, int elements, int per,
                        float out_v, float out_t, float *__restrict__ gvec) {
  __shared__ int32_t lists[SU_WARPS][SU_LIST], row_lists[SU_WARPS][64 + SU_LIST];
  __shared__ float stage[SU_WARPS][32 * 17];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (!EARLY) grid_begin();
  const int chunks = (elements + per - 1) / per;
  if (pair >= nnodes * chunks) {
    if (EARLY) grid_begin();
    return;
  }
  const bool soon = nnodes * chunks <= kSoonWarps;
  const int64_t node = pair / chunks;
  const int z0 = (int)(pair - node * chunks) * per, z1 = z0 + per < elements ? z0 + per : elements;
  SenderElements from(sender, species, row_ptr[node], row_ptr[node + 1], lane);
  SharedRows rows(row_of, row_lists[w], from, EARLY);
  if (EARLY) {
    if (soon) from.look_up<true>();
    grid_begin();
    if (!soon) from.look_up();
  }   // only the gradients of the sums are the kernel before's
  int32_t *list = lists[w];
  float *st = stage[w];
#pragma unroll 1
  for (int z = z0; z < z1; z++) {
    __syncwarp();   // the list of the element before has been read
    float sv, stt;
    uint32_t ph[4][4], pl[4][4];   // A fragments of the 4 K steps
    {
      const int b = z >> 1, width = sums_block_width(elements, b);
      const float *p = gA + (int64_t)b * nnodes * (16 * 128) + (int64_t)slot_of[node] * 16 * width + (z & 1) * ST_H + 8 * t;
      float4 v[2][2][2];   // [piece][row g, g + 8][half of the piece]
      float most = 0.f;
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int r = 0; r < 2; r++) load32(p + (g + 8 * r) * width + 32 * i, v[i][r][0], v[i][r][1]);
      if (z + 1 < z1) {   // the next element's gradients on their way to L1: lane's half of a row of 64
        const int nb = (z + 1) >> 1, nw = sums_block_width(elements, nb);
        const float *block = gA + (int64_t)nb * nnodes * (16 * 128) + (int64_t)slot_of[node] * 16 * nw;
        prefetch_l1(block + (lane >> 1) * nw + ((z + 1) & 1) * ST_H + 32 * (lane & 1));
      }
      if (!EARLY && z == z0) from.look_up();
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
          for (int u = 0; u < 2; u++) {
            most = fmaxf(most, fmaxf(fmaxf(fabsf(v[i][r][u].x), fabsf(v[i][r][u].y)), fmaxf(fabsf(v[i][r][u].z), fabsf(v[i][r][u].w))));
          }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, off));
      int ex = 127 + 13 - ((int)((__float_as_uint(most) >> 23) & 255u) - 127);   // biased exponent of the scale
      ex = ex < 1 ? 1 : (ex > 253 ? 253 : ex);
      const float sc = __uint_as_float((uint32_t)ex << 23), inv = __uint_as_float((uint32_t)(254 - ex) << 23);
      const unsigned long long sc2 = pack2(sc, sc);
      sv = out_v * inv;
      stt = out_t * inv;
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
          for (int r = 0; r < 2; r++) {
            split_half2(mul2(pack2(v[i][r][u].x, v[i][r][u].y), sc2), ph[2 * i + u][r], pl[2 * i + u][r]);
            split_half2(mul2(pack2(v[i][r][u].z, v[i][r][u].w), sc2), ph[2 * i + u][2 + r], pl[2 * i + u][2 + r]);
          }
    }
    if (z == z0) rows.wait();
    for_edges_of_element(from, z, list, rows, [&](int n) {
      for (int j0 = 0; j0 < n; j0 += 32) {
        const int nj = n - j0 < 32 ? n - j0 : 32;
        if (lane < nj) {   // what finish_edge reads
          prefetch_l1(gY1 + (int64_t)list[j0 + lane] * 16);
          prefetch_l1(geo + list[j0 + lane]);
        }
        uint4 hh[2], hl[2], dd[2], dl[2];
        auto load = [&](int j) {   // edge j0 + j + g, or the last one
          const int i = j0 + j + g;
          const int64_t e = rows[i < n ? i : n - 1];
#pragma unroll
          for (int q = 0; q < 2; q++) {
            hh[q] = __ldg(h + e * 16 + t + 4 * q);
            hl[q] = __ldg(h + e * 16 + 8 + t + 4 * q);
            dd[q] = __ldg(dh + e * 16 + t + 4 * q);
            dl[q] = __ldg(dh + e * 16 + 8 + t + 4 * q);
          }
        };
        load(0);
        for (int j = 0; j < nj; j += 8) {
          float ch[4] = {0.f, 0.f, 0.f, 0.f}, cd[4] = {0.f, 0.f, 0.f, 0.f};
          const int i0 = j0 + j + 2 * t;   // this lane's result columns: edges 2 t and 2 t + 1 of the eight
          const int64_t e0 = list[i0 < n ? i0 : n - 1], e1 = list[i0 + 1 < n ? i0 + 1 : n - 1];
          const float y00 = __ldg(Y + e0 * 16 + g), y01 = __ldg(Y + e0 * 16 + g + 8);
          const float y10 = __ldg(Y + e1 * 16 + g), y11 = __ldg(Y + e1 * 16 + g + 8);
#pragma unroll
          for (int q = 0; q < 2; q++) {
            mma_f16(ch, ph[2 * q], hh[q].x, hh[q].y);
            mma_f16(cd, ph[2 * q], dd[q].x, dd[q].y);
            mma_f16(ch, ph[2 * q], hl[q].x, hl[q].y);
            mma_f16(cd, ph[2 * q], dl[q].x, dl[q].y);
            mma_f16(ch, pl[2 * q], hh[q].x, hh[q].y);
            mma_f16(cd, pl[2 * q], dd[q].x, dd[q].y);
            mma_f16(ch, ph[2 * q + 1], hh[q].z, hh[q].w);
            mma_f16(cd, ph[2 * q + 1], dd[q].z, dd[q].w);
            mma_f16(ch, ph[2 * q + 1], hl[q].z, hl[q].w);
            mma_f16(cd, ph[2 * q + 1], dl[q].z, dl[q].w);
            mma_f16(ch, pl[2 * q + 1], hh[q].z, hh[q].w);
            mma_f16(cd, pl[2 * q + 1], dd[q].z, dd[q].w);
          }
          if (j + 8 < nj) load(j + 8);
          float *s0 = st + (j + 2 * t) * 17, *s1 = s0 + 17;
          s0[g] = ch[0] * sv;
          s1[g] = ch[1] * sv;
          s0[g + 8] = ch[2] * sv;
          s1[g + 8] = ch[3] * sv;
          float r0 = fmaf(y00, cd[0], y01 * cd[2]), r1 = fmaf(y10, cd[1], y11 * cd[3]);
#pragma unroll
          for (int off = 4; off < 32; off <<= 1) {
            r0 += __shfl_xor_sync(0xffffffffu, r0, off);
            r1 += __shfl_xor_sync(0xffffffffu, r1, off);
          }
          if (g == 0) {
            s0[16] = r0 * stt;
            s1[16] = r1 * stt;
          }
        }
        __syncwarp();
        if (lane < nj) finish_edge<float>(st + lane * 17, list[j0 + lane], gY1, dr1, geo, gvec);
        __syncwarp();
      }
    });
  }
}

int step_sums_bwd_half(const float *gA, const void *h, const void *dh, const float *Y, const int32_t *sender,
                       const int32_t *row_ptr, const int32_t *species, const int32_t *slot_of, const int32_t *row_of, const float *gY1,
                       const float *dr1, const Quad<float> *geo, int64_t nnodes, int elements, float out_v, float out_t,
                       float *gvec, cudaStream_t st) {
  const int per = elements_per_warp(nnodes, elements);
  const int64_t blocks = (nnodes * ((elements + per - 1) / per) + SU_WARPS - 1) / SU_WARPS;
  if (blocks > 0)
    launch_chained(chain_launches() == Chain::on ? sums_bwd_f16_kernel<true> : sums_bwd_f16_kernel<false>, (unsigned)blocks,
                   SU_WARPS * 32, 0, st, gA, static_cast<const uint4 *>(h), static_cast<const uint4 *>(dh), Y, sender, row_ptr, species,
                   slot_of, row_of, gY1, dr1, geo, nnodes, elements, per, out_v, out_t, gvec);
  return check_launch("cmace_step(sums_back)");
}

// float64: eight edges at a time on the float64 tensor instruction, D = P h^T and P h'^T.  P's A fragments stay in
// registers; K step s of lane (g, t) is k = 16 t + s, so that a lane reads 16 consecutive values of its edge's row (and of
// P's rows g and g + 8).  With fma instructions an edge cost 21 shuffles of two words and eight loads of Y: 404 us at
// 8 000 atoms, 37 us at 192, where its bytes need 115 us at 8 000; now 261 and 20 us.
template <bool EARLY>
__global__ void __launch_bounds__(SU_WARPS * 32, 3)
    sums_bwd_f64_kernel(const double *__restrict__ gA, const double *__restrict__ h, const double *__restrict__ dh,
                    const double *__restrict__ Y, const int32_t *__restrict__ sender, const int32_t *__restrict__ row_ptr,
                    const int32_t *__restrict__ species, const int32_t *__restrict__ slot_of,
                    const int32_t *__restrict__ row_of, const double *__restrict__ gY1, int shares,
                    const Quad<double> *__restrict__ geo, int64_t nnodes, int64_t nedges, int elements,
                    double *__restrict__ gvec) {
  __shared__ int32_t lists[SU_WARPS][SU_LIST], row_lists[SU_WARPS][64 + SU_LIST];
  __shared__ double stage[SU_WARPS][32 * 17];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int64_t pair = (int64_t)blockIdx.x * SU_WARPS + w;
  if (!EARLY) grid_begin();
  if (pair >= nnodes * elements) {
    if (EARLY) grid_begin();
    return;
  }
  const int64_t node = pair / elements;
  const int z = (int)(pair - node * elements);
  SenderElements from(sender, species, row_ptr[node], row_ptr[node + 1], lane);
  SharedRows rows(row_of, row_lists[w], from, EARLY);
  if (EARLY) grid_begin();   // only the gradients of the sums are the kernel before's
  int32_t *list = lists[w];
  double *st = stage[w];
  double2 P[2][8];
  {
    const int b = z >> 1, width = sums_block_width(elements, b);
    const double *p = gA + (int64_t)b * nnodes * (16 * 128) + (int64_t)slot_of[node] * 16 * width + (z & 1) * ST_H + 16 * t;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int q = 0; q < 8; q++) P[i][q] = __ldg(reinterpret_cast<const double2 *>(p + (g + 8 * i) * width) + q);
  }
  from.look_up();
  rows.wait();
  for_edges_of_element(from, z, list, rows, [&](int n) {
    for (int j0 = 0; j0 < n; j0 += 32) {
      const int nj = n - j0 < 32 ? n - j0 : 32;
      if (lane < nj) {   // what finish_edge reads
        for (int k = 0; k < shares; k++) prefetch_l1(gY1 + (k * nedges + list[j0 + lane]) * 16);
        prefetch_l1(geo + list[j0 + lane]);
      }
      for (int j = 0; j < nj; j += 8) {
        const int i = j0 + j + g;   // this lane's row of h: that edge, or the last one
        const int64_t e = rows[i < n ? i : n - 1];
        const double2 *hp = reinterpret_cast<const double2 *>(h + e * ST_H + 16 * t);
        const double2 *dp = reinterpret_cast<const double2 *>(dh + e * ST_H + 16 * t);
        double2 hv[8], dv[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
          hv[q] = __ldg(hp + q);
          dv[q] = __ldg(dp + q);
        }
        const int i0 = j0 + j + 2 * t;   // its result columns: edges 2 t and 2 t + 1 of the eight
        const int64_t e0 = list[i0 < n ? i0 : n - 1], e1 = list[i0 + 1 < n ? i0 + 1 : n - 1];
        const double y00 = __ldg(Y + e0 * 16 + g), y01 = __ldg(Y + e0 * 16 + g + 8);
        const double y10 = __ldg(Y + e1 * 16 + g), y11 = __ldg(Y + e1 * 16 + g + 8);
        double ch[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, cd[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
        for (int q = 0; q < 8; q++) {
          dmma(ch[0], P[0][q].x, hv[q].x);
          dmma(ch[1], P[1][q].x, hv[q].x);
          dmma(cd[0], P[0][q].x, dv[q].x);
          dmma(cd[1], P[1][q].x, dv[q].x);
          dmma(ch[0], P[0][q].y, hv[q].y);
          dmma(ch[1], P[1][q].y, hv[q].y);
          dmma(cd[0], P[0][q].y, dv[q].y);
          dmma(cd[1], P[1][q].y, dv[q].y);
        }
        double *s0 = st + (j + 2 * t) * 17, *s1 = s0 + 17;
        s0[g] = ch[0][0];
        s1[g] = ch[0][1];
        s0[g + 8] = ch[1][0];
        s1[g + 8] = ch[1][1];
        double r0 = fma(y00, cd[0][0], y01 * cd[1][0]), r1 = fma(y10, cd[0][1], y11 * cd[1][1]);
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
          r0 += __shfl_xor_sync(0xffffffffu, r0, off);
          r1 += __shfl_xor_sync(0xffffffffu, r1, off);
        }
        if (g == 0) {
          s0[16] = r0;
          s1[16] = r1;
        }
      }
      __syncwarp();
      if (lane < nj) finish_edge<double>(st + lane * 17, list[j0 + lane], gY1, nullptr, geo, gvec, shares, nedges);
      __syncwarp();
    }
  });
}

template <typename T>
int StepKernels<T>::sums_bwd(const T *gA, const T *h, const T *dh, const T *Y, const int32_t *sender,
                             const int32_t *row_ptr, const int32_t *species, const int32_t *slot_of, const int32_t *row_of,
                             const T *gY1, int shares, const T *dr1, const Quad<T> *geo, int64_t nnodes, int64_t nedges, int elements,
                             T *gvec, cudaStream_t st) {
  const int64_t blocks = (nnodes * elements + SU_WARPS - 1) / SU_WARPS;
  if (blocks > 0) {
    if constexpr (sizeof(T) == 4)
      launch_chained(sums_bwd_tf32_kernel, (unsigned)blocks, SU_WARPS * 32, 0, st, gA, h, dh, Y, sender, row_ptr, species, slot_of,
                                                                      gY1, dr1, geo, nnodes, elements, gvec);
    else
      launch_chained(chain_launches() == Chain::on ? sums_bwd_f64_kernel<true> : sums_bwd_f64_kernel<false>, (unsigned)blocks,
                     SU_WARPS * 32, 0, st, gA, h, dh, Y, sender, row_ptr, species, slot_of, row_of, gY1, shares, geo, nnodes, nedges,
                     elements, gvec);
  }
  return check_launch("cmace_step(sums_bwd)");
}

// ---- tabulated radial weights ---------------------------------------------------------------------------------------
// gradient of every edge's vector from both layers' grad Y and dE/dr, each in `shares` arrays to be added up
template <typename T>
__global__ void __launch_bounds__(256)
    edge_finish_kernel(const T *__restrict__ gY0, const T *__restrict__ dr0, const T *__restrict__ gY1,
                       const T *__restrict__ dr1, const Quad<T> *__restrict__ geo, int64_t nedges, int shares, T *__restrict__ gvec) {
  grid_begin();
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= nedges) return;
  T s[17];
#pragma unroll
  for (int i = 0; i < 17; i++) s[i] = T(0);
  for (int k = 0; k < shares; k++) {
    for (int layer = 0; layer < (k == 0 ? 1 : 2); layer++) {   // finish_edge adds the second layer's first share
      const Quad<T> *g = reinterpret_cast<const Quad<T> *>((layer == 0 ? gY0 : gY1) + (k * nedges + e) * 16);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const Quad<T> q = g[i];
        s[4 * i] += q.x;
        s[4 * i + 1] += q.y;
        s[4 * i + 2] += q.z;
        s[4 * i + 3] += q.w;
      }
      s[16] += (layer == 0 ? dr0 : dr1)[k * nedges + e];
    }
  }
  finish_edge<T>(s, e, gY1, dr1, geo, gvec);
}
template <typename T>
int step_edge_finish(const T *gY0, const T *dr0, const T *gY1, const T *dr1, const Quad<T> *geo, int64_t nedges, int shares,
                     T *gvec, cudaStream_t st) {
  if (nedges > 0)
    launch_chained(edge_finish_kernel<T>, (unsigned)((nedges + 255) / 256), 256, 0, st, gY0, dr0, gY1, dr1, geo, nedges, shares, gvec);
  return check_launch("cmace_step(sums_back)");
}
template int step_edge_finish<float>(const float *, const float *, const float *, const float *, const Quad<float> *, int64_t,
                                     int, float *, cudaStream_t);
template int step_edge_finish<double>(const double *, const double *, const double *, const double *, const Quad<double> *,
                                      int64_t, int, double *, cudaStream_t);

// ---- forces and energies ------------------------------------------------------------------------------------------
// One warp per atom sums its edges' gradients from both groupings (float64, fixed order, no atomics); block 0 adds up
// the energies meanwhile: sums[0] over node_energy, sums[1] over the interaction energies.
template <typename T>
__global__ void __launch_bounds__(256)
    forces_kernel(const T *__restrict__ g, const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ perm,
                  const int32_t *__restrict__ send_ptr, int64_t nrecv, int64_t nsend, double sign,
                  double *__restrict__ out, const int32_t *__restrict__ species_in, int elements,
                  double *__restrict__ inter, double *__restrict__ node_energy, const int32_t *status, const int *stalled,
                  double *__restrict__ sums) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.x == 0) {
    grid_begin();
    __shared__ double part[2][8];
    double a = 0.0, b = 0.0;
    if (species_in && status && *status != 0)   // this call's edge_prep, or one before it, met an index that does not exist
      for (int64_t i = threadIdx.x; i < nrecv; i += 256)
        if (species_in[i] < 0 || species_in[i] >= elements) inter[i] = node_energy[i] = CUDART_NAN;
#pragma unroll 8   // one block: the loads in flight bound it
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
    // non-zero when a bounded wait of this step gave up: the caller reads it with the energies
    if (threadIdx.x == 2) sums[2] = (double)((status ? *status : 0) | (stalled ? *stalled : 0));
    return;
  }
  const int64_t n = (int64_t)(blockIdx.x - 1) * 8 + w;
  if (n >= nsend) {
    grid_begin();
    return;
  }
  double ax = 0.0, ay = 0.0, az = 0.0;
  const Quad<T> *gq = reinterpret_cast<const Quad<T> *>(g);
  const bool receives = n < nrecv;
  const int64_t k0 = send_ptr[n], k1 = send_ptr[n + 1];
  const int64_t r0 = receives ? row_ptr[n] : 0, r1 = receives ? row_ptr[n + 1] : 0;
  if (k0 + 32 * lane < k1) prefetch_l1(perm + k0 + 32 * lane);
  grid_begin();
  // 64 edges of either grouping at a time: the indices of the one are on their way with the gradients of the other
  for (int64_t b = 0; b < k1 - k0 || b < r1 - r0; b += 64) {
    int32_t e[2];
    Quad<T> in[2], out_q[2];
    bool has[2], had[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      has[u] = k0 + b + 32 * u + lane < k1;
      had[u] = r0 + b + 32 * u + lane < r1;
      if (has[u]) e[u] = perm[k0 + b + 32 * u + lane];
      if (had[u]) in[u] = gq[r0 + b + 32 * u + lane];
    }
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (has[u]) out_q[u] = gq[e[u]];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (has[u]) ax += (double)out_q[u].x, ay += (double)out_q[u].y, az += (double)out_q[u].z;
      if (had[u]) ax -= (double)in[u].x, ay -= (double)in[u].y, az -= (double)in[u].z;
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
                           int64_t nrecv, int64_t nsend, double sign, double *out, const int32_t *species_in,
                           int elements, double *inter, double *node_energy, const int32_t *status, const int *stalled,
                           double *sums, cudaStream_t st) {
  const int64_t blocks = 1 + (nsend + 7) / 8;
  launch_chained(forces_kernel<T>, (unsigned)blocks, 256, 0, st, gvec, row_ptr, perm, send_ptr, nrecv, nsend, sign, out,
                 species_in, elements, inter, node_energy, status, stalled, sums);
  return check_launch("cmace_step(forces)");
}

#define CMACE_STEP_EDGES(T)                                                                                         \
  template int StepKernels<T>::edge_prep(const double *, const int32_t *, const int32_t *, const double *,          \
                                         const uint8_t *, const double *, int64_t, int32_t *, int64_t, double, int, \
                                         int, const SplineTable<T> &, Quad<T> *, T *, T *, const int32_t *,         \
                                         const void *, int,                                                         \
                                         int64_t, int64_t, int, int32_t *, int32_t *, int32_t *, int32_t *,         \
                                         int32_t *, int32_t *, const int32_t *, const EdgeRows &, cudaStream_t);    \
  template int StepKernels<T>::sums(const T *, const T *, const int32_t *, const int32_t *, const int32_t *,        \
                                    const int32_t *, const int32_t *, int64_t, int, T *, cudaStream_t);             \
  template int StepKernels<T>::sums_bwd(const T *, const T *, const T *, const T *, const int32_t *,                \
                                        const int32_t *, const int32_t *, const int32_t *, const int32_t *,         \
                                        const T *, int, const T *, const Quad<T> *, int64_t, int64_t, int, T *,     \
                                        cudaStream_t);                                                              \
  template int StepKernels<T>::forces(const T *, const int32_t *, const int32_t *, const int32_t *, int64_t,        \
                                      int64_t, double, double *, const int32_t *, int, double *, double *,          \
                                      const int32_t *, const int *, double *, cudaStream_t);
CMACE_STEP_EDGES(float)
CMACE_STEP_EDGES(double)

}  // namespace cmace
