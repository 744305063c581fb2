// Neighbour list on the device for an orthorhombic cell (the step before the hot path: upstream builds it on the
// host with matscipy / ASE, tests/test_utils.py:97-105 of the reference).  Full list (both directions), receivers =
// the first nrecv atoms, sorted by receiver, i.e. directly the layout InvariantMessagePassing wants:
//
//   edge e:  vector = pos[sender[e]] - pos[receiver[e]] + shift[e],  |vector| < r_cut
//
// Cell list: atoms are binned into cells of at least r_cut per side (cmace_nl_cell_ids_f64), grouped by cell with
// the same radix-sort routine that groups edges by sender (cmace_sender_order with keys = cell ids), then one
// warp per receiver walks the 27 surrounding cells, 32 candidates at a time, once to count and once to fill
// (ballot + prefix inside the warp, so the edges of a receiver come out in a fixed order and nothing is atomic).
// Periodic axes wrap with a lattice shift; a box of one or two cells per periodic axis still works because each of
// the 27 (cell, shift) pairs is distinct as long as the box is at least r_cut long.  Distances are formed with
// the same operations and in the same order as the host list (no fused multiply-add), so both make the same
// decision for every pair.
#include <cub/device/device_scan.cuh>

#include "common.cuh"

namespace cmace {

struct NlGeom {
  double lo[3], len[3], cell[3], rc2;
  int ncell[3], pbc[3];
};

static int make_geom(NlGeom &g, double lox, double loy, double loz, double lx, double ly, double lz, int pbc_mask,
                     double r_cut, const char *what) {
  const double lo[3] = {lox, loy, loz}, len[3] = {lx, ly, lz};
  if (!(r_cut > 0.0)) return fail(CMACE_ERR_ARG, "%s: r_cut must be positive", what);
  for (int d = 0; d < 3; d++) {
    if (!(len[d] > 0.0)) return fail(CMACE_ERR_ARG, "%s: box lengths must be positive", what);
    g.lo[d] = lo[d];
    g.len[d] = len[d];
    g.pbc[d] = (pbc_mask >> d) & 1;
    int64_t n = (int64_t)(len[d] / r_cut);
    if (n < 1) {
      if (g.pbc[d])
        return fail(CMACE_ERR_UNSUPPORTED, "%s: a periodic axis shorter than r_cut needs more than one image", what);
      n = 1;
    }
    if (n > 1024) n = 1024;
    g.ncell[d] = (int)n;
    g.cell[d] = len[d] / (double)n;
  }
  g.rc2 = r_cut * r_cut;
  return CMACE_OK;
}

// wrapped coordinate, cell index and number of lattice translations removed, along axis d
__device__ __forceinline__ void locate(const NlGeom &g, int d, double x, double &xw, int &c, int &w) {
  w = 0;
  xw = x;
  const double t = x - g.lo[d];
  if (g.pbc[d] && !(t >= 0.0 && t < g.len[d])) {   // inside, the quotient rounds below one: no division needed
    w = (int)floor(t / g.len[d]);
    if (w != 0) xw = x - (double)w * g.len[d];
  }
  int ci = (int)floor((xw - g.lo[d]) / g.cell[d]);
  c = ci < 0 ? 0 : (ci >= g.ncell[d] ? g.ncell[d] - 1 : ci);
}

__global__ void nl_cell_ids_kernel(const double *__restrict__ pos, int64_t natoms, const NlGeom g,
                                   int32_t *__restrict__ cell_id) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natoms) return;
  int c[3], w;
  double xw;
  for (int d = 0; d < 3; d++) locate(g, d, pos[3 * i + d], xw, c[d], w);
  cell_id[i] = (c[0] * g.ncell[1] + c[1]) * g.ncell[2] + c[2];
}

// An atom as the walk reads it: wrapped coordinates in cell order, so that a warp's candidates are consecutive and the
// divisions of locate() are done once per atom instead of once per candidate.
struct alignas(16) NlAtom {
  double x, y, z;
  int id, wrapped;   // wrapped: the atom lies outside the box (its lattice translations are recomputed for its edges)
};

__device__ __forceinline__ NlAtom nl_atom(const double *__restrict__ pos, const NlGeom &g, int id) {
  NlAtom a;
  int c, w, any = 0;
  locate(g, 0, pos[3 * (int64_t)id], a.x, c, w);
  any |= w;
  locate(g, 1, pos[3 * (int64_t)id + 1], a.y, c, w);
  any |= w;
  locate(g, 2, pos[3 * (int64_t)id + 2], a.z, c, w);
  any |= w;
  a.id = id;
  a.wrapped = any != 0;
  return a;
}

__global__ void __launch_bounds__(256)
    nl_atoms_kernel(const double *__restrict__ pos, int64_t natoms, const NlGeom g, const int32_t *__restrict__ perm,
                    NlAtom *__restrict__ atoms) {
  const int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (k < natoms) atoms[k] = nl_atom(pos, g, perm[k]);
}

// Binning of a small system in one block: counts, prefix sums and the atoms of every cell in index order (an atom counts
// the smaller indices of its cell: the order of atomics must not show in the edge list).  Bound by the latency of its
// phases; the grouping by radix sort that larger systems take costs five launches.
constexpr int NL_SMALL_ATOMS = 8192, NL_SMALL_CELLS = 8192, NL_SMALL_THREADS = 1024;
constexpr int NL_SMALL_SMEM = (NL_SMALL_ATOMS + NL_SMALL_CELLS + 33) * 4 + NL_SMALL_ATOMS * 2;

// exclusive prefix over count[0 .. n) in shared memory, in place, by the whole block; returns the total
__device__ int block_exclusive_scan(int32_t *count, int n, int32_t *warp_sums) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, per = (n + NL_SMALL_THREADS - 1) / NL_SMALL_THREADS;
  const int lo = tid * per < n ? tid * per : n, hi = lo + per < n ? lo + per : n;
  int mine = 0;
  for (int i = lo; i < hi; i++) mine += count[i];
  int inc = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += o;
  }
  if (lane == 31) warp_sums[w] = inc;
  __syncthreads();
  if (w == 0) {
    int v = warp_sums[lane], t = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, t, off);
      if (lane >= off) t += o;
    }
    warp_sums[lane] = t - v;
    if (lane == 31) warp_sums[32] = t;
  }
  __syncthreads();
  int run = warp_sums[w] + inc - mine;
  for (int i = lo; i < hi; i++) {
    const int c = count[i];
    count[i] = run;
    run += c;
  }
  __syncthreads();
  return warp_sums[32];
}

__global__ void __launch_bounds__(NL_SMALL_THREADS)
    nl_bin_small_kernel(const double *__restrict__ pos, int natoms, int ncells, const NlGeom g,
                        int32_t *__restrict__ cell_ptr, NlAtom *__restrict__ atoms) {
  extern __shared__ int32_t nl_smem[];
  int32_t *ids = nl_smem, *count = nl_smem + NL_SMALL_ATOMS, *sums = count + NL_SMALL_CELLS;
  uint16_t *cells = reinterpret_cast<uint16_t *>(sums + 33);
  const int tid = threadIdx.x;
  for (int c = tid; c < ncells; c += NL_SMALL_THREADS) count[c] = 0;
  __syncthreads();
  for (int i = tid; i < natoms; i += NL_SMALL_THREADS) {
    int c[3], w;
    double xw;
    for (int d = 0; d < 3; d++) locate(g, d, pos[3 * (int64_t)i + d], xw, c[d], w);
    const int cell = (c[0] * g.ncell[1] + c[1]) * g.ncell[2] + c[2];
    cells[i] = (uint16_t)cell;
    atomicAdd(&count[cell], 1);
  }
  __syncthreads();
  block_exclusive_scan(count, ncells, sums);
  for (int c = tid; c <= ncells; c += NL_SMALL_THREADS) cell_ptr[c] = c < ncells ? count[c] : natoms;
  __syncthreads();
  for (int i = tid; i < natoms; i += NL_SMALL_THREADS) ids[atomicAdd(&count[cells[i]], 1)] = i;   // count: the cell's end now
  __syncthreads();
  for (int i = tid; i < natoms; i += NL_SMALL_THREADS) {
    const int c = cells[i], lo = c == 0 ? 0 : count[c - 1], hi = count[c];
    int k = lo;
#pragma unroll 4
    for (int a = lo; a < hi; a++) k += ids[a] < i;
    atoms[k] = nl_atom(pos, g, i);
  }
}

// exclusive prefix of up to a few ten thousand counts in one block, in place (n values, the last one becomes the total)
__global__ void __launch_bounds__(NL_SMALL_THREADS) nl_scan_small_kernel(int32_t *__restrict__ v, int n) {
  extern __shared__ int32_t nl_smem[];
  int32_t *sums = nl_smem + n;
  for (int i = threadIdx.x; i < n; i += NL_SMALL_THREADS) nl_smem[i] = v[i];
  __syncthreads();
  block_exclusive_scan(nl_smem, n, sums);
  for (int i = threadIdx.x; i < n; i += NL_SMALL_THREADS) v[i] = nl_smem[i];
}

// One warp per receiver.  FILL = false: count[i] = number of neighbours; FILL = true: writes them at row_ptr[i].  Lane c
// looks up the range of cell c of the 27; the ranges are then walked as one sequence, four candidates a lane at a time:
// the walk is bound by the latency of its dependent loads, and 27 short loops had one load in flight each (17 and 20 us
// at 3 000 receivers).  atoms: in cell order, or null with perm (the caller's own sequence of calls).
constexpr int NL_AHEAD = 4;

template <bool FILL>
__global__ void __launch_bounds__(128)
    nl_walk_kernel(const double *__restrict__ pos, int64_t nrecv, const NlGeom g, const NlAtom *__restrict__ atoms,
                   const int32_t *__restrict__ perm, const int32_t *__restrict__ cell_ptr, int32_t *__restrict__ count,
                   const int32_t *__restrict__ row_ptr, int32_t *__restrict__ sender, int32_t *__restrict__ receiver,
                   int8_t *__restrict__ shift_idx, double *__restrict__ shifts) {
  __shared__ int32_t first[4][28], base[4][28];   // position of a cell's first candidate in the sequence; its place in atoms
  __shared__ int8_t image[4][28][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 4 + w;
  if (i >= nrecv) return;
  double xi[3];
  int ci[3], wi[3];
  for (int d = 0; d < 3; d++) locate(g, d, pos[3 * i + d], xi[d], ci[d], wi[d]);
  int k0 = 0, length = 0;
  if (lane < 27) {
    const int dd[3] = {lane / 9 - 1, lane / 3 % 3 - 1, lane % 3 - 1};
    int c[3];
    bool skip = false;
    for (int d = 0; d < 3; d++) {
      int cc = ci[d] + dd[d], S = 0;
      if (cc < 0 || cc >= g.ncell[d]) {
        if (!g.pbc[d]) {
          skip = true;
          cc = ci[d];
        } else {
          S = cc < 0 ? -1 : 1;
          cc -= S * g.ncell[d];
        }
      }
      c[d] = cc;
      image[w][lane][d] = (int8_t)S;
    }
    const int cf = (c[0] * g.ncell[1] + c[1]) * g.ncell[2] + c[2];
    k0 = cell_ptr[cf];
    length = skip ? 0 : cell_ptr[cf + 1] - k0;
  }
  int inc = length;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += o;
  }
  if (lane < 28) {   // lane 27: the end of the sequence
    first[w][lane] = inc - length;
    base[w][lane] = k0;
  }
  __syncwarp();
  const int all = __shfl_sync(0xffffffffu, inc, 31);
  int64_t out = FILL ? (int64_t)row_ptr[i] : 0;
  int total = 0, cell = 0;
  for (int t0 = 0; t0 < all; t0 += 32 * NL_AHEAD) {
    NlAtom a[NL_AHEAD];
    int from[NL_AHEAD];
#pragma unroll
    for (int u = 0; u < NL_AHEAD; u++) {
      const int t = t0 + u * 32 + lane;
      from[u] = -1;
      if (t < all) {
        while (t >= first[w][cell + 1]) cell++;   // ends: first[27] = all
        from[u] = cell;
        const int k = base[w][cell] + t - first[w][cell];
        a[u] = atoms ? atoms[k] : nl_atom(pos, g, perm[k]);
      }
    }
#pragma unroll
    for (int u = 0; u < NL_AHEAD; u++) {
      bool hit = false;
      int S[3] = {0, 0, 0};
      if (from[u] >= 0) {
        for (int d = 0; d < 3; d++) S[d] = image[w][from[u]][d];
        // (x_j + shift) - x_i, squared and summed in the order of the host list, without contraction
        const double ddx = __dsub_rn(__dadd_rn(a[u].x, (double)S[0] * g.len[0]), xi[0]);
        const double ddy = __dsub_rn(__dadd_rn(a[u].y, (double)S[1] * g.len[1]), xi[1]);
        const double ddz = __dsub_rn(__dadd_rn(a[u].z, (double)S[2] * g.len[2]), xi[2]);
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)), __dmul_rn(ddz, ddz));
        hit = d2 < g.rc2 && !(S[0] == 0 && S[1] == 0 && S[2] == 0 && (int64_t)a[u].id == i);
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (FILL && hit) {
        const int64_t e = out + __popc(m & ((1u << lane) - 1u));
        sender[e] = a[u].id;
        receiver[e] = (int32_t)i;
        int wj[3] = {0, 0, 0};
        if (a[u].wrapped)
          for (int d = 0; d < 3; d++) {
            double xw;
            int cj;
            locate(g, d, pos[3 * (int64_t)a[u].id + d], xw, cj, wj[d]);
          }
        for (int d = 0; d < 3; d++) {
          const int s = S[d] - wj[d] + wi[d];
          if (shift_idx) shift_idx[3 * e + d] = (int8_t)s;
          if (shifts) shifts[3 * e + d] = (double)s * g.len[d];
        }
      }
      out += __popc(m);
      total += __popc(m);
    }
  }
  if (!FILL && lane == 0) count[i] = total;
}

static bool nl_small(int64_t natoms, int64_t ncells) { return natoms <= NL_SMALL_ATOMS && ncells <= NL_SMALL_CELLS; }
static int64_t nl_align(int64_t x) { return (x + 255) / 256 * 256; }
// atoms in cell order, cell pointers, then (systems that do not fit one block) cell ids, their grouping and its workspace
static int64_t nl_ws_atoms(int64_t n) { return nl_align(n * (int64_t)sizeof(NlAtom)); }
static int64_t nl_ws_cells(int64_t ncells) { return nl_align((ncells + 1) * 4); }

}  // namespace cmace

using namespace cmace;

extern "C" {

int64_t cmace_nl_num_cells(double lx, double ly, double lz, double r_cut) {
  NlGeom g;
  if (make_geom(g, 0, 0, 0, lx, ly, lz, 0, r_cut, "cmace_nl_num_cells")) return 0;
  return (int64_t)g.ncell[0] * g.ncell[1] * g.ncell[2];
}

int cmace_nl_cell_ids_f64(const double *pos, int64_t natoms, double lox, double loy, double loz, double lx, double ly,
                          double lz, int pbc_mask, double r_cut, int32_t *cell_id, cmace_stream_t stream) {
  NlGeom g;
  if (int rc = make_geom(g, lox, loy, loz, lx, ly, lz, pbc_mask, r_cut, "cmace_nl_cell_ids")) return rc;
  if (natoms < 0) return fail(CMACE_ERR_ARG, "cmace_nl_cell_ids: negative size");
  if (natoms == 0) return CMACE_OK;
  if (!pos || !cell_id) return fail(CMACE_ERR_ARG, "cmace_nl_cell_ids: null pointer");
  nl_cell_ids_kernel<<<(unsigned)((natoms + 255) / 256), 256, 0, (cudaStream_t)stream>>>(pos, natoms, g, cell_id);
  return check_launch("cmace_nl_cell_ids");
}

int cmace_nl_count_f64(const double *pos, int64_t natoms, int64_t nrecv, double lox, double loy, double loz, double lx,
                       double ly, double lz, int pbc_mask, double r_cut, const int32_t *perm, const int32_t *cell_ptr,
                       int32_t *count, cmace_stream_t stream) {
  NlGeom g;
  if (int rc = make_geom(g, lox, loy, loz, lx, ly, lz, pbc_mask, r_cut, "cmace_nl_count")) return rc;
  if (natoms < 0 || nrecv < 0 || nrecv > natoms) return fail(CMACE_ERR_ARG, "cmace_nl_count: bad size");
  if (nrecv == 0) return CMACE_OK;
  if (!pos || !perm || !cell_ptr || !count) return fail(CMACE_ERR_ARG, "cmace_nl_count: null pointer");
  nl_walk_kernel<false><<<(unsigned)((nrecv + 3) / 4), 128, 0, (cudaStream_t)stream>>>(
      pos, nrecv, g, nullptr, perm, cell_ptr, count, nullptr, nullptr, nullptr, nullptr, nullptr);
  return check_launch("cmace_nl_count");
}

int cmace_nl_fill_f64(const double *pos, int64_t natoms, int64_t nrecv, double lox, double loy, double loz, double lx,
                      double ly, double lz, int pbc_mask, double r_cut, const int32_t *perm, const int32_t *cell_ptr,
                      const int32_t *row_ptr, int32_t *sender, int32_t *receiver, int8_t *shift_idx, double *shifts,
                      cmace_stream_t stream) {
  NlGeom g;
  if (int rc = make_geom(g, lox, loy, loz, lx, ly, lz, pbc_mask, r_cut, "cmace_nl_fill")) return rc;
  if (natoms < 0 || nrecv < 0 || nrecv > natoms) return fail(CMACE_ERR_ARG, "cmace_nl_fill: bad size");
  if (nrecv == 0) return CMACE_OK;
  if (!pos || !perm || !cell_ptr || !row_ptr || !sender || !receiver)
    return fail(CMACE_ERR_ARG, "cmace_nl_fill: null pointer");
  nl_walk_kernel<true><<<(unsigned)((nrecv + 3) / 4), 128, 0, (cudaStream_t)stream>>>(
      pos, nrecv, g, nullptr, perm, cell_ptr, nullptr, row_ptr, sender, receiver, shift_idx, shifts);
  return check_launch("cmace_nl_fill");
}

int64_t cmace_nl_workspace_bytes(int64_t natoms, int64_t nrecv, double lx, double ly, double lz, double r_cut) {
  const int64_t ncells = cmace_nl_num_cells(lx, ly, lz, r_cut);
  if (ncells < 1 || natoms < 0 || nrecv < 0) return 0;
  int64_t b = nl_ws_atoms(natoms) + nl_ws_cells(ncells) + nl_align(cmace_scan_workspace_bytes(nrecv + 1));
  if (!nl_small(natoms, ncells)) b += 2 * nl_align(natoms * 4) + nl_align(cmace_sender_order_workspace_bytes(natoms));
  return b;
}

int cmace_nl_build_f64(const double *pos, int64_t natoms, int64_t nrecv, double lox, double loy, double loz, double lx,
                       double ly, double lz, int pbc_mask, double r_cut, void *workspace, int64_t workspace_bytes,
                       int32_t *row_ptr, cmace_stream_t stream) {
  NlGeom g;
  if (int rc = make_geom(g, lox, loy, loz, lx, ly, lz, pbc_mask, r_cut, "cmace_nl_build")) return rc;
  if (natoms < 0 || nrecv < 0 || nrecv > natoms || natoms > 0x7ffffff0LL) return fail(CMACE_ERR_ARG, "cmace_nl_build: bad size");
  if (!workspace || !row_ptr || (natoms > 0 && !pos)) return fail(CMACE_ERR_ARG, "cmace_nl_build: null pointer");
  if (workspace_bytes < cmace_nl_workspace_bytes(natoms, nrecv, lx, ly, lz, r_cut))
    return fail(CMACE_ERR_ARG, "cmace_nl_build: workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ncells = (int64_t)g.ncell[0] * g.ncell[1] * g.ncell[2];
  char *w = static_cast<char *>(workspace);
  NlAtom *atoms = reinterpret_cast<NlAtom *>(w);
  int32_t *cell_ptr = reinterpret_cast<int32_t *>(w + nl_ws_atoms(natoms));
  char *scan_ws = w + nl_ws_atoms(natoms) + nl_ws_cells(ncells);
  const int64_t scan_bytes = nl_align(cmace_scan_workspace_bytes(nrecv + 1));
  cudaError_t e = cudaMemsetAsync(row_ptr, 0, (size_t)(nrecv + 1) * 4, st);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "cmace_nl_build: %s", cudaGetErrorString(e));
  if (nrecv == 0) return CMACE_OK;
  if (nl_small(natoms, ncells)) {
    cudaFuncSetAttribute(nl_bin_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NL_SMALL_SMEM);
    nl_bin_small_kernel<<<1, NL_SMALL_THREADS, NL_SMALL_SMEM, st>>>(pos, (int)natoms, (int)ncells, g, cell_ptr, atoms);
  } else {
    char *more = scan_ws + scan_bytes;
    int32_t *ids = reinterpret_cast<int32_t *>(more), *perm = reinterpret_cast<int32_t *>(more + nl_align(natoms * 4));
    nl_cell_ids_kernel<<<(unsigned)((natoms + 255) / 256), 256, 0, st>>>(pos, natoms, g, ids);
    if (int rc = cmace_sender_order(ids, natoms, ncells, perm, cell_ptr, more + 2 * nl_align(natoms * 4),
                                    nl_align(cmace_sender_order_workspace_bytes(natoms)), stream))
      return rc;
    nl_atoms_kernel<<<(unsigned)((natoms + 255) / 256), 256, 0, st>>>(pos, natoms, g, perm, atoms);
  }
  nl_walk_kernel<false><<<(unsigned)((nrecv + 3) / 4), 128, 0, st>>>(pos, nrecv, g, atoms, nullptr, cell_ptr, row_ptr, nullptr,
                                                                     nullptr, nullptr, nullptr, nullptr);
  if (nrecv + 1 <= 16384) {   // one block; longer ones by cub's scan
    const int smem = (int)(nrecv + 1 + 33) * 4;
    cudaFuncSetAttribute(nl_scan_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (16384 + 33) * 4);
    nl_scan_small_kernel<<<1, NL_SMALL_THREADS, smem, st>>>(row_ptr, (int)(nrecv + 1));
    return check_launch("cmace_nl_build");
  }
  if (int rc = check_launch("cmace_nl_build")) return rc;
  return cmace_exclusive_scan_i32(row_ptr, nrecv + 1, row_ptr, scan_ws, scan_bytes, stream);
}

int64_t cmace_scan_workspace_bytes(int64_t n) {
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const int32_t *)nullptr, (int32_t *)nullptr, (int)(n < 1 ? 1 : n));
  return (int64_t)bytes + 256;
}

int cmace_exclusive_scan_i32(const int32_t *in, int64_t n, int32_t *out, void *workspace, int64_t workspace_bytes,
                             cmace_stream_t stream) {
  if (n < 0 || n > 0x7ffffffeLL) return fail(CMACE_ERR_ARG, "cmace_exclusive_scan: bad size");
  if (n == 0) return CMACE_OK;
  if (!in || !out || !workspace) return fail(CMACE_ERR_ARG, "cmace_exclusive_scan: null pointer");
  size_t bytes = (size_t)workspace_bytes;
  cudaError_t e = cub::DeviceScan::ExclusiveSum(workspace, bytes, in, out, (int)n, (cudaStream_t)stream);
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "cmace_exclusive_scan: %s", cudaGetErrorString(e));
  return check_launch("cmace_exclusive_scan");
}

int cmace_nl_emit_f64(const double *pos, int64_t natoms, int64_t nrecv, double lox, double loy, double loz, double lx,
                      double ly, double lz, int pbc_mask, double r_cut, const void *workspace, const int32_t *row_ptr,
                      int32_t *sender, int32_t *receiver, int8_t *shift_idx, double *shifts, cmace_stream_t stream) {
  NlGeom g;
  if (int rc = make_geom(g, lox, loy, loz, lx, ly, lz, pbc_mask, r_cut, "cmace_nl_emit")) return rc;
  if (natoms < 0 || nrecv < 0 || nrecv > natoms) return fail(CMACE_ERR_ARG, "cmace_nl_emit: bad size");
  if (nrecv == 0) return CMACE_OK;
  if (!pos || !workspace || !row_ptr || !sender || !receiver)
    return fail(CMACE_ERR_ARG, "cmace_nl_emit: null pointer");
  const char *w = static_cast<const char *>(workspace);
  nl_walk_kernel<true><<<(unsigned)((nrecv + 3) / 4), 128, 0, (cudaStream_t)stream>>>(
      pos, nrecv, g, reinterpret_cast<const NlAtom *>(w), nullptr, reinterpret_cast<const int32_t *>(w + nl_ws_atoms(natoms)), nullptr,
      row_ptr, sender, receiver, shift_idx, shifts);
  return check_launch("cmace_nl_emit");
}
}
