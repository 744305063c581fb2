// Second layer's radial weights and their derivative, float64:  R = h W,  R' = h' W  [rows, 4C], W [64, 4C].
//
// Bound by the float64 tensor instruction (128 flop a cycle and SM).  The weight slice of a block, 64 x 128, stays in shared
// memory for the whole kernel and the rows' tiles pass by, the next one on its way while one is worked on: a product that
// fetches both operands for every tile has four K slices to hide their latency behind and stood at 73 % of the instruction's
// rate; here 81 %.  h and h' are one list of tiles.  With the edges of a pair sharing a row this is the work that R alone was, and
// the product that formed dE/dr from the gradient of R is gone: 1 015 + 869 -> 912 us at 8 000 atoms and 128 channels, 512 + 455
// -> 463 at 64.  16 warps of 32 rows x 32 columns (TM = 128) or 32 x 16 (TM = 64, while there are
// not two tiles a block otherwise); row strides of 68 and 132 doubles make the fragment loads free of bank conflicts.
#include "step_common.cuh"

namespace cmace {

constexpr int RO_N = 128, RO_THREADS = 512, RO_LDA = 68, RO_LDB = 132;

struct RadialOutArgs64 {
  const double *h[2], *W;
  double *out[2];
  EdgeRows rows;
  int64_t nedges;
  int N;
};

template <int TM>
__global__ void __launch_bounds__(RO_THREADS, 1) radial_out_f64_kernel(const RadialOutArgs64 g) {
  constexpr int WM = TM / 32, WN = 16 / WM, NJ = RO_N / WN / 8;
  extern __shared__ __align__(16) double ro_smem[];
  double *const sB = ro_smem, *const sA = sB + ST_H * RO_LDB;   // two tiles of rows
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fr = lane >> 2, fk = lane & 3;
  const int slices = (g.N + RO_N - 1) / RO_N, slice = (int)(blockIdx.x % (unsigned)slices), n0 = slice * RO_N;
  auto copy = [](double *dst, const double *src, bool there) {   // no source bytes: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(there ? 16 : 0)
                 : "memory");
  };
  for (int i = tid; i < ST_H * RO_N / 2; i += RO_THREADS) {
    const int k = i / (RO_N / 2), c = 2 * (i % (RO_N / 2));
    copy(sB + k * RO_LDB + c, n0 + c < g.N ? g.W + (int64_t)k * g.N + n0 + c : g.W, n0 + c < g.N);
  }
  grid_begin();
  const int64_t nrows = count_rows(g.rows, g.nedges), tiles = (nrows + TM - 1) / TM;
  const int64_t step = gridDim.x / (unsigned)slices;
  auto fetch = [&](int64_t t, double *dst) {
    const bool second = t >= tiles;
    const double *src = second ? g.h[1] : g.h[0];
    const int64_t first = (second ? t - tiles : t) * TM;
    for (int i = tid; i < TM * ST_H / 2; i += RO_THREADS) {
      const int r = i / (ST_H / 2), c = 2 * (i % (ST_H / 2));
      copy(dst + r * RO_LDA + c, first + r < nrows ? src + (first + r) * ST_H + c : src, first + r < nrows);
    }
  };
  int64_t t = blockIdx.x / (unsigned)slices;
  if (t >= 2 * tiles) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  fetch(t, sA);
  asm volatile("cp.async.commit_group;" ::: "memory");
  const int wm = (warp / WN) * 32, wn = (warp % WN) * (8 * NJ);
  for (int turn = 0; t < 2 * tiles; t += step, turn ^= 1) {
    const double *const A = sA + turn * TM * RO_LDA;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // the tile is there, and everybody has left the one before it
    if (t + step < 2 * tiles) fetch(t + step, sA + (turn ^ 1) * TM * RO_LDA);
    asm volatile("cp.async.commit_group;" ::: "memory");
    double acc[4][NJ][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < NJ; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 4
    for (int k = 0; k < ST_H; k += 4) {
      double a[4], b[NJ];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = A[(wm + 8 * i + fr) * RO_LDA + k + fk];
#pragma unroll
      for (int j = 0; j < NJ; j++) b[j] = sB[(k + fk) * RO_LDB + wn + 8 * j + fr];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < NJ; j++) dmma(acc[i][j], a[i], b[j]);
    }
    const bool second = t >= tiles;
    double *const out = second ? g.out[1] : g.out[0];
    const int64_t first = (second ? t - tiles : t) * TM;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int64_t row = first + wm + 8 * i + fr;
      if (row >= nrows) continue;
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const int c = n0 + wn + 8 * j + 2 * fk;
        if (c < g.N) *reinterpret_cast<double2 *>(out + row * g.N + c) = make_double2(acc[i][j][0], acc[i][j][1]);
      }
    }
  }
}

int radial_out_f64(const double *h, const double *dh, const double *W, const EdgeRows &rows, int64_t nedges, int N, double *R,
                   double *dR, cudaStream_t st) {
  const char *what = "cmace_step(radial_out)";
  if (nedges == 0) return CMACE_OK;
  if (N % 2 != 0) return fail(CMACE_ERR_ARG, "%s: bad size", what);
  const RadialOutArgs64 g{{h, dh}, W, {R, dR}, rows, nedges, N};
  const int slices = (N + RO_N - 1) / RO_N;
  const int64_t expected = rows.count ? (nedges + 1) / 2 : nedges;   // a complete list has half as many rows as edges
  const bool wide = 2 * ((expected + 127) / 128) * slices >= 4 * 148;
  auto launch = [&](auto kernel, int tm) -> int {
    const int smem = (ST_H * RO_LDB + 2 * tm * RO_LDA) * (int)sizeof(double);
    const int64_t tiles = 2 * ((nedges + tm - 1) / tm);
    int64_t blocks = 148 / slices;
    if (blocks > tiles) blocks = tiles;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    launch_chained(kernel, (unsigned)(blocks * slices), RO_THREADS, (size_t)smem, st, g);
    return check_launch(what);
  };
  return wide ? launch(radial_out_f64_kernel<128>, 128) : launch(radial_out_f64_kernel<64>, 64);
}

}  // namespace cmace
