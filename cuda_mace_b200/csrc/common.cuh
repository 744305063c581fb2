// Shared helpers of the C-ABI library: status codes, error text, launch checks.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/cuda_mace_b200.h"

namespace cmace {

// thread-local message returned by cmace_last_error()
char *error_buffer();

inline int fail(int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(error_buffer(), 512, fmt, ap);
  va_end(ap);
  return code;
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

inline int check_launch(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return CMACE_OK;
}

// strides of an array of 16 values per edge, over components and over edges: {E, 1} for [16, E], {1, 16} for [E, 16]
struct ImpLayout {
  int64_t m, e;
};

// operator launchers that other translation units call with their own layout of Y
template <typename T>
int imp_fwd(const T *X, const T *Y, const T *R, const int32_t *sender, const int32_t *row_ptr, int64_t nnodes,
            int64_t nedges, ImpLayout ys, int C, T *out, cmace_stream_t stream);
template <typename T>
int imp_bwd_edge(const T *X, const T *Y, const T *R, const T *G, const int32_t *sender, const int32_t *row_ptr,
                 int64_t nnodes, int64_t nedges, ImpLayout ys, int C, T *gradR, T *gradY, T *Tout, T *partial,
                 cmace_stream_t stream);
template <typename T>   // nedges < 0: not known
int imp_bwd_node(const T *Tin, const int32_t *perm, const int32_t *send_ptr, int64_t nnodes, int64_t nedges, int C, T *gradX,
                 cmace_stream_t stream);
int gemm3x_gradr(const float *X, const float *G, const float *Y, ImpLayout ys, const int32_t *sender,
                 const int32_t *receiver, const float *packed, int64_t nedges, int channels, int N, const float *dot,
                 float *out, int32_t *status, cmace_stream_t stream);

// l of each of the 16 (l, m) components
__host__ __device__ constexpr int l_of_lm(int lm) { return lm == 0 ? 0 : (lm < 4 ? 1 : (lm < 9 ? 2 : 3)); }

template <typename T, int VEC>
struct Vec;  // VEC scalars moved with one load/store
template <>
struct Vec<float, 4> { using type = float4; };
template <>
struct Vec<float, 2> { using type = float2; };
template <>
struct Vec<float, 1> { using type = float; };
template <>
struct Vec<double, 2> { using type = double2; };
template <>
struct Vec<double, 1> { using type = double; };

// Vector load/store of VEC consecutive scalars; p must be VEC*sizeof(T) aligned.
template <typename T, int VEC>
__device__ __forceinline__ void load_vec(T (&dst)[VEC], const T *p) {
  using V = typename Vec<T, VEC>::type;
  V v = __ldg(reinterpret_cast<const V *>(p));
  const T *s = reinterpret_cast<const T *>(&v);
#pragma unroll
  for (int i = 0; i < VEC; i++) dst[i] = s[i];
}
// streaming variant for data read exactly once (evict-first)
template <typename T, int VEC>
__device__ __forceinline__ void load_vec_stream(T (&dst)[VEC], const T *p) {
  using V = typename Vec<T, VEC>::type;
  V v = __ldcs(reinterpret_cast<const V *>(p));
  const T *s = reinterpret_cast<const T *>(&v);
#pragma unroll
  for (int i = 0; i < VEC; i++) dst[i] = s[i];
}
template <typename T, int VEC>
__device__ __forceinline__ void store_vec(T *p, const T (&src)[VEC]) {
  using V = typename Vec<T, VEC>::type;
  V v;
  T *d = reinterpret_cast<T *>(&v);
#pragma unroll
  for (int i = 0; i < VEC; i++) d[i] = src[i];
  *reinterpret_cast<V *>(p) = v;
}
template <typename T, int VEC>
__device__ __forceinline__ void store_vec_stream(T *p, const T (&src)[VEC]) {
  using V = typename Vec<T, VEC>::type;
  V v;
  T *d = reinterpret_cast<T *>(&v);
#pragma unroll
  for (int i = 0; i < VEC; i++) d[i] = src[i];
  __stcs(reinterpret_cast<V *>(p), v);
}

// Programmatic dependent launch: a kernel launched by launch_chained() may be resident before its predecessor in the stream
// has finished (launch latency, block scheduling and what stands before grid_wait() overlap the predecessor's last
// blocks), so it reads and writes nothing before grid_wait(), which returns when the predecessor has completed and its
// writes are visible.  grid_release() lets the successor's blocks come once every block of this grid has called it: a
// kernel with tensor memory calls it after its allocation, or a successor's block could take the columns that a block of
// this grid on the same SM still needs, and wait for that block.  Worth about 2 us a kernel in a chain of small ones.
//
// A block's grid_release() comes after its own grid_wait().  So when a kernel's first block runs, everything before its predecessor has
// completed: before grid_wait() it may read what is older than that (constant weights, the caller's list, what kernels before
// the predecessor wrote) and set up barriers and tensor memory, and a chain of small kernels is mostly such beginnings.  What the
// chain itself has written (elements, groupings, rows of pairs) it reads from L2 there (__ldcg, cp.async.cg, bulk copies): the
// order of the waits says that the writes have been performed, nothing says when an SM's L1 has let go of an older line.
// Every block waits on every path: a kernel that ended without having waited would let its successor overtake its predecessor.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_begin() {
  grid_wait();
  grid_release();
}
// It is off unless the caller has switched it on for this thread: blocks that arrive early keep the SM's split between
// shared memory and L1 as the predecessor had it, which costs kernels that live on L1 more than 2 us once they are long.
// from_second: on, but the next kernel waits for all that is before it in the stream (what its beginning reads may be the work of
// a kernel right before it that is none of the chain's), the ones after it are chained to it.
enum class Chain { off, from_second, on };
inline Chain &chain_launches() {
  static thread_local Chain chain = Chain::off;
  return chain;
}
// on for a scope: the layout of the contraction's weights and the program that reads it
struct ChainScope {
  const Chain before = chain_launches();
  ChainScope() { chain_launches() = Chain::on; }
  ~ChainScope() { chain_launches() = before; }
};
template <typename... Params, typename... Args>
inline void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = chain_launches() == Chain::on ? 1 : 0;
  if (chain_launches() == Chain::from_second) chain_launches() = Chain::on;
  cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// One thread of a converged warp, always the same one (elect.sync).  What it guards (tcgen05.mma, TMA and bulk copies) takes
// uniform-register operands: under `lane == 0` the compiler does not know that a single thread is left and wraps every such
// instruction in a loop over the lanes (a tcgen05.mma then costs 125-190 cycles to issue; elected, M = 128 with A in
// tensor memory runs at 9, 16, 32, 64 cycles for N = 16, 32, 64, 128, and with A in shared memory at 39, 40, 48, 64).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}
// a value that is the same in every lane of the warp, known to the compiler as such
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

// ---- two floats in one 64-bit register, handled by one instruction (fma / mul / add / sub .f32x2) --------------
// The kernels that use these are bound by instruction issue, not by the FMA pipe.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// channels handled per lane: the widest 16-byte-or-narrower vector that tiles C in 32-lane chunks
// The 16 harmonics of a pair of edges, lane (16 h + m) -> component m of edge h, handed to all lanes through shared memory:
// a broadcast load gives 16 bytes, a shuffle (two of them in float64) one value.  Two buffers, so that one warp barrier a
// pair is enough.
template <typename T, int WARPS>
struct PairHarmonics {
  T v[WARPS][2][32];
};
template <typename T>
__device__ __forceinline__ void take16(T (&y)[16], const T *p) {
  constexpr int V = 16 / (int)sizeof(T);
  using Piece = typename Vec<T, V>::type;
#pragma unroll
  for (int i = 0; i < 16 / V; i++) {   // p is in shared memory: no read-only load
    const Piece q = reinterpret_cast<const Piece *>(p)[i];
    const T *s = reinterpret_cast<const T *>(&q);
#pragma unroll
    for (int u = 0; u < V; u++) y[V * i + u] = s[u];
  }
}

// Sum of p[m] over the 32 lanes for all 16 m at once: after the call every lane holds the
// total of component (lane >> 1).  16 shuffles instead of 16 * 5.
template <typename T>
__device__ __forceinline__ T warp_reduce16(T (&p)[16], int lane) {
  T q8[8], q4[4], q2[2];
  {
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const T send = up ? p[i] : p[i + 8];
      const T keep = up ? p[i + 8] : p[i];
      q8[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
  }
  {
    const bool up = lane & 8;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const T send = up ? q8[i] : q8[i + 4];
      const T keep = up ? q8[i + 4] : q8[i];
      q4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
  }
  {
    const bool up = lane & 4;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const T send = up ? q4[i] : q4[i + 2];
      const T keep = up ? q4[i + 2] : q4[i];
      q2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
  }
  const bool up = lane & 2;
  const T send = up ? q2[0] : q2[1];
  const T keep = up ? q2[1] : q2[0];
  T r = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

template <typename T>
inline int pick_vec(int channels);
template <>
inline int pick_vec<float>(int c) { return c % 128 == 0 ? 4 : (c % 64 == 0 ? 2 : 1); }
template <>
inline int pick_vec<double>(int c) { return c % 64 == 0 ? 2 : 1; }

}  // namespace cmace
