// Topology preprocessing, run once per neighbour list (not per layer or per step):
//  * receiver CSR from the receiver-sorted edge list (empty rows allowed),
//  * sender-grouped edge permutation (stable radix sort of edge ids by sender) + its CSR,
//  * nodes grouped by chemical element (same routine, keys = element index).
#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"

namespace cmace {

char *error_buffer() {
  static thread_local char buf[512] = {0};
  return buf;
}

// keys sorted ascending -> ptr[k] = first position whose key is >= k, for k = 0..nkeys.
// Thread i looks at the boundary between positions i-1 and i and fills every ptr entry whose
// first position is i, so keys that never occur get an empty range.
__global__ void csr_from_sorted_kernel(const int32_t *__restrict__ keys, int64_t n, int64_t nkeys,
                                       int32_t *__restrict__ ptr) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  int64_t prev = (i == 0) ? -1 : (int64_t)keys[i - 1];
  int64_t cur = (i == n) ? nkeys : (int64_t)keys[i];
  if (cur > nkeys) cur = nkeys;
  if (prev < -1) prev = -1;
  for (int64_t k = prev + 1; k <= cur; k++) ptr[k] = (int32_t)i;
}

__global__ void iota_kernel(int32_t *p, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = (int32_t)i;
}

// Short lists: a stable counting sort and its pointers by one block.  Every warp counts a contiguous piece, lanes with the same key
// together (match); a key's places follow from the warps' counts in order, and a second walk over the piece writes them.  The radix
// sort is eight launches and memsets around two passes; here one launch: 17 -> 7 us at 1 600 entries, 17 -> 11 at 3 000, 31 -> 26 at
// 10 000, but 42 -> 48 at 20 000 (a match of 32 different keys costs 70 cycles of the one SM).  Keys outside 0 .. nkeys - 1 come
// last, as in the radix sort.
constexpr int GS_THREADS = 1024, GS_WARPS = GS_THREADS / 32, GS_AHEAD = 4;
constexpr int64_t GS_MOST = 8192;      // entries: the block's walk takes 2.4 us a thousand, the radix sort 17 to 30 us up to 10 000
constexpr int64_t GS_MOST_KEYS = 1600; // 33 counts a key in shared memory

__global__ void __launch_bounds__(GS_THREADS) group_small_kernel(const int32_t *__restrict__ keys, int n, int nkeys,
                                                                 int32_t *__restrict__ order, int32_t *__restrict__ ptr) {
  extern __shared__ int32_t gs_smem[];
  __shared__ int32_t sums[GS_WARPS];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int ld = nkeys + 1;                 // the last one: keys outside the range
  int32_t *const start = gs_smem, *const count = gs_smem + ld + w * ld;   // [ld], [warps][ld]
  for (int i = tid; i < GS_WARPS * ld; i += GS_THREADS) gs_smem[ld + i] = 0;
  __syncthreads();
  const int per = (n + GS_THREADS - 1) / GS_THREADS * 32, lo = w * per < n ? w * per : n, hi = lo + per < n ? lo + per : n;
  const unsigned below = (1u << lane) - 1u;
  auto key_at = [&](int i) {
    const int32_t k = i < hi ? __ldg(keys + i) : nkeys;
    return (uint32_t)k < (uint32_t)nkeys ? k : nkeys;
  };
  // body(i, rank, peers, key, lanes) for every entry of the piece, in order; rank: among the lanes with its key
  auto walk = [&](auto body) {
    for (int b = lo; b < hi; b += 32 * GS_AHEAD) {
      int key[GS_AHEAD];
#pragma unroll
      for (int u = 0; u < GS_AHEAD; u++) key[u] = key_at(b + 32 * u + lane);
#pragma unroll
      for (int u = 0; u < GS_AHEAD; u++) {
        const int i = b + 32 * u + lane;
        if (b + 32 * u >= hi) break;
        const unsigned active = __ballot_sync(0xffffffffu, i < hi);
        if (i < hi) {
          const unsigned peers = __match_any_sync(active, key[u]);
          body(i, __popc(peers & below), __popc(peers), key[u], active);
        }
        __syncwarp();
      }
    }
  };
  walk([&](int, int rank, int peers, int key, unsigned) {
    if (rank == 0) count[key] += peers;
  });
  __syncthreads();
  // a key's counts become the places of its warps' first entries, then the keys' starts follow by a scan over the block
  int carry = 0;
  for (int b = 0; b < ld; b += GS_THREADS) {
    const int k = b + tid;
    int total = 0;
    if (k < ld)
#pragma unroll 8
      for (int v = 0; v < GS_WARPS; v++) {
        int32_t &c = gs_smem[ld + v * ld + k];
        const int here = c;
        c = total;
        total += here;
      }
    int inc = total;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += o;
    }
    if (lane == 31) sums[w] = inc;
    __syncthreads();
    int before = 0, all = 0;
    for (int v = 0; v < GS_WARPS; v++) {
      before += v < w ? sums[v] : 0;
      all += sums[v];
    }
    if (k < ld) {
      const int at = carry + before + inc - total;
      start[k] = at;
      ptr[k] = at;      // ptr[nkeys]: where the keys outside the range begin, the end of the others
    }
    carry += all;
    __syncthreads();
  }
  walk([&](int i, int rank, int peers, int key, unsigned lanes) {
    const int at = count[key];
    order[start[key] + at + rank] = i;
    __syncwarp(lanes);
    if (rank == 0) count[key] = at + peers;
  });
}

static int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

static int64_t cub_temp_bytes(int64_t n) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const int32_t *)nullptr, (int32_t *)nullptr,
                                  (const int32_t *)nullptr, (int32_t *)nullptr, (int)n);
  return (int64_t)bytes;
}

static int group_by_key(const int32_t *keys, int64_t n, int64_t nkeys, int32_t *order, int32_t *ptr,
                        void *workspace, int64_t workspace_bytes, cudaStream_t st, const char *what) {
  if (n < 0 || nkeys < 0 || n > 0x7fffffffLL) return fail(CMACE_ERR_ARG, "%s: bad size", what);
  if (!ptr) return fail(CMACE_ERR_ARG, "%s: null pointer", what);
  if (n > 0) {
    if (!keys || !order || !workspace) return fail(CMACE_ERR_ARG, "%s: null pointer", what);
    const int64_t need = cmace_sender_order_workspace_bytes(n);
    if (workspace_bytes < need)
      return fail(CMACE_ERR_ARG, "%s: workspace of %lld bytes, %lld needed", what,
                  (long long)workspace_bytes, (long long)need);
    if (n <= GS_MOST && nkeys <= GS_MOST_KEYS && nkeys > 0) {
      const int smem = (int)((GS_WARPS + 1) * (nkeys + 1) * 4), most = (int)((GS_WARPS + 1) * (GS_MOST_KEYS + 1) * 4);
      cudaError_t err = cudaFuncSetAttribute(group_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      if (err != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(err));
      group_small_kernel<<<1, GS_THREADS, smem, st>>>(keys, (int)n, (int)nkeys, order, ptr);
      return check_launch(what);
    }
    char *w = static_cast<char *>(workspace);
    int32_t *keys_sorted = reinterpret_cast<int32_t *>(w);
    int32_t *ids = reinterpret_cast<int32_t *>(w + align256(n * 4));
    void *temp = w + 2 * align256(n * 4);
    size_t temp_bytes = (size_t)(workspace_bytes - 2 * align256(n * 4));
    iota_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ids, n);
    int end_bit = 1;
    while (end_bit < 31 && (1LL << end_bit) < nkeys) end_bit++;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys, keys_sorted, ids, order,
                                                    (int)n, 0, end_bit, st);
    if (e != cudaSuccess) return fail(CMACE_ERR_CUDA, "%s: radix sort: %s", what, cudaGetErrorString(e));
    csr_from_sorted_kernel<<<(unsigned)((n + 1 + 255) / 256), 256, 0, st>>>(keys_sorted, n, nkeys, ptr);
  } else {
    csr_from_sorted_kernel<<<1, 256, 0, st>>>(nullptr, 0, nkeys, ptr);
  }
  return check_launch(what);
}

}  // namespace cmace

using namespace cmace;

extern "C" {

const char *cmace_last_error(void) { return error_buffer(); }
int cmace_abi_version(void) { return 1; }

int cmace_receiver_csr(const int32_t *receiver, int64_t nedges, int64_t nnodes, int32_t *row_ptr,
                       cmace_stream_t stream) {
  if (nedges < 0 || nnodes < 0 || nedges > 0x7fffffffLL)
    return fail(CMACE_ERR_ARG, "cmace_receiver_csr: bad size");
  if (!row_ptr || (nedges > 0 && !receiver)) return fail(CMACE_ERR_ARG, "cmace_receiver_csr: null pointer");
  csr_from_sorted_kernel<<<(unsigned)((nedges + 1 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      receiver, nedges, nnodes, row_ptr);
  return check_launch("cmace_receiver_csr");
}

int64_t cmace_sender_order_workspace_bytes(int64_t n) {
  if (n <= 0) return 0;
  return 2 * align256(n * 4) + align256(cub_temp_bytes(n));
}

int cmace_sender_order(const int32_t *sender, int64_t nedges, int64_t nnodes, int32_t *perm,
                       int32_t *send_ptr, void *workspace, int64_t workspace_bytes, cmace_stream_t stream) {
  return group_by_key(sender, nedges, nnodes, perm, send_ptr, workspace, workspace_bytes,
                      (cudaStream_t)stream, "cmace_sender_order");
}

int cmace_group_by_element(const int32_t *elem, int64_t nnodes, int nelements, int32_t *node_order,
                           int32_t *elem_start, void *workspace, int64_t workspace_bytes,
                           cmace_stream_t stream) {
  return group_by_key(elem, nnodes, nelements, node_order, elem_start, workspace, workspace_bytes,
                      (cudaStream_t)stream, "cmace_group_by_element");
}
}
