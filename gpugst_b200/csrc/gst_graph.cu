// Device side of gst_graph_create: the resident adjacency is built from the
// caller's CSR on the GPU.  Each list is sorted by (weight, neighbour), which
// as a little-endian {neighbour, weight} pair is the order of 64-bit integers:
//   lists of 2 .. 256 arcs     bitonic, one warp and its shared memory each;
//   up to SORT_BLOCK arcs      bitonic, one block each;
//   longer ones                SORT_BLOCK pieces the same way, then merged run
//                              by run: every element's place is its own index
//                              plus its rank in the sibling run.
// Measured on 170k vertices / 13.6M arcs: packing 0.04 ms, lists 0.28, pieces
// 0.35, two merge passes 0.02 and the weight index 0.02; creating the graph, with a
// sort on 16 host threads 105 ms, takes 16 (medians of 60), which is the copy of
// the caller's pageable arrays.  Bound by the bitonic steps' shared-memory passes,
// which is no matter beside that copy.
#include "gst_device.cuh"

namespace gstb {

typedef unsigned long long u64;
constexpr uint32_t SORT_WARP = 256, SORT_WARPS = 8;

__global__ void __launch_bounds__(256) k_pack_arcs(const uint32_t* __restrict__ csr, const uint32_t* __restrict__ w,
                                                   uint2* __restrict__ adj, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    adj[i] = make_uint2(csr[i], w[i]);
}

// Bitonic sort of P (a power of two) keys in shared memory by the lanes
// t = first, first + step, ..; `sync` orders one pass after the other.
template <class Sync>
__device__ __forceinline__ void bitonic(u64* key, uint32_t P, uint32_t first, uint32_t step, Sync sync) {
  for (uint32_t size = 2; size <= P; size <<= 1)
    for (uint32_t j = size >> 1; j > 0; j >>= 1) {
      for (uint32_t t = first; t < P / 2; t += step) {
        const uint32_t a = 2u * t - (t & (j - 1u)), b = a + j;
        const u64 x = key[a], y = key[b];
        if ((x > y) == ((a & size) == 0u)) {
          key[a] = y;
          key[b] = x;
        }
      }
      sync();
    }
}

__device__ __forceinline__ uint32_t pow2_at_least(uint32_t n) { return n <= 1u ? 1u : 1u << (32 - __clz(n - 1u)); }

// Lists of 2 .. SORT_WARP arcs, one warp per vertex.
__global__ void __launch_bounds__(SORT_WARPS * 32) k_sort_lists(const uint32_t* __restrict__ beg, u64* __restrict__ adj,
                                                                uint32_t V) {
  __shared__ u64 keys[SORT_WARPS][SORT_WARP];
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  u64* key = keys[wid];
  for (uint32_t v = blockIdx.x * SORT_WARPS + wid; v < V; v += gridDim.x * SORT_WARPS) {
    const uint32_t a = beg[v], n = beg[v + 1] - a;
    if (n < 2u || n > SORT_WARP) continue;
    const uint32_t P = pow2_at_least(n);
    for (uint32_t i = lane; i < P; i += 32u) key[i] = i < n ? adj[a + i] : ~0ull;
    __syncwarp();
    bitonic(key, P, lane, 32u, [] { __syncwarp(); });
    for (uint32_t i = lane; i < n; i += 32u) adj[a + i] = key[i];
    __syncwarp();
  }
}

// Pieces {first arc, arcs} of at most SORT_BLOCK arcs, one block each.
__global__ void __launch_bounds__(512) k_sort_pieces(const uint2* __restrict__ piece, uint32_t n_pieces,
                                                     u64* __restrict__ adj) {
  __shared__ u64 key[SORT_BLOCK];
  for (uint32_t p = blockIdx.x; p < n_pieces; p += gridDim.x) {
    const uint2 pc = piece[p];
    const uint32_t P = pow2_at_least(pc.y);
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) key[i] = i < pc.y ? adj[pc.x + i] : ~0ull;
    __syncthreads();
    bitonic(key, P, threadIdx.x, blockDim.x, [] { __syncthreads(); });
    for (uint32_t i = threadIdx.x; i < pc.y; i += blockDim.x) adj[pc.x + i] = key[i];
    __syncthreads();
  }
}

// One merge pass over long lists: runs of `width` sorted arcs become runs of
// twice that.  list[s] = {first arc, arcs}, cum[s] = arcs of the lists before s
// (cum[n_lists] = all).  The pass reads the adjacency and writes tmp (where list
// s starts at cum[s]), or the other way round.
__global__ void __launch_bounds__(256) k_merge_runs(const uint2* __restrict__ list, const uint32_t* __restrict__ cum,
                                                    uint32_t n_lists, u64* __restrict__ adj, u64* __restrict__ tmp,
                                                    uint32_t width, int to_tmp) {
  const uint32_t total = cum[n_lists];
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = n_lists;
    while (hi - lo > 1u) {
      const uint32_t mid = (lo + hi) >> 1;
      if (cum[mid] <= e)
        lo = mid;
      else
        hi = mid;
    }
    const uint2 L = list[lo];
    const u64* src = to_tmp ? adj + L.x : tmp + cum[lo];
    u64* dst = to_tmp ? tmp + cum[lo] : adj + L.x;
    const uint32_t i = (uint32_t)e - cum[lo], run = i / width;
    const bool right = run & 1u;
    const u64 x = src[i];
    // the sibling run [s0, s1); equal keys of the left run come first
    const uint32_t s0 = (uint32_t)min((u64)(right ? run - 1u : run + 1u) * width, (u64)L.y);
    const uint32_t s1 = (uint32_t)min((u64)s0 + width, (u64)L.y);
    uint32_t a = s0, b = s1;
    while (a < b) {
      const uint32_t m = a + (b - a) / 2u;
      const u64 y = src[m];
      if (right ? y <= x : y < x)
        a = m + 1u;
      else
        b = m;
    }
    dst[(right ? i - width : i) + (a - s0)] = x;
  }
}

// Weight-bucket index: for each vertex the first arc heavier than 2^b, b = 0..6,
// and its first arc.
__global__ void __launch_bounds__(256) k_weight_index(const uint32_t* __restrict__ beg, const uint2* __restrict__ adj,
                                                      uint32_t* __restrict__ wcut, uint32_t V) {
  const size_t n = (size_t)V * 8;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)(t >> 3), lim = 1u << (t & 7u);
    uint32_t a = beg[v], b = (t & 7u) == 7u ? a : beg[v + 1];
    while (a < b) {
      const uint32_t m = a + (b - a) / 2u;
      if (adj[m].y <= lim)
        a = m + 1u;
      else
        b = m;
    }
    wcut[t] = a;
  }
}

}  // namespace gstb
