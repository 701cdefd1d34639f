// prep.cu -- the resident graph's internal order, built on the GPU.
//
// From the caller's CSR: vertices renamed by degree, highest first (ties by
// caller id), every list renamed and sorted ascending, and GroupBy's hub of
// every vertex (GroupBy.cuh:19-84).  Each of the two orders is one stable LSD
// radix sort of 64-bit keys: (max degree - degree, id) for the vertices, and
// (new source, new neighbour) for the edges, whose sorted low halves are the
// adjacency array.
//
// The sort streams its keys twice per 8-bit digit (histogram, scatter); a
// scatter tile ranks its keys inside its warps (match), sorts the tile in
// shared memory and then writes one run per digit, so that the writes to the
// 256 destinations are coalesced.  What bounds the whole build is the host's
// side of it: the copy of the caller's arrays that the handle keeps and the
// pageable upload (R-MAT scale 22: 0.55 GB, about 110 ms in all).
#include <algorithm>
#include <cstdint>

#include <cuda_runtime.h>

#include "internal.h"

namespace ibfs {
namespace {

using u64 = unsigned long long;

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;                   // keys per thread
constexpr int kTile = kThreads * kItems;     // 4096 keys, 32 KB of shared memory
constexpr int kScanTile = 2048;              // counters per scan block

// ---- exclusive scan of 32-bit counters (in place) or 64-bit degrees ------------
// Every block scans kScanTile entries (8 per thread) and leaves its total in
// sums; the totals are scanned the same way and added back.
template <class T>
__device__ __forceinline__ T block_scan(T x, T* total) {  // exclusive, 256 threads
  __shared__ T s[kWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();
  if (lane == 31) s[w] = incl;
  __syncthreads();
  T before = 0, all = 0;
  for (int i = 0; i < kWarps; i++) {
    if (i < w) before += s[i];
    all += s[i];
  }
  *total = all;
  return before + incl - x;
}

template <class T>
__global__ void __launch_bounds__(kThreads) k_scan(T* a, int64_t n, T* sums) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + threadIdx.x * 8;
  T v[8], own = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    v[i] = base + i < n ? a[base + i] : 0;
    own += v[i];
  }
  T total;
  T at = block_scan<T>(own, &total);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if (base + i < n) a[base + i] = at;
    at += v[i];
  }
  if (threadIdx.x == 0 && sums) sums[blockIdx.x] = total;
}

template <class T>
__global__ void __launch_bounds__(kThreads) k_scan_add(T* a, int64_t n, const T* sums) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + threadIdx.x * 8;
  const T x = sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (base + i < n) a[base + i] += x;
}

// Entries of scratch that scan() needs behind an array of n.
int64_t scan_scratch(int64_t n) {
  int64_t t = 0;
  while (n > kScanTile) {
    n = (n + kScanTile - 1) / kScanTile;
    t += n;
  }
  return t;
}

template <class T>
void scan(T* a, int64_t n, T* scratch, cudaStream_t s) {
  const int64_t blocks = (n + kScanTile - 1) / kScanTile;
  if (blocks <= 1) {
    k_scan<T><<<1, kThreads, 0, s>>>(a, n, nullptr);
    return;
  }
  k_scan<T><<<(unsigned)blocks, kThreads, 0, s>>>(a, n, scratch);
  scan<T>(scratch, blocks, scratch + blocks, s);
  k_scan_add<T><<<(unsigned)blocks, kThreads, 0, s>>>(a, n, scratch);
}

// ---- stable LSD radix sort of 64-bit keys by bits [lo, hi) -----------------------
__global__ void __launch_bounds__(kThreads) k_hist(const u64* key, int64_t n, int shift,
                                                   int64_t ntiles, uint32_t* hist) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kTile;
#pragma unroll 4
  for (int j = 0; j < kItems; j++) {
    const int64_t i = base + j * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(uint32_t)(key[i] >> shift) & 0xFFu], 1u);
  }
  __syncthreads();
  hist[(int64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];  // digit-major
}

// Keys of a tile are taken in input order (warp, step, lane); equal digits
// keep it, so the pass is stable.
__global__ void __launch_bounds__(kThreads) k_scatter(const u64* key, int64_t n, int shift,
                                                      int64_t ntiles, const uint32_t* offs,
                                                      u64* out) {
  __shared__ u64 s_key[kTile];
  __shared__ uint32_t s_cnt[kWarps][256];  // per warp: keys of a digit, then its first rank
  __shared__ uint32_t s_dst[256];          // output offset of a digit minus its tile rank
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int d = lane; d < 256; d += 32) s_cnt[w][d] = 0;
  __syncwarp();
  const int64_t tile0 = (int64_t)blockIdx.x * kTile;
  const int have = (int)min((int64_t)kTile, n - tile0);
  u64 k[kItems];
  uint16_t rank[kItems];
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int at = (w * kItems + j) * 32 + lane;
    k[j] = at < have ? key[tile0 + at] : 0ull;
  }
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int at = (w * kItems + j) * 32 + lane;
    const int d = at < have ? (int)((uint32_t)(k[j] >> shift) & 0xFFu) : 256;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
    const int below = __popc(peers & ((1u << lane) - 1u));
    uint32_t base = 0;
    if (d < 256 && below == 0) {
      base = s_cnt[w][d];
      s_cnt[w][d] = base + __popc(peers);
    }
    base = __shfl_sync(0xFFFFFFFFu, base, __ffs(peers) - 1);
    rank[j] = (uint16_t)(base + below);
    __syncwarp();
  }
  __syncthreads();
  {  // thread = digit: ranks of the warps' first keys, and of the digit itself
    const int d = threadIdx.x;
    uint32_t sum = 0;
    for (int i = 0; i < kWarps; i++) {
      const uint32_t c = s_cnt[i][d];
      s_cnt[i][d] = sum;
      sum += c;
    }
    uint32_t total;
    const uint32_t first = block_scan<uint32_t>(sum, &total);
    for (int i = 0; i < kWarps; i++) s_cnt[i][d] += first;
    s_dst[d] = offs[(int64_t)d * ntiles + blockIdx.x] - first;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int at = (w * kItems + j) * 32 + lane;
    if (at < have) s_key[s_cnt[w][(uint32_t)(k[j] >> shift) & 0xFFu] + rank[j]] = k[j];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < have; i += kThreads) {
    const u64 x = s_key[i];
    out[s_dst[(uint32_t)(x >> shift) & 0xFFu] + (uint32_t)i] = x;
  }
}

// Sorts a (b: the other buffer); returns the one that holds the result.
u64* sort_keys(u64* a, u64* b, int64_t n, int lo, int hi, uint32_t* hist, cudaStream_t s) {
  const int64_t ntiles = (n + kTile - 1) / kTile;
  for (int shift = lo; shift < hi; shift += 8) {
    k_hist<<<(unsigned)ntiles, kThreads, 0, s>>>(a, n, shift, ntiles, hist);
    scan<uint32_t>(hist, 256 * ntiles, hist + 256 * ntiles, s);
    k_scatter<<<(unsigned)ntiles, kThreads, 0, s>>>(a, n, shift, ntiles, hist, b);
    std::swap(a, b);
  }
  return a;
}

// ---- the two orders ------------------------------------------------------------
__global__ void k_vertex_keys(const int64_t* beg, int64_t V, int64_t max_deg, u64* key) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v < V) key[v] = (u64)(max_deg - (beg[v + 1] - beg[v])) << 32 | (u64)v;
}

__global__ void k_rename(const u64* key, int64_t V, const int64_t* beg, int32_t* new_of_old,
                         u64* nbeg) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < V) {
    const uint32_t o = (uint32_t)key[i];
    new_of_old[o] = (int32_t)i;
    nbeg[i] = (u64)(beg[o + 1] - beg[o]);
  } else if (i == V) {
    nbeg[V] = 0;
  }
}

// A warp per vertex of the caller's order; the keys stay at their edge's place.
__global__ void __launch_bounds__(kThreads) k_edge_keys(const int64_t* beg, const int32_t* col,
                                                        int64_t V, const int32_t* new_of_old,
                                                        int bits, u64* key, int32_t* col_max) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * kWarps;
  int32_t top = -1;
  for (int64_t v = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); v < V; v += nw) {
    const int64_t e1 = beg[v + 1];
    const u64 hi = (u64)(uint32_t)new_of_old[v] << bits;
    for (int64_t e = beg[v] + lane; e < e1; e += 32) {
      const int32_t u = new_of_old[col[e]];
      top = max(top, u);
      key[e] = hi | (u64)(uint32_t)u;
    }
  }
  top = __reduce_max_sync(0xFFFFFFFFu, top);
  if (lane == 0 && top >= 0) atomicMax(col_max, top);
}

__global__ void k_columns(const u64* key, int64_t E, uint32_t mask, int32_t* col) {
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * 4;
  if (i + 3 < E) {
    const ulonglong2 a = reinterpret_cast<const ulonglong2*>(key + i)[0];
    const ulonglong2 b = reinterpret_cast<const ulonglong2*>(key + i)[1];
    *reinterpret_cast<int4*>(col + i) =
        make_int4((int)((uint32_t)a.x & mask), (int)((uint32_t)a.y & mask),
                  (int)((uint32_t)b.x & mask), (int)((uint32_t)b.y & mask));
  } else {
    for (int64_t j = i; j < E; j++) col[j] = (int)((uint32_t)key[j] & mask);
  }
}

// GroupBy's hub: for degree <= 128, the first neighbour in the caller's order
// whose degree is above 128.
__global__ void k_groupby_hub(const int64_t* beg, const int32_t* col, int64_t V, int32_t* hub) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= V) return;
  int32_t h = -1;
  const int64_t e0 = beg[v], e1 = beg[v + 1];
  if (e1 - e0 <= 128)
    for (int64_t e = e0; e < e1; e++) {
      const int32_t u = col[e];
      if (beg[u + 1] - beg[u] > 128) {
        h = u;
        break;
      }
    }
  hub[v] = h;
}

int bits_of(u64 x) {
  int b = 0;
  while (b < 63 && (x >> b) != 0) b++;
  return b;
}

}  // namespace

// beg_h/col_h: the caller's CSR on the host (valid; V < 2^31, 0 < E < 2^31).
// Writes beg[V+1], col[E], vmap[V] and hub[V] on the device and the largest
// neighbour id of the new order.  Returns cudaErrorMemoryAllocation when the
// sort's scratch (about 20 bytes per edge and 24 per vertex) does not fit: the
// caller then builds the order on the host.
cudaError_t prep_graph(const int64_t* beg_h, const int32_t* col_h, int64_t V, int64_t E,
                       int64_t max_deg, int64_t* beg, int32_t* col, int32_t* vmap, int32_t* hub,
                       int64_t* col_max, cudaStream_t s) {
  auto a256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const int64_t nkeys = std::max(V, E);
  const int64_t ncnt = 256 * ((nkeys + kTile - 1) / kTile);
  const size_t o_beg = 0;
  const size_t o_col = a256(o_beg + sizeof(int64_t) * (size_t)(V + 1));
  const size_t o_a = a256(o_col + sizeof(int32_t) * (size_t)E);
  const size_t o_b = a256(o_a + sizeof(u64) * (size_t)nkeys);
  const size_t o_hist = a256(o_b + sizeof(u64) * (size_t)nkeys);
  const size_t n_hist = (size_t)(ncnt + scan_scratch(ncnt));
  const size_t o_scan = a256(o_hist + sizeof(uint32_t) * n_hist);
  const size_t o_max = a256(o_scan + sizeof(u64) * (size_t)(scan_scratch(V + 1) + 1));
  uint8_t* w = nullptr;
  cudaError_t e = cudaMalloc(&w, o_max + 256);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return cudaErrorMemoryAllocation;
  }
  int64_t* obeg = reinterpret_cast<int64_t*>(w + o_beg);
  int32_t* ocol = reinterpret_cast<int32_t*>(w + o_col);
  u64* ka = reinterpret_cast<u64*>(w + o_a);
  u64* kb = reinterpret_cast<u64*>(w + o_b);
  uint32_t* hist = reinterpret_cast<uint32_t*>(w + o_hist);
  int32_t* d_max = reinterpret_cast<int32_t*>(w + o_max);
  int32_t h_max = -1;
  auto blocks = [](int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); };
  auto run = [&]() -> cudaError_t {
    cudaError_t r;
    if ((r = cudaMemcpyAsync(obeg, beg_h, sizeof(int64_t) * (size_t)(V + 1),
                             cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return r;
    // the vertex order, while the columns still travel
    k_vertex_keys<<<blocks(V), kThreads, 0, s>>>(obeg, V, max_deg, ka);
    u64* ks = sort_keys(ka, kb, V, 32, 32 + bits_of((u64)max_deg), hist, s);
    u64* nbeg = reinterpret_cast<u64*>(beg);
    k_rename<<<blocks(V + 1), kThreads, 0, s>>>(ks, V, obeg, vmap, nbeg);
    scan<u64>(nbeg, V + 1, reinterpret_cast<u64*>(w + o_scan), s);
    if ((r = cudaMemcpyAsync(ocol, col_h, sizeof(int32_t) * (size_t)E, cudaMemcpyHostToDevice,
                             s)) != cudaSuccess ||
        (r = cudaMemsetAsync(d_max, 0xFF, sizeof(int32_t), s)) != cudaSuccess)
      return r;
    const int bits = std::max(1, bits_of((u64)(V - 1)));
    const int64_t warps = std::min<int64_t>(V, 148 * 64);
    k_edge_keys<<<(unsigned)((warps + kWarps - 1) / kWarps), kThreads, 0, s>>>(
        obeg, ocol, V, vmap, bits, ka, d_max);
    k_groupby_hub<<<blocks(V), kThreads, 0, s>>>(obeg, ocol, V, hub);
    ks = sort_keys(ka, kb, E, 0, 2 * bits, hist, s);
    k_columns<<<blocks((E + 3) / 4), kThreads, 0, s>>>(ks, E, (uint32_t)((1ull << bits) - 1),
                                                       col);
    if ((r = cudaGetLastError()) != cudaSuccess) return r;
    return cudaMemcpyAsync(&h_max, d_max, sizeof(h_max), cudaMemcpyDeviceToHost, s);
  };
  e = run();
  const cudaError_t e2 = cudaStreamSynchronize(s);
  cudaFree(w);
  *col_max = h_max;
  return e != cudaSuccess ? e : e2;
}

}  // namespace ibfs
