// bfs_device.cuh -- device side of the concurrent multi-source BFS.
//
// One batch = up to W sources (W = 32*WORDS status bits per vertex).  Per
// vertex v the status word holds bit s when source s has reached v.  Two
// copies are kept: `last` (status after the previous level) and `curr` (the
// status being built); after every level the vertices whose word changed
// are fixed up (last = curr) so that curr == last holds for every vertex at
// the start of a level.  Reference: comp_t status words and
// depth_comp_last/curr (comm.h:44, allocator.cuh:51-52).
//
// A level is three phases, separated by barriers (grid barriers inside the
// persistent kernel, kernel boundaries in the plain schedule):
//   expand   top-down push over the joint frontier queues (expander.cuh:
//            140-331) or bottom-up pull over all vertices (expander.cuh:
//            341-489); changed vertices go to a 1-bit-per-vertex bitmap
//            (V/8 bytes, L2 resident), double-buffered by level parity so
//            that the bottom-up pull can skip neighbours outside the previous
//            frontier, and on thin top-down levels also to a list (td_kind);
//   inspect  takes the changed vertices (from the list, the bitmap or a
//            sweep): new bits = curr & ~last, last = curr, ORs the new bits
//            into the depth bit-planes of the level number, and accumulates
//            the direction-switch counters; bottom-up levels do this work in
//            the pull itself.  Replaces the O(V) count/scan/gather passes of
//            inspector.cuh:63-525, scan.cuh:455-655 and the per-level
//            depth_merge writes of inspector.cuh:8-56,113-120;
//   qbuild   (only before a top-down level whose queues no thin inspect left
//            behind) turns the bitmap into the small/medium/large queues
//            (replaces td_frontier_count/td_frontier_gather).
// After the last level one pass turns the bit-planes into the depth output
// (either layout), writing every output byte exactly once.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ibfs {

constexpr int kDirTD = 0;
constexpr int kDirBU = 1;
constexpr int kMaxWords = 8;   // W = 256
constexpr int kMaxPlanes = 16; // two-byte depths

// Per-level counters, one of three sets per level (par_at): while level L runs,
// L-1's set is still read and L+1's is being zeroed.
struct Par {
  unsigned long long changed;  // vertices whose status changed
  unsigned long long mf;       // sum of their degrees (frontier edges)
  unsigned long long cdeg;     // sum of degrees of vertices that became complete
  unsigned long long teps;     // sum over new (v, s) pairs of deg(v)
  uint32_t fmask[kMaxWords];   // OR of all new bits (sources still expanding)
  int32_t range_err;           // a level did not fit the depth type
  int32_t hq_cnt;              // deferred bottom-up hub chunks of this level
  int32_t pq_cnt;              // queued sparse-source push chunks of this level
  int32_t t_cnt;               // vertices in the touched list of this level
};

// State of the level loop when it runs as kernels inside a CUDA graph (the
// device-driven schedule): what the persistent kernel keeps in registers
// lives here between kernels.
struct LoopState {
  long long n_total;  // sources of the run (set by the host before the launch)
  int32_t nbatches;   // batches of the run (set by the host before the launch)
  int32_t batch;      // batch the group is traversing
  int32_t level;      // level being expanded / inspected
  int32_t dir;        // direction of `level`
  int32_t max_level;
  int32_t td, bu;
  int32_t err;
  int32_t flip;       // 1: the status "last" lives in GroupBufs::curr and vice versa
  int32_t sync;       // the next top-down level first copies new statuses over old ones
  int32_t nb;         // sources of `batch`
  uint32_t smask[kMaxWords];  // bottom-up level: sources pushed top-down instead
  int32_t tail_clean;         // both status buffers are zero from v_reach on
                              // (batch_end clears its unreachable sources' words)
  int32_t sparse_try;         // this bottom-up level follows a top-down one: count
                              // the sources' frontiers and pick the sparse ones
  int32_t kind;               // how `level` keeps track of its changed vertices (td_kind)
  int32_t have_q;             // the queues of `level` were built by the previous inspect
  unsigned long long m_u, teps, prev_changed;
  unsigned long long t_lvl, t_mid;  // %globaltimer at the level start / inspect start
};

// Control block of one group (one batch at a time).  256-byte aligned.
struct __align__(256) Ctl {
  unsigned int bar_count;  // barrier arrivals of the run so far
  int err;
  int pad0[2];
  Par par[3];
  int32_t tail_src;  // a source of the batch lies at or past Params::v_reach
  __align__(16) int32_t qc[2][4];  // [consumer level parity][small, medium, large-chunks]
  unsigned long long pad1[4];
  LoopState ls;
};

__host__ __device__ inline Par* par_at(Ctl* ctl, int level) { return &ctl->par[level % 3]; }

struct BatchRec {
  int32_t levels;     // levels expanded (incl. the last empty one)
  int32_t max_level;  // deepest level with a new vertex
  int32_t td, bu;
  unsigned long long teps;
  int32_t err;
  int32_t pad;
};

struct LevelRec {
  int32_t batch, level, dir, pad;
  long long frontier, frontier_edges;
  long long expand_ns, inspect_ns;  // device time of the level's phases (persistent)
};

struct GroupBufs {
  uint32_t* last;    // [Vpad][WORDS]
  uint32_t* curr;    // [Vpad][WORDS]
  uint32_t* chg;     // 2 bitmaps of chg_stride words (level parity)
  uint32_t* planes;  // depth bit-planes, plane b at b*plane_stride words
  int32_t* q;        // [V] frontier queue: small vertices from the front, medium
                     // ones from the back (a vertex is in one class only)
  int32_t* tl;       // [V] touched list of a thin top-down level; on a bottom-up
                     // level that picks sparse sources, its first W entries
                     // count each source's previous frontier
  int2* ql;
  int2* hq;          // deferred bottom-up hub chunks (v, chunk)
  Ctl* ctl;
};

struct Params {
  const int64_t* beg;
  const int32_t* col;
  int64_t V, E, nchg;
  long long chg_stride;    // words per bitmap (nchg rounded up to 4)
  long long plane_stride;  // words per bit-plane (Vpad * WORDS)
  const int32_t* src;      // ordered sources [n_total]
  const int32_t* out_row;  // output row of ordered source k (source-major)
  int64_t n_total;
  int C, nbatches, G, cpg;
  int db;                  // depth bytes
  int layout;              // 0 source-major, 1 vertex-major
  uint8_t* out;            // device output
  int sml, lrg, chunk, but;
  int switch_level;
  float alpha, beta;
  int max_levels;
  unsigned long long timeout_ns;
  int withhold;
  GroupBufs* groups;
  BatchRec* brec;
  LevelRec* lrec;
  int lrec_cap;
  int vec_sm;   // source-major rows allow vector stores of this many bytes: 16 (V % 16
                // == 0, 16-byte aligned base), 4 (V % 4 == 0, 4-byte aligned) or 0
  int td_stage;     // top-down stages large vertices' chunks by bulk copies
  int sparse_div;   // device loop: a bottom-up level pushes, top-down, the sources
                    // whose previous frontier is below 1/sparse_div of the average
                    // (0: off; see sparse_count_phase)
  int bu_filter;    // bottom-up skips neighbours outside the previous frontier:
                    // 1 always, 0 never, -1 on levels whose previous frontier
                    // is small (bu_filter_level)
  int col_vec;      // col is 16-byte aligned and padded by 4 entries (vector reads)
  int hub_t;        // bottom-up: a warp scans at most hub_t neighbours of a vertex;
                    // a hub still missing bits defers the rest in chunks
  const int32_t* vmap;  // caller id -> internal id of the resident graph (null:
                        // identical); the output pass reads statuses through it
  long long v_nz;       // bottom-up sweeps [0, v_nz): in the degree order the
                        // vertices from v_nz on have no edges (v_nz a multiple
                        // of 32, or V); a bottom-up pass cannot change them and
                        // a top-down level (a directed graph's sinks) writes
                        // both status buffers through inspect, so they agree
  long long v_reach;    // v_nz when no edge points into [v_nz, V) (symmetric
                        // graphs), else V: vertices from v_reach on are reached
                        // only as sources, at depth 0
  long long big_prefix; // bottom-up: vertices [0, big_prefix) are spread over all warps
                        // (degree-ordered graphs: the vertices above the
                        // thread-path limit; a multiple of 32, at most V; 0
                        // otherwise)
  int32_t* done_flags;  // per batch, in mapped host memory: 1 once the batch's
                        // depths are complete in `out` (device loop), so that
                        // the host can stream them out while later batches run
  // Serving queue (device loop, q_slots > 0): batches are not a fixed list
  // but slots of a ring that the host fills while the graph runs.  The host
  // writes a slot's sources (internal ids), output rows and count, then
  // raises q_tail; a group that finishes a batch claims the next published
  // one (q_head, compare-and-swap), copies the slot into src/out_row (device
  // arrays of q_slots * C entries) and marks it 1 in q_state; after its
  // output pass it writes brec[slot] and marks it 2.  A group that finds no
  // published batch ends its batch loop; the host relaunches the graph for
  // batches published after every group ended.
  int q_slots;
  const long long* q_tail;      // mapped host memory: batches published
  const int32_t* q_n;           // mapped host memory [q_slots]: sources per slot
  const int32_t* q_src;         // mapped host memory [q_slots * C]
  const int32_t* q_rows;        // mapped host memory [q_slots * C]
  int32_t* q_state;             // mapped host memory [q_slots]: 1 claimed, 2 done
  unsigned long long* q_head;   // device memory: batches claimed
  unsigned long long q_wait_ns; // a group that finds no published batch waits this
                                // long for one (%globaltimer) before ending
};

// Neighbours one thread of the bottom-up thread path has in flight per step
// (4 or 8).
#ifndef IBFS_BU_STEP
#define IBFS_BU_STEP 4
#endif
constexpr int kBuStep = IBFS_BU_STEP;
// Steps of kBuStep neighbours a big vertex (degree above the thread-path
// limit) scans on its own lane before the warp takes it (0: none).
#ifndef IBFS_BU_PEEK
#define IBFS_BU_PEEK 2
#endif
constexpr int kBuPeek = IBFS_BU_PEEK;

// Bottom-up frontier filter.  A neighbour u that did not change at level L-1
// cannot give v a bit it lacks at level L: every bit u held before L-1
// reached v by L-1 already (BFS distances of adjacent vertices differ by at
// most one).  So the scan may skip, exactly, every neighbour outside the
// level-(L-1) changed bitmap.  The bitmap test costs a lookup per neighbour;
// it can pay off when the previous frontier is a small part of the graph
// (the tail levels of a traversal), not when it is a large part.
constexpr long long kFilterDiv = 16;  // auto: filter when prev frontier < V / 16
__host__ __device__ inline bool bu_filter_level(int mode, unsigned long long prev_changed,
                                                long long V) {
  if (mode >= 0) return mode > 0;
  return (long long)prev_changed * kFilterDiv < V;
}

// Whether u is in the previous level's changed bitmap; through L1 when the
// pass runs as a kernel of its own (RO: nothing writes that bitmap while it
// runs), else through L2 (the persistent kernel rewrites it at later levels).
template <bool RO>
__device__ __forceinline__ bool in_front(const uint32_t* front, int32_t u) {
  const uint32_t w = RO ? __ldg(front + (u >> 5)) : __ldcg(front + (u >> 5));
  return (w >> (u & 31)) & 1u;
}

// How a top-down level keeps track of the vertices it changes.
//   thin   a list: the first push to change a vertex appends it (one returned
//          atomic), and the inspect step, which reads only the list, queues the
//          next level on the way;
//   bitmap every push that adds bits marks its vertex;
//   wide   nothing: the inspect step compares every vertex's two statuses, in
//          one coalesced sweep, and writes the bitmap itself.
// What a level costs beside its pushes: one appended counter (thin), one more
// reduction per push (bitmap), a sweep of 32 to 64 bytes per reachable vertex
// (wide).  So a frontier of at most 2^20 edges is thin -- with the limit at
// 2^17 / 2^20 / 2^23 edges R-MAT scale 22, 512 sources takes 5.10 / 5.06 / 5.14
// ms, a grid of 4096^2, 256 sources 156.1 / 154.1 / 157.9 ms, R-MAT scale
// 20, 60 sources in 32-bit words 1.55 / 1.56 / 1.61 ms -- and one with an edge
// per two reachable vertices is wide -- at 1/4 / 1 / 4 edges per vertex
// scale 22 takes 4.40 / 4.48 / 4.65 ms, the grid 153.7 / 152.9 / 152.8 ms,
// scale 20 0.79 / 0.79 / 0.84 ms.  The pushes are bound by L2's reductions:
// without the bitmap's the level that pushes 30 M edges of the social graph
// went from 609 to 354 us, its inspect step from 100 to 61 us (coalesced).
constexpr int kTdBitmap = 0;
constexpr int kTdThin = 1;
constexpr int kTdWide = 2;
constexpr unsigned long long kThinEdges = 1ull << 20;
__host__ __device__ inline int td_kind(unsigned long long mf, long long v_reach) {
  if (mf <= kThinEdges) return kTdThin;
  return mf * 2 >= (unsigned long long)v_reach ? kTdWide : kTdBitmap;
}
// The kind of the next level by its direction: a bottom-up pass marks the
// bitmap, which is what an inspect step of its own has to walk.
__host__ __device__ inline int level_kind(int dir, unsigned long long mf, long long v_reach) {
  return dir == kDirTD ? td_kind(mf, v_reach) : kTdBitmap;
}

constexpr int kHubScan = 1024;   // neighbours one warp scans before deferring
constexpr int kHubChunk = 2048;  // edges per deferred chunk (one CTA each)

// Bottom-up positions inside one list are 32 bits (registers are what the
// sweep is short of: 64-bit ones cost the grid and the 256-bit runs 2 %).  Only
// a list with duplicates can be longer than kListMax, which leaves room for a
// step of 128 past the end; a graph that has one runs every level top-down,
// where positions are 64 bits.
constexpr long long kListMax = 0x7FFFF000;
__host__ __device__ inline int switch_level_for(int switch_level, long long max_deg) {
  return max_deg > kListMax ? 0x7FFFFFFF : switch_level;
}

// Neighbour statuses of a bottom-up pass that runs as a kernel of its own
// (RO: nothing writes `last` while it runs) are read through L1 (ld.global.nc):
// most gathers hit the few hub words that the degree order packs into the
// first lines of `last`, and L1 serves them instead of L2.  Measured on
// R-MAT scale 24, one batch at a time: bottom-up 25.1 -> 19.4 ms per
// 1024-source run.  The persistent kernel, whose other phases write `last`
// within the same launch, must not use that path; its sweep reads `last` by
// ordinary cached loads (ld_status_ca), its deferred hub chunks through L2.
#ifndef IBFS_BU_NC
#define IBFS_BU_NC 1
#endif

// A team is the set of threads that share one batch: the whole grid in the
// plain schedule, the CTAs of one group in the persistent kernel.
struct Team {
  int block, nblocks;  // CTA index inside the team, team size in CTAs
  long long tid, nthreads;
  long long warp, nwarps;
  int lane;
};

__host__ __device__ inline uint32_t* chg_at(const GroupBufs& gb, const Params& p, int level) {
  return gb.chg + (level & 1) * p.chg_stride;
}

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
template <int WORDS>
__device__ __forceinline__ void ld_status(const uint32_t* p, uint32_t (&x)[WORDS]) {
  if constexpr (WORDS == 1) {
    x[0] = __ldcg(p);
  } else if constexpr (WORDS == 2) {
    uint2 t = __ldcg(reinterpret_cast<const uint2*>(p));
    x[0] = t.x; x[1] = t.y;
  } else if constexpr (WORDS == 4) {
    uint4 t = __ldcg(reinterpret_cast<const uint4*>(p));
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else {
    uint4 a = __ldcg(reinterpret_cast<const uint4*>(p));
    uint4 b = __ldcg(reinterpret_cast<const uint4*>(p) + 1);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
}

template <int WORDS>
__device__ __forceinline__ void st_status(uint32_t* p, const uint32_t (&x)[WORDS]) {
  if constexpr (WORDS == 1) {
    __stcg(p, x[0]);
  } else if constexpr (WORDS == 2) {
    __stcg(reinterpret_cast<uint2*>(p), make_uint2(x[0], x[1]));
  } else if constexpr (WORDS == 4) {
    __stcg(reinterpret_cast<uint4*>(p), make_uint4(x[0], x[1], x[2], x[3]));
  } else {
    __stcg(reinterpret_cast<uint4*>(p), make_uint4(x[0], x[1], x[2], x[3]));
    __stcg(reinterpret_cast<uint4*>(p) + 1, make_uint4(x[4], x[5], x[6], x[7]));
  }
}

// Status read through the non-coherent (L1) path: only for buffers that no
// thread writes while the kernel runs (`last` during a fused bottom-up pass).
template <int WORDS>
__device__ __forceinline__ void ld_status_nc(const uint32_t* p, uint32_t (&x)[WORDS]) {
  if constexpr (WORDS == 1) {
    x[0] = __ldg(p);
  } else if constexpr (WORDS == 2) {
    uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
    x[0] = t.x; x[1] = t.y;
  } else if constexpr (WORDS == 4) {
    uint4 t = __ldg(reinterpret_cast<const uint4*>(p));
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else {
    uint4 a = __ldg(reinterpret_cast<const uint4*>(p));
    uint4 b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
}

// Status read through L1 inside the persistent kernel, only for a buffer that
// no thread writes during the phase: the team barrier before the phase (release
// by every CTA, acquire by every CTA, then a CTA barrier) makes the earlier
// writes visible to ordinary cached loads.
template <int WORDS>
__device__ __forceinline__ void ld_status_ca(const uint32_t* p, uint32_t (&x)[WORDS]) {
  if constexpr (WORDS == 1) {
    x[0] = __ldca(p);
  } else if constexpr (WORDS == 2) {
    uint2 t = __ldca(reinterpret_cast<const uint2*>(p));
    x[0] = t.x; x[1] = t.y;
  } else {
#pragma unroll
    for (int q = 0; q < WORDS / 4; q++) {
      uint4 t = __ldca(reinterpret_cast<const uint4*>(p) + q);
      x[4 * q] = t.x; x[4 * q + 1] = t.y; x[4 * q + 2] = t.z; x[4 * q + 3] = t.w;
    }
  }
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_volatile_i32(const int* p) {
  return *reinterpret_cast<const volatile int*>(p);
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bit mask of the sources of a batch of n inside word k.
__host__ __device__ __forceinline__ uint32_t full_word(int n, int k) {
  const int lo = k * 32;
  if (n >= lo + 32) return 0xFFFFFFFFu;
  if (n <= lo) return 0u;
  return (1u << (n - lo)) - 1u;
}

// Number of depth bit-planes that levels 0..max_level use.
__host__ __device__ __forceinline__ int planes_for(int max_level) {
  int p = 0;
  while (p < 31 && (max_level >> p) != 0) p++;
  return p;
}

// Bounded team barrier.  Every CTA adds one to a counter that only grows
// (the host zeroes it before a run) and waits for the barrier's own target
// on that counter, so the last arrival releases the waiters directly: one
// reduction and one polled line, instead of a returned atomic, a reset and a
// release store.  All waits end: after timeout_ns the waiting CTA records
// IBFS_ERR_TIMEOUT (6) in ctl->err, and the others leave on seeing it.
// Returns false when the team must stop.
static __device__ __noinline__ bool team_barrier(Ctl* ctl, unsigned nblocks, unsigned target,
                                                 unsigned long long timeout_ns,
                                                 bool withhold) {
  __shared__ int s_ok;
  if (nblocks == 1 && !withhold) {  // a team of one CTA
    __syncthreads();
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    if (!withhold)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->bar_count) : "memory");
    unsigned long long t0 = 0;
    for (unsigned spin = 1; (int)(ld_acquire_u32(&ctl->bar_count) - target) < 0; spin++) {
      if (spin & 63u) continue;
      if (ld_volatile_i32(&ctl->err) != 0) { ok = 0; break; }
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > timeout_ns) {
        atomicCAS(&ctl->err, 0, 6);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// A level's counters, summed over the CTA and added to `par` (every thread
// calls it).  A CTA that changed nothing -- most of them on a thin level --
// leaves after one barrier; otherwise the warps' sums meet in shared memory
// behind a second one and one thread per counter issues its atomic.
template <int WORDS>
__device__ __forceinline__ void cta_flush(Par* par, unsigned long long cnt, unsigned long long mf,
                                          unsigned long long cdeg, unsigned long long teps,
                                          const uint32_t (&fm)[WORDS]) {
  __shared__ unsigned long long s_c[32][4];
  __shared__ uint32_t s_f[32][WORDS];
  bool any = cnt != 0;
#pragma unroll
  for (int k = 0; k < WORDS; k++) any |= fm[k] != 0u;
  if (!__syncthreads_or(any)) return;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (__any_sync(0xFFFFFFFFu, any)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
      mf += __shfl_xor_sync(0xFFFFFFFFu, mf, o);
      cdeg += __shfl_xor_sync(0xFFFFFFFFu, cdeg, o);
      teps += __shfl_xor_sync(0xFFFFFFFFu, teps, o);
    }
    if (l == 0) {
      s_c[w][0] = cnt;
      s_c[w][1] = mf;
      s_c[w][2] = cdeg;
      s_c[w][3] = teps;
    }
#pragma unroll
    for (int k = 0; k < WORDS; k++) {
      const uint32_t r = __reduce_or_sync(0xFFFFFFFFu, fm[k]);
      if (l == 0) s_f[w][k] = r;
    }
  } else {
    if (l < 4) s_c[w][l] = 0;
    if (l < WORDS) s_f[w][l] = 0;
  }
  __syncthreads();
  const int nw = blockDim.x >> 5;
  if (threadIdx.x < 4) {
    unsigned long long t = 0;
    for (int i = 0; i < nw; i++) t += s_c[i][threadIdx.x];
    unsigned long long* dst = threadIdx.x == 0   ? &par->changed
                              : threadIdx.x == 1 ? &par->mf
                              : threadIdx.x == 2 ? &par->cdeg
                                                 : &par->teps;
    if (t) atomicAdd(dst, t);
  } else if (threadIdx.x >= 32 && threadIdx.x < 32 + WORDS) {
    uint32_t t = 0;
    for (int i = 0; i < nw; i++) t |= s_f[i][threadIdx.x - 32];
    if (t) atomicOr(&par->fmask[threadIdx.x - 32], t);
  }
}

// Per-source counts of a level's new bits, for the sparse-source decision:
// shared-memory counters per CTA (every thread calls scnt_begin and
// scnt_flush), one atomic add per counted (vertex, source) pair.
__device__ __forceinline__ void scnt_begin(uint32_t* s_cnt) {
  for (int i = threadIdx.x; i < kMaxWords * 32; i += blockDim.x) s_cnt[i] = 0u;
  __syncthreads();
}
template <int WORDS>
__device__ __forceinline__ void scnt_flush(const uint32_t* s_cnt, int32_t* dst) {
  __syncthreads();
  for (int i = threadIdx.x; i < WORDS * 32; i += blockDim.x)
    if (s_cnt[i]) atomicAdd(&dst[i], (int)s_cnt[i]);
}

__device__ __forceinline__ void zero_words(uint32_t* p, long long nwords, const Team& t) {
  // nwords is a multiple of 4 and p 16-byte aligned (allocation padding)
  uint4* q = reinterpret_cast<uint4*>(p);
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (long long i = t.tid; i < nwords / 4; i += t.nthreads) __stcg(q + i, z);
}

// One warp zeroes a level's counters, a word per lane and step.  (A memset by
// one thread became a chain of byte stores: 67 us for the three sets of a
// batch, which was half of a small run.)
__device__ __forceinline__ void zero_par(Par* par, int lane) {
  static_assert(sizeof(Par) % 8 == 0, "whole words");
  unsigned long long* q = reinterpret_cast<unsigned long long*>(par);
  for (int i = lane; i < (int)(sizeof(Par) / 8); i += 32) q[i] = 0ull;
}

// ---------------------------------------------------------------------------
// Direction choice for the next level (host and device use the same rule).
//   fixed (switch_level >= 0): top-down while level <= switch_level, then
//     bottom-up -- the reference's CLI switch level (expander.cuh:687-723);
//   alpha/beta (Beamer et al., SC'12): top-down -> bottom-up when the
//     frontier's edges exceed unexplored_edges/alpha and the frontier is
//     growing; bottom-up -> top-down when the frontier holds fewer than
//     V/beta vertices and is shrinking.  Without the growing/shrinking
//     tests a long shrinking tail (high-diameter graphs) flips direction
//     every level once the unexplored edges run low, paying a full
//     bottom-up sweep for a handful of frontier vertices.
// ---------------------------------------------------------------------------
__host__ __device__ inline int choose_dir(int next_level, int prev_dir,
                                          int switch_level, float alpha,
                                          float beta, unsigned long long changed,
                                          unsigned long long prev_changed,
                                          unsigned long long mf,
                                          unsigned long long m_u, long long V) {
  if (switch_level >= 0) return next_level <= switch_level ? kDirTD : kDirBU;
  if (prev_dir == kDirTD)
    return ((double)mf * (double)alpha > (double)m_u && changed > prev_changed) ? kDirBU
                                                                                : kDirTD;
  return ((double)changed * (double)beta < (double)V && changed < prev_changed) ? kDirTD
                                                                                : kDirBU;
}

// ---------------------------------------------------------------------------
// Phase: seed the sources of one batch (curr bits + level-0 changed bits, and
// the touched list when the schedule inspects level 0 from it).
// ---------------------------------------------------------------------------
template <int WORDS, bool THIN>
__device__ void seed_phase(const Params& p, const GroupBufs& gb,
                           const int32_t* src_b, int n_b, const Team& t) {
  uint32_t* chg0 = chg_at(gb, p, 0);
  for (long long i = t.tid; i < n_b; i += t.nthreads) {
    const int32_t v = src_b[i];
    atomicOr(gb.curr + (size_t)v * WORDS + (i >> 5), 1u << (i & 31));
    if (v >= p.v_reach) gb.ctl->tail_src = 1;
    const uint32_t bit = 1u << (v & 31);
    const uint32_t old = atomicOr(chg0 + (v >> 5), bit);
    if (THIN && !(old & bit)) gb.tl[atomicAdd(&gb.ctl->par[0].t_cnt, 1)] = v;
  }
}

// Zero depth bit-plane b when `level` = 2^b, the first level that uses it.
__device__ __forceinline__ void zero_plane_if_first(const Params& p, const GroupBufs& gb,
                                                    int level, const Team& t) {
  if (level > 0 && (level & (level - 1)) == 0) {
    const int b = __ffs(level) - 1;
    zero_words(gb.planes + (size_t)b * p.plane_stride, p.plane_stride, t);
  }
}

// Fire-and-forget ORs (red: no value comes back, so nothing waits on them).
__device__ __forceinline__ void red_or_u32(uint32_t* p, uint32_t x) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}
__device__ __forceinline__ void red_or_u64(unsigned long long* p, unsigned long long x) {
  asm volatile("red.relaxed.gpu.global.or.b64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
}

// Inspect work of one changed vertex v of level L: new bits, last = curr,
// counters, planes; deg = its degree.
// RED: the planes take the bits as reductions, with nothing to wait for.  A
// thin level is a chain of dependent accesses, and a read-modify-write per
// pair of set bits of the level number would be most of it; the other levels
// move whole lines either way and keep the loads and stores.
template <int WORDS, bool RED>
__device__ __forceinline__ void inspect_vertex(const Params& p, const GroupBufs& gb, long long v,
                                               int level, bool depth_ok,
                                               const uint32_t (&full)[WORDS], uint32_t (&fm)[WORDS],
                                               unsigned long long& mf, unsigned long long& cnt,
                                               unsigned long long& cdeg,
                                               unsigned long long& teps, long long& deg,
                                               const uint32_t (&c)[WORDS],
                                               const uint32_t (&l)[WORDS]) {
  uint32_t nb[WORDS];
  bool comp = true;
  uint32_t pop = 0;
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    nb[k] = c[k] & ~l[k];
    comp = comp && (c[k] == full[k]);
    pop += __popc(nb[k]);
    fm[k] |= nb[k];
  }
  st_status<WORDS>(gb.last + (size_t)v * WORDS, c);
  deg = p.beg[v + 1] - p.beg[v];
  mf += deg;
  cnt += 1;
  teps += (unsigned long long)deg * pop;
  if (comp) cdeg += deg;
  if (depth_ok) {
    // depth(v, s) = level for the new bits: OR them into the planes of the
    // level's set bits (one coalesced read-modify-write per plane), two
    // planes at a time so that their loads are in flight together.
    uint32_t* q0 = gb.planes + (size_t)v * WORDS;
    unsigned rest = (unsigned)level;
    while (RED && rest) {
      const int b0 = __ffs(rest) - 1;
      rest &= rest - 1;
      uint32_t* qa = q0 + (size_t)b0 * p.plane_stride;
      if constexpr (WORDS == 1) {
        red_or_u32(qa, nb[0]);
      } else {
#pragma unroll
        for (int k = 0; k < WORDS / 2; k++) {
          const unsigned long long w = ((unsigned long long)nb[2 * k + 1] << 32) | nb[2 * k];
          if (w) red_or_u64(reinterpret_cast<unsigned long long*>(qa) + k, w);
        }
      }
    }
    while (!RED && rest) {
      const int b0 = __ffs(rest) - 1;
      rest &= rest - 1;
      uint32_t* qa = q0 + (size_t)b0 * p.plane_stride;
      uint32_t xa[WORDS];
      ld_status<WORDS>(qa, xa);
      if (rest) {
        const int b1 = __ffs(rest) - 1;
        rest &= rest - 1;
        uint32_t* qb = q0 + (size_t)b1 * p.plane_stride;
        uint32_t xb[WORDS];
        ld_status<WORDS>(qb, xb);
#pragma unroll
        for (int k = 0; k < WORDS; k++) xb[k] |= nb[k];
        st_status<WORDS>(qb, xb);
      }
#pragma unroll
      for (int k = 0; k < WORDS; k++) xa[k] |= nb[k];
      st_status<WORDS>(qa, xa);
    }
  }
}

// ---------------------------------------------------------------------------
// Changed-vertex bitmap walk.  A warp takes `wpc` bitmap words per step and
// writes the ids of their set bits, compacted, into its own piece of shared
// memory, so that all lanes have a changed vertex in every full round of 32,
// however thinly the set is spread.  wpc is kWalkWords on large graphs; on
// small ones it
// shrinks until every warp of the team has a step, because a step's rounds
// are serial.  body(first vertex, ids, count) runs once per step.  A step is
// 8 words: the lists of 16 warps then take 8 KB, so that the walks leave L1 to
// the bottom-up kernels that share the SM with them (four groups of R-MAT
// scale 24: 29.9 / 29.6 / 29.4 ms per run with steps of 32 / 16 / 8 words).
// ---------------------------------------------------------------------------
constexpr int kWalkWords = 8;                     // bitmap words of one step at most
constexpr int kWalkIds = kWalkWords * 32;         // ids of one step at most
constexpr int kWalkWarps = 16;                    // warps per CTA at most (512 threads)

__device__ __forceinline__ int walk_words(long long nchg, long long nwarps) {
  int w = kWalkWords;
  while (w > 1 && nchg < (long long)w * nwarps) w >>= 1;
  return w;
}

// One warp's piece of the id lists (a function of its own, so that every walk
// of a kernel shares one array).
__device__ __forceinline__ uint16_t* walk_ids() {
  __shared__ uint16_t s_ids[kWalkWarps][kWalkIds];
  return s_ids[threadIdx.x >> 5];
}

template <class Body>
__device__ __forceinline__ void walk_changed(const uint32_t* chg, long long nchg, const Team& t,
                                             Body&& body) {
  uint16_t* ids = walk_ids();
  const int lane = t.lane;
  const int wpc = walk_words(nchg, t.nwarps);
  const long long nstep = (nchg + wpc - 1) / wpc;
  for (long long c = t.warp; c < nstep; c += t.nwarps) {
    const long long w = c * wpc + lane;
    uint32_t word = (lane < wpc && w < nchg) ? __ldcg(chg + w) : 0u;
    if (__ballot_sync(0xFFFFFFFFu, word != 0u) == 0u) continue;
    const int own = __popc(word);
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    int at = incl - own;
    while (word) {
      ids[at++] = (uint16_t)(lane * 32 + __ffs(word) - 1);
      word &= word - 1;
    }
    __syncwarp();
    body(c * wpc * 32, ids, total);
    __syncwarp();  // the next step overwrites ids
  }
}

// Degree class of a frontier vertex (td_inspect, inspector.cuh:534-626):
// deg < sml -> small (0), deg > lrg -> large (2), else medium (1); vertices
// without edges are dropped (-1).
__device__ __forceinline__ int deg_class(const Params& p, long long deg) {
  return deg <= 0 ? -1 : deg < p.sml ? 0 : deg <= p.lrg ? 1 : 2;
}

// Append one vertex per lane (cls -1: none) to the queues: ballots, and one
// atomic per class, the three of them issued together by three lanes.
__device__ __forceinline__ void q_append(const Params& p, const GroupBufs& gb, int32_t* qc,
                                         int lane, int32_t v, long long deg, int cls) {
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, cls == 0);
  const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, cls == 1);
  const uint32_t m2 = __ballot_sync(0xFFFFFFFFu, cls == 2);
  if (!(m0 | m1 | m2)) return;
  int nch = 0, incl = 0, total = 0;
  if (m2) {  // large vertices are cut into chunks of p.chunk edges
    nch = cls == 2 ? (int)((deg + p.chunk - 1) / p.chunk) : 0;
    incl = nch;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  const int add = lane == 0 ? __popc(m0) : lane == 1 ? __popc(m1) : lane == 2 ? total : 0;
  int base = 0;
  if (add) base = atomicAdd(&qc[lane], add);
  const int b0 = __shfl_sync(0xFFFFFFFFu, base, 0);
  const int b1 = __shfl_sync(0xFFFFFFFFu, base, 1);
  const int b2 = __shfl_sync(0xFFFFFFFFu, base, 2);
  if (cls == 0) gb.q[b0 + __popc(m0 & lt)] = v;
  else if (cls == 1) gb.q[p.V - 1 - (b1 + __popc(m1 & lt))] = v;
  else if (cls == 2)
    for (int c = 0; c < nch; c++) gb.ql[b2 + incl - nch + c] = make_int2(v, c);
}

// ---------------------------------------------------------------------------
// Phase: inspect level L.  Takes the changed vertices from the list, the
// bitmap or a sweep (td_kind), fixes last, and updates the depth bit-planes
// and the counters.  What bounds a thin level is its chain of dependent L2
// reads (queue entry, offsets, column id, status, then list entry, statuses,
// planes), so the step is one vertex per lane and 8 lanes per pushed small
// vertex.  A 256 x 1024 grid without shortcuts (64 sources, 1269 levels, about
// 12,500 vertices each) went from 144 to 34 ms when its levels stopped walking
// the whole bitmap with a few warps.
// ---------------------------------------------------------------------------
template <int WORDS>
__device__ void inspect_phase(const Params& p, const GroupBufs& gb, Par* par, int n_b,
                              int level, bool depth_ok, int kind, int32_t* qc_next,
                              const Team& t) {
  uint32_t full[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) full[k] = full_word(n_b, k);
  unsigned long long mf = 0, cnt = 0, cdeg = 0, teps = 0;
  uint32_t fm[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) fm[k] = 0;
  // the bitmap of level+1 (last used by level-1's expand) must start empty:
  // bottom-up merges into it with atomics
  zero_words(chg_at(gb, p, level + 1), p.chg_stride, t);
  const int lane = t.lane;
  if (kind == kTdThin) {
    const int n = __ldcg(&par->t_cnt);
    for (long long base = t.warp * 32; base < n; base += t.nwarps * 32) {
      int32_t v = -1;
      long long deg = 0;
      if (base + lane < n) {
        v = __ldcg(gb.tl + base + lane);
        uint32_t c[WORDS], l[WORDS];
        ld_status<WORDS>(gb.curr + (size_t)v * WORDS, c);
        ld_status<WORDS>(gb.last + (size_t)v * WORDS, l);
        inspect_vertex<WORDS, true>(p, gb, v, level, depth_ok, full, fm, mf, cnt, cdeg, teps, deg,
                                    c, l);
      }
      q_append(p, gb, qc_next, lane, v, deg, deg_class(p, deg));
    }
  } else if (kind == kTdWide) {
    uint32_t* chg = chg_at(gb, p, level);
    for (long long base = t.warp * 32; base < p.v_reach; base += t.nwarps * 32) {
      const long long v = base + lane;
      bool ch = false;
      if (v < p.V) {
        uint32_t c[WORDS], l[WORDS];
        ld_status<WORDS>(gb.curr + (size_t)v * WORDS, c);
        ld_status<WORDS>(gb.last + (size_t)v * WORDS, l);
#pragma unroll
        for (int k = 0; k < WORDS; k++) ch |= c[k] != l[k];
        long long deg;
        if (ch)
          inspect_vertex<WORDS, false>(p, gb, v, level, depth_ok, full, fm, mf, cnt, cdeg, teps,
                                       deg, c, l);
      }
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, ch);
      if (lane == 0 && bal) __stcg(chg + (base >> 5), bal);
    }
  } else {
    walk_changed(chg_at(gb, p, level), p.nchg, t,
                 [&](long long v0, const uint16_t* ids, int total) {
                   for (int r = lane; r < total; r += 32) {
                     const long long v = v0 + ids[r];
                     long long deg;
                     uint32_t c[WORDS], l[WORDS];
                     ld_status<WORDS>(gb.curr + (size_t)v * WORDS, c);
                     ld_status<WORDS>(gb.last + (size_t)v * WORDS, l);
                     inspect_vertex<WORDS, false>(p, gb, v, level, depth_ok, full, fm, mf, cnt,
                                                  cdeg, teps, deg, c, l);
                   }
                 });
  }
  if (!depth_ok && cnt) par->range_err = 1;
  cta_flush<WORDS>(par, cnt, mf, cdeg, teps, fm);
}

// ---------------------------------------------------------------------------
// Phase: build the joint frontier queues of top-down level L from the
// level-(L-1) bitmap.  The classes of a step's vertices are counted first,
// so that a step of up to 256 vertices costs one round of three atomics
// instead of one per 32 vertices.
// ---------------------------------------------------------------------------
// With `sync` (a top-down level right after a fused bottom-up level, which
// left the new statuses in `last` and the previous ones in `curr`) every
// changed vertex also copies last -> curr, restoring curr == last.
template <int WORDS = 4>
__device__ inline void qbuild_phase(const Params& p, const GroupBufs& gb, int level,
                                    int32_t* qc, const Team& t, bool sync = false) {
  const int lane = t.lane;
  const uint32_t lt = (1u << lane) - 1u;
  walk_changed(chg_at(gb, p, level - 1), p.nchg, t,
               [&](long long v0, uint16_t* ids, int total) {
    // count the classes; the class stays in the id's top bits
    int n0 = 0, n1 = 0, n2 = 0;
    for (int r0 = 0; r0 < total; r0 += 32) {
      int cls = -1, nch = 0;
      if (r0 + lane < total) {
        const uint32_t id = ids[r0 + lane];
        const long long v = v0 + id;
        const long long deg = p.beg[v + 1] - p.beg[v];
        if (sync) {
          uint32_t x[WORDS];
          ld_status<WORDS>(gb.last + (size_t)v * WORDS, x);
          st_status<WORDS>(gb.curr + (size_t)v * WORDS, x);
        }
        cls = deg_class(p, deg);
        if (cls == 2) nch = (int)((deg + p.chunk - 1) / p.chunk);
        ids[r0 + lane] = (uint16_t)(id | (uint32_t)(cls + 1) << 10);
      }
      n0 += __popc(__ballot_sync(0xFFFFFFFFu, cls == 0));
      n1 += __popc(__ballot_sync(0xFFFFFFFFu, cls == 1));
      if (__any_sync(0xFFFFFFFFu, cls == 2)) n2 += __reduce_add_sync(0xFFFFFFFFu, nch);
    }
    __syncwarp();
    const int add = lane == 0 ? n0 : lane == 1 ? n1 : lane == 2 ? n2 : 0;
    int base = 0;
    if (add) base = atomicAdd(&qc[lane], add);
    int b0 = __shfl_sync(0xFFFFFFFFu, base, 0);
    int b1 = __shfl_sync(0xFFFFFFFFu, base, 1);
    int b2 = __shfl_sync(0xFFFFFFFFu, base, 2);
    for (int r0 = 0; r0 < total; r0 += 32) {
      int cls = -1;
      int32_t v = 0;
      if (r0 + lane < total) {
        const uint32_t id = ids[r0 + lane];
        v = (int32_t)(v0 + (id & 1023u));
        cls = (int)(id >> 10) - 1;
      }
      const uint32_t m0 = __ballot_sync(0xFFFFFFFFu, cls == 0);
      const uint32_t m1 = __ballot_sync(0xFFFFFFFFu, cls == 1);
      if (cls == 0) gb.q[b0 + __popc(m0 & lt)] = v;
      if (cls == 1) gb.q[p.V - 1 - (b1 + __popc(m1 & lt))] = v;
      b0 += __popc(m0);
      b1 += __popc(m1);
      if (__any_sync(0xFFFFFFFFu, cls == 2)) {
        const int nch =
            cls == 2 ? (int)((p.beg[v + 1] - p.beg[v] + p.chunk - 1) / p.chunk) : 0;
        int incl = nch;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= o) incl += y;
        }
        for (int c = 0; c < nch; c++) gb.ql[b2 + incl - nch + c] = make_int2(v, c);
        b2 += __shfl_sync(0xFFFFFFFFu, incl, 31);
      }
    }
  });
}

// Top-down edges: push the frontier word P of v into neighbours u[0..cnt).
// The status reads of all cnt neighbours are issued before any of them is
// used, so one thread has cnt gathers in flight instead of one.
// The status read s (through L2) decides everything: every level starts
// with curr == last, so bits of P missing from s are missing from last[u],
// and once ORed in (by this thread or a concurrent one) u has changed at
// this level.  So the ORs into curr[u] and into the changed bitmap are
// reductions whose old value is never needed: the thread issues them and
// goes on instead of waiting for L2 round trips.  A stale s (fewer bits)
// costs at most one redundant OR.
//
// Thin levels (td_kind): the bitmap OR returns the old word,
// which says whether this push was the first to change u at this level, and
// the warp appends those vertices to the list with one atomic per step.  All
// 32 lanes call it together (cnt 0: nothing to push).
constexpr int kTdStep = 4;  // edges one thread has in flight
template <int WORDS, int KIND>
__device__ __forceinline__ void td_push_n(const GroupBufs& gb, uint32_t* chg, int32_t* t_cnt,
                                          const int32_t (&u)[kTdStep], int cnt,
                                          const uint32_t (&P)[WORDS]) {
  uint32_t first = 0;  // bit i: u[i] changed here first
  uint32_t s[kTdStep][WORDS];
#pragma unroll
  for (int i = 0; i < kTdStep; i++) {
    if (i < cnt) {
      ld_status<WORDS>(gb.curr + (size_t)u[i] * WORDS, s[i]);
    } else {
#pragma unroll
      for (int k = 0; k < WORDS; k++) s[i][k] = 0xFFFFFFFFu;
    }
  }
#pragma unroll
  for (int i = 0; i < kTdStep; i++) {
    bool need = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) need |= (P[k] & ~s[i][k]) != 0u;
    if (!need) continue;
    if constexpr (WORDS == 1) {
      red_or_u32(gb.curr + u[i], P[0]);
    } else {
      unsigned long long* q = reinterpret_cast<unsigned long long*>(gb.curr + (size_t)u[i] * WORDS);
#pragma unroll
      for (int k = 0; k < WORDS / 2; k++) {
        const uint32_t n0 = P[2 * k] & ~s[i][2 * k], n1 = P[2 * k + 1] & ~s[i][2 * k + 1];
        if (n0 | n1) red_or_u64(q + k, ((unsigned long long)P[2 * k + 1] << 32) | P[2 * k]);
      }
    }
    const uint32_t bit = 1u << (u[i] & 31);
    if constexpr (KIND == kTdThin) {
      if (!(atomicOr(chg + (u[i] >> 5), bit) & bit)) first |= 1u << i;
    } else if constexpr (KIND == kTdBitmap) {
      red_or_u32(chg + (u[i] >> 5), bit);
    }
  }
  if constexpr (KIND == kTdThin) {
    if (!__any_sync(0xFFFFFFFFu, first != 0u)) return;
    const int lane = threadIdx.x & 31;
    const int own = __popc(first);
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    int base = 0;
    if (lane == 31) base = atomicAdd(t_cnt, incl);
    base = __shfl_sync(0xFFFFFFFFu, base, 31) + incl - own;
#pragma unroll
    for (int i = 0; i < kTdStep; i++)
      if ((first >> i) & 1u) gb.tl[base++] = u[i];
  }
}

// ---- bulk-copy (TMA) staging of large vertices' adjacency chunks ---------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// One untiled bulk copy global -> shared (both addresses 16-byte aligned,
// bytes a multiple of 16), completing on `bar`.  The source is this GPU's
// own CSR; no multicast.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes,
                                         unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for phase `parity` of `bar` (each try_wait suspends the
// thread for a while in hardware; kMbarTries of them is seconds).
constexpr long long kMbarTries = 1LL << 22;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  for (long long i = 0; i < kMbarTries; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

constexpr int kStageInts = 2048 + 8;  // one chunk (threads*4 <= 2048) plus alignment slack

// The two staging buffers (one array for every instance of the phase).
__device__ __forceinline__ int32_t (*td_stage_buf())[kStageInts] {
  __shared__ __align__(128) int32_t s_col[2][kStageInts];
  return s_col;
}

// The column-id range [a0, a1) that covers chunk c of a large vertex with
// 16-byte aligned ends (col is 16-byte aligned and padded by 4 entries).
__device__ __forceinline__ void td_chunk(const Params& p, const GroupBufs& gb, int c, int32_t* v,
                                         long long* b0, long long* b1, long long* a0,
                                         long long* a1) {
  const int2 d = gb.ql[c];
  *v = d.x;
  const long long e_end = p.beg[d.x + 1];
  *b0 = p.beg[d.x] + (long long)d.y * p.chunk;
  *b1 = min(e_end, *b0 + (long long)p.chunk);
  *a0 = *b0 & ~3LL;
  *a1 = (*b1 + 3) & ~3LL;
}

// ---------------------------------------------------------------------------
// Phase: top-down expansion of level L over the three queues: one CTA per
// chunk of a large vertex (td_expand_cta, expander.cuh:276-331), one warp
// per medium vertex (td_expand_warp, expander.cuh:208-267), one thread per
// small vertex (td_expand_thd, expander.cuh:140-199).  Every thread takes
// kTdStep edges at a time: their column ids first, then their statuses.
// STAGE (the phase's own kernel, chunk <= 2048) with Params::td_stage: the
// large vertices' chunks -- the hubs' adjacency -- are staged through shared
// memory by bulk copies (TMA, cp.async.bulk), double-buffered: while the CTA
// pushes one chunk's edges, the next chunk's column ids are already on
// their way, so the pushes never wait for a column read.  Off by default:
// on R-MAT scale 24 the top-down levels are bound by the random status
// gathers, not by the column reads, and staging measured ~1 % slower.
// ---------------------------------------------------------------------------
template <int WORDS, bool STAGE, int KIND>
__device__ __forceinline__ void td_run(const Params& p, const GroupBufs& gb, int level,
                                       const int32_t* qc, const Team& t) {
  uint32_t* chg = chg_at(gb, p, level);
  int32_t* t_cnt = &par_at(gb.ctl, level)->t_cnt;
  const int4 nq = __ldcg(reinterpret_cast<const int4*>(qc));  // small, medium, large chunks
  const int nS = nq.x, nM = nq.y, nL = nq.z;
  if (STAGE && p.td_stage) {
    int32_t (*s_col)[kStageInts] = td_stage_buf();
    __shared__ __align__(8) unsigned long long s_bar[2];
    __shared__ int s_fail;
    if (threadIdx.x == 0) {
      mbar_init(&s_bar[0], 1);
      mbar_init(&s_bar[1], 1);
      mbar_init_fence();
      s_fail = 0;
    }
    __syncthreads();
    auto issue = [&](int i) {  // thread 0: chunk i of this CTA into buffer i & 1
      int32_t v;
      long long b0, b1, a0, a1;
      td_chunk(p, gb, t.block + i * t.nblocks, &v, &b0, &b1, &a0, &a1);
      const unsigned bytes = (unsigned)((a1 - a0) * 4);
      mbar_expect_tx(&s_bar[i & 1], bytes);
      bulk_g2s(s_col[i & 1], p.col + a0, bytes, &s_bar[i & 1]);
    };
    int issued = 0;  // chunks whose copy thread 0 has started
    if (threadIdx.x == 0 && t.block < nL) {
      issue(0);
      issued = 1;
    }
    for (int i = 0;; i++) {
      const int c = t.block + i * t.nblocks;
      if (c >= nL) break;
      if (threadIdx.x == 0 && c + t.nblocks < nL) {
        issue(i + 1);
        issued = i + 2;
      }
      int32_t v;
      long long b0, b1, a0, a1;
      td_chunk(p, gb, c, &v, &b0, &b1, &a0, &a1);
      uint32_t P[WORDS];
      ld_status<WORDS>(gb.last + (size_t)v * WORDS, P);
      if (!mbar_wait(&s_bar[i & 1], (unsigned)((i >> 1) & 1))) s_fail = 1;
      __syncthreads();
      if (s_fail) break;  // uniform
      const int32_t* sc = s_col[i & 1] + (b0 - a0);
      const int n = (int)(b1 - b0);
      for (int j0 = 0; j0 < n; j0 += kTdStep * blockDim.x) {
        const int j = j0 + (int)threadIdx.x;
        int32_t u[kTdStep];
        int cnt = 0;
#pragma unroll
        for (int q = 0; q < kTdStep; q++) {
          const int jq = j + q * (int)blockDim.x;
          u[q] = jq < n ? sc[jq] : 0;
          cnt += jq < n ? 1 : 0;
        }
        td_push_n<WORDS, KIND>(gb, chg, t_cnt, u, cnt, P);
      }
      __syncthreads();  // buffer i & 1 is read: the copy of chunk i + 2 may reuse it
    }
    if (s_fail && threadIdx.x == 0) {
      // a copy did not complete in time: report it, and before the CTA's
      // shared memory goes away, wait (bounded) for every copy it started
      atomicCAS(&gb.ctl->err, 0, 6);
      for (int i = 0; i < issued; i++) (void)mbar_wait(&s_bar[i & 1], (unsigned)((i >> 1) & 1));
    }
  } else {
    for (int c = t.block; c < nL; c += t.nblocks) {
      int32_t v;
      long long b0, b1, a0, a1;
      td_chunk(p, gb, c, &v, &b0, &b1, &a0, &a1);
      uint32_t P[WORDS];
      ld_status<WORDS>(gb.last + (size_t)v * WORDS, P);
      for (long long e0 = b0; e0 < b1; e0 += (long long)kTdStep * blockDim.x) {
        const long long e = e0 + threadIdx.x;
        int32_t u[kTdStep];
        int cnt = 0;
#pragma unroll
        for (int i = 0; i < kTdStep; i++) {
          const long long ei = e + (long long)i * blockDim.x;
          u[i] = ei < b1 ? __ldg(p.col + ei) : 0;
          cnt += ei < b1 ? 1 : 0;
        }
        td_push_n<WORDS, KIND>(gb, chg, t_cnt, u, cnt, P);
      }
    }
  }
  for (long long i = t.warp; i < nM; i += t.nwarps) {
    const int32_t v = __ldcg(gb.q + (p.V - 1 - i));
    uint32_t P[WORDS];
    ld_status<WORDS>(gb.last + (size_t)v * WORDS, P);
    const long long b1 = p.beg[v + 1];
    for (long long e0 = p.beg[v]; e0 < b1; e0 += 32 * kTdStep) {
      const long long e = e0 + t.lane;
      int32_t u[kTdStep];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < kTdStep; j++) {
        const long long ej = e + 32LL * j;
        u[j] = ej < b1 ? __ldg(p.col + ej) : 0;
        cnt += ej < b1 ? 1 : 0;
      }
      td_push_n<WORDS, KIND>(gb, chg, t_cnt, u, cnt, P);
    }
  }
  // A thread per small vertex; a thin level, whose queue leaves most threads
  // of the team without one, gives it 8 lanes instead, so that its list is
  // one step (32 edges) and not a chain of them.
  const int lg = (KIND == kTdThin && (long long)nS * 8 <= t.nthreads) ? 3 : 0;
  for (long long i0 = t.warp << (5 - lg); i0 < nS; i0 += t.nwarps << (5 - lg)) {
    const long long i = i0 + (t.lane >> lg);
    uint32_t P[WORDS];
    long long e = 0, b1 = 0;
    if (i < nS) {
      const int32_t v = __ldcg(gb.q + i);
      ld_status<WORDS>(gb.last + (size_t)v * WORDS, P);
      b1 = p.beg[v + 1];
      e = p.beg[v] + (long long)kTdStep * (t.lane & ((1 << lg) - 1));
    } else {
#pragma unroll
      for (int k = 0; k < WORDS; k++) P[k] = 0u;
    }
    while (__any_sync(0xFFFFFFFFu, e < b1)) {
      int32_t u[kTdStep];
      const int cnt = (int)max(0LL, min((long long)kTdStep, b1 - e));
#pragma unroll
      for (int j = 0; j < kTdStep; j++) u[j] = j < cnt ? __ldg(p.col + e + j) : 0;
      td_push_n<WORDS, KIND>(gb, chg, t_cnt, u, cnt, P);
      e += (long long)kTdStep << lg;
    }
  }
}

// A template instance per kind: the thin one's lists and votes cost the
// large levels registers otherwise.
template <int WORDS, bool STAGE = false>
__device__ void td_phase(const Params& p, const GroupBufs& gb, int level, const int32_t* qc,
                         int kind, const Team& t) {
  if (kind == kTdThin) td_run<WORDS, false, kTdThin>(p, gb, level, qc, t);
  else if (kind == kTdWide) td_run<WORDS, STAGE, kTdWide>(p, gb, level, qc, t);
  else td_run<WORDS, STAGE, kTdBitmap>(p, gb, level, qc, t);
}

// Second bottom-up stage: the hubs that were still missing frontier bits
// after their first hub_t neighbours.  One CTA per chunk of kHubChunk edges
// (frontier neighbours only); a chunk is skipped when curr[v], which the
// other chunks of the same hub merge into with atomics, already covers
// every frontier bit.  So one hub's long scan is spread over many CTAs
// instead of holding one warp -- and the whole level -- for its adjacency.
template <int WORDS, bool RO = false>
__device__ void bu_defer_phase(const Params& p, const GroupBufs& gb, int level,
                               const uint32_t* fmask_g, const int32_t* hq_cnt, const Team& t,
                               bool filt = false, const uint32_t* smask = nullptr) {
  __shared__ uint32_t s_acc[32][kMaxWords];
  __shared__ uint32_t s_cur[kMaxWords];
  __shared__ int s_skip;
  uint32_t fm[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) fm[k] = __ldcg(fmask_g + k) & (smask ? ~__ldcg(smask + k) : ~0u);
  const uint32_t* front = chg_at(gb, p, level - 1);
  uint32_t* out = chg_at(gb, p, level);
  const int n = __ldcg(hq_cnt);
  const int lane = t.lane, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int c = t.block; c < n; c += t.nblocks) {
    const int2 hc = gb.hq[c];
    const int32_t v = hc.x;
    if (threadIdx.x == 0) {  // one read, so that the skip decision is uniform
      uint32_t cur[WORDS];
      ld_status<WORDS>(gb.curr + (size_t)v * WORDS, cur);
      bool need = false;
#pragma unroll
      for (int k = 0; k < WORDS; k++) {
        s_cur[k] = cur[k];
        need |= (fm[k] & ~cur[k]) != 0u;
      }
      s_skip = need ? 0 : 1;
    }
    __syncthreads();
    if (s_skip) {
      __syncthreads();
      continue;
    }
    const long long e_end = p.beg[v + 1];
    const long long b0 = p.beg[v] + p.hub_t + (long long)hc.y * kHubChunk;
    const long long b1 = min(e_end, b0 + (long long)kHubChunk);
    uint32_t acc[WORDS];
#pragma unroll
    for (int k = 0; k < WORDS; k++) acc[k] = 0;
    for (long long e = b0 + threadIdx.x; e < b1; e += blockDim.x) {
      const int32_t u = p.col[e];
      if (filt && !in_front<RO>(front, u)) continue;
      uint32_t x[WORDS];
      if constexpr (RO && IBFS_BU_NC) ld_status_nc<WORDS>(gb.last + (size_t)u * WORDS, x);
      else ld_status<WORDS>(gb.last + (size_t)u * WORDS, x);
#pragma unroll
      for (int k = 0; k < WORDS; k++) acc[k] |= x[k];
    }
#pragma unroll
    for (int k = 0; k < WORDS; k++) {
      const uint32_t r = __reduce_or_sync(0xFFFFFFFFu, acc[k]);
      if (lane == 0) s_acc[wid][k] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t nb[WORDS];
      bool any = false;
#pragma unroll
      for (int k = 0; k < WORDS; k++) {
        uint32_t r = 0;
        for (int i = 0; i < nw; i++) r |= s_acc[i][k];
        nb[k] = r & ~s_cur[k];
        any |= nb[k] != 0u;
      }
      if (any) {
        if constexpr (WORDS == 1) {
          atomicOr(gb.curr + v, nb[0]);
        } else {
          unsigned long long* q = reinterpret_cast<unsigned long long*>(gb.curr + (size_t)v * WORDS);
#pragma unroll
          for (int k = 0; k < WORDS / 2; k++) {
            const unsigned long long w2 = ((unsigned long long)nb[2 * k + 1] << 32) | nb[2 * k];
            if (w2) atomicOr(q + k, w2);
          }
        }
        atomicOr(out + (v >> 5), 1u << (v & 31));
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Phase: bottom-up level L.  Every vertex that still lacks a bit of the
// previous level's frontier mask ORs the `last` words of those neighbours
// that were in the previous frontier (a bit can only come from a vertex
// that gained it at level L-1; the level-(L-1) bitmap, L2 resident, filters
// the others before their status word is read) and stops as soon as no
// frontier bit is missing -- the early exit of expander.cu:298,348,
// generalised from "all bits" to "all bits any frontier vertex carries".
// Low-degree vertices scan with one thread (sw_expand_thd, expander.cuh:
// 431-489), the rest with the whole warp and a warp OR-reduction
// (sw_expand_warp, expander.cuh:341-422).
// ---------------------------------------------------------------------------
//
// FUSED (device loop and persistent kernel) also does the inspect work of the level in the
// same pass, so that bottom-up levels need no inspect pass: every vertex's
// new status goes to `curr` (for all vertices, changed or not: `curr` then
// holds the complete status of the level while `last` keeps the previous
// one, and the caller swaps their roles), the new bits update the depth
// planes and the counters directly (the whole plane b is written at level
// 2^b, so it needs no zeroing), and the changed bitmap is still marked for a
// following top-down level.  Hubs deferred to bu_defer_phase get their
// planes and counters in bu_hub_epilogue.

// Status of neighbour u for a bottom-up scan: from the CTA's shared-memory
// copy of the hubs' statuses when u is one of the first hk vertices, else
// from `last`, which no thread writes during the pass (through L1: the
// read-only path when the pass is a kernel of its own (NC), ordinary cached
// loads in the persistent kernel).
template <int WORDS, int HK, bool NC>
__device__ __forceinline__ void ld_nbr(const uint32_t* last, const uint32_t* s_hub, long long hk,
                                       int32_t u, uint32_t (&x)[WORDS]) {
  if (HK > 0 && u < hk) {
    if constexpr (WORDS >= 4) {
#pragma unroll
      for (int q = 0; q < WORDS / 4; q++) {
        const uint4 t = reinterpret_cast<const uint4*>(s_hub + (size_t)u * WORDS)[q];
        x[4 * q] = t.x; x[4 * q + 1] = t.y; x[4 * q + 2] = t.z; x[4 * q + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < WORDS; k++) x[k] = s_hub[(size_t)u * WORDS + k];
    }
    return;
  }
  if constexpr (NC) ld_status_nc<WORDS>(last + (size_t)u * WORDS, x);
  else ld_status_ca<WORDS>(last + (size_t)u * WORDS, x);
}

// A word of shared memory, read again at every use: kept out of registers on
// purpose (the compiler would hoist a loop-invariant load and spill it).
__device__ __forceinline__ uint32_t lds_again(const uint32_t* p) {
  uint32_t x;
  asm volatile("ld.shared.u32 %0, [%1];"
               : "=r"(x)
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
  return x;
}

// A warp ORs the statuses of the neighbours [e0, e_lim) of one vertex into a
// (the same value in every lane) until no bit of fm is missing; returns
// whether one still is.  The first step reads 32 neighbours (the highest
// degrees, which usually cover the bits), the later ones 128: a long scan is
// a chain of steps, and with 4 gathers per lane in flight it has a quarter
// of them.
template <int WORDS, int HK, bool NC, bool RO>
__device__ __forceinline__ bool warp_scan(const Params& p, const GroupBufs& gb,
                                          const uint32_t* s_hub, long long hk,
                                          const uint32_t* front, bool filt, int lane,
                                          const int32_t* col, int e0, int e_lim,
                                          const uint32_t* s_mask, uint32_t (&a)[WORDS]) {
  // gathers in flight per lane; the kernel of its own, whose 40 registers
  // already spill, keeps one (its warps hide the chain)
  constexpr int D = RO ? 1 : WORDS <= 4 ? 4 : 2;
  bool miss = true;
  int width = 32;
  for (int e = e0; e < e_lim;) {
    uint32_t x[D][WORDS];
#pragma unroll
    for (int i = 0; i < D; i++) {
#pragma unroll
      for (int k = 0; k < WORDS; k++) x[i][k] = 0;
      const int ei = e + lane + 32 * i;
      if (32 * i < width && ei < e_lim) {
        const int32_t u = __ldg(col + ei);
        if (!filt || in_front<RO>(front, u)) ld_nbr<WORDS, HK, NC>(gb.last, s_hub, hk, u, x[i]);
      }
    }
    miss = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) {
      uint32_t r = x[0][k];
#pragma unroll
      for (int i = 1; i < D; i++) r |= x[i][k];
      a[k] |= __reduce_or_sync(0xFFFFFFFFu, r);
      miss |= (lds_again(s_mask + k) & ~a[k]) != 0u;
    }
    if (!miss) break;
    e += width;
    width = 32 * D;
  }
  return miss;
}

// Start fetching the line at p into L2 (no register waits for it).
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// smask (device loop, sparse-source levels): bits pushed top-down after this
// pass (push_queue_phase / push_run_phase); the scan's early exit ignores them.
template <int WORDS, bool FUSED = false, bool RO = FUSED, int HK = 0>
__device__ void bu_phase(const Params& p, const GroupBufs& gb, int level,
                         const uint32_t* fmask_g, int32_t* hq_cnt, const Team& t,
                         Par* par = nullptr, int n_b = 0, bool depth_ok = true,
                         bool filt = false, const uint32_t* smask = nullptr) {
  constexpr bool NC = RO && IBFS_BU_NC;
  // Hub status cache (HK > 0, passes that run as their own kernel: `last` is
  // not written while they run).  The degree order puts the highest-degree vertices at
  // internal ids 0..HK-1 and every adjacency list is ascending, so the first
  // neighbours a scan reads -- the ones that usually complete it -- are these
  // hubs: every CTA copies their previous-level statuses into shared memory
  // once and reads them from there instead of from L2.
  __shared__ __align__(16) uint32_t s_hub[HK > 0 ? HK * WORDS : 4];
  long long hk = 0;
  if constexpr (HK > 0) {
    hk = min((long long)HK, (long long)p.V);
    for (long long i = threadIdx.x; i < hk * WORDS; i += blockDim.x) s_hub[i] = __ldcg(gb.last + i);
    __syncthreads();
  }
  // The frontier mask and the batch's full words stay in shared memory, and
  // list positions are 32 bits relative to the list: the own-kernel build has
  // 40 registers a thread (3 x 512 threads per SM), and what does not fit is
  // spilled inside the sweep.
  __shared__ uint32_t s_mask[kMaxWords], s_full[kMaxWords], s_fm[kMaxWords];
  if (threadIdx.x < WORDS) {
    const int k = threadIdx.x;
    s_mask[k] = __ldcg(fmask_g + k) & (smask ? ~__ldcg(smask + k) : ~0u);
    s_full[k] = full_word(n_b, k);
    s_fm[k] = 0u;  // the OR of the level's new bits
  }
  __syncthreads();
  const uint32_t* front = chg_at(gb, p, level - 1);
  uint32_t* out = chg_at(gb, p, level);
  const int lane = t.lane;
  // FUSED counters (as inspect_phase).  32 bits hold a thread's degree sums: a
  // degree is below 2^31 here, and in the degree order each later vertex of a
  // thread has at most the average degree of the round of vertices before it, so
  // that they add up to at most E / threads (E / warps in the own-kernel prefix
  // loop), below 2^31 for every E that fits the GPU.  (A caller's own order,
  // ibfs_run_static_scratch, could pass that only with lists full of
  // duplicates; the sums steer the direction choice and no depth.)  The kernels
  // are sensitive here: handing a carry on instead cost the grid 1.5 % in the
  // device loop and deep grids 4 % in the persistent kernel.
  uint32_t f_mf = 0, f_cnt = 0, f_cdeg = 0;
  unsigned long long f_teps = 0;
  const bool first_plane = (level & (level - 1)) == 0;
  const int pb = __ffs(level) - 1;
  bool range = false;
  // The degree order puts every vertex above the thread-path limit into the
  // prefix [0, p.big_prefix): one warp per vertex there, so that the hubs,
  // which that order packs into a few warps, are spread over all of them.
  // (The persistent kernel deals them out to lanes instead, below.)
  for (long long v = t.warp; RO && v < p.big_prefix; v += t.nwarps) {
    uint32_t l[WORDS];
    ld_status<WORDS>(gb.last + (size_t)v * WORDS, l);
    const long long e0 = p.beg[v];
    const int deg_v = (int)(p.beg[v + 1] - e0);
    bool need = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) need |= (lds_again(s_mask + k) & ~l[k]) != 0u;
    need = need && deg_v > 0;  // uniform across the warp
    uint32_t a[WORDS];
#pragma unroll
    for (int k = 0; k < WORDS; k++) a[k] = l[k];
    bool defer = false;
    if (need) {
      const int e_lim = min(deg_v, p.hub_t);
      const bool miss = warp_scan<WORDS, HK, NC, RO>(p, gb, s_hub, hk, front, filt, lane,
                                                     p.col + e0, 0, e_lim, s_mask, a);
      defer = miss && e_lim < deg_v;
      if (defer && lane == 0) {
        const int nch = (deg_v - e_lim + kHubChunk - 1) / kHubChunk;
        const int base0 = atomicAdd(hq_cnt, nch);
        for (int c = 0; c < nch; c++) gb.hq[base0 + c] = make_int2((int)v, c);
      }
    }
    bool ch = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) ch |= a[k] != l[k];
    if (lane == 0) {
      if constexpr (!FUSED) {
        if (ch) {
          st_status<WORDS>(gb.curr + (size_t)v * WORDS, a);
          atomicOr(out + (v >> 5), 1u << (v & 31));
        }
      } else {
        st_status<WORDS>(gb.curr + (size_t)v * WORDS, a);  // every vertex: curr = new status
        const bool epi = ch && !defer;
        uint32_t nb[WORDS];
        uint32_t pop = 0;
        bool comp = true;
#pragma unroll
        for (int k = 0; k < WORDS; k++) {
          nb[k] = epi ? (a[k] & ~l[k]) : 0u;
          pop += __popc(nb[k]);
          comp = comp && a[k] == lds_again(s_full + k);
          if (nb[k]) atomicOr(&s_fm[k], nb[k]);
        }
        if (epi) {
          const uint32_t deg = (uint32_t)deg_v;
          f_cnt += 1;
          f_mf += deg;
          f_teps += (unsigned long long)deg * pop;
          if (comp) f_cdeg += deg;
          if (!depth_ok) range = true;
          atomicOr(out + (v >> 5), 1u << (v & 31));
        }
        uint32_t* q0 = gb.planes + (size_t)v * WORDS;
        if (first_plane) {
          st_status<WORDS>(q0 + (size_t)pb * p.plane_stride, nb);
        } else if (epi && depth_ok) {
          unsigned rest = (unsigned)level;
          while (rest) {
            const int b0p = __ffs(rest) - 1;
            rest &= rest - 1;
            uint32_t* qa = q0 + (size_t)b0p * p.plane_stride;
            uint32_t xa[WORDS];
            ld_status<WORDS>(qa, xa);
#pragma unroll
            for (int k = 0; k < WORDS; k++) xa[k] |= nb[k];
            st_status<WORDS>(qa, xa);
          }
        }
      }
    }
  }
  const long long start = p.big_prefix;  // a multiple of 32
  const long long rstep = t.nwarps * 32;
  if (FUSED && first_plane) {
    // the pass writes its first-used plane whole; the edgeless tail it does
    // not sweep gets zeros (an edgeless source keeps depth 0)
    const long long n4 = (p.V - p.v_nz) * WORDS / 4;
    uint4* q = reinterpret_cast<uint4*>(gb.planes + (size_t)pb * p.plane_stride +
                                        (size_t)p.v_nz * WORDS);
    for (long long i = t.tid; i < n4 + ((p.V - p.v_nz) * WORDS % 4 ? 1 : 0); i += t.nthreads)
      __stcg(q + i, make_uint4(0, 0, 0, 0));
  }
  // Persistent kernel: the prefix is dealt out like cards, one vertex per lane
  // and the hubs one per warp, so that the lanes peek at their first
  // neighbours together and a warp scans only the vertices that are still
  // missing bits, one after another.  Then the rest, in ranges of 32.
  const long long first = start + t.warp * 32;
  const long long dealt_v = RO ? 0 : (p.big_prefix + rstep - 1) / rstep * rstep;
  for (long long base = first - dealt_v; base < p.v_nz; base += rstep) {
    const bool dealt = !RO && base < start;
    const long long v = dealt ? base - first + dealt_v + lane * t.nwarps + t.warp : base + lane;
    const bool valid = v < (dealt ? p.big_prefix : p.V);
    uint32_t l[WORDS], acc[WORDS];
    long long b0 = 0;
    int deg_v = 0;
    if (valid) {
      ld_status<WORDS>(gb.last + (size_t)v * WORDS, l);
      b0 = p.beg[v];
      deg_v = (int)(p.beg[v + 1] - b0);
    } else {
#pragma unroll
      for (int k = 0; k < WORDS; k++) l[k] = 0;
    }
    bool need = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) {
      acc[k] = l[k];
      need |= (lds_again(s_mask + k) & ~l[k]) != 0u;
    }
    need = need && deg_v > 0;
    const bool small = need && deg_v <= p.but;
    if (FUSED && need && !first_plane) {
      // the depth planes that a change of this vertex will read
      for (unsigned rest = (unsigned)level; rest; rest &= rest - 1)
        prefetch_l2(gb.planes + (size_t)(__ffs(rest) - 1) * p.plane_stride + (size_t)v * WORDS);
    }
    // Every vertex that needs bits scans on its own lane first: a small one
    // its whole list, a big one only its first kBuPeek steps -- its
    // highest-degree neighbours, which in the degree order usually cover
    // the frontier bits already.  Only big vertices still missing bits go on
    // to the warp scan below, which takes them one at a time.
    bool covered = false;
    const int32_t* col = p.col + b0;
    int e_big = 0;  // where a big vertex's warp scan starts
    if (need) {
      // kBuStep neighbours in flight per step; with col_vec their ids come as
      // aligned 16-byte vectors (col is padded by 4 entries at its end, and
      // a vector is only read when it starts before b1)
      constexpr int S = kBuStep;
      // (a list of one step is read id by id: its vector would often straddle
      // two aligned ones and cost a second step; grid 4096^2 137 -> 133 ms)
      const bool vec = p.col_vec && deg_v > S;
      const int a0 = vec ? -(int)(b0 & 3) : 0;
      const int a_end = small ? deg_v : min(deg_v, a0 + kBuPeek * S);
      if (!small) e_big = max(0, a_end);
      for (int a = a0; a < a_end; a += S) {
        int32_t u[S];
        if (vec) {
#pragma unroll
          for (int q = 0; q < S / 4; q++) {
            int4 c4 = make_int4(0, 0, 0, 0);
            if (q == 0 || a + 4 * q < deg_v)
              c4 = __ldg(reinterpret_cast<const int4*>(col + a + 4 * q));
            u[4 * q] = c4.x; u[4 * q + 1] = c4.y; u[4 * q + 2] = c4.z; u[4 * q + 3] = c4.w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < S; i++) u[i] = a + i < deg_v ? __ldg(col + a + i) : 0;
        }
        bool f[S];
#pragma unroll
        for (int i = 0; i < S; i++) {
          const bool in = (unsigned)(a + i) < (unsigned)deg_v;
          f[i] = in && (!filt || in_front<RO>(front, u[i]));
        }
        uint32_t x[S][WORDS];
#pragma unroll
        for (int i = 0; i < S; i++) {
          if (f[i]) {
            ld_nbr<WORDS, HK, NC>(gb.last, s_hub, hk, u[i], x[i]);
          } else {
#pragma unroll
            for (int k = 0; k < WORDS; k++) x[i][k] = 0;
          }
        }
        bool miss = false;
#pragma unroll
        for (int k = 0; k < WORDS; k++) {
#pragma unroll
          for (int i = 0; i < S; i++) acc[k] |= x[i][k];
          miss |= (lds_again(s_mask + k) & ~acc[k]) != 0u;
        }
        if (!miss) {
          covered = true;
          break;
        }
      }
    }
    bool deferred = false;  // this lane's vertex left chunks to bu_defer_phase
    uint32_t big = __ballot_sync(0xFFFFFFFFu, need && !small && !covered);
    while (big) {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const long long e0 = __shfl_sync(0xFFFFFFFFu, b0, j);
      const int dj = __shfl_sync(0xFFFFFFFFu, deg_v, j);
      const int es = __shfl_sync(0xFFFFFFFFu, e_big, j);
      uint32_t a[WORDS];
#pragma unroll
      for (int k = 0; k < WORDS; k++) a[k] = __shfl_sync(0xFFFFFFFFu, acc[k], j);
      // a warp scans at most hub_t neighbours; the rest of a hub that is
      // still missing frontier bits is deferred to bu_defer_phase
      // (the limit counts from the list's start, as bu_defer_phase does)
      const int e_lim = min(dj, p.hub_t);
      const bool miss = warp_scan<WORDS, HK, NC, RO>(p, gb, s_hub, hk, front, filt, lane,
                                                     p.col + e0, es, e_lim, s_mask, a);
      const bool defer = miss && e_lim < dj;
      if (defer && lane == 0) {
        const int nch = (dj - e_lim + kHubChunk - 1) / kHubChunk;
        const int base0 = atomicAdd(hq_cnt, nch);
        const int vj = dealt ? (int)(base - first + dealt_v + j * t.nwarps + t.warp)
                             : (int)(base + j);
        for (int c = 0; c < nch; c++) gb.hq[base0 + c] = make_int2(vj, c);
      }
      if (lane == j) {
#pragma unroll
        for (int k = 0; k < WORDS; k++) acc[k] = a[k];
        deferred = defer;
      }
    }
    bool ch = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) ch |= acc[k] != l[k];
    ch = ch && need;
    uint32_t nb[WORDS];
#pragma unroll
    for (int k = 0; k < WORDS; k++) nb[k] = 0u;
    if constexpr (!FUSED) {
      if (ch) st_status<WORDS>(gb.curr + (size_t)v * WORDS, acc);
    } else if (valid) {
      st_status<WORDS>(gb.curr + (size_t)v * WORDS, acc);  // every vertex: curr = new status
      const bool epi = ch && !deferred;  // deferred hubs: bu_hub_epilogue
      uint32_t pop = 0;
      bool comp = true;
#pragma unroll
      for (int k = 0; k < WORDS; k++) {
        nb[k] = epi ? (acc[k] & ~l[k]) : 0u;
        pop += __popc(nb[k]);
        comp = comp && acc[k] == lds_again(s_full + k);
      }
      if (epi) {
        const uint32_t deg = (uint32_t)deg_v;
        f_cnt += 1;
        f_mf += deg;
        f_teps += (unsigned long long)deg * pop;
        if (comp) f_cdeg += deg;
        if (!depth_ok) range = true;
      }
      uint32_t* q0 = gb.planes + (size_t)v * WORDS;
      if (first_plane) {
        // level 2^b is the first to use plane b: write it whole (0 where no bit is new)
        st_status<WORDS>(q0 + (size_t)pb * p.plane_stride, nb);
      } else if (epi && depth_ok) {
        unsigned rest = (unsigned)level;
        while (rest) {
          const int b0p = __ffs(rest) - 1;
          rest &= rest - 1;
          uint32_t* qa = q0 + (size_t)b0p * p.plane_stride;
          uint32_t xa[WORDS];
          ld_status<WORDS>(qa, xa);
#pragma unroll
          for (int k = 0; k < WORDS; k++) xa[k] |= nb[k];
          st_status<WORDS>(qa, xa);
        }
      }
      ch = epi;
    }
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, ch);
    if (!bal) continue;
    if constexpr (FUSED) {
      // the level's new bits: every source that still expands is in s_fm
      // after a few ranges, so look before reducing
      bool more = false;
#pragma unroll
      for (int k = 0; k < WORDS; k++) more |= (nb[k] & ~lds_again(s_fm + k)) != 0u;
      if (__any_sync(0xFFFFFFFFu, more)) {
#pragma unroll
        for (int k = 0; k < WORDS; k++) {
          const uint32_t r = __reduce_or_sync(0xFFFFFFFFu, nb[k]);
          if (lane == 0 && r) atomicOr(&s_fm[k], r);
        }
      }
    }
    if (!dealt) {
      if (lane == 0) atomicOr(out + (base >> 5), bal);
    } else if (ch) {
      atomicOr(out + (v >> 5), 1u << (v & 31));
    }
  }
  if constexpr (FUSED) {
    if (range) par->range_err = 1;
    uint32_t fmo[WORDS];  // every thread holds the CTA's OR (s_fm is complete
    __syncthreads();      // behind the barrier)
#pragma unroll
    for (int k = 0; k < WORDS; k++) fmo[k] = s_fm[k];
    cta_flush<WORDS>(par, f_cnt, f_mf, f_cdeg, f_teps, fmo);
  }
}

// FUSED bottom-up, after bu_defer_phase: the inspect work of the hubs whose
// scan was deferred (one entry per hub: chunk 0), from their final status
// in `curr` and the previous one in `last`; and the level+1 bitmap cleared
// for the next expand (what inspect_phase does on other levels).
// keep_next: a sparse-source push follows and still reads the level-(L-1)
// bitmap, which is the same buffer as level L+1's (level parity); the push
// kernel's successor clears it then.
template <int WORDS>
__device__ void bu_hub_epilogue(const Params& p, const GroupBufs& gb, Par* par, int n_b,
                                int level, bool depth_ok, const Team& t, bool keep_next = false) {
  if (!keep_next) zero_words(chg_at(gb, p, level + 1), p.chg_stride, t);
  uint32_t full[WORDS], fm[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    full[k] = full_word(n_b, k);
    fm[k] = 0;
  }
  unsigned long long mf = 0, cnt = 0, cdeg = 0, teps = 0;
  uint32_t* out = chg_at(gb, p, level);
  const int n = __ldcg(&par->hq_cnt);
  for (long long i = t.tid; i < n; i += t.nthreads) {
    const int2 hc = gb.hq[i];
    if (hc.y != 0) continue;
    const long long v = hc.x;
    uint32_t c[WORDS], l[WORDS], nb[WORDS];
    ld_status<WORDS>(gb.curr + (size_t)v * WORDS, c);
    ld_status<WORDS>(gb.last + (size_t)v * WORDS, l);
    bool any = false, comp = true;
    uint32_t pop = 0;
#pragma unroll
    for (int k = 0; k < WORDS; k++) {
      nb[k] = c[k] & ~l[k];
      any |= nb[k] != 0u;
      comp = comp && c[k] == full[k];
      pop += __popc(nb[k]);
      fm[k] |= nb[k];
    }
    if (!any) continue;
    const unsigned long long deg = (unsigned long long)(p.beg[v + 1] - p.beg[v]);
    cnt += 1;
    mf += deg;
    teps += deg * pop;
    if (comp) cdeg += deg;
    if (!depth_ok) par->range_err = 1;
    atomicOr(out + (v >> 5), 1u << (v & 31));
    if (depth_ok) {
      unsigned rest = (unsigned)level;
      while (rest) {
        const int b = __ffs(rest) - 1;
        rest &= rest - 1;
        uint32_t* q = gb.planes + (size_t)b * p.plane_stride + (size_t)v * WORDS;
        uint32_t x[WORDS];
        ld_status<WORDS>(q, x);
#pragma unroll
        for (int k = 0; k < WORDS; k++) x[k] |= nb[k];
        st_status<WORDS>(q, x);
      }
    }
  }
  cta_flush<WORDS>(par, cnt, mf, cdeg, teps, fm);
}

// ---------------------------------------------------------------------------
// Sparse sources (device loop, a bottom-up level L that follows a top-down
// level).  A bottom-up scan stops once a vertex holds every bit of the
// previous frontier.  A source whose level-(L-1) frontier holds only a
// handful of vertices (it started far from the hubs) has not reached most
// vertices yet, so with its bit in the mask almost no vertex can stop early
// and most scan their whole neighbour lists.  So at such a level:
//   sparse_count_phase  counts every source's level-(L-1) frontier;
//   (k_dl_sparse_decide) the sources below 1/sparse_div of the average go
//                       into LoopState::smask, and the bottom-up pass's
//                       early exit ignores their bits;
//   push_queue_phase /  after the pass (and its deferred hubs), those bits
//   push_run_phase      are delivered exactly as a top-down level would:
//                       every vertex that gained a sparse bit at level L-1
//                       pushes it to all its neighbours -- a warp per small
//                       vertex, 2048-edge chunks spread over all CTAs for a
//                       vertex above the large-queue threshold (a hub can be
//                       in a sparse source's frontier).
// Each push takes its new bits from the atomic OR's old value, so the
// level's edge count, its depth planes (OR reductions: other pushes may hit
// the same vertex) and fmask stay exact; the changed count, the frontier-edge
// sum and the completed-degree sum (which only steer the direction choice)
// count a vertex when a push is the first change to it at this level.  The
// result is the BFS of every source: a bit reaches each vertex at its
// distance either way.
// ---------------------------------------------------------------------------
// The bits of `mask` that v gained at level L-1 (`last` holds the statuses
// after level L-1; a bit's depth is L-1 when the planes spell L-1: the planes
// of bits already in `last` no longer change).
template <int WORDS>
__device__ __forceinline__ bool gained_at(const Params& p, const GroupBufs& gb, long long v,
                                          int lp, const uint32_t (&mask)[WORDS],
                                          uint32_t (&P)[WORDS]) {
  ld_status<WORDS>(gb.last + (size_t)v * WORDS, P);
  bool has = false;
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    P[k] &= mask[k];
    has |= P[k] != 0u;
  }
  if (!has) return false;
  const int np = planes_for(lp);
  for (int b = 0; b < np; b++) {
    uint32_t x[WORDS];
    ld_status<WORDS>(gb.planes + (size_t)b * p.plane_stride + (size_t)v * WORDS, x);
    const bool one = (lp >> b) & 1;
#pragma unroll
    for (int k = 0; k < WORDS; k++) P[k] &= one ? x[k] : ~x[k];
  }
  has = false;
#pragma unroll
  for (int k = 0; k < WORDS; k++) has |= P[k] != 0u;
  return has;
}

template <int WORDS>
__device__ void sparse_count_phase(const Params& p, const GroupBufs& gb, int level,
                                   const Team& t) {
  __shared__ uint32_t s_scnt[kMaxWords * 32];
  scnt_begin(s_scnt);
  uint32_t all[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) all[k] = 0xFFFFFFFFu;
  const uint32_t* front = chg_at(gb, p, level - 1);
  for (long long v = t.tid; v < p.V; v += t.nthreads) {
    if (!((__ldcg(front + (v >> 5)) >> (v & 31)) & 1u)) continue;
    uint32_t P[WORDS];
    if (!gained_at<WORDS>(p, gb, v, level - 1, all, P)) continue;
#pragma unroll
    for (int k = 0; k < WORDS; k++) {
      uint32_t r = P[k];
      while (r) {
        atomicAdd(&s_scnt[k * 32 + __ffs(r) - 1], 1u);
        r &= r - 1;
      }
    }
  }
  scnt_flush<WORDS>(s_scnt, gb.tl);
}

struct PushAcc {
  unsigned long long mf = 0, cnt = 0, cdeg = 0, teps = 0;
  uint32_t fm[kMaxWords] = {0, 0, 0, 0, 0, 0, 0, 0};
  bool range = false;
};

// One pushed edge: OR the bits P into u's status and account for the ones
// that were new (see above).
template <int WORDS>
__device__ __forceinline__ void push_edge(const Params& p, const GroupBufs& gb, uint32_t* out,
                                          int level, bool depth_ok, const uint32_t (&full)[WORDS],
                                          int32_t u, const uint32_t (&P)[WORDS], PushAcc& acc) {
  uint32_t s[WORDS];
  ld_status<WORDS>(gb.curr + (size_t)u * WORDS, s);
  bool need = false;
#pragma unroll
  for (int k = 0; k < WORDS; k++) need |= (P[k] & ~s[k]) != 0u;
  if (!need) return;
  uint32_t old[WORDS], nb[WORDS];
  if constexpr (WORDS == 1) {
    old[0] = atomicOr(gb.curr + u, P[0]);
  } else {
    unsigned long long* q = reinterpret_cast<unsigned long long*>(gb.curr + (size_t)u * WORDS);
#pragma unroll
    for (int k = 0; k < WORDS / 2; k++) {
      const unsigned long long pw = ((unsigned long long)P[2 * k + 1] << 32) | P[2 * k];
      const unsigned long long o =
          pw ? atomicOr(q + k, pw) : (((unsigned long long)s[2 * k + 1] << 32) | s[2 * k]);
      old[2 * k] = (uint32_t)o;
      old[2 * k + 1] = (uint32_t)(o >> 32);
    }
  }
  bool any = false;
  uint32_t pop = 0;
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    nb[k] = P[k] & ~old[k];
    any |= nb[k] != 0u;
    pop += __popc(nb[k]);
  }
  if (!any) return;
  uint32_t l[WORDS];
  ld_status<WORDS>(gb.last + (size_t)u * WORDS, l);
  bool first = true, was_full = true, now_full = true;
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    first = first && (old[k] & ~l[k]) == 0u;
    was_full = was_full && old[k] == full[k];
    now_full = now_full && (old[k] | nb[k]) == full[k];
    acc.fm[k] |= nb[k];
  }
  const unsigned long long deg = (unsigned long long)(p.beg[u + 1] - p.beg[u]);
  acc.teps += deg * pop;
  if (first) {
    acc.cnt += 1;
    acc.mf += deg;
  }
  if (now_full && !was_full) acc.cdeg += deg;
  red_or_u32(out + (u >> 5), 1u << (u & 31));
  if (!depth_ok) {
    acc.range = true;
    return;
  }
  unsigned rest = (unsigned)level;
  while (rest) {
    const int b = __ffs(rest) - 1;
    rest &= rest - 1;
    uint32_t* q = gb.planes + (size_t)b * p.plane_stride + (size_t)u * WORDS;
#pragma unroll
    for (int k = 0; k < WORDS; k++)
      if (nb[k]) red_or_u32(q + k, nb[k]);
  }
}

template <int WORDS>
__device__ __forceinline__ void push_acc_flush(const PushAcc& acc, Par* par) {
  if (acc.range) par->range_err = 1;
  uint32_t fm[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) fm[k] = acc.fm[k];
  cta_flush<WORDS>(par, acc.cnt, acc.mf, acc.cdeg, acc.teps, fm);
}

template <int WORDS>
__device__ void push_queue_phase(const Params& p, const GroupBufs& gb, Par* par, int n_b,
                                 int level, bool depth_ok, const uint32_t* smask,
                                 const Team& t) {
  uint32_t sm[WORDS], full[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    sm[k] = __ldcg(smask + k);
    full[k] = full_word(n_b, k);
  }
  const uint32_t* front = chg_at(gb, p, level - 1);
  uint32_t* out = chg_at(gb, p, level);
  PushAcc acc;
  const int lane = t.lane;
  for (long long w = t.warp; w < p.nchg; w += t.nwarps) {
    const uint32_t bits = __ldcg(front + w);
    if (!bits) continue;  // uniform
    const long long v0 = w * 32 + lane;
    uint32_t P[WORDS];
    bool has = false;
#pragma unroll
    for (int k = 0; k < WORDS; k++) P[k] = 0u;
    long long deg = 0;
    if ((bits >> lane) & 1u) {
      has = gained_at<WORDS>(p, gb, v0, level - 1, sm, P);
      if (has) deg = p.beg[v0 + 1] - p.beg[v0];
    }
    // a vertex above the large-queue threshold goes to the chunk queue
    if (has && deg > p.lrg) {
      const int nch = (int)((deg + p.chunk - 1) / p.chunk);
      const int base0 = atomicAdd(&par->pq_cnt, nch);
      for (int c = 0; c < nch; c++) gb.ql[base0 + c] = make_int2((int)v0, c);
      has = false;
    }
    uint32_t pushers = __ballot_sync(0xFFFFFFFFu, has);
    while (pushers) {
      const int j = __ffs(pushers) - 1;
      pushers &= pushers - 1;
      uint32_t Pj[WORDS];
#pragma unroll
      for (int k = 0; k < WORDS; k++) Pj[k] = __shfl_sync(0xFFFFFFFFu, P[k], j);
      const long long v = w * 32 + j;
      const long long e1 = p.beg[v + 1];
      for (long long e = p.beg[v] + lane; e < e1; e += 32)
        push_edge<WORDS>(p, gb, out, level, depth_ok, full, __ldg(p.col + e), Pj, acc);
    }
  }
  push_acc_flush<WORDS>(acc, par);
}

template <int WORDS>
__device__ void push_run_phase(const Params& p, const GroupBufs& gb, Par* par, int n_b,
                               int level, bool depth_ok, const uint32_t* smask, const Team& t) {
  uint32_t sm[WORDS], full[WORDS];
#pragma unroll
  for (int k = 0; k < WORDS; k++) {
    sm[k] = __ldcg(smask + k);
    full[k] = full_word(n_b, k);
  }
  uint32_t* out = chg_at(gb, p, level);
  PushAcc acc;
  const int n = __ldcg(&par->pq_cnt);
  for (int c = t.block; c < n; c += t.nblocks) {
    const int2 d = gb.ql[c];
    uint32_t P[WORDS];
    (void)gained_at<WORDS>(p, gb, d.x, level - 1, sm, P);
    const long long e_end = p.beg[d.x + 1];
    const long long b0 = p.beg[d.x] + (long long)d.y * p.chunk;
    const long long b1 = min(e_end, b0 + (long long)p.chunk);
    for (long long e = b0 + threadIdx.x; e < b1; e += blockDim.x)
      push_edge<WORDS>(p, gb, out, level, depth_ok, full, __ldg(p.col + e), P, acc);
  }
  push_acc_flush<WORDS>(acc, par);
}

// ---------------------------------------------------------------------------
// Phase: write one batch's depths from the bit-planes.  Depth of (v, s) =
// the number whose bit b is bit s of plane b, INFTY (255 / 65535,
// comm.h:120) when bit s of the final status is clear.  Every output byte is
// written once, in whole sectors.
//   source-major: rows out_row[...] of V depths;
//   vertex-major: the batch block [V][n_b] (depth_merge, inspector.cuh:48).
// ---------------------------------------------------------------------------

// 4 bits -> the low bit of 4 bytes (bit i -> bit 8i).
__device__ __forceinline__ uint32_t nib_to_bytes(uint32_t nib) {
  return (nib * 0x00204081u) & 0x01010101u;
}
// In-register transpose of a 32 x 32 bit matrix, LSB-first: afterwards
// bit r of A[j] is what bit j of A[r] was.  Five rounds of block swaps
// (16, 8, 4, 2, 1), 16 masked delta swaps each; rows that are zero at
// compile time fold away.
__device__ __forceinline__ void transpose32(uint32_t (&A)[32]) {
#pragma unroll
  for (int lv = 0; lv < 5; lv++) {
    const int j = 16 >> lv;
    const uint32_t m = lv == 0 ? 0x0000FFFFu : lv == 1 ? 0x00FF00FFu : lv == 2 ? 0x0F0F0F0Fu
                     : lv == 3 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int r = 0; r < 32; r++) {
      if (r & j) continue;
      const uint32_t t = ((A[r] >> j) ^ A[r + j]) & m;
      A[r + j] ^= t;
      A[r] ^= t << j;
    }
  }
}

#ifndef IBFS_OUT_PRMT
#define IBFS_OUT_PRMT 1
#endif
#ifndef IBFS_OUT_FASTST
#define IBFS_OUT_FASTST 1
#endif
#ifndef IBFS_OUT_STCS
#define IBFS_OUT_STCS 1
#endif

// A 4-byte piece of a depth row.  The rows are written once and not read
// again on the device: with IBFS_OUT_STCS they are streaming stores (evict
// first), so that they do not push the gathered statuses and planes out of
// L2.
__device__ __forceinline__ void st_row4(uint8_t* a, uint32_t x) {
#if IBFS_OUT_STCS
  __stcs(reinterpret_cast<unsigned int*>(a), x);
#else
  *reinterpret_cast<uint32_t*>(a) = x;
#endif
}

// The same transpose with its first two rounds (whole 16- and 8-bit blocks)
// as byte permutes, two per row pair instead of a five-instruction masked
// delta swap.  Z: bit r set = row r is zero on entry (a compile-time
// constant), so that pairs of zero rows are skipped; the rounds commute, so
// the order of the five does not matter.
template <uint32_t Z>
__device__ __forceinline__ void transpose32_z(uint32_t (&A)[32]) {
#pragma unroll
  for (int r = 0; r < 16; r++) {
    if (((Z >> r) & 1u) && ((Z >> (r + 16)) & 1u)) continue;
    const uint32_t a = A[r], b = A[r + 16];
    A[r] = __byte_perm(a, b, 0x5410);       // low halves
    A[r + 16] = __byte_perm(a, b, 0x7632);  // high halves
  }
  constexpr uint32_t Z1 = (Z & (Z >> 16) & 0xFFFFu) * 0x10001u;
#pragma unroll
  for (int r = 0; r < 32; r++) {
    if (r & 8) continue;
    if (((Z1 >> r) & 1u) && ((Z1 >> (r + 8)) & 1u)) continue;
    const uint32_t a = A[r], b = A[r + 8];
    A[r] = __byte_perm(a, b, 0x6240);      // bytes 0 and 2 of both
    A[r + 8] = __byte_perm(a, b, 0x7351);  // bytes 1 and 3 of both
  }
#pragma unroll
  for (int lv = 2; lv < 5; lv++) {
    const int j = 16 >> lv;
    const uint32_t m = lv == 2 ? 0x0F0F0F0Fu : lv == 3 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int r = 0; r < 32; r++) {
      if (r & j) continue;
      // m << j == ~m: each row keeps its own half and takes the partner's
      // other half, a shift and a three-input select each
      const uint32_t a = A[r], b = A[r + j];
      A[r] = (a & m) | ((b << j) & ~m);
      A[r + j] = ((a >> j) & m) | (b & ~m);
    }
  }
}

// Rows known zero in output_sm_u8's matrix: 8i + b for NP <= b <= 6.
template <int NP>
__host__ __device__ constexpr uint32_t out_zero_rows() {
  uint32_t z = 0u;
  for (int i = 0; i < 4; i++)
    for (int b = NP; b < 7; b++) z |= 1u << (8 * i + b);
  return z;
}

// Source-major, one-byte depths, NP (<= 8) planes known at compile time:
// lane = 4 consecutive vertices, one 4-byte store per source row.  The
// depth byte of (vertex i, source s) has bit b = bit s of plane b of vertex
// i, or is 0xFF when bit s of the final status is clear: the 32 words
// A[8i + b] form a 32 x 32 bit matrix whose transpose is exactly the 32
// output words, one per source, byte i = vertex i.  With NP <= 7 (depths
// below 128) A[8i + b] = plane_b(i) for b < NP, 0 up to b = 6 and ~status(i)
// for b = 7, and one sign-replicating byte permute per word turns bit 7
// into 0xFF; the zero rows are compile-time constants that fold out of the
// transpose.  With NP = 8, A[8i + b] = plane_b(i) | ~status(i).
template <int WORDS, int NP>
__device__ void output_sm_u8(const Params& p, const GroupBufs& gb, const int32_t* rows, int n_b,
                             const Team& t) {
  static_assert(NP <= 8, "one-byte depths use at most 8 planes");
  const int lane = t.lane;
  const bool tail_src = gb.ctl->tail_src != 0;
  for (long long base = t.warp * 128; base < p.V; base += t.nwarps * 128) {
    const long long v0 = base + 4 * lane;
    const bool full4 = p.vec_sm >= 4 && v0 + 3 < p.V;
    // rows are in the caller's vertex order; statuses in the graph's
    uint32_t vis[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
      vis[i] = v0 + i < p.V ? (uint32_t)(p.vmap ? p.vmap[v0 + i] : v0 + i) : 0u;
#pragma unroll 1
    for (int k = 0; k < WORDS && k * 32 < n_b; k++) {
      const uint32_t mine = full_word(n_b, k);
      uint32_t A[32];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool in = v0 + i < p.V;
        const size_t vi = vis[i];
        // a vertex from v_reach on is reached only as a source, at depth 0:
        // its plane words are zeros (every plane was first written whole
        // during the batch), so they are not gathered
        const bool edged = in && (long long)vi < p.v_reach;
        uint32_t some = 0u;  // sources with a plane bit: reached, depth > 0
#pragma unroll
        for (int b = 0; b < NP; b++) {
          A[8 * i + b] = edged ? gb.planes[(size_t)b * p.plane_stride + vi * WORDS + k] : 0u;
          some |= A[8 * i + b];
        }
        // the others are unreached or the vertex itself: only their status
        // tells, so the status word is gathered where there are such sources
        // (past v_reach: when the batch has a source there)
        uint32_t nst = ~some;
        if (in && (edged ? (some & mine) != mine : tail_src)) nst = ~gb.last[vi * WORDS + k];
        if constexpr (NP <= 7) {
          // planes in rows 0..NP-1, zero rows up to 6 (folded away by the
          // compiler), the unreached flag in row 7
#pragma unroll
          for (int b = NP; b < 7; b++) A[8 * i + b] = 0u;
          A[8 * i + 7] = nst;
        } else {
#pragma unroll
          for (int b = 0; b < 8; b++) A[8 * i + b] |= nst;
        }
      }
#if IBFS_OUT_PRMT
      transpose32_z<out_zero_rows<NP>()>(A);
#else
      transpose32(A);
#endif
      if constexpr (NP <= 7) {
        // byte i = depth (< 128) with bit 7 = unreached: widen bit 7 to the
        // whole byte (prmt in sign-replicating mode), 0xFF = INFTY
#pragma unroll
        for (int j = 0; j < 32; j++) {
          uint32_t m;
          asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(m) : "r"(A[j]));
          A[j] |= m;
        }
      }
      const int js = min(32, n_b - k * 32);
#if IBFS_OUT_FASTST
      if (full4 && js == 32) {
        // the common case: 32 whole rows, 4 in-range vertices per lane
#pragma unroll
        for (int j = 0; j < 32; j++)
          st_row4(p.out + (size_t)rows[k * 32 + j] * (size_t)p.V + v0, A[j]);
        continue;
      }
#endif
#pragma unroll
      for (int j = 0; j < 32; j++) {
        if (j < js) {
          uint8_t* row = p.out + (size_t)rows[k * 32 + j] * (size_t)p.V;
          if (full4) {
            st_row4(row + v0, A[j]);
          } else {
            for (int i = 0; i < 4; i++)
              if (v0 + i < p.V) row[v0 + i] = (uint8_t)(A[j] >> (8 * i));
          }
        }
      }
    }
  }
}

// Vertex-major, one-byte depths.  The batch's block is one byte stream
// [V][n_b] whose rows need not be aligned, so a warp takes 32 / WORDS
// vertices -- a lane per status word -- lays their rows out in shared memory
// at the stream's own 16-byte phase and writes whole 16-byte pieces, with
// bytes only at the two ends.  The next step's words are gathered before this
// one's are expanded.  500,009 vertices x 250 sources in 256-bit words:
// 1,120 us per batch with one thread per vertex storing single bytes,
// 127 us so (1 TB/s of rows).
constexpr int kVmTile = 1024 + 16;  // bytes of a warp's rows, and the phase
__device__ __forceinline__ uint8_t* vm_tile() {
  __shared__ __align__(16) uint8_t s_rows[16][kVmTile];
  return s_rows[threadIdx.x >> 5];
}

template <int WORDS, int NP>
__device__ void output_vm_u8(const Params& p, const GroupBufs& gb, uint8_t* depth_vm, int n_b,
                             const Team& t) {
  constexpr int VPS = 32 / WORDS;  // vertices per step
  const int vl = t.lane / WORDS, k = t.lane % WORDS;
  const int js = min(32, n_b - k * 32);  // sources of this lane's word (<= 0: none)
  uint8_t* tile = vm_tile();
  const long long step = t.nwarps * VPS;
  uint32_t nst = 0, npw[NP > 0 ? NP : 1];
  auto gather = [&](long long v0) {
    const long long v = v0 + vl;
    if (v < p.V && js > 0) {
      const size_t vi = (size_t)(p.vmap ? p.vmap[v] : v);
      nst = gb.last[vi * WORDS + k];
      const bool edged = (long long)vi < p.v_reach;  // as in output_sm_u8
#pragma unroll
      for (int b = 0; b < NP; b++)
        npw[b] = edged ? gb.planes[(size_t)b * p.plane_stride + vi * WORDS + k] : 0u;
    }
  };
  const long long first = t.warp * VPS;
  if (first < p.V) gather(first);
  for (long long v0 = first; v0 < p.V; v0 += step) {
    const uint32_t st = nst;
    uint32_t pw[NP > 0 ? NP : 1];
#pragma unroll
    for (int b = 0; b < NP; b++) pw[b] = npw[b];
    if (v0 + step < p.V) gather(v0 + step);
    uint8_t* dst = depth_vm + (size_t)v0 * n_b;
    const int sh = (int)(reinterpret_cast<uintptr_t>(dst) & 15);
    const int nv = (int)min((long long)VPS, p.V - v0);
    if (vl < nv && js > 0) {
      const int at = sh + vl * n_b + k * 32;
      uint8_t* q = tile + at;
#pragma unroll
      for (int j4 = 0; j4 < 8; j4++) {
        uint32_t w = nib_to_bytes(~(st >> (4 * j4)) & 0xFu) * 0xFFu;
#pragma unroll
        for (int b = 0; b < NP; b++) w |= nib_to_bytes((pw[b] >> (4 * j4)) & 0xFu) << b;
        if (j4 * 4 + 4 <= js) {
          if ((at & 3) == 0) {
            *reinterpret_cast<uint32_t*>(q + j4 * 4) = w;
          } else if ((at & 1) == 0) {
            *reinterpret_cast<uint16_t*>(q + j4 * 4) = (uint16_t)w;
            *reinterpret_cast<uint16_t*>(q + j4 * 4 + 2) = (uint16_t)(w >> 16);
          } else {
            q[j4 * 4] = (uint8_t)w;
            q[j4 * 4 + 1] = (uint8_t)(w >> 8);
            q[j4 * 4 + 2] = (uint8_t)(w >> 16);
            q[j4 * 4 + 3] = (uint8_t)(w >> 24);
          }
        } else {
          for (int i = 0; i < 4 && j4 * 4 + i < js; i++) q[j4 * 4 + i] = (uint8_t)(w >> (8 * i));
        }
      }
    }
    __syncwarp();
    const int end = sh + nv * n_b;
    for (int c = t.lane * 16; c < end; c += 512) {
      if (c >= sh && c + 16 <= end) {
        __stcs(reinterpret_cast<uint4*>(dst - sh + c), *reinterpret_cast<const uint4*>(tile + c));
      } else {
        for (int i = max(c, sh); i < min(c + 16, end); i++) dst[i - sh] = tile[i];
      }
    }
    __syncwarp();
  }
}

// Any depth width and plane count (two-byte depths): lane = vertex.
template <int WORDS>
__device__ void output_generic(const Params& p, const GroupBufs& gb, uint8_t* depth_vm,
                               const int32_t* rows, int n_b, int P, const Team& t) {
  const uint32_t inf = p.db == 1 ? 0xFFu : 0xFFFFu;
  for (long long v = t.tid; v < p.V; v += t.nthreads) {
    const size_t vi = (size_t)(p.vmap ? p.vmap[v] : v);
#pragma unroll 1
    for (int k = 0; k < WORDS && k * 32 < n_b; k++) {
      const uint32_t st = gb.last[vi * WORDS + k];
      const int js = min(32, n_b - k * 32);
      for (int j = 0; j < js; j++) {
        uint32_t d = inf;
        if ((st >> j) & 1u) {
          d = 0;
          for (int b = 0; b < P; b++)
            d |= ((gb.planes[(size_t)b * p.plane_stride + vi * WORDS + k] >> j) & 1u) << b;
        }
        uint8_t* dst = p.layout == 0
                           ? p.out + ((size_t)rows[k * 32 + j] * (size_t)p.V + (size_t)v) * p.db
                           : depth_vm + ((size_t)v * n_b + k * 32 + j) * p.db;
        if (p.db == 1) *dst = (uint8_t)d;
        else *reinterpret_cast<uint16_t*>(dst) = (uint16_t)d;
      }
    }
  }
}

template <int WORDS, int NP>
__device__ __forceinline__ void output_u8(const Params& p, const GroupBufs& gb, uint8_t* depth_vm,
                                          const int32_t* rows, int n_b, const Team& t) {
  if (p.layout == 0) output_sm_u8<WORDS, NP>(p, gb, rows, n_b, t);
  else output_vm_u8<WORDS, NP>(p, gb, depth_vm, n_b, t);
}

template <int WORDS>
__device__ void output_phase(const Params& p, const GroupBufs& gb, uint8_t* depth_vm,
                             const int32_t* rows, int n_b, int max_level, const Team& t) {
  const int P = planes_for(max_level);
  if (p.db == 1) {
    switch (P) {
      case 0: output_u8<WORDS, 0>(p, gb, depth_vm, rows, n_b, t); return;
      case 1: output_u8<WORDS, 1>(p, gb, depth_vm, rows, n_b, t); return;
      case 2: output_u8<WORDS, 2>(p, gb, depth_vm, rows, n_b, t); return;
      case 3: output_u8<WORDS, 3>(p, gb, depth_vm, rows, n_b, t); return;
      case 4: output_u8<WORDS, 4>(p, gb, depth_vm, rows, n_b, t); return;
      case 5: output_u8<WORDS, 5>(p, gb, depth_vm, rows, n_b, t); return;
      case 6: output_u8<WORDS, 6>(p, gb, depth_vm, rows, n_b, t); return;
      case 7: output_u8<WORDS, 7>(p, gb, depth_vm, rows, n_b, t); return;
      case 8: output_u8<WORDS, 8>(p, gb, depth_vm, rows, n_b, t); return;
      default: break;
    }
  }
  output_generic<WORDS>(p, gb, depth_vm, rows, n_b, P, t);
}

}  // namespace ibfs
