// persistent.cuh -- the persistent kernel (IBFS_MODE_PERSISTENT): one
// cooperative launch runs every level of every batch; the grid is cut into
// G groups of CTAs, each group owns one batch at a time and synchronises with
// a bounded team barrier, and the direction decision is taken on the device.
// Each status width is instantiated in a translation unit of its own
// (persistent_w32/64/128/256.cu), which exports the kernels' addresses per
// occupancy level through persistent_fn_w<W>().
#pragma once

#include <cuda_runtime.h>

#include "bfs_device.cuh"
#include "launch_common.cuh"

namespace ibfs {

// THREADS x MINB fixes the register budget (65536 / (THREADS * MINB)) and
// hence how many warps per SM hide the latency of the random gathers.
template <int WORDS, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) persistent_kernel(Params p) {
  // The loop's state that only the decision touches lives here and not in
  // registers, which the phases need (thread 0 writes it; what every thread
  // reads alternates by level parity, with a CTA barrier in between).
  struct LoopShared {
    unsigned long long m_u[2], prev_changed[2], teps, t_lvl, t_mid;
    int td, bu, max_level;
  };
  __shared__ LoopShared s_loop;
  __shared__ int32_t s_rows[kMaxWords * 32];
  const int g = blockIdx.x / p.cpg;
  const Team t = make_team(blockIdx.x % p.cpg, p.cpg);
  GroupBufs gb = p.groups[g];  // last and curr swap roles after bottom-up levels
  Ctl* ctl = gb.ctl;
  const unsigned nb = (unsigned)p.cpg;
  const bool lead = (t.block == 0 && threadIdx.x == 0);
  bool withhold = p.withhold && t.block == 0 && g == 0;
  const long long vpad = (p.V + 31) & ~31LL;

  unsigned bar_target = 0;
#define BARRIER()                                                   \
  do {                                                              \
    bar_target += nb;                                               \
    if (!team_barrier(ctl, nb, bar_target, p.timeout_ns, withhold)) return; \
    withhold = false;                                               \
  } while (0)

  for (int b = g; b < p.nbatches; b += p.G) {
    const long long k0 = (long long)b * p.C;
    const int n_b = (int)min((long long)p.C, p.n_total - k0);
    if (threadIdx.x == 0) {
      s_loop.m_u[0] = (unsigned long long)p.E;
      s_loop.prev_changed[0] = 0;
      s_loop.teps = 0;
      s_loop.td = s_loop.bu = s_loop.max_level = 0;
      s_loop.t_lvl = s_loop.t_mid = global_ns();
    }
    zero_words(gb.last, vpad * WORDS, t);
    zero_words(gb.curr, vpad * WORDS, t);
    zero_words(gb.chg, 2 * p.chg_stride, t);
    load_rows(p, b, n_b, s_rows);
    if (t.block == 0 && threadIdx.x < 32) {
      for (int i = 0; i < 3; i++) zero_par(&ctl->par[i], t.lane);
      if (threadIdx.x < 8) (&ctl->qc[0][0])[threadIdx.x] = 0;
      if (threadIdx.x == 8) ctl->tail_src = 0;
    }
    BARRIER();
    seed_phase<WORDS, true>(p, gb, p.src + k0, n_b, t);
    BARRIER();
    if (lead) s_loop.t_mid = global_ns();
    inspect_phase<WORDS>(p, gb, &ctl->par[0], n_b, 0, true, kTdThin, ctl->qc[1], t);
    BARRIER();
    int level = 0, cur_dir = kDirTD;
    int err = 0;
    bool have_q = true;     // the queues of the next level are built (by a thin inspect)
    bool after_bu = false;  // the level before was bottom-up: `curr` is one level behind
    while (true) {
      // level-1's counters become level+2's: no CTA reads them any more, and
      // none adds to them before the next barrier
      if (t.block == 0 && threadIdx.x >= 32 && threadIdx.x < 64)
        zero_par(par_at(ctl, level + 2), t.lane);
      // Every thread takes the decision from the same counters (two 16-byte
      // loads each), so that no CTA waits for one thread's chain of loads.
      const Par* pr = par_at(ctl, level);
      const ulonglong2 c0 = __ldcg(reinterpret_cast<const ulonglong2*>(&pr->changed));
      const ulonglong2 c1 = __ldcg(reinterpret_cast<const ulonglong2*>(&pr->cdeg));
      const int range = __ldcg(&pr->range_err);
      const unsigned long long changed = c0.x, mf = c0.y, cdeg = c1.x;
      unsigned long long m_u = s_loop.m_u[level & 1];
      m_u = m_u > cdeg ? m_u - cdeg : 0ull;
      int stop = 0;
      if (range) { stop = 1; err = 3; }
      else if (changed == 0) stop = 1;
      else if (level + 1 > p.max_levels) { stop = 1; err = 3; }
      const int nd = choose_dir(level + 1, cur_dir, p.switch_level, p.alpha, p.beta, changed,
                                s_loop.prev_changed[level & 1], mf, m_u, p.V);
      if (threadIdx.x == 0) {
        s_loop.m_u[(level + 1) & 1] = m_u;
        s_loop.prev_changed[(level + 1) & 1] = changed;
        s_loop.teps += c1.y;
        if (changed && !range) s_loop.max_level = level;
        if (!stop && nd == kDirTD) s_loop.td++;
        if (!stop && nd != kDirTD) s_loop.bu++;
        if (lead) {
          if (level < p.lrec_cap) {
            LevelRec r;
            r.batch = b; r.level = level; r.dir = level == 0 ? -1 : cur_dir; r.pad = 0;
            r.frontier = (long long)changed; r.frontier_edges = (long long)mf;
            const unsigned long long t_now = global_ns();
            r.expand_ns = (long long)(s_loop.t_mid - s_loop.t_lvl);
            r.inspect_ns = (long long)(t_now - s_loop.t_mid);
            s_loop.t_lvl = t_now;
            p.lrec[(size_t)b * p.lrec_cap + level] = r;
          }
          if (!stop) ctl->qc[level & 1][0] = ctl->qc[level & 1][1] = ctl->qc[level & 1][2] = 0;
        }
      }
      if (stop) break;
      cur_dir = nd;
      const int kind = td_kind(mf, p.v_reach);
      level++;
      const bool depth_ok = level <= depth_limit(p.db);
      if (cur_dir == kDirTD) {
        zero_plane_if_first(p, gb, level, t);
        if (!have_q) {
          qbuild_phase<WORDS>(p, gb, level, ctl->qc[level & 1], t, after_bu);
          BARRIER();
        }
        td_phase<WORDS>(p, gb, level, ctl->qc[level & 1], kind, t);
        BARRIER();
        if (lead) s_loop.t_mid = global_ns();
        inspect_phase<WORDS>(p, gb, par_at(ctl, level), n_b, level, depth_ok, kind,
                             ctl->qc[(level + 1) & 1], t);
        have_q = kind == kTdThin;
        after_bu = false;
      } else {
        // Fused with its inspect work, as in the device loop: the pass writes
        // every vertex's new status to `curr`, and the buffers swap roles.
        Par* par = par_at(ctl, level);
        const Par* prev = par_at(ctl, level - 1);
        const bool filt = bu_filter_level(p.bu_filter, __ldcg(&prev->changed), p.V);
        // the level-(L+1) bitmap is the buffer of level L-1's, which only the
        // filter reads
        if (!filt) zero_words(chg_at(gb, p, level + 1), p.chg_stride, t);
        bu_phase<WORDS, true, false>(p, gb, level, prev->fmask, &par->hq_cnt, t, par, n_b,
                                     depth_ok, filt);
        BARRIER();
        if (lead) s_loop.t_mid = global_ns();
        if (__ldcg(&par->hq_cnt) > 0) {  // same value in every CTA
          bu_defer_phase<WORDS>(p, gb, level, prev->fmask, &par->hq_cnt, t, filt);
          BARRIER();
          bu_hub_epilogue<WORDS>(p, gb, par, n_b, level, depth_ok, t, !filt);
        } else if (filt) {
          zero_words(chg_at(gb, p, level + 1), p.chg_stride, t);
        }
        uint32_t* x = gb.last;
        gb.last = gb.curr;
        gb.curr = x;
        have_q = false;
        after_bu = true;
        if (!filt && __ldcg(&par->hq_cnt) == 0) continue;  // nothing since the barrier
      }
      BARRIER();
    }
    if (err) {
      if (lead) {
        atomicCAS(&ctl->err, 0, err);
        p.brec[b].err = err;
      }
      return;
    }
    __syncthreads();  // thread 0's last state
    output_phase<WORDS>(p, gb, batch_depth(p, b), s_rows, n_b, s_loop.max_level, t);
    if (lead && level + 1 < p.lrec_cap) {
      // one extra record per batch: dir 2 = the output pass
      LevelRec r;
      r.batch = b; r.level = level + 1; r.dir = 2; r.pad = 0;
      r.frontier = 0; r.frontier_edges = 0;
      r.expand_ns = (long long)(global_ns() - s_loop.t_lvl);
      r.inspect_ns = 0;
      p.lrec[(size_t)b * p.lrec_cap + level + 1] = r;
    }
    if (lead) {
      BatchRec r;
      r.levels = level;
      r.max_level = s_loop.max_level;
      r.td = s_loop.td;
      r.bu = s_loop.bu;
      r.teps = s_loop.teps;
      r.err = 0;
      r.pad = 0;
      p.brec[b] = r;
    }
    BARRIER();
  }
#undef BARRIER
}

// Occupancy levels of the persistent kernel: 512 x 2 (default), 256 x 6,
// 256 x 8 and 512 x 1 threads x CTAs per SM (the register budget; of the third
// level, 28.6 KB of shared memory a CTA let 7 reside).
template <int WORDS>
const void* persistent_fn(int level) {
  switch (level) {
    case 1: return (const void*)persistent_kernel<WORDS, 256, 6>;
    case 2: return (const void*)persistent_kernel<WORDS, 256, 8>;
    case 3: return (const void*)persistent_kernel<WORDS, 512, 1>;
    default: return (const void*)persistent_kernel<WORDS, 512, 2>;
  }
}

}  // namespace ibfs
