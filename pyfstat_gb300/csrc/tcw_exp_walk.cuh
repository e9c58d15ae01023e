// The row-table walk of an exponential column chunk, shared by the map kernels
// and the estimate of the differentiable statistics.
#pragma once

#include <stdint.h>

#include "tcw_cell.h"

namespace tcw {

constexpr uint32_t kExpRowTab = 128;

// The row-table walk of one warp's column chunk [mb, me) (regular rows):
// row tables of kExpRowTab rows built by the warp, then each lane's column
// slides down them (ExpColumn).  The walk starts at row ms - 1 >= me - 1: the
// rows of [me, ms) bring the window sums to the state that a walk from further
// up would have, without an F.  kSegs, kRunUpRows: whether the
// walk may start from segment sums and above me.
template <bool kSegs, bool kRunUpRows, class Column, class Sink>
__device__ __forceinline__ void exp_rows(Column &C, const Geom &g, uint32_t shift, uint32_t nseg,
                                         const float *__restrict__ a8,
                                         const uint32_t *__restrict__ t0s, uint32_t mb,
                                         uint32_t me, uint32_t ms, bool active, Sink &sink,
                                         ExpRow *tab, const float *__restrict__ seg) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t *a8u = reinterpret_cast<const uint32_t *>(a8);
  if (kSegs && seg && active) {  // the walk's first window, where it is long
    const uint32_t t0 = __ldg(t0s + ms - 1u);
    const uint32_t lo = exp_lo(t0, g), d = t0 - g.t0_data;
    ExpRow e;
    e.a = fdiv(d, g.div);
    e.b = d - e.a * g.TAtom;
    const uint32_t top = min(max(C.top_raw(e), 1u), g.numAtoms);
    if (lo < top && top - lo >= (2u << shift))
      C.warm_start(a8, g, seg, shift, nseg, lo, top);
  }
  // the run-up moves the window only (tables as below: rows much finer than
  // the atoms make it hundreds of rows, whose loads and divisions one after the
  // other took longer than the chunk)
  if (kRunUpRows) {
    for (uint32_t ce = ms; ce > me;) {
      const uint32_t cb = ce - me > kExpRowTab ? ce - kExpRowTab : me;
      __syncwarp();
      for (uint32_t r = lane; r < ce - cb; r += 32u) {
        const uint32_t t0 = __ldg(t0s + cb + r), d = t0 - g.t0_data;
        ExpRow e;
        e.lo = exp_lo(t0, g);
        e.nz = 0u;
        e.a = fdiv(d, g.div);
        e.b = d - e.a * g.TAtom;
        tab[r] = e;
      }
      __syncwarp();
      if (active)
        for (uint32_t m = ce; m > cb;) {
          m--;
          C.window(a8, g, tab[m - cb]);
        }
      ce = cb;
    }
  }
  for (uint32_t ce = me; ce > mb;) {
    const uint32_t cb = ce - mb > kExpRowTab ? ce - kExpRowTab : mb;
    __syncwarp();
    uint32_t t0min = 0xFFFFFFFFu;
    for (uint32_t r = lane; r < ce - cb; r += 32u) {
      const uint32_t t0 = __ldg(t0s + cb + r);
      t0min = min(t0min, t0);
      ExpRow e;
      e.lo = exp_lo(t0, g);
      const uint32_t *nz = a8u + (size_t)e.lo * 8u + 3u;
      e.nz = e.lo < g.numAtoms ? (Column::kReadOnly ? __ldg(nz) : *nz) : 0xFFFFFFFFu;
      const uint32_t d = t0 - g.t0_data;
      e.a = fdiv(d, g.div);
      e.b = d - e.a * g.TAtom;
      tab[r] = e;
    }
    __syncwarp();
    // the window end grows with t0: if it is clamped at numAtoms for the
    // chunk's smallest t0, it is for every row of the chunk
    ExpRow e0;
    const uint32_t d0 = __reduce_min_sync(0xffffffffu, t0min) - g.t0_data;
    e0.a = fdiv(d0, g.div);
    e0.b = d0 - e0.a * g.TAtom;
    const bool clamped = __all_sync(0xffffffffu, !active || C.top_raw(e0) >= g.numAtoms);
    // window starts that never grow along the walk (t0 non-decreasing in m)
    bool mono = true;
    for (uint32_t r = lane; r + 1u < ce - cb; r += 32u) mono = mono && tab[r].lo <= tab[r + 1u].lo;
    mono = __all_sync(0xffffffffu, mono);
    if (active) {
      if (clamped && mono) {
        // the rows before the first window with an atom, that row, then the
        // steady rows (row_steady's conditions hold for all of them; after
        // the first window with data, row_steady_data's too)
        uint32_t m = ce;
        while (m > cb) {
          m--;
          const ExpRow &e = tab[m - cb];
          C.row_clamped(a8, g, e, m, sink);
          if (e.lo < g.numAtoms) break;
        }
        // once a window holds data, every later (lower-starting) one does
        while (m > cb) {
          m--;
          const ExpRow &e = tab[m - cb];
          C.row_steady(a8, g, e, m, sink);
          if (e.nz < g.numAtoms) break;
        }
        while (m > cb) {
          m--;
          C.row_steady_data(a8, g, tab[m - cb], m, sink);
        }
      } else if (clamped) {
        for (uint32_t m = ce; m > cb;) {
          m--;
          C.row_clamped(a8, g, tab[m - cb], m, sink);
        }
      } else {
        for (uint32_t m = ce; m > cb;) {
          m--;
          C.row(a8, g, tab[m - cb], m, sink);
        }
      }
    }
    ce = cb;
  }
}

}  // namespace tcw
