// CUDA kernels of the transient-CW F-statistic map for GB300 (sm_103a).
//
//   prefix kernels   compensated exclusive prefix sums of the 7 atom channels of
//                    each rectangular template (a cluster of blocks per template,
//                    one block each where there are many), stored as quantised
//                    double-word rows (see tcw_cell.h)
//   map_kernel       the (t0, tau) cells of a list of tiles; a block owns one tile
//                    (grid launch) or pulls tiles from an atomic counter
//                    (persistent launch).  Rectangular tiles difference two prefix
//                    rows per cell; exponential tiles slide one double-word window
//                    sum down each tau column (atoms enter at the lower window end
//                    and leave at the upper end).  Every block (rect: every warp
//                    of a persistent launch) reduces its cells to
//                    (max F, first argmax, sum exp(F - max F)).
//   repack_kernel    exponential templates' atoms into 32-byte rows (one 256-bit
//                    load per recurrence step)
//   finalize_kernel  per template, merges the tile partials in a fixed order:
//                    maxF, argmax, lnBtSG in FP64.
//   posterior kernels  row / column sums of exp(F - maxF) over written maps and
//                    their argmax (t0 / tau max-posterior bins), for one
//                    template or every template of a plan
//                    (post_sums_kernel, post_argmax_kernel).
// No tensor cores: nothing on this path is a dense contraction.
#include <math.h>
#include <stdint.h>

#include "../../include/tcw_b200.h"
#include "tcw_exp_walk.cuh"
#include "tcw_internal.h"

namespace tcw {

constexpr float kLog2e = 1.4426950408889634f;

// ------------------------------------------------------------------ helpers

__device__ __forceinline__ FF ff_add(FF a, FF b) {
  float s, e;
  two_sum(a.h, b.h, s, e);
  e = fadd(e, fadd(a.l, b.l));
  float s2 = fadd(s, e);
  return FF{s2, fsub(e, fsub(s2, s))};
}

__device__ __forceinline__ FF shfl_up_ff(FF v, int d) {
  return FF{__shfl_up_sync(0xffffffffu, v.h, d), __shfl_up_sync(0xffffffffu, v.l, d)};
}

// Programmatic dependent launch (the chain of small kernels of one map): a
// kernel's blocks may start while the kernel before it still runs and wait
// here until it has finished and its writes are visible; both are no-ops in
// launches without the attribute.  What the chain's own kernels write
// (descriptor, prefix and atom rows, segment sums, partials, results, maps,
// posterior sums) changes while the next kernel is resident, so it is read by
// plain loads: no __restrict__ parameter, no __ldg, no ld.global.nc, which
// promise read-only data and may move above the wait.  Kernels that plans
// launch as well, without the attribute, keep read-only loads there.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One 64-byte prefix row as two 256-bit loads (each lane's request covers
// whole 32-byte sectors); kReadOnly as in load_row8.
template <bool kReadOnly>
__device__ __forceinline__ void ld_row16(const float *p, float r[16]) {
#pragma unroll
  for (int k = 0; k < 2; k++) {
    F2 x[4];
    load_row8<kReadOnly>(p + 8 * k, x);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      r[8 * k + 2 * j] = x[j].x;
      r[8 * k + 2 * j + 1] = x[j].y;
    }
  }
}

// ------------------------------------------------------------------ repack

// One block per 256 atoms of a template (grid y: the template), several where
// the launch has fewer blocks (launch_repack).
__global__ void __launch_bounds__(256) repack_kernel(const TemplateDev *__restrict__ T,
                                                     const uint32_t *__restrict__ exp_list,
                                                     const float *__restrict__ atoms,
                                                     float *__restrict__ A8) {
  const TemplateDev t = T[exp_list[blockIdx.y]];
  for (uint64_t i0 = blockIdx.x * 256u; i0 < t.g.numAtoms; i0 += gridDim.x * 256u) {
    repack_rows(atoms + t.atom_off * 7u, reinterpret_cast<float4 *>(A8 + t.a8_off * 8u),
                t.g.numAtoms, (uint32_t)i0);
    __syncthreads();  // (its shared masks)
  }
}

// One template given by value, left at T for the launches that follow.
__global__ void __launch_bounds__(256) repack_one_kernel(const __grid_constant__ TemplateDev t,
                                                         TemplateDev *__restrict__ T,
                                                         const float *__restrict__ atoms,
                                                         float *__restrict__ A8) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x == 0 && threadIdx.x == 0) *T = t;
  repack_rows(atoms + t.atom_off * 7u, reinterpret_cast<float4 *>(A8 + t.a8_off * 8u),
              t.g.numAtoms, blockIdx.x * 256u);
}

// ------------------------------------------------------------------ prefix

template <bool kComp>
__global__ void __launch_bounds__(256) prefix_kernel(const TemplateDev *__restrict__ T,
                                                     const uint32_t *__restrict__ rect_list,
                                                     const float *__restrict__ atoms,
                                                     float *__restrict__ P) {
  const TemplateDev t = T[rect_list[blockIdx.x]];
  const uint32_t N = t.g.numAtoms;
  const float *x = atoms + t.atom_off * 7u;
  float *out = P + t.p_off * kPrefixStride;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  const uint32_t chunk = (N + 255u) / 256u;
  const uint32_t i0 = min(N, tid * chunk), i1 = min(N, i0 + chunk);

  FF loc[7];
  float sabs[7];
#pragma unroll
  for (int c = 0; c < 7; c++) {
    loc[c] = ff_zero();
    sabs[c] = 0.0f;
  }
#pragma unroll 4
  for (uint32_t i = i0; i < i1; i++) {
#pragma unroll
    for (int c = 0; c < 7; c++) {
      float v = __ldg(x + (size_t)i * 7u + c);
      loc[c] = kComp ? ff_add1(loc[c], v) : FF{fadd(loc[c].h, v), 0.0f};
      sabs[c] += fabsf(v);
    }
  }

  __shared__ FF warp_tot[8][7];
  __shared__ float warp_abs[8][7];
#pragma unroll
  for (int c = 0; c < 7; c++) {
    FF v = loc[c];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      FF o = shfl_up_ff(v, d);
      if (lane >= (uint32_t)d) v = kComp ? ff_add(o, v) : FF{fadd(o.h, v.h), 0.0f};
    }
    FF ex = shfl_up_ff(v, 1);
    if (lane == 0) ex = ff_zero();
    if (lane == 31) warp_tot[wid][c] = v;
    loc[c] = ex;
    float a = sabs[c];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
    if (lane == 0) warp_abs[wid][c] = a;
  }
  __syncthreads();

  float Q[7], invQ[7];
#pragma unroll
  for (int c = 0; c < 7; c++) {
    FF off = ff_zero();
    for (uint32_t w = 0; w < wid; w++)
      off = kComp ? ff_add(off, warp_tot[w][c]) : FF{fadd(off.h, warp_tot[w][c].h), 0.0f};
    loc[c] = kComp ? ff_add(off, loc[c]) : FF{fadd(off.h, loc[c].h), 0.0f};
    float S = 0.0f;
    for (int w = 0; w < 8; w++) S += warp_abs[w][c];
    Q[c] = prefix_quantum(S);
    invQ[c] = 1.0f / Q[c];
  }

  auto write_row = [&](uint32_t j) {
    float r[16];
#pragma unroll
    for (int c = 0; c < 7; c++) {
      if (kComp) {
        quantise_prefix(loc[c].h, loc[c].l, Q[c], invQ[c], r[c], r[8 + c]);
      } else {
        r[c] = loc[c].h;
        r[8 + c] = 0.0f;
      }
    }
    r[7] = 0.0f;
    r[15] = 0.0f;
    float4 *o = reinterpret_cast<float4 *>(out + (size_t)j * kPrefixStride);
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
  };

#pragma unroll 4
  for (uint32_t i = i0; i < i1; i++) {
    write_row(i);
#pragma unroll
    for (int c = 0; c < 7; c++) {
      float v = __ldg(x + (size_t)i * 7u + c);
      loc[c] = kComp ? ff_add1(loc[c], v) : FF{fadd(loc[c].h, v), 0.0f};
    }
  }
  if (i0 < N && i1 == N) write_row(N);
}

// prefix_kernel for few templates: a cluster of eight blocks per template.
// Rank b takes the 32 chunks of prefix_kernel's warp b, eight threads per
// chunk (one channel each, the eighth writes the pads), so that its chains
// run 1792 wide instead of 256 and its loads and row writes are whole
// sectors; one warp per channel scans the block's chunk sums as that warp
// did, and the ranks exchange their totals through distributed shared memory:
// the same sums in the same order, bit for bit.  Bound by the chunks' serial
// double-word sums (numAtoms / 256 steps, twice).  17532 atoms: 107 -> 19 us,
// 480 atoms: 8.3 -> 3.3 us.
constexpr uint32_t kPrefixCluster = 8;

template <bool kComp>
__device__ __forceinline__ void prefix_cluster(const TemplateDev &t, uint32_t rank,
                                               const float *__restrict__ atoms,
                                               float *__restrict__ P) {
  __shared__ FF s_sum[7][32];     // chunk sums, then their offsets in the block
  __shared__ float s_abs[7][32];
  __shared__ float s_tot[kPrefixCluster][7][3];  // every rank's total (h, l) and sum |x|
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint32_t N = t.g.numAtoms;
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  const uint32_t ci = threadIdx.x >> 3, c = threadIdx.x & 7u;
  const float *x = atoms + t.atom_off * 7u + c;
  const uint32_t chunk = (N + 255u) / 256u;
  const uint32_t i0 = min(N, (rank * 32u + ci) * chunk), i1 = min(N, i0 + chunk);
  FF loc = ff_zero();
  if (c < 7u) {
    float sabs = 0.0f;
#pragma unroll 8
    for (uint32_t i = i0; i < i1; i++) {
      const float v = __ldg(x + (size_t)i * 7u);
      loc = kComp ? ff_add1(loc, v) : FF{fadd(loc.h, v), 0.0f};
      sabs += fabsf(v);
    }
    s_sum[c][ci] = loc;
    s_abs[c][ci] = sabs;
  }
  __syncthreads();
  // every rank runs before its shared memory is written to
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (wid < 7u) {
    FF v = s_sum[wid][lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      FF o = shfl_up_ff(v, d);
      if (lane >= (uint32_t)d) v = kComp ? ff_add(o, v) : FF{fadd(o.h, v.h), 0.0f};
    }
    FF ex = shfl_up_ff(v, 1);
    if (lane == 0) ex = ff_zero();
    s_sum[wid][lane] = ex;
    float a = s_abs[wid][lane];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
    // lane r < 8 leaves the totals in rank r's shared memory
    const float th = __shfl_sync(0xffffffffu, v.h, 31), tl = __shfl_sync(0xffffffffu, v.l, 31);
    if (lane < kPrefixCluster) {
      const uint32_t own = (uint32_t)__cvta_generic_to_shared(&s_tot[rank][wid][0]);
      uint32_t far;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(own), "r"(lane));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(far), "f"(th) : "memory");
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(far + 4u), "f"(tl) : "memory");
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(far + 8u), "f"(a) : "memory");
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  float *out = P + t.p_off * kPrefixStride;
  float Q = 1.0f, invQ = 1.0f;
  if (c < 7u) {
    FF off = ff_zero();
    for (uint32_t w = 0; w < rank; w++) {
      const FF tw{s_tot[w][c][0], s_tot[w][c][1]};
      off = kComp ? ff_add(off, tw) : FF{fadd(off.h, tw.h), 0.0f};
    }
    const FF ex = s_sum[c][ci];
    loc = kComp ? ff_add(off, ex) : FF{fadd(off.h, ex.h), 0.0f};
    float S = 0.0f;
    for (uint32_t w = 0; w < kPrefixCluster; w++) S += s_tot[w][c][2];
    Q = prefix_quantum(S);
    invQ = 1.0f / Q;
  }
  auto write_row = [&](uint32_t j) {
    float h = 0.0f, l = 0.0f;
    if (c < 7u) {
      if (kComp)
        quantise_prefix(loc.h, loc.l, Q, invQ, h, l);
      else
        h = loc.h;
    }
    out[(size_t)j * kPrefixStride + c] = h;
    out[(size_t)j * kPrefixStride + 8u + c] = l;
  };
#pragma unroll 8
  for (uint32_t i = i0; i < i1; i++) {
    write_row(i);
    if (c < 7u) {
      const float v = __ldg(x + (size_t)i * 7u);
      loc = kComp ? ff_add1(loc, v) : FF{fadd(loc.h, v), 0.0f};
    }
  }
  if (i0 < N && i1 == N) write_row(N);
}

template <bool kComp>
__global__ void __launch_bounds__(256)
    prefix_cluster_kernel(const TemplateDev *__restrict__ T,
                          const uint32_t *__restrict__ rect_list,
                          const float *__restrict__ atoms, float *__restrict__ P) {
  const TemplateDev t = T[rect_list[blockIdx.x / kPrefixCluster]];
  prefix_cluster<kComp>(t, blockIdx.x % kPrefixCluster, atoms, P);
}

// One template given by value, left at T for the launches that follow.
template <bool kComp>
__global__ void __launch_bounds__(256)
    prefix_one_kernel(const __grid_constant__ TemplateDev t, TemplateDev *__restrict__ T,
                      const float *__restrict__ atoms, float *__restrict__ P) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x == 0 && threadIdx.x == 0) *T = t;
  prefix_cluster<kComp>(t, blockIdx.x, atoms, P);
}

// ------------------------------------------------------------------ reductions

struct Red {
  float mx;        // running max F (= best)
  int64_t bidx;    // its first flat index
  float s, c;      // sum of exp(F - mx), Kahan-compensated
  float f;         // rectangular rows: plain partial sum of the current
                   // 32-column chunk, added to (s, c) by fold()

  __device__ __forceinline__ void init() {
    mx = -INFINITY;
    bidx = INT64_MAX;
    brow = 0;
    last = 0.0f;
    s = 0.0f;
    c = 0.0f;
    f = 0.0f;
  }
  // Adds 2^d (d <= 0, relative to the running max).  Terms below 2^-60 are
  // dropped: the sum is >= 1, so even 2^22 of them change it by < 2^-38.
  __device__ __forceinline__ void add_small(float d) {
    if (d > -60.0f) add_term(ex2_approx(d));
  }
  __device__ __forceinline__ void add_term(float e) {
    float y = fsub(e, c);
    float t = fadd(s, y);
    c = fsub(fsub(t, s), y);
    s = t;
  }
  // Exponential columns visit rows in descending order at a fixed column:
  // the first occurrence of the max in row-major order is the last row seen
  // with it, so only that row is kept per cell (row_to_index forms the flat
  // index once per column).
  uint32_t brow;  // row (exp columns) or column (rect rows) of the max
  // NaN cells are skipped: they fail both comparisons and the -60 test.
  __device__ __forceinline__ void add_row_desc(float F, uint32_t m) {
    if (F >= mx) {  // one test for the common F < mx
      brow = m;
      if (F > mx) {
        const float sc = ex2_approx((mx - F) * kLog2e);
        s *= sc;
        c *= sc;
        mx = F;
        add_term(1.0f);
        return;
      }
    }
    add_small((F - mx) * kLog2e);
  }
  __device__ __forceinline__ void row_to_index(uint32_t N_tau, uint32_t n) {
    if (mx != -INFINITY) bidx = (int64_t)brow * N_tau + n;
  }
  // Rectangular rows visit columns in ascending order at a fixed row: a tie
  // never replaces the earlier maximum, so only the column of a strictly
  // larger F is kept (brow holds the column here); col_to_index forms the
  // flat index once per row.  The terms go into the plain partial f (at
  // most 32 terms <= 1 between folds, and every term is added: 2^d flushes
  // to 0 below 2^-126, and what lies between adds nothing to a sum >= 1),
  // which the row's walk folds into the Kahan pair after each 32-column
  // chunk: one addition per cell instead of a compensated one and a branch
  // (-2.7 % rect kernel time).
  __device__ __forceinline__ void add_col_asc(float F, uint32_t n) {
    if (F != F) return;  // NaN cells are skipped
    if (F > mx) {
      const float sc = ex2_approx((mx - F) * kLog2e);
      s *= sc;
      c *= sc;
      f *= sc;
      mx = F;
      brow = n;
      f = fadd(f, 1.0f);
      last = ex2_approx(0.0f);  // what add_col_asc would add for F again
    } else {
      last = ex2_approx((F - mx) * kLog2e);
      f = fadd(f, last);
    }
  }
  // add_col_asc for the same F as the previous column's: the same term.
  float last;
  __device__ __forceinline__ void add_col_same(float F) {
    if (F != F) return;
    f = fadd(f, last);
  }
  __device__ __forceinline__ void fold() {
    add_term(f);
    f = 0.0f;
  }
  __device__ __forceinline__ void col_to_index(int64_t rowidx) {
    if (mx != -INFINITY) bidx = rowidx + brow;
  }
};

struct RedVal {
  float mx;
  int64_t bidx;
  float s;
};

__device__ __forceinline__ RedVal red_combine(RedVal a, RedVal b) {
  if (a.mx == -INFINITY) return b;
  if (b.mx == -INFINITY) return a;
  RedVal r;
  if (b.mx > a.mx || (b.mx == a.mx && b.bidx < a.bidx)) {
    r.mx = b.mx;
    r.bidx = b.bidx;
  } else {
    r.mx = a.mx;
    r.bidx = a.bidx;
  }
  r.s = a.s * ex2_approx((a.mx - r.mx) * kLog2e) + b.s * ex2_approx((b.mx - r.mx) * kLog2e);
  return r;
}

__device__ __forceinline__ RedVal shfl_down_red(RedVal v, int d) {
  RedVal o;
  o.mx = __shfl_down_sync(0xffffffffu, v.mx, d);
  o.bidx = __shfl_down_sync(0xffffffffu, v.bidx, d);
  o.s = __shfl_down_sync(0xffffffffu, v.s, d);
  return o;
}

// Reduce a block's per-thread reducers and write one Partial (thread 0).
__device__ void block_reduce_store(const Red &red, Partial *out) {
  __shared__ RedVal sh[kBlock / 32];
  RedVal v{red.mx, red.bidx, fsub(red.s, red.c)};
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = red_combine(v, shfl_down_red(v, d));
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    RedVal r = sh[0];
    for (int w = 1; w < kBlock / 32; w++) r = red_combine(r, sh[w]);
    Partial p;
    p.maxF = r.mx;
    p.pad = 0;
    p.argmax = r.bidx;
    p.s = (r.mx == -INFINITY) ? 0.0 : (double)r.s;
    *out = p;
  }
  __syncthreads();
}

// ------------------------------------------------------------------ tiles

// Rectangular tile: each thread owns one row (t0) and walks the tile's
// columns, so the row's start index, its prefix row and the u32-wrap state
// are set up once per row; per cell only the end index and one prefix row
// are needed, and the next cell's prefix row is loaded while the current
// cell is computed.  A call covers the 32 rows of row group my_rg and
// column range my_cg of cgs equal ranges: one-tile-per-block launches give
// the block's 4 warps (rg row groups) x (4/rg column ranges), persistent
// launches give one warp all row groups in turn with cgs = 1.  The columns'
// taus are staged 32 at a time in the warp's `stau` slots of shared memory
// (one coalesced load per 32 columns instead of a global load on every
// cell's end-index chain).  With a map to write, each warp transposes
// 32 x 32 blocks through shared memory so that global stores are
// row-contiguous.
template <bool kWrite, int kPrec, bool kReadOnly>
__device__ void rect_tile(const TemplateDev &t, const WorkItem &w,
                          const uint32_t *__restrict__ t0s_all,
                          const uint32_t *__restrict__ taus_all, const float *__restrict__ P_all,
                          float *__restrict__ Fmn, Red &red, float *smw, uint32_t my_rg,
                          uint32_t cgs, uint32_t my_cg, uint32_t *stau) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t mbase = w.m0 + 32u * my_rg;
  const uint32_t m = mbase + lane;
  const bool row_ok = m < w.m1;
  const uint32_t ncols = w.n1 - w.n0;
  const uint32_t per = (ncols + cgs - 1u) / cgs;
  const uint32_t nb = min(w.n1, w.n0 + my_cg * per), ne = min(w.n1, nb + per);
  const uint32_t *t0s = t0s_all + t.t0_off;
  const uint32_t *taus = taus_all + t.tau_off;
  const float *P = P_all + t.p_off * kPrefixStride;
  const uint32_t tau_first = __ldg(taus);
  uint32_t t0 = 0, j0 = 0, ef = 0;
  bool wr = false;
  float row0[16];
  if (row_ok) {
    t0 = __ldg(t0s + m);
    j0 = idx_start(t0, t.g);
    wr = rect_row_wrapped(t0, tau_first, t.g);
    ef = wr ? idx_end(t0 + tau_first, t.g) : 0u;
    TCW_DCHECK(j0 <= t.g.numAtoms);
    ld_row16<kReadOnly>(P + (size_t)j0 * kPrefixStride, row0);
  }
  auto end_of = [&](uint32_t tau) {
    uint32_t e = idx_end(t0 + tau, t.g);
    return (wr && ef > e) ? ef : e;
  };
  const int64_t rowidx = (int64_t)m * t.N_tau;
  // e < numAtoms always, so prefix row e + 1 exists even for empty windows
  uint32_t e_cur = 0;
  float cur[16], nxt[16];
  if (row_ok && nb < ne) {
    e_cur = end_of(__ldg(taus + nb));
    TCW_DCHECK(e_cur + 1u <= t.g.numAtoms);
    ld_row16<kReadOnly>(P + (size_t)(e_cur + 1u) * kPrefixStride, cur);
  }
  // One cell: F of column n from prefix row `a` (end ea); the next column's
  // prefix row is loaded into `b` (end eb) while this one is computed.  A
  // column whose window end equals the previous column's has the same
  // window, hence the same F: it takes the previous F, and its prefix row is
  // not loaded (the window ends of a row are clamped at the last atom once
  // t0 + tau passes the data, and taus closer than TAtom share ends).
  uint32_t e_prev = 0xFFFFFFFFu;  // end of the previous column (none yet)
  float F_prev = 2.0f;
  auto cell = [&](uint32_t n, uint32_t cb, const float *a, uint32_t ea, float *b,
                  uint32_t &eb) {
    if (row_ok && n + 1u < ne) {
      eb = end_of(n + 1u < cb + 32u ? stau[n + 1u - cb] : __ldg(taus + n + 1u));
      TCW_DCHECK(eb + 1u <= t.g.numAtoms);
      if (eb != ea) ld_row16<kReadOnly>(P + (size_t)(eb + 1u) * kPrefixStride, b);
    }
    float F = F_prev;
    if (row_ok) {
      if (ea != e_prev) F = 2.0f;
      if (ea != e_prev && ea >= j0) {
        bool ok;
        if (kPrec == kPrecPlain32) {
          F = fstat_plain32(fsub(a[0], row0[0]), fsub(a[1], row0[1]), fsub(a[2], row0[2]),
                            fsub(a[3], row0[3]), fsub(a[4], row0[4]), fsub(a[5], row0[5]),
                            fsub(a[6], row0[6]), ok);
        } else {
          FF2 W[4];
#pragma unroll
          for (int k = 0; k < 4; k++) {
            W[k].h = sub2(F2{a[2 * k], a[2 * k + 1]}, F2{row0[2 * k], row0[2 * k + 1]});
            W[k].l = sub2(F2{a[8 + 2 * k], a[9 + 2 * k]}, F2{row0[8 + 2 * k], row0[9 + 2 * k]});
          }
          F = fstat_tiered2<kPrec == kPrecFF_F64Det>(W, ok);
        }
      }
      if (ea != e_prev)
        red.add_col_asc(F, n);
      else
        red.add_col_same(F);
    }
    e_prev = ea;
    F_prev = F;
    if (kWrite) smw[lane * 33u + (n - cb)] = F;
  };
  for (uint32_t cb = nb; cb < ne; cb += 32u) {
    const uint32_t ce = min(ne, cb + 32u);
    __syncwarp();
    if (cb + lane < ne) stau[lane] = __ldg(taus + cb + lane);
    __syncwarp();
    // A chunk inside every warp row's clamped run -- the window ends of the
    // previous column and of column cb at the last atom, the chunk's taus
    // (and the next chunk's first) non-decreasing, t0 + tau past the u32
    // wrap of the reference's end index and without overflow, TAtom >= 2 (so
    // the end index's quotient never reaches 2^31) -- has the last atom as
    // every window end, so every column repeats the previous F.
    const uint32_t nlast = ce - cb - 1u;
    const uint32_t tx = ce < ne ? __ldg(taus + ce) : 0u;
    bool mono = true;
    if (lane < nlast) mono = stau[lane] <= stau[lane + 1u];
    if (lane == nlast && ce < ne) mono = stau[lane] <= tx;
    const uint32_t tmax = ce < ne ? tx : stau[nlast];
    const bool clamped_run =
        !row_ok || (t.g.TAtom >= 2u && e_cur == t.g.numAtoms - 1u &&
                    e_prev == t.g.numAtoms - 1u &&
                    (uint64_t)t0 + stau[0] + t.g.half >= (uint64_t)t.g.t0_data &&
                    (uint64_t)t0 + tmax + t.g.half - t.g.t0_data <= 0xFFFFFFFFull &&
                    (uint64_t)t0 + tmax <= 0xFFFFFFFFull);
    uint32_t n = cb;
    if (__all_sync(0xffffffffu, mono && clamped_run)) {
      for (; n < ce; n++) {
        if (row_ok) red.add_col_same(F_prev);
        if (kWrite) smw[lane * 33u + (n - cb)] = F_prev;
      }
      e_cur = t.g.numAtoms - 1u;  // the end of column ce
    }
    // ping-pong between the two row buffers; `cur` holds column n on entry
    for (; n + 1u < ce; n += 2u) {
      uint32_t e_nxt = 0;
      cell(n, cb, cur, e_cur, nxt, e_nxt);
      cell(n + 1u, cb, nxt, e_nxt, cur, e_cur);
    }
    if (n < ce) {  // odd chunk length: one more cell, then its successor moves to `cur`
      uint32_t e_nxt = 0;
      cell(n, cb, cur, e_cur, nxt, e_nxt);
#pragma unroll
      for (int k = 0; k < 16; k++) cur[k] = nxt[k];
      e_cur = e_nxt;
    }
    if (kWrite) {
      __syncwarp();
      const uint32_t col = cb + lane;
      for (uint32_t r = 0; r < 32u; r++) {
        const uint32_t mr = mbase + r;
        if (mr < w.m1 && col < ce) Fmn[t.map_off + (size_t)mr * t.N_tau + col] = smw[r * 33u + lane];
      }
      __syncwarp();
    }
    red.fold();
  }
  if (row_ok) red.col_to_index(rowidx);
}

template <bool kWrite>
struct MapSink {
  float *Fmn;
  uint32_t N_tau, n;
  Red *red;
  __device__ __forceinline__ void operator()(uint32_t m, float F, bool) {
    TCW_DCHECK(n < N_tau);
    if (kWrite) Fmn[(size_t)m * N_tau + n] = F;
    red->add_row_desc(F, m);
  }
};

// Exponential tile: each thread runs one tau column over a chunk of rows
// (the chunk is the same for the 32 lanes of a warp: tn >= 32).  When every
// row of the warp's chunk satisfies exp_row_regular for its columns' largest
// tau, the per-row quantities (ExpRow: window start, first non-zero atom,
// t0 split by TAtom) are tabulated 128 rows at a time by the warp itself in
// its own shared-memory slots (no block barrier) and every cell takes the
// division-free window end of ExpColumn; otherwise the warp runs
// exp_column2's generic index arithmetic.  Both give identical results.
template <bool kWrite, int kPrec, bool kChunks, bool kWarp>
__device__ void exp_tile(const TemplateDev &t, const WorkItem &w, const float *__restrict__ atoms,
                         const float *__restrict__ atoms8,
                         const uint32_t *__restrict__ t0s_all,
                         const uint32_t *__restrict__ taus_all, float *__restrict__ Fmn,
                         Red &red, ExpRow *tab, const float *__restrict__ G) {
  const uint32_t *t0s = t0s_all + t.t0_off;
  const uint32_t tn = w.tn;
  const uint32_t lane = threadIdx.x & 31u;
  // a warp tile (persistent launches) is 32 columns over all the tile's rows
  const uint32_t col = kWarp ? lane : threadIdx.x % tn;
  const uint32_t rl = kWarp ? 0u : threadIdx.x / tn;
  const uint32_t n = w.n0 + col;
  // the rows [mb, me) of the history that ends at h1: a warp tile's own, or
  // chunk m0 + rl of a single map (uniform per warp, tn >= 32)
  uint32_t mb = w.m0, me = w.m1, h1 = me;
  if (kWarp) {
    // (holds for every tile; with the exit the register allocator spills 48
    // bytes of the whole-column kernel, without it 80)
    if (mb >= t.N_t0) return;
    if (kChunks) h1 = min(t.N_t0, mb / t.e_hist * t.e_hist + t.e_hist);
  } else {
    const uint32_t chunk = w.m0 + rl;
    if (chunk >= w.m1) return;
    const uint32_t h0 = chunk / t.e_sub * t.e_hist;
    h1 = min(t.N_t0, h0 + t.e_hist);
    mb = h0 + chunk % t.e_sub * t.e_rows;
    if (mb >= h1) return;
    me = min(h1, mb + t.e_rows);
  }
  const bool active = n < w.n1;
  const uint32_t tau = active ? __ldg(taus_all + t.tau_off + n) : 0u;
  MapSink<kWrite> sink{kWrite ? Fmn + t.map_off : nullptr, t.N_tau, n, &red};
  if (kPrec == kPrecPlain32) {
    if (active) {
      exp_column<false, false>(atoms + t.atom_off * 7u, t.g, t0s, mb, me, tau, sink, nullptr);
      red.row_to_index(t.N_tau, n);
    }
    return;
  }
  const float *a8 = atoms8 + t.a8_off * 8u;
  const uint32_t taumax = __reduce_max_sync(0xffffffffu, tau);
  // run-up over the history above the chunk (kShortWindow, kRunUp)
  uint32_t ms = me;
  if (kChunks && me < h1) {
    const uint32_t taumin = __reduce_min_sync(0xffffffffu, active ? tau : 0xFFFFFFFFu);
    if (3ull * taumin < (uint64_t)kShortWindow * t.g.TAtom) {
      const uint64_t longest = min((uint64_t)taumax, (uint64_t)kShortWindow * t.g.TAtom / 3u + 1u);
      const uint64_t from = __ldg(t0s + me - 1u) + kRunUp * longest + 8ull * t.g.TAtom;
      uint32_t found = 0;
      for (uint32_t r = me; r < h1 && !found; r += 32u) {
        found = __ballot_sync(0xffffffffu, r + lane < h1 && __ldg(t0s + r + lane) >= from);
        ms = found ? r + __ffs(found) : h1;
      }
    }
  }
  bool reg = true;
  for (uint32_t m = mb + lane; m < ms; m += 32u)
    reg = reg && exp_row_regular(__ldg(t0s + m), taumax, t.g);
  if (!__all_sync(0xffffffffu, reg)) {
    if (active) {
      exp_column2<kPrec == kPrecFF_F64Det, kWarp>(a8, t.g, t0s, mb, me, tau, sink, nullptr);
      red.row_to_index(t.N_tau, n);
    }
    return;
  }
  const float *seg =
      t.g_nseg ? G + (t.g_off + (size_t)(n >> 5) * t.g_nseg) * kSegFloats + lane : nullptr;
  ExpColumn<kPrec == kPrecFF_F64Det, true, false, kWarp> C;
  C.init(t.g, tau);
  exp_rows<kChunks, kChunks>(C, t.g, t.g_shift, t.g_nseg, a8, t0s, mb, me, ms, active, sink, tab, seg);
  if (active) red.row_to_index(t.N_tau, n);
}

// Segment sums of exp columns: a warp takes `per` segments of one
// 32-column group, each lane one column, and enters the segment's atoms into
// an empty window (the map kernel's steps).  They let a column be cut into
// row chunks whose first window is combined from whole segments
// (ExpColumn::warm_start) instead of entered atom by atom, at the price of
// one more pass over the atoms per column -- fully parallel.  Column groups
// whose windows are shorter than two segments are never combined and are
// skipped.  Bound by the FP32 pipe and the latency of the double-word steps:
// 186 us for 17532 atoms x 4096 columns.  The map kernel behind it goes from
// 3331 us (16 chunks per column, each entering up to 17532 atoms) to 440 us
// there (one-year 8192 x 4096 map), from 645 us (whole columns, one warp per
// 32) to 188 us for 12 templates of up to 1500 atoms and 600 x 600 cells.
template <bool kList>
__global__ void __launch_bounds__(128, 8)
    exp_seg_kernel(const TemplateDev *T, const SegItem *__restrict__ items,
                   uint32_t n_items, uint32_t per, const float *atoms8,
                   const uint32_t *__restrict__ taus_all, float *__restrict__ G) {
  const uint32_t wi = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  pdl_begin();
  if (wi >= n_items) return;
  SegItem w;
  if (kList) {
    w = items[wi];
  } else {
    const uint32_t ncg = (T[0].N_tau + 31u) >> 5;
    w.tmpl = 0;
    w.cg = wi % ncg;
    w.j0 = wi / ncg * per;
    w.j1 = min(T[0].g_nseg, w.j0 + per);
  }
  const TemplateDev t = T[w.tmpl];
  const uint32_t n = w.cg * 32u + lane;
  uint32_t tau = n < t.N_tau ? __ldg(taus_all + t.tau_off + n) : 0u;
  const uint32_t taumax = __reduce_max_sync(0xffffffffu, tau);
  // a window holds fewer than 3 tau / TAtom + 2 atoms
  if (3ull * taumax + 2ull * t.g.TAtom < ((uint64_t)t.g.TAtom << (t.g_shift + 1u))) return;
  if (n >= t.N_tau) tau = taumax;
  const float *a8 = atoms8 + t.a8_off * 8u;
  ExpColumn<false, true, false, kList> C;
  C.init(t.g, tau);
  for (uint32_t j = w.j0; j < w.j1; j++) {
    C.reset_window(min(t.g.numAtoms, (j + 1u) << t.g_shift));
    C.enter_to(a8, t.g, j << t.g_shift);
    C.store_sums(G + (t.g_off + (size_t)w.cg * t.g_nseg + j) * kSegFloats + lane);
  }
}

// Minimum resident blocks per SM requested from the register allocator
// (build-time tunables; 1 leaves the allocation to ptxas).
#ifndef TCW_RECT_MIN_BLOCKS
#define TCW_RECT_MIN_BLOCKS 5
#endif
// The persistent exp kernels (the batched plans' hot kernels, with or
// without maps) run fastest at 8 blocks (64 registers, a few spilled); the
// one-tile-per-block exp kernels of single-template calls keep 96 registers
// without spills (their grids are small, so latency matters more than
// occupancy).
#ifndef TCW_EXP_MIN_BLOCKS
#define TCW_EXP_MIN_BLOCKS 8
#endif
#ifndef TCW_EXP_MIN_BLOCKS_OTHER
#define TCW_EXP_MIN_BLOCKS_OTHER 5
#endif

// Launches whose columns are cut are small: registers matter more than
// occupancy (24 templates 210 / 189 / 182 us at 8 / 6 / 5 blocks, 96 templates
// with maps 2.67 / 2.57 / 2.61 ms).
#ifndef TCW_EXP_MIN_BLOCKS_CHUNKS
#define TCW_EXP_MIN_BLOCKS_CHUNKS 6
#endif

template <int kWin, bool kPersist, bool kChunks>
constexpr int map_min_blocks() {
  return kWin == TCW_WINDOW_RECT ? TCW_RECT_MIN_BLOCKS
         : !kPersist             ? TCW_EXP_MIN_BLOCKS_OTHER
         : kChunks               ? TCW_EXP_MIN_BLOCKS_CHUNKS
                                 : TCW_EXP_MIN_BLOCKS;
}

// kChunks (exponential windows): columns may be cut into row chunks within a
// history (TemplateDev::e_sub > 1).
template <int kWin, bool kPersist, bool kWrite, int kPrec, bool kChunks>
__global__ void __launch_bounds__(kBlock, (map_min_blocks<kWin, kPersist, kChunks>()))
    map_kernel(const TemplateDev *T, const WorkItem *__restrict__ items,
               uint32_t n_items, uint32_t *__restrict__ counter, const float *__restrict__ atoms,
               const float *atoms8, const uint32_t *__restrict__ t0s,
               const uint32_t *__restrict__ taus, const float *P, const float *G,
               float *__restrict__ Fmn, Partial *__restrict__ parts) {
  constexpr uint32_t kSmem = kWin == TCW_WINDOW_RECT ? (kWrite ? (kBlock / 32) * 32 * 33 : 1)
                                                     : (kBlock / 32) * kExpRowTab * 4;
  __shared__ __align__(16) uint32_t sm[kSmem];
  __shared__ uint32_t s_tau[kWin == TCW_WINDOW_RECT ? kBlock : 1];
  if (kWin == TCW_WINDOW_RECT && kPersist) {
    // Persistent rectangular launches schedule by warp: each warp fetches
    // whole tiles and walks their 32-row groups in turn, merging the groups'
    // reducers in row order, so no block barrier waits on the slowest warp
    // (rect warps share no shared memory).
    const uint32_t lane = threadIdx.x & 31u;
    float *smw = reinterpret_cast<float *>(sm) + (threadIdx.x >> 5) * (32 * 33);
    for (;;) {
      uint32_t it2 = 0;
      if (lane == 0) it2 = atomicAdd(counter, 1u);
      it2 = __shfl_sync(0xffffffffu, it2, 0);
      if (it2 >= n_items) break;
      const WorkItem w = items[it2];
      const TemplateDev t = T[w.tmpl];
      RedVal acc{-INFINITY, INT64_MAX, 0.0f};
      for (uint32_t g = 0; g < w.tn; g++) {
        Red red;
        red.init();
        rect_tile<kWrite, kPrec, true>(t, w, t0s, taus, P, Fmn, red, smw, g, 1u, 0u,
                                       s_tau + (threadIdx.x >> 5) * 32u);
        acc = red_combine(acc, RedVal{red.mx, red.bidx, fsub(red.s, red.c)});
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc = red_combine(acc, shfl_down_red(acc, d));
      if (lane == 0) {
        Partial pp;
        pp.maxF = acc.mx;
        pp.pad = 0;
        pp.argmax = acc.bidx;
        pp.s = (acc.mx == -INFINITY) ? 0.0 : (double)acc.s;
        parts[w.part] = pp;
      }
    }
    return;
  }
  if (kWin == TCW_WINDOW_EXP && kPersist) {
    // Persistent exponential launches schedule by warp as well: each warp
    // fetches 32-column tiles (all rows of a row chunk), keeps its row table
    // in its own shared-memory slots and reduces its tile itself, so no block
    // barrier waits for the warp with the most removals.
    const uint32_t lane = threadIdx.x & 31u;
    ExpRow *tab = reinterpret_cast<ExpRow *>(sm) + (threadIdx.x >> 5) * kExpRowTab;
    for (;;) {
      uint32_t it2 = 0;
      if (lane == 0) it2 = atomicAdd(counter, 1u);
      it2 = __shfl_sync(0xffffffffu, it2, 0);
      if (it2 >= n_items) break;
      const WorkItem w = items[it2];
      const TemplateDev t = T[w.tmpl];
      Red red;
      red.init();
      exp_tile<kWrite, kPrec, kChunks, true>(t, w, atoms, atoms8, t0s, taus, Fmn, red, tab, G);
      RedVal acc{red.mx, red.bidx, fsub(red.s, red.c)};
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc = red_combine(acc, shfl_down_red(acc, d));
      if (lane == 0) {
        Partial pp;
        pp.maxF = acc.mx;
        pp.pad = 0;
        pp.argmax = acc.bidx;
        pp.s = (acc.mx == -INFINITY) ? 0.0 : (double)acc.s;
        parts[w.part] = pp;
      }
      __syncwarp();
    }
    return;
  }
  if (kPersist) return;
  // one tile of template 0 per block
  pdl_begin();
  const TemplateDev t = T[0];
  WorkItem w;
  w.tmpl = 0;
  w.part = blockIdx.x;
  const uint32_t nt = blockIdx.x / t.tile_rows, mt = blockIdx.x - nt * t.tile_rows;
  w.n0 = nt * t.tile_tn;
  w.n1 = min(t.N_tau, w.n0 + t.tile_tn);
  w.m0 = mt * t.tile_tm;
  Red red;
  red.init();
  if (kWin == TCW_WINDOW_RECT) {
    w.m1 = min(t.N_t0, w.m0 + t.tile_tm);
    w.tn = (uint16_t)(t.tile_tm / 32u);  // row groups of 32 rows (one per warp)
    const uint32_t warp = threadIdx.x >> 5, rg = w.tn;
    rect_tile<kWrite, kPrec, false>(t, w, t0s, taus, P, Fmn, red,
                                    reinterpret_cast<float *>(sm) + warp * (32 * 33), warp % rg,
                                    4u / rg, warp / rg, s_tau + warp * 32u);
  } else {
    w.m1 = w.m0 + t.tile_tm;
    w.tn = (uint16_t)t.tile_tn;
    exp_tile<kWrite, kPrec, kChunks, false>(
        t, w, atoms, atoms8, t0s, taus, Fmn, red,
        reinterpret_cast<ExpRow *>(sm) + (threadIdx.x >> 5) * kExpRowTab, G);
  }
  block_reduce_store(red, parts + w.part);
}

// ------------------------------------------------------------------ finalize

// One warp per template: merge its partials in index order.
__global__ void __launch_bounds__(128) finalize_kernel(const TemplateDev *T,
                                                       uint32_t n_templates,
                                                       const Partial *parts,
                                                       tcw_result *__restrict__ results) {
  const uint32_t tmpl = blockIdx.x * 4u + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31u;
  pdl_begin();
  if (tmpl >= n_templates) return;
  const TemplateDev t = T[tmpl];
  float best = -INFINITY;
  int64_t bidx = INT64_MAX;
  for (uint32_t k = lane; k < t.n_parts; k += 32) {
    const Partial p = parts[t.part_off + k];
    if (p.maxF > best || (p.maxF == best && p.argmax < bidx)) {
      best = p.maxF;
      bidx = p.argmax;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    float ob = __shfl_xor_sync(0xffffffffu, best, d);
    int64_t oi = __shfl_xor_sync(0xffffffffu, bidx, d);
    if (ob > best || (ob == best && oi < bidx)) {
      best = ob;
      bidx = oi;
    }
  }
  double S = 0.0;
  for (uint32_t k = lane; k < t.n_parts; k += 32) {
    const Partial p = parts[t.part_off + k];
    if (p.s > 0.0) S += p.s * (double)exp2f((p.maxF - best) * kLog2e);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) S += __shfl_xor_sync(0xffffffffu, S, d);
  if (lane == 0) {
    tcw_result r;
    r.maxF = best;
    r.argmax = bidx;
    r.lnBtSG = t.ln_prior + (double)best + log(S);
    r.t0_mp_idx = -1;
    r.tau_mp_idx = -1;
    r.status = 0;
    results[tmpl] = r;
  }
}

// ------------------------------------------------------------------ launchers

// Launches `kernel`; `pdl`: as the programmatic dependent of the kernel before
// it in the stream (which must be one of the same chain).
template <class... KArgs, class... Args>
static cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block,
                                 cudaStream_t stream, bool pdl, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t launch_exp_segments(const TemplateDev *d_T, const SegItem *d_items, uint32_t n_items,
                                uint32_t per, const float *d_atoms8, const uint32_t *d_taus,
                                float *d_G, cudaStream_t stream) {
  if (n_items == 0) return cudaSuccess;
  const uint32_t blocks = (n_items + 3u) / 4u;
  if (d_items)
    return launch_kernel(exp_seg_kernel<true>, blocks, 128, stream, false, d_T, d_items, n_items,
                         per, d_atoms8, d_taus, d_G);
  return launch_kernel(exp_seg_kernel<false>, blocks, 128, stream, true, d_T, d_items, n_items,
                       per, d_atoms8, d_taus, d_G);
}

// Templates up to which a prefix scan takes a cluster each; more run one block
// each, which costs no redundant scans.  Above 152 the scans run beside the exp
// map kernel, where a lone block's chain of scans is what the rect tiles wait
// for (one block / cluster per template, whole run: 172 templates 1.28 / 1.25
// ms, 500 2.35 / 2.22, 570 1.81 / 1.78, 700 0.295 / 0.303).
constexpr uint32_t kPrefixFew = 600;

cudaError_t launch_prefix(const TemplateDev *d_T, const uint32_t *d_rect_list, uint32_t n_rect,
                          const float *d_atoms, float *d_P, int prec, cudaStream_t stream) {
  if (n_rect == 0) return cudaSuccess;
  if (n_rect <= kPrefixFew) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_rect * kPrefixCluster);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kPrefixCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return prec == kPrecPlain32
               ? cudaLaunchKernelEx(&cfg, prefix_cluster_kernel<false>, d_T, d_rect_list, d_atoms,
                                    d_P)
               : cudaLaunchKernelEx(&cfg, prefix_cluster_kernel<true>, d_T, d_rect_list, d_atoms,
                                    d_P);
  }
  if (prec == kPrecPlain32)
    prefix_kernel<false><<<n_rect, 256, 0, stream>>>(d_T, d_rect_list, d_atoms, d_P);
  else
    prefix_kernel<true><<<n_rect, 256, 0, stream>>>(d_T, d_rect_list, d_atoms, d_P);
  return cudaGetLastError();
}

cudaError_t launch_prepare_one(const TemplateDev &t, TemplateDev *d_T, const float *d_atoms,
                               float *d_rows, int prec, cudaStream_t stream) {
  if (t.window != TCW_WINDOW_RECT)
    return launch_kernel(repack_one_kernel, (t.g.numAtoms + 255u) / 256u, 256, stream, false, t,
                         d_T, d_atoms, d_rows);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kPrefixCluster);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kPrefixCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return prec == kPrecPlain32
             ? cudaLaunchKernelEx(&cfg, prefix_one_kernel<false>, t, d_T, d_atoms, d_rows)
             : cudaLaunchKernelEx(&cfg, prefix_one_kernel<true>, t, d_T, d_atoms, d_rows);
}

template <int kWin, bool kPersist, bool kWrite, bool kChunks>
static cudaError_t launch_map_prec(int prec, uint32_t grid, cudaStream_t s, int priority,
                                   bool chained,
                                   const TemplateDev *T, const WorkItem *items, uint32_t n_items,
                                   uint32_t *counter, const float *atoms, const float *atoms8,
                                   const uint32_t *t0s, const uint32_t *taus, const float *P,
                                   const float *G, float *Fmn, Partial *parts) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kBlock);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  if (kPersist) {
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = priority;
  } else {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = kPersist || chained ? 1 : 0;
  if (prec == kPrecPlain32)
    return cudaLaunchKernelEx(&cfg, map_kernel<kWin, kPersist, kWrite, kPrecPlain32, false>, T,
                              items, n_items, counter, atoms, atoms8, t0s, taus, P, G, Fmn, parts);
  if (prec == kPrecFF_F64Det)
    return cudaLaunchKernelEx(&cfg, map_kernel<kWin, kPersist, kWrite, kPrecFF_F64Det, kChunks>, T,
                              items, n_items, counter, atoms, atoms8, t0s, taus, P, G, Fmn, parts);
  return cudaLaunchKernelEx(&cfg, map_kernel<kWin, kPersist, kWrite, kPrecFF, kChunks>, T, items,
                            n_items, counter, atoms, atoms8, t0s, taus, P, G, Fmn, parts);
}

template <int kWin>
static cudaError_t launch_map_win(const MapLaunch &L, cudaStream_t stream) {
  if (L.n_items == 0) return cudaSuccess;
  const uint32_t grid = L.persistent ? L.n_blocks : L.n_items;
  constexpr bool kExp = kWin == TCW_WINDOW_EXP;
  auto launch = [&](auto fn) {
    return fn(L.prec, grid, stream, L.priority, L.chained, L.T, L.items, L.n_items, L.counter, L.atoms,
              L.atoms8, L.t0s, L.taus, L.P, L.G, L.Fmn, L.parts);
  };
  if (!L.persistent)
    return L.write_map ? launch(launch_map_prec<kWin, false, true, kExp>)
                       : launch(launch_map_prec<kWin, false, false, kExp>);
  if (kExp && L.chunks)
    return L.write_map ? launch(launch_map_prec<kWin, true, true, kExp>)
                       : launch(launch_map_prec<kWin, true, false, kExp>);
  return L.write_map ? launch(launch_map_prec<kWin, true, true, false>)
                     : launch(launch_map_prec<kWin, true, false, false>);
}

cudaError_t launch_repack(const TemplateDev *d_T, const uint32_t *d_exp_list, uint32_t n_exp,
                          uint32_t max_atoms, const float *d_atoms, float *d_atoms8,
                          cudaStream_t stream) {
  // At most 2^16 blocks: one template of 17532 atoms among 20000 of 48 gave 1.4e6
  // (0.6 of 7.2 ms a run), nearly all of them empty.
  for (uint32_t y0 = 0; y0 < n_exp; y0 += 65535u) {
    const uint32_t ny = n_exp - y0 < 65535u ? n_exp - y0 : 65535u;
    const uint32_t nx = (max_atoms + 255u) / 256u, most = 65536u / ny;
    const dim3 grid(nx < most ? nx : most, ny);
    repack_kernel<<<grid, 256, 0, stream>>>(d_T, d_exp_list + y0, d_atoms, d_atoms8);
  }
  return cudaGetLastError();
}

cudaError_t launch_map(int window, const MapLaunch &L, cudaStream_t stream) {
  cudaError_t e = window == TCW_WINDOW_RECT ? launch_map_win<TCW_WINDOW_RECT>(L, stream)
                                            : launch_map_win<TCW_WINDOW_EXP>(L, stream);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

template <int kWin, bool kChunks>
static int blocks_per_sm_win(int prec) {
  int n = 0;
  cudaError_t e;
  if (prec == kPrecPlain32)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &n, map_kernel<kWin, true, false, kPrecPlain32, false>, kBlock, 0);
  else if (prec == kPrecFF_F64Det)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &n, map_kernel<kWin, true, false, kPrecFF_F64Det, kChunks>, kBlock, 0);
  else
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &n, map_kernel<kWin, true, false, kPrecFF, kChunks>, kBlock, 0);
  if (e != cudaSuccess) {
    cudaGetLastError();
    n = 1;
  }
  return n > 0 ? n : 1;
}

// Resident blocks per SM of the persistent (map-less) kernel of a window.
int map_blocks_per_sm(int window, int prec, bool chunks) {
  return window == TCW_WINDOW_RECT ? blocks_per_sm_win<TCW_WINDOW_RECT, false>(prec)
         : chunks                  ? blocks_per_sm_win<TCW_WINDOW_EXP, true>(prec)
                                   : blocks_per_sm_win<TCW_WINDOW_EXP, false>(prec);
}

// One block per template where there are few (up to thousands of tiles
// each): its partials merged by 256 threads, warps' results combined in warp
// order.
__global__ void __launch_bounds__(256) finalize_block_kernel(const TemplateDev *T,
                                                             const Partial *parts,
                                                             tcw_result *__restrict__ results) {
  __shared__ float s_best[8];
  __shared__ int64_t s_bidx[8];
  __shared__ double s_sum[8];
  pdl_begin();
  const TemplateDev t = T[blockIdx.x];
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  float best = -INFINITY;
  int64_t bidx = INT64_MAX;
  for (uint32_t k = threadIdx.x; k < t.n_parts; k += blockDim.x) {
    const Partial p = parts[t.part_off + k];
    if (p.maxF > best || (p.maxF == best && p.argmax < bidx)) {
      best = p.maxF;
      bidx = p.argmax;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    float ob = __shfl_xor_sync(0xffffffffu, best, d);
    int64_t oi = __shfl_xor_sync(0xffffffffu, bidx, d);
    if (ob > best || (ob == best && oi < bidx)) {
      best = ob;
      bidx = oi;
    }
  }
  if (lane == 0) {
    s_best[wid] = best;
    s_bidx[wid] = bidx;
  }
  __syncthreads();
  best = s_best[0];
  bidx = s_bidx[0];
  for (uint32_t w = 1; w < blockDim.x / 32u; w++)
    if (s_best[w] > best || (s_best[w] == best && s_bidx[w] < bidx)) {
      best = s_best[w];
      bidx = s_bidx[w];
    }
  double S = 0.0;
  for (uint32_t k = threadIdx.x; k < t.n_parts; k += blockDim.x) {
    const Partial p = parts[t.part_off + k];
    if (p.s > 0.0) S += p.s * (double)exp2f((p.maxF - best) * kLog2e);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) S += __shfl_xor_sync(0xffffffffu, S, d);
  if (lane == 0) s_sum[wid] = S;
  __syncthreads();
  if (threadIdx.x == 0) {
    S = 0.0;
    for (uint32_t w = 0; w < blockDim.x / 32u; w++) S += s_sum[w];
    tcw_result r;
    r.maxF = best;
    r.argmax = bidx;
    r.lnBtSG = t.ln_prior + (double)best + log(S);
    r.t0_mp_idx = -1;
    r.tau_mp_idx = -1;
    r.status = 0;
    results[blockIdx.x] = r;
  }
}

cudaError_t launch_finalize(const TemplateDev *d_T, uint32_t n_templates, const Partial *d_parts,
                            void *d_results, bool chained, cudaStream_t stream) {
  if (n_templates == 0) return cudaSuccess;
  if (n_templates <= 1024)  // (a warp each: 38 us for 3 templates of 2100 x 1581 cells)
    return launch_kernel(finalize_block_kernel, n_templates, 256, stream, chained, d_T, d_parts,
                         reinterpret_cast<tcw_result *>(d_results));
  return launch_kernel(finalize_kernel, (n_templates + 3u) / 4u, 128, stream, chained, d_T,
                       n_templates, d_parts, reinterpret_cast<tcw_result *>(d_results));
}

// Posteriors of written maps (tcw:219-287): the row and column sums of
// exp(F - maxF) in one read of the maps, then their first argmaxes.
//
// post_sums_kernel: a block takes `rows` t0 rows x `cols` columns of one
// template (the whole of it in 1024-column strips); its threads walk four rows
// at a time over four columns each, 256 apart (whole-line loads).  Column sums
// are FP32 with Kahan compensation per thread, row sums double-words added
// over the warp by recursive halving (six steps for four rows) and over the
// block's warps in order: no atomics.  Bound by issue (~16 instructions per
// cell) and the map's read: 137e6 cells of 96 templates 924 -> 225 us (2.4
// TB/s; before, one block per template and 1024 columns walked all rows).
// post_argmax_kernel: per template up to kPostParts blocks each for rows and
// columns add the chunks' sums in FP64 and leave their first maximum; the
// template's last block picks among them in index order (same maps: 68 ->
// 33 us with one warp per template before).  The grid is that of the template
// with most parts, fewer blocks (down to one) where there are thousands of
// templates: with 64 for each a run of 2000 templates of 20 x 20 cells took 255
// us for 113.
constexpr uint32_t kPostThreads = 256;
constexpr uint32_t kPostCols = 1024;
constexpr uint32_t kPostMaxRows = 256;

// kChained (both kernels): launched as a dependent in a single map's chain
// (pdl_begin); a plan's launches take read-only loads.
template <bool kChained, class V>
__device__ __forceinline__ V post_load(const V *p) {
  return kChained ? *p : __ldg(p);
}

template <bool kChained>
__global__ void __launch_bounds__(kPostThreads) post_sums_kernel(
    const TemplateDev *T, const uint2 *__restrict__ chunks, uint32_t rows,
    uint32_t cols, const float *maps, const tcw_result *results,
    double *__restrict__ rowsum, double *__restrict__ colsum, uint32_t *__restrict__ ticket) {
  __shared__ float2 srow[kPostThreads / 32][kPostMaxRows];
  pdl_begin();
  uint2 ch;  // template, chunk within it (column chunk fastest)
  if (chunks)
    ch = chunks[blockIdx.x];
  else
    ch = make_uint2(0u, blockIdx.x);
  const TemplateDev t = T[ch.x];
  const uint32_t n_cc = (t.N_tau + cols - 1u) / cols;
  const uint32_t cc = ch.y % n_cc, rc = ch.y / n_cc;
  const uint32_t m0 = rc * rows, m1 = min(t.N_t0, m0 + rows);
  const uint32_t nb = cc * cols, ne = min(t.N_tau, nb + cols);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  if (ch.y == 0u && tid == 0u) ticket[ch.x] = 0u;
  const float maxF = results[ch.x].maxF;
  const float *F = maps + t.map_off;
  for (uint32_t k = lane; k < m1 - m0; k += 32u) srow[wid][k] = make_float2(0.0f, 0.0f);
  __syncwarp();
  // (warps behind a narrow map's last column leave their zeros; tested once, not
  // per strip: that made 1024 x 1024 exponential calls 127 -> 137 us)
  for (uint32_t n0 = nb + wid * 32u < ne ? nb + tid : ne + tid; n0 - tid < ne; n0 += kPostCols) {
    float cs[4] = {0, 0, 0, 0}, cc4[4] = {0, 0, 0, 0};
    for (uint32_t m = m0; m < m1; m += 4u) {
      FF w[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float *row = F + (size_t)(m + q) * t.N_tau;
        float e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t n = n0 + 256u * j;
          e[j] = (m + q < m1 && n < ne) ? ex2_approx((post_load<kChained>(row + n) - maxF) * kLog2e) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float y = fsub(e[j], cc4[j]);
          const float u = fadd(cs[j], y);
          cc4[j] = fsub(fsub(u, cs[j]), y);
          cs[j] = u;
        }
        w[q] = ff_add1(ff_add1(ff_add1(FF{e[0], 0.0f}, e[1]), e[2]), e[3]);
      }
      // four rows over 32 lanes: a lane keeps half of its rows per step
      auto xch = [&](FF v, int d) {
        return FF{__shfl_xor_sync(0xffffffffu, v.h, d), __shfl_xor_sync(0xffffffffu, v.l, d)};
      };
      const bool u16 = (lane & 16u) != 0u, u8 = (lane & 8u) != 0u;
      const FF a0 = ff_add(u16 ? w[2] : w[0], xch(u16 ? w[0] : w[2], 16));
      const FF a1 = ff_add(u16 ? w[3] : w[1], xch(u16 ? w[1] : w[3], 16));
      FF v = ff_add(u8 ? a1 : a0, xch(u8 ? a0 : a1, 8));
      v = ff_add(v, xch(v, 4));
      v = ff_add(v, xch(v, 2));
      v = ff_add(v, xch(v, 1));
      const uint32_t r = m - m0 + (u16 ? 2u : 0u) + (u8 ? 1u : 0u);
      if ((lane & 7u) == 0u && r < m1 - m0) {
        const float2 o = srow[wid][r];
        const FF s = ff_add(FF{o.x, o.y}, v);
        srow[wid][r] = make_float2(s.h, s.l);
      }
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (n0 + 256u * j < ne)
        colsum[t.col_off + (size_t)rc * t.N_tau + n0 + 256u * j] =
            (double)cs[j] - (double)cc4[j];
  }
  __syncthreads();
  for (uint32_t k = tid; k < m1 - m0; k += kPostThreads) {
    double s = 0.0;
#pragma unroll
    for (uint32_t w = 0; w < kPostThreads / 32u; w++)
      s += (double)srow[w][k].x + (double)srow[w][k].y;
    rowsum[t.row_off + (size_t)cc * t.N_t0 + m0 + k] = s;
  }
}

// A sum as an integer of the same order (sums are >= 0; a NaN is below all),
// so that no FP64 comparison stands in the chains.
struct PostBest {
  int64_t v;
  int64_t i;
};
__device__ __forceinline__ int64_t post_key(double x) {
  const int64_t k = __double_as_longlong(x);
  return (uint64_t)k > 0x7FF0000000000000ull ? -1 : k;
}
__device__ __forceinline__ PostBest post_better(PostBest a, PostBest b) {
  return b.v > a.v || (b.v == a.v && b.i < a.i) ? b : a;
}
__device__ __forceinline__ PostBest post_block_best(PostBest best, PostBest *sh) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    PostBest o;
    o.v = __shfl_xor_sync(0xffffffffu, best.v, d);
    o.i = __shfl_xor_sync(0xffffffffu, best.i, d);
    best = post_better(best, o);
  }
  if ((threadIdx.x & 31u) == 0) sh[threadIdx.x >> 5] = best;
  __syncthreads();
  best = sh[0];
  for (uint32_t w = 1; w < kPostThreads / 32u; w++) best = post_better(best, sh[w]);
  return best;
}

template <bool kChained>
__global__ void __launch_bounds__(kPostThreads) post_argmax_kernel(
    const TemplateDev *T, uint32_t rows, uint32_t cols, const double *rowsum,
    const double *colsum,
    PostPart *__restrict__ parts, uint32_t *__restrict__ ticket,
    tcw_result *__restrict__ results) {
  __shared__ PostBest sh[kPostThreads / 32];
  __shared__ uint32_t s_last;
  pdl_begin();
  const uint32_t k = blockIdx.y;
  const TemplateDev t = T[k];
  const uint32_t e_row = post_part_entries(t.N_t0), e_col = post_part_entries(t.N_tau);
  const uint32_t p_row = (t.N_t0 + e_row - 1u) / e_row, p_col = (t.N_tau + e_col - 1u) / e_col;
  const uint32_t n_parts = p_row + p_col;
  PostPart *mine = parts + (size_t)k * (2u * kPostParts);
  bool last = false;
  for (uint32_t part = blockIdx.x; part < n_parts; part += gridDim.x) {
    const bool is_row = part < p_row;
    const uint32_t N = is_row ? t.N_t0 : t.N_tau, e = is_row ? e_row : e_col;
    const uint32_t i0 = (is_row ? part : part - p_row) * e, i1 = min(N, i0 + e);
    const uint32_t n_sum = is_row ? (t.N_tau + cols - 1u) / cols : (t.N_t0 + rows - 1u) / rows;
    const double *S = is_row ? rowsum + t.row_off : colsum + t.col_off;
    PostBest best{-1, INT64_MAX};
    if (n_sum >= 64u && i1 - i0 <= kPostThreads / 8u) {
      // few entries of many sums (a map of many rows and few columns): eight
      // lanes share an entry (100000 x 3 cells: 3 threads adding 6250 sums each
      // 700 us a call, 180 now)
      const uint32_t i = i0 + threadIdx.x / 8u;
      double s = 0.0;
      if (i < i1) {
        const double *col = S + i;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        uint32_t c = threadIdx.x & 7u;
        for (; c + 24u < n_sum; c += 32u)
#pragma unroll
          for (uint32_t q = 0; q < 4u; q++) v[q] += post_load<kChained>(col + (size_t)(c + 8u * q) * N);
        for (; c < n_sum; c += 8u) v[0] += post_load<kChained>(col + (size_t)c * N);
        s = (v[0] + v[1]) + (v[2] + v[3]);
      }
#pragma unroll
      for (int d = 4; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (i < i1) best = PostBest{post_key(s), (int64_t)i};
    } else {
      for (uint32_t i = i0 + threadIdx.x; i < i1; i += kPostThreads) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};  // four chains: FP64 additions are slow to return
        uint32_t c = 0;
        for (; c + 4u <= n_sum; c += 4u)
#pragma unroll
          for (uint32_t q = 0; q < 4u; q++) v[q] += post_load<kChained>(S + (size_t)(c + q) * N + i);
        for (; c < n_sum; c++) v[0] += post_load<kChained>(S + (size_t)c * N + i);
        const int64_t key = post_key((v[0] + v[1]) + (v[2] + v[3]));
        if (key > best.v) best = PostBest{key, (int64_t)i};  // i increases: keeps the first
      }
    }
    best = post_block_best(best, sh);
    if (threadIdx.x == 0) {
      mine[is_row ? part : kPostParts + part - p_row] = PostPart{best.v, best.i};
      if (gridDim.x > 1u) {
        __threadfence();
        s_last = atomicAdd(ticket + k, 1u) == n_parts - 1u ? 1u : 0u;
      } else {
        s_last = 1u;
      }
    }
    __syncthreads();
    last = s_last != 0u;
  }
  if (!last || threadIdx.x >= 2u) return;
  __threadfence();
  // thread 0 the rows' parts, thread 1 the columns'
  const uint32_t n = threadIdx.x == 0 ? p_row : p_col;
  const volatile PostPart *v = mine + threadIdx.x * kPostParts;
  PostBest b{-1, INT64_MAX};
  for (uint32_t q = 0; q < n; q++) b = post_better(b, PostBest{v[q].v, v[q].i});
  const int64_t idx = b.i == INT64_MAX ? -1 : b.i;
  if (threadIdx.x == 0)
    results[k].t0_mp_idx = idx;
  else
    results[k].tau_mp_idx = idx;
}

cudaError_t launch_posteriors(const TemplateDev *d_T, uint32_t n_templates, const PostLayout &L,
                              const float *d_maps, tcw_result *d_results, bool chained,
                              cudaStream_t stream) {
  if (L.n_chunks == 0 || n_templates == 0) return cudaSuccess;
  cudaError_t e = launch_kernel(chained ? post_sums_kernel<true> : post_sums_kernel<false>,
                                L.n_chunks, kPostThreads, stream, chained, d_T, L.chunks, L.rows,
                                L.cols, d_maps, (const tcw_result *)d_results, L.rowsum, L.colsum,
                                L.ticket);
  if (e != cudaSuccess) return e;
  for (uint32_t y0 = 0; y0 < n_templates; y0 += 65535u) {
    const uint32_t ny = n_templates - y0 < 65535u ? n_templates - y0 : 65535u;
    e = launch_kernel(chained ? post_argmax_kernel<true> : post_argmax_kernel<false>,
                      dim3(L.argmax_blocks, ny), kPostThreads, stream, chained && y0 == 0,
                      d_T + y0, L.rows, L.cols, (const double *)L.rowsum, (const double *)L.colsum,
                      L.parts + (size_t)y0 * 2u * kPostParts, L.ticket + y0, d_results + y0);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace tcw

namespace tcw {
// Failed debug checks of this file's kernels (0 unless built with TCW_DEBUG_CHECKS).
unsigned int dcheck_failures_kernels() {
#if defined(TCW_DEBUG_CHECKS)
  return tcw_dcheck_read();
#else
  return 0;
#endif
}
}  // namespace tcw
