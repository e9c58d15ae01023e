// Differentiable transient maps (exponential and rectangular windows):
// forward values and the adjoint.
//
// Per template the tau grid is continuous, tau_n = tau_min + n (tau_max -
// tau_min) / (N_tau - 1), and the outputs are
//   lnBtSG    = ln(70 / (N_t0 N_tau)) + logsumexp_mn F_mn            (tcw:196-217)
//   softmax2F = T logsumexp_mn (2 F_mn / T)        (a smooth max of 2F, T > 0)
// with gradients with respect to the atoms (a2, b2, ab, Fa, Fb) and to
// tau_min / tau_max.  Window boundaries move in steps with tau; only the
// weights are differentiated (the boundaries are piecewise constant).
//
// At T = 0.1 the soft-max weights are exp(20 F), so a gradient good to 1e-4
// needs F to ~1e-9 of its value.  The exponential windows' sums slide down
// each tau column in double-word FP32 (ExpColumn, the map kernels'
// arithmetic, ~1e-14 of the sums' magnitude) rather than in FP64, whose rate
// on GB300 is 1/70 of FP32; for the cells that carry weight (an FP32 tier-1
// F far enough below the maximum or the normaliser skips a cell, whose
// weight is then below e^-40) the forward forms F and the log-sum-exps in
// FP64, the backward F, dF/dW and the sources in double-word FP32:
//
// Exponential templates are tiled by 32 tau columns x a chunk of t0 rows, one
// warp per tile; a chunk's first window is joined from segment sums
// (ExpColumn::warm_start), so that a single template fills the GPU.  Batches of
// templates of few rows keep whole columns (DiffTemplate::whole).
//
//   diff_est_kernel  FP32 only: the tile's largest tier-1 F (`need`, infinite
//            where a cell has none) and a lower bound of the template's
//            maximum.  With a signal almost no tile holds a cell that carries
//            weight, and the FP64 and adjoint work below skips whole tiles.
//   diff_hot_kernel  the tiles whose cells matter by themselves, their columns
//            walked whole (many of them: by the kHot forms of the next two);
//   diff_fwd_kernel  the tiles that may carry weight: double-word window
//            sums, FP64 log-sum-exps of F and 2F/T -> partials -> finalize
//            per template.
//   diff_src_kernel  backward, the tiles that may carry weight: the same walk
//            plus the tau-derivative sums V = sum (i - lo) x r^(i - lo)
//            (ExpColumnV); per cell the adjoint sources G_c = g dF/dW_c
//            (g = dL/dF) go to scratch (no map is kept) and g dF/dtau
//            accumulates per column;
//   diff_atoms_kernel  per column, atoms ascending, the transposed recurrence
//            H(i) = r H(i-1) + sum_{lo(m)=i} G(m) - sum_{hi(m)+1=i} G(m)
//            r^(L(m)) in double-word FP32 gives dL/dx(i) = H(i).  It is linear
//            in H, so it runs in segments of 64 atoms and more side by side: a
//            first pass leaves each segment's end from H = 0, a second one joins
//            the ends below its segment, walks it again and adds each warp's 32
//            columns per atom (recursive halving over the 7 channels) to the
//            FP64 atom gradient.
// Measured (forward + backward, 2000 atoms, 1024 x 1024 cells, signal): one
// template 7.7-9.6 -> 1.6 ms (one block per 128 columns and all rows before),
// 24 templates 16.5 -> 3.0 ms, 256 templates 53 -> 22 ms; noise alone: 6.9 -> 0.9,
// 17.6 -> 7.9, 101 -> 85 ms.
// The window-sum factor e^(-k (t_lo - t0)/tau) is left out everywhere: F does
// not depend on it, so neither do g, dF/dW (in this frame) or dF/dtau.
//
// Rectangular windows: tiles of 32 t0 rows x a chunk of tau columns, one warp
// per tile, one row per lane, the columns in ascending order (the window end
// only grows with tau, as in the reference's running sums, Rect.cu:75-91).
// rect_est_kernel bounds F per tile in FP32 from the map path's prefix rows;
// rect_diff_kernel takes the tiles that may carry weight, with FP64 sums
// (32-atom block sums, then single atoms) brought up to date only at cells
// that do.  The sums of a window do not depend on tau between boundaries, so
// dL/dtau = 0; the atom gradient is scattered as a difference array:
// +sum_n G(m, n) at the row's start index lo(m), -G(m, n) at end(m, n) + 1
// (consecutive cells with the same end merged), then one prefix scan per
// template (rect_diff_scan_kernel) gives dL/dx(i) = sum_{j <= i} D(j).
// Measured (7 templates of 1499 atoms, 777 x 611 cells, signal): forward and
// backward 6.47 -> 0.64 ms (before, one thread per row over all columns and
// FP64 F in every cell).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/tcw_b200.h"
#include "tcw_exp_walk.cuh"
#include "tcw_internal.h"

namespace tcw {

namespace {

constexpr float kLog2eF = 1.4426950408889634f;

__device__ __forceinline__ double tau_of(const DiffTemplate &t, uint32_t n) {
  if (t.N_tau <= 1) return t.tau_min;
  return t.tau_min + (double)n * ((t.tau_max - t.tau_min) / (double)(t.N_tau - 1u));
}

// Upper window end for a real tau (the reference's formula with t1 real).
__device__ __forceinline__ bool exp_hi_real(uint32_t t0, double tau, const Geom &g, uint32_t &hi) {
  const double t1 = (double)t0 + 3.0 * tau;
  if (t1 < (double)g.t0_data) return false;
  const double d = t1 - (double)g.t0_data;
  const double q = floor((d + (double)g.half) / (double)g.TAtom) - 1.0;
  const uint32_t b = q < 0.0 ? 0u
                             : (q >= (double)(g.numAtoms - 1u) ? g.numAtoms - 1u : (uint32_t)q);
  const double l = floor(d / (double)g.TAtom);
  const uint32_t last = l >= 4294967295.0 ? 0xFFFFFFFFu : (uint32_t)l;
  hi = b < last ? b : last;
  return true;
}

// F in FP64 with the reference's conditioning test (Rect.cu:93-118).
struct F64Cell {
  double F, iD;  // F and 1/D
  bool ok;
};

// The conditioning test (sumAB + disc) / (sumAB - disc) < 1e4 is taken as
// sumAB + disc < 1e4 (sumAB - disc) with sumAB - disc > 0 (no division), and
// F = N (1/D) with the one reciprocal the derivatives reuse: FP64 divisions
// are long sequences at GB300's FP64 rate.
// `passes`: the caller knows that the test holds (a tier-1 cell, cond < 32).
__device__ __forceinline__ F64Cell fstat64(const double W[7], bool passes = false) {
  const double A = W[0], B = W[1], C = W[2];
  F64Cell r{2.0, 0.0, false};
  if (!passes) {
    const double sumAB = A + B, diffAB = A - B;
    const double disc = sqrt(diffAB * diffAB + 4.0 * C * C);
    const double denom = sumAB - disc;
    passes = denom > 0.0 && sumAB + disc < 1e4 * denom;
  }
  if (passes) {
    // (explicit roundings: every kernel forms the same bits)
    const double D = fma(A, B, -(C * C));
    if (D > 0.0) {
      const double Fa2 = fma(W[3], W[3], W[4] * W[4]), Fb2 = fma(W[5], W[5], W[6] * W[6]);
      const double re = fma(W[3], W[5], W[4] * W[6]);
      const double N = fma(B, Fa2, fma(A, Fb2, -2.0 * C * re));
      r.iD = 1.0 / D;
      r.F = N * r.iD;
      r.ok = true;
    }
  }
  return r;
}

// Online log-sum-exp in FP64 (exp in FP64 too: the forward values feed
// finite-difference checks, where FP32 rounding of the terms would show).
// Terms below e^-60 of the running maximum are skipped: the sum is >= 1, so
// even 1e9 of them change it by < 1e-17.
// `k`: so many terms v.
__device__ __forceinline__ void lse_add(double &m, double &s, double v, double k = 1.0) {
  if (v > m) {
    s = s * exp(m - v) + k;
    m = v;
  } else if (v - m > -60.0) {
    s += k * exp(v - m);
  }
}

constexpr int kDiffBlock = 128;  // four warps, one tile each

// Order-preserving key of a float for atomicMax; 0 is below every key.
__device__ __forceinline__ uint32_t float_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// ------------------------------------------------------------ exponential backward (double-word)

// Packed double-word helpers of the backward pass.
__device__ __forceinline__ FF2 ff2_add_dw(FF2 a, FF2 b) {  // a + b, low words summed
  const F2 s = add2(a.h, b.h);
  const F2 bb = sub2(s, a.h);
  const F2 e = add2(sub2(a.h, sub2(s, bb)), sub2(b.h, bb));
  return FF2{s, add2(e, add2(a.l, b.l))};
}
__device__ __forceinline__ FF2 ff2_scale_dw(F2 rh, F2 nrh, F2 rl, FF2 S) {  // r S (r = rh + rl)
  const F2 q = mul2(nrh, S.h);  // -p
  F2 pe = fma2(rh, S.h, q);
  pe = fma2(rh, S.l, pe);
  pe = fma2(rl, S.h, pe);
  return FF2{sub2(F2{0.0f, 0.0f}, q), pe};
}
__device__ __forceinline__ FF ff_add_dw(FF a, FF b) {
  float s, e;
  two_sum(a.h, b.h, s, e);
  return FF{s, fadd(e, fadd(a.l, b.l))};
}
__device__ __forceinline__ FF ff_scale_dw(FF r, FF S) {
  const float p = fmul(r.h, S.h);
  float pe = ffma(r.h, S.h, -p);
  pe = ffma(r.h, S.l, pe);
  pe = ffma(r.l, S.h, pe);
  return FF{p, pe};
}
// Double-word arithmetic on FF (hi + lo FP32 pairs, ~2^-44 relative per
// operation) for the adjoint's per-cell values.
__device__ __forceinline__ FF dw_norm(float s, float e) {
  const float h = fadd(s, e);
  return FF{h, fsub(e, fsub(h, s))};
}
__device__ __forceinline__ FF dw_add(FF a, FF b) {
  float s, e;
  two_sum(a.h, b.h, s, e);
  return dw_norm(s, fadd(e, fadd(a.l, b.l)));
}
__device__ __forceinline__ FF dw_sub(FF a, FF b) { return dw_add(a, FF{-b.h, -b.l}); }
__device__ __forceinline__ FF dw_mulf(FF a, float b) {
  const float p = fmul(a.h, b);
  float e = ffma(a.h, b, -p);
  e = ffma(a.l, b, e);
  return dw_norm(p, e);
}
__device__ __forceinline__ FF dw_twice(FF a) { return FF{2.0f * a.h, 2.0f * a.l}; }
__device__ __forceinline__ FF dw_from(double x) {
  const float h = (float)x;
  return FF{h, (float)(x - (double)h)};
}

// F of a cell from its double-word window sums, in double-word arithmetic:
// D = AB - C^2 from exact products of the high words, the conditioning test
// cond < 1e4 as 1e4 S^2 < (1 + 1e4)^2 D (S = A + B), G = B Fa - C Fb and
// F = (|G|^2 + D |Fb|^2) / (B D).
struct DwCell {
  FF F, iD, Gre, Gim, Fb2;
  bool ok;
};
__device__ __forceinline__ DwCell dw_fstat(FF A, FF B, FF C, FF Far, FF Fai, FF Fbr, FF Fbi) {
  DwCell r;
  const float p = fmul(A.h, B.h), pe = ffma(A.h, B.h, -p);
  const float q = fmul(C.h, C.h), qe = ffma(C.h, C.h, -q);
  float s, se;
  two_sum(p, -q, s, se);
  float corr = fadd(se, fsub(pe, qe));
  corr = ffma(A.h, B.l, corr);
  corr = ffma(A.l, B.h, corr);
  corr = ffma(-2.0f * C.h, C.l, corr);
  corr = ffma(A.l, B.l, corr);
  corr = ffma(-C.l, C.l, corr);
  const FF D = dw_norm(s, corr);
  const FF S = dw_add(A, B);
  const FF lhs = dw_mulf(ff_mul(S, S), 1.0e4f);
  const FF rhs = ff_mul(D, FF{100020000.0f, 1.0f});  // (1 + 1e4)^2
  const FF dd = dw_sub(rhs, lhs);
  r.ok = D.h > 0.0f && S.h > 0.0f && dd.h > 0.0f;
  r.Gre = dw_sub(ff_mul(B, Far), ff_mul(C, Fbr));
  r.Gim = dw_sub(ff_mul(B, Fai), ff_mul(C, Fbi));
  r.Fb2 = dw_add(ff_mul(Fbr, Fbr), ff_mul(Fbi, Fbi));
  const FF G2 = dw_add(ff_mul(r.Gre, r.Gre), ff_mul(r.Gim, r.Gim));
  const FF num = dw_add(G2, ff_mul(D, r.Fb2));
  r.iD = r.ok ? ff_recip(D) : FF{0.0f, 0.0f};
  const FF iB = r.ok ? ff_recip(B) : FF{0.0f, 0.0f};
  r.F = ff_mul(ff_mul(num, r.iD), iB);
  return r;
}

// E + x per lane (TwoSum of the high words, x's rounding into the low word).
__device__ __forceinline__ FF2 ff2_add_x(FF2 E, F2 x) {
  const F2 s = add2(E.h, x);
  const F2 bb = sub2(s, E.h);
  const F2 e = add2(sub2(E.h, sub2(s, bb)), sub2(x, bb));
  return FF2{s, add2(E.l, e)};
}


// The backward pass's column: the window sums W of ExpColumn and their
// tau-derivative sums V_c = sum_i (i - lo) x_c(i) r_c^(i - lo) (r_c = r^2
// for A, B, C, r for Fa, Fb), both in double-word FP32 and moved together:
// an atom entering at the bottom gives V' = r_c (V + W) (the old W), one
// leaving at the top with weight exponent e gives V' = V - e x r_c^e.
// dW_c / dtau = k_c (TAtom / tau^2) V_c (k_c = 2 for A, B, C; 1 otherwise).
struct ExpColumnV {
  ExpColumn<false> C;
  __device__ __forceinline__ const ExpColumn<false> &sums() const { return C; }
  FF2 V0, V2, V3;
  FF Vc;

  __device__ __forceinline__ void reset_v() {
    const F2 z{0.0f, 0.0f};
    V0 = V2 = V3 = FF2{z, z};
    Vc = FF{0.0f, 0.0f};
  }

  __device__ __forceinline__ bool slide(const float *__restrict__ atoms8, const Geom &g,
                                        uint32_t lo, uint32_t top, uint32_t nz) {
    if (top > C.wtop || lo > C.wlo || top <= C.wlo) {
      C.reset_window(top);
      reset_v();
    }
    while (C.wtop > top) {
      C.wtop--;
      const uint32_t ex = C.wtop - C.wlo;
      C.power(ex);
      F2 x[4];
      TCW_DCHECK(C.wtop < g.numAtoms);
      load_row8<true>(atoms8 + (size_t)C.wtop * 8u, x);
      const F2 ph0{C.p2.h, C.p2.h}, pl0{C.p2.l, C.p2.l}, nph0{-C.p2.h, -C.p2.h};
      const F2 ph1{C.pw.h, C.pw.h}, pl1{C.pw.l, C.pw.l}, nph1{-C.pw.h, -C.pw.h};
      C.W0 = ff2_sub_scaled_x(C.W0, ph0, nph0, pl0, x[0]);
      C.Wc = ff_sub_scaled_x1(C.Wc, C.p2, x[1].x);
      C.W2 = ff2_sub_scaled_x(C.W2, ph1, nph1, pl1, x[2]);
      C.W3 = ff2_sub_scaled_x(C.W3, ph1, nph1, pl1, x[3]);
      // V: the leaving atom's weight times its exponent
      const FF e2 = ff_mul(C.p2, FF{(float)ex, 0.0f}), e1 = ff_mul(C.pw, FF{(float)ex, 0.0f});
      const F2 eh0{e2.h, e2.h}, el0{e2.l, e2.l}, neh0{-e2.h, -e2.h};
      const F2 eh1{e1.h, e1.h}, el1{e1.l, e1.l}, neh1{-e1.h, -e1.h};
      V0 = ff2_sub_scaled_x(V0, eh0, neh0, el0, x[0]);
      Vc = ff_sub_scaled_x1(Vc, e2, x[1].x);
      V2 = ff2_sub_scaled_x(V2, eh1, neh1, el1, x[2]);
      V3 = ff2_sub_scaled_x(V3, eh1, neh1, el1, x[3]);
    }
    while (C.wlo > lo) {
      C.wlo--;
      F2 x[4];
      TCW_DCHECK(C.wlo < g.numAtoms);
      load_row8<true>(atoms8 + (size_t)C.wlo * 8u, x);
      V0 = ff2_scale_dw(C.k2.rh[0], C.k2.nrh[0], C.k2.rl[0], ff2_add_dw(V0, C.W0));
      Vc = ff_scale_dw(C.k.r2, ff_add_dw(Vc, C.Wc));
      V2 = ff2_scale_dw(C.k2.rh[1], C.k2.nrh[1], C.k2.rl[1], ff2_add_dw(V2, C.W2));
      V3 = ff2_scale_dw(C.k2.rh[1], C.k2.nrh[1], C.k2.rl[1], ff2_add_dw(V3, C.W3));
      C.W0 = ff2_axpy(x[0], C.k2.rh[0], C.k2.nrh[0], C.k2.rl[0], C.W0);
      C.Wc = ff_axpy(x[1].x, C.k.r2, C.Wc);
      C.W2 = ff2_axpy(x[2], C.k2.rh[1], C.k2.nrh[1], C.k2.rl[1], C.W2);
      C.W3 = ff2_axpy(x[3], C.k2.rh[1], C.k2.nrh[1], C.k2.rl[1], C.W3);
    }
    return nz < top;
  }

  // One lane's W and V sums of a segment (stride 32).
  __device__ __forceinline__ void store_sums(float *__restrict__ o) const {
    C.store_sums(o);
    const float v[14] = {V0.h.x, V0.h.y, V0.l.x, V0.l.y, Vc.h,   Vc.l,   V2.h.x,
                         V2.h.y, V2.l.x, V2.l.y, V3.h.x, V3.h.y, V3.l.x, V3.l.y};
#pragma unroll
    for (int f = 0; f < 14; f++) o[32 * (14 + f)] = v[f];
  }

  // ExpColumn::warm_start with the derivative sums: below a segment of
  // S = 2^shift atoms, V = GV_j + r^S (V + S W) with the old W.
  __device__ __forceinline__ void warm_start(const float *__restrict__ atoms8, const Geom &g,
                                             const float *__restrict__ seg, uint32_t shift,
                                             uint32_t nseg, uint32_t lo, uint32_t top,
                                             uint32_t stride) {
    const uint32_t j1 = (lo + (1u << shift) - 1u) >> shift;
    const uint32_t j2 = top == g.numAtoms ? nseg : top >> shift;
    C.reset_window(top);
    reset_v();
    if (top != g.numAtoms) slide(atoms8, g, j2 << shift, top, 0u);
    FF R = C.k.r1;
    for (uint32_t b = 0; b < shift; b++) R = ff_mul(R, R);
    const FF R2 = ff_mul(R, R);
    const F2 rh0{R2.h, R2.h}, nrh0{-R2.h, -R2.h}, rl0{R2.l, R2.l};
    const F2 rh1{R.h, R.h}, nrh1{-R.h, -R.h}, rl1{R.l, R.l};
    const float S = (float)(1u << shift);
    const F2 S2{S, S};
    for (uint32_t j = j2; j > j1;) {
      j--;
      TCW_DCHECK(j < nseg);
      const float *s = seg + (size_t)j * stride;
      const float *v = s + 14 * 32;
      V0 = ff2_axpy_dw(FF2{F2{v[0], v[32]}, F2{v[64], v[96]}}, rh0, nrh0, rl0,
                       ff2_add_dw(V0, FF2{mul2(S2, C.W0.h), mul2(S2, C.W0.l)}));
      Vc = ff_axpy_dw(FF{v[128], v[160]}, R2, ff_add_dw(Vc, FF{S * C.Wc.h, S * C.Wc.l}));
      V2 = ff2_axpy_dw(FF2{F2{v[192], v[224]}, F2{v[256], v[288]}}, rh1, nrh1, rl1,
                       ff2_add_dw(V2, FF2{mul2(S2, C.W2.h), mul2(S2, C.W2.l)}));
      V3 = ff2_axpy_dw(FF2{F2{v[320], v[352]}, F2{v[384], v[416]}}, rh1, nrh1, rl1,
                       ff2_add_dw(V3, FF2{mul2(S2, C.W3.h), mul2(S2, C.W3.l)}));
      C.W0 = ff2_axpy_dw(FF2{F2{s[0], s[32]}, F2{s[64], s[96]}}, rh0, nrh0, rl0, C.W0);
      C.Wc = ff_axpy_dw(FF{s[128], s[160]}, R2, C.Wc);
      C.W2 = ff2_axpy_dw(FF2{F2{s[192], s[224]}, F2{s[256], s[288]}}, rh1, nrh1, rl1, C.W2);
      C.W3 = ff2_axpy_dw(FF2{F2{s[320], s[352]}, F2{s[384], s[416]}}, rh1, nrh1, rl1, C.W3);
    }
    C.wlo = j1 << shift;
  }
};

// ------------------------------------------------------------ exponential tiles

constexpr uint32_t kDiffRowTab = 128;

// Grid y: the template; the first `n_atom_blocks` blocks of x repack its atoms
// (256 each), the others form its column constants (256 each).
__global__ void __launch_bounds__(256) diff_prep_kernel(const DiffTemplate *__restrict__ T,
                                                        const uint32_t *__restrict__ list,
                                                        uint32_t n_atom_blocks,
                                                        const float *__restrict__ atoms,
                                                        float *__restrict__ atoms8,
                                                        ColConsts *__restrict__ cols) {
  const DiffTemplate t = T[list[blockIdx.y]];
  if (blockIdx.x < n_atom_blocks) {
    repack_rows(atoms + t.atom_off * 7u, reinterpret_cast<float4 *>(atoms8 + t.atom_off * 8u),
                t.g.numAtoms, blockIdx.x * 256u);
    return;
  }
  const uint32_t n = (blockIdx.x - n_atom_blocks) * 256u + threadIdx.x;
  if (n >= t.N_tau) return;
  ExpColumn<false> C;
  C.init_real(t.g, tau_of(t, n));
  cols[t.col_off + n] = C.consts();
}

// One warp's share of a template: its column group, this lane's column and
// the warp's largest tau (rounded up, for the regularity test).
struct DiffLane {
  DiffTemplate t;
  uint32_t n, taumax;
  bool active;
  double tau;
  const float *a8;
  const uint32_t *t0s;

  __device__ __forceinline__ void columns(const float *atoms8, const uint32_t *t0s_all,
                                          uint32_t cg) {
    n = cg * 32u + (threadIdx.x & 31u);
    active = n < t.N_tau;
    tau = tau_of(t, active ? n : cg * 32u);
    const uint32_t up = !active ? 0u
                        : (tau >= 4294967295.0 ? 0xFFFFFFFFu : (uint32_t)ceil(tau));
    taumax = __reduce_max_sync(0xffffffffu, up);
    a8 = atoms8 + t.atom_off * 8u;
    t0s = t0s_all + t.t0_off;
  }
  // this lane's constants (a lane without a column takes the group's first)
  __device__ __forceinline__ ColConsts consts(const ColConsts *__restrict__ cols) const {
    return cols[t.col_off + (active ? n : n & ~31u)];
  }
};

template <bool kFast, bool kWide>
__device__ __forceinline__ const ExpColumn<false, kFast, kWide> &sums_of(
    const ExpColumn<false, kFast, kWide> &C) {
  return C;
}
__device__ __forceinline__ const ExpColumn<false> &sums_of(const ExpColumnV &C) { return C.C; }

// Walks rows [mb, me) of one tile from the last one down and calls
// cell(m, lo, top, data) for each: data says that the window [lo, top) holds
// data and that the column holds its sums.  Rows that are not regular for
// the group's taus (t0 + 3 tau + TAtom/2 beyond u32, or TAtom < 2) take the
// window end from exp_hi_real.  `seg`: this lane's segment sums of the group,
// `stride` floats apart (NULL: the first window is entered atom by atom).
template <class Col, class Cell>
__device__ __forceinline__ void diff_rows(const DiffLane &L, uint32_t mb, uint32_t me, Col &C,
                                          const float *__restrict__ seg, uint32_t stride,
                                          ExpRow *tab, Cell &&cell) {
  const DiffTemplate &t = L.t;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t *a8u = reinterpret_cast<const uint32_t *>(L.a8);
  if (seg && L.active) {
    const uint32_t t0 = __ldg(L.t0s + me - 1u);
    if (exp_row_regular(t0, L.taumax, t.g)) {
      const uint32_t lo = exp_lo(t0, t.g), d = t0 - t.g.t0_data;
      ExpRow e;
      e.a = fdiv(d, t.g.div);
      e.b = d - e.a * t.g.TAtom;
      const uint32_t top = sums_of(C).top_of(t.g, e);
      if (lo < top && top - lo >= (2u << t.g_shift))
        C.warm_start(L.a8, t.g, seg, t.g_shift, t.g_nseg, lo, top, stride);
    }
  }
  for (uint32_t ce = me; ce > mb;) {
    const uint32_t cb = ce - mb > kDiffRowTab ? ce - kDiffRowTab : mb;
    bool reg = true;
    for (uint32_t r = lane; r < ce - cb; r += 32u)
      reg = reg && exp_row_regular(__ldg(L.t0s + cb + r), L.taumax, t.g);
    reg = __all_sync(0xffffffffu, reg);
    __syncwarp();
    for (uint32_t r = lane; r < ce - cb; r += 32u) {
      const uint32_t t0 = __ldg(L.t0s + cb + r);
      ExpRow e;
      e.lo = exp_lo(t0, t.g);
      e.nz = e.lo < t.g.numAtoms ? __ldg(a8u + (size_t)e.lo * 8u + 3u) : 0xFFFFFFFFu;
      const uint32_t d = t0 - t.g.t0_data;
      e.a = reg ? fdiv(d, t.g.div) : t0;  // irregular chunks: the generic branch reads t0
      e.b = reg ? d - e.a * t.g.TAtom : 0u;
      tab[r] = e;
    }
    __syncwarp();
    if (L.active) {
      for (uint32_t m = ce; m > cb;) {
        m--;
        const ExpRow e = tab[m - cb];
        uint32_t top = 0;
        bool data = false;
        if (reg) {
          top = sums_of(C).top_of(t.g, e);
          data = e.lo < top && C.slide(L.a8, t.g, e.lo, top, e.nz);
        } else {
          uint32_t hi;
          if (exp_hi_real(e.a, L.tau, t.g, hi) && e.lo <= hi) {
            top = hi + 1u;
            data = C.slide(L.a8, t.g, e.lo, top, e.nz);
          }
        }
        cell(m, e.lo, top, data);
      }
    }
    ce = cb;
  }
}

// Tier-1 F of a column's current sums; false where it needs the test.
__device__ __forceinline__ bool diff_tier1(const ExpColumn<false> &C, float &F32) {
  const F2 s0 = add2(C.W0.h, C.W0.l), s2 = add2(C.W2.h, C.W2.l), s3 = add2(C.W3.h, C.W3.l);
  const float sc = fadd(C.Wc.h, C.Wc.l);
  return fstat_fast_sums(s0.x, s0.y, sc, s2.x, s2.y, s3.x, s3.y, F32);
}

// The largest F of every tile in FP32 (`need`, good to ~1.5e-6 relative: tier
// 1, else tier 2 with the conditioning cut widened by 1e-3, so that no cell
// that FP64 lets pass is missed; infinite for a NaN; at least 2 where a cell
// has no data) and the largest F of the template's cells that surely pass
// (`est`, a lower bound of its maximum to within 1.5e-6).  One W-only walk
// with the map kernels' steps: on the benchmark's differentiation data
// (maximum F 400, F within 62 of it in 4e-6 of the cells) it replaces the
// FP64 work of 99.6 % of the tiles.
struct EstSink {
  float top, most;
  __device__ __forceinline__ void operator()(uint32_t, float F, bool ok) {
    if (!(F == F)) F = INFINITY;
    else if (ok) top = fmaxf(top, F);
    most = fmaxf(most, F);
  }
};

__global__ void __launch_bounds__(kDiffBlock, 8)
    diff_est_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                    const float *__restrict__ atoms8, const uint32_t *__restrict__ t0s_all,
                    const ColConsts *__restrict__ cols, const float *__restrict__ seg,
                    float *__restrict__ need, uint32_t *__restrict__ est) {
  __shared__ __align__(16) ExpRow s_tab[kDiffBlock / 32][kExpRowTab];
  DiffLane L;
  const uint32_t k = list[blockIdx.y];
  L.t = T[k];
  const uint32_t tile = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  const uint32_t cg = tile / L.t.n_chunk, mb = tile % L.t.n_chunk * L.t.chunk_rows;
  if (cg >= L.t.n_cg || L.t.whole == kDiffWholeBlind) return;
  const uint32_t me = min(L.t.N_t0, mb + L.t.chunk_rows);
  L.columns(atoms8, t0s_all, cg);
  ExpColumn<false, true, true> C;
  C.init_consts(L.consts(cols));
  const float *sg =
      L.t.g_nseg ? seg + (L.t.seg_off + (size_t)cg * L.t.g_nseg) * kDiffSegFloats + lane : nullptr;
  EstSink sink{-INFINITY, -INFINITY};
  bool reg = true;
  for (uint32_t m = mb + lane; m < me; m += 32u)
    reg = reg && exp_row_regular(__ldg(L.t0s + m), L.taumax, L.t.g);
  ExpRow *tab = s_tab[threadIdx.x >> 5];
  if (__all_sync(0xffffffffu, reg)) {
    exp_rows<true, false>(C, L.t.g, L.t.g_shift, L.t.g_nseg, L.a8, L.t0s, mb, me, me, L.active, sink, tab, sg);
  } else {
    diff_rows(L, mb, me, C, sg, kDiffSegFloats, tab,
              [&](uint32_t m, uint32_t, uint32_t, bool data) {
                if (data)
                  C.emit(m, sink);
                else
                  sink(m, 2.0f, false);
              });
  }
  float top1 = sink.top, most = sink.most;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    top1 = fmaxf(top1, __shfl_xor_sync(0xffffffffu, top1, d));
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
  }
  if (lane == 0) {
    need[L.t.part_off + tile] = most;
    if (top1 > -INFINITY) atomicMax(est + k, float_key(top1));
  }
}

// ------------------------------------------------------------ exponential forward

// A cell so far below the largest F weighs less than e^-62 in both sums:
// e^(F - max) in lnBtSG, e^(2 (F - max) / T) in the soft-max, whose weights
// fall slower than lnBtSG's above T = 2.
__device__ __forceinline__ double no_weight_below(double temp) {
  return 62.0 * fmax(1.0, 0.5 * temp);
}

// From the key of a template's estimated maximum: cells below `skip` carry no
// weight in either sum, tiles that reach `hot` may hold a cell whose last bits
// show (lnBtSG: e^-8 of the largest; the soft-max multiplies them by 2/T,
// where this is large its weights fall as much faster).  Without an estimate
// (key 0: no cell surely passes the conditioning test, F is 2 almost
// everywhere) nothing is skipped and only NaN tiles are hot.
struct FwdBounds {
  float skip, hot;
  __device__ __forceinline__ FwdBounds(uint32_t key, double temp) {
    skip = -INFINITY;
    hot = INFINITY;
    if (key) {
      const double top = (double)key_float(key);
      skip = (float)(top - 1e-5 * fabs(top) - no_weight_below(temp) - 1.0);
      hot = (float)(top - 1e-5 * fabs(top) - 8.0);
    }
  }
};

// FP64 log-sum-exps of F and 2F/T over the cells of one lane, then over the
// warp; cells below `skip` carry no weight.
struct DiffLse {
  double m1, s1, m2, s2, twoT;
  float skip;
  __device__ __forceinline__ DiffLse(double temp, float bound)
      : m1(-INFINITY), s1(0.0), m2(-INFINITY), s2(0.0), twoT(2.0 / temp), skip(bound) {}
  __device__ __forceinline__ void add(double F, double k = 1.0) {
    lse_add(m1, s1, F, k);
    lse_add(m2, s2, F * twoT, k);
  }
  __device__ __forceinline__ void cell(bool data, const double W[7], bool t1, float F32) {
    if (!data) {
      if (!(2.0f < skip)) add(2.0);
    } else if (!(t1 && F32 < skip)) {
      add(fstat64(W, t1).F);
    }
  }
  // without an estimate: the bound of this lane's own largest F so far
  __device__ __forceinline__ void follow(double below) {
    const float bound = (float)(m1 - 1e-5 * fabs(m1) - below - 1.0);
    if (bound > skip) skip = bound;
  }
  // every lane's sums brought to the warp's maximum (one exp per sum), added
  __device__ __forceinline__ DiffPartial merge() const {
    double M1 = m1, M2 = m2;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      M1 = fmax(M1, __shfl_xor_sync(0xffffffffu, M1, d));
      M2 = fmax(M2, __shfl_xor_sync(0xffffffffu, M2, d));
    }
    double S1 = s1 > 0.0 ? s1 * exp(m1 - M1) : 0.0, S2 = s2 > 0.0 ? s2 * exp(m2 - M2) : 0.0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      S1 += __shfl_xor_sync(0xffffffffu, S1, d);
      S2 += __shfl_xor_sync(0xffffffffu, S2, d);
    }
    return DiffPartial{M1, S1, M2, S2};
  }
};

// Which kernel walks a group's hot tiles: diff_hot_kernel, a block per column
// group, where few column groups have any; else the kHot tile kernels, a warp per
// column group with the same steps -- the block's walk is a third as long, but
// an SM holds one block and four warps of the other on each scheduler.
// `groups` (NULL: blocks) counts the column groups with hot tiles
// (diff_route_kernel), `few` is two blocks per SM.  Forward / backward by blocks
// and by warps, noise: 2000 templates of 1500 atoms, 600 x 4 cells 18.0 / 16.2 ->
// 9.1 / 11.1 ms; of 400 atoms, 32 x 128 cells 5.7 / 7.4 -> 2.6 / 5.2; 256 of 2000
// atoms, 1024 x 1024 cells and a signal 11.8 / 17.2 -> 7.8 / 17.3; 24 of those
// have few hot groups and keep the blocks (1.46 / 1.82 ms).
struct HotRoute {
  const uint32_t *groups;
  uint32_t few;
  __device__ __forceinline__ bool warps() const { return groups && __ldg(groups) > few; }
};

// One column group's hot tiles (at or above `hot` and not below `skip`), for a
// warp that walks its rows from the last one down.
struct HotGroup {
  const float *nd;
  uint32_t n_chunk, chunk_rows, first, row0;
  float skip, hot;
  bool on;
  __device__ __forceinline__ HotGroup(const float *need, const DiffTemplate &t, float skip_,
                                      float hot_)
      : nd(need), n_chunk(t.n_chunk), chunk_rows(t.chunk_rows), first(0xFFFFFFFFu),
        row0(0xFFFFFFFFu), skip(skip_), hot(hot_), on(false) {}
  __device__ __forceinline__ bool is_hot(uint32_t c) const {
    return !(nd[c] < skip) && !(nd[c] < hot);
  }
  // all lanes: finds the first hot tile
  __device__ __forceinline__ bool any() {
    for (uint32_t c = threadIdx.x & 31u; c < n_chunk; c += 32u)
      if (is_hot(c)) first = min(first, c);
    first = __reduce_min_sync(0xffffffffu, first);
    return first != 0xFFFFFFFFu;
  }
  // whether row m, below those asked for before, is in a hot tile
  __device__ __forceinline__ bool row(uint32_t m) {
    if (m < row0) {
      const uint32_t c = m / chunk_rows;
      row0 = c * chunk_rows;
      on = is_hot(c);
    }
    return on;
  }
};

// Forward pass of the tiles that may carry weight (lnBtSG and the soft-max
// 2F): the window sums in double-word FP32 (ExpColumn; sums good to ~1e-14 of
// the window's magnitude, against FP64 recurrences at GB300's 1/70 FP64
// rate), F of the weighted cells in FP64 from them (the reference's formula
// and conditioning test, fstat64) into FP64 log-sum-exps.  A cell whose
// tier-1 F lies more than 62 max(1, T/2) below a lower bound of the template's
// maximum carries less than e^-60 in both sums (no_weight_below) and is skipped
// -- the tier-1 F is good to ~1.5e-6 relative and passes only for cond < 32,
// where the FP64 test passes too.
// kHot: the hot tiles of one column group per warp, their columns walked whole
// (HotGroup), where diff_hot_kernel leaves them to it.
template <bool kHot>
__global__ void __launch_bounds__(kDiffBlock, 5)
    diff_fwd_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                    const float *__restrict__ atoms8, const uint32_t *__restrict__ t0s_all,
                    const ColConsts *__restrict__ cols, const float *__restrict__ seg,
                    const float *__restrict__ need, const uint32_t *__restrict__ est, double temp,
                    DiffPartial *__restrict__ parts, HotRoute route) {
  __shared__ __align__(16) ExpRow s_tab[kDiffBlock / 32][kDiffRowTab];
  if (kHot && !route.warps()) return;
  DiffLane L;
  const uint32_t k = list[blockIdx.y];
  L.t = T[k];
  const uint32_t warp = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  const uint32_t cg = kHot ? warp : warp / L.t.n_chunk;
  if (cg >= L.t.n_cg || (kHot && L.t.whole)) return;
  const FwdBounds bd(est[k], temp);
  const float skip0 = bd.skip;
  DiffPartial *out = parts + L.t.part_off + (kHot ? (size_t)cg * L.t.n_chunk : warp);
  uint32_t mb, me = L.t.N_t0;
  HotGroup hot(need + L.t.part_off + (size_t)cg * L.t.n_chunk, L.t, skip0, bd.hot);
  if (kHot) {
    if (!hot.any()) return;
    mb = hot.first * L.t.chunk_rows;
  } else {
    if (L.t.whole != kDiffWholeBlind) {
      const float nd = need[L.t.part_off + warp];
      if (nd < skip0) {
        if (lane == 0) *out = DiffPartial{-INFINITY, 0.0, -INFINITY, 0.0};
        return;
      }
      if (!(nd < bd.hot) && !L.t.whole) return;  // a hot tile
    }
    mb = warp % L.t.n_chunk * L.t.chunk_rows;
    me = min(me, mb + L.t.chunk_rows);
  }
  L.columns(atoms8, t0s_all, cg);
  ExpColumn<false> C;
  C.init_consts(L.consts(cols));
  const float *sg = !kHot && L.t.g_nseg
                        ? seg + (L.t.seg_off + (size_t)cg * L.t.g_nseg) * kDiffSegFloats + lane
                        : nullptr;
  DiffLse lse(temp, skip0);
  const bool blind = L.t.whole == kDiffWholeBlind;
  const double below = no_weight_below(temp);
  diff_rows(L, mb, me, C, sg, kDiffSegFloats, s_tab[threadIdx.x >> 5],
            [&](uint32_t m, uint32_t, uint32_t, bool data) {
              if (kHot && !hot.row(m)) return;
              float F32 = 0.0f;
              const bool t1 = data && diff_tier1(C, F32);
              double W[7] = {0, 0, 0, 0, 0, 0, 0};
              if (data && !(t1 && F32 < lse.skip)) {
                W[0] = (double)C.W0.h.x + (double)C.W0.l.x;
                W[1] = (double)C.W0.h.y + (double)C.W0.l.y;
                W[2] = (double)C.Wc.h + (double)C.Wc.l;
                W[3] = (double)C.W2.h.x + (double)C.W2.l.x;
                W[4] = (double)C.W2.h.y + (double)C.W2.l.y;
                W[5] = (double)C.W3.h.x + (double)C.W3.l.x;
                W[6] = (double)C.W3.h.y + (double)C.W3.l.y;
              }
              lse.cell(data, W, t1, F32);
              if (!kHot && blind) lse.follow(below);
            });
  const DiffPartial p = lse.merge();
  if (!kHot) {
    if (lane == 0) *out = p;
    return;
  }
  // the group's hot cells are one partial, its other hot tiles' are empty
  for (uint32_t c = lane; c < L.t.n_chunk; c += 32u)
    if (hot.is_hot(c)) out[c] = c == hot.first ? p : DiffPartial{-INFINITY, 0.0, -INFINITY, 0.0};
}

// Whether a template's cells below `skip` carry no weight in the gradient: a
// cell's weight g = gB e^(F - Z1) + 2 gS e^(2F/T - Z2) (Z1 = logsumexp F,
// Z2 = logsumexp 2F/T, from the forward outputs) is below e^-40 when its
// tier-1 F (good to ~1e-5 of F) lies more than 42 below Z1 (the lnBtSG term,
// gB != 0) and more than 40 T + 1 below (T/2) Z2 (the soft-max term, gS != 0:
// its exponent is then below -80).
// `hot`: above it a single cell may carry more than e^-6 of either gradient
// (without an estimate, key 0, only NaN tiles are, as in the forward).
struct DiffWeights {
  double z1, z2, gb, gs;
  float skip, hot;
  __device__ __forceinline__ DiffWeights(const DiffTemplate &t, uint32_t k, uint32_t key,
                                         double temp, const double *lnZ1, const double *lnZ2,
                                         const double *gB, const double *gS) {
    z1 = lnZ1[k] - log(70.0 / ((double)t.N_t0 * (double)t.N_tau));
    z2 = lnZ2[k] / temp;
    gb = gB[k];
    gs = gS[k];
    const double sk1 = gb != 0.0 ? z1 - 42.0 : INFINITY;
    const double sk2 = gs != 0.0 ? 0.5 * temp * (z2 - 80.0) - 1.0 : INFINITY;
    skip = (float)fmin(sk1, sk2);
    hot = (float)fmin(gb != 0.0 ? z1 - 1e-5 * fabs(z1) - 7.0 : INFINITY,
                      gs != 0.0 ? 0.5 * temp * (z2 - 1e-5 * fabs(z2) - 25.0) - 0.1 : INFINITY);
    if (!key) hot = INFINITY;
  }
};

// Segment sums (exp_seg_kernel's, with TwoSum steps; kV: with the tau
// derivatives, only for column groups that diff_src_kernel walks).
template <bool kV>
__global__ void __launch_bounds__(kDiffBlock)
    diff_seg_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                    const float *__restrict__ atoms8, const uint32_t *__restrict__ t0s_all,
                    const ColConsts *__restrict__ cols, const float *__restrict__ need,
                    const uint32_t *__restrict__ est, double temp,
                    const double *__restrict__ lnZ1, const double *__restrict__ lnZ2,
                    const double *__restrict__ gB, const double *__restrict__ gS, uint32_t per,
                    float *__restrict__ seg) {
  DiffLane L;
  const uint32_t k = list[blockIdx.y];
  L.t = T[k];
  const uint32_t w = blockIdx.x * 4u + (threadIdx.x >> 5);
  const uint32_t cg = w % L.t.n_cg, j0 = w / L.t.n_cg * per;
  if (j0 >= L.t.g_nseg) return;
  if (kV) {
    const DiffWeights w(L.t, k, est[k], temp, lnZ1, lnZ2, gB, gS);
    const float *nd = need + L.t.part_off + (size_t)cg * L.t.n_chunk;
    bool any = false;
    for (uint32_t c = threadIdx.x & 31u; c < L.t.n_chunk; c += 32u)
      any = any || (!(nd[c] < w.skip) && nd[c] < w.hot);
    if (!__any_sync(0xffffffffu, any)) return;
  }
  L.columns(atoms8, t0s_all, cg);
  const uint32_t shift = L.t.g_shift, j1 = min(L.t.g_nseg, j0 + per);
  // a window holds fewer than 3 tau / TAtom + 2 atoms: shorter ones are never joined
  if (3ull * L.taumax + 2ull * L.t.g.TAtom < ((uint64_t)L.t.g.TAtom << (shift + 1u))) return;
  for (uint32_t j = j0; j < j1; j++) {
    const uint32_t lo = j << shift, top = min(L.t.g.numAtoms, (j + 1u) << shift);
    if (kV) {
      ExpColumnV C;
      C.C.init_consts(L.consts(cols));
      C.reset_v();
      C.slide(L.a8, L.t.g, lo, top, 0u);
      C.store_sums(seg + (L.t.seg_off + (size_t)cg * L.t.g_nseg + j) * kDiffSegFloatsV +
                   (threadIdx.x & 31u));
    } else {
      ExpColumn<false> C;
      C.init_consts(L.consts(cols));
      C.slide(L.a8, L.t.g, lo, top, 0u);
      C.store_sums(seg + (L.t.seg_off + (size_t)cg * L.t.g_nseg + j) * kDiffSegFloats +
                   (threadIdx.x & 31u));
    }
  }
}

// The cell's gradient dL/dF dF/dW_c (Gf) from its double-word window sums in
// double-word arithmetic, and G_c k_c V_c added to dtw; false (and Gf
// untouched) where the conditioning test fails.
struct DiffGrad {
  FF z1w, z2w, twoT;
  float gbf, gsf;
  DiffGrad() = default;
  __device__ __forceinline__ DiffGrad(const DiffWeights &w, double temp)
      : z1w(dw_from(w.z1)), z2w(dw_from(w.z2)), twoT(dw_from(2.0 / temp)), gbf((float)w.gb),
        gsf((float)w.gs) {}
  __device__ __forceinline__ bool cell(const FF W[7], const FF V[7], float Gf[7], FF &dtw) const {
    const FF A = W[0], B = W[1], Cc = W[2], Far = W[3], Fai = W[4], Fbr = W[5], Fbi = W[6];
    const DwCell fc = dw_fstat(A, B, Cc, Far, Fai, Fbr, Fbi);
    if (!fc.ok) return false;
    const FF F = fc.F;
    // exponents of the weights from double-word differences
    const FF d1 = dw_sub(F, z1w);
    const FF d2 = dw_sub(ff_mul(F, twoT), z2w);
    const float g = gbf * exp2f(fadd(d1.h, d1.l) * kLog2eF) +
                    gsf * 2.0f * exp2f(fadd(d2.h, d2.l) * kLog2eF);
    const FF Fa2 = dw_add(ff_mul(Far, Far), ff_mul(Fai, Fai));
    const FF re = dw_add(ff_mul(Far, Fbr), ff_mul(Fai, Fbi));
    FF dF[7];
    dF[0] = ff_mul(dw_sub(fc.Fb2, ff_mul(F, B)), fc.iD);
    dF[1] = ff_mul(dw_sub(Fa2, ff_mul(F, A)), fc.iD);
    dF[2] = dw_twice(ff_mul(dw_sub(ff_mul(F, Cc), re), fc.iD));
    dF[3] = dw_twice(ff_mul(fc.Gre, fc.iD));
    dF[4] = dw_twice(ff_mul(fc.Gim, fc.iD));
    dF[5] = dw_twice(ff_mul(dw_sub(ff_mul(A, Fbr), ff_mul(Cc, Far)), fc.iD));
    dF[6] = dw_twice(ff_mul(dw_sub(ff_mul(A, Fbi), ff_mul(Cc, Fai)), fc.iD));
#pragma unroll
    for (int c = 0; c < 7; c++) {
      const FF Gc = dw_mulf(dF[c], g);
      Gf[c] = fadd(Gc.h, Gc.l);
      const FF tv = ff_mul(Gc, V[c]);
      dtw = dw_add(dtw, c < 3 ? dw_twice(tv) : tv);
    }
    return true;
  }
};

// r^L, L = top - lo, for the removal in the transposed recurrence (FP64, one
// multiplication when L moves by one), as a float pair.
struct DiffPower {
  double r1 = 0.0, inv_r1 = 0.0, pw = 1.0;
  uint32_t len = 0;
  bool init = false;
  __device__ __forceinline__ FF at(const DiffLane &L, uint32_t n) {
    if (!init) {
      r1 = exp(-(double)L.t.g.TAtom / L.tau);
      inv_r1 = r1 > 1e-280 ? 1.0 / r1 : 0.0;
      init = true;
    }
    if (n != len) {
      if (n == len + 1u) {
        pw *= r1;
      } else if (n + 1u == len && inv_r1 > 0.0) {
        pw *= inv_r1;
      } else {  // square and multiply: pow()'s chain of FP64 steps is ten times as long
        double base = r1;
        pw = 1.0;
        for (uint32_t q = n; q; q >>= 1) {
          if (q & 1u) pw *= base;
          base *= base;
        }
      }
      len = n;
    }
    const float h = (float)pw;
    return FF{h, (float)(pw - (double)h)};
  }
};

__device__ __forceinline__ void add_grad_tau(const DiffLane &L, FF dtw, double *grad_tau) {
  const double dtau = (double)dtw.h + (double)dtw.l;
  const double scale = L.active ? (double)L.t.g.TAtom / (L.tau * L.tau) * dtau : 0.0;
  const double fr = (L.active && L.t.N_tau > 1) ? (double)L.n / (double)(L.t.N_tau - 1u) : 0.0;
  double dmax = scale * fr,
         dmin = scale * (L.active && L.t.N_tau > 1 ? 1.0 - fr : (L.active ? 1.0 : 0.0));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    dmax += __shfl_down_sync(0xffffffffu, dmax, d);
    dmin += __shfl_down_sync(0xffffffffu, dmin, d);
  }
  if ((threadIdx.x & 31u) == 0) {
    atomicAdd(grad_tau, dmin);
    atomicAdd(grad_tau + 1, dmax);
  }
}

// Adjoint sources of the tiles that may carry weight: W and V slide down each
// tau column in double-word FP32 (ExpColumnV); a cell gets F, dF/dW and its
// sources (in double-word arithmetic, dw_fstat) only when it carries weight
// (DiffWeights).  kHot: as in diff_fwd_kernel.
template <bool kHot>
__global__ void __launch_bounds__(kDiffBlock)
    diff_src_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                    const float *__restrict__ atoms8, const uint32_t *__restrict__ t0s_all,
                    const ColConsts *__restrict__ cols, const float *__restrict__ seg,
                    float *__restrict__ need, const uint32_t *__restrict__ est, double temp,
                    const double *__restrict__ lnZ1, const double *__restrict__ lnZ2,
                    const double *__restrict__ gB, const double *__restrict__ gS, uint32_t cg0,
                    uint32_t cgs, float *__restrict__ scratch, double *__restrict__ grad_tau,
                    HotRoute route) {
  __shared__ __align__(16) ExpRow s_tab[kDiffBlock / 32][kDiffRowTab];
  if (kHot && !route.warps()) return;
  DiffLane L;
  const uint32_t k = list[blockIdx.y];
  L.t = T[k];
  const DiffTemplate &t = L.t;
  // the slice's tiles; scratch holds those of column groups [cg0, cg0 + cgs)
  const uint32_t warp = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  const uint32_t scg = kHot ? warp : warp / t.n_chunk, cg = cg0 + scg;
  if (scg >= cgs || cg >= t.n_cg || (kHot && t.whole)) return;
  const DiffWeights w(t, k, est[k], temp, lnZ1, lnZ2, gB, gS);
  uint32_t mb, me = t.N_t0;
  HotGroup hot(need + t.part_off + (size_t)cg * t.n_chunk, t, w.skip, w.hot);
  if (kHot) {
    if (!hot.any()) return;
    mb = hot.first * t.chunk_rows;
  } else {
    if (!t.whole) {
      const float nd = need[t.part_off + cg0 * t.n_chunk + warp];
      if (nd < w.skip) return;     // diff_atoms_kernel skips its rows
      if (!(nd < w.hot)) return;  // a hot tile
    }
    mb = warp % t.n_chunk * t.chunk_rows;
    me = min(me, mb + t.chunk_rows);
  }
  L.columns(atoms8, t0s_all, cg);
  const DiffGrad grad(w, temp);
  DiffPower power;
  FF dtw{0.0f, 0.0f};
  bool some = false;
  ExpColumnV CV;
  CV.C.init_consts(L.consts(cols));
  CV.reset_v();
  const float *sg = !kHot && t.g_nseg
                        ? seg + (t.seg_off + (size_t)cg * t.g_nseg) * kDiffSegFloatsV + lane
                        : nullptr;
  // (a column group's rows in order: its tiles are chunk_rows each but for the last)
  float *my = scratch + t.scr_off +
              (size_t)scg * t.n_chunk * t.chunk_rows * (TCW_DIFF_SLOTS * 32u) + lane;
  diff_rows(L, mb, me, CV, sg, kDiffSegFloatsV, s_tab[threadIdx.x >> 5],
            [&](uint32_t m, uint32_t lo, uint32_t top, bool data) {
              if (kHot && !hot.row(m)) return;
              float Gf[7] = {0, 0, 0, 0, 0, 0, 0};
              FF p1{0.0f, 0.0f};
              if (data) {
                const ExpColumn<false> &C = CV.C;
                float F32;
                const bool t1 = diff_tier1(C, F32);
                if (!(t1 && F32 < w.skip)) {
                  const FF W[7] = {FF{C.W0.h.x, C.W0.l.x}, FF{C.W0.h.y, C.W0.l.y}, C.Wc,
                                   FF{C.W2.h.x, C.W2.l.x}, FF{C.W2.h.y, C.W2.l.y},
                                   FF{C.W3.h.x, C.W3.l.x}, FF{C.W3.h.y, C.W3.l.y}};
                  const FF V[7] = {FF{CV.V0.h.x, CV.V0.l.x}, FF{CV.V0.h.y, CV.V0.l.y}, CV.Vc,
                                   FF{CV.V2.h.x, CV.V2.l.x}, FF{CV.V2.h.y, CV.V2.l.y},
                                   FF{CV.V3.h.x, CV.V3.l.x}, FF{CV.V3.h.y, CV.V3.l.y}};
                  if (grad.cell(W, V, Gf, dtw)) {
                    p1 = power.at(L, top - lo);
                    some = true;
                  }
                }
              }
              TCW_DCHECK(m < t.N_t0);
              float *scr = my + (size_t)m * (TCW_DIFF_SLOTS * 32u);
#pragma unroll
              for (int c = 0; c < 7; c++) scr[32 * c] = Gf[c];
              scr[32 * 7] = p1.h;
              scr[32 * 8] = p1.l;
            });
  add_grad_tau(L, dtw, grad_tau + 2u * k);
  if (!kHot && t.whole) {  // (no estimate: for diff_atoms_kernel)
    some = __any_sync(0xffffffffu, some);
    if (lane == 0) need[t.part_off + cg] = some ? INFINITY : -INFINITY;
  }
}

// Most atoms of a template that diff_hot_kernel keeps in shared memory.
constexpr uint32_t kHotAtoms = 7000;
// Its evaluating warps, and the rows of each half of its ring of window sums.
constexpr uint32_t kHotEval = 2;
constexpr uint32_t kHotThreads = (7u + kHotEval) * 32u;

// Barriers of diff_hot_kernel: all its warps, when a half of the ring is full;
// the seven walking warps.
__device__ __forceinline__ void hot_ring_sync() {
  asm volatile("barrier.sync 1, %0;" ::"r"(kHotThreads) : "memory");
}
__device__ __forceinline__ void hot_walk_sync() {
  asm volatile("barrier.sync 2, %0;" ::"r"(7u * 32u) : "memory");
}

// The tiles whose cells matter by themselves.  Their F enters the results
// through exponents of 20 F, where the last bits of the window sums show, so
// their columns are walked whole from the last row down -- a tile started
// from segment sums agrees to ~1e-14 of the sums only.  A whole walk by one
// thread per column is a long serial chain (W, V and the removal powers of 7
// channels: 2.4 ms for 1024 rows); here a block takes 32 columns with one
// warp per channel, whose steps are the packed pairs' bit for bit, and two
// more warps evaluate the hot rows from shared memory while the others walk
// on.  Column groups without a hot tile leave at once, and so do all of them
// where more have one than blocks are good for (HotRoute).
// Bound by the latency of each walking warp's own dependent instructions
// (~1000 cycles per row of 2 atoms), so: the loops hold no evaluation code,
// the next removal power is prepared beside the present sums, and a block may
// use all the registers (96 by the compiler's own choice cost 30 %).  Forward
// / backward of one 1024 x 1024 template 756 / 816 -> 517 / 577 us against one
// evaluating warp and powers in the chain, of 24 templates 1096 / 972 -> 650 /
// 757 (73 pairs of hot rows in a group: evaluating one takes as long as
// walking two, one warp alone 870 / 947, three as two).
template <bool kBack>
__global__ void __launch_bounds__(kHotThreads, 1)
    diff_hot_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                    const float *__restrict__ atoms8, const uint32_t *__restrict__ t0s_all,
                    const ColConsts *__restrict__ cols, const float *__restrict__ need,
                    const uint32_t *__restrict__ est, double temp,
                    const double *__restrict__ lnZ1, const double *__restrict__ lnZ2,
                    const double *__restrict__ gB, const double *__restrict__ gS, uint32_t cg0,
                    float *__restrict__ scratch, double *__restrict__ grad_tau,
                    DiffPartial *__restrict__ parts, uint32_t smem_atoms, HotRoute route) {
  extern __shared__ float s_x[];  // channel-major atoms, where a template's fit
  __shared__ float2 s_pow[32][32];  // r^(2^b) of the lanes' columns
  constexpr int kWords = kBack ? 4 : 2;
  __shared__ __align__(16) ExpRow tab[kDiffRowTab];
  struct HotRow {
    ExpRow e;
    uint32_t m;
    bool reg;
  };
  __shared__ float s_sum[2][kHotEval][7][kWords][32];
  __shared__ HotRow s_row[2][kHotEval];
  __shared__ DiffPartial s_part[kHotEval];
  __shared__ uint8_t s_hot[kDiffRowTab];
  if (route.warps()) return;
  DiffLane L;
  const uint32_t k = list[blockIdx.y], cg = cg0 + blockIdx.x;  // (grid x: a slice's groups)
  L.t = T[k];
  const DiffTemplate &t = L.t;
  if (cg >= t.n_cg || t.whole) return;
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  const float *nd = need + t.part_off + (size_t)cg * t.n_chunk;
  // the first and last hot chunk
  float hot, skip;
  DiffGrad grad;
  if (kBack) {
    const DiffWeights w(t, k, est[k], temp, lnZ1, lnZ2, gB, gS);
    hot = w.hot;
    skip = w.skip;
    grad = DiffGrad(w, temp);
  } else {
    const FwdBounds bd(est[k], temp);
    hot = bd.hot;
    skip = bd.skip;
  }
  auto is_hot = [&](uint32_t c) { return !(nd[c] < skip) && !(nd[c] < hot); };
  uint32_t c0 = 0xFFFFFFFFu;
  for (uint32_t c = lane; c < t.n_chunk; c += 32u)
    if (is_hot(c)) c0 = min(c0, c);
  c0 = __reduce_min_sync(0xffffffffu, c0);
  if (c0 == 0xFFFFFFFFu) return;  // the same in every warp
  const uint32_t mb = c0 * t.chunk_rows;  // rows below the last hot one are not walked
  L.columns(atoms8, t0s_all, cg);
  const uint32_t *a8u = reinterpret_cast<const uint32_t *>(L.a8);
  const ColConsts cc = L.consts(cols);
  const ExpConsts kc = cc.consts();

  const uint32_t N = t.g.numAtoms;
  const bool staged = N <= smem_atoms;
  if (staged)
    for (uint32_t i = threadIdx.x; i < N * 8u; i += blockDim.x)
      if ((i & 7u) != 3u) s_x[((i & 7u) - ((i & 7u) > 3u ? 1u : 0u)) * N + (i >> 3)] = __ldg(L.a8 + i);
  if (wid == 7u) {  // ff_pow's squarings, once per column
    FF base = kc.r1;
    for (uint32_t b = 0; b < 32u && (1ull << b) <= N; b++) {
      s_pow[b][lane] = make_float2(base.h, base.l);
      base = ff_mul(base, base);
    }
  }
  __syncthreads();

  // this warp's channel (warps 0..6)
  const uint32_t ch = wid < 7u ? wid : 0u;
  const uint32_t slot = ch < 3u ? ch : ch + 1u;
  const FF r = ch < 3u ? kc.r2 : kc.r1;
  FF W{0.0f, 0.0f}, V{0.0f, 0.0f}, pw{1.0f, 0.0f};
  uint32_t wlo = 0, wtop = 0, Lp = 0;
  bool pinit = false;
  // this channel's atoms, in shared memory or not: one generic load, no branch
  const float *xp = staged ? s_x + ch * N : L.a8 + slot;
  const uint32_t xs = staged ? 1u : 8u;
  auto atom = [&](uint32_t i) {  // (the index below atom 0 reads atom 0)
    return xp[(size_t)(i < N ? i : 0u) * xs];
  };
  float xl = 0.0f, xe = 0.0f;  // the atoms that leave and enter next
  // A lone warp waits for every instruction's result, so what counts is the
  // longest dependent chain of a step: the next leaving atom's power is
  // prepared beside the sums of the present step, and taken over (pw, Lp)
  // only when an atom leaves.
  FF np{1.0f, 0.0f}, pc{1.0f, 0.0f}, pv{0.0f, 0.0f};
  uint32_t ex = 0;
  auto prepare = [&]() {  // ExpColumn::power
    ex = wtop - 1u - wlo;
    const bool same = ex == Lp, up = ex == Lp + 1u, down = ex + 1u == Lp && kc.has_inv;
    const FF step = ff_mul(pw, up ? kc.r1 : kc.r1inv);
    np = up || down ? step : pw;
    FF sq = ff_mul(np, np);
    if (!(pinit && (same || up || down)) && wtop > wlo) {
      np = FF{1.0f, 0.0f};  // ff_pow from the table
      for (uint32_t q = ex; q; q &= q - 1u) {
        const float2 f = s_pow[__ffs(q) - 1][lane];
        np = ff_mul(np, FF{f.x, f.y});
      }
      sq = ff_mul(np, np);
    }
    pc = ch < 3u ? sq : np;  // this channel's weight, and times its exponent
    if (kBack) pv = ff_mul(pc, FF{(float)ex, 0.0f});
  };
  auto leave = [&](bool on) {
    const FF w = ff_sub_scaled_x1(W, pc, xl);
    if (kBack) {
      const FF v = ff_sub_scaled_x1(V, pv, xl);
      V = on ? v : V;
    }
    W = on ? w : W;
    pw = on ? np : pw;
    Lp = on ? ex : Lp;
    pinit = pinit || on;
    wtop -= on ? 1u : 0u;
    xl = atom(wtop - 1u);
  };
  auto enter = [&](bool on) {
    if (kBack) {
      const FF v = ff_scale_dw(r, ff_add_dw(V, W));
      V = on ? v : V;
    }
    const FF w = ff_axpy(xe, r, W);
    W = on ? w : W;
    wlo -= on ? 1u : 0u;
    xe = atom(wlo - 1u);
  };
  // an evaluating warp's state
  DiffLse lse(temp, skip);
  FF dtw{0.0f, 0.0f};
  DiffPower power;
  uint32_t half = 0, fill = 0;  // the ring's half that is being filled, its rows so far

  auto window = [&](const ExpRow &e, bool reg, uint32_t &top) {
    if (reg) {
      top = e.a + cc.Qp1 - ((e.b + cc.RmT) >> 31);  // ExpColumn::top_of
      top = top < 1u ? 1u : top;
      top = top < t.g.numAtoms ? top : t.g.numAtoms;
      return e.lo < top;
    }
    uint32_t hi;
    const bool some = exp_hi_real(e.a, L.tau, t.g, hi) && e.lo <= hi;
    top = some ? hi + 1u : 0u;
    return some;
  };
  // row `wid - 7` of the half that was filled before the last barrier
  auto evaluate = [&](uint32_t filled, uint32_t rows) {
    const uint32_t q = wid - 7u;
    if (wid < 7u || q >= rows || !L.active) return;
    const HotRow row = s_row[filled][q];
    float(*sum)[kWords][32] = s_sum[filled][q];
    uint32_t top;
    const bool data = window(row.e, row.reg, top) && row.e.nz < top;
    FF Wr[7];
#pragma unroll
    for (int c = 0; c < 7; c++) Wr[c] = FF{sum[c][0][lane], sum[c][1][lane]};
    float F32 = 0.0f;
    const bool t1 = data && fstat_fast(Wr, F32);
    if (!kBack) {
      double Wd[7] = {0, 0, 0, 0, 0, 0, 0};
      if (data && !(t1 && F32 < lse.skip)) {
#pragma unroll
        for (int c = 0; c < 7; c++) Wd[c] = (double)Wr[c].h + (double)Wr[c].l;
      }
      lse.cell(data, Wd, t1, F32);
    } else {
      float Gf[7] = {0, 0, 0, 0, 0, 0, 0};
      FF p1{0.0f, 0.0f};
      if (data && !(t1 && F32 < skip)) {
        FF Vr[7];
#pragma unroll
        for (int c = 0; c < 7; c++)
          Vr[c] = FF{sum[c][kWords - 2][lane], sum[c][kWords - 1][lane]};
        if (grad.cell(Wr, Vr, Gf, dtw)) p1 = power.at(L, top - row.e.lo);
      }
      const uint32_t c = row.m / t.chunk_rows;
      float *scr = scratch + t.scr_off +
                   ((size_t)((cg - cg0) * t.n_chunk + c) * t.chunk_rows +
                    (row.m - c * t.chunk_rows)) *
                       (TCW_DIFF_SLOTS * 32u) +
                   lane;
#pragma unroll
      for (int c7 = 0; c7 < 7; c7++) scr[32 * c7] = Gf[c7];
      scr[32 * 7] = p1.h;
      scr[32 * 8] = p1.l;
    }
  };

  if (wid >= 7u) {  // the evaluating warps: a barrier for every half that is filled
    uint32_t rows = 0;  // hot rows, all of them at or above mb
    for (uint32_t c = lane; c < t.n_chunk; c += 32u)
      if (is_hot(c)) rows += min(t.N_t0, (c + 1u) * t.chunk_rows) - c * t.chunk_rows;
    rows = __reduce_add_sync(0xffffffffu, rows);
    for (; rows; half ^= 1u) {
      const uint32_t n = min(rows, kHotEval);
      hot_ring_sync();
      evaluate(half, n);
      rows -= n;
    }
  } else {
    for (uint32_t ce = t.N_t0; ce > mb;) {
      const uint32_t cb = ce - mb > kDiffRowTab ? ce - kDiffRowTab : mb;
      bool reg = true;  // the same in every warp
      for (uint32_t q = lane; q < ce - cb; q += 32u)
        reg = reg && exp_row_regular(__ldg(L.t0s + cb + q), L.taumax, t.g);
      reg = __all_sync(0xffffffffu, reg);
      hot_walk_sync();
      for (uint32_t q = threadIdx.x; q < ce - cb; q += 7u * 32u) {
        const uint32_t t0 = __ldg(L.t0s + cb + q);
        ExpRow e;
        e.lo = exp_lo(t0, t.g);
        e.nz = e.lo < t.g.numAtoms ? __ldg(a8u + (size_t)e.lo * 8u + 3u) : 0xFFFFFFFFu;
        const uint32_t d = t0 - t.g.t0_data;
        e.a = reg ? fdiv(d, t.g.div) : t0;  // irregular chunks: the generic branch reads t0
        e.b = reg ? d - e.a * t.g.TAtom : 0u;
        tab[q] = e;
        s_hot[q] = is_hot((cb + q) / t.chunk_rows) ? 1 : 0;
      }
      hot_walk_sync();
#pragma unroll 1
      for (uint32_t m = ce; m > cb;) {
        m--;
        const ExpRow e = tab[m - cb];
        const bool hot_row = s_hot[m - cb];
        uint32_t top;
        if (window(e, reg, top) && L.active) {
          if (top > wtop || e.lo > wlo || top <= wlo) {
            wlo = wtop = top;
            xl = xe = atom(top - 1u);
            W = V = FF{0.0f, 0.0f};
          }
          // ExpColumn::slide alternates, ExpColumnV::slide does not
          const uint32_t nl = wtop - top;
          if (kBack) {
#pragma unroll 1
            for (uint32_t j = 0; j < nl; j++) {
              leave(true);
              prepare();
            }
          } else {
            const uint32_t ne = wlo - e.lo, n = max(nl, min(ne, nl + 2u));
#pragma unroll 1
            for (uint32_t j = 0; j < n; j++) {
              leave(j < nl);
              enter(j < ne);
              prepare();
            }
          }
          if (wlo > e.lo) {
#pragma unroll 1
            while (wlo > e.lo) enter(true);
            prepare();
          }
        }
        if (!hot_row) continue;
        float(*sum)[kWords][32] = s_sum[half][fill];
        sum[ch][0][lane] = W.h;
        sum[ch][1][lane] = W.l;
        if (kBack) {
          sum[ch][kWords - 2][lane] = V.h;
          sum[ch][kWords - 1][lane] = V.l;
        }
        if (threadIdx.x == 0) s_row[half][fill] = HotRow{e, m, reg};
        if (++fill < kHotEval) continue;
        hot_ring_sync();  // (the readers of the other half are done, too)
        half ^= 1u;
        fill = 0;
      }
      ce = cb;
    }
    if (fill) hot_ring_sync();
  }
  if (kBack) {
    if (wid >= 7u) add_grad_tau(L, dtw, grad_tau + 2u * k);
    return;
  }
  // the group's hot cells are one partial, its other hot tiles' are empty
  if (wid >= 7u) {
    const DiffPartial p = lse.merge();
    if (lane == 0) s_part[wid - 7u] = p;
  }
  __syncthreads();
  if (wid != 7u) return;
  DiffPartial sum{-INFINITY, 0.0, -INFINITY, 0.0};
  for (uint32_t q = 0; q < kHotEval; q++) {
    sum.m1 = fmax(sum.m1, s_part[q].m1);
    sum.m2 = fmax(sum.m2, s_part[q].m2);
  }
  for (uint32_t q = 0; q < kHotEval; q++) {
    if (s_part[q].s1 != 0.0) sum.s1 += s_part[q].s1 * exp(s_part[q].m1 - sum.m1);
    if (s_part[q].s2 != 0.0) sum.s2 += s_part[q].s2 * exp(s_part[q].m2 - sum.m2);
  }
  for (uint32_t c = lane; c < t.n_chunk; c += 32u)
    if (is_hot(c))
      parts[t.part_off + (size_t)cg * t.n_chunk + c] =
          c == c0 ? sum : DiffPartial{-INFINITY, 0.0, -INFINITY, 0.0};
}

// Counts the column groups that have a hot tile (HotRoute), a thread each.
template <bool kBack>
__global__ void __launch_bounds__(kDiffBlock)
    diff_route_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                      const float *__restrict__ need, const uint32_t *__restrict__ est,
                      double temp, const double *__restrict__ lnZ1,
                      const double *__restrict__ lnZ2, const double *__restrict__ gB,
                      const double *__restrict__ gS, uint32_t *__restrict__ groups) {
  const uint32_t k = list[blockIdx.y], cg = blockIdx.x * kDiffBlock + threadIdx.x;
  const DiffTemplate t = T[k];
  bool any = false;
  if (cg < t.n_cg && !t.whole) {
    float skip, hot;
    if (kBack) {
      const DiffWeights w(t, k, est[k], temp, lnZ1, lnZ2, gB, gS);
      skip = w.skip;
      hot = w.hot;
    } else {
      const FwdBounds bd(est[k], temp);
      skip = bd.skip;
      hot = bd.hot;
    }
    const HotGroup g(need + t.part_off + (size_t)cg * t.n_chunk, t, skip, hot);
    for (uint32_t c = 0; c < t.n_chunk && !any; c++) any = g.is_hot(c);
  }
  const uint32_t n = __syncthreads_count(any);
  if (threadIdx.x == 0 && n) atomicAdd(groups, n);
}

// The transposed recurrence over one segment of 2^a_shift atoms of one column
// group, in double-word FP32, from the adjoint sources of the rows in the
// group's weighted chunks.  kEnds: leaves H at the segment's end, started from
// zero, in `cend` (but for the last segment, whose end nothing reads); else
// starts from the ends below and adds every atom's sum over the warp's columns
// to the gradient.
template <bool kEnds>
__global__ void __launch_bounds__(kDiffBlock)
    diff_atoms_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                      const float *__restrict__ atoms8, const uint32_t *__restrict__ t0s_all,
                      const ColConsts *__restrict__ cols, const float *__restrict__ need,
                      const uint32_t *__restrict__ est, double temp,
                      const double *__restrict__ lnZ1, const double *__restrict__ lnZ2,
                      const double *__restrict__ gB, const double *__restrict__ gS, uint32_t cg0,
                      uint32_t cgs, const float *__restrict__ scratch, float *__restrict__ cend,
                      double *__restrict__ grad_atoms) {
  DiffLane L;
  const uint32_t k = list[blockIdx.y];
  L.t = T[k];
  const DiffTemplate &t = L.t;
  const uint32_t wi = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  const uint32_t scg = wi / t.n_aseg, cg = cg0 + scg, as = wi % t.n_aseg;
  if (scg >= cgs || cg >= t.n_cg || (kEnds && as + 1u >= t.n_aseg)) return;
  // the group's weighted chunks: first and last
  uint32_t c0 = 0xFFFFFFFFu, c1 = 0;
  {
    const DiffWeights w(t, k, est[k], temp, lnZ1, lnZ2, gB, gS);
    const float *nd = need + t.part_off + (size_t)cg * t.n_chunk;
    for (uint32_t c = lane; c < t.n_chunk; c += 32u)
      if (!(nd[c] < w.skip)) {
        c0 = min(c0, c);
        c1 = max(c1, c + 1u);
      }
    c0 = __reduce_min_sync(0xffffffffu, c0);
    c1 = __reduce_max_sync(0xffffffffu, c1);
    if (c0 >= c1) return;
    L.columns(atoms8, t0s_all, cg);
    const uint32_t rb = c0 * t.chunk_rows, re = min(t.N_t0, c1 * t.chunk_rows);
    const uint32_t *t0s = L.t0s;
    const ColConsts cc = L.consts(cols);
    // one past the window end of row m (the window start for empty windows:
    // removal right after injection), from the integer split on regular
    // rows, else from the real t1
    auto row_end = [&](uint32_t m) -> uint32_t {
      const uint32_t t0 = __ldg(t0s + m);
      const uint32_t lo = exp_lo(t0, t.g);
      if (exp_row_regular(t0, L.taumax, t.g)) {
        const uint32_t dd = t0 - t.g.t0_data;
        const uint32_t a = fdiv(dd, t.g.div), b = dd - a * t.g.TAtom;
        uint32_t top = a + cc.Qp1 - ((b + cc.RmT) >> 31);
        top = top < 1u ? 1u : (top < t.g.numAtoms ? top : t.g.numAtoms);
        return lo < top ? top : lo;
      }
      uint32_t hi;
      return (exp_hi_real(t0, L.tau, t.g, hi) && lo <= hi) ? hi + 1u : lo;
    };
    // the group's atoms: from its first weighted row's window start to the
    // largest window end
    const uint32_t i_begin = exp_lo(__ldg(t0s + rb), t.g);
    const uint32_t i_end =
        __reduce_max_sync(0xffffffffu, L.active ? row_end(re - 1u) : i_begin);
    const uint32_t a = max(i_begin, as << t.a_shift);
    const uint32_t b = as + 1u < t.n_aseg ? min(i_end, (as + 1u) << t.a_shift) : i_end;
    if (a >= b) return;
    const ExpConsts kc = cc.consts();
    const ExpConsts2 kp = exp_consts2(kc);
    // H: (A,B) and C decay with r^2, (Fa) and (Fb) with r
    const F2 zp{0.0f, 0.0f};
    FF2 H01{zp, zp}, H34{zp, zp}, H56{zp, zp};
    FF H2{0.0f, 0.0f};
    float *ends = cend + (t.cend_off + (size_t)scg * t.n_aseg) * kDiffSegFloats + lane;
    if (!kEnds) {  // H = r^len H + end, segment by segment from the first
      const uint32_t s0 = i_begin >> t.a_shift;
      FF R = kc.r1;  // r^(2^a_shift)
#pragma unroll 1
      for (uint32_t q = 0; q < t.a_shift; q++) R = ff_mul(R, R);
      const FF R2 = ff_mul(R, R);
      const F2 rh0{R2.h, R2.h}, nrh0{-R2.h, -R2.h}, rl0{R2.l, R2.l};
      const F2 rh1{R.h, R.h}, nrh1{-R.h, -R.h}, rl1{R.l, R.l};
      for (uint32_t j = s0; j < as; j++) {
        const float *s = ends + (size_t)j * kDiffSegFloats;
        H01 = ff2_axpy_dw(FF2{F2{s[0], s[32]}, F2{s[64], s[96]}}, rh0, nrh0, rl0, H01);
        H2 = ff_axpy_dw(FF{s[128], s[160]}, R2, H2);
        H34 = ff2_axpy_dw(FF2{F2{s[192], s[224]}, F2{s[256], s[288]}}, rh1, nrh1, rl1, H34);
        H56 = ff2_axpy_dw(FF2{F2{s[320], s[352]}, F2{s[384], s[416]}}, rh1, nrh1, rl1, H56);
      }
    }
    // the first row whose window starts at or after atom a, and this
    // column's first row that ends at or after it (earlier ones are removed)
    uint32_t mi = rb, hiw = re;
    if (a > i_begin) {
      while (mi < hiw) {
        const uint32_t mid = (mi + hiw) >> 1;
        if (exp_lo(__ldg(t0s + mid), t.g) < a) mi = mid + 1u; else hiw = mid;
      }
    }
    uint32_t mr = rb;
    hiw = re;
    if (a > i_begin) {
      while (mr < hiw) {
        const uint32_t mid = (mr + hiw) >> 1;
        if (row_end(mid) < a) mr = mid + 1u; else hiw = mid;
      }
    }
    uint32_t lo_next = mi < re ? exp_lo(__ldg(t0s + mi), t.g) : 0u;
    uint32_t end_r = mr < re ? row_end(mr) : 0u;
    const float *scr0 = scratch + t.scr_off + lane;
    auto sources = [&](uint32_t m) -> const float * {  // NULL: the row carries no weight
      const uint32_t c = m / t.chunk_rows;
      if (nd[c] < w.skip) return nullptr;
      return scr0 + ((size_t)(scg * t.n_chunk + c) * t.chunk_rows + (m - c * t.chunk_rows)) *
                        (TCW_DIFF_SLOTS * 32u);
    };
    for (uint32_t i = a; i < b; i++) {
      if (L.active) {
        H01 = ff2_scale_dw(kp.rh[0], kp.nrh[0], kp.rl[0], H01);
        H2 = ff_scale_dw(kc.r2, H2);
        H34 = ff2_scale_dw(kp.rh[1], kp.nrh[1], kp.rl[1], H34);
        H56 = ff2_scale_dw(kp.rh[1], kp.nrh[1], kp.rl[1], H56);
        while (mi < re && lo_next <= i) {
          const float *scr = sources(mi);
          if (scr) {
            H01 = ff2_add_x(H01, F2{scr[0], scr[32 * 1]});
            H2 = ff_add1(H2, scr[32 * 2]);
            H34 = ff2_add_x(H34, F2{scr[32 * 3], scr[32 * 4]});
            H56 = ff2_add_x(H56, F2{scr[32 * 5], scr[32 * 6]});
          }
          mi++;
          if (mi < re) lo_next = exp_lo(__ldg(t0s + mi), t.g);
        }
        while (mr < mi && end_r <= i) {
          const float *scr = sources(mr);
          if (scr) {
            const FF p1{scr[32 * 7], scr[32 * 8]};
            const FF p2 = ff_mul(p1, p1);
            const F2 ph0{p2.h, p2.h}, pl0{p2.l, p2.l}, nph0{-p2.h, -p2.h};
            const F2 ph1{p1.h, p1.h}, pl1{p1.l, p1.l}, nph1{-p1.h, -p1.h};
            H01 = ff2_sub_scaled_x(H01, ph0, nph0, pl0, F2{scr[0], scr[32 * 1]});
            H2 = ff_sub_scaled_x1(H2, p2, scr[32 * 2]);
            H34 = ff2_sub_scaled_x(H34, ph1, nph1, pl1, F2{scr[32 * 3], scr[32 * 4]});
            H56 = ff2_sub_scaled_x(H56, ph1, nph1, pl1, F2{scr[32 * 5], scr[32 * 6]});
          }
          mr++;
          if (mr < re) end_r = row_end(mr);
        }
      }
      if (kEnds) continue;
      // reduce the warp's columns' contributions to atom i by recursive
      // halving over 8 channel slots in double-word arithmetic: at each step a
      // lane keeps half of its slots, sends the other half to its partner and
      // adds what it receives (9 double-word additions per lane); lane L ends
      // with channel (L >> 2) & 7 summed over the warp
      const bool u16 = (lane & 16u) != 0u, u8 = (lane & 8u) != 0u, u4 = (lane & 4u) != 0u;
      const FF zf{0.0f, 0.0f};
      const FF slot[8] = {L.active ? FF{H01.h.x, H01.l.x} : zf,
                          L.active ? FF{H01.h.y, H01.l.y} : zf,
                          L.active ? H2 : zf,
                          L.active ? FF{H34.h.x, H34.l.x} : zf,
                          L.active ? FF{H34.h.y, H34.l.y} : zf,
                          L.active ? FF{H56.h.x, H56.l.x} : zf,
                          L.active ? FF{H56.h.y, H56.l.y} : zf,
                          zf};
      auto xch = [&](FF send, int d) {
        return FF{__shfl_xor_sync(0xffffffffu, send.h, d), __shfl_xor_sync(0xffffffffu, send.l, d)};
      };
      FF k4[4], k2[2];
#pragma unroll
      for (int j = 0; j < 4; j++)
        k4[j] = ff_add_dw(u16 ? slot[4 + j] : slot[j], xch(u16 ? slot[j] : slot[4 + j], 16));
#pragma unroll
      for (int j = 0; j < 2; j++)
        k2[j] = ff_add_dw(u8 ? k4[2 + j] : k4[j], xch(u8 ? k4[j] : k4[2 + j], 8));
      FF v = ff_add_dw(u4 ? k2[1] : k2[0], xch(u4 ? k2[0] : k2[1], 4));
      v = ff_add_dw(v, xch(v, 2));
      v = ff_add_dw(v, xch(v, 1));
      const uint32_t ch = (lane >> 2) & 7u;
      if ((lane & 3u) == 0u && ch < 7u && i < t.g.numAtoms) {
        const double x = (double)v.h + (double)v.l;
        if (x != 0.0) atomicAdd(grad_atoms + (t.atom_off + i) * 7u + ch, x);
      }
    }
    if (kEnds) {
      // a first segment that starts inside its atoms ends at the same atom as
      // a whole one: joins decay by r^(2^a_shift) from end to end
      float *o = ends + (size_t)as * kDiffSegFloats;
      const float v[14] = {H01.h.x, H01.h.y, H01.l.x, H01.l.y, H2.h,    H2.l,    H34.h.x,
                           H34.h.y, H34.l.x, H34.l.y, H56.h.x, H56.h.y, H56.l.x, H56.l.y};
#pragma unroll
      for (int f = 0; f < 14; f++) o[32 * f] = v[f];
    }
  }
}

// ------------------------------------------------------------ rectangular windows

// FP64 sums of aligned 32-atom blocks (8 doubles per block, 7 used).
__global__ void __launch_bounds__(256)
    rect_blocks_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                       const float *__restrict__ atoms, double *__restrict__ B64) {
  const DiffTemplate t = T[list[blockIdx.y]];
  const uint32_t w = blockIdx.x * 256u + threadIdx.x, b = w >> 3, c = w & 7u;
  if (b * 32u >= t.g.numAtoms || c == 7u) return;
  const float *x = atoms + t.atom_off * 7u + c;
  double s = 0.0;
  for (uint32_t i = b * 32u; i < min(t.g.numAtoms, b * 32u + 32u); i++)
    s += (double)__ldg(x + (size_t)i * 7u);
  B64[(t.seg_off + b) * 8u + c] = s;
}

// One warp's tile of a rectangular template: this lane's row and its window
// starts and ends.
struct RectLane {
  DiffTemplate t;
  uint32_t tile, m, nb, ne, lo;
  bool ok;
  double t0d;
  const float *x;

  // false: no such tile
  __device__ __forceinline__ bool init(const DiffTemplate *T, uint32_t k, uint32_t tl,
                                       const float *atoms, const uint32_t *t0s_all) {
    t = T[k];
    tile = tl;
    const uint32_t rg = tile / t.n_chunk;
    if (rg >= t.n_cg) return false;
    m = rg * 32u + (threadIdx.x & 31u);
    ok = m < t.N_t0;
    nb = tile % t.n_chunk * t.chunk_rows;
    ne = min(t.N_tau, nb + t.chunk_rows);
    const uint32_t t0 = __ldg(t0s_all + t.t0_off + (ok ? m : t.N_t0 - 1u));
    t0d = (double)t0;
    lo = idx_start(t0, t.g);
    x = atoms + t.atom_off * 7u;
    return true;
  }
  // rect_end_real without its division: the real end's distance from the
  // data is a sum of exact steps after t0 + tau, so its floor divided as an
  // integer is the floor of the quotient
  __device__ __forceinline__ uint32_t end(double tau) const {
    const double d = t0d + tau - (double)t.g.t0_data + (double)t.g.half;
    const uint32_t q = fdiv((uint32_t)d, t.g.div);
    return q < 1u ? 0u : min(q - 1u, t.g.numAtoms - 1u);
  }
  // cell(end) for every column of the tile; all lanes call it together
  template <class Cell>
  __device__ __forceinline__ void columns(double *s_tau, Cell &&cell) const {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t cb = nb; cb < ne; cb += 32u) {
      __syncwarp();
      if (cb + lane < ne) s_tau[lane] = tau_of(t, cb + lane);
      __syncwarp();
      const uint32_t ce = min(ne, cb + 32u);
      if (ok)
        for (uint32_t n = cb; n < ce; n++) cell(end(s_tau[n - cb]));
    }
  }
};

// Prefix rows of a row's windows (the rectangular map kernel's): FP32 F of
// the window [lo, e].
struct RectPrefix {
  const float *P;
  float row0[16];
  __device__ __forceinline__ void init(const RectLane &L, const float *P_all) {
    P = P_all + L.t.p_off * kPrefixStride;
    TCW_DCHECK(L.lo <= L.t.g.numAtoms);
    for (int c = 0; c < 16; c++) row0[c] = __ldg(P + (size_t)L.lo * kPrefixStride + c);
  }
  __device__ __forceinline__ void window(uint32_t e, FF2 W[4]) const {
    float a[16];
    const float4 *r = reinterpret_cast<const float4 *>(P + (size_t)(e + 1u) * kPrefixStride);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float4 v = __ldg(r + q);
      a[4 * q] = v.x;
      a[4 * q + 1] = v.y;
      a[4 * q + 2] = v.z;
      a[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      W[q].h = sub2(F2{a[2 * q], a[2 * q + 1]}, F2{row0[2 * q], row0[2 * q + 1]});
      W[q].l = sub2(F2{a[8 + 2 * q], a[9 + 2 * q]}, F2{row0[8 + 2 * q], row0[9 + 2 * q]});
    }
  }
  __device__ __forceinline__ static bool tier1(const FF2 W[4], float &F) {
    const F2 s0 = add2(W[0].h, W[0].l), s1 = add2(W[1].h, W[1].l);
    const F2 s2 = add2(W[2].h, W[2].l), s3 = add2(W[3].h, W[3].l);
    return fstat_fast_sums(s0.x, s0.y, s1.x, s1.y, s2.x, s2.y, s3.x, F);
  }
};

// diff_est_kernel's `need` and `est` for rectangular tiles.
__global__ void __launch_bounds__(kDiffBlock)
    rect_est_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                    const float *__restrict__ atoms, const uint32_t *__restrict__ t0s_all,
                    const float *__restrict__ P, float *__restrict__ need,
                    uint32_t *__restrict__ est) {
  __shared__ double s_tau[kDiffBlock / 32][32];
  const uint32_t k = list[blockIdx.y], wid = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  RectLane L;
  if (!L.init(T, k, blockIdx.x * (blockDim.x >> 5) + wid, atoms, t0s_all)) return;
  RectPrefix R;
  R.init(L, P);
  EstSink sink{-INFINITY, -INFINITY};
  uint32_t prev = 0xFFFFFFFFu;
  L.columns(s_tau[wid], [&](uint32_t e) {
    if (e == prev) return;  // the same window
    prev = e;
    float F = 2.0f;
    bool ok = false;
    if (e >= L.lo) {
      FF2 W[4];
      R.window(e, W);
      ok = RectPrefix::tier1(W, F);
      if (!ok) {
        FF w[7];
        ff2_unpack(W, w);
        F = fstat_ff<false, true>(w[0], w[1], w[2], w[3], w[4], w[5], w[6], ok);
      }
    }
    sink(0u, F, ok);
  });
  float top1 = sink.top, most = sink.most;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    top1 = fmaxf(top1, __shfl_xor_sync(0xffffffffu, top1, d));
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
  }
  if (lane == 0) {
    need[L.t.part_off + L.tile] = most;
    if (top1 > -INFINITY) atomicMax(est + k, float_key(top1));
  }
}

__device__ __forceinline__ void flush_diff(double *D, uint32_t row, const double v[7], double sgn,
                                           uint32_t numAtoms) {
  TCW_DCHECK(row <= numAtoms);
#pragma unroll
  for (int c = 0; c < 7; c++)
    if (v[c] != 0.0) atomicAdd(D + (size_t)row * 8u + c, sgn * v[c]);
}

// The tiles that may carry weight.  kPass 0: FP64 log-sum-exps of F and 2F/T;
// 1: the atom gradient's difference rows.  Columns with the same window count
// together.
template <int kPass>
__global__ void __launch_bounds__(kDiffBlock)
    rect_diff_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                     const float *__restrict__ atoms, const uint32_t *__restrict__ t0s_all,
                     const float *__restrict__ P, const double *__restrict__ B64,
                     const float *__restrict__ need, const uint32_t *__restrict__ est,
                     double temp, DiffPartial *__restrict__ parts,
                     const double *__restrict__ lnZ1, const double *__restrict__ lnZ2,
                     const double *__restrict__ gB, const double *__restrict__ gS,
                     double *__restrict__ D64) {
  __shared__ double s_tau[kDiffBlock / 32][32];
  const uint32_t k = list[blockIdx.y], wid = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  RectLane L;
  if (!L.init(T, k, blockIdx.x * (blockDim.x >> 5) + wid, atoms, t0s_all)) return;
  const DiffTemplate &t = L.t;
  DiffPartial *out = kPass == 0 ? parts + t.part_off + L.tile : nullptr;
  double z1 = 0.0, z2 = 0.0, gb = 0.0, gs = 0.0;
  float skip0;
  if (kPass == 0) {
    skip0 = FwdBounds(est[k], temp).skip;
  } else {  // a cell whose weights are below e^-62 in both sums has no gradient
    z1 = lnZ1[k] - log(70.0 / ((double)t.N_t0 * (double)t.N_tau));
    z2 = lnZ2[k] / temp;
    gb = gB[k];
    gs = gS[k];
    skip0 = (float)fmin(gb != 0.0 ? z1 - 1e-5 * fabs(z1) - 63.0 : INFINITY,
                        gs != 0.0 ? 0.5 * temp * (z2 - 1e-5 * fabs(z2) - 62.0) - 1.0 : INFINITY);
  }
  if (need[t.part_off + L.tile] < skip0) {
    if (kPass == 0 && lane == 0) *out = DiffPartial{-INFINITY, 0.0, -INFINITY, 0.0};
    return;
  }
  RectPrefix R;
  R.init(L, P);
  const double *B = B64 + t.seg_off * 8u;
  double *D = kPass == 1 ? D64 + t.p_off * 8u : nullptr;
  DiffLse lse(temp, skip0);
  double S[7] = {0, 0, 0, 0, 0, 0, 0}, Rs[7] = {0, 0, 0, 0, 0, 0, 0};
  uint32_t next = L.lo, prev = 0xFFFFFFFFu, count = 0;
  bool weighs = false;   // the current window carries weight
  F64Cell fc{2.0, 0.0, false};
  // the columns of the current window, all at once
  auto finish = [&]() {
    if (!weighs || count == 0u) return;
    if (kPass == 0) {
      lse.add(fc.F, (double)count);
    } else {
      // dL/dF of the cells (FP32 exponentials: relative 1e-7 on a gradient term)
      const double F = fc.F;
      double g = gb * (double)exp2f((float)(F - z1) * kLog2eF) +
                 gs * 2.0 * (double)exp2f((float)(2.0 * F / temp - z2) * kLog2eF);
      if (g == 0.0) return;
      g *= (double)count;
      const double A = S[0], B2 = S[1], C = S[2], iD = fc.iD;
      const double Fa2 = S[3] * S[3] + S[4] * S[4], Fb2 = S[5] * S[5] + S[6] * S[6];
      const double re = S[3] * S[5] + S[4] * S[6];
      double G[7];
      G[0] = (Fb2 - F * B2) * iD;
      G[1] = (Fa2 - F * A) * iD;
      G[2] = (2.0 * F * C - 2.0 * re) * iD;
      G[3] = 2.0 * (B2 * S[3] - C * S[5]) * iD;
      G[4] = 2.0 * (B2 * S[4] - C * S[6]) * iD;
      G[5] = 2.0 * (A * S[5] - C * S[3]) * iD;
      G[6] = 2.0 * (A * S[6] - C * S[4]) * iD;
#pragma unroll
      for (int c = 0; c < 7; c++) {
        G[c] *= g;
        Rs[c] += G[c];
      }
      flush_diff(D, prev + 1u, G, -1.0, t.g.numAtoms);
    }
  };
  L.columns(s_tau[wid], [&](uint32_t e) {
    if (e == prev) {
      count++;
      return;
    }
    finish();
    prev = e;
    count = 1u;
    if (e < L.lo) {  // no atoms: F = 2, no gradient
      fc = F64Cell{2.0, 0.0, false};
      weighs = kPass == 0 && !(2.0f < lse.skip);
      return;
    }
    FF2 W[4];
    float F32 = 0.0f;
    R.window(e, W);
    const bool t1 = RectPrefix::tier1(W, F32);
    weighs = !(t1 && F32 < lse.skip);
    if (!weighs) return;
    while (next <= e) {
      TCW_DCHECK(next < t.g.numAtoms);
      if ((next & 31u) == 0u && next + 31u <= e) {
#pragma unroll
        for (int c = 0; c < 7; c++) S[c] += __ldg(B + (size_t)(next >> 5) * 8u + c);
        next += 32u;
      } else {
#pragma unroll
        for (int c = 0; c < 7; c++) S[c] += (double)__ldg(L.x + (size_t)next * 7u + c);
        next++;
      }
    }
    fc = fstat64(S, t1);
    if (kPass == 1 && !fc.ok) weighs = false;
  });
  if (L.ok) finish();
  if (kPass == 0) {
    const DiffPartial p = lse.merge();
    if (lane == 0) *out = p;
  } else if (L.ok) {
    flush_diff(D, L.lo, Rs, 1.0, t.g.numAtoms);
  }
}

// dL/dx(i) = sum_{j <= i} D(j) for i < numAtoms, one block per rectangular
// template: per-thread chunk sums, an exclusive scan of the chunk sums, then
// each chunk written in order.
constexpr int kScanBlock = 256;

__global__ void __launch_bounds__(kScanBlock)
    rect_diff_scan_kernel(const DiffTemplate *__restrict__ T, const uint32_t *__restrict__ list,
                          const double *__restrict__ D64, double *__restrict__ grad_atoms) {
  __shared__ double sh[kScanBlock / 32][7];
  const DiffTemplate t = T[list[blockIdx.x]];
  const uint32_t n = t.g.numAtoms, lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  const double *D = D64 + t.p_off * 8u;
  const uint32_t chunk = (n + kScanBlock - 1u) / kScanBlock;
  const uint32_t a0 = min(n, threadIdx.x * chunk), a1 = min(n, a0 + chunk);
  double s[7] = {0, 0, 0, 0, 0, 0, 0};
  for (uint32_t i = a0; i < a1; i++)
#pragma unroll
    for (int c = 0; c < 7; c++) s[c] += D[(size_t)i * 8u + c];
  // exclusive scan of the chunk sums: within the warp, then over the warps
  double run[7];
#pragma unroll
  for (int c = 0; c < 7; c++) {
    double v = s[c];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double o = __shfl_up_sync(0xffffffffu, v, d);
      if (lane >= (uint32_t)d) v += o;
    }
    if (lane == 31u) sh[wid][c] = v;
    const double ex = __shfl_up_sync(0xffffffffu, v, 1);
    run[c] = lane ? ex : 0.0;
  }
  __syncthreads();
  for (uint32_t w = 0; w < wid; w++)
#pragma unroll
    for (int c = 0; c < 7; c++) run[c] += sh[w][c];
  for (uint32_t i = a0; i < a1; i++) {
#pragma unroll
    for (int c = 0; c < 7; c++) {
      run[c] += D[(size_t)i * 8u + c];
      grad_atoms[(t.atom_off + i) * 7u + c] = run[c];
    }
  }
}

// One block per template: its partials brought to their maximum and added
// (one warp: 33 us for the 2048 partials of a lone template, now 8), one warp
// where there are few, as the FP64 maxima and sums of idle warps cost as much as
// theirs (2000 templates of 4 x 4 cells 73 us by eight warps each).
__global__ void __launch_bounds__(256)
    diff_finalize_kernel(const DiffTemplate *__restrict__ T, const DiffPartial *__restrict__ parts,
                         double temp, double *__restrict__ lnB, double *__restrict__ soft) {
  __shared__ DiffPartial sh[8];
  const uint32_t k = blockIdx.x, lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  const uint32_t warps = blockDim.x >> 5;
  const DiffTemplate t = T[k];
  DiffPartial a{-INFINITY, 0.0, -INFINITY, 0.0};
  for (uint32_t p = threadIdx.x; p < t.n_parts; p += blockDim.x) {
    a.m1 = fmax(a.m1, parts[t.part_off + p].m1);
    a.m2 = fmax(a.m2, parts[t.part_off + p].m2);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    a.m1 = fmax(a.m1, __shfl_xor_sync(0xffffffffu, a.m1, d));
    a.m2 = fmax(a.m2, __shfl_xor_sync(0xffffffffu, a.m2, d));
  }
  if (lane == 0) sh[wid] = a;
  __syncthreads();
  for (uint32_t w = 0; w < warps; w++) {
    a.m1 = fmax(a.m1, sh[w].m1);
    a.m2 = fmax(a.m2, sh[w].m2);
  }
  for (uint32_t p = threadIdx.x; p < t.n_parts; p += blockDim.x) {
    const DiffPartial q = parts[t.part_off + p];
    if (q.s1 != 0.0) a.s1 += q.s1 * exp(q.m1 - a.m1);
    if (q.s2 != 0.0) a.s2 += q.s2 * exp(q.m2 - a.m2);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    a.s1 += __shfl_xor_sync(0xffffffffu, a.s1, d);
    a.s2 += __shfl_xor_sync(0xffffffffu, a.s2, d);
  }
  __syncthreads();  // every thread has read the maxima
  if (lane == 0) sh[wid] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s1 = 0.0, s2 = 0.0;
    for (uint32_t w = 0; w < warps; w++) {
      s1 += sh[w].s1;
      s2 += sh[w].s2;
    }
    lnB[k] = log(70.0 / ((double)t.N_t0 * (double)t.N_tau)) + a.m1 + log(s1);
    soft[k] = temp * (a.m2 + log(s2));
  }
}

}  // namespace

// `side`: a second stream for diff_hot_kernel, whose few long blocks run beside
// the tiles that need no whole walk; fork and join are the caller's events.
cudaError_t launch_diff(int pass, const DiffLaunch &L, const DiffGroup *groups, uint32_t n_groups,
                        const DiffClass *classes, cudaStream_t stream, cudaStream_t side,
                        cudaEvent_t fork, cudaEvent_t join) {
  cudaError_t e = cudaSuccess;
  if (L.n_exp) {
    e = cudaFuncSetAttribute(pass == 0 ? (const void *)diff_hot_kernel<false>
                                       : (const void *)diff_hot_kernel<true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kHotAtoms * 28u));
    if (e != cudaSuccess) return e;
    for (uint32_t q = 0; q < n_groups; q++) {
      const DiffGroup &g = groups[q];
      const DiffClass *c0 = classes + g.c0, *c1 = c0 + g.n_classes;
      // atoms that diff_hot_kernel stages in shared memory (28 bytes each)
      const uint32_t smem_atoms = g.max_atoms < kHotAtoms ? g.max_atoms : kHotAtoms;
      auto warps = [](const DiffClass *c, uint32_t n) { return dim3((n + 3u) / 4u, c->ny); };
      for (const DiffClass *c = c0; c < c1; c++) {
        const uint32_t atom_blocks = (c->max_atoms + 255u) / 256u;
        diff_prep_kernel<<<dim3(atom_blocks + (c->max_cols + 255u) / 256u, c->ny), 256, 0,
                           stream>>>(L.T, L.exp_list + c->y0, atom_blocks, L.atoms, L.atoms8,
                                     L.cols);
      }
      for (const DiffClass *c = c0; c < c1; c++)
        if (c->max_segs)
          diff_seg_kernel<false><<<warps(c, c->max_segs), kDiffBlock, 0, stream>>>(
              L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, nullptr, nullptr, L.temp, nullptr,
              nullptr, nullptr, nullptr, g.seg_per, L.seg);
      for (const DiffClass *c = c0; c < c1; c++)
        if (c->est_tiles)
          diff_est_kernel<<<warps(c, c->est_tiles), kDiffBlock, 0, stream>>>(
              L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.seg, L.need, L.est);
      // (one slice unless the group is one large template in its backward pass)
      for (uint32_t cg0 = 0; cg0 < g.max_cg; cg0 += g.cg_slice) {
        const uint32_t cgs = g.max_cg - cg0 < g.cg_slice ? g.max_cg - cg0 : g.cg_slice;
        const dim3 hot(cgs, g.ny);
        const HotRoute route{g.hot > 2u * L.n_sms ? L.hot_groups + q : nullptr, 2u * L.n_sms};
        if (g.hot) {
          if (route.groups && cg0 == 0) {
            const dim3 all((g.max_cg + kDiffBlock - 1u) / kDiffBlock, g.ny);
            if (pass == 0)
              diff_route_kernel<false><<<all, kDiffBlock, 0, stream>>>(
                  L.T, L.exp_list + g.y0, L.need, L.est, L.temp, nullptr, nullptr, nullptr,
                  nullptr, L.hot_groups + q);
            else
              diff_route_kernel<true><<<all, kDiffBlock, 0, stream>>>(
                  L.T, L.exp_list + g.y0, L.need, L.est, L.temp, L.lnZ1, L.lnZ2, L.gB, L.gS,
                  L.hot_groups + q);
          }
          if ((e = cudaEventRecord(fork, stream)) != cudaSuccess ||
              (e = cudaStreamWaitEvent(side, fork, 0)) != cudaSuccess)
            return e;
          if (pass == 0)
            diff_hot_kernel<false><<<hot, kHotThreads, (size_t)smem_atoms * 28u, side>>>(
                L.T, L.exp_list + g.y0, L.atoms8, L.t0s, L.cols, L.need, L.est, L.temp, nullptr,
                nullptr, nullptr, nullptr, cg0, nullptr, nullptr, L.parts, smem_atoms, route);
          else
            diff_hot_kernel<true><<<hot, kHotThreads, (size_t)smem_atoms * 28u, side>>>(
                L.T, L.exp_list + g.y0, L.atoms8, L.t0s, L.cols, L.need, L.est, L.temp, L.lnZ1,
                L.lnZ2, L.gB, L.gS, cg0, L.scratch, L.grad_tau, nullptr, smem_atoms, route);
          for (const DiffClass *c = c0; route.groups && c < c1; c++) {
            if (pass == 0)
              diff_fwd_kernel<true><<<warps(c, c->slice_cg), kDiffBlock, 0, side>>>(
                  L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.seg, L.need, L.est, L.temp,
                  L.parts, route);
            else
              diff_src_kernel<true><<<warps(c, c->slice_cg), kDiffBlock, 0, side>>>(
                  L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.seg, L.need, L.est, L.temp,
                  L.lnZ1, L.lnZ2, L.gB, L.gS, cg0, cgs, L.scratch, L.grad_tau, route);
          }
        }
        if (pass == 0) {
          for (const DiffClass *c = c0; c < c1; c++)
            diff_fwd_kernel<false><<<warps(c, c->max_tiles), kDiffBlock, 0, stream>>>(
                L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.seg, L.need, L.est, L.temp,
                L.parts, route);
        } else {
          for (const DiffClass *c = c0; c < c1; c++)
            if (c->max_segs && cg0 == 0)  // (over the window sums, which nothing reads any more)
              diff_seg_kernel<true><<<warps(c, c->max_segs), kDiffBlock, 0, stream>>>(
                  L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.need, L.est, L.temp, L.lnZ1,
                  L.lnZ2, L.gB, L.gS, g.seg_per, L.seg);
          for (const DiffClass *c = c0; c < c1; c++)
            diff_src_kernel<false><<<warps(c, c->slice_tiles), kDiffBlock, 0, stream>>>(
                L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.seg, L.need, L.est, L.temp,
                L.lnZ1, L.lnZ2, L.gB, L.gS, cg0, cgs, L.scratch, L.grad_tau, route);
        }
        if (g.hot && ((e = cudaEventRecord(join, side)) != cudaSuccess ||
                      (e = cudaStreamWaitEvent(stream, join, 0)) != cudaSuccess))
          return e;
        if (pass == 1) {
          for (const DiffClass *c = c0; c < c1; c++)
            if (c->slice_ends)
              diff_atoms_kernel<true><<<warps(c, c->slice_ends), kDiffBlock, 0, stream>>>(
                  L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.need, L.est, L.temp, L.lnZ1,
                  L.lnZ2, L.gB, L.gS, cg0, cgs, L.scratch, L.cend, L.grad_atoms);
          for (const DiffClass *c = c0; c < c1; c++)
            diff_atoms_kernel<false><<<warps(c, c->slice_aseg), kDiffBlock, 0, stream>>>(
                L.T, L.exp_list + c->y0, L.atoms8, L.t0s, L.cols, L.need, L.est, L.temp, L.lnZ1,
                L.lnZ2, L.gB, L.gS, cg0, cgs, L.scratch, L.cend, L.grad_atoms);
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
      }
    }
  }
  for (uint32_t y0 = 0; y0 < L.n_rect; y0 += 65535u) {
    const uint32_t ny = L.n_rect - y0 < 65535u ? L.n_rect - y0 : 65535u;
    const uint32_t *list = L.rect_list + y0;
    // four tiles per block, fewer where templates have fewer: warps without a tile
    // keep their registers until the block ends (1000 templates of 480 atoms, 32 x
    // 32 cells in one tile each 0.86 / 1.02 -> 0.71 / 0.81 ms)
    const uint32_t warps = L.max_rect_tiles < 4u ? L.max_rect_tiles : 4u, threads = warps * 32u;
    const dim3 tiles((L.max_rect_tiles + warps - 1u) / warps, ny);
    const dim3 blocks((L.max_rect_atoms + 1023u) / 1024u, ny);  // 32 blocks of 32 atoms each
    if (y0 == 0) {
      e = launch_prefix(L.rect_T, L.rect_ident, L.n_rect, L.atoms, L.P, kPrecFF, stream);
      if (e != cudaSuccess) return e;
    }
    rect_blocks_kernel<<<blocks, 256, 0, stream>>>(L.T, list, L.atoms, L.B64);
    rect_est_kernel<<<tiles, threads, 0, stream>>>(L.T, list, L.atoms, L.t0s, L.P, L.need,
                                                      L.est);
    if (pass == 0) {
      rect_diff_kernel<0><<<tiles, threads, 0, stream>>>(
          L.T, list, L.atoms, L.t0s, L.P, L.B64, L.need, L.est, L.temp, L.parts, nullptr, nullptr,
          nullptr, nullptr, nullptr);
    } else {
      rect_diff_kernel<1><<<tiles, threads, 0, stream>>>(
          L.T, list, L.atoms, L.t0s, L.P, L.B64, L.need, L.est, L.temp, nullptr, L.lnZ1, L.lnZ2,
          L.gB, L.gS, L.D64);
      rect_diff_scan_kernel<<<ny, kScanBlock, 0, stream>>>(L.T, list, L.D64, L.grad_atoms);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_diff_finalize(const DiffTemplate *T, uint32_t n_templates, uint32_t max_parts,
                                 const DiffPartial *parts, double temp, double *lnB, double *soft,
                                 cudaStream_t stream) {
  if (n_templates == 0) return cudaSuccess;
  const uint32_t threads = max_parts <= 64u ? 32u : 256u;
  diff_finalize_kernel<<<n_templates, threads, 0, stream>>>(T, parts, temp, lnB, soft);
  return cudaGetLastError();
}

}  // namespace tcw

namespace tcw {
// Failed debug checks of this file's kernels (0 unless built with TCW_DEBUG_CHECKS).
unsigned int dcheck_failures_diff() {
#if defined(TCW_DEBUG_CHECKS)
  return tcw_dcheck_read();
#else
  return 0;
#endif
}
}  // namespace tcw
