// Internal device-side data structures shared by the kernels and the C-ABI
// layer.  Not part of the public interface (include/tcw_b200.h).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tcw_b200.h"
#include "tcw_cell.h"

namespace tcw {

constexpr int kBlock = 128;  // threads per map block

enum PrecisionMode : int {
  kPrecFF = 0,        // double-word window sums, FP32 error-free D (default)
  kPrecFF_F64Det = 1, // double-word window sums, native FP64 D
  kPrecPlain32 = 2,   // uncompensated FP32 (precision report only)
};

// One template as the kernels see it.  Offsets index the concatenated
// arrays of a call: atoms in rows of 7 floats, grids in u32 entries, prefix
// rows of 16 floats, the output map in floats, per-item partials.
struct TemplateDev {
  uint64_t atom_off;
  uint64_t t0_off;
  uint64_t tau_off;
  uint64_t p_off;
  uint64_t a8_off;  // exp templates: first row in the 8-float atom rows
  uint64_t map_off;
  Geom g;
  uint32_t window;  // 1 rect, 2 exp
  uint32_t N_t0, N_tau;
  uint32_t part_off, n_parts;
  uint32_t pad;
  uint64_t row_off, col_off;  // posterior row and column sums (PostLayout)
  // exp templates whose columns are cut into row chunks: segment sums of
  // 2^g_shift atoms (exp_seg_kernel), g_nseg segments per 32-column group
  // (0: none), starting at float g_off * kSegFloats
  uint64_t g_off;
  uint32_t g_shift, g_nseg;
  uint32_t e_hist, e_rows, e_sub;  // row chunks (ExpSplit)
  // single-template launches: tiles of tile_tn columns x tile_tm rows (rect)
  // or row chunks (exp), row tiles fastest (plain_tile)
  uint32_t tile_tn, tile_tm, tile_rows;  // tile_rows: row tiles per column tile
  double ln_prior;                 // ln(70 / (N_t0 N_tau))
};
// Floats of one 32-column segment sum (7 channels x hi, lo x 32 lanes).
constexpr uint32_t kSegFloats = 14u * 32u;
// Segments of one warp of exp_seg_kernel: up to 4 amortise the column's FP64
// exp, fewer where that leaves resident warps (32 per SM) without one (480
// atoms x 512 columns: 4 per warp 22.8 us; 24 templates: 24 -> 16 us).
inline uint32_t segs_per_warp(uint64_t segments, int n_sms) {
  const uint64_t per = segments / ((uint64_t)n_sms * 32u);
  return per < 1 ? 1u : (per > 4 ? 4u : (uint32_t)per);
}

// A tile of one template, rows [m0, m1) x columns [n0, n1).  Rectangular: tn
// groups of 32 rows.  Exponential: 32 columns, walked by one warp (within one
// history).
struct WorkItem {
  uint32_t tmpl;
  uint32_t part;
  uint32_t m0, m1;
  uint32_t n0, n1;
  uint16_t tn;            // rect: row groups; exp: columns (32)
  uint16_t pad16;
  uint32_t pad;
};

// Segments [j0, j1) of 32-column group cg of one exp template.
struct SegItem {
  uint32_t tmpl, cg, j0, j1;
};

// How an exp template's columns are cut into row chunks.  `hist` rows are one
// history: a window's sums keep the roundings of the rows above it in the
// same history and start afresh at the next one.  Each history is walked in
// `sub` chunks of `rows` rows, side by side, whose starts are combined from
// nseg segment sums of 2^shift atoms (0: every chunk enters its whole window
// atom by atom, sub is 1).
struct ExpSplit {
  uint32_t hist, rows, sub, shift, nseg;
  uint32_t chunks(uint32_t N_t0) const { return (N_t0 + hist - 1u) / hist * sub; }
  uint64_t seg_floats(uint32_t N_tau) const {
    return (uint64_t)((N_tau + 31u) / 32u) * nseg * kSegFloats;
  }
};
constexpr uint64_t kSegBytesMax = 1ull << 30;
// Windows of fewer atoms have a history that F shows (a near-singular F
// amplifies the roundings that Fast2Sum leaves in Fa and Fb by up to
// 2 sqrt(1e4)): a chunk whose columns have such windows starts kRunUp tau
// earlier, where a rounding's weight is below e^-12 and F is that of the whole
// history (without the run-up maxF of ~2 % of the benchmark's exp templates
// moved by up to 2e-7; with 64 atoms and 18 tau the run-up was as long as
// the chunks: 406 against 227 us per run of 24 templates of up to 1500 atoms).
constexpr uint32_t kShortWindow = 32;
constexpr uint32_t kRunUp = 12;

// At least `chunks` chunks per column where histories allow it (8 rows or
// more each).  Segments of about sqrt(numAtoms) atoms: a chunk start costs up
// to 2 x 2^shift entering steps and numAtoms / 2^shift joins.
inline ExpSplit exp_split(uint32_t numAtoms, uint32_t N_t0, uint32_t N_tau, uint32_t hist,
                          uint64_t chunks) {
  ExpSplit s{hist, hist, 1, 5, 0};
  const uint64_t n_hist = (N_t0 + hist - 1u) / hist;
  const uint64_t sub = (chunks + n_hist - 1) / n_hist;
  if (chunks <= 1 || numAtoms < 2u * kShortWindow) return s;
  const uint64_t rows = (hist + sub - 1) / sub;
  s.rows = rows < 8 ? 8u : (uint32_t)rows;
  s.sub = (hist + s.rows - 1u) / s.rows;
  while ((4ull << (2u * s.shift)) <= numAtoms) s.shift++;
  s.nseg = (uint32_t)(((uint64_t)numAtoms + (1u << s.shift) - 1u) >> s.shift);
  if (n_hist * s.sub <= 1 || s.seg_floats(N_tau) * sizeof(float) > kSegBytesMax)
    return ExpSplit{hist, hist, 1, 5, 0};
  return s;
}

// Row chunks of a single-template exp map: 16 histories per column, cut
// further (`cut`) until there are about TCW_PLAIN_EXP_WARPS warps per
// scheduler (one-year 8192 x 4096 map, whole call: 4 warps 908 us, 6 762 us,
// 8 687 us, 12 709 us).
#ifndef TCW_PLAIN_EXP_WARPS
#define TCW_PLAIN_EXP_WARPS 8
#endif
inline ExpSplit plain_exp_split(uint32_t numAtoms, uint32_t N_t0, uint32_t N_tau, int n_sms,
                                bool cut) {
  uint32_t hist = (N_t0 + 15u) / 16u;
  hist = hist < 8u ? 8u : hist;
  hist = hist < N_t0 ? hist : N_t0;
  hist = hist < 65535u ? hist : 65535u;
  const uint64_t groups = (N_tau + 31u) / 32u;
  const uint64_t want = (uint64_t)n_sms * 4u * TCW_PLAIN_EXP_WARPS;
  return exp_split(numAtoms, N_t0, N_tau, hist, cut ? (want + groups - 1u) / groups : 1u);
}

// Whether a single map's tiles are launched as the dependent of the kernel
// before (prepare or segment sums): where that one leaves most of the GPU
// idle.  Tiles that arrive while thousands of segment blocks still run settle
// on the SMs that happen to be free (one-year exp map 650 -> 760 us); behind
// the eight blocks of a prefix scan they save the launch (one-year rect map
// 250 -> 233 us, 480 x 480 53 -> 29 us per call with the other launches).
inline bool plain_map_chained(uint32_t n_seg_items, uint32_t numAtoms, int n_sms) {
  const uint32_t before = n_seg_items ? (n_seg_items + 3u) / 4u : (numAtoms + 255u) / 256u;
  return before <= (uint32_t)n_sms;
}

// Tiles of a single-template map (tile_tn, tile_tm, tile_rows); the number of
// tiles, each one block.  Rect: 32 rows x as many columns as give ~4 blocks per
// SM, 16 to 256 (at least 4 per warp).  Exp: 32 columns x 4 row chunks (a warp
// each), t.e_* set.
inline uint64_t plain_tiles(TemplateDev &t, int n_sms) {
  if (t.window == 1u) {
    t.tile_tm = 32;
    t.tile_rows = (t.N_t0 + 31u) / 32u;
    const uint64_t c = (uint64_t)t.N_tau * t.tile_rows / ((uint64_t)n_sms * 4u);
    t.tile_tn = (uint32_t)(c < 16 ? 16 : (c > 256 ? 256 : c));
  } else {
    t.tile_tn = 32;
    t.tile_tm = kBlock / 32;
    const uint32_t chunks = (t.N_t0 + t.e_hist - 1u) / t.e_hist * t.e_sub;
    t.tile_rows = (chunks + t.tile_tm - 1u) / t.tile_tm;
  }
  return (uint64_t)t.tile_rows * (((uint64_t)t.N_tau + t.tile_tn - 1u) / t.tile_tn);
}

inline void set_split(TemplateDev &t, const ExpSplit &sp) {
  t.e_hist = sp.hist;
  t.e_rows = sp.rows;
  t.e_sub = sp.sub;
  t.g_shift = sp.shift;
  t.g_nseg = sp.nseg;
}

// Per-item reduction result.  s = sum over the item's cells of exp(F - maxF).
struct Partial {
  float maxF;
  uint32_t pad;
  int64_t argmax;  // flat m*N_tau + n, smallest index among ties
  double s;
};

#if defined(__CUDACC__)
// 256 of one template's atoms from i0 on (rows of 7 floats, x) into 32-byte
// rows [a2 b2 ab nz Fa_re Fa_im Fb_re Fb_im] (o), by a block of 256 threads,
// one atom each; nz (as u32 bits) is the lowest atom index >= i with a2 or b2
// non-zero (0xFFFFFFFF: none), from the warps' ballots and, past the block's
// atoms, a search upwards 256 at a time (one step unless a gap is that long).
// (One block walking all atoms: 46 us for 17532 atoms.)
__device__ __forceinline__ void repack_rows(const float *__restrict__ x, float4 *__restrict__ o,
                                            uint32_t N, uint32_t i0) {
  __shared__ uint32_t s_mask[8];
  if (i0 >= N) return;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5, i = i0 + tid;
  float r[7] = {0, 0, 0, 0, 0, 0, 0};
  if (i < N)
    for (int c = 0; c < 7; c++) r[c] = __ldg(x + (size_t)i * 7u + c);
  const uint32_t mine = __ballot_sync(0xffffffffu, r[0] != 0.0f || r[1] != 0.0f);
  if (lane == 0) s_mask[wid] = mine;
  __syncthreads();
  uint32_t nz = 0xFFFFFFFFu;
  const uint32_t here = mine >> lane;
  if (here) {
    nz = i + __ffs(here) - 1u;
  } else {
    for (uint32_t w = wid + 1u; w < 8u; w++)
      if (s_mask[w]) {
        nz = i0 + w * 32u + __ffs(s_mask[w]) - 1u;
        break;
      }
  }
  // the lanes without one look above the block (all threads take part)
  bool search = __syncthreads_or(i < N && nz == 0xFFFFFFFFu) != 0;
  for (uint32_t base = i0 + 256u; search && base < N; base += 256u) {
    const uint32_t j = base + tid;
    const bool hit = j < N && (__ldg(x + (size_t)j * 7u) != 0.0f ||
                               __ldg(x + (size_t)j * 7u + 1) != 0.0f);
    const uint32_t m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) s_mask[wid] = m;
    if (__syncthreads_or(hit)) {
      if (nz == 0xFFFFFFFFu)
        for (uint32_t w = 0; w < 8u; w++)
          if (s_mask[w]) {
            nz = base + w * 32u + __ffs(s_mask[w]) - 1u;
            break;
          }
      search = false;
    }
  }
  if (i < N) {
    o[2u * i] = make_float4(r[0], r[1], r[2], __uint_as_float(nz));
    o[2u * i + 1u] = make_float4(r[3], r[4], r[5], r[6]);
  }
}
#endif

// Launchers (tcw_kernels.cu).  All asynchronous on `stream`.
cudaError_t launch_prefix(const TemplateDev *d_T, const uint32_t *d_rect_list, uint32_t n_rect,
                          const float *d_atoms, float *d_P, int prec, cudaStream_t stream);
// The first kernel of a single-template map: prefix rows (rect) or repacked
// rows (exp) of `t`, which it leaves at d_T for the launches that follow (no
// control data is uploaded).
cudaError_t launch_prepare_one(const TemplateDev &t, TemplateDev *d_T, const float *d_atoms,
                               float *d_rows, int prec, cudaStream_t stream);
// Exp templates' atoms (rows of 7 floats) into rows of 8 (repack_rows);
// max_atoms: the most atoms of one of them.
cudaError_t launch_repack(const TemplateDev *d_T, const uint32_t *d_exp_list, uint32_t n_exp,
                          uint32_t max_atoms, const float *d_atoms, float *d_atoms8,
                          cudaStream_t stream);
// Segment sums of exp templates (the chunk starts of exp tiles are combined
// from them): items == NULL means template 0's columns and segments, with
// n_items = column groups x ceil(segments / per).
cudaError_t launch_exp_segments(const TemplateDev *d_T, const SegItem *d_items, uint32_t n_items,
                                uint32_t per, const float *d_atoms8, const uint32_t *d_taus, float *d_G,
                                cudaStream_t stream);
struct MapLaunch {
  const TemplateDev *T;
  const WorkItem *items;  // this window's tiles (persistent launches)
  uint32_t n_items;
  uint32_t *counter;      // persistent launches: tile counter, zeroed before
  uint32_t n_blocks;      // persistent grid size
  bool persistent, write_map;
  bool chunks;            // persistent exp launches: some columns are cut (e_sub > 1)
  int prec;
  int priority;           // stream-priority value of a persistent launch
  bool chained;           // single maps: programmatic dependent of the launch before
  const float *atoms;
  const float *atoms8;    // exp tiles: atoms in 32-byte rows
  const float *G;         // exp tiles: segment sums (NULL where no template has any)
  const uint32_t *t0s, *taus;
  const float *P;
  float *Fmn;
  Partial *parts;
};
cudaError_t launch_map(int window, const MapLaunch &L, cudaStream_t stream);
// Resident blocks per SM of the persistent (map-less) kernel of a window.
int map_blocks_per_sm(int window, int prec, bool chunks);

// `chained` (finalize, posteriors): part of a single map's chain of programmatic
// dependent launches.
cudaError_t launch_finalize(const TemplateDev *d_T, uint32_t n_templates, const Partial *d_parts,
                            void *d_results, bool chained, cudaStream_t stream);
// Posterior indices of templates whose maps were written: blocks of `rows`
// t0 rows x `cols` columns (a multiple of 1024) leave row sums per column
// chunk (rowsum + row_off + chunk * N_t0) and column sums per row chunk
// (colsum + col_off + chunk * N_tau); up to kPostParts blocks per template and
// direction then leave their first maximum in `parts`.
constexpr uint32_t kPostParts = 32;
struct PostPart {
  int64_t v, i;  // the sum's key (its bits: sums are >= 0) and index
};
struct PostLayout {
  uint32_t rows, cols, n_chunks;
  uint32_t argmax_blocks;  // blocks per template, up to the most parts of one (post_parts)
  const uint2 *chunks;  // (template, chunk); NULL: template 0's chunks
  double *rowsum, *colsum;
  PostPart *parts;      // 2 kPostParts per template
  uint32_t *ticket;     // one per template
};
#if defined(__CUDACC__)
__host__ __device__
#endif
inline uint32_t post_part_entries(uint32_t n) {
  const uint32_t e = (n + kPostParts - 1u) / kPostParts;
  return e < 256u ? 256u : e;
}
// Parts of one template: those of its rows, then those of its columns.
inline uint32_t post_parts(uint32_t N_t0, uint32_t N_tau) {
  const uint32_t r = post_part_entries(N_t0), c = post_part_entries(N_tau);
  return (uint32_t)(((uint64_t)N_t0 + r - 1u) / r + ((uint64_t)N_tau + c - 1u) / c);
}
// Rows per block for maps of `cells` cells in all: 256, fewer where that
// leaves fewer than 8 blocks per SM, 16 at least.
inline uint32_t post_rows(uint64_t cells, int n_sms) {
  uint32_t rows = 256;
  while (rows > 16u && cells / ((uint64_t)rows * 1024u) < (uint64_t)n_sms * 8u) rows >>= 1;
  return rows;
}
cudaError_t launch_posteriors(const TemplateDev *d_T, uint32_t n_templates, const PostLayout &L,
                              const float *d_maps, tcw_result *d_results, bool chained,
                              cudaStream_t stream);

// ---------------------------------------------------------------- differentiable path
// One template with a continuous tau grid (tcw_diff.cu).  Exponential
// templates are tiled by 32 tau columns x chunk_rows t0 rows (n_cg x n_chunk
// tiles, tile = cg * n_chunk + chunk), rectangular ones by 32 t0 rows x
// chunk_rows tau columns (n_cg row groups, n_chunk column chunks); these own
// (numAtoms + 1) prefix rows at p_off, as many difference rows of their atom
// gradient in the backward pass, and FP64 block sums at seg_off.
struct DiffTemplate {
  uint64_t atom_off, t0_off;
  Geom g;
  uint32_t N_t0, N_tau;
  double tau_min, tau_max;
  uint32_t part_off, n_parts;  // this template's tiles (need, partials)
  uint32_t window;
  uint32_t whole;  // its tiles are whole columns, none walked apart: kDiffWhole, kDiffWholeBlind
  uint64_t p_off;
  uint32_t n_cg, n_chunk, chunk_rows;
  uint32_t g_shift, g_nseg;          // segment sums
  uint32_t n_aseg, a_shift;          // segments of 2^a_shift atoms of the transposed recurrence
  uint64_t col_off;   // column constants
  uint64_t seg_off;   // segment sums, in 32-lane blocks of one segment
  uint64_t scr_off;   // backward: adjoint sources, in floats
  uint64_t cend_off;  // backward: recurrence ends, in 32-lane blocks
};
// Adjoint sources of one cell in the backward pass's scratch (7 channels and
// r^L as a float pair), least atoms per segment of the transposed recurrence and
// most segments (a segment joins the ends of all below it).
#define TCW_DIFF_SLOTS 9u
constexpr uint32_t kDiffAtomShift = 6u, kDiffAtomSeg = 1u << kDiffAtomShift;
constexpr uint32_t kDiffMaxAseg = 4096u;
// DiffTemplate::whole: with an estimate, without one.
constexpr uint32_t kDiffWhole = 1u, kDiffWholeBlind = 2u;
// Floats of one 32-column segment: window sums (forward), with their
// tau derivatives (backward).
constexpr uint32_t kDiffSegFloats = 14u * 32u;
constexpr uint32_t kDiffSegFloatsV = 28u * 32u;

struct DiffPartial {
  double m1, s1, m2, s2;
};
// Exponential templates [y0, y0 + ny) of exp_list (largest first) whose tiles
// one launch takes, as a grid of the most that one of them has x ny.
struct DiffClass {
  uint32_t y0, ny;
  // most tiles / segments / atoms / columns of one template
  uint32_t max_tiles, max_segs, max_atoms, max_cols;
  uint32_t slice_tiles, slice_aseg;  // most tiles / atom segments in a slice
  uint32_t slice_cg;                 // most column groups in a slice
  // most tiles that are estimated, most atom segments that leave their ends
  uint32_t est_tiles, slice_ends;
};
// Exponential templates [y0, y0 + ny) of exp_list with workspaces of their
// own: a backward pass runs in groups that bound the scratch, a group of one
// large template in slices of cg_slice column groups.  Its launches go by
// classes [c0, c0 + n_classes).
struct DiffGroup {
  uint32_t y0, ny, c0, n_classes;
  uint32_t max_cg, max_atoms;  // most column groups / atoms of one template
  uint32_t cg_slice;
  uint32_t hot;  // column groups of templates whose hot tiles are walked apart
  uint32_t seg_per;  // segments per warp
  uint64_t seg_floats, scr_floats, cend_floats;
};
struct DiffLaunch {
  const DiffTemplate *T;
  const float *atoms;
  float *atoms8;                     // exponential templates' atoms in 32-byte rows
                                     // (same row index as `atoms`), written by the launch
  const uint32_t *exp_list;          // the exponential templates' indices
  uint32_t n_exp;                    // their number
  ColConsts *cols;                   // per exponential column, written by the launch
  float *seg;                        // segment sums
  float *need;                       // per exp tile: an upper bound of its F
  uint32_t *est;                     // per template: key of a lower bound of max F (zeroed)
  uint32_t *hot_groups;              // per group: column groups with hot tiles (zeroed)
  uint32_t n_sms;
  const uint32_t *t0s;
  double temp;
  DiffPartial *parts;                // pass A output
  const double *lnZ1, *lnZ2, *gB, *gS;  // pass B inputs per template: lnBtSG, softmax2F,
                                        // dL/dlnBtSG, dL/dsoftmax2F
  float *scratch;                    // backward: adjoint sources of a group's tiles
  float *cend;                       // backward: recurrence ends of a group
  double *grad_atoms, *grad_tau;     // pass B/C outputs (accumulated; zero them first)
  // rectangular templates: the list of their indices, their geometry for the
  // prefix kernel (rect_ident counts 0, 1, ...) with the prefix rows it fills,
  // FP64 32-atom block sums and (backward) the difference rows of the atom
  // gradient (zeroed by the caller)
  const uint32_t *rect_list, *rect_ident;
  uint32_t n_rect, max_rect_tiles, max_rect_atoms;
  const TemplateDev *rect_T;
  float *P;
  double *B64, *D64;
};
cudaError_t launch_diff(int pass, const DiffLaunch &L, const DiffGroup *groups, uint32_t n_groups,
                        const DiffClass *classes, cudaStream_t stream, cudaStream_t side, cudaEvent_t fork,
                        cudaEvent_t join);
// Failed device-side debug checks per translation unit (TCW_DEBUG_CHECKS).
unsigned int dcheck_failures_kernels();
unsigned int dcheck_failures_diff();
unsigned int dcheck_failures_f64();
unsigned int dcheck_failures_noalloc();
// Full-FP64 direct-summation map of rows rows[0..n_rows) (all rows when rows
// is NULL) into F[r * N_tau + n]; cond optional.
cudaError_t launch_map_f64(int window, const float *atoms, const Geom &g, const uint32_t *t0s,
                           const uint32_t *taus, uint32_t N_tau, const uint32_t *rows,
                           uint32_t n_rows, double *F, double *cond, cudaStream_t stream);
// max_parts: the most tiles of one template.
cudaError_t launch_diff_finalize(const DiffTemplate *T, uint32_t n_templates, uint32_t max_parts,
                                 const DiffPartial *parts, double temp, double *lnB, double *soft,
                                 cudaStream_t stream);

}  // namespace tcw
