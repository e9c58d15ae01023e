// Plain per-template map for callers that cannot allocate device memory.
//
// Some host programs may not call cudaMalloc at all: code running inside a
// memory-pool-managed framework that forbids raw device allocations, code
// that must not synchronise the device (cudaMalloc/cudaFree can), or
// real-time loops that pre-budget every byte at start-up.  They still need
// scratch memory for the map: the compensated prefix rows (rectangular
// window) or the 32-byte atom rows (exponential window), the tile list, the
// per-tile partial reductions and the posterior sums.  This file gives them
// tcw_map_plain_noalloc(): the caller passes inputs and outputs as device
// pointers and a stream; the scratch lives in one file-scope device array
// of kNoallocScratchBytes that every GPU loading the library holds until the
// process exits.  The entry point makes no cudaMalloc / cudaFree call and
// uses no allocating library routine.
//
// Set-up: the first call on a device looks up the device address of the
// array (cudaGetSymbolAddress, with that device current) and caches it per
// device ordinal; make that first call before any stream capture.  The
// cached address belongs to the runtime's primary context of that device:
// after cudaDeviceReset of the device, or with another context made current
// on it through the driver API, the array may live elsewhere and the cached
// address is stale -- this entry point is for processes that keep the
// primary context for their lifetime.  All calls on a
// device share the array and it keeps the last call's contents, so calls
// whose work overlaps on the GPU (different streams, or threads racing to the
// same stream) corrupt each other's scratch: serialise them.  Everything a
// call reads from the array it has written earlier in the same call
// (descriptor, prefix or atom rows, partials), so no clearing is needed
// between calls.
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

#include "../../include/tcw_b200.h"
#include "tcw_internal.h"

using namespace tcw;

namespace {

constexpr size_t kNoallocScratchBytes = TCW_NOALLOC_SCRATCH_BYTES;
constexpr int kMaxDevices = 64;

__device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];
// the posterior argmax's partial maxima and ticket, apart from the scratch
__device__ PostPart g_noalloc_post[2u * kPostParts + 1u];

std::mutex g_scratch_mu;
void *g_scratch_ptr[kMaxDevices] = {nullptr};
void *g_post_ptr[kMaxDevices] = {nullptr};

// Device addresses of the two arrays on the current device (cached).
int scratch_address(int device, unsigned char **out, PostPart **post) {
  if (device < 0 || device >= kMaxDevices) return TCW_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_ptr[device]) {
    void *p = nullptr, *q = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&q, g_noalloc_post);
    if (e != cudaSuccess || !p || !q) {
      cudaGetLastError();
      return TCW_ERR_CUDA;
    }
    g_post_ptr[device] = q;
    g_scratch_ptr[device] = p;
  }
  *post = static_cast<PostPart *>(g_post_ptr[device]);
  *out = static_cast<unsigned char *>(g_scratch_ptr[device]);
  return TCW_OK;
}

size_t align256(size_t x) { return (x + 255u) / 256u * 256u; }

}  // namespace

extern "C" int tcw_map_plain_noalloc(void *stream, const float *d_atoms, uint32_t numAtoms,
                                     uint32_t TAtom, uint32_t t0_data, int window,
                                     const uint32_t *d_t0s, uint32_t N_t0,
                                     const uint32_t *d_taus, uint32_t N_tau, float *d_Fmn,
                                     tcw_result *d_result, int flags) {
  if (!d_atoms || !d_t0s || !d_taus || !d_result) return TCW_ERR_INVALID_ARG;
  if (window != TCW_WINDOW_RECT && window != TCW_WINDOW_EXP) return TCW_ERR_INVALID_ARG;
  if (numAtoms == 0 || TAtom == 0 || N_t0 == 0 || N_tau == 0) return TCW_ERR_INVALID_ARG;
  if ((uint64_t)t0_data + (uint64_t)numAtoms * TAtom > 0xFFFFFFFFull) return TCW_ERR_OVERFLOW;
  const bool post = (flags & TCW_FLAG_POSTERIORS) != 0;
  if (post && !d_Fmn) return TCW_ERR_INVALID_ARG;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_NO_DEVICE;
  }
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_NO_DEVICE;
  }

  const int prec = (flags & TCW_FLAG_UNCOMPENSATED) ? kPrecPlain32
                   : (flags & TCW_FLAG_FP64_DET)    ? kPrecFF_F64Det
                                                    : kPrecFF;
  // tile shapes and scratch layout: the same rules as the handle-based plain
  // entry point; exp columns stay whole histories (`cut` false) where their
  // segment sums do not fit the scratch
  TemplateDev t{};
  t.g = make_geom(numAtoms, TAtom, t0_data);
  t.window = (uint32_t)window;
  t.N_t0 = N_t0;
  t.N_tau = N_tau;
  t.ln_prior = log(70.0 / ((double)N_t0 * (double)N_tau));
  ExpSplit sp{};
  // posterior sums by blocks of p_rows x p_cols cells; documented: 64 rows of
  // all columns
  uint32_t p_rows = 64u, p_cols = 0xFFFFFC00u, n_rc = 0, n_cc = 0;
  size_t o_T = 0, o_parts = 0, o_rows = 0, o_row = 0, o_col = 0, o_G = 0;
  auto layout = [&](bool cut, bool documented) {
    if (window == TCW_WINDOW_EXP) {
      sp = plain_exp_split(numAtoms, N_t0, N_tau, sms, cut);
      set_split(t, sp);
    }
    const uint64_t tiles = plain_tiles(t, sms);
    if (tiles > 0x7FFFFFFFull) return false;
    t.n_parts = (uint32_t)tiles;
    size_t off = 0;
    o_T = off;
    off = align256(off + sizeof(TemplateDev));
    if (documented) off += 256u + align256(sizeof(WorkItem) * (size_t)tiles);
    o_parts = off;
    off = align256(off + sizeof(Partial) * (size_t)tiles);
    o_rows = off;
    off = align256(off + (window == TCW_WINDOW_RECT
                              ? sizeof(float) * kPrefixStride * ((size_t)numAtoms + 1u)
                              : sizeof(float) * 8u * (size_t)numAtoms));
    o_row = off;
    n_rc = (uint32_t)(((uint64_t)N_t0 + p_rows - 1u) / p_rows);
    n_cc = (uint32_t)(((uint64_t)N_tau + p_cols - 1u) / p_cols);
    if (post) off = align256(off + sizeof(double) * (size_t)N_t0 * n_cc);
    o_col = off;
    if (post) off = align256(off + sizeof(double) * (size_t)n_rc * N_tau);
    o_G = off;
    if (sp.nseg) off = align256(off + sizeof(float) * sp.seg_floats(N_tau));
    return off <= kNoallocScratchBytes;
  };
  // admitted by the documented sizes (with a tile list, whole histories); what
  // they admit fits without the list
  if (!layout(false, true)) return TCW_ERR_OVERFLOW;
  const bool cut = window == TCW_WINDOW_EXP && prec != kPrecPlain32;
  // the handle's posterior blocks (post_rows x 1024 columns), larger ones where
  // their sums do not fit (64 x 60000 cells: one block for all of them 1781 us
  // a call, 236 blocks 64 us)
  auto fit = [&](bool c) {
    p_rows = post_rows((uint64_t)N_t0 * N_tau, sms);
    p_cols = 1024u;
    while (!layout(c, false)) {
      if (p_rows < 64u)
        p_rows *= 2u;
      else if (n_cc > 1u)
        p_cols *= 2u;
      else
        return false;
    }
    return true;
  };
  if (!fit(cut)) fit(false);

  unsigned char *base = nullptr;
  PostPart *pp = nullptr;
  int rc = scratch_address(device, &base, &pp);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  TemplateDev *dT = reinterpret_cast<TemplateDev *>(base + o_T);
  Partial *dparts = reinterpret_cast<Partial *>(base + o_parts);
  float *drows = reinterpret_cast<float *>(base + o_rows);
  if (launch_prepare_one(t, dT, d_atoms, drows, prec, s) != cudaSuccess) return TCW_ERR_CUDA;
  float *dG = reinterpret_cast<float *>(base + o_G);
  const uint32_t groups = (N_tau + 31u) / 32u;
  const uint32_t per = segs_per_warp((uint64_t)groups * sp.nseg, sms);
  const uint32_t n_seg_items = groups * ((sp.nseg + per - 1u) / per);
  if (launch_exp_segments(dT, nullptr, n_seg_items, per, drows, d_taus, dG, s) != cudaSuccess)
    return TCW_ERR_CUDA;
  MapLaunch ml{};
  ml.T = dT;
  ml.n_items = t.n_parts;
  ml.persistent = false;
  ml.chained = plain_map_chained(n_seg_items, numAtoms, sms);
  ml.write_map = d_Fmn != nullptr;
  ml.prec = prec;
  ml.atoms = d_atoms;
  ml.atoms8 = window == TCW_WINDOW_EXP ? drows : nullptr;
  ml.t0s = d_t0s;
  ml.taus = d_taus;
  ml.G = dG;
  ml.P = window == TCW_WINDOW_RECT ? drows : nullptr;
  ml.Fmn = d_Fmn;
  ml.parts = dparts;
  if (launch_map(window, ml, s) != cudaSuccess) return TCW_ERR_CUDA;
  if (launch_finalize(dT, 1, dparts, d_result, true, s) != cudaSuccess) return TCW_ERR_CUDA;
  if (post) {
    const PostLayout pl{p_rows, p_cols, n_rc * n_cc, post_parts(N_t0, N_tau), nullptr,
                        reinterpret_cast<double *>(base + o_row),
                        reinterpret_cast<double *>(base + o_col), pp,
                        reinterpret_cast<uint32_t *>(pp + 2u * kPostParts)};
    if (launch_posteriors(dT, 1, pl, d_Fmn, d_result, true, s) != cudaSuccess) return TCW_ERR_CUDA;
  }
  return TCW_OK;
}

namespace tcw {
// Failed debug checks of this file's kernels (0 unless built with TCW_DEBUG_CHECKS).
unsigned int dcheck_failures_noalloc() {
#if defined(TCW_DEBUG_CHECKS)
  return tcw_dcheck_read();
#else
  return 0;
#endif
}
}  // namespace tcw
