// C-ABI layer of the GB300 transient-CW F-statistic map (include/tcw_b200.h).
//
// Host-side responsibilities: argument validation (with the reference's
// u32 time conventions), tiling of maps into work items, workspace
// management, stream ordering, CUDA-graph capture of batched runs, and
// status codes instead of exceptions.  All compute is in tcw_kernels.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <thread>
#include <vector>

#include "../../include/tcw_b200.h"
#include "tcw_internal.h"

using namespace tcw;

struct tcw_handle {
  int device = 0;
  int n_sms = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaStream_t side_stream = nullptr;  // second branch of batched runs
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
  // pipelined host-buffer runs: uploads on their own stream, ordered after
  // the previous run's prefix/repack kernels (the readers of the atoms)
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t consumed_ev = nullptr, consumed_side_ev = nullptr, copied_ev = nullptr;
  bool consumed_pending = false;
  int prio_high = 0, prio_low = 0;
  char *d_ws = nullptr;
  size_t ws_cap = 0;
  char *h_stage = nullptr;
  size_t stage_cap = 0;
  cudaEvent_t stage_ev = nullptr;
  bool stage_pending = false;
  int fail_alloc_countdown = 0;
  char err[512] = {0};
};

struct tcw_plan {
  int device = 0;
  int prec = kPrecFF;
  int flags = 0;
  uint32_t n_templates = 0, n_items = 0, n_rect = 0;
  uint32_t n_items_rect = 0, n_items_exp = 0, n_blocks_rect = 0, n_blocks_exp = 0;
  uint64_t n_cells = 0, n_atom_rows = 0, p_rows = 0;
  tcw_tile_config cfg{};
  char *d_buf = nullptr;  // one allocation for all plan-owned device arrays
  TemplateDev *d_T = nullptr;
  WorkItem *d_items = nullptr;
  Partial *d_parts = nullptr;
  uint32_t *d_rect_list = nullptr, *d_exp_list = nullptr, *d_t0s = nullptr, *d_taus = nullptr;
  uint32_t n_exp = 0, max_exp_atoms = 0;
  float *d_A8 = nullptr;  // exp templates' atoms in rows of 8 floats
  // row-chunked exp columns: segments and their sums
  SegItem *d_segs = nullptr;
  uint32_t n_segs = 0;
  bool exp_chunks = false;  // some columns are cut within a history
  float *d_G = nullptr;
  uint32_t *d_counter = nullptr;  // [0] rect tiles, [1] exp tiles
  float *d_P = nullptr;
  // graph state
  cudaGraphExec_t gexec = nullptr;
  const float *g_atoms = nullptr;
  tcw_result *g_results = nullptr;
  float *g_maps = nullptr;
  cudaStream_t g_stream = nullptr;
  // buffers of the host-buffer entry point
  float *d_atoms_in = nullptr;
  tcw_result *d_res_out = nullptr;
  float *d_maps_out = nullptr;  // maps of tcw_plan_run_maps_host (n_cells floats)
  // posterior plans: chunks and the row / column sums
  PostLayout post{};
};

namespace {

int set_err(tcw_handle *h, int code, const char *fmt, ...) {
  if (h) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(h->err, sizeof(h->err), fmt, ap);
    va_end(ap);
  }
  return code;
}

int cuda_err(tcw_handle *h, cudaError_t e, const char *what) {
  return set_err(h, TCW_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

#define TCW_CUDA(h, call)                          \
  do {                                             \
    cudaError_t _e = (call);                       \
    if (_e != cudaSuccess) return cuda_err(h, _e, #call); \
  } while (0)

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

int ws_alloc(tcw_handle *h, void **p, size_t bytes) {
  if (h->fail_alloc_countdown > 0 && --h->fail_alloc_countdown == 0)
    return set_err(h, TCW_ERR_ALLOC, "workspace allocation of %zu bytes failed (test hook)",
                   bytes);
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_err(h, TCW_ERR_ALLOC, "cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
  }
  return TCW_OK;
}

// Grow-only device workspace.  Growing waits for the handle's stream so that
// no queued kernel still uses the old buffer.
int ensure_ws(tcw_handle *h, size_t bytes) {
  if (bytes <= h->ws_cap) return TCW_OK;
  TCW_CUDA(h, cudaStreamSynchronize(h->stream));
  if (h->d_ws) cudaFree(h->d_ws);
  h->d_ws = nullptr;
  h->ws_cap = 0;
  size_t cap = align_up(bytes + bytes / 4, 1 << 20);
  void *p = nullptr;
  int rc = ws_alloc(h, &p, cap);
  if (rc) return rc;
  h->d_ws = static_cast<char *>(p);
  h->ws_cap = cap;
  return TCW_OK;
}

// Pinned host staging for small control data (descriptors, tile lists).
int ensure_stage(tcw_handle *h, size_t bytes) {
  if (h->stage_pending) {
    TCW_CUDA(h, cudaEventSynchronize(h->stage_ev));
    h->stage_pending = false;
  }
  if (bytes <= h->stage_cap) return TCW_OK;
  if (h->h_stage) cudaFreeHost(h->h_stage);
  h->h_stage = nullptr;
  h->stage_cap = 0;
  size_t cap = align_up(bytes + bytes / 4, 1 << 16);
  void *p = nullptr;
  cudaError_t e = cudaMallocHost(&p, cap);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_err(h, TCW_ERR_ALLOC, "cudaMallocHost(%zu) failed", cap);
  }
  h->h_stage = static_cast<char *>(p);
  h->stage_cap = cap;
  return TCW_OK;
}

struct Layout {
  size_t total = 0;
  size_t add(size_t bytes) {
    size_t off = total;
    total = align_up(total + bytes, 256);
    return off;
  }
};

bool valid_window(int w) { return w == TCW_WINDOW_RECT || w == TCW_WINDOW_EXP; }

int check_geometry(tcw_handle *h, uint32_t numAtoms, uint32_t TAtom, uint32_t t0_data,
                   uint32_t N_t0, uint32_t N_tau) {
  if (numAtoms == 0) return set_err(h, TCW_ERR_INVALID_ARG, "numAtoms must be >= 1");
  if (TAtom == 0) return set_err(h, TCW_ERR_INVALID_ARG, "TAtom must be >= 1");
  if (N_t0 == 0 || N_tau == 0)
    return set_err(h, TCW_ERR_INVALID_ARG, "empty grid: N_t0=%u N_tau=%u", N_t0, N_tau);
  if ((uint64_t)t0_data + (uint64_t)numAtoms * TAtom > 0xFFFFFFFFull)
    return set_err(h, TCW_ERR_OVERFLOW,
                   "atom timestamps t0_data + i*TAtom exceed the u32 range (t0_data=%u, "
                   "numAtoms=%u, TAtom=%u)",
                   t0_data, numAtoms, TAtom);
  if ((uint64_t)N_t0 * (uint64_t)N_tau > (1ull << 62))
    return set_err(h, TCW_ERR_OVERFLOW, "N_t0*N_tau overflows");
  return TCW_OK;
}

// Host-side grid checks (only where the grids are host memory).
int check_grids(tcw_handle *h, int window, const uint32_t *t0s, uint32_t N_t0,
                const uint32_t *taus, uint32_t N_tau) {
  uint32_t t0max = 0, taumax = 0;
  for (uint32_t m = 0; m < N_t0; m++) t0max = std::max(t0max, t0s[m]);
  for (uint32_t n = 0; n < N_tau; n++) {
    taumax = std::max(taumax, taus[n]);
    if (taus[n] == 0 && window == TCW_WINDOW_EXP)
      return set_err(h, TCW_ERR_INVALID_ARG, "exponential window needs tau > 0 (taus[%u]=0)", n);
    if (window == TCW_WINDOW_RECT && n > 0 && taus[n] < taus[n - 1])
      return set_err(h, TCW_ERR_INVALID_ARG,
                     "rectangular window needs a non-decreasing tau grid (taus[%u] < taus[%u])",
                     n, n - 1);
  }
  uint64_t reach = (uint64_t)t0max + (uint64_t)taumax * (window == TCW_WINDOW_EXP ? 3u : 1u);
  if (reach > 0xFFFFFFFFull)
    return set_err(h, TCW_ERR_OVERFLOW, "t0 + %stau exceeds the u32 time range",
                   window == TCW_WINDOW_EXP ? "3*" : "");
  return TCW_OK;
}

int prec_of(int flags) {
  if (flags & TCW_FLAG_UNCOMPENSATED) return kPrecPlain32;
  if (flags & TCW_FLAG_FP64_DET) return kPrecFF_F64Det;
  return kPrecFF;
}

// Time of an exp column in recurrence steps (one atom entering or leaving its
// window): a row's F and table entry take that of kExpRowSteps, and of
// kExpShortRowSteps where windows are so short that F is often near-singular
// and evaluated in double-word FP32 (kShortWindow).  Chunks of equal steps
// rather than equally many per column: with one weight per row the rows of the
// shortest windows were left running when the other warps had ended (35 % of
// the time; 96 templates with maps 1.82 -> 1.55 ms; weights of 3 / 6 / 10 for
// the short windows' rows 1.81 / 1.63 / 1.56).
constexpr double kExpRowSteps = 3.0, kExpShortRowSteps = 10.0;

// The columns of one 32-column group, whose first duration is tau.
struct ExpGroupSteps {
  double atoms, window, per_row, row, t_atom;
  ExpGroupSteps(double n_atoms, uint32_t TAtom, uint32_t N_t0, uint32_t tau)
      : atoms(n_atoms), window(3.0 * tau / TAtom), per_row(n_atoms / N_t0),
        row(window < kShortWindow ? kExpShortRowSteps : kExpRowSteps), t_atom(TAtom) {}
  // Most steps of a chunk's first window.
  double start(const ExpSplit &sp) const {
    return std::min(window, 2.0 * ((1u << sp.shift) + (double)sp.nseg));
  }
  // Atoms of a chunk's run-up (kRunUp); last_tau: the group's longest duration.
  double run_up_atoms(uint32_t last_tau) const {
    return window < kShortWindow
               ? std::min(atoms, kRunUp * std::min(last_tau / t_atom, kShortWindow / 3.0))
               : 0.0;
  }
  // Steps of `rows` rows from row m0 on (starts spread over the data): the
  // atoms that enter, those that leave while the window ends before the data
  // do, and the rows.
  double rows(uint32_t m0, uint32_t n) const {
    const double enter = per_row * n;
    return enter + std::min(enter, std::max(0.0, atoms - window - per_row * m0)) + row * n;
  }
};

// A plan's tiles of one template.  Rect: tn columns x tm rows.  Exp: 32 columns
// x a row chunk of about `chunk_steps` steps where the template has segment
// sums to start one from (8 rows or more), else a history.
void tile_template(uint32_t tmpl, const TemplateDev &t, const tcw_tile_config &cfg,
                   const uint32_t *taus, double chunk_steps, std::vector<WorkItem> &items,
                   std::vector<double> &cost) {
  const uint32_t N_t0 = t.N_t0, N_tau = t.N_tau;
  if (t.window == TCW_WINDOW_RECT) {
    const uint32_t tn = cfg.rect_tn, tm = cfg.rect_tm;
    for (uint32_t n0 = 0; n0 < N_tau; n0 += tn)
      for (uint32_t m0 = 0; m0 < N_t0; m0 += tm) {
        WorkItem w{};
        w.tmpl = tmpl;
        w.m0 = m0;
        w.m1 = std::min(N_t0, m0 + tm);
        w.n0 = n0;
        w.n1 = std::min(N_tau, n0 + tn);
        w.tn = (uint16_t)(tm / 32u);  // row groups of 32 rows (one per warp)
        items.push_back(w);
        cost.push_back((double)(w.m1 - w.m0) * (w.n1 - w.n0));
      }
  } else {
    const double atoms = (double)t.g.numAtoms;
    for (uint32_t n0 = 0; n0 < N_tau; n0 += 32u) {
      uint32_t rows = t.e_hist;
      double run_up = 0.0;  // rows of a chunk's run-up
      const ExpGroupSteps steps(atoms, t.g.TAtom, N_t0, taus[n0]);
      double start = 0.0;  // most steps of a chunk's first window
      if (t.g_nseg) {
        start = steps.start(ExpSplit{t.e_hist, t.e_rows, t.e_sub, t.g_shift, t.g_nseg});
        const double n = steps.rows(0, N_t0) / chunk_steps;
        run_up = steps.run_up_atoms(taus[std::min(N_tau, n0 + 32u) - 1u]) / steps.per_row;
        rows = std::min(rows, (uint32_t)std::max(8.0, ceil(N_t0 / std::max(1.0, ceil(n)))));
      }
      for (uint32_t h0 = 0; h0 < N_t0; h0 += t.e_hist)
        for (uint32_t m0 = h0, h1 = std::min(N_t0, h0 + t.e_hist); m0 < h1; m0 += rows) {
          WorkItem w{};
          w.tmpl = tmpl;
          w.m0 = m0;
          w.m1 = std::min(h1, m0 + rows);
          w.n0 = n0;
          w.n1 = std::min(N_tau, n0 + 32u);
          w.tn = 32;
          items.push_back(w);
          // Whole columns: one cost for all of a template's groups, so that
          // they stay neighbours in the queue and the warps of an SM read the
          // same atoms (ordered by each group's own steps, 1000 templates of up
          // to 600 x 600 cells take 3.45 ms for 2.30).
          if (!t.g_nseg)
            cost.push_back((w.m1 - m0) * (4.0 * std::max(1.0, steps.per_row) + 1.0) +
                           2.0 * std::min(atoms, 3.0 * N_tau));
          else
            cost.push_back(std::min(start, atoms - steps.per_row * w.m1) +
                           (w.m1 < h1 ? run_up : 0.0) + steps.rows(m0, w.m1 - m0));
        }
    }
  }
}

#ifndef TCW_PLAN_RECT_WARPS
#define TCW_PLAN_RECT_WARPS 10
#endif
#ifndef TCW_PLAN_EXP_WARPS
#define TCW_PLAN_EXP_WARPS 8
#endif
// Rows of a history for exp_rows of a tile configuration (0: whole columns).
uint32_t exp_hist(uint32_t exp_rows, uint32_t N_t0) {
  return std::min(std::min(exp_rows ? exp_rows : N_t0, N_t0), 65535u);
}

void fill_cfg_defaults(tcw_tile_config &c) {
  if (c.rect_tm != 32 && c.rect_tm != 64 && c.rect_tm != 128) c.rect_tm = 128;
  if (c.rect_tn == 0) c.rect_tn = 128;
  c.exp_tn = 32;  // exp tiles are 32 columns (tile_template)
  if (c.blocks_per_sm == 0) c.blocks_per_sm = 32;  // cap; occupancy decides below it
}

TemplateDev make_tdev(uint32_t numAtoms, uint32_t TAtom, uint32_t t0_data, int window,
                      uint32_t N_t0, uint32_t N_tau) {
  TemplateDev t{};
  t.g = make_geom(numAtoms, TAtom, t0_data);
  t.window = (uint32_t)window;
  t.N_t0 = N_t0;
  t.N_tau = N_tau;
  t.ln_prior = log(70.0 / ((double)N_t0 * (double)N_tau));
  return t;
}

int set_device(tcw_handle *h) {
  TCW_CUDA(h, cudaSetDevice(h->device));
  return TCW_OK;
}

}  // namespace

// ====================================================================== ABI

extern "C" {

int tcw_abi_version(void) { return TCW_ABI_VERSION; }

const char *tcw_strerror(int status) {
  switch (status) {
    case TCW_OK: return "ok";
    case TCW_ERR_INVALID_ARG: return "invalid argument";
    case TCW_ERR_CUDA: return "CUDA error";
    case TCW_ERR_NO_DEVICE: return "no usable CUDA device";
    case TCW_ERR_ALLOC: return "allocation failed";
    case TCW_ERR_TIMEOUT: return "timed out waiting for the device";
    case TCW_ERR_UNSUPPORTED: return "unsupported";
    case TCW_ERR_OVERFLOW: return "size or time range overflow";
    case TCW_ERR_IO: return "file input/output error";
    case TCW_ERR_FORMAT: return "malformed line in a text file";
    default: return "unknown status";
  }
}

const char *tcw_last_error(const tcw_handle *h) { return h ? h->err : "null handle"; }

int tcw_device_count(int *count) {
  if (!count) return TCW_ERR_INVALID_ARG;
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *count = 0;
    return TCW_ERR_NO_DEVICE;
  }
  *count = n;
  return TCW_OK;
}

int tcw_device_info(int device, char *name, size_t name_len, int *cc_major, int *cc_minor,
                    size_t *total_mem) {
  cudaDeviceProp prop;
  cudaError_t e = cudaGetDeviceProperties(&prop, device);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_NO_DEVICE;
  }
  if (name && name_len) {
    strncpy(name, prop.name, name_len - 1);
    name[name_len - 1] = 0;
  }
  if (cc_major) *cc_major = prop.major;
  if (cc_minor) *cc_minor = prop.minor;
  if (total_mem) *total_mem = prop.totalGlobalMem;
  return TCW_OK;
}

int tcw_device_memory(int device, size_t *free_bytes, size_t *total_bytes) {
  if (!free_bytes || !total_bytes) return TCW_ERR_INVALID_ARG;
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_NO_DEVICE;
  }
  if (cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_NO_DEVICE;
  }
  size_t f = 0, t = 0;
  const cudaError_t e = cudaMemGetInfo(&f, &t);
  cudaSetDevice(prev);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_CUDA;
  }
  *free_bytes = f;
  *total_bytes = t;
  return TCW_OK;
}

int tcw_create(tcw_handle **out, int device) {
  if (!out) return TCW_ERR_INVALID_ARG;
  *out = nullptr;
  int n = 0;
  if (tcw_device_count(&n) != TCW_OK || n == 0) return TCW_ERR_NO_DEVICE;
  if (device < 0 || device >= n) return TCW_ERR_NO_DEVICE;
  tcw_handle *h = new (std::nothrow) tcw_handle();
  if (!h) return TCW_ERR_ALLOC;
  h->device = device;
  int rc = set_device(h);
  if (rc) {
    delete h;
    return rc;
  }
  cudaDeviceProp prop;
  // The kernels are built for sm_103a only: architecture-specific code that
  // loads on compute capability 10.3 and on no other device.
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess || prop.major != 10 ||
      prop.minor != 3) {
    cudaGetLastError();
    delete h;
    return TCW_ERR_NO_DEVICE;
  }
  h->n_sms = prop.multiProcessorCount;
  if (cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->stage_ev, cudaEventDisableTiming) != cudaSuccess) {
    cudaGetLastError();
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    delete h;
    return TCW_ERR_CUDA;
  }
  h->stream = h->own_stream;
  if (cudaDeviceGetStreamPriorityRange(&h->prio_low, &h->prio_high) != cudaSuccess ||
      cudaStreamCreateWithPriority(&h->side_stream, cudaStreamNonBlocking, h->prio_low) !=
          cudaSuccess ||
      cudaEventCreateWithFlags(&h->fork_ev, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->join_ev, cudaEventDisableTiming) != cudaSuccess ||
      cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->consumed_ev, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->consumed_side_ev, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->copied_ev, cudaEventDisableTiming) != cudaSuccess) {
    cudaGetLastError();
    tcw_destroy(h);
    return TCW_ERR_CUDA;
  }
  *out = h;
  return TCW_OK;
}

int tcw_destroy(tcw_handle *h) {
  if (!h) return TCW_ERR_INVALID_ARG;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  if (h->d_ws) cudaFree(h->d_ws);
  if (h->h_stage) cudaFreeHost(h->h_stage);
  if (h->stage_ev) cudaEventDestroy(h->stage_ev);
  if (h->side_stream) {
    cudaStreamSynchronize(h->side_stream);
    cudaStreamDestroy(h->side_stream);
  }
  if (h->fork_ev) cudaEventDestroy(h->fork_ev);
  if (h->join_ev) cudaEventDestroy(h->join_ev);
  if (h->copy_stream) {
    cudaStreamSynchronize(h->copy_stream);
    cudaStreamDestroy(h->copy_stream);
  }
  if (h->consumed_ev) cudaEventDestroy(h->consumed_ev);
  if (h->consumed_side_ev) cudaEventDestroy(h->consumed_side_ev);
  if (h->copied_ev) cudaEventDestroy(h->copied_ev);
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
  cudaGetLastError();
  delete h;
  return TCW_OK;
}

int tcw_get_stream(tcw_handle *h, void **stream) {
  if (!h || !stream) return TCW_ERR_INVALID_ARG;
  *stream = (void *)h->stream;
  return TCW_OK;
}

int tcw_set_stream(tcw_handle *h, void *stream) {
  if (!h) return TCW_ERR_INVALID_ARG;
  h->stream = stream ? (cudaStream_t)stream : h->own_stream;
  return TCW_OK;
}

int tcw_sync(tcw_handle *h, int timeout_ms) {
  if (!h) return TCW_ERR_INVALID_ARG;
  int rc = set_device(h);
  if (rc) return rc;
  auto t0 = std::chrono::steady_clock::now();
  for (;;) {
    cudaError_t e = cudaStreamQuery(h->stream);
    if (e == cudaSuccess) return TCW_OK;
    if (e != cudaErrorNotReady) return cuda_err(h, e, "cudaStreamQuery");
    auto ms = std::chrono::duration_cast<std::chrono::milliseconds>(
                  std::chrono::steady_clock::now() - t0)
                  .count();
    if (timeout_ms >= 0 && ms >= timeout_ms)
      return set_err(h, TCW_ERR_TIMEOUT, "stream not done after %d ms", timeout_ms);
    std::this_thread::sleep_for(std::chrono::microseconds(50));
  }
}

int tcw_pinned_alloc(void **ptr, size_t bytes) {
  if (!ptr) return TCW_ERR_INVALID_ARG;
  *ptr = nullptr;
  if (cudaHostAlloc(ptr, std::max<size_t>(bytes, 16), cudaHostAllocDefault) != cudaSuccess) {
    cudaGetLastError();
    *ptr = nullptr;
    return TCW_ERR_ALLOC;
  }
  return TCW_OK;
}

int tcw_pinned_free(void *ptr) {
  if (!ptr) return TCW_OK;
  if (cudaFreeHost(ptr) != cudaSuccess) {
    cudaGetLastError();
    return TCW_ERR_CUDA;
  }
  return TCW_OK;
}

int tcw_debug_fail_alloc(tcw_handle *h, int n) {
  if (!h || n < 0) return TCW_ERR_INVALID_ARG;
  h->fail_alloc_countdown = n;
  return TCW_OK;
}

// ---------------------------------------------------------------- plain map

// Inputs of a host-buffer map that go through page-locked staging.
constexpr size_t kStagedInputs = 1u << 20;

// Descriptor and workspace of one single-template map behind `off` bytes.
struct PlainLayout {
  TemplateDev t;
  uint32_t n_items, n_seg_items, seg_per, post_rows, post_chunks;
  size_t o_T, o_parts, o_rows, o_G, o_row, o_col, o_pp, total;
};

static int plain_layout(tcw_handle *h, uint32_t numAtoms, uint32_t TAtom, uint32_t t0_data,
                        int window, uint32_t N_t0, uint32_t N_tau, int flags, size_t off,
                        bool cut, PlainLayout &P) {
  TemplateDev &t = P.t;
  t = make_tdev(numAtoms, TAtom, t0_data, window, N_t0, N_tau);
  uint64_t seg_floats = 0;
  P.n_seg_items = 0;
  P.seg_per = 1;
  if (window == TCW_WINDOW_EXP) {
    const ExpSplit sp =
        plain_exp_split(numAtoms, N_t0, N_tau, h->n_sms, cut && prec_of(flags) != kPrecPlain32);
    set_split(t, sp);
    seg_floats = sp.seg_floats(N_tau);
    const uint32_t groups = (N_tau + 31u) / 32u;
    P.seg_per = segs_per_warp((uint64_t)groups * sp.nseg, h->n_sms);
    P.n_seg_items = groups * ((sp.nseg + P.seg_per - 1u) / P.seg_per);
  }
  const uint64_t tiles = plain_tiles(t, h->n_sms);
  if (tiles > 0x7FFFFFFFull) return set_err(h, TCW_ERR_OVERFLOW, "too many tiles");
  P.n_items = t.n_parts = (uint32_t)tiles;
  const bool post = (flags & TCW_FLAG_POSTERIORS) != 0;
  P.post_rows = post_rows((uint64_t)N_t0 * N_tau, h->n_sms);
  const uint32_t n_rc = (N_t0 + P.post_rows - 1u) / P.post_rows, n_cc = (N_tau + 1023u) / 1024u;
  P.post_chunks = n_rc * n_cc;
  Layout L;
  L.total = off;
  P.o_T = L.add(sizeof(TemplateDev));
  P.o_parts = L.add(sizeof(Partial) * P.n_items);
  P.o_rows = L.add(window == TCW_WINDOW_RECT
                       ? sizeof(float) * kPrefixStride * ((size_t)numAtoms + 1)
                       : sizeof(float) * 8u * (size_t)numAtoms);
  P.o_G = L.add(sizeof(float) * seg_floats);
  P.o_row = post ? L.add(sizeof(double) * (size_t)N_t0 * n_cc) : 0;
  P.o_col = post ? L.add(sizeof(double) * (size_t)n_rc * N_tau) : 0;
  P.o_pp = post ? L.add(sizeof(PostPart) * 2u * kPostParts + sizeof(uint32_t)) : 0;
  P.total = L.total;
  return TCW_OK;
}

// Layout and workspace of one map.  Where the memory for the segment sums of
// exp columns (up to 1 GiB) is not to be had, the columns stay whole histories.
static int plain_fit(tcw_handle *h, uint32_t numAtoms, uint32_t TAtom, uint32_t t0_data,
                     int window, uint32_t N_t0, uint32_t N_tau, int flags, size_t off,
                     PlainLayout &P) {
  for (bool cut : {true, false}) {
    int rc =
        plain_layout(h, numAtoms, TAtom, t0_data, window, N_t0, N_tau, flags, off, cut, P);
    if (rc) return rc;
    rc = ensure_ws(h, P.total);
    if (rc != TCW_ERR_ALLOC || P.n_seg_items == 0) return rc;
  }
  return TCW_ERR_ALLOC;
}

// One map: prepare (prefix or repacked rows, the descriptor), exp segment sums,
// map tiles, finalize, posteriors -- a chain of programmatic dependent
// launches that needs nothing from the host but their arguments (and the
// workspace that L was fitted into).
static int plain_enqueue(tcw_handle *h, const PlainLayout &L, const float *d_atoms,
                         const uint32_t *d_t0s, const uint32_t *d_taus, float *d_Fmn,
                         tcw_result *d_result, int flags) {
  char *ws = h->d_ws;
  const int prec = prec_of(flags), window = (int)L.t.window;
  const uint32_t numAtoms = L.t.g.numAtoms;
  const bool rect = window == TCW_WINDOW_RECT;
  TemplateDev *dT = reinterpret_cast<TemplateDev *>(ws + L.o_T);
  float *drows = reinterpret_cast<float *>(ws + L.o_rows);
  Partial *dparts = reinterpret_cast<Partial *>(ws + L.o_parts);
  TCW_CUDA(h, launch_prepare_one(L.t, dT, d_atoms, drows, prec, h->stream));
  float *dG = reinterpret_cast<float *>(ws + L.o_G);
  TCW_CUDA(h, launch_exp_segments(dT, nullptr, L.n_seg_items, L.seg_per, drows, d_taus, dG,
                                  h->stream));
  MapLaunch ml{};
  ml.T = dT;
  ml.n_items = L.n_items;
  ml.persistent = false;
  ml.chained = plain_map_chained(L.n_seg_items, numAtoms, h->n_sms);
  ml.write_map = d_Fmn != nullptr;
  ml.prec = prec;
  ml.atoms = d_atoms;
  ml.atoms8 = rect ? nullptr : drows;
  ml.G = dG;
  ml.t0s = d_t0s;
  ml.taus = d_taus;
  ml.P = rect ? drows : nullptr;
  ml.Fmn = d_Fmn;
  ml.parts = dparts;
  TCW_CUDA(h, launch_map(window, ml, h->stream));
  TCW_CUDA(h, launch_finalize(dT, 1, dparts, d_result, true, h->stream));
  if (flags & TCW_FLAG_POSTERIORS) {
    PostPart *pp = reinterpret_cast<PostPart *>(ws + L.o_pp);
    const PostLayout pl{L.post_rows, 1024u, L.post_chunks, post_parts(L.t.N_t0, L.t.N_tau),
                        nullptr,
                        reinterpret_cast<double *>(ws + L.o_row),
                        reinterpret_cast<double *>(ws + L.o_col), pp,
                        reinterpret_cast<uint32_t *>(pp + 2u * kPostParts)};
    TCW_CUDA(h, launch_posteriors(dT, 1, pl, d_Fmn, d_result, true, h->stream));
  }
  return TCW_OK;
}

int tcw_map_plain(tcw_handle *h, const float *d_atoms, uint32_t numAtoms, uint32_t TAtom,
                  uint32_t t0_data, int window, const uint32_t *d_t0s, uint32_t N_t0,
                  const uint32_t *d_taus, uint32_t N_tau, float *d_Fmn, tcw_result *d_result,
                  int flags) {
  if (!h) return TCW_ERR_INVALID_ARG;
  if (!d_atoms || !d_t0s || !d_taus || !d_result)
    return set_err(h, TCW_ERR_INVALID_ARG, "null device pointer");
  if (!valid_window(window))
    return set_err(h, TCW_ERR_INVALID_ARG,
                   "invalid window type %d: the device entry point takes "
                   "TCW_WINDOW_RECT or TCW_WINDOW_EXP",
                   window);
  int rc = check_geometry(h, numAtoms, TAtom, t0_data, N_t0, N_tau);
  if (rc) return rc;
  if ((flags & TCW_FLAG_POSTERIORS) && !d_Fmn)
    return set_err(h, TCW_ERR_INVALID_ARG, "posteriors need a map (d_Fmn is NULL)");
  rc = set_device(h);
  if (rc) return rc;
  PlainLayout P;
  rc = plain_fit(h, numAtoms, TAtom, t0_data, window, N_t0, N_tau, flags, 0, P);
  if (rc) return rc;
  return plain_enqueue(h, P, d_atoms, d_t0s, d_taus, d_Fmn, d_result, flags);
}

int tcw_map_plain_host(tcw_handle *h, const float *atoms, uint32_t numAtoms, uint32_t TAtom,
                       uint32_t t0_data, int window, const uint32_t *t0s, uint32_t N_t0,
                       const uint32_t *taus, uint32_t N_tau, float *Fmn, tcw_result *result,
                       int flags) {
  if (!h) return TCW_ERR_INVALID_ARG;
  if (!atoms || !result) return set_err(h, TCW_ERR_INVALID_ARG, "null host pointer");
  if (window < 0 || window > TCW_WINDOW_EXP)
    return set_err(h, TCW_ERR_INVALID_ARG, "Unknown window-type (%d) passed as input. Allowed are [0,%d].",
                   window, TCW_WINDOW_EXP);
  uint32_t none_t0 = t0_data, none_tau = 0;
  if (window == TCW_WINDOW_NONE) {
    // one rectangular cell spanning all data (tcw_fstat_map_funcs.py:742-749)
    if ((uint64_t)numAtoms * TAtom > 0xFFFFFFFFull)
      return set_err(h, TCW_ERR_OVERFLOW, "data span exceeds the u32 range");
    none_tau = numAtoms * TAtom;
    window = TCW_WINDOW_RECT;
    t0s = &none_t0;
    taus = &none_tau;
    N_t0 = N_tau = 1;
  }
  if (!t0s || !taus) return set_err(h, TCW_ERR_INVALID_ARG, "null grid pointer");
  int rc = check_geometry(h, numAtoms, TAtom, t0_data, N_t0, N_tau);
  if (rc) return rc;
  rc = check_grids(h, window, t0s, N_t0, taus, N_tau);
  if (rc) return rc;
  rc = set_device(h);
  if (rc) return rc;
  // Workspace: the inputs (atoms, t0s, taus) back to back, the result record,
  // the map, then plain_enqueue's own.  The inputs go up in one copy from
  // page-locked staging (three pageable copies cost the caller ~10 us each)
  // where they are small; the record comes back through staging, too.
  const bool want_map = Fmn != nullptr || (flags & TCW_FLAG_POSTERIORS);
  const size_t b_atoms = sizeof(float) * 7u * (size_t)numAtoms, b_t0 = sizeof(uint32_t) * N_t0,
               b_tau = sizeof(uint32_t) * N_tau;
  Layout L;
  const size_t o_atoms = L.add(b_atoms);
  const size_t o_t0 = L.add(b_t0);
  const size_t o_tau = L.add(b_tau);
  const size_t in_bytes = L.total;
  const size_t o_res = L.add(sizeof(tcw_result));
  const size_t o_map = want_map ? L.add(sizeof(float) * (size_t)N_t0 * N_tau) : 0;
  PlainLayout P;
  rc = plain_fit(h, numAtoms, TAtom, t0_data, window, N_t0, N_tau, flags, L.total, P);
  if (rc) return rc;
  const bool staged = in_bytes <= kStagedInputs;
  const size_t s_res = align_up(staged ? in_bytes : 0, 64);
  rc = ensure_stage(h, s_res + sizeof(tcw_result));
  if (rc) return rc;
  char *ws = h->d_ws;
  if (staged) {
    memcpy(h->h_stage + o_atoms, atoms, b_atoms);
    memcpy(h->h_stage + o_t0, t0s, b_t0);
    memcpy(h->h_stage + o_tau, taus, b_tau);
    TCW_CUDA(h, cudaMemcpyAsync(ws, h->h_stage, in_bytes, cudaMemcpyHostToDevice, h->stream));
  } else {
    TCW_CUDA(h, cudaMemcpyAsync(ws + o_atoms, atoms, b_atoms, cudaMemcpyHostToDevice, h->stream));
    TCW_CUDA(h, cudaMemcpyAsync(ws + o_t0, t0s, b_t0, cudaMemcpyHostToDevice, h->stream));
    TCW_CUDA(h, cudaMemcpyAsync(ws + o_tau, taus, b_tau, cudaMemcpyHostToDevice, h->stream));
  }
  float *dmap = want_map ? reinterpret_cast<float *>(ws + o_map) : nullptr;
  tcw_result *dres = reinterpret_cast<tcw_result *>(ws + o_res);
  rc = plain_enqueue(h, P, reinterpret_cast<const float *>(ws + o_atoms),
                     reinterpret_cast<const uint32_t *>(ws + o_t0),
                     reinterpret_cast<const uint32_t *>(ws + o_tau), dmap, dres, flags);
  // on any error below the stream is drained first: the staging and the
  // caller's buffers must not be in use when this returns
  if (rc == TCW_OK) {
    cudaError_t e = cudaMemcpyAsync(h->h_stage + s_res, dres, sizeof(tcw_result),
                                    cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess && Fmn)
      e = cudaMemcpyAsync(Fmn, dmap, sizeof(float) * (size_t)N_t0 * N_tau,
                          cudaMemcpyDeviceToHost, h->stream);
    if (e != cudaSuccess) rc = cuda_err(h, e, "result download");
  }
  const cudaError_t es = cudaStreamSynchronize(h->stream);
  if (rc) return rc;
  if (es != cudaSuccess) return cuda_err(h, es, "cudaStreamSynchronize");
  memcpy(result, h->h_stage + s_res, sizeof(tcw_result));
  return TCW_OK;
}

// ---------------------------------------------------------------- batched plans

// `cut`: exp columns may be cut into row chunks; *segments: some were, and the
// plan's buffer has their sums.
static int plan_create(tcw_handle *h, const tcw_template_desc *desc, uint32_t n_templates,
                       const uint32_t *t0s, uint64_t n_t0s, const uint32_t *taus, uint64_t n_taus,
                       const tcw_tile_config *cfg_in, int flags, bool cut, bool *segments,
                       tcw_plan **out) {
  if (!desc || n_templates == 0 || !t0s || !taus)
    return set_err(h, TCW_ERR_INVALID_ARG, "empty or null template list / grids");
  int rc = set_device(h);
  if (rc) return rc;
  tcw_tile_config cfg{};
  if (cfg_in) cfg = *cfg_in;
  fill_cfg_defaults(cfg);

  tcw_plan *p = new (std::nothrow) tcw_plan();
  if (!p) return TCW_ERR_ALLOC;
  p->device = h->device;
  p->prec = prec_of(flags);
  p->flags = flags;
  p->n_templates = n_templates;
  std::vector<uint2> post_chunks;
  uint64_t post_row_sums = 0, post_col_sums = 0;
  std::vector<TemplateDev> T(n_templates);
  std::vector<WorkItem> items;
  std::vector<double> cost;
  std::vector<uint32_t> rect_list, exp_list;
  uint64_t p_rows = 0, a8_rows = 0, atom_rows = 0, cells = 0;
  // Row chunks of exp columns when the caller leaves them to the library
  // (exp_rows 0).  A lone warp is bound by its own latency, eight share a
  // scheduler's issue slots, and one wave of whole columns lasts as long as its
  // longest: plans with fewer column tiles than `limit` times `want` (eight
  // warps per scheduler) are cut into chunks of equal steps that bring the warp
  // tiles there, started from segment sums.  Equal columns are cut up to about
  // `want` tiles, columns of unequal length up to 1.3 of it (`most`); a start
  // and its run-up cost up to two and a half times their steps (they run beside
  // fewer warps, behind the segment sums), less where rect tiles keep the SMs
  // busy meanwhile.  Short columns (the longest of few starts' length) stay whole
  // where their chunks would crowd schedulers that whole columns leave free
  // (`crowded`: 97 templates of 200 atoms, 64 x 32 cells: 776 chunks 0.150 ms a
  // run, 97 columns 0.102; 9 templates 0.091 / 0.099).  Per run, cut / whole: 96 templates with maps and posteriors
  // 1.55 / 3.55 ms, 24 templates 0.18 / 0.67; exp templates of up to 2500 atoms
  // and 700 x 700 cells at 0.6, 0.95 and 1.3 `want` 1.01 / 1.40, 1.48 / 1.73,
  // 1.90 / 1.77; 500 atoms, 60 x 60 cells at 0.25, 0.8, 1.0 0.34 / 0.41, 0.65 /
  // 0.63, 0.77 / 0.64; 100 atoms, 20 x 20 at 0.1, 0.8 0.116 / 0.073, 0.220 /
  // 0.154; of each pair the rule takes the smaller (to within 5 % but for a few
  // sizes at its line).  6 or 12 warps are no faster (96 templates 1.66 and
  // 1.64 ms).
  uint64_t seg_blocks = 0;
  double chunk_steps = 0.0;  // 0: whole columns
  if (cut && cfg.exp_rows == 0 && p->prec != kPrecPlain32) {
    double tiles = 0.0, steps = 0.0, most = 0.0, most_mean = 0.0, starts = 0.0, pieces = 0.0;
    bool rect = false;
    for (uint32_t k = 0; k < n_templates; k++) {
      const tcw_template_desc &d = desc[k];
      rect = rect || d.window == TCW_WINDOW_RECT;
      if (d.window != TCW_WINDOW_EXP || d.tau_offset + d.N_tau > n_taus || d.numAtoms == 0 ||
          d.N_t0 == 0)
        continue;
      const ExpSplit sp = exp_split(d.numAtoms, d.N_t0, d.N_tau, d.N_t0, 2);
      const double before = steps;
      for (uint32_t n0 = 0; n0 < d.N_tau; n0 += 32u) {
        const uint32_t *tau = taus + d.tau_offset;
        const ExpGroupSteps g(d.numAtoms, d.TAtom, d.N_t0, tau[n0]);
        const double s = g.rows(0, d.N_t0);
        tiles += 1.0;
        steps += s;
        most = std::max(most, s);
        pieces += ceil(d.N_t0 / 8.0);
        starts += g.start(sp) + 3.0 * g.run_up_atoms(tau[std::min(d.N_tau, n0 + 32u) - 1u]);
      }
      most_mean = std::max(most_mean, (steps - before) / ceil(d.N_tau / 32.0));
    }
    const double want = (double)h->n_sms * 4.0 * TCW_PLAN_EXP_WARPS;
    const double limit =
        std::min(1.3, 0.75 + 0.3 * most * tiles / steps) *
        (1.0 - (rect ? 1.5 * starts : 2.5 * starts + 100.0 * tiles) / steps);
    const double scheds = (double)h->n_sms * 4.0;
    const bool crowded =
        most_mean * tiles < 6.0 * starts && pieces > scheds && tiles < (rect ? 0.5 : 1.0) * scheds;
    if (tiles > 0.0 && tiles <= limit * want && !crowded) chunk_steps = steps / want;
  }
  // Rect tiles when the caller leaves them to the library: 128 x 128 while
  // these give every scheduler TCW_PLAN_RECT_WARPS warps' worth of tiles, else
  // 32 rows x as many columns (32..128) as do (rect map kernel of 24
  // templates: 182 -> 38 us).
  tcw_tile_config rcfg = cfg;
  if (!cfg_in || (cfg_in->rect_tn == 0 && cfg_in->rect_tm == 0)) {
    uint64_t rect_cells = 0;
    for (uint32_t k = 0; k < n_templates; k++)
      if (desc[k].window == TCW_WINDOW_RECT) rect_cells += (uint64_t)desc[k].N_t0 * desc[k].N_tau;
    const uint64_t per = rect_cells / ((uint64_t)h->n_sms * 4u * TCW_PLAN_RECT_WARPS);
    if (per < (uint64_t)cfg.rect_tn * cfg.rect_tm) {
      rcfg.rect_tm = 32;
      rcfg.rect_tn =
          (uint32_t)std::max<uint64_t>(32, std::min<uint64_t>(128, per / 32u / 32u * 32u));
    }
  }
  p->cfg = rcfg;
  std::vector<SegItem> segs;
  {
    uint64_t all = 0;
    for (uint32_t k = 0; k < n_templates; k++) all += (uint64_t)desc[k].N_t0 * desc[k].N_tau;
    // post_rows, but no more blocks than 12 per SM where small maps give them
    // (2000 maps of 20 x 20 cells: 2 blocks of 16 rows each 54 us, one block each
    // 30; a block for both directions of a template's argmax 18 -> 14)
    const uint32_t least = post_rows(all, h->n_sms);
    p->post.cols = 1024u;
    for (p->post.rows = 256u; p->post.rows > least; p->post.rows >>= 1) {
      uint64_t blocks = 0;
      for (uint32_t k = 0; k < n_templates; k++)
        blocks += ((uint64_t)desc[k].N_t0 + p->post.rows - 1u) / p->post.rows *
                  (((uint64_t)desc[k].N_tau + 1023u) / 1024u);
      if (blocks >= (uint64_t)h->n_sms * 12u) break;
    }
  }
  try {
    for (uint32_t k = 0; k < n_templates; k++) {
      const tcw_template_desc &d = desc[k];
      if (!valid_window(d.window)) {
        delete p;
        return set_err(h, TCW_ERR_INVALID_ARG, "template %u: invalid window type %d", k,
                       d.window);
      }
      rc = check_geometry(h, d.numAtoms, d.TAtom, d.t0_data, d.N_t0, d.N_tau);
      if (rc) {
        delete p;
        return rc;
      }
      if (d.t0_offset + d.N_t0 > n_t0s || d.tau_offset + d.N_tau > n_taus) {
        delete p;
        return set_err(h, TCW_ERR_INVALID_ARG, "template %u: grid range outside the arrays", k);
      }
      rc = check_grids(h, d.window, t0s + d.t0_offset, d.N_t0, taus + d.tau_offset, d.N_tau);
      if (rc) {
        delete p;
        return rc;
      }
      TemplateDev t = make_tdev(d.numAtoms, d.TAtom, d.t0_data, d.window, d.N_t0, d.N_tau);
      t.atom_off = d.atom_offset;
      t.t0_off = d.t0_offset;
      t.tau_off = d.tau_offset;
      t.map_off = cells;  // maps of tcw_plan_run_maps: templates in descriptor order
      t.row_off = post_row_sums;
      t.col_off = post_col_sums;
      if (flags & TCW_FLAG_POSTERIORS) {
        const uint32_t n_cc = (d.N_tau + 1023u) / 1024u;
        const uint32_t n_rc = (d.N_t0 + p->post.rows - 1u) / p->post.rows;
        p->post.argmax_blocks = std::max(p->post.argmax_blocks, post_parts(d.N_t0, d.N_tau));
        post_row_sums += (uint64_t)d.N_t0 * n_cc;
        post_col_sums += (uint64_t)d.N_tau * n_rc;
        for (uint32_t c = 0; c < n_cc * n_rc; c++) post_chunks.push_back(make_uint2(k, c));
      }
      if (d.window == TCW_WINDOW_RECT) {
        t.p_off = p_rows;
        p_rows += (uint64_t)d.numAtoms + 1u;
        rect_list.push_back(k);
      } else {
        t.a8_off = a8_rows;
        a8_rows += d.numAtoms;
        exp_list.push_back(k);
        p->max_exp_atoms = std::max(p->max_exp_atoms, d.numAtoms);
      }
      atom_rows = std::max<uint64_t>(atom_rows, d.atom_offset + d.numAtoms);
      cells += (uint64_t)d.N_t0 * d.N_tau;
      const size_t first = items.size();
      if (d.window == TCW_WINDOW_EXP) {
        const uint32_t hist = exp_hist(cfg.exp_rows, d.N_t0), groups = (d.N_tau + 31u) / 32u;
        // cut where the shortest windows' columns hold more than a chunk
        const bool more = chunk_steps > 0.0 &&
                          ExpGroupSteps(d.numAtoms, d.TAtom, d.N_t0, taus[d.tau_offset])
                                  .rows(0, d.N_t0) > chunk_steps;
        ExpSplit sp = exp_split(d.numAtoms, d.N_t0, d.N_tau, hist, more ? 2 : 1);
        if ((seg_blocks + (uint64_t)groups * sp.nseg) * kSegFloats * sizeof(float) > kSegBytesMax)
          sp = exp_split(d.numAtoms, d.N_t0, d.N_tau, hist, 1);
        set_split(t, sp);
        p->exp_chunks = p->exp_chunks || sp.sub > 1u || sp.nseg > 0u;
        t.g_off = seg_blocks;
        seg_blocks += (uint64_t)groups * sp.nseg;
      }
      tile_template(k, t, rcfg, taus + d.tau_offset, chunk_steps, items, cost);
      t.part_off = (uint32_t)first;
      t.n_parts = (uint32_t)(items.size() - first);
      for (size_t i = first; i < items.size(); i++) items[i].part = (uint32_t)i;
      T[k] = t;
    }
    p->post.argmax_blocks = std::min(p->post.argmax_blocks,
                                     std::max(1u, (uint32_t)h->n_sms * 12u / n_templates));
    const uint32_t per = segs_per_warp(seg_blocks, h->n_sms);
    size_t n_segs = 0;
    for (uint32_t k : exp_list)
      n_segs += (size_t)((T[k].N_tau + 31u) / 32u) * ((T[k].g_nseg + per - 1u) / per);
    segs.reserve(n_segs);
    for (uint32_t k : exp_list)
      for (uint32_t cg = 0; cg < (T[k].N_tau + 31u) / 32u; cg++)
        for (uint32_t j = 0; j < T[k].g_nseg; j += per)
          segs.push_back(SegItem{k, cg, j, std::min(T[k].g_nseg, j + per)});
    // two queues (rect tiles, then exp tiles), each in longest-processing-time
    // order to within 1 % (a counting sort by the cost's exponent and upper
    // mantissa bits)
    auto bucket = [&](size_t i) {
      const float c = (float)cost[i];
      uint32_t bits;
      memcpy(&bits, &c, sizeof bits);
      return (T[items[i].tmpl].window == TCW_WINDOW_RECT ? 0u : 0x8000u) + 0x7FFFu - (bits >> 16);
    };
    std::vector<uint16_t> key(items.size());
    uint32_t nr = 0;
    for (size_t i = 0; i < items.size(); i++) {
      key[i] = (uint16_t)bucket(i);
      nr += key[i] < 0x8000u ? 1u : 0u;
    }
    std::vector<WorkItem> sorted(items.size());
    if (items.size() < 4096u) {  // (40 us for the counts alone)
      std::vector<uint32_t> order(items.size());
      for (size_t i = 0; i < order.size(); i++) order[i] = (uint32_t)i;
      std::stable_sort(order.begin(), order.end(),
                       [&](uint32_t a, uint32_t b) { return key[a] < key[b]; });
      for (size_t i = 0; i < order.size(); i++) sorted[i] = items[order[i]];
    } else {
      std::vector<uint32_t> at(0x10001u, 0u);
      for (uint16_t k : key) at[k + 1u]++;
      for (uint32_t b = 0; b < 0x10000u; b++) at[b + 1u] += at[b];
      for (size_t i = 0; i < items.size(); i++) sorted[at[key[i]]++] = items[i];
    }
    items.swap(sorted);
    p->n_items_rect = nr;
    p->n_items_exp = (uint32_t)items.size() - nr;
  } catch (const std::bad_alloc &) {
    delete p;
    return set_err(h, TCW_ERR_ALLOC, "host allocation failed while planning");
  }
  if (items.size() > 0xFFFFFFF0ull) {
    delete p;
    return set_err(h, TCW_ERR_OVERFLOW, "too many tiles");
  }
  p->n_items = (uint32_t)items.size();
  p->n_rect = (uint32_t)rect_list.size();
  p->n_exp = (uint32_t)exp_list.size();
  p->n_segs = (uint32_t)segs.size();
  *segments = p->n_segs != 0;
  p->n_cells = cells;
  p->n_atom_rows = atom_rows;
  p->p_rows = p_rows;
  {
    const uint32_t br = (uint32_t)std::min<int>(map_blocks_per_sm(TCW_WINDOW_RECT, p->prec, false),
                                                (int)cfg.blocks_per_sm);
    const uint32_t be = (uint32_t)std::min<int>(map_blocks_per_sm(TCW_WINDOW_EXP, p->prec, p->exp_chunks),
                                                (int)cfg.blocks_per_sm);
    p->n_blocks_rect = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>(p->n_items_rect, (uint64_t)br * h->n_sms));
    p->n_blocks_exp = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>(p->n_items_exp, (uint64_t)be * h->n_sms));
  }

  Layout L;
  const size_t o_T = L.add(sizeof(TemplateDev) * n_templates);
  const size_t o_items = L.add(sizeof(WorkItem) * p->n_items);
  const size_t o_list = L.add(sizeof(uint32_t) * std::max<size_t>(1, rect_list.size()));
  const size_t o_elist = L.add(sizeof(uint32_t) * std::max<size_t>(1, exp_list.size()));
  const size_t o_t0 = L.add(sizeof(uint32_t) * n_t0s);
  const size_t o_tau = L.add(sizeof(uint32_t) * n_taus);
  const size_t o_segs = L.add(sizeof(SegItem) * segs.size());
  const size_t ctl_end = L.total;
  const size_t o_parts = L.add(sizeof(Partial) * p->n_items);
  const size_t o_G = L.add(sizeof(float) * kSegFloats * seg_blocks);
  const size_t o_P = L.add(sizeof(float) * kPrefixStride * std::max<uint64_t>(1, p_rows));
  const size_t o_A8 = L.add(sizeof(float) * 8u * std::max<uint64_t>(1, a8_rows));
  const size_t o_cnt = L.add(2 * sizeof(uint32_t));
  const bool post = (flags & TCW_FLAG_POSTERIORS) != 0;
  const size_t o_chunks = post ? L.add(sizeof(uint2) * std::max<size_t>(1, post_chunks.size())) : 0;
  const size_t o_rowsum = post ? L.add(sizeof(double) * post_row_sums) : 0;
  const size_t o_colsum = post ? L.add(sizeof(double) * post_col_sums) : 0;
  const size_t o_pp = post ? L.add(sizeof(PostPart) * 2u * kPostParts * (size_t)n_templates) : 0;
  const size_t o_ticket = post ? L.add(sizeof(uint32_t) * n_templates) : 0;
  void *buf = nullptr;
  rc = ws_alloc(h, &buf, L.total);
  if (rc) {
    delete p;
    return rc;
  }
  p->d_buf = static_cast<char *>(buf);
  p->d_T = reinterpret_cast<TemplateDev *>(p->d_buf + o_T);
  p->d_items = reinterpret_cast<WorkItem *>(p->d_buf + o_items);
  p->d_rect_list = reinterpret_cast<uint32_t *>(p->d_buf + o_list);
  p->d_exp_list = reinterpret_cast<uint32_t *>(p->d_buf + o_elist);
  p->d_A8 = reinterpret_cast<float *>(p->d_buf + o_A8);
  p->d_segs = reinterpret_cast<SegItem *>(p->d_buf + o_segs);
  p->d_G = reinterpret_cast<float *>(p->d_buf + o_G);
  p->d_t0s = reinterpret_cast<uint32_t *>(p->d_buf + o_t0);
  p->d_taus = reinterpret_cast<uint32_t *>(p->d_buf + o_tau);
  p->d_parts = reinterpret_cast<Partial *>(p->d_buf + o_parts);
  p->d_P = reinterpret_cast<float *>(p->d_buf + o_P);
  p->d_counter = reinterpret_cast<uint32_t *>(p->d_buf + o_cnt);
  if (post) {
    p->post.chunks = reinterpret_cast<const uint2 *>(p->d_buf + o_chunks);
    p->post.n_chunks = (uint32_t)post_chunks.size();
    p->post.rowsum = reinterpret_cast<double *>(p->d_buf + o_rowsum);
    p->post.colsum = reinterpret_cast<double *>(p->d_buf + o_colsum);
    p->post.parts = reinterpret_cast<PostPart *>(p->d_buf + o_pp);
    p->post.ticket = reinterpret_cast<uint32_t *>(p->d_buf + o_ticket);
  }
  // control data: a synchronous copy (plans are built once)
  std::vector<char> host(ctl_end);
  memcpy(host.data() + o_T, T.data(), sizeof(TemplateDev) * n_templates);
  memcpy(host.data() + o_items, items.data(), sizeof(WorkItem) * p->n_items);
  if (!rect_list.empty())
    memcpy(host.data() + o_list, rect_list.data(), sizeof(uint32_t) * rect_list.size());
  if (!exp_list.empty())
    memcpy(host.data() + o_elist, exp_list.data(), sizeof(uint32_t) * exp_list.size());
  memcpy(host.data() + o_t0, t0s, sizeof(uint32_t) * n_t0s);
  memcpy(host.data() + o_tau, taus, sizeof(uint32_t) * n_taus);
  if (!segs.empty()) memcpy(host.data() + o_segs, segs.data(), sizeof(SegItem) * segs.size());
  cudaError_t e = cudaMemcpy(p->d_buf, host.data(), ctl_end, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && post && !post_chunks.empty())
    e = cudaMemcpy(p->d_buf + o_chunks, post_chunks.data(), sizeof(uint2) * post_chunks.size(),
                   cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(p->d_buf);
    delete p;
    return cuda_err(h, e, "plan upload");
  }
  *out = p;
  return TCW_OK;
}

int tcw_plan_create(tcw_handle *h, const tcw_template_desc *desc, uint32_t n_templates,
                    const uint32_t *t0s, uint64_t n_t0s, const uint32_t *taus, uint64_t n_taus,
                    const tcw_tile_config *cfg, int flags, tcw_plan **out) {
  if (!h || !out) return TCW_ERR_INVALID_ARG;
  *out = nullptr;
  bool segments = false;
  int rc = plan_create(h, desc, n_templates, t0s, n_t0s, taus, n_taus, cfg, flags, true,
                       &segments, out);
  // without the memory for segment sums (up to 1 GiB): whole columns
  if (rc == TCW_ERR_ALLOC && segments)
    rc = plan_create(h, desc, n_templates, t0s, n_t0s, taus, n_taus, cfg, flags, false,
                     &segments, out);
  return rc;
}

int tcw_plan_destroy(tcw_plan *p) {
  if (!p) return TCW_ERR_INVALID_ARG;
  cudaSetDevice(p->device);
  cudaDeviceSynchronize();
  if (p->gexec) cudaGraphExecDestroy(p->gexec);
  if (p->d_buf) cudaFree(p->d_buf);
  if (p->d_atoms_in) cudaFree(p->d_atoms_in);
  if (p->d_res_out) cudaFree(p->d_res_out);
  if (p->d_maps_out) cudaFree(p->d_maps_out);
  cudaGetLastError();
  delete p;
  return TCW_OK;
}

int tcw_plan_info(const tcw_plan *p, uint64_t *n_cells, uint32_t *n_items,
                  uint64_t *n_atom_rows, tcw_tile_config *cfg) {
  if (!p) return TCW_ERR_INVALID_ARG;
  if (n_cells) *n_cells = p->n_cells;
  if (n_items) *n_items = p->n_items;
  if (n_atom_rows) *n_atom_rows = p->n_atom_rows;
  if (cfg) *cfg = p->cfg;
  return TCW_OK;
}

static MapLaunch plan_launch(const tcw_handle *h, const tcw_plan *p, int window,
                             const float *d_atoms, float *d_maps) {
  MapLaunch ml{};
  const bool rect = window == TCW_WINDOW_RECT;
  ml.T = p->d_T;
  ml.items = p->d_items + (rect ? 0 : p->n_items_rect);
  ml.n_items = rect ? p->n_items_rect : p->n_items_exp;
  ml.counter = p->d_counter + (rect ? 0 : 1);
  ml.n_blocks = rect ? p->n_blocks_rect : p->n_blocks_exp;
  ml.persistent = true;
  ml.chunks = p->exp_chunks;
  ml.write_map = d_maps != nullptr;
  ml.prec = p->prec;
  ml.priority = rect ? h->prio_low : h->prio_high;
  ml.atoms = d_atoms;
  ml.atoms8 = p->d_A8;
  ml.G = p->d_G;
  ml.t0s = p->d_t0s;
  ml.taus = p->d_taus;
  ml.P = p->d_P;
  ml.Fmn = d_maps;
  ml.parts = p->d_parts;
  return ml;
}

// (repack -> exp tiles on the main stream at high priority) || (prefix ->
// rect tiles on the side stream) -> finalize.  The exp tiles are the long
// ones; the rect kernel's blocks fill SMs as exp blocks retire.
// `inputs_read` / `inputs_read_side`, if set, are recorded once the atoms
// have been read (after the repack kernel on the main stream and the prefix
// kernel on the side stream; the map kernels read only their outputs).
static int plan_enqueue(tcw_handle *h, tcw_plan *p, const float *d_atoms, tcw_result *d_results,
                        float *d_maps, cudaEvent_t inputs_read = nullptr,
                        cudaEvent_t inputs_read_side = nullptr) {
  TCW_CUDA(h, cudaMemsetAsync(p->d_counter, 0, 2 * sizeof(uint32_t), h->stream));
  // Two branches from the start: repack -> exp tiles (main stream, high
  // priority) || prefix -> rect tiles (side stream, low priority), so the
  // exp kernel does not wait for the rect templates' prefix scans; the
  // persistent rect blocks take the SMs that exp blocks leave as the exp
  // tile queue runs dry (its tail).
  TCW_CUDA(h, cudaEventRecord(h->fork_ev, h->stream));
  TCW_CUDA(h, cudaStreamWaitEvent(h->side_stream, h->fork_ev, 0));
  TCW_CUDA(h, launch_repack(p->d_T, p->d_exp_list, p->n_exp, p->max_exp_atoms, d_atoms, p->d_A8,
                            h->stream));
  if (inputs_read) TCW_CUDA(h, cudaEventRecord(inputs_read, h->stream));
  TCW_CUDA(h, launch_exp_segments(p->d_T, p->d_segs, p->n_segs, 0, p->d_A8, p->d_taus, p->d_G,
                                  h->stream));
  TCW_CUDA(h, launch_prefix(p->d_T, p->d_rect_list, p->n_rect, d_atoms, p->d_P, p->prec,
                            h->side_stream));
  if (inputs_read_side) TCW_CUDA(h, cudaEventRecord(inputs_read_side, h->side_stream));
  TCW_CUDA(h, launch_map(TCW_WINDOW_EXP, plan_launch(h, p, TCW_WINDOW_EXP, d_atoms, d_maps),
                         h->stream));
  TCW_CUDA(h, launch_map(TCW_WINDOW_RECT, plan_launch(h, p, TCW_WINDOW_RECT, d_atoms, d_maps),
                         h->side_stream));
  TCW_CUDA(h, cudaEventRecord(h->join_ev, h->side_stream));
  TCW_CUDA(h, cudaStreamWaitEvent(h->stream, h->join_ev, 0));
  TCW_CUDA(h, launch_finalize(p->d_T, p->n_templates, p->d_parts, d_results, false,
                              h->stream));
  if (d_maps && (p->flags & TCW_FLAG_POSTERIORS))
    TCW_CUDA(h, launch_posteriors(p->d_T, p->n_templates, p->post, d_maps, d_results, false,
                                  h->stream));
  return TCW_OK;
}

}  // extern "C"

static int plan_run(tcw_handle *h, tcw_plan *p, const float *d_atoms, tcw_result *d_results,
                    float *d_maps, int use_graph) {
  if (!h || !p) return TCW_ERR_INVALID_ARG;
  if (!d_atoms || !d_results) return set_err(h, TCW_ERR_INVALID_ARG, "null device pointer");
  if ((p->flags & TCW_FLAG_POSTERIORS) && !d_maps)
    return set_err(h, TCW_ERR_INVALID_ARG,
                   "posteriors need the maps: run the plan with tcw_plan_run_maps");
  if (p->device != h->device)
    return set_err(h, TCW_ERR_INVALID_ARG, "plan and handle are on different devices");
  int rc = set_device(h);
  if (rc) return rc;
  // stream capture is not allowed on the legacy default stream: run directly
  if (!use_graph || h->stream == nullptr || h->stream == cudaStreamLegacy)
    return plan_enqueue(h, p, d_atoms, d_results, d_maps);
  if (!p->gexec || p->g_atoms != d_atoms || p->g_results != d_results || p->g_maps != d_maps ||
      p->g_stream != h->stream) {
    if (p->gexec) {
      cudaGraphExecDestroy(p->gexec);
      p->gexec = nullptr;
    }
    TCW_CUDA(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    rc = plan_enqueue(h, p, d_atoms, d_results, d_maps);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
    if (rc) {
      if (graph) cudaGraphDestroy(graph);
      return rc;
    }
    if (e != cudaSuccess) return cuda_err(h, e, "cudaStreamEndCapture");
    e = cudaGraphInstantiate(&p->gexec, graph, cudaGraphInstantiateFlagUseNodePriority);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      p->gexec = nullptr;
      return cuda_err(h, e, "cudaGraphInstantiate");
    }
    p->g_atoms = d_atoms;
    p->g_results = d_results;
    p->g_maps = d_maps;
    p->g_stream = h->stream;
  }
  TCW_CUDA(h, cudaGraphLaunch(p->gexec, h->stream));
  return TCW_OK;
}

extern "C" {

int tcw_plan_run(tcw_handle *h, tcw_plan *p, const float *d_atoms, tcw_result *d_results,
                 int use_graph) {
  return plan_run(h, p, d_atoms, d_results, nullptr, use_graph);
}

int tcw_plan_run_maps(tcw_handle *h, tcw_plan *p, const float *d_atoms, tcw_result *d_results,
                      float *d_maps, int use_graph) {
  if (h && !d_maps) return set_err(h, TCW_ERR_INVALID_ARG, "null map buffer");
  return plan_run(h, p, d_atoms, d_results, d_maps, use_graph);
}

int tcw_plan_run_timed(tcw_handle *h, tcw_plan *p, const float *d_atoms, tcw_result *d_results,
                       float *ms) {
  if (!h || !p || !ms) return TCW_ERR_INVALID_ARG;
  if (!d_atoms || !d_results) return set_err(h, TCW_ERR_INVALID_ARG, "null device pointer");
  int rc = set_device(h);
  if (rc) return rc;
  cudaEvent_t ev[5];
  for (int i = 0; i < 5; i++) TCW_CUDA(h, cudaEventCreate(&ev[i]));
  TCW_CUDA(h, cudaMemsetAsync(p->d_counter, 0, 2 * sizeof(uint32_t), h->stream));
  TCW_CUDA(h, cudaEventRecord(ev[0], h->stream));
  TCW_CUDA(h, launch_prefix(p->d_T, p->d_rect_list, p->n_rect, d_atoms, p->d_P, p->prec,
                            h->stream));
  TCW_CUDA(h, launch_repack(p->d_T, p->d_exp_list, p->n_exp, p->max_exp_atoms, d_atoms, p->d_A8,
                            h->stream));
  TCW_CUDA(h, cudaEventRecord(ev[1], h->stream));
  TCW_CUDA(h, launch_map(TCW_WINDOW_RECT, plan_launch(h, p, TCW_WINDOW_RECT, d_atoms, nullptr),
                         h->stream));
  TCW_CUDA(h, cudaEventRecord(ev[2], h->stream));
  TCW_CUDA(h, launch_exp_segments(p->d_T, p->d_segs, p->n_segs, 0, p->d_A8, p->d_taus, p->d_G,
                                  h->stream));
  TCW_CUDA(h, launch_map(TCW_WINDOW_EXP, plan_launch(h, p, TCW_WINDOW_EXP, d_atoms, nullptr),
                         h->stream));
  TCW_CUDA(h, cudaEventRecord(ev[3], h->stream));
  TCW_CUDA(h, launch_finalize(p->d_T, p->n_templates, p->d_parts, d_results, false,
                              h->stream));
  TCW_CUDA(h, cudaEventRecord(ev[4], h->stream));
  TCW_CUDA(h, cudaEventSynchronize(ev[4]));
  for (int i = 0; i < 4; i++) TCW_CUDA(h, cudaEventElapsedTime(&ms[i], ev[i], ev[i + 1]));
  for (int i = 0; i < 5; i++) cudaEventDestroy(ev[i]);
  return TCW_OK;
}

// ---------------------------------------------------------------- differentiable path

// Validates descriptors, uploads descriptors, tiles and grids into the
// handle's workspace; returns the layout of what follows them.
struct DiffSetup {
  size_t o_T, o_parts, o_t0, o_est, o_hot, o_rlist, o_ident, o_RT, o_P, o_B64, o_D64, o_elist, o_A8;
  size_t o_cols, o_seg, o_need, o_scratch, o_cend, total;
  uint32_t n_rect, max_rect_tiles, max_rect_atoms, n_exp;
  uint32_t max_parts;  // most tiles of one template
  uint64_t p_rows, seg_floats;
  std::vector<DiffGroup> groups;
  std::vector<DiffClass> classes;
};

// Backward workspace of one group of exponential templates (adjoint sources
// and recurrence ends; the segment sums of a pass have as much again) and the
// most templates of one (grid y dimension).  A template that needs more is a
// group by itself, in slices of column groups within kDiffSliceBytes for the
// sources and for the ends; of the sources at least one column group per SM,
// the width at which diff_hot_kernel fills the GPU.
constexpr uint64_t kDiffGroupBytes = 1ull << 30;
constexpr uint64_t kDiffSliceBytes = 4ull << 30;
constexpr uint32_t kDiffGroupMax = 65535u;

// Adjoint sources (unpadded row chunks) and recurrence ends of one column group.
static uint64_t diff_source_bytes(const DiffTemplate &t) {
  return (uint64_t)t.N_t0 * TCW_DIFF_SLOTS * 32u * sizeof(float);
}
static uint64_t diff_end_bytes(const DiffTemplate &t) {
  return ((uint64_t)t.g.numAtoms + kDiffAtomSeg - 1u) / kDiffAtomSeg * kDiffSegFloats *
         sizeof(float);
}

// Tiles of the exponential templates elist[y0, y1): as many row chunks per
// column as give every resident warp (32 per SM) four tiles, at least 16 rows
// each; chunks start from segment sums of 2^shift atoms (exp_split).  Four
// rather than one: the tiles that carry weight are few, and the kernels that
// walk them last as long as their longest tile (24 templates 3.19 -> 2.99 ms,
// 100 5.4 -> 5.0, 600 17.8 -> 12.9; two 2.98 / 5.1 / 14.3, eight 3.1: the
// estimate starts too many chunks).
// Where whole columns give most schedulers a warp, templates of few rows and
// atoms keep whole columns (so do the shortest columns of any batch, 10 x 10
// cells of 48 atoms 235 -> 223 us): a handful of chunks per column buys little,
// most of them hold a cell that matters by itself, and the walk that
// diff_hot_kernel would repeat is then the tile's own, bit for bit.  Whole columns
// go without the estimate, a walk as long as their own that skips nothing where
// signals are weak -- but for the forward pass of few atoms per row, whose FP64 F
// is most of the work (kDiffEstAtoms; with / without it, noise and a loud signal:
// 500 templates of 400 atoms, 32 x 600 cells 2.6, 1.3 / 1.9, 1.7 ms, 2000 of 1500,
// 32 x 128 6.0, 4.4 / 2.7, 2.7) -- and, from four warps per scheduler on, without
// the segments of the transposed recurrence (one pass in place of two).  More atoms make the
// walk the longest chain (64 rows of 17532 atoms among 300 templates: 12.5 + 14.7
// -> 26 + 34 ms), so they are cut.
constexpr uint32_t kDiffFewRows = 64, kDiffFewAtoms = 2048, kDiffEstAtoms = 14;
// Warps of a class's grid that have no tile: above this, half a millisecond of
// empty blocks, the templates of unequal size go in launches of their own,
// each of which lasts as long as its longest tile (gradients of 2000 templates
// of 32 x 32 cells beside one of 17532 atoms and 1024 x 2048: one grid for all
// 8.3 + 21.1 ms, two classes 5.2 + 8.8; 300 templates of log-uniform sizes: one
// 12.1 + 14.3, three 13.1 + 17.0).
constexpr uint64_t kDiffEmptyWarps = 1ull << 22;
static void diff_tile_group(const tcw_handle *h, std::vector<DiffTemplate> &T,
                            const std::vector<uint32_t> &elist, uint32_t y0, uint32_t y1,
                            int pass, bool cut, DiffGroup &g, std::vector<DiffClass> &classes) {
  uint64_t total_cg = 0;
  for (uint32_t y = y0; y < y1; y++) total_cg += (T[elist[y]].N_tau + 31u) / 32u;
  const uint64_t chunks = ((uint64_t)h->n_sms * 128u + total_cg - 1u) / total_cg;
  const bool filled = total_cg >= (uint64_t)h->n_sms * 3u;
  const bool full = total_cg >= (uint64_t)h->n_sms * 16u;
  const uint64_t seg_floats = pass ? kDiffSegFloatsV : kDiffSegFloats;
  uint64_t seg = 0, scr = 0, cend = 0;
  g = DiffGroup{};
  g.y0 = y0;
  g.ny = y1 - y0;
  g.c0 = (uint32_t)classes.size();
  uint64_t most_warps = 0, class_warps = 0;  // of one template, of all of the class
  g.cg_slice = 0xFFFFFFFFu;
  if (pass && g.ny == 1u) {
    const DiffTemplate &t = T[elist[y0]];
    const uint64_t src = std::max<uint64_t>(h->n_sms, kDiffSliceBytes / diff_source_bytes(t));
    const uint64_t end = std::max<uint64_t>(1, kDiffSliceBytes / diff_end_bytes(t));
    g.cg_slice = (uint32_t)std::min<uint64_t>(g.cg_slice, std::min(src, end));
  }
  for (uint32_t y = y0; y < y1; y++) {
    DiffTemplate &t = T[elist[y]];
    t.n_cg = (t.N_tau + 31u) / 32u;
    const uint64_t most = (t.N_t0 + 15u) / 16u;
    uint64_t nc = cut && !(filled && t.N_t0 <= kDiffFewRows && t.g.numAtoms <= kDiffFewAtoms)
                      ? std::max<uint64_t>(1, std::min(chunks, most))
                      : 1;
    t.g_shift = 5;
    while ((4ull << (2u * t.g_shift)) <= t.g.numAtoms) t.g_shift++;
    t.g_nseg = (uint32_t)(((uint64_t)t.g.numAtoms + (1u << t.g_shift) - 1u) >> t.g_shift);
    if (nc > 1 && (seg + (uint64_t)t.n_cg * t.g_nseg) * seg_floats * sizeof(float) > kDiffGroupBytes)
      nc = 1;
    t.chunk_rows = (uint32_t)((t.N_t0 + nc - 1) / nc);
    t.n_chunk = (t.N_t0 + t.chunk_rows - 1u) / t.chunk_rows;
    if (t.n_chunk == 1u || t.g.numAtoms < 64u) t.g_nseg = 0;
    const bool tiny = 2u * (uint64_t)t.g.numAtoms + 10u * (uint64_t)t.N_t0 <= 512u;
    if (t.n_chunk == 1u && ((filled && t.g.numAtoms <= kDiffFewAtoms) || tiny))
      t.whole = !pass && filled && t.g.numAtoms / kDiffEstAtoms < t.N_t0 ? kDiffWhole
                                                                       : kDiffWholeBlind;
    if (!t.whole) g.hot += t.n_cg;
    t.a_shift = kDiffAtomShift;
    while (((t.g.numAtoms - 1u) >> t.a_shift) >= (t.whole && full ? 1u : kDiffMaxAseg)) t.a_shift++;
    t.n_aseg = ((t.g.numAtoms - 1u) >> t.a_shift) + 1u;
    t.seg_off = seg;
    t.scr_off = scr;
    t.cend_off = cend;
    seg += (uint64_t)t.n_cg * t.g_nseg;
    const uint32_t cgs = std::min(t.n_cg, g.cg_slice);
    scr += (uint64_t)cgs * t.n_chunk * t.chunk_rows * TCW_DIFF_SLOTS * 32u;
    cend += (uint64_t)cgs * t.n_aseg;
    g.max_cg = std::max(g.max_cg, t.n_cg);
    g.max_atoms = std::max(g.max_atoms, t.g.numAtoms);
    const uint64_t warps = std::max<uint64_t>(
        (t.g.numAtoms + kDiffAtomSeg - 1u) / kDiffAtomSeg,  // (diff_prep_kernel)
        (uint64_t)cgs * std::max(std::max(t.n_chunk, t.g_nseg), pass ? t.n_aseg : 0u));
    const uint64_t most_now = std::max(most_warps, warps);
    if (y == y0 || (classes.back().ny + 1u) * most_now > class_warps + warps + kDiffEmptyWarps) {
      classes.push_back(DiffClass{});
      classes.back().y0 = y;
      most_warps = warps;
      class_warps = 0;
    } else {
      most_warps = most_now;
    }
    class_warps += warps;
    DiffClass &c = classes.back();
    c.ny++;
    c.max_tiles = std::max(c.max_tiles, t.n_cg * t.n_chunk);
    c.max_segs = std::max(c.max_segs, t.n_cg * t.g_nseg);
    c.max_atoms = std::max(c.max_atoms, t.g.numAtoms);
    c.max_cols = std::max(c.max_cols, t.N_tau);
    c.slice_tiles = std::max(c.slice_tiles, cgs * t.n_chunk);
    c.slice_aseg = std::max(c.slice_aseg, cgs * t.n_aseg);
    c.slice_cg = std::max(c.slice_cg, cgs);
    if (t.whole != kDiffWholeBlind) c.est_tiles = std::max(c.est_tiles, t.n_cg * t.n_chunk);
    if (t.n_aseg > 1u) c.slice_ends = std::max(c.slice_ends, cgs * t.n_aseg);
  }
  g.n_classes = (uint32_t)classes.size() - g.c0;
  g.seg_per = segs_per_warp(seg, h->n_sms);
  g.seg_floats = seg * seg_floats;
  g.scr_floats = pass ? scr : 0;
  g.cend_floats = pass ? cend * kDiffSegFloats : 0;
}

static int diff_setup(tcw_handle *h, const tcw_diff_desc *desc, uint32_t n, const uint32_t *t0s,
                      uint64_t n_t0s, int pass, bool cut, DiffSetup &S) {
  S = DiffSetup{};
  if (!desc || n == 0 || !t0s) return set_err(h, TCW_ERR_INVALID_ARG, "empty template list");
  std::vector<DiffTemplate> T;
  std::vector<TemplateDev> RT;
  std::vector<uint32_t> rlist, elist, ident;
  uint64_t p_rows = 0, atom_rows = 0, n_cols = 0, n_tiles = 0, b_rows = 0, row_groups = 0;
  S.max_rect_tiles = S.max_rect_atoms = 0;
  uint64_t seg_floats = 0, scr_floats = 0, cend_floats = 0;
  try {
    T.resize(n);
    for (uint32_t k = 0; k < n; k++) {
      const tcw_diff_desc &d = desc[k];
      int rc = check_geometry(h, d.numAtoms, d.TAtom, d.t0_data, d.N_t0, d.N_tau);
      if (rc) return rc;
      if (d.t0_offset + d.N_t0 > n_t0s)
        return set_err(h, TCW_ERR_INVALID_ARG, "template %u: t0 grid outside the array", k);
      if (!(d.tau_min > 0.0) || !(d.tau_max >= d.tau_min))
        return set_err(h, TCW_ERR_INVALID_ARG, "template %u: need 0 < tau_min <= tau_max", k);
      const uint32_t *g = t0s + d.t0_offset;
      if ((uint64_t)g[0] + d.TAtom / 2u < d.t0_data)
        return set_err(h, TCW_ERR_INVALID_ARG, "template %u: t0 grid starts before the data", k);
      for (uint32_t m = 1; m < d.N_t0; m++)
        if (g[m] < g[m - 1])
          return set_err(h, TCW_ERR_INVALID_ARG, "template %u: t0 grid must be non-decreasing", k);
      if (d.window != 0 && d.window != TCW_WINDOW_EXP && d.window != TCW_WINDOW_RECT)
        return set_err(h, TCW_ERR_INVALID_ARG, "template %u: invalid window type %u", k,
                       d.window);
      const bool rect = d.window == TCW_WINDOW_RECT;
      if ((double)g[d.N_t0 - 1] + (rect ? 1.0 : 3.0) * d.tau_max >= 4294967295.0)
        return set_err(h, TCW_ERR_OVERFLOW, "template %u: window end exceeds the u32 range", k);
      DiffTemplate t{};
      t.atom_off = d.atom_offset;
      t.t0_off = d.t0_offset;
      t.g = make_geom(d.numAtoms, d.TAtom, d.t0_data);
      t.N_t0 = d.N_t0;
      t.N_tau = d.N_tau;
      t.tau_min = d.tau_min;
      t.tau_max = d.tau_max;
      t.window = rect ? (uint32_t)TCW_WINDOW_RECT : (uint32_t)TCW_WINDOW_EXP;
      if (rect) {
        t.n_cg = (d.N_t0 + 31u) / 32u;
        row_groups += t.n_cg;
        t.p_off = p_rows;
        p_rows += (uint64_t)d.numAtoms + 1u;
        t.seg_off = b_rows;
        b_rows += ((uint64_t)d.numAtoms + 31u) / 32u;
        TemplateDev rt = make_tdev(d.numAtoms, d.TAtom, d.t0_data, TCW_WINDOW_RECT, d.N_t0, d.N_tau);
        rt.atom_off = t.atom_off;
        rt.p_off = t.p_off;
        ident.push_back((uint32_t)RT.size());
        RT.push_back(rt);
        S.max_rect_atoms = std::max(S.max_rect_atoms, d.numAtoms);
        rlist.push_back(k);
      } else {
        t.col_off = n_cols;
        n_cols += d.N_tau;
        elist.push_back(k);
        atom_rows = std::max<uint64_t>(atom_rows, d.atom_offset + d.numAtoms);
      }
      T[k] = t;
    }
    // largest templates first, so that those of a launch are of like size
    auto size_of = [&](uint32_t k) {
      const DiffTemplate &t = T[k];
      return ((uint64_t)t.N_tau + 31u) / 32u *
             (t.N_t0 / 16u + (uint64_t)t.g.numAtoms / kDiffAtomSeg + 1u);
    };
    std::stable_sort(elist.begin(), elist.end(),
                     [&](uint32_t a, uint32_t b) { return size_of(a) > size_of(b); });
    // groups of exponential templates within the workspace bound, one template
    // at least
    for (uint32_t y0 = 0; y0 < elist.size();) {
      uint32_t y1 = y0;
      uint64_t bytes = 0;
      while (y1 < elist.size() && y1 - y0 < kDiffGroupMax) {
        const DiffTemplate &t = T[elist[y1]];
        const uint64_t b =
            ((uint64_t)t.N_tau + 31u) / 32u * (diff_source_bytes(t) + diff_end_bytes(t));
        if (pass && y1 > y0 && bytes + b > kDiffGroupBytes) break;
        bytes += b;
        y1++;
      }
      DiffGroup g;
      diff_tile_group(h, T, elist, y0, y1, pass, cut, g, S.classes);
      S.groups.push_back(g);
      seg_floats = std::max(seg_floats, g.seg_floats);
      scr_floats = std::max(scr_floats, g.scr_floats);
      cend_floats = std::max(cend_floats, g.cend_floats);
      y0 = y1;
    }
    // rectangular tiles: as many column chunks per row group as give every
    // resident warp a tile, at least 16 columns each; where the row groups alone
    // keep the FP64 pipe busy (two warps per SM) 64 columns, as each chunk sums
    // its first window anew (forward / backward, noise: 500 templates of 1500
    // atoms, 4 x 128 cells 1.45 / 1.58 -> 1.07 / 1.40 ms; of 100 atoms, 128 x 32
    // 0.84 / 1.32 -> 0.67 / 1.07; 2000 of 480, 32 x 32 1.49 / 1.53 -> 1.29 / 1.42)
    const bool busy = row_groups >= (uint64_t)h->n_sms * 2u;
    const uint64_t rchunks =
        row_groups ? ((uint64_t)h->n_sms * 32u + row_groups - 1u) / row_groups : 1u;
    for (uint32_t k : rlist) {
      DiffTemplate &t = T[k];
      uint64_t nc = std::max<uint64_t>(1, std::min<uint64_t>(rchunks, (t.N_tau + 15u) / 16u));
      if (busy)
        nc = std::min<uint64_t>(nc, (t.N_tau + 63u) / 64u);
      t.chunk_rows = (uint32_t)((t.N_tau + nc - 1) / nc);
      t.n_chunk = (t.N_tau + t.chunk_rows - 1u) / t.chunk_rows;
      S.max_rect_tiles = std::max(S.max_rect_tiles, t.n_cg * t.n_chunk);
    }
    for (const std::vector<uint32_t> *l : {&elist, &rlist})
      for (uint32_t k : *l) {
        T[k].part_off = (uint32_t)n_tiles;
        T[k].n_parts = T[k].n_cg * T[k].n_chunk;
        S.max_parts = std::max(S.max_parts, T[k].n_parts);
        n_tiles += T[k].n_parts;
        if (n_tiles > 0xFFFFFFF0ull) return set_err(h, TCW_ERR_OVERFLOW, "too many tiles");
      }
  } catch (const std::bad_alloc &) {
    return set_err(h, TCW_ERR_ALLOC, "host allocation failed");
  }
  S.n_rect = (uint32_t)rlist.size();
  S.n_exp = (uint32_t)elist.size();
  S.p_rows = p_rows;
  Layout L;
  S.o_T = L.add(sizeof(DiffTemplate) * n);
  S.o_t0 = L.add(sizeof(uint32_t) * n_t0s);
  S.o_est = L.add(sizeof(uint32_t) * n);
  S.o_hot = L.add(sizeof(uint32_t) * S.groups.size());
  S.o_rlist = L.add(sizeof(uint32_t) * std::max<size_t>(1, rlist.size()));
  S.o_elist = L.add(sizeof(uint32_t) * std::max<size_t>(1, elist.size()));
  S.o_ident = L.add(sizeof(uint32_t) * ident.size());
  S.o_RT = L.add(sizeof(TemplateDev) * RT.size());
  const size_t ctl = L.total;
  S.o_parts = L.add(sizeof(DiffPartial) * n_tiles);
  S.o_need = L.add(sizeof(float) * n_tiles);
  S.o_cols = L.add(sizeof(ColConsts) * n_cols);
  S.seg_floats = seg_floats;
  S.o_seg = L.add(sizeof(float) * seg_floats);
  S.o_scratch = L.add(sizeof(float) * scr_floats);
  S.o_cend = L.add(sizeof(float) * cend_floats);
  S.o_P = L.add(sizeof(float) * kPrefixStride * p_rows);
  S.o_B64 = L.add(sizeof(double) * 8u * b_rows);
  S.o_D64 = pass == 1 ? L.add(sizeof(double) * 8u * std::max<uint64_t>(1, p_rows)) : 0;
  // the exponential templates' atoms in 32-byte rows, at their own row index
  S.o_A8 = S.n_exp ? L.add(sizeof(float) * 8u * std::max<uint64_t>(1, atom_rows)) : 0;
  S.total = L.total;
  int rc = ensure_ws(h, S.total);
  if (rc) return rc;
  rc = ensure_stage(h, ctl);
  if (rc) return rc;
  memcpy(h->h_stage + S.o_T, T.data(), sizeof(DiffTemplate) * n);
  memcpy(h->h_stage + S.o_t0, t0s, sizeof(uint32_t) * n_t0s);
  memset(h->h_stage + S.o_est, 0, sizeof(uint32_t) * n);
  memset(h->h_stage + S.o_hot, 0, sizeof(uint32_t) * S.groups.size());
  if (!rlist.empty()) {
    memcpy(h->h_stage + S.o_rlist, rlist.data(), sizeof(uint32_t) * rlist.size());
    memcpy(h->h_stage + S.o_ident, ident.data(), sizeof(uint32_t) * ident.size());
    memcpy(h->h_stage + S.o_RT, RT.data(), sizeof(TemplateDev) * RT.size());
  }
  if (!elist.empty()) memcpy(h->h_stage + S.o_elist, elist.data(), sizeof(uint32_t) * elist.size());
  TCW_CUDA(h, cudaMemcpyAsync(h->d_ws, h->h_stage, ctl, cudaMemcpyHostToDevice, h->stream));
  TCW_CUDA(h, cudaEventRecord(h->stage_ev, h->stream));
  h->stage_pending = true;
  return TCW_OK;
}

static int diff_prepare(tcw_handle *h, const tcw_diff_desc *desc, uint32_t n,
                        const uint32_t *t0s, uint64_t n_t0s, int pass, DiffSetup &S) {
  int rc = diff_setup(h, desc, n, t0s, n_t0s, pass, true, S);
  // without the memory for segment sums (up to 1 GiB): whole columns
  if (rc == TCW_ERR_ALLOC && S.seg_floats) rc = diff_setup(h, desc, n, t0s, n_t0s, pass, false, S);
  return rc;
}

static DiffLaunch diff_launch(tcw_handle *h, const DiffSetup &S, const float *d_atoms,
                              double temperature) {
  DiffLaunch L{};
  L.T = reinterpret_cast<const DiffTemplate *>(h->d_ws + S.o_T);
  L.atoms = d_atoms;
  L.t0s = reinterpret_cast<const uint32_t *>(h->d_ws + S.o_t0);
  L.temp = temperature;
  L.parts = reinterpret_cast<DiffPartial *>(h->d_ws + S.o_parts);
  L.cols = reinterpret_cast<ColConsts *>(h->d_ws + S.o_cols);
  L.seg = reinterpret_cast<float *>(h->d_ws + S.o_seg);
  L.need = reinterpret_cast<float *>(h->d_ws + S.o_need);
  L.est = reinterpret_cast<uint32_t *>(h->d_ws + S.o_est);
  L.hot_groups = reinterpret_cast<uint32_t *>(h->d_ws + S.o_hot);
  L.n_sms = (uint32_t)h->n_sms;
  L.scratch = reinterpret_cast<float *>(h->d_ws + S.o_scratch);
  L.cend = reinterpret_cast<float *>(h->d_ws + S.o_cend);
  L.rect_list = reinterpret_cast<const uint32_t *>(h->d_ws + S.o_rlist);
  L.n_rect = S.n_rect;
  L.rect_ident = reinterpret_cast<const uint32_t *>(h->d_ws + S.o_ident);
  L.rect_T = reinterpret_cast<const TemplateDev *>(h->d_ws + S.o_RT);
  L.max_rect_tiles = S.max_rect_tiles;
  L.max_rect_atoms = S.max_rect_atoms;
  L.P = reinterpret_cast<float *>(h->d_ws + S.o_P);
  L.B64 = reinterpret_cast<double *>(h->d_ws + S.o_B64);
  L.D64 = S.o_D64 ? reinterpret_cast<double *>(h->d_ws + S.o_D64) : nullptr;
  L.atoms8 = S.o_A8 ? reinterpret_cast<float *>(h->d_ws + S.o_A8) : nullptr;
  L.exp_list = reinterpret_cast<const uint32_t *>(h->d_ws + S.o_elist);
  L.n_exp = S.n_exp;
  return L;
}

int tcw_map_forward(tcw_handle *h, const tcw_diff_desc *desc, uint32_t n_templates,
                    const float *d_atoms, const uint32_t *t0s, uint64_t n_t0s,
                    double temperature, double *d_lnBtSG, double *d_softmax2F) {
  if (!h) return TCW_ERR_INVALID_ARG;
  if (!d_atoms || !d_lnBtSG || !d_softmax2F)
    return set_err(h, TCW_ERR_INVALID_ARG, "null device pointer");
  if (!(temperature > 0.0)) return set_err(h, TCW_ERR_INVALID_ARG, "temperature must be > 0");
  int rc = set_device(h);
  if (rc) return rc;
  DiffSetup S;
  rc = diff_prepare(h, desc, n_templates, t0s, n_t0s, 0, S);
  if (rc) return rc;
  DiffLaunch L = diff_launch(h, S, d_atoms, temperature);
  TCW_CUDA(h, launch_diff(0, L, S.groups.data(), (uint32_t)S.groups.size(), S.classes.data(),
                          h->stream, h->side_stream, h->fork_ev, h->join_ev));
  TCW_CUDA(h, launch_diff_finalize(L.T, n_templates, S.max_parts, L.parts, temperature, d_lnBtSG,
                                   d_softmax2F, h->stream));
  return TCW_OK;
}

int tcw_map_backward(tcw_handle *h, const tcw_diff_desc *desc, uint32_t n_templates,
                     const float *d_atoms, const uint32_t *t0s, uint64_t n_t0s,
                     double temperature, const double *d_lnBtSG, const double *d_softmax2F,
                     const double *d_grad_lnBtSG, const double *d_grad_softmax2F,
                     double *d_grad_atoms, uint64_t n_atom_rows, double *d_grad_tau) {
  if (!h) return TCW_ERR_INVALID_ARG;
  if (!d_atoms || !d_lnBtSG || !d_softmax2F || !d_grad_lnBtSG || !d_grad_softmax2F ||
      !d_grad_atoms || !d_grad_tau)
    return set_err(h, TCW_ERR_INVALID_ARG, "null device pointer");
  if (!(temperature > 0.0)) return set_err(h, TCW_ERR_INVALID_ARG, "temperature must be > 0");
  for (uint32_t k = 0; desc && k < n_templates; k++)
    if (desc[k].atom_offset + desc[k].numAtoms > n_atom_rows)
      return set_err(h, TCW_ERR_INVALID_ARG, "template %u: atoms outside the gradient array", k);
  int rc = set_device(h);
  if (rc) return rc;
  DiffSetup S;
  rc = diff_prepare(h, desc, n_templates, t0s, n_t0s, 1, S);
  if (rc) return rc;
  DiffLaunch L = diff_launch(h, S, d_atoms, temperature);
  L.lnZ1 = d_lnBtSG;
  L.lnZ2 = d_softmax2F;
  L.gB = d_grad_lnBtSG;
  L.gS = d_grad_softmax2F;
  L.grad_atoms = d_grad_atoms;
  L.grad_tau = d_grad_tau;
  TCW_CUDA(h, cudaMemsetAsync(d_grad_atoms, 0, sizeof(double) * 7u * n_atom_rows, h->stream));
  TCW_CUDA(h, cudaMemsetAsync(d_grad_tau, 0, sizeof(double) * 2u * n_templates, h->stream));
  if (S.n_rect)
    TCW_CUDA(h, cudaMemsetAsync(L.D64, 0, sizeof(double) * 8u * S.p_rows, h->stream));
  TCW_CUDA(h, launch_diff(1, L, S.groups.data(), (uint32_t)S.groups.size(), S.classes.data(),
                          h->stream, h->side_stream, h->fork_ev, h->join_ev));
  return TCW_OK;
}

int tcw_plan_run_host(tcw_handle *h, tcw_plan *p, const float *atoms, tcw_result *results) {
  if (!h || !p) return TCW_ERR_INVALID_ARG;
  if (!atoms || !results) return set_err(h, TCW_ERR_INVALID_ARG, "null host pointer");
  int rc = set_device(h);
  if (rc) return rc;
  const size_t abytes = sizeof(float) * 7u * (size_t)p->n_atom_rows;
  if (!p->d_atoms_in) {
    void *a = nullptr, *r = nullptr;
    rc = ws_alloc(h, &a, std::max<size_t>(abytes, 16));
    if (rc) return rc;
    rc = ws_alloc(h, &r, sizeof(tcw_result) * p->n_templates);
    if (rc) {
      cudaFree(a);
      return rc;
    }
    p->d_atoms_in = static_cast<float *>(a);
    p->d_res_out = static_cast<tcw_result *>(r);
  }
  TCW_CUDA(h, cudaMemcpyAsync(p->d_atoms_in, atoms, abytes, cudaMemcpyHostToDevice, h->stream));
  rc = tcw_plan_run(h, p, p->d_atoms_in, p->d_res_out, 1);
  if (rc) return rc;
  TCW_CUDA(h, cudaMemcpyAsync(results, p->d_res_out, sizeof(tcw_result) * p->n_templates,
                              cudaMemcpyDeviceToHost, h->stream));
  TCW_CUDA(h, cudaStreamSynchronize(h->stream));
  return TCW_OK;
}

int tcw_plan_run_host_async(tcw_handle *h, tcw_plan *p, const float *atoms,
                            tcw_result *results) {
  if (!h || !p) return TCW_ERR_INVALID_ARG;
  if (!atoms || !results) return set_err(h, TCW_ERR_INVALID_ARG, "null host pointer");
  if (p->flags & TCW_FLAG_POSTERIORS)
    return set_err(h, TCW_ERR_INVALID_ARG,
                   "posteriors need the maps: run the plan with tcw_plan_run_maps");
  if (p->device != h->device)
    return set_err(h, TCW_ERR_INVALID_ARG, "plan and handle are on different devices");
  int rc = set_device(h);
  if (rc) return rc;
  const size_t abytes = sizeof(float) * 7u * (size_t)p->n_atom_rows;
  if (!p->d_atoms_in) {
    void *a = nullptr, *r = nullptr;
    rc = ws_alloc(h, &a, std::max<size_t>(abytes, 16));
    if (rc) return rc;
    rc = ws_alloc(h, &r, sizeof(tcw_result) * p->n_templates);
    if (rc) {
      cudaFree(a);
      return rc;
    }
    p->d_atoms_in = static_cast<float *>(a);
    p->d_res_out = static_cast<tcw_result *>(r);
  }
  // the upload may start as soon as the previous run has read its atoms, so
  // it overlaps that run's map kernels
  if (h->consumed_pending) {
    TCW_CUDA(h, cudaStreamWaitEvent(h->copy_stream, h->consumed_ev, 0));
    TCW_CUDA(h, cudaStreamWaitEvent(h->copy_stream, h->consumed_side_ev, 0));
  }
  TCW_CUDA(h, cudaMemcpyAsync(p->d_atoms_in, atoms, abytes, cudaMemcpyHostToDevice,
                              h->copy_stream));
  TCW_CUDA(h, cudaEventRecord(h->copied_ev, h->copy_stream));
  TCW_CUDA(h, cudaStreamWaitEvent(h->stream, h->copied_ev, 0));
  // the compensated map kernels read only the prefix and repacked rows; the
  // uncompensated exp kernel reads the atoms themselves
  const bool maps_read_atoms = p->prec == kPrecPlain32;
  rc = plan_enqueue(h, p, p->d_atoms_in, p->d_res_out, nullptr,
                    maps_read_atoms ? nullptr : h->consumed_ev,
                    maps_read_atoms ? nullptr : h->consumed_side_ev);
  if (rc) return rc;
  if (maps_read_atoms) {
    TCW_CUDA(h, cudaEventRecord(h->consumed_ev, h->stream));
    TCW_CUDA(h, cudaEventRecord(h->consumed_side_ev, h->stream));
  }
  h->consumed_pending = true;
  TCW_CUDA(h, cudaMemcpyAsync(results, p->d_res_out, sizeof(tcw_result) * p->n_templates,
                              cudaMemcpyDeviceToHost, h->stream));
  return TCW_OK;
}

int tcw_plan_run_maps_host(tcw_handle *h, tcw_plan *p, const float *atoms, tcw_result *results,
                           float *maps) {
  if (!h || !p) return TCW_ERR_INVALID_ARG;
  if (!atoms || !results || !maps) return set_err(h, TCW_ERR_INVALID_ARG, "null host pointer");
  int rc = set_device(h);
  if (rc) return rc;
  const size_t abytes = sizeof(float) * 7u * (size_t)p->n_atom_rows;
  const size_t mbytes = sizeof(float) * (size_t)p->n_cells;
  if (!p->d_atoms_in) {
    void *a = nullptr, *r = nullptr;
    rc = ws_alloc(h, &a, std::max<size_t>(abytes, 16));
    if (rc) return rc;
    rc = ws_alloc(h, &r, sizeof(tcw_result) * p->n_templates);
    if (rc) {
      cudaFree(a);
      return rc;
    }
    p->d_atoms_in = static_cast<float *>(a);
    p->d_res_out = static_cast<tcw_result *>(r);
  }
  if (!p->d_maps_out) {
    void *m = nullptr;
    rc = ws_alloc(h, &m, std::max<size_t>(mbytes, 16));
    if (rc) return rc;
    p->d_maps_out = static_cast<float *>(m);
  }
  TCW_CUDA(h, cudaMemcpyAsync(p->d_atoms_in, atoms, abytes, cudaMemcpyHostToDevice, h->stream));
  rc = plan_run(h, p, p->d_atoms_in, p->d_res_out, p->d_maps_out, 1);
  if (rc) return rc;
  TCW_CUDA(h, cudaMemcpyAsync(results, p->d_res_out, sizeof(tcw_result) * p->n_templates,
                              cudaMemcpyDeviceToHost, h->stream));
  TCW_CUDA(h, cudaMemcpyAsync(maps, p->d_maps_out, mbytes, cudaMemcpyDeviceToHost, h->stream));
  TCW_CUDA(h, cudaStreamSynchronize(h->stream));
  return TCW_OK;
}

int tcw_map_batched(tcw_handle *h, const tcw_template_desc *desc, uint32_t n_templates,
                    const uint32_t *t0s, uint64_t n_t0s, const uint32_t *taus, uint64_t n_taus,
                    const float *atoms_concat, const tcw_tile_config *cfg, float *max2F,
                    int64_t *argmax, double *lnBtSG) {
  if (!h) return TCW_ERR_INVALID_ARG;
  if (!atoms_concat || !max2F || !argmax || !lnBtSG)
    return set_err(h, TCW_ERR_INVALID_ARG, "null host pointer");
  tcw_plan *p = nullptr;
  int rc = tcw_plan_create(h, desc, n_templates, t0s, n_t0s, taus, n_taus, cfg, TCW_FLAG_LNBTSG,
                           &p);
  if (rc) return rc;
  std::vector<tcw_result> res;
  try {
    res.resize(n_templates);
  } catch (const std::bad_alloc &) {
    tcw_plan_destroy(p);
    return set_err(h, TCW_ERR_ALLOC, "host allocation failed");
  }
  rc = tcw_plan_run_host(h, p, atoms_concat, res.data());
  tcw_plan_destroy(p);
  if (rc) return rc;
  for (uint32_t k = 0; k < n_templates; k++) {
    max2F[k] = 2.0f * res[k].maxF;
    argmax[k] = res[k].argmax;
    lnBtSG[k] = res[k].lnBtSG;
  }
  return TCW_OK;
}

int tcw_debug_check_failures(uint32_t *count) {
  if (!count) return TCW_ERR_INVALID_ARG;
  uint64_t n = (uint64_t)dcheck_failures_kernels() + dcheck_failures_diff() +
               dcheck_failures_f64() + dcheck_failures_noalloc();
  *count = (uint32_t)std::min<uint64_t>(n, 0xFFFFFFFFull);
#if defined(TCW_DEBUG_CHECKS)
  return TCW_OK;
#else
  return TCW_ERR_UNSUPPORTED;
#endif
}

int tcw_map_f64(tcw_handle *h, const float *d_atoms, uint32_t numAtoms, uint32_t TAtom,
                uint32_t t0_data, int window, const uint32_t *d_t0s, uint32_t N_t0,
                const uint32_t *d_taus, uint32_t N_tau, const uint32_t *rows, uint32_t n_rows,
                double *d_F, double *d_cond) {
  if (!h) return TCW_ERR_INVALID_ARG;
  if (!d_atoms || !d_t0s || !d_taus || !d_F)
    return set_err(h, TCW_ERR_INVALID_ARG, "null device pointer");
  if (!valid_window(window))
    return set_err(h, TCW_ERR_INVALID_ARG,
                   "invalid window type %d: TCW_WINDOW_RECT or TCW_WINDOW_EXP", window);
  int rc = check_geometry(h, numAtoms, TAtom, t0_data, N_t0, N_tau);
  if (rc) return rc;
  if (!rows && n_rows != N_t0)
    return set_err(h, TCW_ERR_INVALID_ARG, "without a row list n_rows must equal N_t0");
  if (n_rows == 0) return set_err(h, TCW_ERR_INVALID_ARG, "no rows requested");
  if (rows)
    for (uint32_t k = 0; k < n_rows; k++)
      if (rows[k] >= N_t0)
        return set_err(h, TCW_ERR_INVALID_ARG, "row %u (entry %u) outside the t0 grid of %u",
                       rows[k], k, N_t0);
  rc = set_device(h);
  if (rc) return rc;
  const uint32_t *d_rows = nullptr;
  if (rows) {
    const size_t bytes = sizeof(uint32_t) * (size_t)n_rows;
    rc = ensure_ws(h, bytes);
    if (rc) return rc;
    rc = ensure_stage(h, bytes);
    if (rc) return rc;
    memcpy(h->h_stage, rows, bytes);
    TCW_CUDA(h, cudaMemcpyAsync(h->d_ws, h->h_stage, bytes, cudaMemcpyHostToDevice, h->stream));
    TCW_CUDA(h, cudaEventRecord(h->stage_ev, h->stream));
    h->stage_pending = true;
    d_rows = reinterpret_cast<const uint32_t *>(h->d_ws);
  }
  const Geom g = make_geom(numAtoms, TAtom, t0_data);
  TCW_CUDA(h, launch_map_f64(window, d_atoms, g, d_t0s, d_taus, N_tau, d_rows, n_rows, d_F,
                             d_cond, h->stream));
  return TCW_OK;
}

}  // extern "C"
