"""Workloads of the transient F-statistic map, as programs use it.

Each case goes through a public entry point:

* ``dropin``  one map per call through the PyFstat-facing dispatcher
  (``call_compute_transient_fstat_map('b200', ...)``): host atoms in, the map,
  the ML point, lnBtSG and the posterior estimates back;
* ``host``    one map per call from host arrays on an explicit grid
  (``Handle.map_plain_host``; log-spaced taus);
* ``plain``   one map on device buffers (``Handle.map_plain``), map written;
* ``batch``   many templates in one launch, no maps (``TransientMapBatch``);
* ``maps``    many templates with their maps and posteriors
  (``Plan.run_maps`` of a plan with ``TCW_FLAG_POSTERIORS``);
* ``grad``    lnBtSG and the soft maximum of 2F with their gradients
  (``autograd.transient_stats``, forward and backward);
* ``grid``    a whole transient grid search over Doppler points
  (``search.TransientGridBatch``).

Data are the synthetic atoms of ``pyfstat_gb300.synth`` (the same antenna
patterns, noise, injection and gaps), made on the GPU where they are many.
"""

import math

import numpy as np
import torch

from pyfstat_gb300 import _lib, synth
from pyfstat_gb300 import tcw_fstat_map_funcs as tcw
from pyfstat_gb300.autograd import DiffBatch, transient_stats
from pyfstat_gb300.batched import TransientMapBatch
from pyfstat_gb300.search import TransientGridBatch
from pyfstat_gb300.window import transientWindowRange_t

T0 = synth.T0_DEFAULT
TSFT = synth.TSFT_DEFAULT
RECT, EXP = 1, 2


def listed():
    return [
        # one day of one detector, the geometry of PyFstat's own test of this
        # path: the smallest map a search asks for, one call per Doppler point
        dict(name="dropin_day_rect", kind="dropin", window=RECT, nsft=48, ndet=1, gap=0.0,
             n_t0=47, n_tau=47),
        # ten days, every start and every duration in SFT steps
        dict(name="dropin_480_rect", kind="dropin", window=RECT, nsft=480, ndet=1, gap=0.0,
             n_t0=480, n_tau=480),
        # two detectors merged, exponential windows, log-spaced taus beyond
        # the data span
        dict(name="host_480_exp_log", kind="host", window=EXP, nsft=480, ndet=2, gap=0.0,
             n_t0=480, n_tau=512),
        # one year of data on a fine grid, the map kept on the device
        dict(name="plain_year_rect", kind="plain", window=RECT, nsft=17532, ndet=1, gap=0.05,
             n_t0=8192, n_tau=4096, post=False),
        dict(name="plain_year_exp", kind="plain", window=EXP, nsft=17532, ndet=2, gap=0.05,
             n_t0=8192, n_tau=4096, post=False),
        # a handful of Doppler points of ragged sizes, mixed windows
        dict(name="batch_24", kind="batch", n=24, nsft_max=1500, grid_max=600),
        # a full search step: the library's benchmark workload
        dict(name="batch_4096", kind="batch", n=4096, nsft_max=4000, grid_max=2048),
        # templates with the maps and the t0 / tau posteriors
        dict(name="maps_96_posteriors", kind="maps", n=96, nsft_max=4000, grid_max=2048),
        # following up one candidate by gradients
        dict(name="grad_1_exp", kind="grad", window=EXP, n=1, nsft=2000, ndet=2, n_t0=1024,
             n_tau=1024),
        # a few candidates of odd sizes, rectangular windows
        dict(name="grad_7_rect", kind="grad", window=RECT, n=7, nsft=1499, ndet=1, n_t0=777,
             n_tau=611),
        # gradients of a batch of templates
        dict(name="grad_24_exp", kind="grad", window=EXP, n=24, nsft=2000, ndet=2, n_t0=1024,
             n_tau=1024),
        # a grid search with transient Bayes factors, from host atoms
        dict(name="grid_32_rect", kind="grid", window=RECT, n=32, nsft=480, n_t0=240,
             n_tau=240),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "host", "plain", "plain", "batch", "batch", "maps", "grad",
                       "grad", "grid"])
    window = rng.choice([RECT, EXP])
    if kind in ("dropin", "host"):
        nsft = _log(rng, 40, 2000)
        return dict(kind=kind, window=EXP if kind == "host" else window, nsft=nsft,
                    ndet=rng.choice([1, 2]), gap=rng.choice([0.0, round(rng.random() * 0.3, 3)]),
                    n_t0=_log(rng, 20, min(700, nsft)), n_tau=_log(rng, 20, min(700, nsft)))
    if kind == "plain":
        return dict(kind=kind, window=window, nsft=_log(rng, 100, 17532),
                    ndet=rng.choice([1, 2]), gap=round(rng.random() * 0.3, 3),
                    n_t0=_log(rng, 64, 6000), n_tau=_log(rng, 64, 4096),
                    post=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 2, 1500), nsft_max=_log(rng, 300, 4000),
                    grid_max=_log(rng, 100, 2048))
    if kind == "maps":
        return dict(kind=kind, n=_log(rng, 2, 90), nsft_max=_log(rng, 300, 4000),
                    grid_max=_log(rng, 100, 2000))
    if kind == "grad":
        return dict(kind=kind, window=window, n=_log(rng, 1, 16), nsft=_log(rng, 100, 2000),
                    ndet=rng.choice([1, 2]), n_t0=_log(rng, 50, 1000),
                    n_tau=_log(rng, 50, 1000))
    nsft = _log(rng, 60, 600)
    return dict(kind="grid", window=window, n=_log(rng, 3, 32), nsft=nsft,
                n_t0=_log(rng, 20, min(300, nsft)), n_tau=_log(rng, 20, min(300, nsft)))


# ------------------------------------------------------------------ inputs


def _atoms_cuda(seed, nsfts, gaps, ndet):
    """Binned atoms of several templates, (sum nsft, 7) float32 on the GPU,
    distributed as synth.detector_atoms (bins of gap SFTs are zero)."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    n, nmax = len(nsfts), int(max(nsfts))
    ns = torch.as_tensor(np.asarray(nsfts), device=dev)[:, None]
    gap = torch.as_tensor(np.asarray(gaps, np.float64), device=dev)[:, None]
    k = torch.arange(nmax, device=dev, dtype=torch.float64)[None, :]
    out = torch.zeros((n, nmax, 7), dtype=torch.float32, device=dev)
    om = 2.0 * math.pi / synth.SIDEREAL_DAY
    for x in range(ndet):
        t = T0 + (x * TSFT) // 3 + k * TSFT
        ph = 2.0 * math.pi * torch.rand((2, n, 1), generator=g, device=dev, dtype=torch.float64)
        a = 0.4 + 0.3 * torch.cos(om * t + ph[0])
        b = 0.3 * torch.sin(om * t + ph[1])
        z = torch.randn((4, n, nmax), generator=g, device=dev, dtype=torch.float64)
        sig = ((k >= synth.INJECT_RANGE[0]) & (k <= synth.INJECT_RANGE[1])).to(torch.float64)
        z[0] += 3.0 * a * sig
        z[2] += 3.0 * b * sig
        keep = torch.rand((n, nmax), generator=g, device=dev) >= gap
        keep |= (k == 0) | (k == ns - 1)
        a2, b2, ab = (v.to(torch.float32) for v in (a * a, b * b, a * b))
        sa, sb = torch.sqrt(a2.double() / 2.0), torch.sqrt(b2.double() / 2.0)
        row = torch.stack((a2, b2, ab, (sa * z[0]).float(), (sa * z[1]).float(),
                           (sb * z[2]).float(), (sb * z[3]).float()), dim=2)
        out += torch.where(keep[:, :, None], row, torch.zeros_like(row))
    return out[k < ns].contiguous()


def _uniform(start, step, n):
    return (np.uint64(start) + np.arange(n, dtype=np.uint64) * np.uint64(step)).astype(np.uint32)


def _span_grid(nsft, n_t0, n_tau):
    """Uniform grid over the data span: (t0s, taus, dt0, dtau)."""
    span = nsft * TSFT
    dt0 = max(1, span // n_t0)
    dtau = max(1, (span - TSFT) // max(1, n_tau - 1))
    return _uniform(T0, dt0, n_t0), _uniform(TSFT, dtau, n_tau), dt0, dtau


def _batch_geometry(case):
    """SFT counts, gap fractions and grid sizes of a batch: fixed by the case,
    as a search's templates share their data span and grid set-up."""
    r = np.random.default_rng([case["n"], case["nsft_max"], case["grid_max"]])
    n = case["n"]
    nsft = r.integers(max(20, case["nsft_max"] // 20), case["nsft_max"] + 1, n)
    gaps = r.uniform(0.0, 0.3, n)
    nt0 = r.integers(max(16, case["grid_max"] // 8), case["grid_max"] + 1, n)
    ntau = r.integers(max(16, case["grid_max"] // 8), case["grid_max"] + 1, n)
    return nsft, gaps, nt0, ntau


def _dropin_range(case):
    """Starts over the data and durations from one SFT up, in whole SFTs
    where the grid is as fine as the data."""
    dt0 = max(1, case["nsft"] // case["n_t0"]) * TSFT
    dtau = max(1, case["nsft"] // case["n_tau"]) * TSFT
    return dict(type=case["window"], t0=T0, t0Band=(case["n_t0"] - 1) * dt0, dt0=dt0, tau=TSFT,
                tauBand=(case["n_tau"] - 1) * dtau, dtau=dtau)


def _grad_tau(case):
    """Durations of at least a quarter of a day up to a good part of the data."""
    lo = 12.0 * TSFT + 75.0
    return lo, lo + 0.6 * case["nsft"] * TSFT


def _i32(a):
    return torch.from_numpy(a.view(np.int32)).cuda()


# What a program sets up once and keeps: the version's features and context,
# one library handle on one stream of its own (graphs cannot be captured on
# the legacy default stream), and one handle for the gradients, which run on
# torch's current stream.
_PROGRAM = {}


def _features():
    if "features" not in _PROGRAM:
        _PROGRAM["features"], _PROGRAM["context"] = tcw.init_transient_fstat_map_features("b200")
    return _PROGRAM["features"]


def _handle():
    if "handle" not in _PROGRAM:
        _PROGRAM["stream"] = torch.cuda.Stream()
        _PROGRAM["handle"] = _lib.Handle(torch.cuda.current_device())
        _PROGRAM["handle"].set_stream(_PROGRAM["stream"].cuda_stream)
    return _PROGRAM["handle"]


def _grad_handle():
    if "grad_handle" not in _PROGRAM:
        _PROGRAM["grad_handle"] = _lib.Handle(torch.cuda.current_device())
    return _PROGRAM["grad_handle"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        _features()
        multi = synth.multi_detector_atoms(seed, case["nsft"], case["ndet"],
                                           gap_frac=case["gap"])
        return dict(kind=kind, multi=multi, range=_dropin_range(case))
    if kind == "host":
        _, A = synth.merged_atoms(seed, case["nsft"], case["ndet"], gap_frac=case["gap"])
        dt0 = max(1, case["nsft"] // case["n_t0"]) * TSFT
        return dict(kind=kind, handle=_handle(), A=A, window=case["window"],
                    t0s=_uniform(T0, dt0, case["n_t0"]),
                    taus=synth.log_tau_grid(TSFT, 3 * case["nsft"], case["n_tau"]))
    if kind == "plain":
        A = _atoms_cuda(seed, [case["nsft"]], [case["gap"]], case["ndet"])
        t0s, taus, _, _ = _span_grid(case["nsft"], case["n_t0"], case["n_tau"])
        flags = _lib.TCW_FLAG_LNBTSG | (_lib.TCW_FLAG_POSTERIORS if case["post"] else 0)
        return dict(kind=kind, handle=_handle(), A=A, window=case["window"], t0s=_i32(t0s),
                    taus=_i32(taus), flags=flags,
                    F=torch.empty((t0s.size, taus.size), dtype=torch.float32, device="cuda"),
                    res=torch.zeros((1, 5), dtype=torch.float64, device="cuda"))
    if kind in ("batch", "maps"):
        nsft, gaps, nt0, ntau = _batch_geometry(case)
        d_atoms = _atoms_cuda(seed, nsft, gaps, 1)
        host = d_atoms.cpu().numpy()
        ends = np.cumsum(nsft)
        templates = []
        for j in range(case["n"]):
            t0s, taus, _, _ = _span_grid(int(nsft[j]), int(nt0[j]), int(ntau[j]))
            templates.append(dict(atoms=host[ends[j] - nsft[j]:ends[j]], TAtom=TSFT, t0_data=T0,
                                  window=RECT if j % 2 == 0 else EXP, t0s=t0s, taus=taus))
        flags = _lib.TCW_FLAG_LNBTSG | (_lib.TCW_FLAG_POSTERIORS if kind == "maps" else 0)
        b = TransientMapBatch(templates, handle=_handle(), flags=flags)
        st = dict(kind=kind, batch=b, atoms=d_atoms,
                  res=torch.zeros((case["n"], 5), dtype=torch.float64, device="cuda"))
        if kind == "maps":
            st["maps"] = torch.empty(b.n_cells, dtype=torch.float32, device="cuda")
        return st
    if kind == "grad":
        n, nsft = case["n"], case["nsft"]
        A = _atoms_cuda(seed, [nsft] * n, [0.0] * n, case["ndet"])
        host = A.cpu().numpy()
        t0s = _uniform(T0 + 450, max(1, nsft * TSFT // case["n_t0"]), case["n_t0"])
        lo, hi = _grad_tau(case)
        b = DiffBatch([dict(atoms=host[j * nsft:(j + 1) * nsft], TAtom=TSFT, t0_data=T0, t0s=t0s,
                            N_tau=case["n_tau"], window=case["window"]) for j in range(n)],
                      handle=_grad_handle())
        one = torch.ones(n, dtype=torch.float64, device="cuda")
        return dict(kind=kind, batch=b, A=A.requires_grad_(),
                    tau_min=torch.full((n,), lo, dtype=torch.float64, requires_grad=True),
                    tau_max=torch.full((n,), hi, dtype=torch.float64, requires_grad=True),
                    one=one)
    points = [synth.multi_detector_atoms(100003 * (seed % 10007) + j, case["nsft"], 2,
                                         gap_frac=0.1) for j in range(case["n"])]
    return dict(kind=kind, points=points, range=_dropin_range(case))


# ------------------------------------------------------------------ one pass


def _records(res):
    """The fields of device result records, as views."""
    words = res.view(torch.int64)
    return dict(lnBtSG=res[:, 0], argmax=words[:, 1], maxF=res.view(torch.float32)[:, 8],
                t0_mp=words[:, 2], tau_mp=words[:, 3])


def run(st):
    kind = st["kind"]
    if kind == "dropin":
        m, _ = tcw.call_compute_transient_fstat_map(
            "b200", _features(), st["multi"], transientWindowRange_t(**st["range"]),
            BtSG=True)
        return dict(F=m.F_mn, maxF=m.maxF, t0_ML=m.t0_ML, tau_ML=m.tau_ML, lnBtSG=m.lnBtSG,
                    t0_MP=m.t0_MP, tau_MP=m.tau_MP)
    if kind == "host":
        F, r = st["handle"].map_plain_host(
            st["A"], TSFT, T0, st["window"], st["t0s"], st["taus"],
            flags=_lib.TCW_FLAG_LNBTSG | _lib.TCW_FLAG_POSTERIORS)
        return dict(F=F, maxF=float(r["maxF"]), argmax=int(r["argmax"]),
                    lnBtSG=float(r["lnBtSG"]), t0_mp=int(r["t0_mp_idx"]),
                    tau_mp=int(r["tau_mp_idx"]))
    if kind == "plain":
        st["handle"].map_plain(st["A"], st["A"].shape[0], TSFT, T0, st["window"], st["t0s"],
                               st["t0s"].shape[0], st["taus"], st["taus"].shape[0], st["F"],
                               st["res"], flags=st["flags"])
        return dict(F=st["F"], **_records(st["res"]))
    if kind == "batch":
        st["batch"].run_device(st["atoms"], st["res"])
        return _records(st["res"])
    if kind == "maps":
        st["batch"].plan.run_maps(st["atoms"], st["res"], st["maps"])
        return dict(maps=st["maps"], **_records(st["res"]))
    if kind == "grad":
        lnB, soft = transient_stats(st["A"], st["tau_min"], st["tau_max"], st["batch"])
        ga, g0, g1 = torch.autograd.grad((lnB, soft), (st["A"], st["tau_min"], st["tau_max"]),
                                         (st["one"], st["one"]))
        return dict(lnBtSG=lnB.detach(), softmax2F=soft.detach(), grad_atoms=ga, grad_tau_min=g0,
                    grad_tau_max=g1)
    out = TransientGridBatch(st["points"], transientWindowRange_t(**st["range"]), BtSG=True).run()
    return {k: np.ascontiguousarray(out[k]) for k in out.dtype.names}


def _cells(case):
    if case["kind"] in ("batch", "maps"):
        nsft, _, nt0, ntau = _batch_geometry(case)
        c = nt0.astype(np.int64) * ntau
        return int(nsft.sum()), int(c[0::2].sum()), int(c[1::2].sum()), int(case["n"])
    n = case.get("n", 1)
    c = n * case["n_t0"] * case["n_tau"]
    rect = case["window"] == RECT
    ndet = 2 if case["kind"] == "grid" else 1
    return n * case["nsft"] * ndet, c if rect else 0, 0 if rect else c, n


def work(case):
    """Each atom (28 bytes) read once, results and, where they are asked for,
    maps and gradients written once; FP32 operations per cell of the plain
    formulae (34 rectangular, 55 exponential; a gradient pass evaluates every
    cell twice and adds its derivatives)."""
    atoms, rect, exp, n = _cells(case)
    nbytes = 28.0 * atoms + 40.0 * n
    flops = 34.0 * rect + 55.0 * exp
    if case["kind"] in ("dropin", "host", "plain", "maps"):
        nbytes += 4.0 * (rect + exp)
    if case["kind"] == "grad":
        nbytes += 28.0 * atoms + 28.0 * atoms
        flops = 2.0 * flops + 60.0 * (rect + exp)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ 64 bits


class _Windows64:
    """Window sums and F of one template in 64 bits: prefix sums for
    rectangular windows, E(i) = x(i) + r^k E(i+1) per tau column for
    exponential ones.  taus are real; t0s start at or after the data."""

    def __init__(self, A, window, t0s, taus, want_v=False):
        dev = A.device
        self.A = A.double()
        self.N = N = A.shape[0]
        self.window = window
        t0 = torch.as_tensor(np.asarray(t0s, np.float64), device=dev) - T0
        tau = torch.as_tensor(np.asarray(taus, np.float64), device=dev)
        reach = tau if window == RECT else 3.0 * tau
        start = torch.floor((t0 + TSFT // 2) / TSFT).clamp(max=N - 1)
        end = (torch.floor((t0[:, None] + reach[None, :] + TSFT // 2) / TSFT) - 1).clamp(0, N - 1)
        if window == EXP:
            start = torch.maximum(start, torch.ceil(t0 / TSFT))
            end = torch.minimum(end, torch.floor((t0[:, None] + reach[None, :]) / TSFT))
        self.lo = start.long()
        self.top = end.long() + 1
        self.any = self.lo[:, None] < self.top
        nz = torch.cat((torch.zeros(1, dtype=torch.long, device=dev),
                        torch.cumsum((A[:, 0] != 0) | (A[:, 1] != 0), 0)))
        lo_in = self.lo.clamp(max=N)
        self.any &= nz[self.top] > nz[lo_in][:, None]
        self.tau = tau
        W, V = [], []
        if window == RECT:
            P = torch.cat((torch.zeros((1, 7), dtype=torch.float64, device=dev),
                           torch.cumsum(self.A, 0)))
            for c in range(7):
                W.append(P[:, c][self.top] - P[:, c][lo_in][:, None])
        else:
            L = (self.top - self.lo[:, None]).clamp(min=0).double()
            for c in range(7):
                k = 2.0 if c < 3 else 1.0
                r = torch.exp(-k * TSFT / tau)
                E = torch.zeros((N + 1, tau.numel()), dtype=torch.float64, device=dev)
                x = self.A[:, c].contiguous()
                for i in range(N - 1, -1, -1):
                    torch.addcmul(x[i].expand_as(r), r, E[i + 1], out=E[i])
                rl = torch.exp(-k * TSFT / tau * L)
                Et = E.gather(0, self.top)
                W.append(E[lo_in] - rl * Et)
                if want_v:  # sum (i - lo) x(i) r^(i - lo)
                    Q = torch.zeros_like(E)
                    for i in range(N - 1, -1, -1):
                        torch.mul(r, Q[i + 1] + E[i + 1], out=Q[i])
                    V.append(Q[lo_in] - rl * (Q.gather(0, self.top) + L * Et))
        self.W, self.V = W, V

    def F(self):
        A, B, C, ar, ai, br, bi = self.W
        S = A + B
        disc = torch.sqrt((A - B) ** 2 + 4.0 * C * C)
        self.D = A * B - C * C
        self.ok = self.any & (S - disc > 0) & (S + disc < 1e4 * (S - disc)) & (self.D > 0)
        num = B * (ar * ar + ai * ai) + A * (br * br + bi * bi) - 2.0 * C * (ar * br + ai * bi)
        return torch.where(self.ok, num / self.D, torch.full_like(num, 2.0))


def _ln_btsg(F):
    return (math.log(70.0 / F.numel()) + torch.logsumexp(F.reshape(-1), 0)).reshape(1)


def _grad64(w, n_tau, T=0.1):
    """(lnBtSG, softmax2F, dL/datoms, dL/dtau_min, dL/dtau_max) of
    L = lnBtSG + softmax2F for one template."""
    F = w.F()
    v = F.reshape(-1)
    lnB = _ln_btsg(F)
    z2 = torch.logsumexp(2.0 * v / T, 0)
    g = torch.exp(F - torch.logsumexp(v, 0)) + 2.0 * torch.exp(2.0 * F / T - z2)
    A, B, C, ar, ai, br, bi = w.W
    gi = torch.where(w.ok, g / w.D, torch.zeros_like(g))
    G = [gi * (br * br + bi * bi - F * B), gi * (ar * ar + ai * ai - F * A),
         2.0 * gi * (F * C - (ar * br + ai * bi)), 2.0 * gi * (B * ar - C * br),
         2.0 * gi * (B * ai - C * bi), 2.0 * gi * (A * br - C * ar), 2.0 * gi * (A * bi - C * ai)]
    dev = F.device
    ga = torch.zeros((w.N, 7), dtype=torch.float64, device=dev)
    dtau = torch.zeros_like(w.tau)
    lo_in = w.lo.clamp(max=w.N)
    for c in range(7):
        k = 2.0 if c < 3 else 1.0
        inj = torch.zeros((w.N + 1, w.tau.numel()), dtype=torch.float64, device=dev)
        inj.index_add_(0, lo_in, G[c])
        if w.window == RECT:
            inj.scatter_add_(0, w.top, -G[c])
            ga[:, c] = torch.cumsum(inj.sum(1), 0)[:w.N]
            continue
        L = (w.top - w.lo[:, None]).clamp(min=0).double()
        inj.scatter_add_(0, w.top, -G[c] * torch.exp(-k * TSFT / w.tau * L))
        r = torch.exp(-k * TSFT / w.tau)
        for i in range(1, w.N):
            inj[i].addcmul_(r, inj[i - 1])
        ga[:, c] = inj[:w.N].sum(1)
        dtau += (G[c] * w.V[c]).sum(0) * (k * TSFT / w.tau ** 2)
    fr = torch.arange(n_tau, dtype=torch.float64, device=dev) / max(1, n_tau - 1)
    return lnB, (T * z2).reshape(1), ga, (dtau * (1.0 - fr)).sum(), (dtau * fr).sum()


def exact(case, seed):
    kind = case["kind"]
    if kind == "dropin" or kind == "host":
        _, A = synth.merged_atoms(seed, case["nsft"], case["ndet"], gap_frac=case["gap"])
        if kind == "dropin":
            r = _dropin_range(case)
            t0s, taus = (_uniform(r["t0"], r["dt0"], case["n_t0"]),
                         _uniform(r["tau"], r["dtau"], case["n_tau"]))
        else:
            t0s = _uniform(T0, max(1, case["nsft"] // case["n_t0"]) * TSFT, case["n_t0"])
            taus = synth.log_tau_grid(TSFT, 3 * case["nsft"], case["n_tau"])
        F = _Windows64(torch.from_numpy(A).cuda(), case["window"], t0s, taus).F()
        out = dict(F=F, maxF=F.max(), lnBtSG=_ln_btsg(F)[0])
        rest = ("t0_ML", "tau_ML", "t0_MP", "tau_MP") if kind == "dropin" else (
            "argmax", "t0_mp", "tau_mp")
        return {**out, **{k: None for k in rest}}
    if kind == "plain":
        A = _atoms_cuda(seed, [case["nsft"]], [case["gap"]], case["ndet"])
        t0s, taus, _, _ = _span_grid(case["nsft"], case["n_t0"], case["n_tau"])
        F = _Windows64(A, case["window"], t0s, taus).F()
        return dict(F=F, lnBtSG=_ln_btsg(F), argmax=None, maxF=F.max().reshape(1), t0_mp=None,
                    tau_mp=None)
    if kind in ("batch", "maps"):
        if case["n"] > 200:
            return None
        nsft, gaps, nt0, ntau = _batch_geometry(case)
        A = _atoms_cuda(seed, nsft, gaps, 1)
        ends = np.cumsum(nsft)
        maps = []
        for j in range(case["n"]):
            t0s, taus, _, _ = _span_grid(int(nsft[j]), int(nt0[j]), int(ntau[j]))
            maps.append(_Windows64(A[int(ends[j] - nsft[j]):int(ends[j])],
                                   RECT if j % 2 == 0 else EXP, t0s, taus).F())
        out = dict(lnBtSG=torch.cat([_ln_btsg(F) for F in maps]), argmax=None,
                   maxF=torch.stack([F.max() for F in maps]), t0_mp=None, tau_mp=None)
        if kind == "maps":
            out["maps"] = torch.cat([F.reshape(-1) for F in maps])
        return out
    if kind == "grad":
        n, nsft = case["n"], case["nsft"]
        A = _atoms_cuda(seed, [nsft] * n, [0.0] * n, case["ndet"])
        t0s = _uniform(T0 + 450, max(1, nsft * TSFT // case["n_t0"]), case["n_t0"])
        lo, hi = _grad_tau(case)
        taus = lo + np.arange(case["n_tau"]) * ((hi - lo) / max(1, case["n_tau"] - 1))
        rows = [_grad64(_Windows64(A[j * nsft:(j + 1) * nsft], case["window"], t0s, taus,
                                   want_v=case["window"] == EXP), case["n_tau"])
                for j in range(n)]
        return dict(lnBtSG=torch.cat([r[0] for r in rows]),
                    softmax2F=torch.cat([r[1] for r in rows]),
                    grad_atoms=torch.cat([r[2] for r in rows]),
                    grad_tau_min=torch.stack([r[3] for r in rows]),
                    grad_tau_max=torch.stack([r[4] for r in rows]))
    cols = dict(twoF=[], maxTwoF=[], lnBtSG=[])
    r = _dropin_range(case)
    t0s = _uniform(r["t0"], r["dt0"], case["n_t0"])
    taus = _uniform(r["tau"], r["dtau"], case["n_tau"])
    for j in range(case["n"]):
        _, A = synth.merged_atoms(100003 * (seed % 10007) + j, case["nsft"], 2, gap_frac=0.1)
        A = torch.from_numpy(A).cuda()
        F = _Windows64(A, case["window"], t0s, taus).F()
        full = _Windows64(A, RECT, [T0], [A.shape[0] * TSFT]).F()
        cols["twoF"].append(2.0 * full.max())
        cols["maxTwoF"].append(2.0 * F.max())
        cols["lnBtSG"].append(_ln_btsg(F)[0])
    out = {k: torch.stack(v) for k, v in cols.items()}
    return {**out, "t0_ML": None, "tau_ML": None, "t0_MP": None, "tau_MP": None}
