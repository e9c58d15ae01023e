"""Exponential columns without segment sums: where their memory is not to be
had (injected allocation failure) and beyond the 1 GiB that they may take."""

import numpy as np
import pytest
from _helpers import REL_TOL, rel_err

from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu


def small():
    t0_data, A = synth.merged_atoms(9, 700, 1, gap_frac=0.1)
    return dict(window=2, atoms=A, TAtom=1800, t0_data=t0_data,
                t0s=(t0_data + 1800 * np.arange(300)).astype(np.uint32),
                taus=(3600 + 5400 * np.arange(70)).astype(np.uint32))


@pytest.mark.parametrize("entry", ["host", "device", "plan", "forward", "backward"])
def test_calls_succeed_without_the_memory_for_segment_sums(oracle, entry):
    """The first workspace allocation fails; the call runs whole columns."""
    torch = pytest.importorskip("torch")
    from pyfstat_gb300 import _lib
    from pyfstat_gb300.autograd import DiffBatch
    from pyfstat_gb300.batched import TransientMapBatch

    t = small()
    A, t0s, taus = t["atoms"], t["t0s"], t["taus"]
    h = _lib.Handle(0)
    if entry in ("forward", "backward"):
        ref = _lib.Handle(0)
        d = dict(atoms=A, TAtom=1800, t0_data=t["t0_data"], t0s=t0s, N_tau=70)
        out = []
        for hd in (ref, h):
            b = DiffBatch([d], handle=hd)
            atoms = torch.from_numpy(b.atoms).cuda()
            lim = np.array([9075.0]), np.array([369075.0])
            if hd is h and entry == "forward":
                hd.fail_alloc(1)
            lnB, soft = b.forward_raw(atoms, *lim)
            if hd is h and entry == "backward":  # a fresh handle: its workspace is too small
                hd = b.handle = _lib.Handle(0)
                hd.fail_alloc(1)
            g = torch.ones_like(lnB)
            out.append([x.cpu().numpy() for x in (lnB, soft, *b.backward_raw(
                atoms, *lim, lnB, soft, g, g))])
        for x, y in zip(*out):
            np.testing.assert_allclose(y, x, rtol=1e-5, atol=1e-9 * np.abs(x).max())
        assert np.allclose(out[0][0], out[1][0], rtol=1e-12, atol=0)
        return
    F64, cond = oracle.map_f64(A, 1800, t["t0_data"], 2, t0s, taus, with_cond=True)
    h.fail_alloc(1)
    if entry == "host":
        F, r = h.map_plain_host(A, 1800, t["t0_data"], 2, t0s, taus)
    elif entry == "device":
        dev = [torch.from_numpy(x).cuda() for x in (A, t0s.view(np.int32), taus.view(np.int32))]
        dF = torch.empty((300, 70), device="cuda")
        res = torch.zeros(5, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        h.map_plain(dev[0], 700, 1800, t["t0_data"], 2, dev[1], 300, dev[2], 70, dF, res)
        h.sync()
        F, r = dF.cpu().numpy(), res.cpu().numpy().view(_lib.RESULT_DTYPE)[0]
    else:
        batch = TransientMapBatch([t], handle=h)
        res, F = batch.plan.run_maps_host(batch.atoms)
        r = res[0]
        batch.close()
    rel, _ = rel_err(F.reshape(F64.shape), F64, cond)
    assert rel.max() <= REL_TOL
    assert float(r["lnBtSG"]) == pytest.approx(oracle.lnBtSG(F64), rel=REL_TOL)
    h.close()


NSFT, N_T0 = 100000, 24  # segments of 256 atoms, 700672 bytes per 32 columns


def large(n_tau):
    t0_data, A = synth.merged_atoms(13, NSFT, 1, Tsft=600, inject=(0, NSFT), amp=0.2)
    return dict(window=2, atoms=A, TAtom=600, t0_data=t0_data,
                t0s=(t0_data + 300 + 2400000 * np.arange(N_T0)).astype(np.uint32),
                taus=(600000 + 400 * np.arange(n_tau)).astype(np.uint32))


def test_templates_beyond_the_segment_limit_take_whole_columns():
    """Two templates of 0.58 GiB of segment sums each: the second one keeps
    whole columns, the bits of a plan whose exp_rows asks for them; a single
    map of 1.1 GiB keeps whole histories."""
    from pyfstat_gb300 import _lib
    from pyfstat_gb300.batched import TransientMapBatch

    t = large(28672)
    h = _lib.Handle(0)
    auto = TransientMapBatch([t, t], handle=h)
    _, F = auto.plan.run_maps_host(auto.atoms)
    F = F.reshape(2, N_T0, -1)
    whole = TransientMapBatch([t], tile_config=dict(exp_rows=N_T0), handle=h)
    _, W = whole.plan.run_maps_host(whole.atoms)
    W = W.reshape(F[0].shape)
    assert np.array_equal(F[1].view(np.uint32), W.view(np.uint32))
    np.testing.assert_allclose(F[0], W, rtol=REL_TOL)
    t = large(50048)
    P, _ = h.map_plain_host(t["atoms"], 600, t["t0_data"], 2, t["t0s"], t["taus"])
    np.testing.assert_allclose(P[:, :28672], W, rtol=REL_TOL)
    for b in (auto, whole):
        b.close()
    h.close()


def test_gradients_beyond_the_segment_limit():
    """100096 columns of 100000 atoms: whole columns in both passes, 8.8 GB of
    recurrence ends in three slices, against the template's halves in tau
    (whole columns as well: sums over 100000 atoms that are cut differently
    agree to 1e-7 only)."""
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch, transient_stats

    t = large(1)
    N, lo, step = 100096, 600075.0, 400.0
    vals, grads = [], []
    for n, first in ((N, lo), (N // 2, lo), (N // 2, lo + step * (N // 2))):
        b = DiffBatch([dict(atoms=t["atoms"], TAtom=600, t0_data=t["t0_data"], N_tau=n,
                            t0s=t["t0s"])], temperature=100.0)
        atoms = torch.from_numpy(b.atoms).cuda().requires_grad_(True)
        lim = [torch.tensor([x], dtype=torch.float64) for x in (first, first + step * (n - 1))]
        lnB, soft = transient_stats(atoms, *lim, b)
        g, = torch.autograd.grad(soft.sum(), atoms)
        vals.append(float(soft.detach()) / 100.0)
        grads.append(g.double().cpu().numpy())
        b.handle.close()
    top = max(vals[1:])
    z = top + np.log(sum(np.exp(v - top) for v in vals[1:]))
    assert vals[0] == pytest.approx(z, rel=1e-9)
    w = [np.exp(v - z) for v in vals[1:]]
    assert min(w) > 1e-3  # both halves count
    ref = w[0] * grads[1] + w[1] * grads[2]
    # FP32 weights, exponents within 20: 2 (2.5 x 20 + 8) 2^-24 = 7e-6 of the terms
    np.testing.assert_allclose(grads[0], ref, rtol=0, atol=2e-5 * np.abs(ref).max())
