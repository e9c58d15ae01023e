"""Workspace bounds of the differentiable statistics' backward pass: groups of
templates with many atoms and few cells, and one template in slices of column
groups."""

import numpy as np
import pytest

from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu


def test_many_templates_of_many_atoms_and_one_row():
    """20000 templates of one t0 and 1024 taus over the same 17532 atoms: few
    cells, but 16 MB of recurrence ends each (314 GB in one group)."""
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch

    n, nsft = 20000, 17532
    t0_data, A = synth.merged_atoms(3, nsft, 1)
    t = dict(atoms=A, TAtom=1800, t0_data=t0_data, N_tau=1024, tau_min=9075.0, tau_max=18075.0,
             t0s=np.array([t0_data + 450], np.uint32))
    one = DiffBatch([t])
    many = DiffBatch([t], handle=one.handle)
    many.desc = np.repeat(one.desc, n)  # (all read and differentiate the same rows)
    many.n_templates = n
    atoms = torch.from_numpy(one.atoms).cuda()
    out = []
    for b in (one, many):
        taus = [np.full(b.n_templates, t[k]) for k in ("tau_min", "tau_max")]
        lnB, soft = b.forward_raw(atoms, *taus)
        g = torch.ones_like(lnB)
        out.append([v.cpu().numpy() for v in (lnB, soft, *b.backward_raw(atoms, *taus, lnB, soft,
                                                                         g, g))])
    (lnB1, soft1, ga1, gt1), (lnB, soft, ga, gt) = out
    assert np.array_equal(lnB, np.repeat(lnB1, n)) and np.array_equal(soft, np.repeat(soft1, n))
    # FP64 sums of n x 32 equal terms in any order
    np.testing.assert_allclose(ga, n * ga1, rtol=1e-9, atol=0)
    np.testing.assert_allclose(gt, np.repeat(gt1, n, 0), rtol=1e-9, atol=0)
    one.handle.close()


def test_slices_of_a_large_template_add_up():
    """8192 t0 x 16384 taus (two slices) against its two halves in tau (one
    slice each): the halves' sums and gradients weigh in by their shares of
    the log-sum-exps.  The windows end behind the data, so that F changes
    slowly with tau and every column counts."""
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch, transient_stats

    T, N = 100.0, 16384
    t0_data, A = synth.merged_atoms(11, 300, 2, amp=1.0, inject=(0, 300))
    t0s = (t0_data + 450 + 60 * np.arange(8192)).astype(np.uint32)
    lo, step = 720075.0, 90.0
    # (number of taus, first tau): the whole and its halves
    grids = [(N, lo), (N // 2, lo), (N // 2, lo + step * (N // 2))]
    vals, grads = [], []
    for n, first in grids:
        b = DiffBatch([dict(atoms=A, TAtom=1800, t0_data=t0_data, N_tau=n, t0s=t0s)],
                      temperature=T)
        atoms = torch.from_numpy(b.atoms).cuda().requires_grad_(True)
        tmin = torch.tensor([first], dtype=torch.float64)
        tmax = torch.tensor([first + step * (n - 1)], dtype=torch.float64)
        lnB, soft = transient_stats(atoms, tmin, tmax, b)
        gl, = torch.autograd.grad(lnB.sum(), atoms, retain_graph=True)
        gs, = torch.autograd.grad(soft.sum(), atoms)
        # (the number of cells out of lnBtSG)
        vals.append((float(lnB.detach()) + np.log(n), float(soft.detach())))
        grads.append([g.double().cpu().numpy() for g in (gl, gs)])
        b.handle.close()
    for q, scale in ((0, 1.0), (1, T)):
        z = [v[q] / scale for v in vals]
        top = max(z[1:])
        whole = top + np.log(sum(np.exp(v - top) for v in z[1:]))
        assert z[0] == pytest.approx(whole, rel=1e-9)
        w = [np.exp(v - whole) for v in z[1:]]
        assert min(w) > 1e-3  # both halves count
        ref = w[0] * grads[1][q] + w[1] * grads[2][q]
        # FP32 weights, exponents within 20: 2 (2.5 x 20 + 8) 2^-24 = 7e-6 of the terms
        np.testing.assert_allclose(grads[0][q], ref, rtol=0, atol=2e-5 * np.abs(ref).max())
