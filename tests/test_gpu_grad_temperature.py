"""Differentiable statistics over the range of soft-max temperatures, against
FP64 torch autograd: above T = 2 the soft-max's weights reach further below the
maximum than lnBtSG's."""

import numpy as np
import pytest

import _torch_ref as R
from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu

N_T0, N_TAU, NSFT = 21, 18, 160


def template(window):
    t0_data, A = synth.merged_atoms(31 + window, NSFT, 2, amp=6.0, inject=(50, 90))
    return dict(atoms=A, TAtom=1800, t0_data=t0_data, window=window, N_tau=N_TAU,
                tau_min=9075.0, tau_max=9075.0 + 5400.0 * (N_TAU - 1),
                t0s=(t0_data + 450 + 12600 * np.arange(N_T0)).astype(np.uint32))


def cell_jacobian(t, T):
    """FP64 values, F per cell and |dF| of every cell to atoms, tau_min, tau_max."""
    import torch

    x = torch.from_numpy(t["atoms"].astype(np.float64)).requires_grad_(True)
    a = torch.tensor(t["tau_min"], dtype=torch.float64, requires_grad=True)
    b = torch.tensor(t["tau_max"], dtype=torch.float64, requires_grad=True)
    lnB, soft, F = R.stats(x, 1800, t["t0_data"], t["t0s"], a, b, N_TAU, T, t["window"])
    rows = []
    for f in F.reshape(-1):
        if not f.requires_grad:
            rows.append(np.zeros(x.numel() + 2))
            continue
        g = torch.autograd.grad(f, (x, a, b), retain_graph=True, allow_unused=True)
        rows.append(np.concatenate([np.zeros(n) if q is None else q.numpy().reshape(-1)
                                    for q, n in zip(g, (x.numel(), 1, 1))]))
    return float(lnB.detach()), float(soft.detach()), F.detach().numpy().reshape(-1), np.array(rows)


@pytest.mark.parametrize("T", [0.1, 5.0, 20.0, 100.0, 1000.0])
@pytest.mark.parametrize("window", [1, 2])
def test_temperatures_match_torch_autograd(window, T):
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch, transient_stats

    t = template(window)
    batch = DiffBatch([t], temperature=T)
    atoms = torch.from_numpy(batch.atoms).cuda().requires_grad_(True)
    tmin = torch.tensor([t["tau_min"]], dtype=torch.float64, requires_grad=True)
    tmax = torch.tensor([t["tau_max"]], dtype=torch.float64, requires_grad=True)
    lnB, soft = transient_stats(atoms, tmin, tmax, batch)
    rl, rs, F, J = cell_jacobian(t, T)
    assert F.max() > 140.0  # cells beyond 62 of the maximum
    assert float(lnB[0].detach()) == pytest.approx(rl, rel=1e-9)
    assert float(soft[0].detach()) == pytest.approx(rs, rel=1e-9)
    (0.5 * lnB.sum() + 1.5 * soft.sum()).backward()
    got = np.concatenate([atoms.grad.double().cpu().numpy().reshape(-1), tmin.grad.numpy(),
                          tmax.grad.numpy()])
    # dL/dF of every cell; its FP32 weights are good to (2.5 |exponent| + 8) 2^-24
    e1 = F - (rl - np.log(70.0 / (N_T0 * N_TAU)))
    e2 = 2.0 * F / T - rs / T
    g1, g2 = 0.5 * np.exp(e1), 3.0 * np.exp(e2)
    ref = (g1 + g2) @ J
    unit = 2.0 ** -24 * (g1 * (2.5 * np.abs(e1) + 8.0) + g2 * (2.5 * np.abs(e2) + 8.0))
    bound = unit @ np.abs(J)
    # what is left of a cell's term behind its window (double-word removal, 2^-46)
    bound[:-2] += 1e-12 * ((g1 + g2) @ np.abs(J))[:-2].max()
    assert (np.abs(got - ref) <= bound + 1e-15).all(), np.max(np.abs(got - ref) / (bound + 1e-15))
