"""Tiles of the rectangular differentiable statistics (column chunks, tiles
without weight left out, FP64 sums from block sums) against FP64 torch
autograd."""

import numpy as np
import pytest

import _torch_ref as R
from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu

# per template: SFTs, t0 points, t0 step in seconds, tau points, first tau, tau
# step, signal amplitude, gap fraction.  Row groups of 32 and column chunks of
# 16 and their neighbours, 32-atom blocks and their neighbours, taus closer
# than an SFT (windows that repeat), windows clamped at the data's end, a
# start half an SFT before the data, noise alone and strong signals, templates
# of unequal size side by side.
CASES = [
    [(31, 33, 1800, 17, 5400.0, 450.0, 0.0, 0.0)],
    [(32, 32, 900, 16, 7200.0, 1800.0, 8.0, 0.2), (33, 31, 1800, 15, 9000.0, 3600.0, 0.0, 0.0),
     (97, 1, 1800, 70, 3600.0, 1234.5, 6.0, 0.0)],
    [(300, 70, 5400, 40, 21600.0, 14400.0, 10.0, 0.05), (64, 64, 1800, 1, 36000.0, 1.0, 0.0, 0.3)],
]


@pytest.mark.parametrize("weights", [(1.0, 0.5), (0.0, -2.0)])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_rect_tiles_match_torch_autograd(case, weights):
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch, transient_stats

    tl = []
    for k, (nsft, n_t0, dt0, n_tau, tau, dtau, amp, gap) in enumerate(CASES[case]):
        t0_data, A = synth.merged_atoms(170 + 10 * case + k, nsft, 2, amp=amp,
                                        inject=(nsft // 3, nsft // 2), gap_frac=gap)
        tl.append(dict(atoms=A, TAtom=1800, t0_data=t0_data, window=1, N_tau=n_tau,
                       tau_min=tau, tau_max=tau + dtau * (n_tau - 1),
                       t0s=(t0_data - 900 + 450 * k + dt0 * np.arange(n_t0)).astype(np.uint32)))
    batch = DiffBatch(tl)
    atoms = torch.from_numpy(batch.atoms).cuda().requires_grad_(True)
    tmin = torch.tensor([t["tau_min"] for t in tl], dtype=torch.float64, requires_grad=True)
    tmax = torch.tensor([t["tau_max"] for t in tl], dtype=torch.float64, requires_grad=True)
    lnB, soft = transient_stats(atoms, tmin, tmax, batch)
    (weights[0] * lnB.sum() + weights[1] * soft.sum()).backward()
    ga = atoms.grad.double().cpu().numpy()
    assert float(tmin.grad.abs().max()) == 0.0 and float(tmax.grad.abs().max()) == 0.0
    row = 0
    for k, t in enumerate(tl):
        x = torch.from_numpy(t["atoms"].astype(np.float64)).requires_grad_(True)
        rl, rs, _ = R.stats(x, 1800, t["t0_data"], t["t0s"],
                            torch.tensor(t["tau_min"], dtype=torch.float64),
                            torch.tensor(t["tau_max"], dtype=torch.float64), t["N_tau"], window=1)
        assert float(lnB[k].detach()) == pytest.approx(float(rl.detach()), rel=1e-9)
        assert float(soft[k].detach()) == pytest.approx(float(rs.detach()), rel=1e-9)
        (weights[0] * rl + weights[1] * rs).backward()
        n = t["atoms"].shape[0]
        ref = x.grad.numpy()
        # a weight's exponent (down to -63) is rounded to FP32 before exp2 and
        # multiplied by log2(e) there: up to 2 x 91 x 2^-24 = 1.1e-5 of a weight
        np.testing.assert_allclose(ga[row:row + n], ref, rtol=1.2e-5,
                                   atol=1e-9 * np.abs(ref).max())
        row += n
