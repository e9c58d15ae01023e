"""Tiles of the exponential differentiable statistics (row chunks started from
segment sums, tiles without weight left out, hot columns walked whole, the
transposed recurrence in atom segments) against FP64 torch autograd."""

import numpy as np
import pytest

import _torch_ref as R
from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu

# per template: SFTs, t0 points, t0 step in SFTs, tau points, tau step, signal
# amplitude, gap fraction.  Sizes around the smallest atom count with
# segments (64), one and two 64-atom segments, one chunk of 16 rows and its
# neighbours, one column group and its neighbours; noise alone (every cell
# carries weight) and strong signals (most tiles carry none); templates of
# unequal size side by side; more atoms than the staged walk keeps.
CASES = [
    [(63, 17, 3, 33, 1200, 0.0, 0.0)],
    [(64, 16, 4, 32, 1500, 20.0, 0.1), (65, 15, 4, 31, 900, 0.0, 0.3), (129, 130, 1, 1, 300, 5.0, 0.0)],
    [(200, 70, 2, 70, 2400, 30.0, 0.05), (40, 33, 1, 9, 600, 0.0, 0.0)],
    [(7100, 7, 1000, 3, 90000, 10.0, 0.0)],
]


@pytest.mark.parametrize("weights", [(1.0, 0.5), (1.0, 0.0), (0.0, -2.0)])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_tiles_match_torch_autograd(case, weights):
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch, transient_stats

    tl = []
    for k, (nsft, n_t0, dt0, n_tau, step, amp, gap) in enumerate(CASES[case]):
        t0_data, A = synth.merged_atoms(70 + 10 * case + k, nsft, 2, amp=amp,
                                        inject=(nsft // 3, nsft // 2), gap_frac=gap)
        tau_min = 6675.0 + 900.0 * k
        tl.append(dict(atoms=A, TAtom=1800, t0_data=t0_data, N_tau=n_tau, tau_min=tau_min,
                       tau_max=tau_min + step * (n_tau - 1),
                       t0s=(t0_data + 450 + 1800 * dt0 * np.arange(n_t0)).astype(np.uint32)))
    batch = DiffBatch(tl)
    atoms = torch.from_numpy(batch.atoms).cuda().requires_grad_(True)
    tmin = torch.tensor([t["tau_min"] for t in tl], dtype=torch.float64, requires_grad=True)
    tmax = torch.tensor([t["tau_max"] for t in tl], dtype=torch.float64, requires_grad=True)
    lnB, soft = transient_stats(atoms, tmin, tmax, batch)
    (weights[0] * lnB.sum() + weights[1] * soft.sum()).backward()
    ga = atoms.grad.double().cpu().numpy()
    row = 0
    for k, t in enumerate(tl):
        x = torch.from_numpy(t["atoms"].astype(np.float64)).requires_grad_(True)
        a = torch.tensor(t["tau_min"], dtype=torch.float64, requires_grad=True)
        b = torch.tensor(t["tau_max"], dtype=torch.float64, requires_grad=True)
        rl, rs, _ = R.stats(x, 1800, t["t0_data"], t["t0s"], a, b, t["N_tau"])
        assert float(lnB[k].detach()) == pytest.approx(float(rl.detach()), rel=1e-9)
        assert float(soft[k].detach()) == pytest.approx(float(rs.detach()), rel=1e-9)
        (weights[0] * rl + weights[1] * rs).backward()
        n = t["atoms"].shape[0]
        ref = x.grad.numpy()
        # a weight's exponent (down to -80) is rounded to FP32 before exp2:
        # 80 x 2^-24 = 5e-6 of the weight, with as much again for its product
        # with log2(e) and the sums
        np.testing.assert_allclose(ga[row:row + n], ref, rtol=1e-5,
                                   atol=1e-9 * np.abs(ref).max())
        if t["N_tau"] > 1:
            assert float(tmax.grad[k]) == pytest.approx(float(b.grad), rel=1e-5, abs=1e-15)
        assert float(tmin.grad[k]) == pytest.approx(float(a.grad), rel=1e-5, abs=1e-15)
        row += n


@pytest.mark.parametrize("kind", ["one antenna pattern", "zero atoms"])
def test_templates_whose_cells_all_fail_the_conditioning_test(kind):
    """F = 2 in every cell (no lower bound of the maximum to sort tiles by):
    the closed forms of both statistics, no gradient, and the template beside
    them as by itself."""
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.autograd import DiffBatch

    def template(k, nsft, n_t0, n_tau, flat):
        t0_data, A = synth.merged_atoms(40 + k, nsft, 2, amp=3.0)
        if flat:
            A = np.zeros_like(A) if kind == "zero atoms" else A * np.float32([1, 0, 0, 1, 1, 0, 0])
        return dict(atoms=A, TAtom=1800, t0_data=t0_data, N_tau=n_tau, tau_min=9075.0,
                    tau_max=9075.0 + 900.0 * (n_tau - 1),
                    t0s=(t0_data + 450 + 3600 * np.arange(n_t0)).astype(np.uint32))

    tl = [template(0, 200, 90, 70, True), template(1, 120, 17, 33, False),
          template(2, 65, 16, 1, True), template(3, 30, 1, 40, True)]

    def run(tl):
        b = DiffBatch(tl)
        atoms = torch.from_numpy(b.atoms).cuda()
        lim = [np.array([t[k] for t in tl]) for k in ("tau_min", "tau_max")]
        lnB, soft = b.forward_raw(atoms, *lim)
        g = torch.ones_like(lnB)
        out = [x.cpu().numpy() for x in (lnB, soft, *b.backward_raw(atoms, *lim, lnB, soft, g, g))]
        b.handle.close()
        return out

    lnB, soft, ga, gt = run(tl)
    first = np.cumsum([0] + [t["atoms"].shape[0] for t in tl])
    for k in (0, 2, 3):
        n = len(tl[k]["t0s"]) * tl[k]["N_tau"]
        assert lnB[k] == pytest.approx(np.log(70.0) + 2.0, rel=1e-12)
        assert soft[k] == pytest.approx(4.0 + 0.1 * np.log(n), rel=1e-12)
        assert not ga[first[k]:first[k + 1]].any() and not gt[k].any()
    one = run([tl[1]])
    assert lnB[1] == pytest.approx(one[0][0], rel=1e-11)
    assert soft[1] == pytest.approx(one[1][0], rel=1e-11)
    # FP32 weights, exponents down to -80
    np.testing.assert_allclose(ga[first[1]:first[2]], one[2], rtol=1.3e-5,
                               atol=1e-9 * np.abs(one[2]).max())
