"""Differentiable statistics of many templates of few rows: whole columns by one
warp, against the channel-split walk of hot columns (bit for bit) and against
FP64 torch autograd."""

import numpy as np
import pytest

import _torch_ref as R
from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu

MANY = 700  # column groups that fill the GPU with whole columns


def template(seed, nsft, n_t0, n_tau, dt0=9000, amp=8.0, gap=0.2):
    t0_data, A = synth.merged_atoms(seed, nsft, 2, amp=amp, inject=(nsft // 3, nsft // 2),
                                    gap_frac=gap)
    return dict(atoms=A, TAtom=1800, t0_data=t0_data, N_tau=n_tau, tau_min=9075.0,
                tau_max=9075.0 + 2700.0 * (n_tau - 1),
                t0s=(t0_data + 450 + dt0 * np.arange(n_t0)).astype(np.uint32))


def run(tl, T):
    import torch
    from pyfstat_gb300.autograd import DiffBatch

    b = DiffBatch(tl, temperature=T)
    atoms = torch.from_numpy(b.atoms).cuda()
    lim = [np.array([t[k] for t in tl]) for k in ("tau_min", "tau_max")]
    lnB, soft = b.forward_raw(atoms, *lim)
    z, g = torch.zeros_like(lnB), torch.ones_like(lnB)
    out = [x.cpu().numpy() for x in (lnB, soft, *b.backward_raw(atoms, *lim, lnB, soft, z, g))]
    b.handle.close()
    return out


@pytest.mark.parametrize("nsft", [31, 64, 200, 256])
def test_whole_columns_have_the_bits_of_the_channel_split_walk(nsft):
    """At T = 1e-4 one cell (with atoms entered and removed above it) carries all
    the weight: the value (window sums) and the tau gradients (derivative sums)
    of one template, walked by diff_hot_kernel when alone and by the tiles' own
    warps among 700, are equal bit for bit.  Behind the window's end the atom
    gradients differ by the removal power r^L, an FP64 product stepped from row
    to row: by 16 steps of 2^-53 for one warp, for each second row's warp by
    others."""
    pytest.importorskip("torch")
    t = template(5, nsft, 16, 1, dt0=nsft * 1800 // 20)
    _, soft1, ga1, gt1 = run([t], 1e-4)
    _, soft, ga, gt = run([t] * MANY, 1e-4)
    assert np.abs(ga1).max() > 0.0
    assert np.array_equal(soft, np.repeat(soft1, MANY))
    np.testing.assert_allclose(ga, np.tile(ga1, (MANY, 1)), rtol=0,
                               atol=2 * 16 * 2.0 ** -53 * np.abs(ga1).max())
    assert np.array_equal(gt, np.repeat(gt1, MANY, 0))


def test_few_rows_in_a_full_batch_match_torch_autograd():
    """Rows around the limits of 64 and 16 and atoms around that of 256, one and
    two column groups, beside templates that are cut."""
    torch = pytest.importorskip("torch")
    shapes = [(40, 1, 1), (50, 63, 33), (63, 64, 32), (64, 65, 31), (65, 64, 9), (90, 17, 64),
              (70, 150, 20), (256, 40, 9), (257, 40, 9), (330, 16, 10), (330, 17, 10)]
    tl = [template(k, n, rows, cols, dt0=max(450, n * 1800 // rows // 450 * 450),
                   amp=[0.0, 1.0, 6.0][k % 3])
          for k, (n, rows, cols) in enumerate(shapes * (MANY // len(shapes)))]
    lnB, soft, ga, gt = run(tl, 0.1)
    first = np.cumsum([0] + [t["atoms"].shape[0] for t in tl])
    for k in list(range(len(shapes))) + list(range(len(tl) - len(shapes), len(tl))):
        t = tl[k]
        x = torch.from_numpy(t["atoms"].astype(np.float64)).requires_grad_(True)
        a = torch.tensor(t["tau_min"], dtype=torch.float64, requires_grad=True)
        b = torch.tensor(t["tau_max"], dtype=torch.float64, requires_grad=True)
        rl, rs, _ = R.stats(x, 1800, t["t0_data"], t["t0s"], a, b, t["N_tau"])
        assert lnB[k] == pytest.approx(float(rl.detach()), rel=1e-9)
        assert soft[k] == pytest.approx(float(rs.detach()), rel=1e-9)
        rs.backward()
        ref = x.grad.numpy()
        # FP32 weights, exponents down to -80: (2.5 x 80 + 8) 2^-24 = 1.2e-5
        np.testing.assert_allclose(ga[first[k]:first[k + 1]], ref, rtol=1.3e-5,
                                   atol=1e-9 * np.abs(ref).max())
        assert gt[k, 0] == pytest.approx(float(a.grad), rel=1.3e-5, abs=1e-15)
        if t["N_tau"] > 1:
            assert gt[k, 1] == pytest.approx(float(b.grad), rel=1.3e-5, abs=1e-15)


def test_templates_of_unequal_size_match_those_alone():
    """2000 small templates around one of 17532 atoms and 400 x 256 cells: launches
    of their own for the large one, each template's result as by itself."""
    pytest.importorskip("torch")
    big = template(77, 17532, 400, 256, dt0=72000, gap=0.05)
    small = [template(k, 90 + k, 30, 33) for k in range(4)]
    tl = small * 300 + [big] + small * 200
    lnB, soft, ga, gt = run(tl, 0.1)
    first = np.cumsum([0] + [t["atoms"].shape[0] for t in tl])
    for k in (0, 1, 2, 3, 1200, 1201, len(tl) - 1):
        l1, s1, ga1, gt1 = run([tl[k]], 0.1)
        assert lnB[k] == pytest.approx(l1[0], rel=1e-11)
        assert soft[k] == pytest.approx(s1[0], rel=1e-11)
        # other chunks and sums: F to 1e-13, 2F/T to 1e-9; FP32 weights 1.2e-5
        np.testing.assert_allclose(ga[first[k]:first[k + 1]], ga1, rtol=1.3e-5,
                                   atol=1e-9 * np.abs(ga1).max())
        np.testing.assert_allclose(gt[k], gt1[0], rtol=1.3e-5, atol=1e-15)
