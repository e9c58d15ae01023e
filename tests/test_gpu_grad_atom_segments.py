"""Atom segments of the gradient's transposed recurrence: one per column where
whole columns fill the GPU, longer ones for very many atoms."""

import numpy as np
import pytest

from test_gpu_grad_whole_columns import run, template

pytestmark = pytest.mark.gpu


def close(got, want):
    """Other segments and partial sums: F to 1e-13; FP32 weights 1.2e-5."""
    (l, s, ga, gt), (l1, s1, ga1, gt1) = got, want
    assert l == pytest.approx(l1, rel=1e-11)
    assert s == pytest.approx(s1, rel=1e-11)
    np.testing.assert_allclose(ga, ga1, rtol=1.3e-5, atol=1e-9 * np.abs(ga1).max())
    np.testing.assert_allclose(gt, gt1, rtol=1.3e-5, atol=1e-15)


@pytest.mark.parametrize("sms", [15, 17])
def test_whole_columns_below_and_above_four_warps_per_scheduler(sms):
    """`sms` column groups per SM, atoms around a segment and the limit of 2048,
    rows around that of 64: each template as by itself."""
    torch = pytest.importorskip("torch")
    shapes = [(63, 5, 1), (64, 64, 33), (65, 64, 20), (129, 3, 40), (700, 63, 9), (2048, 16, 33),
              (2049, 16, 5), (300, 65, 8)]
    kinds = [template(k, n, rows, cols, dt0=max(450, n * 1800 // rows // 450 * 450),
                      amp=[0.0, 1.0, 6.0][k % 3]) for k, (n, rows, cols) in enumerate(shapes)]
    groups = sum((t["N_tau"] + 31) // 32 for t in kinds)
    n = torch.cuda.get_device_properties(0).multi_processor_count * sms // groups
    tl = kinds * n
    lnB, soft, ga, gt = run(tl, 0.1)
    first = np.cumsum([0] + [t["atoms"].shape[0] for t in tl])
    for k in [*range(len(kinds)), *range(len(tl) - len(kinds), len(tl))]:
        l1, s1, ga1, gt1 = run([tl[k]], 0.1)
        close((lnB[k], soft[k], ga[first[k]:first[k + 1]], gt[k]), (l1[0], s1[0], ga1, gt1[0]))


@pytest.mark.parametrize("nsft", [262144, 262145])
def test_very_many_atoms_match_the_part_that_the_windows_see(nsft):
    """4096 segments of 64 atoms, and more than these cover: a template of `nsft`
    atoms whose windows lie in the last 5000 against those atoms alone."""
    pytest.importorskip("torch")
    from pyfstat_gb300 import synth
    cut = nsft - 5000
    t0_data, A = synth.merged_atoms(9, 5000, 2, amp=8.0, inject=(1500, 2000), gap_frac=0.1)
    rng = np.random.default_rng(1)
    before = np.abs(rng.standard_normal((cut, 7))).astype(np.float32)
    t0 = t0_data - 1800 * cut
    grid = dict(TAtom=1800, t0s=(t0_data + 450 + 90000 * np.arange(40)).astype(np.uint32),
                N_tau=40, tau_min=9075.0, tau_max=909075.0)
    part = run([dict(grid, atoms=A, t0_data=t0_data)], 0.1)
    lnB, soft, ga, gt = run([dict(grid, atoms=np.concatenate([before, A]), t0_data=t0)], 0.1)
    assert not ga[:cut].any()
    close((lnB, soft, ga[cut:], gt), part)
