"""Hot tiles of many column groups: walked by a warp per group, against a block
per group (a template by itself), bit for bit where one cell carries all the
weight."""

import numpy as np
import pytest

from test_gpu_grad_whole_columns import run, template

pytestmark = pytest.mark.gpu


def few():
    import torch
    return 2 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("nsft,n_t0,n_tau", [(64, 65, 1), (130, 100, 33), (257, 129, 32),
                                             (400, 300, 9)])
def test_warps_have_the_bits_of_the_block_walk(nsft, n_t0, n_tau):
    """At T = 1e-4 one cell carries all the weight, so value and tau gradients
    show its window sums.  Atom gradients: the removal power r^L is an FP64 product
    stepped from row to row, by every row for the one, every second for the
    other."""
    pytest.importorskip("torch")
    t = template(5, nsft, n_t0, n_tau, dt0=max(450, nsft * 1800 // n_t0 // 450 * 450))
    n = few() // ((n_tau + 31) // 32) + 1
    _, soft1, ga1, gt1 = run([t], 1e-4)
    _, soft, ga, gt = run([t] * n, 1e-4)
    assert np.abs(ga1).max() > 0.0
    assert np.array_equal(soft, np.repeat(soft1, n))
    np.testing.assert_allclose(ga, np.tile(ga1, (n, 1)), rtol=0,
                               atol=2 * n_t0 * 2.0 ** -53 * np.abs(ga1).max())
    assert np.array_equal(gt, np.repeat(gt1, n, 0))


@pytest.mark.parametrize("extra", [0, 1])
def test_around_the_limit_match_those_alone(extra):
    """Two blocks per SM and one group more, noise and signals: each template as by
    itself (other partial sums, FP32 weights: 1.2e-5)."""
    pytest.importorskip("torch")
    kinds = [template(k, 150 + 10 * k, 70 + 15 * k, 20, dt0=2250, amp=[0.0, 1.0, 8.0][k])
             for k in range(3)]
    tl = [kinds[k % 3] for k in range(few() + extra)]
    lnB, soft, ga, gt = run(tl, 0.1)
    first = np.cumsum([0] + [t["atoms"].shape[0] for t in tl])
    for k in (0, 1, 2, len(tl) - 3, len(tl) - 2, len(tl) - 1):
        l1, s1, ga1, gt1 = run([tl[k]], 0.1)
        assert lnB[k] == pytest.approx(l1[0], rel=1e-11)
        assert soft[k] == pytest.approx(s1[0], rel=1e-11)
        np.testing.assert_allclose(ga[first[k]:first[k + 1]], ga1, rtol=1.3e-5,
                                   atol=1e-9 * np.abs(ga1).max())
        np.testing.assert_allclose(gt[k], gt1[0], rtol=1.3e-5, atol=1e-15)
