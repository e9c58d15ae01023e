"""Gradients of rectangular templates whose row groups alone fill the GPU: fewer,
wider column chunks, against each template by itself."""

import numpy as np
import pytest

from test_gpu_grad_whole_columns import run, template

pytestmark = pytest.mark.gpu


def test_wide_chunks_match_those_alone():
    """Row groups around one and four per template, columns around a chunk of 16
    and of 64; FP64 sums in other pieces (F to 1e-13), FP32 weights 1.2e-5."""
    torch = pytest.importorskip("torch")
    shapes = [(60, 4, 1), (70, 32, 16), (90, 33, 17), (130, 97, 64), (130, 129, 65), (257, 1, 129),
              (300, 32, 128)]
    kinds = [dict(template(k, n, rows, cols, dt0=max(450, n * 1800 // rows // 450 * 450),
                           amp=[0.0, 1.0, 6.0][k % 3]), window=1)
             for k, (n, rows, cols) in enumerate(shapes)]
    groups = sum((t["t0s"].size + 31) // 32 for t in kinds)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tl = kinds * (2 * sms // groups + 1)
    lnB, soft, ga, gt = run(tl, 0.1)
    first = np.cumsum([0] + [t["atoms"].shape[0] for t in tl])
    for k in [*range(len(kinds)), *range(len(tl) - len(kinds), len(tl))]:
        l1, s1, ga1, gt1 = run([tl[k]], 0.1)
        assert lnB[k] == pytest.approx(l1[0], rel=1e-11)
        assert soft[k] == pytest.approx(s1[0], rel=1e-11)
        np.testing.assert_allclose(ga[first[k]:first[k + 1]], ga1, rtol=1.3e-5,
                                   atol=1e-9 * np.abs(ga1).max())
        assert not gt[k].any() and not gt1.any()
