"""Posterior indices of plans of very many maps (one argmax block per template,
row chunks by the number of blocks) from the maps that the same run wrote."""

import numpy as np
import pytest

from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu


# t0 and tau points: around a warp, a part of the argmax (256), a row quad and
# a strip of 1024 columns; repeated until there are `n` templates
SHAPES = [(20, 20), (1, 1), (257, 3), (3, 257), (31, 33), (600, 40), (5, 1030), (256, 32), (16, 64)]


@pytest.mark.parametrize("n", [9, 180, 2000])
def test_posteriors_of_many_maps(n):
    torch = pytest.importorskip("torch")
    from pyfstat_gb300 import _lib
    from pyfstat_gb300.batched import TransientMapBatch

    tl = []
    for k in range(n):
        n_t0, n_tau = SHAPES[k % len(SHAPES)]
        t0_data, A = synth.merged_atoms(k % 11, 60 + k % 5, 1)
        tl.append(dict(window=1 + k % 2, atoms=A, TAtom=1800, t0_data=t0_data,
                       t0s=(t0_data + 300 * np.arange(n_t0)).astype(np.uint32),
                       taus=(1800 + 97 * np.arange(n_tau)).astype(np.uint32)))
    b = TransientMapBatch(tl, flags=_lib.TCW_FLAG_LNBTSG | _lib.TCW_FLAG_POSTERIORS)
    atoms = torch.from_numpy(b.atoms).cuda()
    res = torch.zeros(5 * n, dtype=torch.float64, device="cuda")
    maps = torch.empty(b.n_cells, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):  # the second run meets the first one's sums
        b.plan.run_maps(atoms, res, maps)
        b.handle.sync()
    rec, F = res.cpu().numpy().view(_lib.RESULT_DTYPE), maps.cpu().numpy()
    off = 0
    for k, t in enumerate(tl):
        shape = len(t["t0s"]), len(t["taus"])
        f = F[off:off + shape[0] * shape[1]].reshape(shape).astype(np.float64)
        off += f.size
        e = np.exp(f - f.max())
        for field, sums in (("t0_mp_idx", e.sum(1)), ("tau_mp_idx", e.sum(0))):
            # FP32 terms of 1e-7: the index of the largest sum, or of one as large
            assert sums[rec[field][k]] >= sums.max() * (1.0 - 1e-6), (k, field)
    b.close()


# 63, 64 and 65 sums of 16 rows per column, up to 32 columns (eight lanes each)
# and more, and many sums
@pytest.mark.parametrize("shape", [(1008, 32), (1009, 32), (1024, 33), (1025, 1), (1040, 31),
                                   (30000, 3), (30011, 32)])
def test_posteriors_of_tall_maps(shape):
    from pyfstat_gb300 import _lib

    n_t0, n_tau = shape
    t0_data, A = synth.merged_atoms(2, 90, 1)
    t0s = (t0_data + 5 * np.arange(n_t0)).astype(np.uint32)
    taus = (1800 + 3600 * np.arange(n_tau)).astype(np.uint32)
    h = _lib.Handle(0)
    F, r = h.map_plain_host(A, 1800, t0_data, 1, t0s, taus,
                            flags=_lib.TCW_FLAG_LNBTSG | _lib.TCW_FLAG_POSTERIORS)
    e = np.exp(F.astype(np.float64) - F.max())
    for idx, sums in ((r["t0_mp_idx"], e.sum(1)), (r["tau_mp_idx"], e.sum(0))):
        assert sums[idx] >= sums.max() * (1.0 - 1e-6)
    h.close()
