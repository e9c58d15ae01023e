"""Exponential columns cut into row chunks whose starts are combined from
segment sums: against the FP64 oracle and against columns walked whole."""

import numpy as np
import pytest
from _helpers import REL_TOL, argmax_ok, rel_err

from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu

# (SFTs, t0 points, tau points, t0 step, first tau, tau step, gap fraction):
# atoms just below, at and above the smallest size that is cut and around a
# power of four (segment length), one and several column groups with a
# ragged last one, fewer t0 points than atoms and more, windows clamped at
# the data's end and not, long gaps, taus shorter than an SFT
CASES = [(63, 40, 33, 1800, 1800, 900, 0.0), (64, 64, 32, 1800, 1800, 1800, 0.1),
         (129, 9, 1, 25200, 90000, 1, 0.0), (255, 300, 65, 1500, 1800, 5400, 0.0),
         (1024, 200, 70, 9000, 43200, 7200, 0.3), (1023, 700, 40, 2600, 600, 1111, 0.9),
         (2500, 17, 31, 240000, 3600, 140000, 0.05)]


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_chunked_columns_match_the_oracle_and_whole_columns(oracle, case, shuffled):
    torch = pytest.importorskip("torch")
    from pyfstat_gb300 import _lib
    from pyfstat_gb300.batched import TransientMapBatch

    nsft, n_t0, n_tau, dt0, tau, dtau, gap = case
    t0_data, A = synth.merged_atoms(nsft, nsft, 1, gap_frac=gap)
    t0s = (t0_data + dt0 * np.arange(n_t0)).astype(np.uint32)
    if shuffled:
        t0s = np.random.default_rng(1).permutation(t0s)
    taus = (tau + dtau * np.arange(n_tau)).astype(np.uint32)
    F64, cond = oracle.map_f64(A, 1800, t0_data, 2, t0s, taus, with_cond=True)
    t = dict(window=2, atoms=A, TAtom=1800, t0_data=t0_data, t0s=t0s, taus=taus)
    batch = TransientMapBatch([t, t])
    res, maps = batch.plan.run_maps_host(batch.atoms)
    whole = TransientMapBatch([t], tile_config=dict(exp_rows=n_t0), handle=batch.handle)
    wres, wmap = whole.plan.run_maps_host(whole.atoms)
    Fp, rp = batch.handle.map_plain_host(A, 1800, t0_data, 2, t0s, taus)
    for name, F, r in (("batch", maps[:n_t0 * n_tau], res[0]),
                       ("batch again", maps[n_t0 * n_tau:], res[1]),
                       ("whole", wmap, wres[0]), ("plain", Fp.reshape(-1), rp)):
        rel, _ = rel_err(F.reshape(F64.shape), F64, cond)
        assert rel.max() <= REL_TOL, (name, rel.max())
        assert float(r["maxF"]) == F.max(), name
        assert argmax_ok(int(r["argmax"]), F64, label=f"exp chunks {case} {name}"), name
        assert float(r["lnBtSG"]) == pytest.approx(oracle.lnBtSG(F64), rel=REL_TOL), name
    # the fused run takes the same chunks as the run that writes maps
    d_atoms = torch.from_numpy(batch.atoms).cuda()
    d_res = torch.zeros(10, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    batch.run_device(d_atoms, d_res)
    batch.handle.sync()
    fused = d_res.cpu().numpy().view(_lib.RESULT_DTYPE)
    assert np.array_equal(fused["maxF"], res["maxF"])
    assert np.array_equal(fused["argmax"], res["argmax"])
    for b in (batch, whole):
        b.close()


# rows much finer than the atoms: run-ups of a chunk's short windows over
# several row tables (128 rows), chunks of different lengths side by side
@pytest.mark.parametrize("case", [(217, 1754, 70, 222, 1800, 331, 0.1),
                                  (100, 129, 33, 900, 1800, 60, 0.0),
                                  (64, 2600, 40, 44, 600, 97, 0.2)])
def test_chunks_of_rows_finer_than_the_atoms(oracle, case):
    test_chunked_columns_match_the_oracle_and_whole_columns(oracle, case, False)
