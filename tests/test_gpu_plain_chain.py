"""Single maps through the chain of dependent launches: map, result record and
posterior bins against the FP64 oracle at the edges of tiles and chunks."""

import numpy as np
import pytest
from _helpers import REL_TOL, argmax_ok, index_ok, rel_err

from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu

# window, SFTs, t0 points, t0 step, tau points, tau step: one cell; one more
# and one fewer than a row tile, a column strip of the posteriors, a part of
# their argmax and a row chunk; few rows under long windows; more input than
# one staging copy takes
CASES = [(1, 1, 1, 1800, 1, 1800), (2, 40, 1, 1800, 33, 1800), (1, 300, 33, 9000, 1025, 450),
         (2, 300, 31, 9000, 1023, 900), (1, 120, 8193, 25, 17, 5400),
         (2, 900, 257, 6300, 40, 36000), (2, 4000, 40, 180000, 70, 90000),
         (1, 40000, 9, 7200000, 5, 9000000)]


@pytest.mark.parametrize("case", CASES)
def test_chain_matches_the_oracle(oracle, case):
    from pyfstat_gb300 import _lib

    window, nsft, n_t0, dt0, n_tau, dtau = case
    t0_data, A = synth.merged_atoms(nsft, nsft, 1, gap_frac=0.1, inject=(nsft // 4, nsft // 3))
    t0s = (t0_data + dt0 * np.arange(n_t0)).astype(np.uint32)
    taus = (3600 + dtau * np.arange(n_tau)).astype(np.uint32)
    F64, cond = oracle.map_f64(A, 1800, t0_data, window, t0s, taus, with_cond=True)
    h = _lib.Handle(0)
    flags = _lib.TCW_FLAG_LNBTSG | _lib.TCW_FLAG_POSTERIORS
    for _ in range(2):  # the second call reuses the workspace
        F, r = h.map_plain_host(A, 1800, t0_data, window, t0s, taus, flags=flags)
        rel, _ = rel_err(F, F64, cond)
        assert rel.max() <= REL_TOL
        assert float(r["maxF"]) == F.max()
        assert argmax_ok(int(r["argmax"]), F64, label=f"chain {case}")
        assert float(r["lnBtSG"]) == pytest.approx(oracle.lnBtSG(F64), rel=REL_TOL)
        # marginals from the written map, as the posteriors are defined
        e = np.exp(F.astype(np.float64) - float(r["maxF"]))
        assert index_ok(int(r["t0_mp_idx"]), e.sum(1), tol=1e-6, label=f"chain t0 {case}")
        assert index_ok(int(r["tau_mp_idx"]), e.sum(0), tol=1e-6, label=f"chain tau {case}")
    # no map, no posteriors: the same record
    _, q = h.map_plain_host(A, 1800, t0_data, window, t0s, taus, want_map=False,
                            flags=_lib.TCW_FLAG_LNBTSG)
    for k in ("maxF", "argmax", "lnBtSG"):
        assert q[k] == r[k], k
    assert int(q["t0_mp_idx"]) == -1
    h.close()
