"""Prefix rows from a cluster per template against one block per template, and
repacked atom rows across gaps longer than a block."""

import numpy as np
import pytest
from _helpers import REL_TOL, rel_err

from pyfstat_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsft", [1, 7, 255, 256, 257, 511, 2049, 5000])
def test_prefix_cluster_gives_the_block_kernels_bits(nsft):
    """601 rectangular templates take one block each, a single one a cluster:
    the maps are the same bit for bit."""
    from pyfstat_gb300.batched import TransientMapBatch

    t0_data, A = synth.merged_atoms(nsft, nsft, 1, gap_frac=0.1)
    t0s = (t0_data + max(1, nsft // 40) * 1800 * np.arange(33)).astype(np.uint32)
    taus = (1800 + max(1, nsft // 30) * 1800 * np.arange(35)).astype(np.uint32)
    t = dict(window=1, atoms=A, TAtom=1800, t0_data=t0_data, t0s=t0s, taus=taus)
    many = TransientMapBatch([t] * 601)
    _, maps = many.plan.run_maps_host(many.atoms)
    one, _ = many.handle.map_plain_host(A, 1800, t0_data, 1, t0s, taus)
    maps = maps.reshape(601, 33, 35).view(np.uint32)
    assert np.array_equal(maps[0], one.view(np.uint32))
    assert np.array_equal(maps[600], maps[0])
    many.close()


@pytest.mark.parametrize("zeros", [(0, 300), (250, 257), (200, 900), (700, 1000), (0, 1000)])
def test_windows_in_gaps_longer_than_a_repack_block(oracle, zeros):
    """Atoms zeros[0]..zeros[1]-1 of 1000 hold no data: windows inside the gap
    have F = 2, windows that reach across it see the first atom behind it."""
    from pyfstat_gb300 import _lib

    t0_data, A = synth.merged_atoms(5, 1000, 1)
    A[zeros[0]:zeros[1]] = 0.0
    t0s = (t0_data + 12600 * np.arange(143)).astype(np.uint32)
    taus = (5400 + 19800 * np.arange(40)).astype(np.uint32)
    F64, cond = oracle.map_f64(A, 1800, t0_data, 2, t0s, taus, with_cond=True)
    h = _lib.Handle(0)
    F, _ = h.map_plain_host(A, 1800, t0_data, 2, t0s, taus)
    rel, _ = rel_err(F, F64, cond)
    assert rel.max() <= REL_TOL
    h.close()


@pytest.mark.parametrize("n", [1, 3, 400])
@pytest.mark.parametrize("cfg", [None, dict(rect_tm=64, rect_tn=48)])
def test_plan_info_reports_the_rect_tiles_in_use(n, cfg):
    """Small plans take small rectangular tiles: the reported shape gives the
    reported number of tiles."""
    from pyfstat_gb300.batched import TransientMapBatch

    t0_data, A = synth.merged_atoms(3, 300, 1)
    t = dict(window=1, atoms=A, TAtom=1800, t0_data=t0_data,
             t0s=(t0_data + 1800 * np.arange(290)).astype(np.uint32),
             taus=(1800 + 1800 * np.arange(270)).astype(np.uint32))
    batch = TransientMapBatch([t] * n, tile_config=cfg)
    c = batch.tile_config
    assert batch.plan.n_items == n * -(-290 // c["rect_tm"]) * -(-270 // c["rect_tn"]), c
    assert c["exp_tn"] == 32
    if cfg:
        assert (c["rect_tm"], c["rect_tn"]) == (64, 48)
    batch.close()


@pytest.mark.parametrize("n", [0, 70, 9000])
def test_long_template_among_many_short_ones(n):
    """A template of 17532 atoms (gaps across blocks of 256) has the same map by
    itself and behind n templates of 40 atoms, whose launch gives it a few
    blocks only."""
    from pyfstat_gb300.batched import TransientMapBatch

    def template(nsft, n_t0, n_tau):
        t0_data, A = synth.merged_atoms(nsft, nsft, 1, gap_frac=0.1)
        A[nsft // 3:nsft // 2] = 0.0
        span = nsft * 1800
        return dict(window=2, atoms=A, TAtom=1800, t0_data=t0_data,
                    t0s=(t0_data + span // n_t0 * np.arange(n_t0)).astype(np.uint32),
                    taus=(1800 + span // n_tau * np.arange(n_tau)).astype(np.uint32))

    cfg = dict(exp_rows=1 << 16)  # whole columns in both plans
    big, small = template(17532, 21, 33), template(40, 3, 2)
    one = TransientMapBatch([big], tile_config=cfg)
    _, F = one.plan.run_maps_host(one.atoms)
    many = TransientMapBatch([small] * n + [big, small], tile_config=cfg, handle=one.handle)
    _, M = many.plan.run_maps_host(many.atoms)
    assert np.array_equal(M[6 * n:6 * n + F.size].view(np.uint32), F.view(np.uint32))
    many.close()
    one.close()
