"""Host logic of the tile autotuner: workload signature, template sampling
and sub-batch extraction (no GPU); its timing and a whole tuning on the GPU."""

import numpy as np
import pytest

from pyfstat_gb300 import _lib, autotune, synth
from pyfstat_gb300.batched import pack_templates


def templates(n=40, seed=7):
    return synth.batched_templates(n, seed=seed, nsft_range=(20, 120), grid_range=(4, 60))


def test_subset_equals_packing_the_chosen_templates():
    tl = templates()
    atoms, desc, t0s, taus = pack_templates(tl)
    idx = np.array([1, 4, 5, 17, 38])
    sd, st0, stau, sa = autotune.subset(desc, t0s, taus, atoms, idx)
    ra, rd, rt0, rtau = pack_templates([tl[i] for i in idx])
    assert np.array_equal(sd, rd)
    assert np.array_equal(st0, rt0) and np.array_equal(stau, rtau)
    assert np.array_equal(sa, ra)


def test_sample_covers_both_windows_and_the_budget():
    _, desc, _, _ = pack_templates(templates())
    cells = desc["N_t0"].astype(np.float64) * desc["N_tau"]
    idx = autotune.sample_templates(desc, budget_cells=2000.0, seed=3)
    for w in (_lib.TCW_WINDOW_RECT, _lib.TCW_WINDOW_EXP):
        sel = idx[desc["window"][idx] == w]
        assert sel.size >= 1
        # the sample reaches the budget unless it takes every template of the type
        assert cells[sel].sum() >= 2000.0 or sel.size == np.sum(desc["window"] == w)
    # a budget above the total takes every template
    idx_all = autotune.sample_templates(desc, budget_cells=1e12)
    assert np.array_equal(np.sort(idx_all), np.arange(desc.shape[0]))
    # seeded
    assert np.array_equal(idx, autotune.sample_templates(desc, budget_cells=2000.0, seed=3))


def test_signature_depends_on_the_mix_not_on_the_order():
    tl = templates()
    _, desc, _, _ = pack_templates(tl)
    _, desc_rev, _, _ = pack_templates(tl[::-1])
    assert autotune.signature(desc) == autotune.signature(desc_rev)
    _, desc_rect, _, _ = pack_templates([t for t in tl if t["window"] == 1])
    assert autotune.signature(desc_rect) != autotune.signature(desc)
    assert "w2:0" in autotune.signature(desc_rect)


def test_cache_round_trip(tmp_path, monkeypatch):
    p = tmp_path / "tiles.json"
    monkeypatch.setenv("PYFSTAT_GB300_TUNE_CACHE", str(p))
    assert autotune.cache_path() == str(p)
    autotune._store_cache(str(p), {"k": {"rect_tm": 64}})
    assert autotune._load_cache(str(p)) == {"k": {"rect_tm": 64}}
    assert autotune._load_cache(str(tmp_path / "missing.json")) == {}


def test_choices_of_other_tile_rules_are_not_taken(monkeypatch):
    """The cache key names the version of the library's tile rules, and its own
    tiles are a candidate for both windows."""
    _, desc, _, _ = pack_templates(templates())
    key = autotune.cache_key("GB300", 1, desc)
    assert autotune.signature(desc) in key
    assert key != f"GB300|flags1|{autotune.signature(desc)}"  # the key before the rules had a version
    monkeypatch.setattr(autotune, "TILE_RULES", autotune.TILE_RULES + 1)
    assert autotune.cache_key("GB300", 1, desc) != key
    assert (0, 0) in autotune.RECT_CANDIDATES and (32, 0) in autotune.EXP_CANDIDATES


@pytest.mark.gpu
def test_timed_run_counts_the_segment_sums_as_exponential():
    """17532 atoms x 4096 taus in one plan: segment sums of some 0.2 ms beside a
    repack of a few microseconds."""
    torch = pytest.importorskip("torch")
    from pyfstat_gb300.batched import TransientMapBatch

    t0_data, A = synth.merged_atoms(1, 17532, 1)
    t = dict(window=2, atoms=A, TAtom=1800, t0_data=t0_data,
             t0s=(t0_data + 61200 * np.arange(512)).astype(np.uint32),
             taus=(7200 + 7200 * np.arange(4096)).astype(np.uint32))
    batch = TransientMapBatch([t])
    atoms = torch.from_numpy(batch.atoms).cuda()
    res = torch.zeros(5, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ms = np.min([batch.plan.run_timed(atoms, res) for _ in range(6)], 0)
    assert ms[0] < 0.15 * ms[2], ms
    batch.close()


@pytest.mark.gpu
def test_tune_chooses_among_the_candidates(tmp_path, monkeypatch):
    pytest.importorskip("torch")
    from pyfstat_gb300.batched import TransientMapBatch

    monkeypatch.setenv("PYFSTAT_GB300_TUNE_CACHE", str(tmp_path / "tiles.json"))
    tl = templates(12)
    atoms, desc, t0s, taus = pack_templates(tl)
    h = _lib.Handle(0)
    cfg = autotune.tune(desc, t0s, taus, atoms, h)
    assert (cfg["rect_tm"], cfg["rect_tn"]) in autotune.RECT_CANDIDATES
    assert (cfg["exp_tn"], cfg["exp_rows"]) in autotune.EXP_CANDIDATES
    assert autotune.tune(desc, t0s, taus, atoms, h) == cfg  # from the cache
    res = [TransientMapBatch(tl, tile_config=c, handle=h).run() for c in (cfg, None)]
    np.testing.assert_allclose(res[0]["maxF"], res[1]["maxF"], rtol=1e-6)
    h.close()
