"""The pruning screen's parent-pair table at the sizes where it can go wrong:
two elites, table sizes around a bitmap word, the largest bitmap (362 elites)
and the first table read directly (363), the most elites the library takes,
with and without a linear tail, in the reference's order and the FP64 ranking.
Every screen must return the unpruned screen's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("tail", [False, True])
@pytest.mark.parametrize("ne", [2, 3, 33, 362, 363, 1536])
def test_pair_table_sizes(monkeypatch, ne, tail):
    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    rng = np.random.default_rng(ne + 7 * tail)
    w = rng.normal(0, 1, 166 if tail else 153).astype(np.float32)
    if tail:
        w[17:30] *= 5
    m = screen.Model.from_compact(w)
    el = wl.seeded_elites(ne, seed=ne)
    el["g"][0, :4] = [0.0, 1.0, 7.5, np.nan]  # boxes cut by [0, 1], clamped and NaN genes
    for form in (0, _lib.FLAG_TC_BF16):
        for sigma in (0.12, 0.004, 0.9):
            got, n = screen.screen(screen.Cfg(700_001, 100, 5, threads=3, sigma=sigma, flags=form), m, el)
            ref, k = screen.screen(screen.Cfg(700_001, 100, 5, threads=3, sigma=sigma,
                                              flags=form | _lib.FLAG_NO_PRUNE), m, el)
            assert n == k == 700_001
            assert got.tobytes() == ref.tobytes(), (form, sigma)


@pytest.mark.parametrize("sigma,tail", [(0.0, False), (0.0, True), (0.05, False)])
def test_tied_survivors_with_pair_tables(monkeypatch, sigma, tail):
    """Streams replayed for exact ties through the pair tables: integer weights
    on genes of a coarse grid tie by the hundred (sigma 0), in the pruned single
    screen and in a batch; the unpruned screen replays them without tables."""
    from codec_arena_gb300 import _lib, islands, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    rng = np.random.default_rng(5)
    w = rng.integers(-3, 4, 166 if tail else 153).astype(np.float32)
    m = screen.Model.from_compact(w)
    el = wl.seeded_elites(40, seed=2)
    el["g"] = np.round(el["g"] * 4) / 4
    cfg = screen.Cfg(2_000_003, 100, 9, threads=3, sigma=sigma)
    got, n = screen.screen(cfg, m, el)
    ref, _ = screen.screen(screen.Cfg(2_000_003, 100, 9, threads=3, sigma=sigma, flags=_lib.FLAG_NO_PRUNE), m, el)
    assert n == 2_000_003
    if sigma == 0.0:
        assert len(set(zip(ref["score"].tolist(), ref["stream"].tolist()))) < len(ref)  # ties inside a stream
    assert got.tobytes() == ref.tobytes()
    for surv, k in islands.screen_batch([cfg, cfg], [m, m], [el, el]):
        assert k == n and surv.tobytes() == ref.tobytes()


@pytest.mark.parametrize("keep,ne,tail", [(2048, 1024, False), (2048, 1025, True), (4096, 1100, False)])
def test_long_lists_beside_many_elites(monkeypatch, orc, keep, ne, tail):
    """Lists of 4096 entries leave no room for the box table of more than 1024
    elites: the kernel reads it where it is, with the oracle's survivors."""
    import os

    from codec_arena_gb300 import screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    rng = np.random.default_rng(keep + ne)
    w = rng.normal(0, 1, 166 if tail else 153).astype(np.float32)
    el = wl.seeded_elites(ne, seed=3)
    got, n = screen.screen(screen.Cfg(300_001, keep, 5, threads=3), screen.Model.from_compact(w), el)
    assert screen.last_run_info()["screen_ctas"] > 0
    want, wn = orc.screen(orc.cfg(300_001, keep, 5, threads=3), orc.model_from_compact(w), el,
                          cpu_threads=os.cpu_count() or 4)
    assert n == wn == 300_001 and got.tobytes() == want.tobytes()


@pytest.mark.parametrize("lam,nf,flag", [(22_800_000, 153, 0), (23_000_000, 153, 0), (2_300_000, 161, 0x20),
                                         (2_400_000, 161, 0x20), (20_000_000, 465, 0), (22_000_000, 465, 0)])
def test_both_sides_of_the_pruning_floor(monkeypatch, lam, nf, flag):
    """The automatic choice at 64 elites, either side of the floor (128 + 68
    candidates per thread; 20 with FP64 ranking; 180 on the full surface),
    against the screen without pruning."""
    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.delenv("CSX_PRUNE_MIN_CANDS", raising=False)
    w = np.random.default_rng(nf).normal(0, 0.3, nf).astype(np.float32)
    m = screen.ModelFull.from_compact(w) if nf == 465 else screen.Model.from_compact(w)
    el = wl.seeded_elites(64, seed=3)
    got, n = screen.screen(screen.Cfg(lam, 192, 5, threads=4, flags=flag), m, el)
    ref, k = screen.screen(screen.Cfg(lam, 192, 5, threads=4, flags=flag | _lib.FLAG_NO_PRUNE), m, el)
    assert n == k == lam and got.tobytes() == ref.tobytes()


@pytest.mark.parametrize("floor", ["79999", "80001"])
def test_batch_prunes_by_its_mean_island(monkeypatch, floor):
    """Islands of 40,000, 40,000 and 160,000 candidates (a mean of 80,000) and an
    empty one, either side of the floor; each equals its single screen."""
    from codec_arena_gb300 import islands, screen, workloads as wl

    rng = np.random.default_rng(2)
    models = [screen.Model.from_compact(rng.normal(0, 1, 153).astype(np.float32)) for _ in range(4)]
    el = [wl.seeded_elites(20 + j, seed=j) for j in range(4)]
    cfgs = [screen.Cfg(lam, 30, 5 + j, threads=2) for j, lam in enumerate((40_000, 40_000, 0, 160_000))]
    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", floor)
    res = islands.screen_batch(cfgs, models, el)
    for c, m, e, (surv, n) in zip(cfgs, models, el, res):
        assert n == c.lambda_
        if c.lambda_:
            want, _ = screen.screen(c, m, e)
            assert surv.tobytes() == want.tobytes()


@pytest.mark.parametrize("ne", [5, 33, 64, 362])
def test_thresholds_that_settle_elsewhere(monkeypatch, ne):
    """Lists longer than a CTA's own finds: its first finite threshold arrives from
    other CTAs while it screens, at the rounds that rebuild the pair bitmap."""
    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    m = screen.Model.from_compact(np.random.default_rng(ne).normal(0, 1, 153).astype(np.float32))
    el = wl.seeded_elites(ne, seed=ne)
    for seed in range(8):
        for lam, keep in ((900_001, 700), (5_000_003, 1500)):
            got, n = screen.screen(screen.Cfg(lam, keep, seed, threads=5), m, el)
            ref, _ = screen.screen(screen.Cfg(lam, keep, seed, threads=5, flags=_lib.FLAG_NO_PRUNE), m, el)
            assert n == lam and got.tobytes() == ref.tobytes(), (seed, lam)


@pytest.mark.parametrize("keep,nf", [(700, 161), (2047, 161), (4096, 161), (2047, 465)])
def test_long_lists_share_a_threshold(monkeypatch, keep, nf):
    """Lists longer than four survivors per CTA: the published positions still
    cover K, so that a small part of 5e7 candidates is scored in full (the
    threshold of 4,096 of them lies 3.8 s.d. up, a CTA's own 4,096 of 330,000 2.2)."""
    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    m = (screen.ModelFull.from_compact(wl.seeded_normal_model(seed=3, n=465)) if nf == 465
         else screen.Model.from_compact(wl.surrogate_161()))
    el = wl.seeded_elites(64, seed=2)
    got, n = screen.screen(screen.Cfg(50_000_000, keep, 3, threads=4, flags=_lib.FLAG_STAGE_TIMES), m, el)
    evals = screen.last_run_info()["exact_evals"]
    ref, _ = screen.screen(screen.Cfg(50_000_000, keep, 3, threads=4, flags=_lib.FLAG_NO_PRUNE), m, el)
    assert n == 50_000_000 and got.tobytes() == ref.tobytes()
    assert evals < 0.2 * n, evals / n


@pytest.mark.parametrize("nf,ne,kw", [(161, 64, {}), (161, 2, {"imm_p": 0.0, "jump_p": 1.0}), (166, 33, {"imm_p": 0.0}),
                                      (153, 300, {"imm_p": 0.5}), (161, 40, {"imm_p": 1.0})])
@pytest.mark.parametrize("lam,keep", [(400_001, 7), (30_000_001, 192)])
def test_bounds_that_rule_out_nothing(monkeypatch, nf, ne, kw, lam, keep):
    """Elites that are alike and at the top (and candidates that are always
    scored): most rounds score without the bounds, each candidate once, instead of
    queueing nearly all of them."""
    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    m = screen.Model.from_compact(wl.surrogate_161() if nf == 161 else wl.seeded_normal_model(seed=8, n=nf))
    el = wl.seeded_elites(max(ne, 64), seed=2)
    for gen in range(3):
        top, _ = screen.screen(screen.Cfg(2_000_000, 64, gen, threads=4), m, el)
        el["g"][:64] = top["g"]
    el = el[:ne].copy()
    el["g"] = top["g"][0] + 0.01 * np.random.default_rng(1).random((ne, 29), dtype=np.float32)
    got, n = screen.screen(screen.Cfg(lam, keep, 3, threads=3, sigma=0.07, flags=_lib.FLAG_STAGE_TIMES, **kw), m, el)
    evals = screen.last_run_info()["exact_evals"]
    ref, _ = screen.screen(screen.Cfg(lam, keep, 3, threads=3, sigma=0.07, flags=_lib.FLAG_NO_PRUNE, **kw), m, el)
    assert n == lam and got.tobytes() == ref.tobytes()
    if lam > 1e7:
        assert evals < 0.3 * n, evals / n


@pytest.mark.parametrize("nf", [161, 465])
def test_tie_replay_where_the_tables_rule_out_nothing(orc, monkeypatch, nf):
    """Elites of one genome at 0 and 1 and no mutation: every crossover candidate
    ties with the best, so that the replay's tables leave whole chunks and the later
    ones are read without them (a stream of 1e6 has chunks past 2^18)."""
    import os

    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    w = np.random.default_rng(4).integers(-2, 3, nf).astype(np.float32)
    el = wl.seeded_elites(12, seed=2)
    el["g"] = np.round(el["g"][0])
    kw = dict(threads=2, sigma=0.0, jump_p=0.1, imm_p=0.05)
    m = (screen.ModelFull if nf == 465 else screen.Model).from_compact(w)
    got, n = screen.screen(screen.Cfg(2_000_001, 50, 9, **kw), m, el)
    ref, _ = screen.screen(screen.Cfg(2_000_001, 50, 9, flags=_lib.FLAG_NO_PRUNE, **kw), m, el)
    assert n == 2_000_001 and got.tobytes() == ref.tobytes()
    if nf == 161:
        want, _ = orc.screen(orc.cfg(2_000_001, 50, 9, **kw), orc.model_from_compact(w), el,
                             cpu_threads=os.cpu_count() or 4)
        assert got.tobytes() == want.tobytes()
