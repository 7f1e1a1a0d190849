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
