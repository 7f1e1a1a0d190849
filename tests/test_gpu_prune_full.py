"""The full surface's pruning screen against the unpruned one: the same
survivors, bytes and count, for one and many elites (shared memory for three,
two and one CTA per SM), tied surfaces, elites outside [0, 1], branch
probabilities at their ends, mutations as wide as the range (the bound leaves
everything and turns itself off), and item ranges of streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


def _both(monkeypatch, w, el, lam, keep, streams=None, **kw):
    from codec_arena_gb300 import _lib, screen

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    m = screen.ModelFull.from_compact(w)
    a, na = screen.screen(screen.Cfg(lam, keep, 11, threads=3, **kw), m, el, streams=streams)
    b, nb = screen.screen(screen.Cfg(lam, keep, 11, threads=3, flags=_lib.FLAG_NO_PRUNE, **kw), m, el,
                          streams=streams)
    assert na == nb
    assert a.tobytes() == b.tobytes()
    return a


@pytest.mark.parametrize("ne", [2, 33, 64, 512, 1536])
@pytest.mark.parametrize("sigma", [0.12, 0.01, 0.0, 0.9])
def test_full_prune_equals_unpruned(monkeypatch, ne, sigma):
    from codec_arena_gb300 import workloads as wl

    el = wl.seeded_elites(ne, seed=ne)
    el["g"][0, :4] = [-3.0, 7.5, np.nan, 1.0]
    w = np.random.default_rng(ne).normal(0, 0.3, 465).astype(np.float32)
    _both(monkeypatch, w, el, 900_001, 100, sigma=sigma)


@pytest.mark.parametrize("imm,jump", [(0.0, 0.0), (1.0, 0.0), (0.0, 1.0), (0.3, 0.3)])
def test_full_prune_branches(monkeypatch, imm, jump):
    from codec_arena_gb300 import workloads as wl

    w = wl.seeded_normal_model(seed=3, n=465)
    _both(monkeypatch, w, wl.seeded_elites(24, seed=4), 300_001, 40, imm_p=imm, jump_p=jump)


def test_full_prune_ties_and_stream_ranges(monkeypatch):
    from codec_arena_gb300 import workloads as wl

    rng = np.random.default_rng(2)
    w = rng.integers(-2, 3, 465).astype(np.float32)
    el = wl.seeded_elites(20, seed=6)
    el["g"] = np.round(el["g"] * 2) / 2
    a = _both(monkeypatch, w, el, 600_001, 80, sigma=0.0)
    assert len(set(zip(a["score"].tolist(), a["stream"].tolist()))) < len(a)
    for k in ([0, 1], [1, 3]):
        _both(monkeypatch, w * 0 + rng.normal(0, 1, 465).astype(np.float32), el, 600_001, 80, streams=tuple(k))
    _both(monkeypatch, np.zeros(465, np.float32), el, 100_001, 30)
