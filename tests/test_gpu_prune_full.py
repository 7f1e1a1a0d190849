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


@pytest.mark.parametrize("ne", [2, 40])
def test_full_prune_backs_off(monkeypatch, ne):
    """A surface that the bound is used for (its slack is within the limit of
    its spread over uniform genes), elites that are alike, and nothing but
    crossover and mutation: the bound of every candidate is the elites' score
    and the slack, above every score there is, so each round that computes it
    leaves everything. 1.5e8 candidates are some 80 rounds of 456 CTAs: past the
    sixteenth that leaves more than half, and into the longer pauses."""
    from codec_arena_gb300 import _lib, screen, workloads as wl

    monkeypatch.setenv("CSX_PRUNE_MIN_CANDS", "0")
    m = screen.ModelFull.from_compact(wl.seeded_normal_model(seed=3, n=465))
    el = wl.seeded_elites(ne, seed=4)
    el["g"] = el["g"][0]
    lam, kw = 150_000_001, dict(threads=3, imm_p=0.0, jump_p=0.0)
    got, n = screen.screen(screen.Cfg(lam, 60, 11, flags=_lib.FLAG_STAGE_TIMES, **kw), m, el)
    evals = screen.last_run_info()["exact_evals"]  # the unpruned kernel counts none
    ref, nr = screen.screen(screen.Cfg(lam, 60, 11, flags=_lib.FLAG_NO_PRUNE, **kw), m, el)
    assert n == nr == lam and got.tobytes() == ref.tobytes()
    assert evals > 0.99 * lam
