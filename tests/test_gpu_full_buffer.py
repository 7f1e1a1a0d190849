"""Screens whose candidates nearly all tie with the K-th score, so that every
flush of a CTA's queue finds its entry buffer without room and merges first: the
pruning screens, the filter, the precision form, the batch and the unfiltered
forms against each other (and, for the ones that rank in the reference's order,
the oracle)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


def _tied(n, seed):
    """Integer weights on few genes, elites at 0 and 1: a handful of exact scores."""
    from codec_arena_gb300 import workloads as wl

    rng = np.random.default_rng(seed)
    w = np.zeros(n, np.float32)
    w[1:4] = rng.integers(0, 2, 3)
    el = wl.seeded_elites(24, seed=seed)
    el["g"] = np.round(el["g"])
    return w, el


@pytest.mark.parametrize("keep", [1, 40, 1000])
@pytest.mark.parametrize("lam,T", [(250_000, 3), (60_001, 1)])
def test_reference_order(orc, keep, lam, T):
    from codec_arena_gb300 import _lib, islands, screen

    w, el = _tied(161, keep)
    kw = dict(threads=T, sigma=0.0, jump_p=0.2)
    want, _ = orc.screen(orc.cfg(lam, keep, 5, **kw), orc.model_from_compact(w), el, cpu_threads=os.cpu_count() or 4)
    m = screen.Model.from_compact(w)
    for flags in (0, _lib.FLAG_NO_PRUNE, _lib.FLAG_EXACT_ALL):
        cfg = screen.Cfg(lam, keep, 5, flags=flags, **kw)
        got, n = screen.screen(cfg, m, el)
        assert n == lam and got.tobytes() == want.tobytes(), flags
        both = islands.screen_batch([cfg, cfg], [m, m], [el, el])
        assert all(n == lam and s.tobytes() == want.tobytes() for s, n in both), flags


@pytest.mark.parametrize("keep", [1, 40, 1000])
def test_precision_and_full_surface(keep):
    from codec_arena_gb300 import _lib, screen

    w, el = _tied(161, keep)
    kw = dict(threads=3, sigma=0.0, jump_p=0.2)
    for tc in (_lib.FLAG_TC_BF16, _lib.FLAG_TC_FP16):
        a, b = (screen.screen(screen.Cfg(250_000, keep, 5, flags=tc | f, **kw), screen.Model.from_compact(w), el)[0]
                for f in (0, _lib.FLAG_NO_PRUNE))
        assert a.tobytes() == b.tobytes()
    w, el = _tied(465, keep)
    a, b = (screen.screen(screen.Cfg(250_000, keep, 5, flags=f, **kw), screen.ModelFull.from_compact(w), el)[0]
            for f in (0, _lib.FLAG_NO_PRUNE))
    assert a.tobytes() == b.tobytes()
