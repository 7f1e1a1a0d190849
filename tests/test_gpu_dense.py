"""Work items from block maps (small generations) against the walk's items
(CSX_SEG_CANDS selects the walk): the same survivors, bytes and count, where a
stream ends inside a block, at a block's end and a group's, with one stream
of several tiles of groups and with many short streams, at every branch
probability, on both sides of the block sizes and of the budget limit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("lam,T,imm,jump", [
    (2_000, 1, 0.01, 0.02), (16_384, 1, 0.0, 0.0), (16_385, 1, 0.0, 0.0), (264_258, 1, 0.0, 0.0),
    (33_000, 2, 1.0, 0.0), (33_001, 3, 1.0, 1.0), (40_000, 1, 0.0, 1.0), (90_001, 5, 0.5, 0.5),
    (500_000, 4, 0.01, 0.02), (500_001, 4, 0.01, 0.02), (1_000_000, 3000, 0.01, 0.02), (3_000_000, 1, 0.01, 0.02),
    (7_999_999, 7, 0.01, 0.02), (8_000_001, 7, 0.01, 0.02)])
def test_dense_items_equal_the_walks(monkeypatch, lam, T, imm, jump):
    from codec_arena_gb300 import _lib, screen, workloads as wl

    m = screen.Model.from_compact(wl.surrogate_161())
    el = wl.seeded_elites(24, seed=3)
    cfg = screen.Cfg(lam, 100, 11, threads=T, imm_p=imm, jump_p=jump, flags=_lib.FLAG_NO_PRUNE)
    a, na = screen.screen(cfg, m, el)
    shards = [screen.screen(cfg, m, el, items=(r, 3)) for r in range(3)]
    monkeypatch.setenv("CSX_SEG_CANDS", "5000")
    b, nb = screen.screen(cfg, m, el)
    assert na == nb == lam == sum(n for _, n in shards)
    assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("lam,T,cands", [(2_000, 1000, 64), (200_000, 4, 8), (500_001, 4, 16), (8_000_000, 7, 16),
                                         (8_000_001, 7, 64)])
def test_run_info_describes_the_items(monkeypatch, lam, T, cands):
    """Streams of one item, block maps of both sizes, and the walk past them."""
    from codec_arena_gb300 import screen, workloads as wl

    for name in ("CSX_SEG_CANDS", "CSX_ITEM_CANDS"):
        monkeypatch.delenv(name, raising=False)
    screen.screen(screen.Cfg(lam, 100, 11, threads=T), screen.Model.from_compact(wl.surrogate_161()),
                  wl.seeded_elites(24, seed=3))
    info = screen.last_run_info()
    assert info["item_cands"] == cands
    if lam <= 8_000_000:
        assert info["segments"] == info["seg_draws"] == 0
    else:
        assert info["segments"] >= T and info["seg_draws"] > 0
    if T > 500:
        assert info["items"] == T
    else:  # all but the streams' and the segments' ends hold that many
        assert 0.95 * cands <= lam / info["items"] <= 1.1 * cands
