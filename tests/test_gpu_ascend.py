"""The ascent's two kernels (sixteen lanes per row up to 30,000 rows, a thread
per row above) and its copying form: the same bits as the in-place call on a
clone, extra columns kept, the input untouched, for each layout's gene count,
strided and overlapping rows, rows around a CTA's sixteen and the limit, no
step, one and several; and tensors whose clone has a place in a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


def _inplace(rows, coef, eta, steps):
    import torch

    from codec_arena_gb300 import _lib

    out = rows.clone()
    sc = torch.empty(len(out), device="cuda")
    _lib.check(_lib.lib().csx_sg_ascend(coef.data_ptr(), coef.numel(), out.data_ptr(), len(out), out.stride(0), eta,
                                        steps, sc.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return out, sc


@pytest.mark.parametrize("ng", [16, 17, 29])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 1000])
@pytest.mark.parametrize("steps", [0, 1, 7])
def test_few_rows_equal_many(n, ng, steps):
    import torch

    from codec_arena_gb300 import surrogate

    g = torch.Generator(device="cuda").manual_seed(n + ng)
    rows = torch.rand(30_001, 32, device="cuda", generator=g)
    coef = torch.randn(1 + ng + 136, device="cuda", generator=g)
    big, bs = _inplace(rows, coef, 0.01, steps)                 # a thread per row
    keep = rows.clone()
    for src in (rows[:n], rows[:n, :30], rows[:n].contiguous()):
        new, sc = surrogate.ascend(src, coef, 0.01, steps)      # lanes, copying
        assert torch.equal(new[:, :ng], big[:n, :ng]) and torch.equal(sc, bs[:n])
        assert torch.equal(new[:, ng:], src[:, ng:])
    many, ms = surrogate.ascend(rows, coef, 0.01, steps)        # a thread per row, copying
    assert torch.equal(many[:, :ng], big[:, :ng]) and torch.equal(many[:, ng:], keep[:, ng:]) and torch.equal(ms, bs)
    small, ss = _inplace(rows[:n], coef, 0.01, steps)           # lanes in place
    assert torch.equal(small[:, :ng], big[:n, :ng]) and torch.equal(ss, bs[:n])
    assert torch.equal(rows, keep)


def test_clones_with_a_place_of_their_own():
    import torch

    from codec_arena_gb300 import surrogate

    rows = torch.rand(40, 29, device="cuda")
    coef = torch.randn(166, device="cuda")
    want, ws = surrogate.ascend(rows, coef, 0.01, 3)
    new, sc = surrogate.ascend(rows.clone().requires_grad_(True), coef, 0.01, 3)
    assert new.requires_grad and torch.equal(new.detach(), want) and torch.equal(sc, ws)
    one = rows[:1].expand(5, 29)                                # rows that overlap
    new, sc = surrogate.ascend(one, coef, 0.01, 3)
    assert torch.equal(new, want[:1].expand(5, 29)) and new.is_contiguous()


def test_dual_numbers_keep_their_tangent():
    import torch
    import torch.autograd.forward_ad as fwd

    from codec_arena_gb300 import surrogate

    rows, t = torch.rand(40, 29, device="cuda"), torch.rand(40, 29, device="cuda")
    coef = torch.randn(166, device="cuda")
    want, ws = surrogate.ascend(rows, coef, 0.01, 3)
    with fwd.dual_level():
        new, sc = surrogate.ascend(fwd.make_dual(rows, t), coef, 0.01, 3)
        primal, tangent = fwd.unpack_dual(new)
        assert torch.equal(primal, want) and torch.equal(tangent, t) and torch.equal(sc, ws)
        new, sc = surrogate.ascend(rows, coef, 0.01, 3)
        assert torch.equal(new, want) and fwd.unpack_dual(new).tangent is None
