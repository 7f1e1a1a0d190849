"""score's gradients on column slices of a wider table and on rows that overlap
past the layout's genes: the bits of the contiguous copy's gradients (the
kernel writes rows at the stride it reads them)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


def _grads(rows, coef, gout, precision):
    import torch

    from codec_arena_gb300 import surrogate

    c = coef.clone().requires_grad_(True)
    s = surrogate.score(rows, c, precision)
    return (s.detach(), *torch.autograd.grad(s, (rows, c), gout))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ng,cols,ld", [(16, 16, 32), (16, 20, 29), (29, 29, 32), (29, 30, 32), (29, 29, 29),
                                        (29, 32, 30)])
@pytest.mark.parametrize("n", [1, 255, 257, 1000])
def test_strided_rows(n, ng, cols, ld, precision):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(n + ld)
    table = torch.rand(n * ld + 64, device="cuda", generator=gen)
    rows = table.as_strided((n, cols), (ld, 1)).requires_grad_(True)
    coef = torch.randn(1 + ng + 136, device="cuda", generator=gen)
    gout = torch.randn(n, device="cuda", generator=gen)
    want = _grads(rows.detach().clone(memory_format=torch.contiguous_format).requires_grad_(True), coef, gout, precision)
    got = _grads(rows, coef, gout, precision)
    for a, b in zip(got, want):
        assert a.shape == b.shape and torch.equal(a, b)
    assert not want[1][:, ng:].any()
