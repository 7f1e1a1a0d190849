"""score's backward allocates what its kernel writes: n rows of the stride that
is passed, for column slices of a wider table, single rows of any stride and
rows that overlap past the layout's genes. The library's calls are replaced by
a recorder: the host's side alone, on CPU tensors."""
import pytest
import torch

from codec_arena_gb300 import _lib, surrogate


@pytest.mark.parametrize("n", [0, 1, 7])
@pytest.mark.parametrize("cols,ld", [(29, 32), (29, 29), (32, 30), (29, 100)])
def test_gradient_rows_hold_what_the_kernel_writes(monkeypatch, n, cols, ld):
    seen = []

    class Lib:
        def csx_sg_forward(self, *a):
            return 0

        def csx_sg_backward_f32(self, coef, nf, genes, n, ldg, precision, gout, dgenes, *a):
            seen.append((n, ldg, dgenes))
            return 0

    monkeypatch.setattr(surrogate, "lib", Lib)
    monkeypatch.setattr(surrogate, "_genes", lambda g: g)
    monkeypatch.setattr(surrogate, "_stream", lambda device: 0)
    rows = torch.rand(8 * ld + 64).as_strided((n, cols), (ld, 1)).requires_grad_(True)
    s = surrogate.score(rows, torch.randn(166), _lib.SG_FP32)
    (dg,) = torch.autograd.grad(s, (rows,), torch.ones(n))
    ((rows_n, ldg, ptr),) = seen
    assert rows_n == n and dg.shape == rows.shape and dg.data_ptr() == ptr
    assert dg.untyped_storage().nbytes() >= 4 * n * ldg
    assert n < 2 or dg.stride(0) == ldg
