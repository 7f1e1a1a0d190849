"""The cluster's ridge solve at the sizes where its layout changes: fewer rows
than CTAs, a panel's remainders, a last block of unknowns of one to 32, the
largest layout held in one CTA and the full surface's; many solves in a row
on one and on several streams, which start while earlier clusters still run.

Tolerance: the matrices are diagonally dominant (row sums of the off-diagonal
below half of the diagonal), so LDL' has no growth and a condition number below
3; every unknown passes at most n roundings per sum of the factorisation and of
the two substitutions: 8 n 2^-53 of the largest unknown, with room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


def _system(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(n, n))
    a = (a + a.T) / 2
    np.fill_diagonal(a, 0.0)
    np.fill_diagonal(a, 2 * np.abs(a).sum(1) + 1)
    return a, rng.normal(size=n), rng.normal(size=n)


def _close(w, a, b, n):
    want = np.linalg.solve(a, b)
    np.testing.assert_allclose(w, want, rtol=0, atol=8 * n * 2.0 ** -53 * np.abs(want).max() + 1e-300)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 63, 64, 65, 153, 161, 165, 166, 465])
def test_solve_sizes(n):
    import torch

    from codec_arena_gb300 import surrogate

    a, b, prior = _system(n, n)
    w = surrogate.ridge_solve(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), 0.5,
                              torch.from_numpy(prior).cuda())
    _close(w.cpu().numpy(), a + 0.5 * np.eye(n), b + 0.5 * prior, n)


@pytest.mark.parametrize("n", [1, 9, 166])
def test_solves_in_a_row(n):
    import torch

    from codec_arena_gb300 import _lib

    streams = [torch.cuda.Stream() for _ in range(3)]
    sys = [_system(n, 100 * n + i) for i in range(12)]
    dev = [(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()) for a, b, _ in sys]
    out = torch.full((12, n), float("nan"), dtype=torch.float64, device="cuda")
    status = torch.full((12,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for rep in range(20):
        for i, (a, b) in enumerate(dev):
            _lib.check(_lib.lib().csx_sg_ridge_solve(n, a.data_ptr(), b.data_ptr(), 0.0, None, out[i].data_ptr(),
                                                     status[i:].data_ptr(), streams[i % 3].cuda_stream))
    torch.cuda.synchronize()
    assert not status.any()
    for i, (a, b, _) in enumerate(sys):
        _close(out[i].cpu().numpy(), a, b, n)


@pytest.mark.parametrize("n", [1, 4, 33, 153, 166, 465])
@pytest.mark.parametrize("lo,hi", [(-500, -500), (500, 500), (-480, 480), (-535, -530)])
def test_rows_of_any_exponent(n, lo, hi):
    """Rows and columns multiplied by powers of two: the unscaled system's bits,
    scaled back (down to a diagonal of subnormals, where the matrix is diagonal)."""
    import torch

    from codec_arena_gb300 import surrogate

    a, b, _ = _system(n, n + 1)
    if lo < -500:
        a = np.diag(2.0 ** np.random.default_rng(n).integers(0, 20, n))
    s = np.random.default_rng(n).integers(lo, hi + 1, n)
    scaled = np.ldexp(np.ldexp(a, s[:, None]), s[None, :])
    w0 = surrogate.ridge_solve(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), 0.0).cpu().numpy()
    w = surrogate.ridge_solve(torch.from_numpy(scaled).cuda(), torch.from_numpy(np.ldexp(b, s)).cuda(), 0.0)
    assert np.isfinite(w0).all()
    np.testing.assert_array_equal(w.cpu().numpy(), np.ldexp(w0, -s))


@pytest.mark.parametrize("n", [1, 9, 166, 465])
@pytest.mark.parametrize("pivot", [0.0, -1.0, float("nan")])
def test_a_failed_factorisation_leaves_no_weights(n, pivot):
    import torch

    from codec_arena_gb300 import _lib

    k = n // 2
    a = np.eye(n)
    a[k, k] = pivot
    g, b = torch.from_numpy(a).cuda(), torch.ones(n, dtype=torch.float64, device="cuda")
    w = torch.zeros(n, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().csx_sg_ridge_solve(n, g.data_ptr(), b.data_ptr(), 0.0, None, w.data_ptr(),
                                             status.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert status.item() == k + 1 and w.isnan().all()


def test_pivot_reciprocal():
    """1 / d of a diagonal matrix's pivots, over significands (ones next to powers
    of two among them) and exponents. Two Newton steps square the seed's 2^-22
    twice, so the last step's rounding is what is left: at most one unit of 2^-52
    of the result (a half, and room for the residual's)."""
    import torch

    from codec_arena_gb300 import surrogate

    rng = np.random.default_rng(1)
    for rep in range(40):
        m = 1.0 + rng.random(465)
        m[:8] = [1.0, 1 + 2.0 ** -52, 2 - 2.0 ** -52, 1 + 2.0 ** -23, 2 - 2.0 ** -23, 1.5, 4 / 3, 1 + 2.0 ** -29]
        d = np.ldexp(m, rng.integers(-1021, 1022, 465))
        w = surrogate.ridge_solve(torch.from_numpy(np.diag(d)).cuda(), torch.ones(465, dtype=torch.float64).cuda(), 0.0)
        want = 1.0 / d
        assert np.all(np.abs(w.cpu().numpy() - want) <= 2.0 ** -52 * want)
