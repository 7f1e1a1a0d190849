"""The refit's normal equations on the tensor cores (fixed point) against
wider host arithmetic, at the edges of a stage (32 rows), a drain (128) and the
row chunks, for each layout's gene count, with signed genes, zero columns,
exact ones, wide exponents and subnormals; and tables with a non-finite entry,
which the FP64 kernel takes.

Tolerance: a scaled feature is rounded by at most 2^-56, so a row's product by
2^-55; the digit products past the seventh add at most 6.1 x 2^-56. Per entry
n x 8.1 x 2^-56 < n x 2^-52 of the columns' scales (each gene's largest value
rounded up to a power of two), and the final rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(csx):
    from conftest import has_gpu

    if not has_gpu():
        pytest.skip("no CUDA device")


def _phi(g, ng):
    ii, jj = np.tril_indices(16)
    one = np.ones((len(g), 1), g.dtype)
    return np.concatenate([one, g[:, :ng], g[:, ii] * g[:, jj]], axis=1)


def _run(genes, y, nf):
    import torch

    from codec_arena_gb300 import surrogate

    gram, rhs = surrogate.normal_equations(torch.from_numpy(genes).cuda(), torch.from_numpy(y).cuda(), nf)
    return gram.cpu().numpy(), rhs.cpu().numpy()


@pytest.mark.parametrize("ng", [16, 17, 29])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 6400, 6401, 9001])
def test_normal_equations_fixed_point(n, ng):
    rng = np.random.default_rng(n + ng)
    g = rng.random((n, ng), dtype=np.float32)
    g[:, 1] = 2 * g[:, 1] - 1                                     # signed
    g[:, 2] = np.round(g[:, 2])                                   # exact zeros and ones
    g[:, 3] = 0.0                                                 # an empty column
    g[:, 4] *= np.float32(2.0) ** rng.integers(-60, 20, n).astype(np.float32)
    g[:, 5] = rng.integers(0, 9, n).astype(np.float32) * np.float32(1e-45)  # subnormals
    g[:, 6] = np.round(g[:, 6], 4)
    y = rng.normal(0, 30, n)
    y[:: 7] *= 1e-9
    gram, rhs = _run(g, y, 1 + ng + 136)
    wide = g.astype(np.longdouble)
    phi = _phi(wide, ng)
    want, wrhs = phi.T @ phi, phi.T @ y.astype(np.longdouble)
    top = np.abs(g).max(0).astype(np.float64)
    scale = np.where(top > 0, 2.0 ** np.ceil(np.log2(np.where(top > 0, top, 1.0))), 1.0)
    fs = _phi(scale[None, :], ng)[0]
    ys = 2.0 ** np.ceil(np.log2(np.abs(y).max()))
    assert np.all(np.abs(gram - want) <= n * 2.0 ** -52 * np.outer(fs, fs) + 2.0 ** -52 * np.abs(want))
    assert np.all(np.abs(rhs - wrhs) <= n * 2.0 ** -52 * fs * ys + 2.0 ** -52 * np.abs(wrhs))
    np.testing.assert_array_equal(gram, gram.T)


@pytest.mark.parametrize("where", ["gene", "y"])
def test_non_finite_tables_keep_the_fp64_kernel(where):
    rng = np.random.default_rng(3)
    g = rng.random((700, 29), dtype=np.float32)
    y = rng.normal(0, 1, 700)
    if where == "gene":
        g[123, 20] = np.inf
    else:
        y[5] = np.nan
    gram, rhs = _run(g, y, 166)
    with np.errstate(invalid="ignore"):
        phi = _phi(g.astype(np.float64), 29)
        want, wrhs = phi.T @ phi, phi.T @ y
    np.testing.assert_allclose(gram, want, rtol=1e-12)
    np.testing.assert_allclose(rhs, wrhs, rtol=1e-9, atol=1e-9)


@pytest.mark.parametrize("off", [0, 8, 16, 24])
@pytest.mark.parametrize("ng", [16, 29])
def test_workspace_at_any_double(off, ng):
    """A workspace of the stated size from any 8-byte boundary: the same bits, and
    nothing written around it."""
    import torch

    from codec_arena_gb300 import _lib, surrogate

    rng = np.random.default_rng(ng)
    n, nf = 6401, 1 + ng + 136
    genes = torch.from_numpy(rng.random((n, ng), dtype=np.float32)).cuda()
    y = torch.from_numpy(rng.normal(0, 3, n)).cuda()
    want, wrhs = surrogate.normal_equations(genes, y, nf)
    size = int(_lib.lib().csx_sg_workspace_bytes(nf))
    buf = torch.full((size + 64,), 0x5a, dtype=torch.uint8, device="cuda")
    assert buf.data_ptr() % 16 == 0
    gram = torch.empty((nf, nf), dtype=torch.float64, device="cuda")
    rhs = torch.empty(nf, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().csx_sg_normal_equations(nf, genes.data_ptr(), n, ng, y.data_ptr(), gram.data_ptr(),
                                                  rhs.data_ptr(), buf.data_ptr() + off,
                                                  torch.cuda.current_stream().cuda_stream))
    assert torch.equal(gram, want) and torch.equal(rhs, wrhs)
    assert (buf[:off] == 0x5a).all() and (buf[off + size:] == 0x5a).all()


def _table(kind, n, ng, rng):
    import os

    from codec_arena_gb300 import genome, workloads as wl

    g = rng.random((n, ng), dtype=np.float32)
    if kind.startswith("pop"):
        pop = genome.load_elites(os.path.join(wl.GOLDEN_DIR, "pop_seed_96.txt"), v6_fix=True)["g"]
        p = np.clip(pop[rng.integers(0, len(pop), n), :ng] + 0.24 * (rng.random((n, ng)) - 0.5), 0, 1)
        g = np.where(rng.random((n, 1)) < 0.05, g, p)
    y = _phi(g.astype(np.float64), ng) @ rng.normal(0, 1, 1 + ng + 136) + 0.5 * rng.standard_t(3, n)
    if kind.startswith("apart"):  # two genes (of two parts, of one, a linear-only one) never large together
        small = np.float32(float(kind.split()[1]))
        k = rng.random(n) < 0.5
        for a, b in ((3, 9), (4, 5), (2, ng - 1)):
            g[:, a] = np.where(k, g[:, a], g[:, a] * small)
            g[:, b] = np.where(k, g[:, b] * small, g[:, b])
    if kind == "rare":            # one row carries a column's largest value and the targets'
        g[1:, 7] *= np.float32(1e-7)
        y[0] = 1e9
        g[0, 11] = np.float32(1e-8)
    if kind == "disjoint":        # genes that are never nonzero together
        k = rng.random(n) < 0.5
        g[:, 3] = np.where(k, g[:, 3], 0)
        g[:, 9] = np.where(k, 0, g[:, 9])
    if kind == "zero":
        g[:, 3] = 0
        y = np.zeros(n)
    if kind.endswith("4 decimals"):
        g = np.round(g, 4)
    return np.ascontiguousarray(g, np.float32), y


@pytest.mark.parametrize("ng", [16, 22, 29])
@pytest.mark.parametrize("n", [1, 33, 1500])
@pytest.mark.parametrize("kind", ["uniform", "uniform 4 decimals", "pop 4 decimals", "apart 1e-2", "apart 1e-4",
                                  "apart 1e-6", "apart 1e-9", "apart 1e-30", "rare", "disjoint", "zero"])
def test_normal_equations_entry_by_entry(kind, n, ng):
    """Each entry against its own magnitude sum_r |phi_i phi_j|, whatever the
    columns' largest values. FP64 sums are within 2^-53 of it per rounding: the
    rows of a part (32 at a time dealt to 152), 19 parts per thread, 8 threads, the
    product. Fixed-point sums are taken only where the magnitude is at least
    sqrt(n) / 8 of the scale, of which a row is within 8.1 x 2^-56: 8.1 sqrt(n) x
    2^-53 of the magnitude, and two roundings at the end."""
    _entry_by_entry(kind, n, ng)


@pytest.mark.parametrize("ng", [16, 29])
@pytest.mark.parametrize("n", [31, 32, 127, 128, 129, 255, 257, 6400, 6401, 9001])
def test_fixed_point_entries_at_stage_edges(n, ng):
    """The same where the rows end around a stage, a drain and a chunk."""
    _entry_by_entry("uniform", n, ng)


def _entry_by_entry(kind, n, ng):
    g, y = _table(kind, n, ng, np.random.default_rng(n + ng))
    gram, rhs = _run(g, y, 1 + ng + 136)
    phi = _phi(g.astype(np.longdouble), ng)
    yl = y.astype(np.longdouble)
    mag, mrhs = np.abs(phi).T @ np.abs(phi), np.abs(phi).T @ np.abs(yl)
    want, wrhs = (mag, phi.T @ yl) if g.min() >= 0 else (phi.T @ phi, phi.T @ yl)
    rows = 32 * -(-(-(-n // 32)) // 152)
    tol = (max(8.1 * np.sqrt(n), rows + 28) + 2) * 2.0 ** -53
    assert np.all(np.abs(gram - want) <= tol * mag)
    assert np.all(np.abs(rhs - wrhs) <= tol * mrhs)
