"""The triangular solves (panel_trsv.hpp:310-758) at the sizes where their 128-row blocks can go wrong."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factors(rng, n):
    """Column-major LU of a matrix with a dominant diagonal: multipliers near 2/n, U's diagonal near n/4."""
    m = rng.uniform(-0.5, 0.5, (n, n)).astype(np.float32)
    m[np.tril_indices(n, -1)] *= np.float32(4.0 / n)
    m[np.arange(n), np.arange(n)] = np.float32(0.25 * n + 1.0)
    return m


def _solve(m, x, lower):
    """Substitution in FP64 (the FP32 entries convert exactly)."""
    a = m.astype(np.float64)
    y = x.copy()
    n = len(x)
    for i in range(n) if lower else reversed(range(n)):
        y[i] -= a[i, :i] @ y[:i] if lower else a[i, i + 1:] @ y[i + 1:]
        if not lower:
            y[i] /= a[i, i]
    return y


# one block and its remainders, whole and ragged block rows, an odd leading dimension and an unaligned base (the
# 4-byte copies), more block rows than the GPU has SMs
@pytest.mark.parametrize("n,lda,off", [(1, 1, 0), (31, 32, 0), (127, 129, 0), (128, 128, 0), (129, 132, 0), (257, 257, 1),
                                       (1000, 1004, 0), (2500, 2501, 3), (19200, 19264, 0)])
def test_trsv_leaf_edges(hplai, torch_cuda, n, lda, off):
    """Dominant factors as the LU leaves them: their blocks are well conditioned, so the forward error is a few eps."""
    torch = torch_cuda
    rng = np.random.default_rng(n)
    if n <= 2500:
        m = _factors(rng, n)
        buf = np.zeros(n * lda + off + 4, dtype=np.float32)
        buf[off:off + n * lda].reshape(n, lda)[:, :n] = m.T   # column j at j * lda
        a = torch.from_numpy(buf).cuda()
    else:
        g = torch.Generator(device="cuda").manual_seed(n)
        a = torch.zeros((n, lda), device="cuda")
        a[:, :n] = torch.rand((n, n), generator=g, device="cuda") - 0.5
        i = torch.arange(n, device="cuda")
        for c in range(0, n, 2048):
            a[c:c + 2048, :n].mul_(torch.where(i[None, :] > i[c:c + 2048, None], 4.0 / n, 1.0))
        a[i, i] = 0.25 * n
    x = rng.uniform(-1, 1, n)
    ws = hplai.trsv_workspace(n)
    w = torch.zeros(ws, dtype=torch.uint8, device="cuda")
    ptr = a.data_ptr() + 4 * off
    for lower in (True, False, True):   # one workspace for solve after solve
        xd = torch.from_numpy(x).cuda()
        fn = hplai.trsv_lower if lower else hplai.trsv_upper
        hplai.check(fn(n, ptr, lda, xd.data_ptr(), w.data_ptr(), ws, None))
        got = xd.cpu().numpy()
        if n <= 2500:
            ref = _solve(m, x, lower)
        else:
            d = a[:, :n].T.double()
            ref = torch.linalg.solve_triangular(d, torch.from_numpy(x).cuda()[:, None], upper=not lower,
                                                unitriangular=lower)[:, 0].cpu().numpy()
            del d
        assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max(), lower


def _leaf(hplai, torch, m, x, lower):
    n = len(x)
    a = torch.from_numpy(np.ascontiguousarray(m.T)).cuda()
    xd = torch.from_numpy(x).cuda()
    w = torch.zeros(hplai.trsv_workspace(n), dtype=torch.uint8, device="cuda")
    fn = hplai.trsv_lower if lower else hplai.trsv_upper
    hplai.check(fn(n, a.data_ptr(), n, xd.data_ptr(), w.data_ptr(), w.numel(), None))
    return xd.cpu().numpy()


@pytest.mark.parametrize("n", [20, 33, 65, 97, 128, 130, 300, 513])
@pytest.mark.parametrize("lower", [True, False])
def test_trsv_leaf_any_triangle(hplai, torch_cuda, n, lower):
    """Triangles from dominant to condition numbers of 1e9 a block, a solution that does not grow: substitution is
    backward stable for each, row by row |T x - b| <= g (|T| |x| + |b|) with g = (n + 4) eps of FP64 for its n products,
    sums and one quotient."""
    rng = np.random.default_rng(n)
    for size in (0.1, 0.5, 1.0):
        m = rng.uniform(-size, size, (n, n)).astype(np.float32)
        m[np.arange(n), np.arange(n)] = np.where(rng.random(n) < 0.5, -1, 1) * rng.uniform(0.5, 1, n)
        t = m.astype(np.longdouble)
        t = np.tril(t, -1) + np.eye(n) if lower else np.triu(t)
        b = (t @ np.ones(n)).astype(np.float64)
        x = _leaf(hplai, torch_cuda, m, b, lower)
        r = np.abs(t @ x.astype(np.longdouble) - b)
        assert np.all(r <= (n + 4) * 2.0 ** -53 * (np.abs(t) @ np.abs(x) + np.abs(b))), size


def test_trsv_leaf_quotients(hplai, torch_cuda):
    """A diagonal U: the quotients of FP64, to one unit in the last place, over zeros, the smallest and the largest."""
    rng = np.random.default_rng(3)
    n = 200
    d = (rng.uniform(1, 2, n) * 2.0 ** rng.integers(-20, 20, n)).astype(np.float32)
    b = rng.uniform(-1, 1, n)
    d[5], d[40], d[70], d[71], d[150] = 2.0 ** -140, 2.0 ** 127, np.inf, 1e-45, 3e-39
    b[20], b[21], b[60], b[90], b[130], b[150] = 0.0, -0.0, 1e-300, 5e-324, 1e300, 1e250
    x = _leaf(hplai, torch_cuda, np.diag(d), b, False)
    ref = b / d.astype(np.float64)
    assert np.all(np.abs(x - ref) <= 2.0 ** -52 * np.abs(ref))


def test_trsv_leaf_inverse_quotients(hplai, torch_cuda):
    """An ordinary diagonal U takes its inverse: the corrected reciprocal (1/2 ulp but for a few parts in 2^50) and the
    product's rounding, 2^-53 of the quotient each."""
    rng = np.random.default_rng(4)
    n = 1000
    d = (rng.uniform(1, 2, n) * 2.0 ** rng.integers(-55, 55, n) * rng.choice((-1, 1), n)).astype(np.float32)
    b = rng.uniform(-1, 1, n)
    ref = b / d.astype(np.float64)
    x = _leaf(hplai, torch_cuda, np.diag(d), b, False)
    assert np.all(np.abs(x - ref) <= 2.0 ** -52 * (1 + 2.0 ** -20) * np.abs(ref))


@pytest.mark.parametrize("lower", [True, False])
def test_trsv_leaf_infinite_entry(hplai, torch_cuda, lower):
    """The rows solved before the one with an infinite right-hand side do not see it."""
    rng = np.random.default_rng(9)
    m, b = _factors(rng, 200), rng.uniform(-1, 1, 200)
    ref = _solve(m, b, lower)
    b[70] = np.inf
    x = _leaf(hplai, torch_cuda, m, b, lower)
    clean = slice(0, 70) if lower else slice(71, 200)
    assert np.abs(x[clean] - ref[clean]).max() <= 1e-13 * np.abs(ref).max()
    assert not np.any(np.isfinite(x[71:] if lower else x[:70])) and not np.isfinite(x[70])


def test_trsv_leaf_workspace_limits(hplai, torch_cuda):
    """A workspace shared by two orders; one byte too few is refused; an address off the 16-byte boundary works."""
    torch = torch_cuda
    rng = np.random.default_rng(5)
    ws = hplai.trsv_workspace(600)
    w = torch.zeros(ws + 16, dtype=torch.uint8, device="cuda")
    for n in (600, 130, 600, 7):
        m = _factors(rng, n)
        a = torch.from_numpy(np.ascontiguousarray(m.T)).cuda()
        x = rng.uniform(-1, 1, n)
        xd = torch.from_numpy(x).cuda()
        hplai.check(hplai.trsv_lower(n, a.data_ptr(), n, xd.data_ptr(), w.data_ptr() + 4, ws, None))
        ref = _solve(m, x, True)
        assert np.abs(xd.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
    a = torch.zeros((600, 600), device="cuda")
    xd = torch.zeros(600, dtype=torch.float64, device="cuda")
    assert hplai.trsv_lower(600, a.data_ptr(), 600, xd.data_ptr(), w.data_ptr(), ws - 1, None) == hplai.HPLAI_EINVAL


@pytest.mark.parametrize("n,b", [(100, 100), (700, 100), (1280, 128), (1290, 30)])
def test_transposed_solve_ragged(hplai, oracle, torch_cuda, n, b):
    """The transposed triangles (and their register-held inverses) through the adjoint solve: x and lambda against
    the dense FP64 solves."""
    g = np.random.default_rng(n).uniform(-1, 1, n)
    with hplai.Solver(n, b) as s:
        s.generate(42)
        s.factor()
        lam, r = s.solve_transpose(g)
        x, q = s.solve_rhs(g)
    assert r.status == hplai.HPLAI_OK and q.status == hplai.HPLAI_OK
    a = oracle.dense_matrix_f64(n)
    assert np.abs(lam - np.linalg.solve(a.T, g)).max() <= 1e-12 * np.abs(lam).max()
    assert np.abs(x - np.linalg.solve(a, g)).max() <= 1e-12 * np.abs(x).max()
