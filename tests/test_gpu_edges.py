"""The tiled kernels at the edges of their tiles, splits and dispatch rules, against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _put(torch, m, lda, off):
    """Column-major m at element `off` of a device buffer with leading dimension lda."""
    r, c = m.shape
    buf = np.zeros(c * lda + off + 4, dtype=m.dtype)
    buf[off:off + c * lda].reshape(c, lda)[:, :r] = m.T
    t = torch.from_numpy(buf).cuda()
    return t, t.data_ptr() + off * m.dtype.itemsize


def _take(t, r, c, lda, off):
    return t.cpu().numpy()[off:off + c * lda].reshape(c, lda)[:, :r].T


def _dominant(rng, n):
    m = rng.uniform(-0.5, 0.5, (n, n)).astype(np.float32)
    m[np.arange(n), np.arange(n)] = np.abs(m).sum(1) + 1
    return np.asfortranarray(m)


def _same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


# one to four tiles a side and remainders, the widest block, odd leading dimensions and unaligned bases (4-byte copies)
@pytest.mark.parametrize("b,lda,off", [(1, 1, 0), (31, 32, 0), (33, 36, 0), (64, 64, 0), (65, 65, 0), (97, 100, 1),
                                       (130, 131, 0), (160, 160, 2), (1023, 1024, 0), (1024, 1028, 0)])
def test_getrf_tile_edges(hplai, oracle, torch_cuda, b, lda, off):
    m = _dominant(np.random.default_rng(b), b)
    t, p = _put(torch_cuda, m, lda, off)
    hplai.check(hplai.getrf_nopiv(b, p, lda, None))
    assert _same_bits(_take(t, b, b, lda, off), oracle.getrf_nopiv(m))


@pytest.mark.parametrize("n,b,side", [(3072, 1024, 2), (3072, 1024, 7), (3072, 1024, 16), (3072, 1024, 12), (2700, 900, 9), (2048, 512, 4),
                                      (1280, 320, 3)])
def test_getrf_on_few_sms(hplai, torch_cuda, n, b, side):
    """More tiles than a team has places for in shared memory, odd numbers of teams: the factors of the whole GPU."""
    def lu(flags):
        with hplai.Solver(n, b, flags=flags) as s:
            if flags:
                s.set_schedule(flags, side)
            s.generate(42)
            s.factor()
            return s.lu()
    assert _same_bits(lu(0), lu(hplai.FLAG_LOOKAHEAD))


@pytest.mark.parametrize("scale", [2.0 ** -127, 2.0 ** -140, 2.0 ** 120])
def test_getrf_pivots_without_normal_reciprocals(hplai, oracle, torch_cuda, scale):
    """Subnormal pivots, and pivots whose reciprocals are subnormal, take the reciprocal that keeps subnormals."""
    m = np.asfortranarray((_dominant(np.random.default_rng(7), 100) * np.float32(scale)).astype(np.float32))
    t, p = _put(torch_cuda, m, 100, 0)
    hplai.check(hplai.getrf_nopiv(100, p, 100, None))
    got, ref = _take(t, 100, 100, 100, 0), oracle.getrf_nopiv(m)
    nan = np.isnan(ref)
    assert np.array_equal(nan, np.isnan(got)) and _same_bits(np.where(nan, 0, got), np.where(nan, 0, ref))


# rows around a CTA's 32 or 64 and the rule's 4736, widths around the 16-column steps and 128-column blocks
@pytest.mark.parametrize("m,b,off", [(1, 1, 0), (31, 15, 0), (33, 16, 1), (65, 17, 0), (100, 127, 0), (64, 128, 0),
                                     (70, 129, 0), (200, 260, 3), (40, 1000, 0), (4736, 48, 0), (4737, 50, 0)])
def test_panel_solve_edges(hplai, oracle, torch_cuda, m, b, off):
    torch = torch_cuda
    rng = np.random.default_rng(m + b)
    lu = _dominant(rng, b)
    lu[np.tril_indices(b, -1)] *= np.float32(4.0 / max(b, 4))
    d, dp = _put(torch, lu, b, off)
    ldh = (b + 7) // 8 * 8
    x = np.asfortranarray(rng.uniform(-0.5, 0.5, (m, b)).astype(np.float32))
    t, p = _put(torch, x, m, off)
    h = torch.zeros((m, ldh), dtype=torch.float16, device="cuda")
    hplai.check(hplai.trsm_right_upper(m, b, dp, b, p, m, h.data_ptr(), ldh, 2.0, None))
    ref = oracle.trsm_right_upper(np.triu(lu), x)
    assert _same_bits(_take(t, m, b, m, off), ref)
    assert np.array_equal(h.cpu().numpy()[:, :b], (np.float32(2.0) * ref).astype(np.float16))
    y = np.asfortranarray(rng.uniform(-0.5, 0.5, (b, m)).astype(np.float32))
    t, p = _put(torch, y, b, off)
    hplai.check(hplai.trsm_left_lower(b, m, dp, b, p, b, h.data_ptr(), ldh, 1.0, None))
    ref = oracle.trsm_left_lower_unit(np.tril(lu, -1) + np.eye(b, dtype=np.float32), y)
    assert _same_bits(_take(t, b, m, b, off), ref)
    assert np.array_equal(h.cpu().numpy()[:, :b], ref.T.astype(np.float16))


# around the rules' 32 and 64 columns and their 4736, 9472 and 16000 rows, blocks of 64 columns and remainders
@pytest.mark.parametrize("m,b,off", [(33, 32, 0), (16001, 31, 0), (16001, 32, 0), (16000, 20, 1), (65, 33, 0), (40, 64, 0),
                                     (4737, 64, 0), (9473, 65, 0), (9473, 128, 0), (9472, 129, 0), (9473, 200, 3),
                                     (9500, 260, 0)])
def test_panel_solve_widths(hplai, oracle, torch_cuda, m, b, off):
    test_panel_solve_edges(hplai, oracle, torch_cuda, m, b, off)


@pytest.mark.parametrize("n,b,flags", [(1200, 60, 0), (770, 70, 0), (1000, 125, 0), (1280, 128, 0), (2048, 512, 2),
                                       (1200, 50, 2)])
def test_small_panels_are_the_substitution_panels(hplai, torch_cuda, n, b, flags):
    """Below the size rule the default panels are the bit-exact substitution (HPLAI_FLAG_SIMT_PANELS), both panels in
    one launch: the same factors bit for bit, on one stream and with look-ahead."""
    def lu(f):
        with hplai.Solver(n, b, flags=f) as s:
            s.generate(42)
            s.factor()
            return s.lu()
    assert _same_bits(lu(flags), lu(flags | hplai.FLAG_SIMT_PANELS))


@pytest.mark.parametrize("n,b", [(9248, 136), (5520, 240), (5200, 260), (3840, 384), (2560, 640), (2700, 900)])
def test_inverse_panels_at_block_edges(hplai, torch_cuda, n, b):
    """Panels above the size rule, b past one, two, three and five 128-blocks of the triangular inverses: against the
    substitution, within the products' 2^-18 and the substitution's b eps, both of |X| |T| |T^-1|."""
    def first(f):
        with hplai.Solver(n, b, flags=f) as s:
            s.generate(42)
            s.factor_steps(1)
            lu = s.lu()
        return lu[:b, :b].astype(np.float64), lu[-400:, :b].astype(np.float64), lu[:b, -400:].astype(np.float64)
    d, lcol, urow = first(0)
    d2, lref, uref = first(hplai.FLAG_SIMT_PANELS)
    assert np.array_equal(d, d2)
    u, l = np.triu(d), np.tril(d, -1) + np.eye(b)
    eps = 2.0 ** -18 + b * 2.0 ** -23
    assert np.all(np.abs(lcol - lref) <= eps * (np.abs(lref) @ np.abs(u) @ np.abs(np.linalg.inv(u))))
    assert np.all(np.abs(urow - uref) <= eps * (np.abs(np.linalg.inv(l)) @ np.abs(l) @ np.abs(uref)))


@pytest.mark.parametrize("n,b", [(1539, 513), (1280, 640), (2048, 1024)])
def test_inverse_panels_of_wide_blocks(hplai, torch_cuda, n, b):
    """Past b = 512 the last panels, however small, are formed by the inverses as well."""
    test_inverse_panels_at_block_edges(hplai, torch_cuda, n, b)


def test_inverse_panels_of_extreme_diagonals(hplai, torch_cuda):
    """The panels by inverses (the precision form's TF32 path) under a diagonal block with an infinite pivot, one whose
    reciprocal is subnormal and, last, one whose reciprocal overflows: as in the substitution, x / inf is 0 and every other
    column is finite, x / d to TF32's 2^-10."""
    n, b = 90, 30
    rng = np.random.default_rng(11)
    a = np.asfortranarray(rng.uniform(0.25, 0.5, (n, n)).astype(np.float32))
    d = rng.uniform(1, 2, b).astype(np.float32)
    d[3], d[7], d[b - 1] = 2.0 ** 127, np.inf, 2.0 ** -140
    a[:b, :b] = np.diag(d)
    a[b:, b:] += 100 * np.eye(n - b, dtype=np.float32)
    with hplai.Solver(n, b, precision=hplai.F32_F8) as s:
        s.upload(a, np.ones(n), np.full(n, 100.0))
        s.factor_steps(1)
        lu = s.lu()
    got, ref = lu[b:, :b - 1].astype(np.float64), a[b:, :b - 1] / d[:b - 1].astype(np.float64)
    assert np.all(got[:, 7] == 0)
    assert np.all(np.abs(got - ref) <= 2.0 ** -9 * np.abs(ref) + 2.0 ** -126)
    assert np.all(np.abs(lu[:b, b:] - a[:b, b:]) <= 2.0 ** -9 * a[:b, b:])


@pytest.mark.parametrize("n,i0,j0,nr,nc,lda,off", [(1000, 3, 5, 1, 1, 1, 0), (1000, 0, 100, 127, 33, 127, 0),
                                                   (4000, 1, 7, 1023, 31, 1024, 0), (4000, 9, 0, 1025, 65, 1025, 0),
                                                   (4000, 0, 2000, 2050, 40, 2052, 1)])
def test_fill_edges(hplai, oracle, torch_cuda, n, i0, j0, nr, nc, lda, off):
    t, p = _put(torch_cuda, np.zeros((nr, nc), dtype=np.float32), lda, off)
    hplai.check(hplai.fill_panel(n, i0, j0, nr, nc, p, lda, 42, 0, None))
    assert _same_bits(_take(t, nr, nc, lda, off), oracle.fill_panel(n, i0, j0, nr, nc, calc_diag=False))


@pytest.mark.parametrize("n,i0,count", [(1, 0, 1), (5, 0, 5), (37, 3, 30), (1000, 31, 400), (1001, 970, 31)])
def test_diag_edges(hplai, oracle, torch_cuda, n, i0, count):
    torch = torch_cuda
    d = torch.empty(count, dtype=torch.float64, device="cuda")
    hplai.check(hplai.gen_diag(n, 42, i0, count, d.data_ptr(), None))
    assert np.array_equal(d.cpu().numpy(), np.array([oracle.calc_diag(i, n, 42) for i in range(i0, i0 + count)]))


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 300, 2047, 2049, 4100])
def test_gemv_edges(hplai, oracle, torch_cuda, n):
    """Rows around a warp's 64 and a CTA's, columns around a chunk's 2048 and its pieces: 1e-14 of ||A|| ||x||."""
    torch = torch_cuda
    rng = np.random.default_rng(n)
    a = oracle.dense_matrix_f64(n)
    x, y0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    xd, dd = torch.from_numpy(x).cuda(), torch.from_numpy(np.ascontiguousarray(np.diag(a))).cuda()
    ws = hplai.otf_gemv_workspace(n)
    w = torch.empty(ws, dtype=torch.uint8, device="cuda")
    for beta in (0.0, 1.0):
        yd = torch.from_numpy(y0).cuda()
        hplai.check(hplai.otf_gemv(n, -1.0, xd.data_ptr(), beta, yd.data_ptr(), 42, dd.data_ptr(), w.data_ptr(), ws, None))
        ref = beta * y0 - a @ x
        assert np.abs(yd.cpu().numpy() - ref).max() <= 1e-14 * (np.abs(a).sum(1).max() + 1)


# a row per thread past 2048 blocks of 256 rows x 2048 columns (transposed: 800): odd orders past the rules' lines
def test_gemv_of_large_orders(hplai, oracle, torch_cuda):
    torch = torch_cuda
    n = 33001
    rng = np.random.default_rng(n)
    x, y0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    dd = torch.empty(n, dtype=torch.float64, device="cuda")
    hplai.check(hplai.gen_diag(n, 42, 0, n, dd.data_ptr(), None))
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y0).cuda()
    ws = hplai.otf_gemv_workspace(n)
    w = torch.empty(ws, dtype=torch.uint8, device="cuda")
    hplai.check(hplai.otf_gemv(n, -1.0, xd.data_ptr(), 1.0, yd.data_ptr(), 42, dd.data_ptr(), w.data_ptr(), ws, None))
    got = yd.cpu().numpy()
    rows = np.array([0, 31, 32, 255, 256, 2047, 2048, 16384, 32767, 32768, 32999, 33000])
    ref = oracle.residual_rows(n, x, rows, rhs_v=y0)
    assert np.abs(got[rows] - ref).max() <= 1e-14 * 2 * float(dd.max())


def test_transposed_residual_of_large_orders(hplai, oracle, torch_cuda):
    """lambda of A^T lambda = g has the residual that the refinement reports for it, on sampled rows."""
    n, b = 20808, 72
    g = np.random.default_rng(n).uniform(-1, 1, n)
    with hplai.Solver(n, b) as s:
        s.generate(42)
        s.factor()
        lam, r = s.solve_transpose(g)
        d = s.diag()
    assert r.status == hplai.HPLAI_OK
    rows = np.array([0, 1, 31, 255, 256, 2048, 10007, 20479, 20480, 20735, 20807])
    res = oracle.residual_rows(n, lam, rows, trans=True, rhs_v=g)
    assert np.abs(res).max() <= r.residual + 1e-14 * 2 * d.max() * np.abs(lam).max()


@pytest.mark.parametrize("n", [[2], [127, 129, 128], [640, 100, 36], [1500, 1536]])
def test_batch_edges(hplai, oracle, torch_cuda, n):
    """Orders around the 128-wide steps, one to eight right-hand sides."""
    nrhs = [(3 * i + 8 - len(n)) % 8 + 1 for i in range(len(n))]
    with hplai.Batch(n, nrhs, list(range(5, 5 + len(n)))) as bt:
        assert bt.solve() == hplai.HPLAI_OK
        for s, m in enumerate(n):
            a = oracle.dense_matrix_f64(m, 5 + s)
            ref = np.linalg.solve(a, oracle.rhs_cols(m, 5 + s, 0, nrhs[s]))
            assert np.abs(bt.x(s) - ref).max() <= 1e-12 * np.abs(ref).max()
