"""FP64 products on the INT8 tensor cores (chfsi_zgemm_cn, chfsi_zgemm_tn above
the sizes where that path is taken) at the edges of its tiles (128 rows, 64
columns, 32 of K), over row scales, with several K chunks and groups, and with
inf and NaN.

Bounds: digits keep 2^-62 of a row's largest part, so K terms leave at most
K 2^-60 max|a| max|b| (under 2^-53 |a||b| for the sizes here); every T1, T2, T3
and the sums over chunks are rounded a few times at most 2 |a||b|, |.| the
2-norms of the two vectors: 64 2^-52 |a||b| holds both, and the error of the
reference sums as well."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 64 * 2.0 ** -52


def _gauss(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn(*shape, 2, generator=g, device="cuda",
                                             dtype=torch.float64))


def _cn(chfsi, a, b):
    m, k = a.shape
    n = b.shape[0]
    c = torch.full((m, n), float("nan"), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    before = chfsi.launch_count()
    chfsi.zgemm_cn(a.data_ptr(), k, b.data_ptr(), k, m, n, k, c.data_ptr())
    return c, chfsi.launch_count() - before


def _row_norms(a):
    top = a.abs().amax(dim=1)  # squares of 1e200 overflow
    top = torch.where(top > 0, top, torch.ones_like(top))
    return top * torch.linalg.vector_norm(a / top[:, None], dim=1)


def _norms(a, b):
    return _row_norms(a)[:, None] * _row_norms(b)[None, :]


@pytest.mark.parametrize("m,n,k", [(256, 160, 37073), (257, 161, 16001), (255, 129, 24031),
                                   (128, 576, 23840), (1153, 576, 40000), (576, 576, 576),
                                   (20, 20, 2945)])
def test_projection(chfsi, m, n, k):
    a, b = _gauss((m, k), 1), _gauss((n, k), 2)
    # rows of very different size, plane waves that decay
    a *= torch.logspace(-12, 3, m, device="cuda", dtype=torch.float64)[:, None]
    b *= 1.0 / (1.0 + torch.arange(k, device="cuda", dtype=torch.float64) / 50.0)
    c, launches = _cn(chfsi, a, b)
    assert launches >= (2 if m == 20 else 4)  # slicing, slicing, products, sums
    assert float(((c - a.conj() @ b.T).abs() / _norms(a, b)).max()) < TOL


@pytest.mark.parametrize("m,n,k,alpha,beta", [(160, 37073, 160, 1.0, 0.0), (161, 8001, 512, 0.5, -2.0),
                                              (64, 37073, 256, 1.0, 1.0), (576, 2945, 576, 1.0, 0.0),
                                              (577, 4097, 33, 1.0, 0.0), (1728, 513, 1728, 1.0, 1.0),
                                              (576, 100000, 576, 1.0, 0.0), (20, 2945, 20, 1.0, 0.0)])
def test_expansion(chfsi, m, n, k, alpha, beta):
    w, x, o0 = _gauss((k, m), 3), _gauss((k, n), 4), _gauss((m, n), 5)
    x *= torch.logspace(-9, 2, n, device="cuda", dtype=torch.float64)[None, :]
    o = o0.clone()
    torch.cuda.synchronize()
    chfsi.zgemm_tn(w.data_ptr(), m, x.data_ptr(), n, o.data_ptr(), n, m, n, k, alpha, beta)
    ref = alpha * (w.T @ x) + beta * o0
    bound = abs(alpha) * _norms(w.T, x.T) + abs(beta) * o0.abs() / 16
    assert float(((o - ref).abs() / bound).max()) < TOL


def test_extreme_rows(chfsi):
    m, n, k = 256, 192, 20000
    a, b = _gauss((m, k), 6), _gauss((n, k), 7)
    a[3] *= 1e-200
    b[5] *= 1e200
    a[7] = 0.0
    b[9] = 0.0
    c, launches = _cn(chfsi, a, b)
    assert launches == 4
    norm = _norms(a, b)
    assert bool((c[7] == 0).all()) and bool((c[:, 9] == 0).all())
    norm[7], norm[:, 9] = 1.0, 1.0
    assert float(((c - a.conj() @ b.T).abs() / norm).max()) < TOL


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_non_finite_rows_stay_in_their_row(chfsi, value):
    m, n, k = 256, 160, 20000
    a, b = _gauss((m, k), 8), _gauss((n, k), 9)
    clean, launches = _cn(chfsi, a, b)
    assert launches == 4
    a[130, 19999] = value
    b[65, 0] = value
    c, _ = _cn(chfsi, a, b)
    hit = torch.zeros((m, n), dtype=torch.bool, device="cuda")
    hit[130], hit[:, 65] = True, True
    assert not bool(torch.isfinite(c[hit].real).any())
    assert bool((c[~hit] == clean[~hit]).all())


def test_same_inputs_same_bits(chfsi):
    a, b = _gauss((300, 30000), 10), _gauss((200, 30000), 11)
    c, _ = _cn(chfsi, a, b)
    d, _ = _cn(chfsi, a, b)
    assert bool((c == d).all())


def test_rows_at_both_ends_of_the_exponents(chfsi):
    """A row near 2^1000 times one near 2^-1000 is an ordinary number."""
    m, n, k = 256, 192, 20000
    a, b = _gauss((m, k), 12), _gauss((n, k), 13)
    ref, norm = a.conj() @ b.T, _norms(a, b)
    ea = torch.zeros(m, dtype=torch.int64, device="cuda")
    eb = torch.zeros(n, dtype=torch.int64, device="cuda")
    ea[1:4] = torch.tensor([990, -1000, 970])
    eb[1:4] = torch.tensor([-990, 1000, -1005])

    def scaled(x, e):
        two = torch.tensor(2.0, dtype=torch.float64, device="cuda")
        return x * two ** (e // 2) * two ** (e - e // 2)

    c, launches = _cn(chfsi, scaled(a, ea[:, None]), scaled(b, eb[None, :].T))
    assert launches == 4
    e = ea[:, None] + eb[None, :]
    ordinary = e.abs() <= 1000
    assert bool(ordinary[1, 1] and ordinary[2, 2] and ordinary[3, 3])
    err = (scaled(c, torch.where(ordinary, -e, 0)) - ref).abs() / norm
    assert float(err[ordinary].max()) < TOL


# ---- element by element: |error| <= c K 2^-53 sum |a||b|, the bound of FP64 sums.
# The digits alone are relative to the rows' largest parts (at most 2^-55 of their
# product per term, 2^-59 sqrt(K) of it over random digits); products whose terms
# are smaller than that go to the FP64 tensor path.  c = 8: the reference's sums,
# the three-multiplication form there (3) and its own.
def _spread(kind, rows, k, seed):
    a = _gauss((rows, k), seed)
    i = torch.arange(k, device="cuda", dtype=torch.float64)
    if kind == "pairs":  # one large element that meets a small one, one ordinary
        a[:] = 0
        a[:, 100] = 1.0 if seed % 2 else 2.0 ** -60
        a[:, 200] = 1.23 * 2.0 ** -40 if seed % 2 else 1.0
    elif kind == "underflow":  # 2^-63 against 1, where the row's largest meets zero
        a[:] = 0
        a[:, 100] = 1.0 if seed % 2 else 0.0
        a[:, 200] = 2.0 ** -63 if seed % 2 else 1.0
    elif kind == "dominant":  # one element of 1, the rest near 2^-20 with full digits
        a *= 2.0 ** -20
        a[:, 7 if seed % 2 else 9] = 1.0
    elif kind == "slope":  # 2^-30 from one end of the row to the other, in opposite directions
        a *= 2.0 ** (-30.0 * (i if seed % 2 else k - 1 - i) / k)
    elif kind == "shuffled slope":
        a *= 2.0 ** (-30.0 * ((i * (7919 if seed % 2 else 104729)) % k) / k)
    elif kind == "apart":  # no common support: exact zeros
        a *= (i < k // 2) if seed % 2 else (i >= k // 2)
    elif kind == "one row":  # a single element of the result that the digits do not hold
        a[3] = 0
        a[3, 100] = 1.0 if seed % 2 else 2.0 ** -50
        a[3, 200] = 2.0 ** -50 if seed % 2 else 1.0
    return a


KINDS = ["pairs", "underflow", "dominant", "slope", "shuffled slope", "apart", "one row", "plain"]


def _elementwise(c, ref, terms, k):
    assert bool(((c - ref).abs() <= 8 * k * 2.0 ** -53 * terms).all())


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,n,k", [(256, 160, 20000), (130, 65, 60000)])
def test_projection_element_by_element(chfsi, kind, m, n, k):
    a, b = _spread(kind, m, k, 1), _spread(kind, n, k, 2)
    c, launches = _cn(chfsi, a, b)
    _elementwise(c, a.conj() @ b.T, a.abs() @ b.abs().T, k)
    assert launches == (4 if kind == "plain" else launches)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,n,k,alpha,beta", [(160, 20000, 512, 1.0, 0.0), (160, 20000, 512, 0.5, -2.0),
                                              (576, 100000, 576, 1.0, 1.0)])
def test_expansion_element_by_element(chfsi, kind, m, n, k, alpha, beta):
    w, x = _spread(kind, m, k, 3).T.contiguous(), _spread(kind, n, k, 4).T.contiguous()
    o0 = _gauss((m, n), 5)
    o = o0.clone()
    torch.cuda.synchronize()
    chfsi.zgemm_tn(w.data_ptr(), m, x.data_ptr(), n, o.data_ptr(), n, m, n, k, alpha, beta)
    ref = alpha * (w.T @ x) + beta * o0
    _elementwise(o, ref, abs(alpha) * (w.abs().T @ x.abs()) + abs(beta) * o0.abs() * 4 / k, k)
