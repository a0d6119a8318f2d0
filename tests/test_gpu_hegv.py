"""chfsi_hegv_dev at the edges of its kernels: tiles of 32 in the Cholesky factor,
leaves of at most 24 rows, the cluster (n <= 256) and grid forms of the
tridiagonal reduction, and spectra that deflate (equal and clustered
eigenvalues, diagonal input, decoupled blocks).

Bounds: each stage is backward stable, so residual and loss of orthogonality are
a modest multiple of n 2^-53 (factor 40 taken), times the condition number of S
where S is not the identity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EPS = 2.0 ** -53


def _gauss(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn(n, n, 2, generator=g, device="cuda",
                                             dtype=torch.float64))


def _unitary(n, seed):
    return torch.linalg.qr(_gauss(n, seed))[0]


def _solve(chfsi, h, s):
    n = h.shape[0]
    h, s = h.contiguous(), s.contiguous()
    v = torch.full((n, n), float("nan"), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    w = chfsi.hegv_dev(h.data_ptr(), s.data_ptr(), n, v.data_ptr())
    return torch.from_numpy(w).cuda(), v


def _check(h, s, w, v, kappa):
    n = h.shape[0]
    scale = float(torch.linalg.matrix_norm(h, 2)) + 1e-300
    tol = 40 * n * EPS * kappa
    assert bool((w[1:] >= w[:-1]).all())
    assert float((h @ v - (s @ v) * w).abs().max()) <= tol * scale
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    assert float((v.mH @ s @ v - eye).abs().max()) <= tol
    low = torch.linalg.cholesky(s)
    b = torch.linalg.solve_triangular(low, h, upper=False)
    b = torch.linalg.solve_triangular(low, b.mH, upper=False).mH
    ref = torch.linalg.eigvalsh((b + b.mH) / 2)
    assert float((w - ref).abs().max()) <= tol * scale


@pytest.mark.parametrize("n", [1, 2, 3, 5, 20, 24, 25, 31, 32, 33, 48, 49, 63, 64, 65, 97, 160, 161,
                               255, 256, 257, 400, 576, 600])
def test_random_pencil(chfsi, n):
    h = _gauss(n, n)
    h = (h + h.mH) / 2
    x = torch.eye(n, dtype=torch.complex128, device="cuda") + 0.3 * _gauss(n, n + 1) / n ** 0.5
    s = x.mH @ x
    s = (s + s.mH) / 2
    w, v = _solve(chfsi, h, s)
    _check(h, s, w, v, float(torch.linalg.cond(s)))


@pytest.mark.parametrize("n", [24, 60, 160, 300])
@pytest.mark.parametrize("kind", ["equal", "clusters", "diagonal", "blocks", "zero", "graded", "rank1"])
def test_spectra_that_deflate(chfsi, n, kind):
    e = torch.linspace(-1.0, 1.0, n, device="cuda", dtype=torch.float64)
    if kind == "equal":
        e = torch.full_like(e, 0.7)
    elif kind == "clusters":
        e = torch.round(2 * e) + 1e-14 * torch.arange(n, device="cuda", dtype=torch.float64)
    elif kind == "graded":
        e = 2.0 ** -torch.arange(n, device="cuda", dtype=torch.float64).clamp(max=60)
    elif kind == "rank1":
        e = torch.zeros_like(e)
        e[-1] = 3.0
    elif kind == "zero":
        e = torch.zeros_like(e)
    q = _unitary(n, 7)
    if kind == "diagonal":
        h = torch.diag(e.flip(0)).to(torch.complex128)
    elif kind == "blocks":
        h = torch.zeros(n, n, dtype=torch.complex128, device="cuda")
        for i in range(0, n, 12):
            b = _gauss(min(12, n - i), 3)  # the same block again and again
            h[i:i + 12, i:i + 12] = (b + b.mH) / 2
    else:
        h = q @ (e[:, None] * q.mH)
        h = (h + h.mH) / 2
    s = torch.eye(n, dtype=torch.complex128, device="cuda")
    w, v = _solve(chfsi, h, s)
    _check(h, s, w, v, 1.0)


@pytest.mark.parametrize("n", [33, 160, 300])
def test_ill_conditioned_filtered_block(chfsi, n):
    """Bands amplified over five decades: the pivots stay positive."""
    x = (torch.eye(n, dtype=torch.complex128, device="cuda") + 0.05 * _gauss(n, 4) / n ** 0.5)
    x = x * torch.logspace(0, -5, n, device="cuda", dtype=torch.float64)[None, :]
    e = torch.linspace(-0.4, 0.9, n, device="cuda", dtype=torch.float64)
    h, s = x.mH @ (e[:, None] * x), x.mH @ x
    w, _ = _solve(chfsi, (h + h.mH) / 2, (s + s.mH) / 2)
    # column scaling leaves the Ritz values alone: only cond(I + 0.05 G) enters
    assert float((w - e).abs().max()) <= 40 * n * EPS * 2.0


@pytest.mark.parametrize("n", [20, 64, 300])
def test_errors(chfsi, n):
    h = _gauss(n, 1)
    h = (h + h.mH) / 2
    s = torch.eye(n, dtype=torch.complex128, device="cuda")
    bad = s.clone()
    bad[n - 1, n - 1] = -1.0
    with pytest.raises(chfsi.RayleighRitzFailed, match="positive definite"):
        _solve(chfsi, h, bad)
    h[2, 3] = float("nan")
    h[3, 2] = float("nan")
    with pytest.raises(chfsi.RayleighRitzFailed, match="did not converge"):
        _solve(chfsi, h, s)
    h = _gauss(n, 2)
    h = (h + h.mH) / 2
    w, v = _solve(chfsi, h, s)
    _check(h, s, w, v, 1.0)


@pytest.mark.parametrize("n", [1, 2, 24, 25, 160, 300])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_non_finite_h_is_reported(chfsi, n, value):
    """Whatever the solver makes of it, an eigenvalue that is not a number does not
    come back as a success; n = 1 has no iteration that could notice."""
    s = torch.eye(n, dtype=torch.complex128, device="cuda")
    h = _gauss(n, 5)
    h = (h + h.mH) / 2
    h[n // 2, n // 2] = value
    with pytest.raises(chfsi.RayleighRitzFailed, match="did not converge"):
        _solve(chfsi, h, s)


@pytest.mark.parametrize("n", [2, 5, 20, 60, 160, 300])
@pytest.mark.parametrize("exponent", [-480, -300, -200, 200, 300, 480])
def test_scaled_matrix(chfsi, n, exponent):
    """A power of two on H goes through to the eigenvalues, whatever squares and
    cubes of its entries do to the range of the exponents."""
    h = _gauss(n, n + 3)
    h = (h + h.mH) / 2
    s = torch.eye(n, dtype=torch.complex128, device="cuda")
    w0, v0 = _solve(chfsi, h, s)
    _check(h, s, w0, v0, 1.0)
    w, v = _solve(chfsi, h * 2.0 ** exponent, s)
    assert float((w * 2.0 ** -exponent - w0).abs().max()) <= 40 * n * EPS * float(w0.abs().max())
    _check(h, s, w * 2.0 ** -exponent, v, 1.0)


@pytest.mark.parametrize("n", [20, 60, 160, 300])
@pytest.mark.parametrize("size", [1e-60, 1e-80, 1e-100, 1e-130])
def test_blocks_with_a_negligible_coupling(chfsi, n, size):
    h = size * _gauss(n, 9)
    for i in range(0, n, 7):
        h[i:i + 7, i:i + 7] = _gauss(min(7, n - i), i + 1)
    h = (h + h.mH) / 2
    s = torch.eye(n, dtype=torch.complex128, device="cuda")
    w, v = _solve(chfsi, h, s)
    _check(h, s, w, v, 1.0)


@pytest.mark.parametrize("n", [768, 769, 1025, 1163, 1164])
def test_largest_sizes(chfsi, n):
    """Past 768 rows the back transformation holds 40 entries per lane, past 1,024
    the reduction a fifth entry per thread and the deflation over 48 KB; 1,163 is the
    last size whose rows fit the grid's shared memory, 1,164 goes to the Jacobi."""
    h = _gauss(n, n)
    h = (h + h.mH) / 2
    s = torch.eye(n, dtype=torch.complex128, device="cuda")
    w, v = _solve(chfsi, h, s)
    _check(h, s, w, v, 1.0)
