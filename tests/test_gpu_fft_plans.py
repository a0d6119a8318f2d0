"""Local H|psi> and the density on every FFT plan with compile-time kernels and
on grids that take the generic ones, against torch FFTs in 64 bits: columns of
all lengths, plane-wave sets with holes and in any order, z axes on another plan
than x and y, one band and odd counts, occupations with zeros.

Bound: a 3D FFT of N^3 points errs by a few 2^-53 log2(N^3) of the 2-norm; there
and back 16 x 2^-53 x 21 = 4e-14 of each band's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 4e-14
# two-radix plans of the compile-time kernels, then grids without one
CUBES = [30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 27, 15, 20]
BOXES = [(40, 40, 36), (40, 36, 40), (64, 64, 50), (32, 32, 25), (72, 72, 54), (48, 48, 120)]


def _basis(n3, seed, holes):
    r = [max(2, int(n / 4.3)) for n in n3]
    h = [np.arange(-k, k + 1) for k in r]
    y, x, z = np.meshgrid(h[1], h[0], h[2], indexing="ij")
    s = (x / (r[0] + 0.5)) ** 2 + (y / (r[1] + 0.5)) ** 2 + (z / (r[2] + 0.5)) ** 2
    m = np.stack([x[s <= 1], y[s <= 1], z[s <= 1]], axis=1).astype(np.int32)
    rng = np.random.default_rng(seed)
    if holes:
        m = m[rng.random(len(m)) < 0.6]
    order = np.lexsort((m[:, 2], m[:, 0] % n3[0], m[:, 1] % n3[1]))
    m = np.ascontiguousarray(m[order])
    return m, rng.random(len(m))


def _grid(psi, m, n3):
    nx, ny, nz = n3
    at = torch.from_numpy((m[:, 0] % nx + nx * (m[:, 1] % ny + ny * (m[:, 2].astype(np.int64) % nz)))).cuda()
    g = torch.zeros(psi.shape[0], nx * ny * nz, dtype=torch.complex128, device="cuda")
    g[:, at] = psi
    return torch.fft.ifftn(g.view(-1, nz, ny, nx), dim=(1, 2, 3), norm="forward"), at


@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("n3", [(n, n, n) for n in CUBES] + BOXES)
def test_local_h(chfsi, n3, holes):
    m, kin = _basis(n3, 3, holes)
    nb = 5
    ctx = chfsi.Context(dims={"ngrid": n3, "n_pw": len(m), "n_bands": nb})
    ctx.set_basis(m, kin, 2.0)
    rng = np.random.default_rng(4)
    v = rng.standard_normal(n3[0] * n3[1] * n3[2])
    ctx.set_veff(v)
    psi = torch.from_numpy(rng.standard_normal((nb, len(m))) + 1j * rng.standard_normal((nb, len(m)))).cuda()
    grid, at = _grid(psi, m, n3)
    vr = torch.from_numpy(v).cuda().view(n3[2], n3[1], n3[0])
    ref = torch.fft.fftn(grid * vr, dim=(1, 2, 3), norm="forward").reshape(nb, -1)[:, at]
    ref = ref + psi * torch.from_numpy(kin).cuda()
    for bands in (nb, 1, 2):
        out = torch.full_like(psi, float("nan"))
        torch.cuda.synchronize()
        ctx.apply_h_local(psi.data_ptr(), out.data_ptr(), bands)
        err = torch.linalg.vector_norm(out[:bands] - ref[:bands], dim=1)
        scale = torch.linalg.vector_norm(ref[:bands], dim=1) + v.std() * torch.linalg.vector_norm(psi[:bands], dim=1)
        assert float((err / scale).max()) < TOL, (n3, bands)
        assert bool(torch.isnan(out[bands:].real).all())


@pytest.mark.parametrize("n", [40, 64, 72, 100, 30])
def test_local_h_many_bands(chfsi, n):
    """Blocks of the inverse z pass that take several bands in turn, of columns
    that fill the axis (more plane waves than a thread keeps places of)."""
    h = np.arange(-9, 10)
    x, y, z = np.meshgrid(h, h, np.arange(-((n - 1) // 2), (n - 1) // 2 + 1), indexing="ij")
    on = x ** 2 + y ** 2 <= 90
    m = np.stack([x[on], y[on], z[on]], axis=1).astype(np.int32)
    m = np.ascontiguousarray(m[np.lexsort((m[:, 2], m[:, 0] % n, m[:, 1] % n))])  # device order
    rng = np.random.default_rng(n)
    kin, v, nb = rng.random(len(m)), rng.standard_normal(n ** 3), 322
    ctx = chfsi.Context(dims={"ngrid": (n, n, n), "n_pw": len(m), "n_bands": nb})
    ctx.set_basis(m, kin, 2.0)
    ctx.set_veff(v)
    gen = torch.Generator("cuda").manual_seed(n)
    psi = torch.randn(nb, len(m), dtype=torch.complex128, device="cuda", generator=gen)
    out = torch.full_like(psi, float("nan"))
    torch.cuda.synchronize()
    ctx.apply_h_local(psi.data_ptr(), out.data_ptr(), nb)
    vr, kt = torch.from_numpy(v).cuda().view(n, n, n), torch.from_numpy(kin).cuda()
    for b in range(0, nb, 46):
        part = psi[b:b + 46]
        grid, at = _grid(part, m, (n, n, n))
        ref = torch.fft.fftn(grid * vr, dim=(1, 2, 3), norm="forward").reshape(len(part), -1)[:, at] + part * kt
        err = torch.linalg.vector_norm(out[b:b + 46] - ref, dim=1)
        scale = torch.linalg.vector_norm(ref, dim=1) + v.std() * torch.linalg.vector_norm(part, dim=1)
        assert float((err / scale).max()) < TOL
    one = torch.empty_like(psi[:1])
    torch.cuda.synchronize()
    for b in (0, 1, 2, nb - 1):
        ctx.apply_h_local(psi[b:b + 1].data_ptr(), one.data_ptr(), 1)
        torch.cuda.synchronize()
        assert bool((one[0] == out[b]).all())


def test_local_h_with_infinite_and_nan_bands(chfsi):
    """A band with an inf or NaN leaves the others alone."""
    n3 = (40, 40, 40)
    m, kin = _basis(n3, 5, False)
    ctx = chfsi.Context(dims={"ngrid": n3, "n_pw": len(m), "n_bands": 3})
    ctx.set_basis(m, kin, 2.0)
    ctx.set_veff(np.random.default_rng(6).standard_normal(40 ** 3))
    psi = torch.randn(3, len(m), dtype=torch.complex128, device="cuda")
    a, b = torch.empty_like(psi), torch.empty_like(psi)
    torch.cuda.synchronize()
    ctx.apply_h_local(psi.data_ptr(), a.data_ptr(), 3)
    psi[1, 7] = float("nan")
    torch.cuda.synchronize()
    ctx.apply_h_local(psi.data_ptr(), b.data_ptr(), 3)
    assert bool((a[[0, 2]] == b[[0, 2]]).all()) and bool(torch.isnan(b[1].real).all())


@pytest.mark.parametrize("n", [30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 27])
def test_density(chfsi, n):
    s = chfsi.SyntheticSystem(config_index=0, ecut=4.0, ngrid=[n] * 3, ngrid_density=[n] * 3, n_bands=23)
    ctx = chfsi.Context(s)
    occ = np.random.default_rng(n).random(23) * 2
    occ[[1, 4, 5]] = 0.0
    ctx.set_occupations(occ)
    psi = s.psi0()
    ctx.set_psi(psi)
    rho = ctx.construct_density()
    grid, _ = _grid(torch.from_numpy(psi).cuda(), s.miller(), (n, n, n))
    ref = (torch.from_numpy(occ).cuda()[:, None, None, None] * grid.abs() ** 2).sum(0) / s.omega
    ref = ref.reshape(-1).cpu().numpy()
    assert np.linalg.norm(rho - ref) < TOL * np.linalg.norm(ref)
    assert np.array_equal(rho, ctx.construct_density())
    ctx.set_occupations(np.zeros(23))
    assert not ctx.construct_density().any()


@pytest.mark.parametrize("at", [0, 31, 8192, 100003])
def test_spectral_bound_sees_every_potential_value(chfsi, at):
    """The filter's upper bound holds the potential's range, wherever its
    extremes lie."""
    n3 = (48, 48, 48)
    m, kin = _basis(n3, 1, False)
    ctx = chfsi.Context(dims={"ngrid": n3, "n_pw": len(m), "n_bands": 4})
    ctx.set_basis(m, kin, 2.0)
    v = np.zeros(48 ** 3)
    v[at], v[-1] = 3.0, -2.0
    ctx.set_veff(v)
    rng = np.random.default_rng(2)
    ctx.set_psi(rng.standard_normal((4, len(m))) + 1j * rng.standard_normal((4, len(m))))
    ctx.chebyshev_filter(1)
    assert abs(ctx.bounds()[0] - (2.0 + 5.0)) < 1e-13
