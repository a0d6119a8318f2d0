"""The FP32 filter on every FFT plan with compile-time FP32 kernels (two bands to
an element: odd counts leave the last one alone) and on grids that take the
generic ones, against the FP64 filter from the same bands.

Bound: FP32 rounding of one application, about 20 x 2^-24 of H's range, times the
spread of a degree-4 filter's gain over the block, under 1e3: angles between the
two filtered subspaces below 1e-3, so that cosines stay above 1 - 1e-6 and Ritz
values, second order in the angle, within 1e-6 of H's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GRIDS = [(n, n, n) for n in (40, 48, 64, 72, 108, 45, 60)] + [
    (40, 40, 144), (72, 72, 108), (108, 108, 40), (48, 64, 72)]


def _system(n3, seed):
    """Plane waves of a sphere inside the grid, kinetic energies up to 10."""
    r = min(n3) / 4.3
    k = np.arange(-int(r), int(r) + 1)
    y, x, z = np.meshgrid(k, k, k, indexing="ij")
    s = x * x + y * y + z * z
    on = s <= r * r
    m = np.stack([x[on], y[on], z[on]], axis=1).astype(np.int32)
    order = np.lexsort((m[:, 2], m[:, 0] % n3[0], m[:, 1] % n3[1]))
    kin = 10.0 * s[on][order] / (r * r)
    v = 0.3 * np.random.default_rng(seed).standard_normal(n3[::-1])
    return np.ascontiguousarray(m[order]), kin, v


@pytest.mark.parametrize("nb", [2, 5, 8])
@pytest.mark.parametrize("n3", GRIDS)
def test_filtered_subspace(chfsi, n3, nb):
    m, kin, v = _system(n3, 2)
    rng = np.random.default_rng(nb)
    psi = (rng.standard_normal((nb, len(m))) + 1j * rng.standard_normal((nb, len(m)))) / (1.0 + kin ** 2)

    def context(precision):
        ctx = chfsi.Context(dims={"ngrid": n3, "n_pw": len(m), "n_bands": nb}, precision=precision)
        ctx.set_basis(m, kin, np.sqrt(20.0))
        ctx.set_veff(v)
        return ctx

    ref, ctx = context(chfsi.PREC_FP64), context(chfsi.PREC_MIXED)
    ref.set_psi(psi)
    w0 = ref.diagonalize(6)
    ctx.set_psi(ref.get_psi())
    w = ref.diagonalize(4, w0)
    w32 = ctx.diagonalize(4, w0)
    a, b = torch.from_numpy(ref.get_psi()).cuda(), torch.from_numpy(ctx.get_psi()).cuda()
    cosines = torch.linalg.svdvals(a.conj() @ b.T)
    assert float(cosines.min()) > 1.0 - 1e-6
    assert float(cosines.min()) < 1.0 - 1e-15  # FP32 it was
    assert np.abs(w - w32).max() <= 1e-6 * (10.0 + np.ptp(v))
