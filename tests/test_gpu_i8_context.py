"""The INT8 products of a context (digits of the projectors, scratch and error
word beside its FP64 buffers) when something about them fails or changes: memory
that is not to be had, waits that run out, projectors set anew.  The FP64 tensor
path computes the same products, so each case is compared with a context that
nothing happened to.

Bound: H psi of unit-norm bands, two ways of summing the same FP64 products: K
terms each at most |beta||psi| in sum, 64 2^-52 of the largest |H psi| holds it
with room (the products themselves are compared in test_gpu_i8_gemm.py)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 64 * 2.0 ** -52


@pytest.fixture(scope="module")
def sys_kb(chfsi):
    # 64-atom supercell at a low cutoff: projections and expansions on INT8
    return chfsi.SyntheticSystem(config_index=0, n_rep=2, ngrid=[45] * 3, ngrid_density=[45] * 3,
                                 ecut=8.0, n_bands=160, n_shell=1, lmax=1,
                                 rc_proj=[1.2, 1.4, 0, 0], d_min=0.5, d_max=2.0)


@pytest.fixture(autouse=True)
def _clear(chfsi):
    yield
    chfsi.inject_fault(chfsi.INJECT_NONE)


def _psi(s, nb=None):
    g = torch.Generator(device="cuda").manual_seed(3)
    psi = torch.view_as_complex(torch.randn(nb or s.n_bands, s.n_pw, 2, generator=g, device="cuda",
                                            dtype=torch.float64))
    return psi / torch.linalg.vector_norm(psi, dim=1, keepdim=True)


def _apply_h(ctx, psi):
    out = torch.full_like(psi, float("nan"))
    torch.cuda.synchronize()
    ctx.apply_h(psi.data_ptr(), out.data_ptr(), len(psi))
    return out


def _context(chfsi, s, **kw):
    ctx = chfsi.Context(s, **kw)
    ctx.set_veff(ctx.get_vloc())
    return ctx


def _same(a, b):
    return float((a - b).abs().max()) <= TOL * float(b.abs().max())


def test_context_without_the_scratch(chfsi, sys_kb):
    """The scratch is the one allocation of a creation that may fail first: what was
    asked for still runs, and its status does not come from memory that the
    process gave back before (the error word is mapped host memory)."""
    rt = ctypes.CDLL("libcudart.so.12")
    dirty = []
    for _ in range(64):
        p = ctypes.c_void_p()
        assert rt.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(4), 2) == 0
        ctypes.cast(p, ctypes.POINTER(ctypes.c_int))[0] = 7
        dirty.append(p)
    for p in dirty:
        rt.cudaFreeHost(p)
    psi = _psi(sys_kb)
    ref = _apply_h(_context(chfsi, sys_kb), psi)
    dims = {"ngrid": list(sys_kb.ngrid), "n_pw": sys_kb.n_pw, "n_bands": sys_kb.n_bands,
            "n_proj": sys_kb.n_proj, "n_ions": sys_kb.n_ions}
    for nth in range(200):
        chfsi.inject_fault(chfsi.INJECT_ALLOC_FAIL, nth)
        try:
            chfsi.Context(dims=dims)
            break
        except chfsi.OutOfMemory:
            pass
    chfsi.inject_fault(chfsi.INJECT_ALLOC_FAIL, nth)
    ctx = chfsi.Context(sys_kb)
    chfsi.inject_fault(chfsi.INJECT_NONE)
    ctx.set_veff(ctx.get_vloc())
    out = _apply_h(ctx, psi)
    assert _same(out, ref)
    assert not bool((out == ref).all())  # the other path did compute it


def _operands(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b, o = [torch.view_as_complex(torch.randn(*shape, 2, generator=g, device="cuda", dtype=torch.float64))
               for shape in ((m, k), (n, k), (m, n))]
    torch.cuda.synchronize()
    return a, b, o


def test_products_report_a_wait_that_ran_out(chfsi):
    m, n, k = 256, 160, 20000
    a, b, c = _operands(m, n, k)
    args = (a.data_ptr(), k, b.data_ptr(), k, m, n, k, c.data_ptr())
    chfsi.zgemm_cn(*args)
    ref = c.clone()
    chfsi.inject_fault(chfsi.INJECT_I8_NO_LOADS, 0)
    with pytest.raises(chfsi.Timeout, match="timed out"):
        chfsi.zgemm_cn(*args)
    chfsi.zgemm_cn(*args)
    assert bool((c == ref).all())
    m, n, k = 160, 20000, 256
    w, x = _operands(k, 1, m)[0], _operands(k, 1, n)[0]
    o = torch.empty(m, n, dtype=torch.complex128, device="cuda")
    args = (w.data_ptr(), m, x.data_ptr(), n, o.data_ptr(), n, m, n, k)
    chfsi.zgemm_tn(*args)
    ref = o.clone()
    chfsi.inject_fault(chfsi.INJECT_I8_NO_LOADS, 0)
    with pytest.raises(chfsi.Timeout, match="timed out"):
        chfsi.zgemm_tn(*args)
    chfsi.zgemm_tn(*args)
    assert bool((o == ref).all())


CALLS = {
    "apply_h": lambda c, s: _apply_h(c, _psi(s)),
    "diagonalize": lambda c, s: c.diagonalize(2),
    "construct_density": lambda c, s: c.construct_density(),
    "band_cg": lambda c, s: c.band_cg(1),
    "scf": lambda c, s: c.run_scf(2, max_iter=1, first_passes=1, kT=0.01),
    "scf, two iterations with cg": lambda c, s: c.run_scf(1, max_iter=2, first_passes=1, kT=0.01, cg_steps=1),
}


@pytest.mark.parametrize("name", CALLS)
def test_every_call_reports_its_own_time_out(chfsi, name):
    """Each INT8 product of a call in turn runs into its time limit: that call
    fails, also where the product is its last, and the next one does not."""
    s = chfsi.SyntheticSystem(config_index=2, n_rep=1, ecut=8.0, ngrid=[0, 0, 0], n_bands=24)
    ctx = _context(chfsi, s)
    psi0, psi = s.psi0(), _psi(s)
    ref = _apply_h(ctx, psi)
    for launches in range(200):
        ctx.set_psi(psi0)
        chfsi.inject_fault(chfsi.INJECT_I8_NO_LOADS, launches)
        try:
            CALLS[name](ctx, s)
            failed = False
        except chfsi.Timeout:
            failed = True
        chfsi.inject_fault(chfsi.INJECT_NONE)
        ctx.set_veff(ctx.get_vloc())
        out = _apply_h(ctx, psi)  # raises what the call before it did not
        # (an ultrasoft SCF leaves the screened D behind: another H)
        assert name.startswith("scf") or bool((out == ref).all())
        if not failed:
            break
    assert launches >= (2 if name.startswith("scf") else 1)


def test_captured_pass_takes_new_projectors(chfsi):
    """A captured pass holds the addresses of the projectors' digits and of D: new
    values go to the same place, and a change of their layout is refused."""
    s = chfsi.SyntheticSystem(config_index=0, n_shell=1, lmax=1, rc_proj=[1.2, 0, 0, 0],
                              d_min=0.5, d_max=2.0)
    beta, dmat, off = 0.9 * s.beta(), 1.1 * s.dmat(), s.proj_offsets()

    def prepared():
        ctx = _context(chfsi, s, precision=chfsi.PREC_MIXED)
        ctx.set_tc_shapes(0, 0)
        return ctx, ctx.diagonalize(8, ctx.diagonalize(8))

    ref, w = prepared()
    ref.set_projectors(beta, off, dmat)
    ref = ref.diagonalize(8, w)
    ctx, _ = prepared()
    batch = chfsi.Batch([ctx])
    batch.capture(8)
    held = [torch.empty(1 << k, device="cuda") for k in range(10, 24)]  # takes what is given back
    ctx.set_projectors(beta, off, dmat)
    held += [torch.zeros(1 << k, device="cuda") for k in range(10, 24)]
    torch.cuda.synchronize()
    np.testing.assert_allclose(batch.run()[0], ref, atol=1e-12, rtol=0)
    assert abs(ref - w).max() > 1e-6
    # other blocks: D lies elsewhere
    split = np.arange(0, s.n_proj + 1, s.n_proj // s.n_ions, dtype=np.int32)
    merged = split.copy()
    merged[1] += 1
    sizes = np.diff(merged)
    ctx.set_projectors(beta, merged, np.concatenate([1e-3 * np.eye(k).ravel() for k in sizes]))
    with pytest.raises(chfsi.BadInput, match="capture again"):
        batch.run()
    batch.capture(8)
    batch.run()


def test_int8_memory_is_given_back_before_an_allocation_is_refused(chfsi, sys_kb):
    psi = _psi(sys_kb)
    plain = _context(chfsi, sys_kb)
    ref_f, ref_h = plain.forces(), _apply_h(plain, psi)
    ctx = _context(chfsi, sys_kb)
    free = torch.cuda.mem_get_info()[0]
    chfsi.inject_fault(chfsi.INJECT_ALLOC_FAIL, 0)
    f = ctx.forces()  # allocates at its first call
    chfsi.inject_fault(chfsi.INJECT_NONE)
    assert torch.cuda.mem_get_info()[0] > free
    assert np.abs(f - ref_f).max() <= TOL * sys_kb.n_pw * np.abs(ref_f).max()  # sums that cancel
    out = _apply_h(ctx, psi)
    assert _same(out, ref_h) and not bool((out == ref_h).all())
    ctx.set_projectors(sys_kb.beta(), sys_kb.proj_offsets(), sys_kb.dmat())
    assert bool((_apply_h(ctx, psi) == out).all())
    # nothing left to give: the failure is reported, and the context still works
    chfsi.inject_fault(chfsi.INJECT_ALLOC_FAIL, 0)
    with pytest.raises(chfsi.OutOfMemory):
        ctx.band_cg(1)
    chfsi.inject_fault(chfsi.INJECT_NONE)
    assert bool((_apply_h(ctx, psi) == out).all())


def test_memory_that_a_captured_pass_uses_is_kept(chfsi, sys_kb):
    ctx = _context(chfsi, sys_kb, precision=chfsi.PREC_MIXED)
    ctx.set_tc_shapes(0, 0)
    ctx.diagonalize(4, ctx.diagonalize(4))
    psi = ctx.get_psi()
    batch = chfsi.Batch([ctx])
    batch.capture(4)
    w = batch.run()[0]
    chfsi.inject_fault(chfsi.INJECT_ALLOC_FAIL, 0)
    with pytest.raises(chfsi.OutOfMemory):
        ctx.forces()
    chfsi.inject_fault(chfsi.INJECT_NONE)
    assert np.isfinite(batch.run()[0]).all()
    assert np.isfinite(w).all() and np.isfinite(psi).all()


def test_scratch_of_a_process_without_contexts(chfsi):
    m, n, k = 256, 160, 20000
    a, b, c = _operands(m, n, k)
    chfsi.zgemm_cn(a.data_ptr(), k, b.data_ptr(), k, m, n, k, c.data_ptr())  # loads the kernels
    chfsi.release_scratch()
    free = torch.cuda.mem_get_info()[0]
    chfsi.zgemm_cn(a.data_ptr(), k, b.data_ptr(), k, m, n, k, c.data_ptr())
    assert torch.cuda.mem_get_info()[0] < free
    chfsi.release_scratch()
    assert torch.cuda.mem_get_info()[0] == free


def test_products_in_groups_with_cut_projectors(chfsi):
    """A projection whose second operand and partial sums are past the 1 GiB of
    scratch runs in groups along the plane waves, against digits cut once for all
    of them."""
    n, radius, np_, nb = 108, 28.8, 256, 400
    r = np.arange(-28, 29)
    y, x, z = np.meshgrid(r, r, r, indexing="ij")
    on = x * x + y * y + z * z <= radius * radius
    m = np.stack([x[on], y[on], z[on]], axis=1).astype(np.int32)
    m = np.ascontiguousarray(m[np.lexsort((m[:, 2], m[:, 0] % n, m[:, 1] % n))])
    npw = len(m)
    assert 7 * 64 * npw * 24 > 2 ** 30  # the digits of the bands alone
    g = torch.Generator(device="cuda").manual_seed(1)
    beta, psi = [torch.view_as_complex(torch.randn(rows, npw, 2, generator=g, device="cuda",
                                                   dtype=torch.float64)) / npw ** 0.5 for rows in (np_, nb)]
    d = torch.randn(np_, generator=g, device="cuda", dtype=torch.float64)
    ctx = chfsi.Context(dims={"ngrid": [n] * 3, "n_pw": npw, "n_bands": nb, "n_proj": np_, "n_ions": np_})
    ctx.set_basis(m, np.zeros(npw), 1.0)
    ctx.set_veff(np.zeros((n, n, n)))
    ctx.set_projectors(beta.cpu().numpy(), np.arange(np_ + 1), d.cpu().numpy().astype(complex))
    before = chfsi.launch_count()
    out = _apply_h(ctx, psi)
    # cuts, products and sums of two groups, D, the expansion's two, three passes
    assert chfsi.launch_count() - before == 2 * 3 + 1 + 2 + 3
    c = beta.conj() @ psi.T
    ref = (d[:, None] * c).T @ beta
    # sums of K products of unit rows, then of np_ of them: TOL covers one each
    bound = TOL * float(d.abs().max()) * torch.linalg.vector_norm(beta, dim=0)[None, :]
    bound = bound * torch.linalg.vector_norm(c, dim=0)[:, None] + TOL * np_ ** 0.5 * float(d.abs().max()) * 0.1
    assert bool(((out - ref).abs() <= bound).all())


def test_overlap_of_larger_blocks(chfsi):
    """Projectors set anew with other blocks, and then q of that larger size."""
    s = chfsi.SyntheticSystem(config_index=2, n_rep=1, ecut=8.0, ngrid=[0, 0, 0], n_bands=24)
    off = np.zeros(s.n_ions + 1, dtype=np.int32)
    off[1:] = np.arange(1, s.n_ions + 1)
    off[-1] = s.n_proj  # one large block
    rng = np.random.default_rng(8)
    sizes = np.diff(off)
    d = [np.diag(rng.standard_normal(k)).astype(complex) for k in sizes]
    q = [np.diag(0.1 + 0.1 * rng.random(k)).astype(complex) for k in sizes]
    assert sum(k * k for k in sizes) > len(s.dmat())
    ctx = _context(chfsi, s)
    ctx.set_projectors(s.beta(), off, np.concatenate([x.ravel() for x in d]))
    ctx.set_qmat(np.concatenate([x.ravel() for x in q]))
    psi = _psi(s)
    out, local = torch.empty_like(psi), torch.empty_like(psi)
    torch.cuda.synchronize()
    ctx.apply_sinv_h(psi.data_ptr(), out.data_ptr(), len(psi))
    ctx.apply_h_local(psi.data_ptr(), local.data_ptr(), len(psi))
    beta = torch.from_numpy(s.beta()).cuda()
    diag = [torch.from_numpy(np.concatenate([np.diag(x) for x in m])).cuda() for m in (d, q)]
    h = local + (diag[0][:, None] * (beta.conj() @ psi.T)).T @ beta
    back = out + (diag[1][:, None] * (beta.conj() @ out.T)).T @ beta  # S S^-1 H psi
    # a solve with S on either side of the products: cond(S) is below 1e3 here
    assert float((back - h).abs().max()) <= 1e3 * TOL * float(h.abs().max())
