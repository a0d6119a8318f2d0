"""Calls of different sizes from several threads, each on a stream and with data
of its own: a kernel's limit of dynamic shared memory belongs to the kernel, not
to the call, so a small call must not lower what a large one is about to use.

Every thread repeats its call and compares with its first, single-threaded
result; the calls are deterministic, so the bits are the same."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _run_threads(calls):
    errors = []

    def loop(call):
        try:
            call()
        except Exception as e:  # reported below, with the thread's own message
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_eigenproblems_of_different_sizes(chfsi):
    calls = []
    for n in (20, 64, 160, 256):
        g = torch.Generator(device="cuda").manual_seed(n)
        h = torch.view_as_complex(torch.randn(n, n, 2, generator=g, device="cuda", dtype=torch.float64))
        h = (h + h.mH).contiguous()
        s = (torch.eye(n, dtype=torch.complex128, device="cuda") + 0.01 * h / n).contiguous()
        st = torch.cuda.Stream()
        v = torch.empty_like(h)
        torch.cuda.synchronize()
        ref = chfsi.hegv_dev(h.data_ptr(), s.data_ptr(), n, v.data_ptr(), st.cuda_stream)

        def call(h=h, s=s, v=v, n=n, st=st, ref=ref):
            for _ in range(150):
                w = chfsi.hegv_dev(h.data_ptr(), s.data_ptr(), n, v.data_ptr(), st.cuda_stream)
                np.testing.assert_array_equal(w, ref)

        calls.append(call)
    _run_threads(calls)


def test_local_h_of_different_band_counts(chfsi):
    """108^3: two buffers per z-stick block with many bands, one with few."""
    n, radius = 108, 20.0
    r = np.arange(-20, 21)
    z, y, x = np.meshgrid(r, r, r, indexing="ij")
    keep = x * x + y * y + z * z <= radius * radius
    miller = np.ascontiguousarray(np.stack([x[keep], y[keep], z[keep]], axis=1), dtype=np.int32)
    kin = 0.5 * 0.04 * (miller.astype(np.float64) ** 2).sum(axis=1)
    rng = np.random.default_rng(1)
    veff = rng.standard_normal((n, n, n))
    calls = []
    for nb in (1, 96, 2, 64):
        ctx = chfsi.Context(dims={"ngrid": [n] * 3, "n_pw": len(kin), "n_bands": nb})
        ctx.set_basis(miller, kin, 0.2 * radius)
        ctx.set_veff(veff)
        psi = torch.from_numpy(rng.standard_normal((nb, len(kin)))
                               + 1j * rng.standard_normal((nb, len(kin)))).cuda()
        out = torch.empty_like(psi)
        torch.cuda.synchronize()
        ctx.apply_h_local(psi.data_ptr(), out.data_ptr(), nb)
        ref = out.clone()

        def call(ctx=ctx, psi=psi, out=out, nb=nb, ref=ref):
            for _ in range(300 if nb < 10 else 100):
                ctx.apply_h_local(psi.data_ptr(), out.data_ptr(), nb)
            assert bool((out == ref).all())

        calls.append(call)
    torch.cuda.synchronize()
    _run_threads(calls)
