"""Workloads of the ChFSI library as its users call it.

A case is a dict of plain values; its "kind" names the public entry point:

  local    Context.apply_h_local on device arrays: T + V_loc of a block of bands
  hpsi     Context.apply_h: the same with separable (Kleinman-Bylander) projectors
  sinv     Context.apply_sinv_h: the ultrasoft filter operator S^-1 H
  cn, tn   zgemm_cn (projections, overlaps) and zgemm_tn (rotations, expansions)
  ritz     hegv_dev on a subspace pair, then the density matrix of the occupied
           states (zgemm_cn), which does not depend on eigenvector phases
  pass     one SCF iteration by hand: build_v_eff(rho), set_psi, diagonalize,
           construct_density, in FP64 or mixed precision

Sizes follow the repository's own cells: 8 atoms (40^3 grid, 2,945 plane
waves, 20 bands), 64 atoms (72^3, 37,073, 160 bands, 256 or 512 projectors) and
216 atoms (108^3, 173,925, 576 bands, 1,728 projectors).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "chemrust-scf_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import chfsi  # noqa: E402

A0 = 10.26  # conventional diamond cell, bohr
C128, F64 = torch.complex128, torch.float64
SMOOTH = [30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 90, 96, 100, 108]


def listed():
    return [
        # smallest call of an SCF step: local H of the 8-atom cell's 20 bands
        {"name": "local_8atom", "kind": "local", "n": 40, "radius": 8.95, "nb": 20},
        # the same at 216 atoms, all 576 bands: what a filter step spends outside the projectors
        {"name": "local_216atom", "kind": "local", "n": 108, "radius": 34.64, "nb": 576},
        # full H with separable projectors, 64 atoms
        {"name": "hpsi_kb_64atom", "kind": "hpsi", "n_rep": 2, "n": 72, "ecut": 20.0, "nb": 160,
         "n_shell": 1},
        # ultrasoft operator, 64 atoms with 8 projectors each, an odd number of bands
        {"name": "sinvh_us_64atom", "kind": "sinv", "n_rep": 2, "n": 72, "ecut": 20.0, "nb": 161,
         "n_shell": 2},
        # beta^H psi of the 216-atom ultrasoft cell
        {"name": "project_216atom", "kind": "cn", "m": 1728, "n": 576, "k": 173925},
        # psi <- psi V of the 216-atom cell
        {"name": "rotate_216atom", "kind": "tn", "m": 576, "n": 173925, "k": 576},
        # odd, ragged band block against a k-point sized sphere
        {"name": "project_ragged", "kind": "cn", "m": 261, "n": 77, "k": 23847},
        # subspace problem in mid-SCF (nearly diagonal in the previous Ritz basis), 64 atoms
        {"name": "ritz_160", "kind": "ritz", "n": 160, "mix": 0.03},
        # subspace problem from a random start, 216 atoms
        {"name": "ritz_576", "kind": "ritz", "n": 576, "mix": 1.0},
        # whole SCF iterations: small cell (launch-bound), 64 atoms in FP64 and mixed precision
        {"name": "pass_8atom", "kind": "pass", "n_rep": 1, "n": 40, "ecut": 15.0, "nb": 20,
         "n_shell": 0, "ndeg": 12, "mixed": False, "kx": 0.0},
        {"name": "pass_kb_64atom", "kind": "pass", "n_rep": 2, "n": 72, "ecut": 20.0, "nb": 160,
         "n_shell": 1, "ndeg": 16, "mixed": False, "kx": 0.0},
        {"name": "pass_kb_64atom_mixed", "kind": "pass", "n_rep": 2, "n": 72, "ecut": 20.0,
         "nb": 160, "n_shell": 1, "ndeg": 16, "mixed": True, "kx": 0.0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _grid(n_rep, ecut):
    """Smallest listed grid that holds the products of a sphere of that cutoff."""
    need = 3.1 * math.sqrt(2.0 * ecut) * A0 * n_rep / (2.0 * math.pi)
    return next(n for n in SMOOTH if n >= need)


def draw(rng):
    kind = rng.choice(["local", "hpsi", "sinv", "cn", "tn", "ritz", "pass", "pass"])
    if kind == "local":
        n = rng.choice(SMOOTH)
        most = max(1, int(576 * (108.0 / n) ** 3))
        return {"kind": kind, "n": n, "radius": round(n / rng.uniform(3.15, 4.6), 3),
                "nb": _log_int(rng, 1, min(576, most))}
    if kind in ("hpsi", "sinv"):
        n_rep = rng.choice([1, 2])
        ecut = round(rng.uniform(10.0, 20.0), 2)
        return {"kind": kind, "n_rep": n_rep, "n": _grid(n_rep, ecut), "ecut": ecut,
                "nb": _log_int(rng, 17, 45) if n_rep == 1 else _log_int(rng, 129, 200),
                "n_shell": rng.choice([1, 2]) if kind == "hpsi" else 2}
    if kind == "cn":
        return {"kind": kind, "m": _log_int(rng, 1, 1728), "n": _log_int(rng, 1, 576),
                "k": _log_int(rng, 500, 173925)}
    if kind == "tn":
        return {"kind": kind, "m": _log_int(rng, 1, 576), "n": _log_int(rng, 500, 173925),
                "k": _log_int(rng, 1, 1728)}
    if kind == "ritz":
        return {"kind": kind, "n": _log_int(rng, 8, 576),
                "mix": round(10.0 ** rng.uniform(-3.0, 0.0), 5)}
    n_rep = rng.choice([1, 1, 2])
    ecut = round(rng.uniform(10.0, 20.0), 2)
    return {"kind": kind, "n_rep": n_rep, "n": _grid(n_rep, ecut), "ecut": ecut,
            "nb": rng.randint(18, 45) if n_rep == 1 else rng.randint(129, 180),
            "n_shell": rng.choice([0, 1]), "ndeg": rng.randint(8, 16),
            "mixed": rng.random() < 0.4, "kx": rng.choice([0.0, 0.25])}


# --------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1 + int(seed))


def _gauss(shape, gen):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, device="cuda", dtype=F64))


def _envelope(n, gen):
    """Decay of plane-wave coefficients over n plane waves spread through a sphere."""
    t = torch.rand(n, generator=gen, device="cuda", dtype=F64) ** (1.0 / 3.0)
    return 1.0 / (1.0 + 30.0 * t ** 4)


def _bands(nb, kin, gen):
    """Band-like vectors: random, smooth at large kinetic energy, unit norm."""
    psi = _gauss((nb, len(kin)), gen)
    psi *= 1.0 / (1.0 + (kin / 1.5) ** 2)
    psi /= torch.linalg.vector_norm(psi, dim=1, keepdim=True)
    return psi


def _sphere(n, radius):
    """Miller indices of a sphere, by (y, x) column and then z, and their squares."""
    r = int(radius)
    h = np.arange(-r, r + 1)
    k, x, z = np.meshgrid(h, h, h, indexing="ij")
    keep = x * x + k * k + z * z <= radius * radius
    m = np.stack([x[keep], k[keep], z[keep]], axis=1)
    order = np.lexsort((m[:, 2], m[:, 0] % n, m[:, 1] % n))
    m = np.ascontiguousarray(m[order], dtype=np.int32)
    return m, (m.astype(np.float64) ** 2).sum(axis=1)


def _sphere_case(case):
    """Context inputs of a "local" case: cutoff 25 Ha, one cell of that size."""
    miller, sq = _sphere(case["n"], case["radius"])
    unit = math.sqrt(50.0) / case["radius"]
    return miller, 0.5 * unit * unit * sq, unit * math.sqrt(sq.max())


def _potential(n, seed):
    """Smooth seeded potential, about -1.5 .. 0.5 Ha."""
    gen = _generator(seed + 77)
    c = _gauss((n, n, n), gen)
    f = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=F64)
    g2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + f[None, None, :] ** 2
    v = torch.fft.ifftn(c * torch.exp(-g2 / 18.0) / (1.0 + g2), norm="forward").real
    return 0.4 * v / v.std() - 0.5


def _system(case, seed):
    params = {"n_rep": case["n_rep"], "ngrid": [case["n"]] * 3, "ngrid_density": [case["n"]] * 3,
              "ecut": case["ecut"], "n_bands": case["nb"], "n_shell": case["n_shell"],
              "seed": 1000 + int(seed)}
    if case["kind"] != "sinv" and case["n_shell"]:
        params.update(lmax=1, rc_proj=[1.2, 1.4, 0, 0], d_min=0.5, d_max=2.0)
    if case.get("kx"):
        params["kpt"] = [case["kx"], 0.0, 0.0]
    return chfsi.SyntheticSystem(config_index=2 if case["kind"] == "sinv" else 0, **params)


def _veff_of(system):
    n = system.ngrid
    vg = torch.from_numpy(system.vloc_g()).cuda().reshape(n[2], n[1], n[0])
    return torch.fft.ifftn(vg, norm="forward").real.contiguous()


def _subspace(n, mix, gen):
    """H and S of a filtered block: Ritz vectors mixed by `mix`, amplified band by band."""
    occ = (3 * n) // 4
    e = torch.cat([torch.linspace(-0.35, 0.15, occ, device="cuda", dtype=F64),
                   torch.linspace(0.30, 0.90, n - occ, device="cuda", dtype=F64)])
    e = e + 0.2 / n * (torch.rand(n, generator=gen, device="cuda", dtype=F64) - 0.5)
    x = torch.eye(n, device="cuda", dtype=C128) + mix * _gauss((n, n), gen) / math.sqrt(2.0 * n)
    x = x * torch.exp(-3.0 * torch.linspace(0, 1, n, device="cuda", dtype=F64))[None, :]
    h = x.mH @ (e[:, None] * x)
    s = x.mH @ x
    return (h + h.mH) / 2, (s + s.mH) / 2, occ


def _blocks(flat, offsets):
    """Per-ion blocks as one dense matrix."""
    out = np.zeros((offsets[-1], offsets[-1]), dtype=np.complex128)
    at = 0
    for a, b in zip(offsets[:-1], offsets[1:]):
        out[a:b, a:b] = flat[at:at + (b - a) ** 2].reshape(b - a, b - a)
        at += (b - a) ** 2
    return torch.from_numpy(out).cuda()


class _Model:
    """Plain torch restatement of H, S, the filter and the density, in 64 bits."""

    def __init__(self, n, miller, kin, veff, system=None):
        self.n, self.veff = n, veff
        self.kin = torch.from_numpy(np.asarray(kin)).cuda()
        m = torch.from_numpy(miller.astype(np.int64)).cuda() % n
        self.at = m[:, 0] + n * (m[:, 1] + n * m[:, 2])
        self.beta = self.q = None
        if system is not None and system.n_proj:
            self.beta = torch.from_numpy(system.beta()).cuda()
            off = system.proj_offsets()
            self.d = _blocks(system.dmat(), off)
            if system.uspp:
                self.q = _blocks(system.qmat(), off)

    def grid(self, psi):
        g = torch.zeros(psi.shape[0], self.n ** 3, device="cuda", dtype=C128)
        g[:, self.at] = psi
        return torch.fft.ifftn(g.view(-1, self.n, self.n, self.n), dim=(1, 2, 3), norm="forward")

    def h(self, psi):
        out = psi * self.kin
        step = max(1, int(6e8 / self.n ** 3) // 16)
        for b in range(0, psi.shape[0], step):
            r = torch.fft.fftn(self.grid(psi[b:b + step]) * self.veff, dim=(1, 2, 3), norm="forward")
            out[b:b + step] += r.reshape(r.shape[0], -1)[:, self.at]
        if self.beta is not None:
            out += (self.d @ (self.beta.conj() @ psi.T)).T @ self.beta
        return out

    def sinv(self, y):
        """S^-1 y for S = 1 + beta q beta^H."""
        b = self.beta.conj() @ self.beta.T
        c = self.beta.conj() @ y.T
        eye = torch.eye(len(b), device="cuda", dtype=C128)
        return y - (self.q @ torch.linalg.solve(eye + b @ self.q, c)).T @ self.beta

    def filtered(self, psi, ndeg, gmax, eig):
        lm = 0.5 * gmax * gmax + float(self.veff.max() - self.veff.min())
        cut = min(eig[-1] + 0.2 * (eig[-1] - eig[0]), 0.95 * lm)
        c, e = (lm + cut) / 2.0, (lm - cut) / 2.0
        prev, cur = psi, (self.h(psi) - c * psi) / e
        for _ in range(ndeg - 1):
            prev, cur = cur, 2.0 / e * (self.h(cur) - c * cur) - prev
        return cur

    def ritz(self, psi):
        """Ritz values and vectors of a block, through its orthonormalised rows."""
        q = torch.linalg.qr(psi.T.contiguous())[0].T.contiguous()
        h = q.conj() @ self.h(q).T
        w, v = torch.linalg.eigh((h + h.mH) / 2)
        return w, v.T @ q

    def density(self, psi, occ, omega):
        rho = torch.zeros(self.n, self.n, self.n, device="cuda", dtype=F64)
        for b in range(0, len(occ), 16):
            f = occ[b:b + 16]
            rho += (f[:, None, None, None] * self.grid(psi[b:b + 16][:len(f)]).abs() ** 2).sum(0)
        return rho / omega


def _pz(rho):
    """Perdew-Zunger exchange-correlation energy per electron and potential."""
    rs = (3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0)
    ex = -0.4581652932831429 / rs
    sr, lr = rs.sqrt(), rs.log()
    den = 1.0 + 1.0529 * sr + 0.3334 * rs
    far = -0.1423 / den
    vfar = far * (1.0 + 7.0 / 6.0 * 1.0529 * sr + 4.0 / 3.0 * 0.3334 * rs) / den
    near = 0.0311 * lr - 0.048 + 0.0020 * rs * lr - 0.0116 * rs
    vnear = (0.0311 * lr + (-0.048 - 0.0311 / 3.0) + 2.0 / 3.0 * 0.0020 * rs * lr
             + (2.0 * -0.0116 - 0.0020) / 3.0 * rs)
    return ex + torch.where(rs >= 1.0, far, near), 4.0 / 3.0 * ex + torch.where(rs >= 1.0, vfar, vnear)


def _v_eff(rho, vloc, a):
    """V_eff of a density in a cubic cell, with the Hartree and XC energies."""
    n = rho.shape[0]
    f = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=F64) * (2.0 * math.pi / a)
    g2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + f[None, None, :] ** 2
    rg = torch.fft.fftn(rho.to(C128), norm="forward")
    g2[0, 0, 0] = 1.0
    vh = 4.0 * math.pi * rg / g2
    vh[0, 0, 0] = 0.0
    exc, vxc = _pz(rho)
    eh = 0.5 * a ** 3 * float((rg.conj() * vh).real.sum())
    e = [eh, float((rho * exc).sum()) * a ** 3 / n ** 3]
    return vloc + torch.fft.ifftn(vh, norm="forward").real + vxc, e


def _pass_inputs(case, seed):
    """Density, bands and band energies as an SCF run has them a few iterations in."""
    s = _system(case, seed)
    a = A0 * case["n_rep"]
    gen = _generator(seed)
    vloc = _veff_of(s)
    bump = torch.exp(-2.0 * vloc)
    rho = (0.4 + 0.6 * bump / bump.mean()) * s.n_elec / s.omega
    model = _Model(case["n"], s.miller(), s.kinetic(), _v_eff(rho, vloc, a)[0], s)
    psi = _bands(case["nb"], model.kin, gen)
    w, psi = model.ritz(psi)
    for _ in range(2):
        w, psi = model.ritz(model.filtered(psi, 8, s.gmax, w.tolist()))
    return s, a, vloc, rho, psi, w.cpu().numpy()


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    kind = case["kind"]
    if kind == "local":
        miller, kin, gmax = _sphere_case(case)
        ctx = chfsi.Context(dims={"ngrid": [case["n"]] * 3, "n_pw": len(kin), "n_bands": case["nb"]})
        ctx.set_basis(miller, kin, gmax)
        ctx.set_veff(_potential(case["n"], seed).cpu().numpy())
        psi = _bands(case["nb"], torch.from_numpy(kin).cuda(), _generator(seed))
        return {"kind": kind, "ctx": ctx, "psi": psi, "out": torch.empty_like(psi)}
    if kind in ("hpsi", "sinv"):
        s = _system(case, seed)
        ctx = chfsi.Context(s)
        ctx.set_veff(_veff_of(s).cpu().numpy())
        psi = _bands(case["nb"], torch.from_numpy(s.kinetic()).cuda(), _generator(seed))
        return {"kind": kind, "ctx": ctx, "psi": psi, "out": torch.empty_like(psi)}
    if kind in ("cn", "tn"):
        a, b = _gemm_inputs(case, seed)
        out = torch.empty(case["m"], case["n"], device="cuda", dtype=C128)
        return {"kind": kind, "a": a, "b": b, "out": out, "size": (case["m"], case["n"], case["k"])}
    if kind == "ritz":
        h, s, occ = _subspace(case["n"], case["mix"], _generator(seed))
        return {"kind": kind, "h": h.contiguous(), "s": s.contiguous(), "occ": occ, "n": case["n"],
                "v": torch.empty_like(h), "p": torch.empty_like(h)}
    s, _, _, rho, psi, w = _pass_inputs(case, seed)
    ctx = chfsi.Context(s, precision=chfsi.PREC_MIXED if case["mixed"] else chfsi.PREC_FP64)
    if case["mixed"] and s.n_proj:
        ctx.set_tc_shapes(2, 0)  # the same tensor-core launch shapes on every run
    host = torch.empty(psi.shape, dtype=C128, pin_memory=True)
    host.copy_(psi)
    return {"kind": kind, "ctx": ctx, "rho": rho.cpu().numpy(), "host": host, "psi": host.numpy(),
            "eig": w, "ndeg": case["ndeg"]}


def _gemm_inputs(case, seed):
    gen = _generator(seed)
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "cn":
        env = _envelope(k, gen)
        return _gauss((m, k), gen) * env, _gauss((n, k), gen) * env / math.sqrt(k)
    return _gauss((k, m), gen) / math.sqrt(k), _gauss((k, n), gen) * _envelope(n, gen)


def run(state):
    kind = state["kind"]
    if kind == "local":
        state["ctx"].apply_h_local(state["psi"].data_ptr(), state["out"].data_ptr(), len(state["psi"]))
        return state["out"]
    if kind == "hpsi":
        state["ctx"].apply_h(state["psi"].data_ptr(), state["out"].data_ptr(), len(state["psi"]))
        return state["out"]
    if kind == "sinv":
        state["ctx"].apply_sinv_h(state["psi"].data_ptr(), state["out"].data_ptr(), len(state["psi"]))
        return state["out"]
    if kind == "cn":
        m, n, k = state["size"]
        chfsi.zgemm_cn(state["a"].data_ptr(), k, state["b"].data_ptr(), k, m, n, k, state["out"].data_ptr())
        return state["out"]
    if kind == "tn":
        m, n, k = state["size"]
        chfsi.zgemm_tn(state["a"].data_ptr(), m, state["b"].data_ptr(), n, state["out"].data_ptr(), n,
                       m, n, k)
        return state["out"]
    if kind == "ritz":
        n, v = state["n"], state["v"].data_ptr()
        w = chfsi.hegv_dev(state["h"].data_ptr(), state["s"].data_ptr(), n, v)
        chfsi.zgemm_cn(v, n, v, n, n, n, state["occ"], state["p"].data_ptr())
        return {"w": w, "p": state["p"]}
    ctx = state["ctx"]
    e = ctx.build_v_eff(state["rho"])
    ctx.set_psi(state["psi"])
    w = ctx.diagonalize(state["ndeg"], state["eig"])
    return {"e": e, "w": w, "rho": ctx.construct_density()}


# ------------------------------------------------------------- what they cost
def _n_pw(case):
    if case["kind"] == "local":
        return 4.0 / 3.0 * math.pi * case["radius"] ** 3
    return (A0 * case["n_rep"]) ** 3 / (6.0 * math.pi ** 2) * (2.0 * case["ecut"]) ** 1.5


def _n_proj(case):
    return 8 * case["n_rep"] ** 3 * 4 * case["n_shell"] if "n_shell" in case else 0


def _fft_flops(n):
    """One 3D transform each way with the lines the sphere needs (about 0.45 of all)."""
    return 2 * 0.45 * 5.0 * n ** 3 * math.log2(n ** 3)


def work(case):
    kind = case["kind"]
    if kind in ("cn", "tn"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 16.0 * (m * k + n * k + m * n), "flops": 8.0 * m * n * k}
    if kind == "ritz":
        n = case["n"]
        return {"bytes": 16.0 * 4 * n * n, "flops": 4.0 * 12.0 * n ** 3}
    npw, nb, n, npr = _n_pw(case), case["nb"], case["n"], _n_proj(case)
    size = 16.0 * npw
    apply_flops = nb * (_fft_flops(n) + 10.0 * npw)
    if kind == "local":
        return {"bytes": 2 * nb * size + 8.0 * n ** 3, "flops": apply_flops}
    if kind == "hpsi":
        return {"bytes": (2 * nb + npr) * size + 8.0 * n ** 3, "flops": apply_flops + 16.0 * npr * nb * npw}
    if kind == "sinv":
        return {"bytes": (2 * nb + npr) * size + 8.0 * n ** 3, "flops": apply_flops + 24.0 * npr * nb * npw}
    deg = case["ndeg"] + 1
    word = 8.0 if case["mixed"] else 16.0
    return {"bytes": deg * (3 * nb + npr) * word * npw + 2 * nb * size,
            "flops": deg * (apply_flops + 16.0 * npr * nb * npw) + 24.0 * nb * nb * npw}


# ------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "local":
        miller, kin, _ = _sphere_case(case)
        model = _Model(case["n"], miller, kin, _potential(case["n"], seed))
        return model.h(_bands(case["nb"], model.kin, _generator(seed)))
    if kind in ("hpsi", "sinv"):
        s = _system(case, seed)
        model = _Model(case["n"], s.miller(), s.kinetic(), _veff_of(s), s)
        h = model.h(_bands(case["nb"], model.kin, _generator(seed)))
        return h if kind == "hpsi" else model.sinv(h)
    if kind in ("cn", "tn"):
        a, b = _gemm_inputs(case, seed)
        return a.conj() @ b.T if kind == "cn" else a.T @ b
    if kind == "ritz":
        h, s, occ = _subspace(case["n"], case["mix"], _generator(seed))
        low = torch.linalg.cholesky(s)
        t = torch.linalg.solve_triangular(low, h, upper=False)
        t = torch.linalg.solve_triangular(low, t.mH, upper=False).mH
        w, u = torch.linalg.eigh((t + t.mH) / 2)
        v = torch.linalg.solve_triangular(low.mH, u, upper=True)[:, :occ]
        return {"w": w, "p": v.conj() @ v.T}
    s, a, vloc, rho, psi, w = _pass_inputs(case, seed)
    veff, e = _v_eff(rho, vloc, a)
    model = _Model(case["n"], s.miller(), s.kinetic(), veff, s)
    w, psi = model.ritz(model.filtered(psi, case["ndeg"], s.gmax, w.tolist()))
    occ = torch.from_numpy(s.occupations()).cuda()
    return {"e": np.array(e), "w": w, "rho": model.density(psi, occ[occ > 0], s.omega).reshape(-1)}

