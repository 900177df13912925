"""The work this framework does for its users, as cases to be timed and checked.

A case is one call (or one pass of a few calls that belong together) through the
package's public entry points, on a system of a size that the package's own
configurations use: the H psi microbench boxes, and silicon cells from Si2 to Si64.
``listed`` names fixed sizes, ``draw`` gives further ones of the same ranges.
``exact`` restates what a pass computes in 64 bits with plain torch, without the package.
"""

from __future__ import annotations

import functools
import itertools
import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "ad-dft_gb300"))

import addft_gb300 as ad  # noqa: E402
from addft_gb300 import autograd, observables, ops, solver, system  # noqa: E402
from addft_gb300.psp import Pseudo, dion_full  # noqa: E402

A_SI = 10.26   # Bohr
F64, C128 = torch.float64, torch.complex128
TWO_PI = 2.0 * math.pi


def listed():
    return [
        # One H psi of the small microbench box in double precision: latency and launches count.
        dict(name="hpsi_micro15_f64", kind="hpsi", family="micro", n=15, nb=64, nat=8, dtype="f64"),
        # The microbench's headline: 64 bands on the 72^3 box, 8 atoms x 4 projectors, single precision.
        dict(name="hpsi_micro72_f32", kind="hpsi", family="micro", n=72, nb=64, nat=8, dtype="f32"),
        # The smallest structure of the batch workload: Si2 on a 2x2x2 k mesh, single precision.
        dict(name="hpsi_si2_kmesh_f32", kind="hpsi", family="si", nat=2, ecut=8.0, nk=2, nb=4, dtype="f32"),
        # The inner loop of the large SCF: every band of Si64 at Gamma, many projectors, single precision.
        dict(name="hpsi_si64_f32", kind="hpsi", family="si", nat=64, ecut=15.0, nk=1, nb=168, dtype="f32"),
        # The same call of the plain double-precision SCF (and of the refinement's anchors).
        dict(name="hpsi_si64_f64", kind="hpsi", family="si", nat=64, ecut=15.0, nk=1, nb=160, dtype="f64"),
        # Differentiation workload: H psi forward and its gradients in psi and V(r) on Si8.
        dict(name="hpsi_grad_si8_f64", kind="hpsi_grad", nat=8, ecut=10.0, nk=1, nb=20, dtype="f64"),
        # The band density that closes every SCF step of Si64.
        dict(name="density_si64_f64", kind="density", nat=64, ecut=15.0, nk=1, nb=160, dtype="f64"),
        # Hartree + exchange-correlation + local: the effective potential of every SCF step.
        dict(name="potential_si64", kind="potential", nat=64, ecut=15.0),
        # A new geometry (relaxation, dynamics): local potential, projector tables, kinetic diagonal.
        dict(name="geometry_si64", kind="geometry", nat=64, ecut=15.0, nk=1),
        # Forces and strain derivative of a converged state.
        dict(name="gradients_si64", kind="gradients", nat=64, ecut=15.0, nk=1, nb=160),
        # The refinement's subspace product conj(X) Y^T on the Si64 shapes.
        dict(name="subspace_si64", kind="subspace", m=168, n=336, k=23847, form="project"),
        # A whole call: SCF, free energy and forces of the two-atom cell, double precision.
        dict(name="scf_si2_f64", kind="scf", ecut=2.0, nb=2),
    ]


SMOOTH = [n for n in range(9, 81)
          if functools.reduce(lambda x, p: x // p if x % p == 0 else x, (2, 2, 2, 2, 2, 2, 3, 3, 3, 3, 5, 5), n) == 1]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hpsi", "hpsi", "hpsi", "hpsi_grad", "density", "potential", "geometry", "gradients",
                       "subspace", "scf"])
    nat = rng.choice([2, 4, 8, 16, 32, 64])
    ecut = round(rng.uniform(5.0, 15.0), 2)
    nk = 2 if nat <= 16 and rng.random() < 0.5 else 1
    nb = max(1, int(nat * rng.uniform(1.5, 2.6)))
    dtype = rng.choice(["f32", "f64"])
    if kind == "hpsi" and rng.random() < 0.5:
        n = rng.choice(SMOOTH)
        return dict(kind="hpsi", family="micro", n=n, nb=_log_int(rng, 1, 96 if dtype == "f32" else 48),
                    nat=rng.randint(1, 10), dtype=dtype)
    if kind == "hpsi":
        return dict(kind="hpsi", family="si", nat=nat, ecut=ecut, nk=nk, nb=nb, dtype=dtype)
    if kind in ("hpsi_grad", "density"):
        return dict(kind=kind, nat=nat, ecut=ecut, nk=nk, nb=nb, dtype="f64" if kind == "hpsi_grad" else dtype)
    if kind == "potential":
        return dict(kind=kind, nat=nat, ecut=ecut)
    if kind == "geometry":
        return dict(kind=kind, nat=nat, ecut=ecut, nk=nk)
    if kind == "gradients":
        return dict(kind=kind, nat=nat, ecut=ecut, nk=nk, nb=nb)
    if kind == "subspace":
        m = _log_int(rng, 4, 200)
        if rng.random() < 0.5:
            return dict(kind=kind, m=m, n=_log_int(rng, 4, 336), k=_log_int(rng, 300, 24000), form="project")
        return dict(kind=kind, m=m, n=_log_int(rng, 300, 24000), k=m, form="rotate")
    return dict(kind="scf", ecut=round(rng.uniform(1.8, 3.5), 2), nb=rng.choice([2, 3]))


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------
def _lattice(nat):
    a = A_SI
    return {2: 0.5 * a * np.array([[0, 1, 1], [1, 0, 1], [1, 1, 0]]),
            4: np.array([[a / 2, a / 2, 0], [-a / 2, a / 2, 0], [0, 0, a]]),
            8: np.eye(3) * a, 16: np.diag([a, a, 2 * a]), 32: np.diag([2 * a, 2 * a, a]), 64: np.eye(3) * 2 * a}[nat]


@functools.lru_cache(maxsize=8)
def _static(nat, ecut, nk, nb):
    """What a program keeps over many geometries: the frozen basis with its plans."""
    from addft_gb300.batch import diamond_cell
    lat = _lattice(nat)
    frac = diamond_cell(lat)
    mesh = ad.monkhorst_pack((nk,) * 3) if nk > 1 else ad.gamma()
    return ad.setup(lat, frac, ecut=ecut, nband=nb, kmesh=mesh), lat, frac


def _system(case, seed):
    s, lat, frac = _static(case["nat"], case["ecut"], case.get("nk", 1), case.get("nb", 4))
    rng = np.random.default_rng(seed)
    frac = frac + rng.normal(0, 0.05, frac.shape) @ np.linalg.inv(lat)
    return ad.System(geo=ad.Cell(lattice=lat, frac=frac), static=s.static)


@functools.lru_cache(maxsize=8)
def _micro_plan(n):
    """The microbench's sphere of radius 0.45 n in the n^3 box and its plan."""
    r = int(0.45 * n)
    m = np.stack(np.meshgrid(*(np.arange(-r, r + 1),) * 3, indexing="ij"), -1).reshape(-1, 3)
    m = m[np.sum(m * m, axis=1) <= (0.45 * n) ** 2]
    m = m[np.lexsort((m[:, 2], m[:, 1], m[:, 0], np.sum(m * m, axis=1)))].astype(np.int32)
    return ops.Plan((n,) * 3, m), m


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + salt)


def _bands(g, nk, nb, kin):
    """Orthonormal bands (nk, nb, nG) whose coefficients fall off with the kinetic energy."""
    out = []
    for k in range(nk):
        c = torch.randn((nb, kin.shape[-1]), dtype=C128, device="cuda", generator=g) / (1.0 + kin[k])
        L = torch.linalg.cholesky(c.conj() @ c.T)
        out.append(torch.linalg.solve_triangular(L.conj(), c, upper=False))
    return torch.stack(out)


def _gvec(miller, lat):
    b = torch.as_tensor(TWO_PI * np.linalg.inv(np.asarray(lat)).T, dtype=F64, device="cuda")
    return torch.as_tensor(np.asarray(miller), dtype=F64, device="cuda") @ b


def _tables(miller, lat, kpts, pos, psp):
    """Kinetic diagonal (nk, nG) and projectors (nk, nat * nh, nG) in 64 bits."""
    omega = abs(float(np.linalg.det(lat)))
    G = _gvec(miller, lat)
    kin, proj = [], []
    pos = torch.as_tensor(np.asarray(pos), dtype=F64, device="cuda")
    for k in np.asarray(kpts):
        v = G + torch.as_tensor(k, dtype=F64, device="cuda")
        kin.append(0.5 * (v * v).sum(-1))
        proj.append(_projectors(v, pos, psp, omega))
    return torch.stack(kin), torch.stack(proj)


def _projectors(v, pos, psp, omega):
    q2 = (v * v).sum(-1)
    q = torch.where(q2 > 1e-30, torch.sqrt(torch.where(q2 > 1e-30, q2, 1.0)), 0.0)
    qs = torch.where(q2 > 1e-30, q, 1.0)
    rows = []
    for l, w, b in zip(psp.proj_l, psp.proj_w, psp.proj_b):
        qq = torch.clamp(q, min=1e-12)
        beta = w * qq ** l * torch.exp(-0.5 * (qq * b) ** 2)
        if l == 0:
            rows.append(beta * math.sqrt(1.0 / (4.0 * math.pi)))
        else:
            c = math.sqrt(3.0 / (4.0 * math.pi))
            rows += [beta * c * v[:, 2] / qs, -beta * c * v[:, 0] / qs, -beta * c * v[:, 1] / qs]
    form = torch.stack(rows)                                  # (nh, nG)
    arg = pos @ v.T                                           # (nat, nG)
    ph = torch.complex(torch.cos(arg), -torch.sin(arg))
    return (ph[:, None, :] * form[None] / math.sqrt(omega)).reshape(-1, v.shape[0])


def _density_like(case, seed, geo, static):
    """A smooth positive density with the cell's electron count: superposed Gaussians on the atoms."""
    n = static.basis.fft_shape
    lat = np.asarray(geo.lattice)
    m = torch.as_tensor(static.basis.miller, dtype=F64, device="cuda")
    G = _gvec(static.basis.miller, lat)
    pos = torch.as_tensor(geo.frac @ lat, dtype=F64, device="cuda")
    arg = pos @ G.T
    s = torch.complex(torch.cos(arg), -torch.sin(arg)).sum(0) * torch.exp(-0.45 * (G * G).sum(-1))
    box = _scatter(s[None], n, m.to(torch.int64))
    rho = torch.fft.ifftn(box, dim=(1, 2, 3)).real.reshape(-1)
    rho = rho - rho.min() + 1e-3 * (rho.max() - rho.min())
    omega = abs(float(np.linalg.det(lat)))
    rho = rho * (static.nelec / (rho.sum() * omega / rho.numel()))
    g = _gen(seed, 5)
    return rho * (1.0 + 1e-3 * torch.rand(rho.shape, generator=g, device="cuda", dtype=F64))


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _hpsi_inputs(case, seed):
    """(plan, miller, box, psi, kin, v, proj, dion), cast to the case's type."""
    g = _gen(seed)
    if case.get("family", "si") == "micro":
        n = case["n"]
        plan, miller = _micro_plan(n)
        lat = np.eye(3) * (0.5 * n)
        rng = np.random.default_rng(seed)
        pos = rng.uniform(0, 1, (case["nat"], 3)) @ lat
        psp = Pseudo(proj_w=(1.0, 1.0), proj_b=(1.0, 1.0), proj_l=(0, 1), dion=np.eye(2))
        kin, proj = _tables(miller, lat, np.zeros((1, 3)), pos, psp)
        dion = torch.eye(proj.shape[1], dtype=F64, device="cuda")
        pick = miller[rng.integers(1, miller.shape[0], 16)]
        ax = torch.arange(n, dtype=F64, device="cuda") * (TWO_PI / n)
        v = torch.zeros((n, n, n), dtype=F64, device="cuda")
        for m, amp, ph in zip(pick, rng.uniform(0, 0.5, 16), rng.uniform(0, TWO_PI, 16)):
            v += amp * torch.cos(int(m[0]) * ax[:, None, None] + int(m[1]) * ax[None, :, None]
                                 + int(m[2]) * ax[None, None, :] + ph)
        psi = torch.randn((1, case["nb"], miller.shape[0]), dtype=C128, device="cuda", generator=g)
        L = torch.linalg.cholesky(psi[0].conj() @ psi[0].T)
        psi = torch.linalg.solve_triangular(L.conj(), psi[0], upper=False)[None]
        box = (n,) * 3
    else:
        s = _system(case, seed)
        st, geo = s.static, s.geo
        plan, miller, box = st.device().wfc, st.basis.miller, st.basis.fft_shape
        kin, proj = _tables(miller, geo.lattice, st.kpts, geo.frac @ geo.lattice, st.psp)
        dion = torch.as_tensor(dion_full(st.psp, st.natom), dtype=F64, device="cuda")
        rho = _density_like(case, seed, geo, st)
        v = 0.3 * torch.sin(rho / rho.mean()) - 0.5 * (rho / rho.mean()) ** (1.0 / 3.0)
        psi = _bands(g, st.nk, case["nb"], kin)
    rdt, cdt = (torch.float32, torch.complex64) if case["dtype"] == "f32" else (F64, C128)
    return (plan, miller, box, psi.to(cdt).contiguous(), kin.to(rdt), v.reshape(-1).to(rdt).contiguous(),
            proj.to(cdt).contiguous(), dion.to(rdt))


def _occ(seed, nk, nb):
    """Occupations between 0 and 1 with a Fermi edge."""
    g = _gen(seed, 3)
    f = torch.sigmoid((0.6 * nb - torch.arange(nb, dtype=F64, device="cuda")[None]) * 0.5
                      + torch.randn((nk, 1), dtype=F64, device="cuda", generator=g) * 0.1)
    return f.expand(nk, nb).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "hpsi":
        plan, _, _, psi, kin, v, proj, dion = _hpsi_inputs(case, seed)
        return dict(kind=kind, plan=plan, psi=psi, kin=kin, v=v, proj=proj, dion=dion)
    if kind == "hpsi_grad":
        plan, _, _, psi, kin, v, proj, dion = _hpsi_inputs(case, seed)
        g = torch.randn(psi.shape, dtype=psi.dtype, device="cuda", generator=_gen(seed, 1))
        return dict(kind=kind, plan=plan, psi=psi.requires_grad_(True), kin=kin, v=v.requires_grad_(True), proj=proj,
                    dion=dion, g=g)
    if kind == "density":
        s = _system(case, seed)
        plan, _, _, psi, *_ = _hpsi_inputs(case, seed)
        wocc = 2.0 / s.static.nk * _occ(seed, s.static.nk, case["nb"])
        return dict(kind=kind, plan=plan, psi=psi, wocc=wocc, omega=ad.volume(s.geo.lattice))
    if kind in ("potential", "geometry", "gradients"):
        s = _system(case, seed)
        out = dict(kind=kind, geo=s.geo, static=s.static)
        s.static.device()
        if kind == "potential":
            out["cache"] = system.build_geometry_cache(s.geo, s.static)
            out["rho"] = _density_like(case, seed, s.geo, s.static)
        if kind == "gradients":
            out["cache"] = system.build_geometry_cache(s.geo, s.static)
            out["state"] = _state(case, seed, s)
        return out
    if kind == "subspace":
        m, n, k = case["m"], case["n"], case["k"]
        g = _gen(seed)
        if case["form"] == "project":          # conj(X) Y^T: rows of plane-wave coefficients
            fall = 1.0 / (1.0 + torch.arange(k, dtype=F64, device="cuda") / (0.05 * k)) ** (2.0 / 3.0)
            a = torch.randn((m, k), dtype=C128, device="cuda", generator=g) * fall
            b = torch.randn((n, k), dtype=C128, device="cuda", generator=g) * fall
            a, b = (x / torch.linalg.vector_norm(x, dim=1, keepdim=True) for x in (a, b))
            return dict(kind=kind, a=a, b=b.transpose(0, 1), conj_a=True)
        # U X: a unitary rotation of the bands
        u = torch.linalg.qr(torch.randn((k, k), dtype=C128, device="cuda", generator=g))[0][:, :m]
        fall = 1.0 / (1.0 + torch.arange(n, dtype=F64, device="cuda") / (0.05 * n)) ** (2.0 / 3.0)
        b = torch.randn((k, n), dtype=C128, device="cuda", generator=g) * fall
        return dict(kind=kind, a=u.transpose(0, 1), b=b / torch.linalg.vector_norm(b, dim=1, keepdim=True),
                    conj_a=False)
    return dict(kind=kind, system=_fixture(case, seed))


def _fixture(case, seed):
    rng = np.random.default_rng(seed)
    frac = np.array([[0.0, 0.0, 0.0], [0.53, 0.47, 0.49]]) + rng.normal(0, 0.004, (2, 3))
    return ad.setup(np.eye(3) * 6.0, frac, ecut=case["ecut"], nband=case["nb"], density_factor=4.0)


def _state(case, seed, s):
    """A state as an SCF leaves it: orthonormal bands, occupations and their density."""
    st = s.static
    G = _gvec(st.basis.miller, s.geo.lattice)
    kin = torch.stack([0.5 * ((G + torch.as_tensor(k, dtype=F64, device="cuda")) ** 2).sum(-1) for k in st.kpts])
    psi = _bands(_gen(seed), st.nk, case["nb"], kin)
    occ = _occ(seed, st.nk, case["nb"])
    wocc = (2.0 / st.nk * occ)[..., None]
    rho = _exact_density(psi, wocc, st.basis.fft_shape, st.basis.miller, ad.volume(s.geo.lattice))
    return system.SCFState(psi=psi, eig=torch.zeros_like(occ), occ=occ, mu=torch.zeros(1, dtype=F64, device="cuda"),
                       rho_r=rho, n_iter=1, residual=0.0)


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "hpsi":
        return ops.hpsi(s["plan"], s["psi"], s["kin"], s["v"], s["proj"], s["dion"])
    if kind == "hpsi_grad":
        y = autograd.hpsi(s["plan"], s["psi"], s["kin"], s["v"], s["proj"], s["dion"])
        gpsi, gv = torch.autograd.grad(y, (s["psi"], s["v"]), s["g"])
        return {"y": y.detach(), "psi": gpsi, "v": gv}
    if kind == "density":
        return ops.density(s["plan"], s["psi"], s["wocc"], s["omega"])
    if kind == "potential":
        v, parts = solver.effective_potential(s["static"], s["cache"], s["rho"])
        return {"v_eff": v, "v_h": parts["v_h"], "v_xc": parts["v_xc"], "e_h": parts["e_h"], "xc": parts["xc_sums"]}
    if kind == "geometry":
        c = system.build_geometry_cache(s["geo"], s["static"])
        return {"v_loc": c.v_loc_r, "proj": c.proj, "kin": c.kin}
    if kind == "gradients":
        dR, deps = observables.envelope_gradients(s["geo"], s["static"], s["state"], s["cache"])
        return {"dR": dR, "deps": deps}
    if kind == "subspace":
        return ops.zgemm_df(s["a"], s["b"], conj_a=s["conj_a"])
    e, f = ad.energy_and_forces(s["system"])
    return {"energy": e, "forces": f}


# ---------------------------------------------------------------------------
# work: each input read once, each output written once; textbook operation counts
# ---------------------------------------------------------------------------
def _sizes(case):
    if case.get("family", "si") == "micro":
        plan, m = _micro_plan(case["n"])
        return 1, m.shape[0], case["n"] ** 3, 4 * case["nat"], 0
    s, _, _ = _static(case["nat"], case["ecut"], case.get("nk", 1), case.get("nb", 4))
    b = s.static.basis
    return s.static.nk, b.nG, b.nfft, 4 * case["nat"], b.nG_rho


def work(case):
    kind = case["kind"]
    if kind == "subspace":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 16.0 * (m * k + k * n + m * n), "flops": 8.0 * m * n * k}
    if kind == "scf":
        s = _fixture(case, 0).static
        N, nG, nb = s.basis.nfft, s.basis.nG, case["nb"]
        # 80 iterations of a dense eigenproblem, its H columns, the density and the potential
        fl = 80.0 * (40.0 * nG ** 3 + 10.0 * N * math.log2(N) * (nG + nb + 3))
        return {"bytes": 80.0 * 16.0 * (2 * nG * nG + 4 * N), "flops": fl}
    nk, nG, N, P, nGr = _sizes(case)
    nb = case.get("nb", 0)
    c = 8 if case.get("dtype") == "f32" else 16
    r = c // 2
    fft = 5.0 * N * math.log2(N)
    if kind in ("hpsi", "hpsi_grad"):
        by = 2.0 * c * nk * nb * nG + r * N + r * nk * nG + c * nk * P * nG + r * P * P
        fl = nk * nb * (2 * fft + 16.0 * P * nG + 8.0 * nG)
        if kind == "hpsi":
            return {"bytes": by, "flops": fl}
        # forward, the adjoint H g, and the cross density conj(g(r)) psi(r)
        return {"bytes": by + 2.0 * c * nk * nb * nG + r * N, "flops": 2 * fl + nk * nb * (2 * fft + 8.0 * N)}
    if kind == "density":
        return {"bytes": c * nk * nb * nG + 8.0 * N, "flops": nk * nb * (fft + 4.0 * N)}
    if kind == "potential":
        return {"bytes": 8.0 * 5 * N, "flops": 2 * fft + 100.0 * N}
    if kind == "geometry":
        return {"bytes": 8.0 * N + 16.0 * nk * P * nG + 8.0 * nk * nG,
                "flops": fft + case["nat"] * 8.0 * nGr + 8.0 * nk * P * nG}
    nt = 17.0 ** 3 + 21.0 ** 3
    return {"bytes": 16.0 * nk * nb * nG + 8.0 * N,
            "flops": nk * nb * (fft + 4.0 * N + 32.0 * P * nG) + 3 * fft + case["nat"] * 16.0 * nGr
            + 20.0 * nk * P * nG + 10.0 * case["nat"] ** 2 * nt}


# ---------------------------------------------------------------------------
# exact: the same outputs in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _scatter(c, box, miller):
    idx = torch.as_tensor(np.asarray(miller.cpu() if isinstance(miller, torch.Tensor) else miller),
                          dtype=torch.int64, device="cuda")
    f = ((idx[:, 0] % box[0]) * box[1] + idx[:, 1] % box[1]) * box[2] + idx[:, 2] % box[2]
    out = torch.zeros((c.shape[0], box[0] * box[1] * box[2]), dtype=C128, device="cuda")
    out[:, f] = c
    return out.reshape((-1,) + tuple(box))


def _gather(x, box, miller):
    idx = torch.as_tensor(np.asarray(miller), dtype=torch.int64, device="cuda")
    f = ((idx[:, 0] % box[0]) * box[1] + idx[:, 1] % box[1]) * box[2] + idx[:, 2] % box[2]
    return x.reshape(x.shape[0], -1)[:, f]


def _exact_hpsi(psi, kin, v, proj, dion, box, miller):
    out = torch.empty_like(psi)
    vb = v.reshape(box)
    for k in range(psi.shape[0]):
        for b0 in range(0, psi.shape[1], 32):
            c = psi[k, b0:b0 + 32]
            r = torch.fft.ifftn(_scatter(c, box, miller), dim=(1, 2, 3)) * vb
            out[k, b0:b0 + 32] = kin[k] * c + _gather(torch.fft.fftn(r, dim=(1, 2, 3)), box, miller)
        if proj is not None:
            becp = proj[k].conj() @ psi[k].T
            out[k] += (dion.to(C128) @ becp).T @ proj[k]
    return out


def _exact_density(psi, wocc, box, miller, omega):
    N = box[0] * box[1] * box[2]
    rho = torch.zeros(N, dtype=F64, device="cuda")
    for k in range(psi.shape[0]):
        for b0 in range(0, psi.shape[1], 32):
            r = torch.fft.ifftn(_scatter(psi[k, b0:b0 + 32], box, miller), dim=(1, 2, 3), norm="forward")
            rho += (wocc[k, b0:b0 + 32].reshape(-1, 1) * (r.real ** 2 + r.imag ** 2).reshape(-1, N)).sum(0)
    return rho / omega


def _exc(n):
    """LDA exchange and correlation energies per electron (Perdew-Zunger 1981)."""
    rs = (3.0 / (4.0 * math.pi * n)) ** (1.0 / 3.0)
    ex = -0.75 * (3.0 * n / math.pi) ** (1.0 / 3.0)
    lo = torch.clamp(rs, max=1.0)
    hi = torch.clamp(rs, min=1.0)
    ln = torch.log(lo)
    small = 0.0311 * ln - 0.048 + 0.0020 * lo * ln - 0.0116 * lo
    large = -0.1423 / (1.0 + 1.0529 * torch.sqrt(hi) + 0.3334 * hi)
    return ex, torch.where(rs < 1.0, small, large)


def _vxc(rho):
    n = torch.clamp(rho, min=1e-14).detach().requires_grad_(True)
    ex, ec = _exc(n)
    v, = torch.autograd.grad((n * (ex + ec)).sum(), n)
    return torch.where(rho > 1e-14, v, 0.0), (n * ex).sum().detach(), (n * ec).sum().detach()


def _exact_potential(rho, box, lat, miller, v_loc):
    N, omega = rho.numel(), abs(float(np.linalg.det(lat)))
    G = _gvec(miller, lat)
    q2 = (G * G).sum(-1)
    n = _gather(torch.fft.fftn(rho.reshape(box).to(C128)[None], dim=(1, 2, 3)) / N, box, miller)[0]
    vg = torch.where(q2 > 1e-14, 4.0 * math.pi / torch.where(q2 > 1e-14, q2, 1.0), 0.0) * n
    e_h = 0.5 * omega * (n.conj() * vg).real.sum()
    v_h = torch.fft.ifftn(_scatter(vg[None], box, miller), dim=(1, 2, 3), norm="forward").real.reshape(-1)
    v_xc, sx, sc = _vxc(rho)
    return {"v_eff": v_loc + v_h + v_xc, "v_h": v_h, "v_xc": v_xc, "e_h": e_h.reshape(1),
            "xc": torch.stack([sx, sc, (v_xc * rho).sum()])}


def _structure(G, pos):
    s = torch.zeros(G.shape[0], dtype=C128, device="cuda")
    for r in pos:
        a = G @ r
        s = s + torch.complex(torch.cos(a), -torch.sin(a))
    return s


def _exact_vloc(static, lat, pos):
    omega = abs(float(np.linalg.det(lat)))
    G = _gvec(static.basis.miller_rho, lat)
    amp = -static.psp.vloc_amp * torch.exp(-0.5 * (G * G).sum(-1) * static.psp.vloc_sigma ** 2)
    vg = amp * _structure(G, torch.as_tensor(pos, dtype=F64, device="cuda")) / omega
    box = static.basis.fft_shape
    return torch.fft.ifftn(_scatter(vg[None], box, static.basis.miller_rho), dim=(1, 2, 3),
                           norm="forward").real.reshape(-1)


def _ewald(lat, pos, z, eta, nmax=8):
    """Ewald energy, differentiable in the lattice rows and positions."""
    omega = torch.abs(torch.linalg.det(lat))
    nat = pos.shape[0]
    ax = torch.arange(-nmax, nmax + 1, dtype=F64, device="cuda")
    T = torch.cartesian_prod(ax, ax, ax) @ lat
    d0 = (pos[:, None, :] - pos[None, :, :]).reshape(-1, 3)
    eye = torch.eye(nat, dtype=torch.bool, device="cuda").reshape(-1)
    origin = torch.cartesian_prod(ax, ax, ax).abs().sum(-1) == 0
    e = 0.0
    for c in range(0, T.shape[0], max(1, 2_000_000 // (nat * nat))):
        t = slice(c, c + max(1, 2_000_000 // (nat * nat)))
        e = e + torch.utils.checkpoint.checkpoint(_ewald_real, d0, T[t], eye, origin[t], eta, z, use_reentrant=False)
    nr = nmax + 2
    ar = torch.arange(-nr, nr + 1, dtype=F64, device="cuda")
    m = torch.cartesian_prod(ar, ar, ar)
    m = m[m.abs().sum(-1) > 0]
    G = m @ (TWO_PI * torch.linalg.inv(lat).T)
    q2 = (G * G).sum(-1)
    arg = G @ pos.T
    s2 = torch.cos(arg).sum(-1) ** 2 + torch.sin(arg).sum(-1) ** 2
    e = e + 2.0 * math.pi / omega * z * z * (torch.exp(-q2 / (4.0 * eta * eta)) / q2 * s2).sum()
    return e - eta / math.sqrt(math.pi) * nat * z * z - math.pi * (nat * z) ** 2 / (2.0 * omega * eta * eta)


def _ewald_real(d0, T, eye, origin, eta, z):
    d = d0[:, None, :] + T[None]
    r2 = (d * d).sum(-1)
    skip = eye[:, None] & origin[None]
    r = torch.sqrt(torch.where(skip, 1.0, r2))
    return 0.5 * z * z * torch.where(skip, 0.0, torch.erfc(eta * r) / r).sum()


def _energy(static, lat0, pos0, psi, wocc, eps, dpos):
    """Total energy of frozen bands under a strain eps and displacements dpos, differentiable in both."""
    I = torch.eye(3, dtype=F64, device="cuda")
    F = I + eps
    lat0 = torch.as_tensor(lat0, dtype=F64, device="cuda")
    lat = lat0 @ F
    pos = (torch.as_tensor(pos0, dtype=F64, device="cuda") + dpos) @ F
    omega0, omega = torch.abs(torch.linalg.det(lat0)), torch.abs(torch.linalg.det(lat))
    bvec = TWO_PI * torch.linalg.inv(lat).T
    b, psp = static.basis, static.psp
    mw = torch.as_tensor(b.miller, dtype=F64, device="cuda")
    mr = torch.as_tensor(b.miller_rho, dtype=F64, device="cuda")
    N = b.nfft
    rho = _exact_density(psi, wocc, b.fft_shape, b.miller, 1.0) / omega
    box = torch.fft.fftn((rho * omega).detach().reshape(b.fft_shape).to(C128)[None], dim=(1, 2, 3)) / N
    Gr = mr @ bvec
    nr = _gather(box, b.fft_shape, b.miller_rho)[0] / omega
    amp = -psp.vloc_amp * torch.exp(-0.5 * (Gr * Gr).sum(-1) * psp.vloc_sigma ** 2)
    e = (amp * (_structure(Gr, pos) * nr.conj()).real).sum()
    Gw = mw @ bvec
    q2 = (Gw * Gw).sum(-1)
    nw = _gather(box, b.fft_shape, b.miller)[0] / omega
    ok = q2 > 1e-14
    e = e + 0.5 * omega * torch.where(ok, 4.0 * math.pi * (nw.real ** 2 + nw.imag ** 2) / torch.where(ok, q2, 1.0),
                                      0.0).sum()
    ex, ec = _exc(torch.clamp(rho, min=1e-14))
    e = e + omega / N * (torch.clamp(rho, min=1e-14) * (ex + ec)).sum()
    d = torch.as_tensor(dion_full(psp, static.natom), dtype=C128, device="cuda")
    for k in range(psi.shape[0]):
        v = Gw + torch.as_tensor(static.kpts[k], dtype=F64, device="cuda")
        w = wocc[k].reshape(-1)
        e = e + (0.5 * (v * v).sum(-1) * (w[:, None] * (psi[k].real ** 2 + psi[k].imag ** 2)).sum(0)).sum()
        becp = torch.utils.checkpoint.checkpoint(lambda vv, pp, om, kk=k: _projectors(vv, pp, psp, 1.0).conj()
                                                 @ psi[kk].T / torch.sqrt(om), v, pos, omega, use_reentrant=False)
        e = e + (w * (becp.conj() * (d @ becp)).sum(0).real).sum()
    return e + _ewald(lat, pos, psp.zval, static.eta_ewald)


def _gradients(static, lat, pos, psi, wocc):
    eps = torch.zeros((3, 3), dtype=F64, device="cuda", requires_grad=True)
    dpos = torch.zeros((static.natom, 3), dtype=F64, device="cuda", requires_grad=True)
    e = _energy(static, lat, pos, psi, wocc, eps, dpos)
    deps, dR = torch.autograd.grad(e, (eps, dpos))
    return e.detach(), dR, deps


def _fermi(eig, nelec, sigma):
    lo, hi = eig.min() - 20.0, eig.max() + 20.0
    for _ in range(200):
        mu = 0.5 * (lo + hi)
        if 2.0 * torch.sigmoid((mu - eig) / sigma).sum() < nelec:
            lo = mu
        else:
            hi = mu
    return torch.sigmoid((0.5 * (lo + hi) - eig) / sigma)


def _exact_scf(s):
    """Self-consistent free energy and forces of a small cell at Gamma from dense matrices."""
    st, lat = s.static, s.geo.lattice
    pos = s.geo.frac @ lat
    b, N = st.basis, st.basis.nfft
    kin, proj = _tables(b.miller, lat, st.kpts, pos, st.psp)
    dion = torch.as_tensor(dion_full(st.psp, st.natom), dtype=F64, device="cuda")
    v_loc = _exact_vloc(st, lat, pos)
    omega = abs(float(np.linalg.det(lat)))
    eye = torch.eye(b.nG, dtype=C128, device="cuda")[None]

    def step(rho):
        v = _exact_potential(rho, b.fft_shape, lat, b.miller, v_loc)["v_eff"]
        H = _exact_hpsi(eye, kin, v, proj, dion, b.fft_shape, b.miller)[0].T
        w, u = torch.linalg.eigh(0.5 * (H + H.conj().T))
        eig, psi = w[:st.nband], u[:, :st.nband].T.contiguous()[None]
        f = _fermi(eig, st.nelec, st.sigma)
        return _exact_density(psi, (2.0 * f)[None], b.fft_shape, b.miller, omega), psi, f

    rho = torch.full((N,), st.nelec / omega, dtype=F64, device="cuda")
    hist = []
    for it in range(300):
        out, psi, f = step(rho)
        r = out - rho
        if float(r.abs().sum()) * omega / N / st.nelec < 2e-14:
            break
        hist = (hist + [(rho, r)])[-8:]
        R = torch.stack([h[1] for h in hist])
        if len(hist) > 1:                       # Anderson: residual differences in the least-squares sense
            D = (R[1:] - R[:-1]).T
            X = torch.stack([h[0] for h in hist])
            c = torch.linalg.lstsq(D, r[:, None], driver="gels").solution[:, 0]
            rho = rho + 0.5 * r - ((X[1:] - X[:-1]).T + 0.5 * D) @ c
        else:
            rho = rho + 0.5 * r
    wocc = (2.0 * f)[None]
    e, dR, _ = _gradients(st, lat, pos, psi, wocc)
    g = torch.clamp(f, 1e-14, 1.0 - 1e-14)
    ent = -(g * torch.log(g) + (1.0 - g) * torch.log(1.0 - g)).sum()
    return {"energy": float(e - 2.0 * st.sigma * ent), "forces": -dR}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hpsi", "hpsi_grad"):
        plan, miller, box, psi, kin, v, proj, dion = _hpsi_inputs(case, seed)
        psi, proj = psi.to(C128), proj.to(C128)
        kin, v, dion = kin.to(F64), v.to(F64), dion.to(F64)
        y = _exact_hpsi(psi, kin, v, proj, dion, box, miller)
        if kind == "hpsi":
            return y
        g = torch.randn(psi.shape, dtype=psi.dtype, device="cuda", generator=_gen(seed, 1))
        N = box[0] * box[1] * box[2]
        gv = torch.zeros(N, dtype=F64, device="cuda")
        for k, b in itertools.product(range(psi.shape[0]), range(0, psi.shape[1], 16)):
            p, q = (torch.fft.ifftn(_scatter(x[k, b:b + 16], box, miller), dim=(1, 2, 3), norm="forward")
                    for x in (psi, g))
            gv += (q.conj() * p).real.sum(0).reshape(-1) / N
        return {"y": y, "psi": _exact_hpsi(g, kin, v, proj, dion, box, miller), "v": gv}
    if kind == "subspace":
        s = prepare(case, seed)
        return (s["a"].conj() if s["conj_a"] else s["a"]) @ s["b"]
    if kind == "scf":
        return _exact_scf(_fixture(case, seed))
    s = _system(case, seed)
    st, lat = s.static, s.geo.lattice
    pos = s.geo.frac @ lat
    if kind == "density":
        _, miller, box, psi, *_ = _hpsi_inputs(case, seed)
        wocc = 2.0 / st.nk * _occ(seed, st.nk, case["nb"])
        return _exact_density(psi.to(C128), wocc[..., None], box, miller, ad.volume(lat))
    if kind == "potential":
        return _exact_potential(_density_like(case, seed, s.geo, st), st.basis.fft_shape, lat, st.basis.miller,
                                _exact_vloc(st, lat, pos))
    if kind == "geometry":
        kin, proj = _tables(st.basis.miller, lat, st.kpts, pos, st.psp)
        return {"v_loc": _exact_vloc(st, lat, pos), "proj": proj, "kin": kin}
    state = _state(case, seed, s)
    wocc = (2.0 / st.nk * state.occ)[..., None]
    _, dR, deps = _gradients(st, lat, pos, state.psi, wocc)
    return {"dR": dR, "deps": deps}
