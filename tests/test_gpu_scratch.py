"""Caller-held scratch: every size from an entry point's least on is taken, gives the same values, and is
not written past; tuning that asks for the FFT kernels reaches every FP64 transform."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if torch.cuda.is_available():
    from addft_gb300 import ops
    from addft_gb300.psp import synthetic
    from addft_gb300._lib import LIB, dbl_array

BOX = (45, 45, 48)
LAT = np.diag([14.0, 14.0, 15.0])
B = 2 * np.pi * np.linalg.inv(LAT).T
OMEGA = float(np.linalg.det(LAT))
F64 = torch.float64


def al256(n):
    return (n + 255) // 256 * 256


def sphere(frac):
    r = [int(frac * n) for n in BOX]
    m = np.stack(np.meshgrid(*(np.arange(-k, k + 1) for k in r), indexing="ij"), -1).reshape(-1, 3)
    return m[np.sum((m / (np.asarray(BOX) * frac)) ** 2, axis=1) <= 1.0].astype(np.int32)


def full():
    return np.stack(np.meshgrid(*(np.arange(n) for n in BOX), indexing="ij"), -1).reshape(-1, 3).astype(np.int32)


def atoms(nat):
    return np.random.default_rng(3).uniform(0, 1, (nat, 3)) @ LAT


def stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def p(t):
    return C.c_void_p(t.data_ptr())


def potentials(plan, wplan, kplan, nat):
    """name -> (call(work, bytes) -> output, least scratch, scratch asked for)"""
    rho = torch.rand(plan.N, dtype=F64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) + 0.5
    psp, pos = synthetic().c_struct(), dbl_array(atoms(nat).reshape(-1))
    bv = dbl_array(B.reshape(-1))

    def slab(q):
        return q.nplanes * BOX[1] * BOX[2] * 16

    def hartree(w, n):
        v, e = torch.empty(plan.N, dtype=F64, device="cuda"), torch.empty(1, dtype=F64, device="cuda")
        assert LIB.addft_hartree(plan.handle, bv, OMEGA, p(rho), p(v), p(e), p(w), n, stream()) == 0
        return torch.cat([v, e])

    def vloc(w, n):
        v = torch.empty(plan.N, dtype=F64, device="cuda")
        assert LIB.addft_local_potential(plan.handle, bv, OMEGA, nat, pos, C.byref(psp), p(v), p(w), n, stream()) == 0
        return v

    def kerker(w, n):
        v = torch.empty(plan.N, dtype=F64, device="cuda")
        assert LIB.addft_kerker(kplan.handle, bv, p(rho), 0.6, 1.1, p(v), p(w), n, stream()) == 0
        return v

    def grads(w, n):
        g = torch.empty(5 + 3 * nat + 18, dtype=F64, device="cuda")
        assert LIB.addft_density_gradients(wplan.handle, plan.handle, bv, OMEGA, nat, pos, C.byref(psp), p(rho), p(g),
                                           p(w), n, stream()) == 0
        return g

    part, g1, gw, gk = al256(10 * 304 * 8), al256(plan.nG * 16), al256(wplan.nG * 16), al256(kplan.nG * 16)
    return {
        "hartree": (hartree, part + 256 + 2 * g1 + slab(plan), LIB.addft_hartree_work_bytes(plan.handle)),
        "vloc": (vloc, g1 + slab(plan), LIB.addft_local_potential_work_bytes(plan.handle)),
        "kerker": (kerker, gk + slab(kplan), LIB.addft_kerker_work_bytes(kplan.handle)),
        "grads": (grads, 2 * part + 2 * 256 + al256(nat * 16 * 3 * 8) + gw + g1 + al256(max(slab(plan), slab(wplan))),
                  LIB.addft_density_gradients_work_bytes(wplan.handle, plan.handle, nat)),
    }


def plans():
    return ops.Plan(BOX, sphere(0.45)), ops.Plan(BOX, sphere(0.24)), ops.Plan(BOX, full())


@pytest.mark.parametrize("nat", [1, 5, 40])   # 40 atoms x 4e4 G: phases as products, with less scratch directly
@pytest.mark.parametrize("name", ["hartree", "vloc", "kerker", "grads"])
def test_potentials_take_the_scratch_of_one_slab(name, nat):
    call, least, asked = potentials(*plans(), nat)[name]
    whole = call(torch.empty(asked, dtype=torch.uint8, device="cuda"), asked)
    for nbytes in (least, least + 1, least + 255, (least + asked) // 2, asked):
        w = torch.full((nbytes + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        out = call(w, nbytes)
        # both forms are FP64 transforms of a field of 1e5 points: their difference is rounding
        assert bool(((out - whole).abs() <= 1e-12 * whole.abs().max()).all()), (nbytes, least, asked)
        assert bool((w[nbytes:] == 0xA5).all())


@pytest.mark.parametrize("key", [{"colfft": 0}, {"plane_split": 1}])
def test_tuning_for_the_fft_kernels_reaches_every_potential(key):
    tuned, plain = plans(), plans()
    for q in tuned:
        q.set_tuning(**key)
    for name in ("hartree", "vloc", "kerker", "grads"):
        call, least, asked = potentials(*tuned, 2)[name]
        cut = slice(0, 2) if name == "grads" else slice(None)   # energies: forces are split by the scratch
        room = torch.empty(max(asked, potentials(*plain, 2)[name][2]), dtype=torch.uint8, device="cuda")
        ffts = call(torch.empty(least, dtype=torch.uint8, device="cuda"), least)[cut]   # holds no other form
        assert torch.equal(call(room, room.numel())[cut], ffts), name
        assert not torch.equal(potentials(*plain, 2)[name][0](room, room.numel())[cut], ffts), name


def test_scratch_limits_hold_where_the_products_start(monkeypatch):
    """The wrappers' byte limits where more bands at once bring a form with larger bands."""
    sizes = []
    keep = ops.workspace
    monkeypatch.setattr(ops, "workspace", lambda n: (sizes.append(n), keep(n))[1])
    for box, nb in (((24, 24, 24), 200), ((30, 30, 32), 64), ((45, 45, 45), 20)):
        r = [int(0.45 * n) for n in box]
        m = np.stack(np.meshgrid(*(np.arange(-k, k + 1) for k in r), indexing="ij"), -1).reshape(-1, 3)
        plan = ops.Plan(box, m[np.sum((m / (np.asarray(box) * 0.45)) ** 2, axis=1) <= 1.0].astype(np.int32))
        psi = torch.zeros((1, nb, plan.nG), dtype=torch.complex128, device="cuda")
        kin = torch.zeros((1, plan.nG), dtype=F64, device="cuda")
        v = torch.zeros(plan.N, dtype=F64, device="cuda")
        for limit in (12 << 20, 24 << 20, 48 << 20, 96 << 20):
            sizes.clear()
            ops.hpsi(plan, psi, kin, v, max_work=limit)
            ops._chunk_work(plan, 1, nb, extra=1000, max_bytes=limit)
            for n in sizes:
                assert n <= limit
            assert all(n >= limit // 4 or n >= plan.work_bytes(nb, 1) for n in sizes)


def test_local_potential_of_few_atoms_asks_for_little():
    """Phase tables are sized for the atoms of the call, not for the most that there can be."""
    plan = plans()[0]
    cell = LIB.addft_local_potential_work_bytes(plan.handle)
    seen = []
    keep = ops.workspace
    ops.workspace = lambda n: (seen.append(n), keep(n))[1]
    try:
        ops.local_potential(plan, B, OMEGA, atoms(2), synthetic())
    finally:
        ops.workspace = keep
    assert seen[0] < cell / 2
    big = atoms(40)                                  # 40 atoms x 4e4 G: the products
    assert 40 * plan.nG > 5e5
    v = ops.local_potential(plan, B, OMEGA, big, synthetic())
    w = torch.empty(al256(plan.nG * 16) + plan.nplanes * BOX[1] * BOX[2] * 16, dtype=torch.uint8, device="cuda")
    ref = torch.empty_like(v)                        # scratch of one slab: a sincos per atom and G
    psp = synthetic().c_struct()
    assert LIB.addft_local_potential(plan.handle, dbl_array(B.reshape(-1)), OMEGA, 40, dbl_array(big.reshape(-1)),
                                     C.byref(psp), p(ref), p(w), w.numel(), stream()) == 0
    assert bool(((v - ref).abs() <= 1e-12 * ref.abs().max()).all())


@pytest.mark.parametrize("nat", [1, 2, 33, 70, 256])
def test_ewald_takes_less_scratch(nat):
    """From the scratch that the sums over pairs and a few reciprocal CTAs need (what was enough before the
    reciprocal sum kept partial sums per CTA) up to what the size query returns."""
    pos, z = atoms(nat), np.random.default_rng(5).uniform(0.5, 4.0, nat)
    nmax = 3
    whole = ops.ewald(LAT, pos, z, nmax=nmax)
    asked = LIB.addft_ewald_work_bytes(nat)
    pairs = al256(nat * nat * 13 * 8)
    for nbytes in (pairs + 24320 + 256 + al256(nat * 24), pairs + 4 * (10 + 3 * nat) * 8, (pairs + asked) // 2):
        w = torch.full((nbytes + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        out = torch.empty_like(whole)
        assert LIB.addft_ewald(dbl_array(LAT.reshape(-1)), nat, dbl_array(pos.reshape(-1)), dbl_array(z), 0.9, nmax,
                               p(out), p(w), nbytes, stream()) == 0
        # sums in another order: a few hundred roundings of the largest output
        assert bool(((out - whole).abs() <= 1e-12 * whole.abs().max()).all()), nbytes
        assert bool((w[nbytes:] == 0xA5).all())


@pytest.mark.parametrize("dt", [1, 0])
@pytest.mark.parametrize("nat,nb", [(1, 3), (6, 40), (40, 20)])
def test_nonlocal_gradients_take_less_scratch(dt, nat, nb):
    plan = ops.Plan(BOX, sphere(0.24))
    psp = synthetic()
    nh, nG, nk, csz = psp.nh, plan.nG, 1, 16 if dt else 8
    P = nat * nh
    pos = atoms(nat)
    g = torch.Generator(device="cuda").manual_seed(nat)
    psi = torch.randn((nk, nb, nG), dtype=torch.complex128, device="cuda", generator=g) / nG ** 0.5
    w_occ = torch.rand((nk, nb), dtype=F64, device="cuda", generator=g)
    dion = torch.diag(torch.linspace(-1.0, 1.0, P, dtype=F64, device="cuda"))
    if not dt:
        psi = psi.to(torch.complex64)
    whole = ops.nonlocal_gradients(plan, B, OMEGA, np.zeros((1, 3)), pos, psp, psi, w_occ, dion)
    asked = LIB.addft_nonlocal_gradients_work_bytes(dt, nk, nb, nG, nat, nh)
    # the same split-K partial sums as the size query's least (becp's default splits), one range of G
    tiles = -(-P // 32) * -(-nb // 64) * nk
    ns = max(1, min(-(-8 * 152 // tiles), -(-nG // 64)))
    partials = al256((ns + -(-ns // 8)) * nk * P * nb * csz) if ns > 1 else 0
    least = 2 * al256(nk * P * nG * csz) + 3 * al256(nk * P * nb * csz) + al256(nk * nb * 8) + al256(nk * P * 12 * 8)
    d = dion.to(F64 if dt else torch.float32).contiguous()
    cs = psp.c_struct()
    tol = 1e-12 if dt else 2e-6
    taken = 0
    for nbytes in sorted({least + partials, least + 4 * partials, (least + partials + asked) // 2, asked}):
        w = torch.full((nbytes + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        out = torch.empty_like(whole)
        st = LIB.addft_nonlocal_gradients(plan.handle, dt, dbl_array(B.reshape(-1)), OMEGA, nk, dbl_array([0.0] * 3), nb,
                                          nat, dbl_array(pos.reshape(-1)), C.byref(cs), p(psi), p(w_occ), p(d), p(out),
                                          p(w), nbytes, stream())
        assert st == 0 or (st == 1 and nbytes == least + partials)   # the test's guess of the least partials
        if st == 0:
            taken += nbytes < asked
            assert bool(((out - whole).abs() <= tol * whole.abs().max()).all()), nbytes
            assert bool((w[nbytes:] == 0xA5).all())
    assert taken >= 1 or asked <= least + 4 * partials
