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


@pytest.mark.parametrize("nat", [1, 5])
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
