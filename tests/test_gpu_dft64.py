"""The FP64 transforms as digit-slice products on the tensor cores against torch's FP64 FFTs: ragged
boxes, spheres and full boxes, one band to several blocks of lines.

Tolerance: a stage rounds each of its outputs once (2^-53 of it) and slices its inputs 62 bits below
the line's largest; what a coefficient set of l1 norm s can carry through the three stages of a
transform stays below 4 x 2^-53 s, and the reference's own FFT is granted the same."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if torch.cuda.is_available():
    from addft_gb300 import ops
    from addft_gb300._lib import LIB

U = 2.0 ** -53
C128, F64 = torch.complex128, torch.float64


def sphere(box, frac):
    r = [int(frac * n) for n in box]
    m = np.stack(np.meshgrid(*(np.arange(-k, k + 1) for k in r), indexing="ij"), -1).reshape(-1, 3)
    m = m[np.sum((m / (np.asarray(box) * frac)) ** 2, axis=1) <= 1.0]
    rng = np.random.default_rng(1)
    return m[rng.permutation(len(m))].astype(np.int32)


def full(box):
    return np.stack(np.meshgrid(*(np.arange(n) for n in box), indexing="ij"), -1).reshape(-1, 3).astype(np.int32)


def scatter(c, box, m):
    i = torch.as_tensor(m, dtype=torch.int64, device="cuda")
    f = ((i[:, 0] % box[0]) * box[1] + i[:, 1] % box[1]) * box[2] + i[:, 2] % box[2]
    x = torch.zeros((c.shape[0], int(np.prod(box))), dtype=C128, device="cuda")
    x[:, f] = c
    return x.reshape((-1,) + tuple(box)), f


CASES = [((30, 32, 36), 0.45, 1), ((27, 30, 28 + 2), 0.25, 3), ((45, 45, 45), 0.45, 5), ((75, 72, 80), 0.24, 2),
         ((100, 96, 108), 0.3, 1), ((32, 32, 32), None, 1), ((128, 40, 9), 0.4, 2), ((64, 64, 64), 0.45, 33),
         ((30, 32, 36), 0.45, 11), ((27, 30, 30), 0.25, 40), ((128, 40, 9), 0.4, 10), ((15, 12, 16), 0.45, 45),
         ((32, 32, 32), None, 10), ((9, 9, 9), 0.45, 160)]


@pytest.mark.parametrize("box,frac,nb", CASES)
def test_transforms_hpsi_and_density(box, frac, nb):
    m = full(box) if frac is None else sphere(box, frac)
    plan = ops.Plan(box, m)
    g = torch.Generator(device="cuda").manual_seed(nb)
    c = torch.randn((nb, plan.nG), dtype=C128, device="cuda", generator=g)
    c = c * 10.0 ** (-6.0 * torch.rand(plan.nG, dtype=F64, device="cuda", generator=g))   # several decades
    N = plan.N
    x, f = scatter(c, box, m)
    r = torch.fft.ifftn(x, dim=(1, 2, 3), norm="forward").reshape(nb, N)
    l1 = c.abs().sum(1, keepdim=True)
    out = ops.psi_to_real(plan, c, 1.0)
    assert bool(((out - r).abs() <= 8 * U * l1).all())
    back = ops.real_to_psi(plan, r, 1.0)
    ref = torch.fft.fftn(r.reshape((nb,) + box), dim=(1, 2, 3)).reshape(nb, N)[:, f] / N
    assert bool(((back - ref).abs() <= 8 * U * r.abs().sum(1, keepdim=True) / N * np.sqrt(N)).all())
    v = torch.randn(N, dtype=F64, device="cuda", generator=g)
    kin = torch.rand((1, plan.nG), dtype=F64, device="cuda", generator=g) * 10
    h = ops.hpsi(plan, c[None], kin, v)[0]
    href = kin * c + torch.fft.fftn((r * v).reshape((nb,) + box), dim=(1, 2, 3)).reshape(nb, N)[:, f] / N
    assert bool(((h - href).abs() <= 16 * U * l1 * v.abs().max() + 4 * U * (kin * c).abs()).all())
    w = torch.rand((1, nb), dtype=F64, device="cuda", generator=g)
    rho = ops.density(plan, c[None], w, 2.5)
    rref = (w[0][:, None] * (r.real ** 2 + r.imag ** 2)).sum(0) / 2.5
    tol = (w[0][:, None] * (16 * U * l1 * r.abs() + 8 * U * (r.abs() ** 2))).sum(0) / 2.5 + nb * 4 * U * rref
    assert bool(((rho - rref).abs() <= tol + 1e-300).all())
    assert LIB.addft_tc05_status() == 0


@pytest.mark.parametrize("nb", [3, 13])
def test_lines_that_are_not_finite_stay_with_their_band(nb):
    box = (32, 32, 32)
    m = sphere(box, 0.4)
    plan = ops.Plan(box, m)
    g = torch.Generator(device="cuda").manual_seed(2)
    c = torch.randn((nb, plan.nG), dtype=C128, device="cuda", generator=g)
    good = ops.psi_to_real(plan, c, 1.0)
    c[1, 7] = complex(float("nan"), 0.0)
    out = ops.psi_to_real(plan, c, 1.0)
    rest = [0] + list(range(2, nb))
    assert torch.equal(out[rest], good[rest])
    assert bool(torch.isnan(torch.view_as_real(out[1])).all())


@pytest.mark.parametrize("box,nb", [((45, 45, 45), 5), ((25, 27, 45), 9)])
def test_density_in_scratch_of_every_size_around_its_groups(box, nb):
    """Scratch of g slabs of partial sums and one band, and up to 300 bytes more or less: one chunk of bands
    at a time, in as many groups as fit; nothing is written past the buffer's end."""
    import ctypes as C
    m = sphere(box, 0.45)
    plan = ops.Plan(box, m)
    g = torch.Generator(device="cuda").manual_seed(nb)
    c = torch.randn((1, nb, plan.nG), dtype=C128, device="cuda", generator=g)
    w = torch.rand((1, nb), dtype=F64, device="cuda", generator=g)
    x, _ = scatter(c[0], box, m)
    r = torch.fft.ifftn(x, dim=(1, 2, 3), norm="forward").reshape(nb, plan.N)
    ref = (w[0][:, None] * (r.real ** 2 + r.imag ** 2)).sum(0) / 2.5
    l1 = c[0].abs().sum(1, keepdim=True)
    tol = (w[0][:, None] * (16 * U * l1 * r.abs() + 8 * U * (r.abs() ** 2))).sum(0) / 2.5 + nb * 4 * U * ref
    band = plan.work_bytes(nb, 1) - plan.work_bytes(nb - 1, 1)
    for groups in (1, 2, 3, 4):
        for more in (-256, -1, 0, 1, 100, 191, 192, 255, 256, 300):
            nbytes = groups * 16 * plan.N + band + more
            work = torch.full((nbytes + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
            rho = torch.full((plan.N,), float("nan"), dtype=F64, device="cuda")
            st = LIB.addft_density(plan.handle, 1, 1, nb, 2.5, C.c_void_p(c.data_ptr()), C.c_void_p(w.data_ptr()),
                                   C.c_void_p(rho.data_ptr()), C.c_void_p(work.data_ptr()), nbytes,
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream))
            if st != 0:        # refused only below the least scratch of one band
                assert st == 1 and nbytes < plan.work_bytes(1, 1), (groups, more)
                continue
            assert bool(((rho - ref).abs() <= tol).all()), (groups, more)
            assert bool((work[nbytes:] == 0xA5).all()), (groups, more)


def test_more_bands_than_a_grid_has_rows():
    """Small boxes in large batches: the reordering kernel's grid holds 65,535 bands of one z tile."""
    box, nb = (4, 4, 5), 66000
    m = sphere(box, 0.45)
    plan = ops.Plan(box, m)
    g = torch.Generator(device="cuda").manual_seed(4)
    c = torch.randn((nb, plan.nG), dtype=C128, device="cuda", generator=g)
    out = ops.psi_to_real(plan, c, 1.0)
    x, _ = scatter(c, box, m)
    ref = torch.fft.ifftn(x, dim=(1, 2, 3), norm="forward").reshape(nb, plan.N)
    assert bool(((out - ref).abs() <= 8 * U * c.abs().sum(1, keepdim=True)).all())


# boxes of every size class from where the products start, and one band below
@pytest.mark.parametrize("box,frac,nb", [((12, 12, 12), 0.45, 46), ((9, 10, 15), 0.45, 60), ((20, 20, 20), 0.25, 165),
                                         ((24, 24, 24), 0.45, 58), ((25, 25, 50), 0.25, 14), ((32, 32, 32), None, 19),
                                         ((30, 32, 36), 0.45, 30), ((36, 36, 36), 0.25, 9), ((32, 32, 64), 0.45, 7)])
def test_where_the_products_start(box, frac, nb):
    for n in (nb, nb - 1):
        test_transforms_hpsi_and_density(box, frac, n)


def test_many_bands_in_scratch_for_a_few_run_the_ffts():
    """24^3 x 64 bands in 8 MB: the products would go in four chunks of six launches."""
    import ctypes as C
    box = (24, 24, 24)
    m = sphere(box, 0.45)
    plan = ops.Plan(box, m)
    g = torch.Generator(device="cuda").manual_seed(3)
    c = torch.randn((1, 64, plan.nG), dtype=C128, device="cuda", generator=g)
    v = torch.randn(plan.N, dtype=F64, device="cuda", generator=g)
    kin = torch.rand((1, plan.nG), dtype=F64, device="cuda", generator=g)
    whole = ops.hpsi(plan, c, kin, v)
    out = torch.empty_like(c)
    n = LIB.addft_launch_count()
    st = LIB.addft_hpsi_noalloc(plan.handle, 1, 1, 64, C.c_void_p(c.data_ptr()), C.c_void_p(kin.data_ptr()),
                                C.c_void_p(v.data_ptr()), 0, C.c_void_p(0), C.c_void_p(0), C.c_void_p(out.data_ptr()),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0 and LIB.addft_launch_count() - n <= 12
    l1 = c[0].abs().sum(1, keepdim=True)
    assert bool(((out - whole).abs() <= 16 * U * l1 * v.abs().max() + 4 * U * (kin[:, None] * c).abs()).all())
