"""The tensor-core form of the FP64 contractions (exact digit slices) against FP64 on the same
operands: double-float entry point (7 digits), becp and the V_NL apply (8 digits), at the edges of
its tiles (128 rows, 32 columns, 16 k per stage, 128 k per accumulation block)."""

from __future__ import annotations

import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if torch.cuda.is_available():
    from addft_gb300 import ops
    from addft_gb300._lib import LIB

U = 2.0 ** -53


def rnd(seed, *s, spread=0.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.complex(torch.randn(*s, generator=g, device="cuda", dtype=torch.float64),
                      torch.randn(*s, generator=g, device="cuda", dtype=torch.float64))
    if spread:   # components over `spread` decades, as plane-wave coefficients have
        x = x * 10.0 ** (-spread * torch.rand(*s, generator=g, device="cuda", dtype=torch.float64))
    return x


def bound(a, b, bits):
    """Slicing (2^-bits of the row's and the column's largest components per term, on both operands
    and for the dropped levels) plus the rounding of an FP64 sum of K terms in the reference."""
    K = a.shape[1]
    big = a.abs().amax(1)[:, None] * b.abs().amax(0)[None]
    return 8.0 * K * big * 2.0 ** -bits + (math.sqrt(K) + 4.0) * 4 * U * (a.abs() @ b.abs())


@pytest.mark.parametrize("M,N,K", [(128, 32, 6000), (129, 33, 2049), (127, 31, 2047), (1, 70, 20000), (300, 5, 1111),
                                   (64, 96, 1024), (65, 257, 4099), (37, 1700, 40), (200, 3000, 130)])
@pytest.mark.parametrize("spread", [0.0, 9.0])
def test_zgemm_df_tiles(M, N, K, spread):
    a, b = rnd(M, M, K, spread=spread), rnd(N + 1, N, K, spread=spread)
    out = ops.zgemm_df(a, b.transpose(0, 1), conj_a=True)
    ref = a.conj() @ b.T
    assert bool(((out - ref).abs() <= bound(a, b.T, 55)).all())
    c = rnd(3, K, N)                       # rotation: the right operand's rows are contiguous along N
    out = ops.zgemm_df(a, c)
    assert bool(((out - a @ c).abs() <= bound(a, c, 55)).all())
    out = ops.zgemm_df(a.T.contiguous().T, c.T.contiguous().T, conj_b=True)   # both operands transposed
    assert bool(((out - a @ c.conj()).abs() <= bound(a, c, 55)).all())


@pytest.mark.parametrize("nk,nb,P,nG", [(1, 64, 32, 1301), (2, 33, 129, 2050), (3, 31, 8, 4097), (1, 160, 64, 3001),
                                        (1, 1, 260, 5000), (8, 4, 8, 20000)])
def test_becp_and_apply_tiles(nk, nb, P, nG):
    proj, psi = rnd(1, nk, P, nG, spread=6.0), rnd(2, nk, nb, nG)
    b = ops.becp(proj, psi)
    dion = torch.diag(torch.linspace(-2.0, 1.0, P, dtype=torch.float64, device="cuda"))
    h0 = rnd(4, nk, nb, nG)
    h = ops.vnl_apply(proj, dion, b, h0.clone())
    for k in range(nk):
        ref = proj[k].conj() @ psi[k].T
        assert bool(((b[k] - ref).abs() <= bound(proj[k], psi[k].T, 60)).all())
        db = dion.to(torch.complex128) @ b[k]
        add = db.T @ proj[k]
        assert bool(((h[k] - (h0[k] + add)).abs() <= bound(db.T, proj[k], 60) + 2 * U * h0[k].abs()).all())


def test_scales_zeros_and_values_that_are_not_finite():
    M, N, K = 40, 50, 3000
    a, b = rnd(1, M, K), rnd(2, N, K)
    a[0] *= 1e-290
    a[1] *= 1e250
    b[2] *= 1e-200
    a[3] = 0
    a[4, 1:] = 0
    a[5] = 0.7                              # every digit of every term alike: the largest sums
    b[5] = 0.9
    a[6] = complex(5e-324, 0)               # subnormal
    ref = a.conj() @ b.T
    out = ops.zgemm_df(a, b.transpose(0, 1), conj_a=True)
    rows = [i for i in range(M) if i != 6]
    ok = (out - ref).abs() <= bound(a, b.T, 55) + 1e-323
    assert bool(ok[rows].all())
    a[7, 11] = complex(float("inf"), 0.0)
    b[9, 13] = complex(0.0, float("nan"))
    out2 = ops.zgemm_df(a, b.transpose(0, 1), conj_a=True)
    bad = torch.zeros((M, N), dtype=torch.bool, device="cuda")
    bad[7], bad[:, 9] = True, True
    assert bool((~torch.isfinite(torch.view_as_real(out2)).all(-1) == bad).all())
    assert torch.equal(out2[~bad], out[~bad])
    assert LIB.addft_tc05_status() == 0


def test_pieces_of_a_product_when_scratch_is_short():
    """The same product with the scratch of the whole and with an eighth of it (K, rows in pieces)."""
    import ctypes as C
    M, N, K = 100, 90, 9000
    a, b = rnd(1, M, K), rnd(2, N, K)
    need = int(LIB.addft_zgemm_df_work_bytes(M, N, K))
    outs = []
    for nbytes in (need, need // 4):
        w = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        out = torch.empty((M, N), dtype=torch.complex128, device="cuda")
        st = LIB.addft_zgemm_df(M, N, K, C.c_void_p(a.data_ptr()), K, 1, 1, C.c_void_p(b.data_ptr()), 1, K, 0,
                                C.c_void_p(out.data_ptr()), N, C.c_void_p(w.data_ptr()), nbytes,
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        torch.cuda.synchronize()
        outs.append(out)
    for o in outs:
        assert bool(((o - a.conj() @ b.T).abs() <= bound(a, b.T, 55)).all())


def guarded(nbytes):
    """A work buffer of `nbytes` before 32 MB of a pattern."""
    w = torch.full((nbytes + (32 << 20),), 0xA5, dtype=torch.uint8, device="cuda")
    return w, lambda: bool((w[nbytes:] == 0xA5).all())


@pytest.mark.parametrize("M,N,K,mb", [(1280, 320, 2432, 70),    # cut along K: the last piece would take more splits
                                      (591, 1316, 3000, 40),    # K, then rows and columns
                                      (1500, 700, 200, 3),      # rows and columns
                                      (40, 3000, 130, 2)])
def test_pieces_stay_within_the_scratch(M, N, K, mb):
    import ctypes as C
    a, b = rnd(1, M, K, spread=3.0), rnd(2, N, K)
    nbytes = mb << 20
    assert nbytes < int(LIB.addft_zgemm_df_work_bytes(M, N, K))
    w, clean = guarded(nbytes)
    out = torch.empty((M, N), dtype=torch.complex128, device="cuda")
    st = LIB.addft_zgemm_df(M, N, K, C.c_void_p(a.data_ptr()), K, 1, 1, C.c_void_p(b.data_ptr()), 1, K, 0,
                            C.c_void_p(out.data_ptr()), N, C.c_void_p(w.data_ptr()), nbytes,
                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    assert bool(((out - a.conj() @ b.T).abs() <= bound(a, b.T, 55)).all()) and clean()


@pytest.mark.parametrize("nk,nb,P,nG,mb", [(5, 40, 72, 3001, 40), (3, 70, 130, 2200, 24)])
def test_pieces_of_a_batch_stay_within_the_scratch(nk, nb, P, nG, mb):
    import ctypes as C
    proj, psi = rnd(1, nk, P, nG), rnd(2, nk, nb, nG)
    w, clean = guarded(mb << 20)
    out = torch.empty((nk, P, nb), dtype=torch.complex128, device="cuda")
    st = LIB.addft_becp(1, nk, nb, nG, P, C.c_void_p(proj.data_ptr()), C.c_void_p(psi.data_ptr()),
                        C.c_void_p(out.data_ptr()), C.c_void_p(w.data_ptr()), mb << 20,
                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    for k in range(nk):
        assert bool(((out[k] - proj[k].conj() @ psi[k].T).abs() <= bound(proj[k], psi[k].T, 60)).all())
    assert clean()


@pytest.mark.parametrize("K", [128, 384, 1024])
def test_aligned_digits(K):
    """Equal components whose digits are all next to the largest: the sums of a level pass 2^24 in its FP32
    accumulator.  What it drops, and what the dropped levels hold, stays below four roundings of the result (in
    products that are not split along K: the split sums are added in FP64)."""
    from fractions import Fraction
    x = float(Fraction(63, 64) + sum(Fraction(127, 64 * 256 ** i) for i in range(1, 6)))
    M, N = 400, 200
    a = torch.full((M, K), complex(x, x), dtype=torch.complex128, device="cuda")
    b = torch.full((N, K), complex(x, -x), dtype=torch.complex128, device="cuda")
    want = float(2 * K * Fraction(x) ** 2)
    for out in (ops.zgemm_df(a, b.transpose(0, 1)), ops.becp(a.conj().resolve_conj()[None], b[None])[0]):
        assert bool(((out.real - want).abs() <= 4 * U * want).all())
        assert bool((out.imag.abs() <= 4 * U * want).all())


@pytest.mark.parametrize("decades", [3, 6, 9, 12])
@pytest.mark.parametrize("K", [40, 512, 6000])
def test_graded_rows_meet_the_stated_bound(decades, K):
    """A large component against a zero, the rest far below it: errors are relative to the largest components
    of row and column (2^-50 K with 7 digits, 2^-56 K with 8), as stated, not to the result."""
    M, N = 130, 70
    a, b = rnd(1, M, K) * 10.0 ** -decades, rnd(2, N, K)
    a[:, 3] = 1.0
    b[:, 3] = 0.0
    ref = a.conj() @ b.T
    big = a.abs().amax(1)[:, None] * b.abs().amax(1)[None]
    fp64 = (math.sqrt(K) + 4.0) * 4 * U * (a.abs() @ b.abs().T)
    assert bool(((ops.zgemm_df(a, b.transpose(0, 1), conj_a=True) - ref).abs() <= K * 2.0 ** -50 * big + fp64).all())
    assert bool(((ops.becp(a[None], b[None])[0] - ref).abs() <= K * 2.0 ** -56 * big + fp64).all())


@pytest.mark.parametrize("K", [15, 16, 17, 33, 48, 95, 96])
@pytest.mark.parametrize("M,N", [(129, 1500), (63, 3100), (64, 3000), (65, 1200), (31, 5003), (33, 4097)])
def test_few_k_in_one_launch_give_the_bits_of_the_passes(M, N, K):
    """Products of up to 96 k find their exponents and digits in one launch; with zeros to 112 k the passes of longer
    products run.  Every order of both operands, conjugates, graded rows, a row and a column that are not finite."""
    if M * N * K < 2e6:
        pytest.skip("a small product in plain FP64")
    a, b = rnd(M, M, K, spread=6.0), rnd(N, K, N)
    a[5] = 0
    a[7, 3] = complex(float("inf"), 0.0)
    b[2, 9] = complex(0.0, float("nan"))
    a2 = torch.cat([a, torch.zeros((M, 112 - K), dtype=a.dtype, device="cuda")], 1)
    b2 = torch.cat([b, torch.zeros((112 - K, N), dtype=a.dtype, device="cuda")], 0)
    ok = torch.ones((M, N), dtype=torch.bool, device="cuda")
    ok[7], ok[:, 9] = False, False                      # zeros against what is not finite are NaN in the longer one
    for x, x2 in ((a, a2), (a.T.contiguous().T, a2.T.contiguous().T)):
        for y, y2 in ((b, b2), (b.T.contiguous().T, b2.T.contiguous().T)):
            for ca, cb in ((False, False), (True, False), (False, True)):
                o, p = ops.zgemm_df(x, y, conj_a=ca, conj_b=cb), ops.zgemm_df(x2, y2, conj_a=ca, conj_b=cb)
                assert torch.equal(torch.view_as_real(o)[ok], torch.view_as_real(p)[ok])
                assert bool((torch.isfinite(torch.view_as_real(o)).all(-1) == ok).all())


@pytest.mark.parametrize("nk,nb,P,nG", [(8, 24, 32, 700), (3, 31, 96, 1301)])
def test_few_k_of_a_batch(nk, nb, P, nG):
    """The V_NL apply of few projectors: all k points in one launch, added to H psi."""
    proj, b = rnd(1, nk, P, nG, spread=6.0), rnd(2, nk, P, nb)
    dion = torch.diag(torch.linspace(-2.0, 1.0, P, dtype=torch.float64, device="cuda"))
    h0 = rnd(4, nk, nb, nG)
    h = ops.vnl_apply(proj, dion, b, h0.clone())
    for k in range(nk):
        db = dion.to(torch.complex128) @ b[k]
        assert bool(((h[k] - (h0[k] + db.T @ proj[k])).abs() <= bound(db.T, proj[k], 60) + 2 * U * h0[k].abs()).all())
