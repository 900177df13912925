"""FP32 projector contractions on the tensor cores, at the edges of their tiles.

becp: 32 G per stage, 32 projectors and 16 to 96 bands per tile; apply: 128 G x 32 to 96 bands per
unit, 16 projectors per stage.  Against 64-bit sums of the same operands, elementwise within
c 2^-23 sum |a| |x|.  A stage's accumulator takes 8 (becp) or 24 (apply) truncating additions, each off by
less than 2^-23 of the sum of magnitudes, three or four products of the split add less than
2 units together, and the FP32 sums over stages and splits (at most 60 here, 2^-24 each) 30: c = 40 and
56.  The apply adds 2^-23 of the value it adds to.
"""

import pytest
import torch

from conftest import gpu_available

pytestmark = pytest.mark.gpu
if not gpu_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from addft_gb300 import ops  # noqa: E402
from addft_gb300._lib import LIB  # noqa: E402

EPS = 2.0 ** -23


def _rnd(g, *s):
    x = torch.complex(torch.randn(*s, generator=g, device="cuda"), torch.randn(*s, generator=g, device="cuda"))
    return x * torch.exp(2.0 * torch.randn(s[-1], generator=g, device="cuda"))   # a wide range over G or bands


@pytest.mark.parametrize("nk,nb,P,nG", [(1, 1, 1, 1), (1, 16, 32, 31), (2, 17, 33, 33), (1, 96, 8, 64), (1, 97, 31, 1025),
                                        (3, 40, 65, 4865), (1, 192, 64, 700), (1, 193, 5, 9729)])
def test_becp(nk, nb, P, nG):
    g = torch.Generator(device="cuda").manual_seed(11)
    proj, psi = _rnd(g, nk, P, nG), _rnd(g, nk, nb, nG)
    b = ops.becp(proj, psi).to(torch.complex128)
    p64, x64 = proj.to(torch.complex128), psi.to(torch.complex128)
    ref = torch.einsum("kpg,kbg->kpb", p64.conj(), x64)
    mag = torch.einsum("kpg,kbg->kpb", p64.abs(), x64.abs())
    assert float(((b - ref).abs() / mag).max()) < 40 * EPS
    assert LIB.addft_tc05_status() == 0


@pytest.mark.parametrize("nk,nb,P,nG", [(1, 32, 33, 19457), (1, 33, 48, 19456), (2, 96, 49, 9729), (1, 97, 64, 14593),
                                        (1, 1, 100, 9000), (1, 160, 257, 2000), (3, 65, 40, 6527), (1, 8, 64, 500)])
def test_apply(nk, nb, P, nG):
    g = torch.Generator(device="cuda").manual_seed(12)
    proj, b, h0 = _rnd(g, nk, P, nG), _rnd(g, nk, P, nb), _rnd(g, nk, nb, nG)
    d = torch.randn(P, generator=g, device="cuda")
    h = ops.vnl_apply(proj, torch.diag(d), b, h0.clone()).to(torch.complex128)   # D becp is then one product
    db = (d[:, None] * b).to(torch.complex128)
    p64 = proj.to(torch.complex128)
    ref = h0.to(torch.complex128) + torch.einsum("kpg,kpb->kbg", p64, db)
    mag = torch.einsum("kpg,kpb->kbg", p64.abs(), db.abs()) + h0.abs()
    assert float(((h - ref).abs() / mag).max()) < 56 * EPS
    assert LIB.addft_tc05_status() == 0
