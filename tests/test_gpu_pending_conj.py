"""Views with a pending conjugation or sign (x.conj(), x.conj().imag) are the values they stand for, in every
wrapper that hands memory to the library, and as incoming gradients."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if torch.cuda.is_available():
    from addft_gb300 import autograd, ops

BOX = (12, 15, 16)


def case():
    r = [int(0.4 * n) for n in BOX]
    m = np.stack(np.meshgrid(*(np.arange(-k, k + 1) for k in r), indexing="ij"), -1).reshape(-1, 3)
    plan = ops.Plan(BOX, m[np.sum((m / (np.asarray(BOX) * 0.4)) ** 2, axis=1) <= 1.0].astype(np.int32))
    g = torch.Generator(device="cuda").manual_seed(1)
    c = [torch.randn(s, dtype=torch.complex128, device="cuda", generator=g)
         for s in ((1, 6, plan.nG), (1, 4, plan.nG), (6, plan.N))]
    return plan, *c, torch.randn(plan.N, dtype=torch.float64, device="cuda", generator=g)


def test_wrappers_read_the_values():
    plan, psi, proj, field, v = case()
    kin = torch.rand((1, plan.nG), dtype=torch.float64, device="cuda")
    dion = torch.eye(4, dtype=torch.float64, device="cuda")
    w = torch.rand((1, 6), dtype=torch.float64, device="cuda")
    for f in (lambda x, p, r: ops.hpsi(plan, x, kin, v, p, dion), lambda x, p, r: ops.becp(p, x),
              lambda x, p, r: ops.psi_to_real(plan, x[0], 2.0), lambda x, p, r: ops.real_to_psi(plan, r, 2.0),
              lambda x, p, r: ops.density(plan, x, w, 2.0), lambda x, p, r: ops.zgemm_df(x[0], p[0].T),
              lambda x, p, r: ops.zgemm_df(x[0], p[0].T, conj_a=True, conj_b=True)):
        lazy = f(psi.conj(), proj.conj(), field.conj())
        assert torch.equal(lazy, f(*(t.conj().resolve_conj() for t in (psi, proj, field))))
    neg = torch.randn(plan.N, dtype=torch.complex128, device="cuda").conj().imag        # a pending sign
    assert neg.is_neg()
    assert torch.equal(ops.hpsi(plan, psi, kin, neg), ops.hpsi(plan, psi, kin, neg.resolve_neg()))


def test_incoming_gradients():
    plan, psi, _, field, _ = case()
    x = psi[0].clone().requires_grad_(True)
    y = autograd.psi_to_real(plan, x, 2.0)
    lazy, = torch.autograd.grad(y, x, field.conj(), retain_graph=True)
    plain, = torch.autograd.grad(y, x, field.conj().resolve_conj())
    assert torch.equal(lazy, plain)
