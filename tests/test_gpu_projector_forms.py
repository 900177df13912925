"""The two forms of the projectors, a thread per (projector, G) and phase tables, around where the tables start: the
same tables k point by k point (few projectors) and all at once."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if torch.cuda.is_available():
    from addft_gb300 import ops
    from addft_gb300.psp import synthetic


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("box,nat,nk", [((36, 36, 36), 4, 8),      # tables of e12
                                        ((27, 40, 36), 7, 5), ((18, 18, 18), 33, 8),   # few G per table entry: never tables
                                        ((128, 120, 9), 8, 8),     # two-axis products of the tables do not fit
                                        ((36, 36, 36), 1, 30)])    # one atom: its rows hold the form factors
def test_forms_agree(box, nat, nk, dtype):
    r = [int(0.25 * n) for n in box]
    m = np.stack(np.meshgrid(*(np.arange(-k, k + 1) for k in r), indexing="ij"), -1).reshape(-1, 3)
    m = m[np.sum((m / (np.asarray(box) * 0.25)) ** 2, axis=1) <= 1.0].astype(np.int32)
    plan = ops.Plan(box, m)
    lat = np.diag(np.asarray(box) / 3.0) + 0.3
    B = 2 * np.pi * np.linalg.inv(lat).T
    rng = np.random.default_rng(nat)
    pos, kpts = rng.uniform(-1, 1, (nat, 3)) @ lat, rng.uniform(-0.3, 0.3, (nk, 3))
    om, dt = abs(float(np.linalg.det(lat))), getattr(torch, dtype)
    whole = ops.projectors(plan, B, om, kpts, pos, synthetic(), dtype=dt)
    if plan.nG >= 2000:
        assert nk * nat * synthetic().nh * plan.nG >= 3e5 > nat * synthetic().nh * plan.nG
    one = torch.cat([ops.projectors(plan, B, om, k[None], pos, synthetic(), dtype=dt) for k in kpts])
    # |(k + G) . R| stays below 1e3: its rounding moves a phase by 2e-13 at most
    tol = (4e-13 if dtype == "complex128" else 1.2e-7) * float(whole.abs().max())
    assert bool(((whole - one).abs() <= tol).all())
