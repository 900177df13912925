"""A tensor-core kernel whose bounded wait runs out returns without results: the calls that hand results to
the user say so.  The status is a fake here; no wait is made to run out."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import FRAC_DISTORTED, LATTICE, gpu_available


class _Status:
    """The library with another answer to addft_tc05_status."""

    def __init__(self, lib, bits):
        self._lib, self._bits, self.looks = lib, bits, 0

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def addft_tc05_status(self):
        self.looks += 1
        return self._bits


def test_status_bits_raise(monkeypatch):
    from addft_gb300 import ops
    from addft_gb300._lib import AddftError
    monkeypatch.setattr(ops, "LIB", _Status(ops.LIB, 0))
    ops.raise_on_device_errors()
    for bits in (1, 0xffffffff):                     # a wait ran out; the status itself could not be read
        monkeypatch.setattr(ops, "LIB", _Status(ops.LIB, bits))
        with pytest.raises(AddftError, match="gave up waiting"):
            ops.raise_on_device_errors()


@pytest.mark.gpu
def test_calls_of_a_user_look_at_the_status(monkeypatch):
    if not gpu_available():
        pytest.skip("needs a CUDA device")
    import addft_gb300 as ad
    from addft_gb300 import observables as obs
    from addft_gb300 import ops
    from addft_gb300._lib import AddftError
    from addft_gb300.response import implicit_grad
    s = ad.setup(LATTICE, FRAC_DISTORTED, ecut=2.0, nband=2, density_factor=4.0)
    st = ad.scf(s)
    g = np.ones(s.static.basis.nfft)
    import torch
    gt = torch.as_tensor(g, device="cuda")
    calls = {"scf": lambda: ad.scf(s), "energy": lambda: ad.energy(s, st),
             "terms": lambda: obs.energy_terms(s.geo, s.static, st),
             "gradients": lambda: obs.envelope_gradients(s.geo, s.static, st),
             "implicit": lambda: implicit_grad(s.geo, s.static, st, gt)}
    for f in calls.values():
        f()                                          # and with the true status they pass
    for name, f in calls.items():
        with monkeypatch.context() as m:
            m.setattr(ops, "LIB", _Status(ops.LIB, 1))
            with pytest.raises(AddftError, match="gave up waiting"):
                f()
            assert ops.LIB.looks == 1, name
