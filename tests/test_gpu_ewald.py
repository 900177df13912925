"""Ewald sums beyond the small cells: more atoms than a warp has lanes (other rows of threads), and more
pairs times translations than 32 bits count."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if torch.cuda.is_available():
    from addft_gb300 import ops
    from oracle import pw


@pytest.mark.parametrize("nat", [31, 32, 33, 65, 97])
def test_more_atoms_than_a_warp(nat):
    rng = np.random.default_rng(nat)
    lat = np.array([[9.0, 0.4, 0.0], [0.0, 8.0, 0.7], [0.3, 0.0, 10.0]])
    frac, z = rng.uniform(0, 1, (nat, 3)), rng.uniform(0.5, 4.0, nat)
    out = ops.ewald(lat, frac @ lat, z, nmax=2).cpu().numpy()
    e = pw.ewald_energy(lat, frac, z, nmax=2)
    dR, deps = pw.ewald_gradients(lat, frac, z, nmax=2)
    # random positions bring pairs of 0.1 Bohr: sums of 1e4 terms, against the largest
    assert abs(out[0] - e) < 1e-11 * (abs(e) + 1)
    assert np.max(np.abs(out[1:1 + 3 * nat].reshape(nat, 3) - dR)) < 1e-11 * (np.max(np.abs(dR)) + 1)
    assert np.max(np.abs(out[1 + 3 * nat:].reshape(3, 3) - deps)) < 1e-11 * (np.max(np.abs(deps)) + 1)


def test_pairs_times_translations_beyond_32_bits():
    """16 atoms and 1.4e8 translations each: a width that reaches 258 cells gives the sum of the usual width.
    The terms cancel from 1e5 (pi z^2 / 2 omega eta^2), in sums of 1e8 roundings of a part of it per thread block."""
    lat, nat = np.eye(3) * 4.0, 16
    rng = np.random.default_rng(2)
    frac, z = rng.uniform(0, 1, (nat, 3)), rng.uniform(0.5, 3.0, nat)
    usual = ops.ewald(lat, frac @ lat, z, eta=0.9, nmax=8).cpu().numpy()
    eta, nmax = 0.0097, 262
    far = ops.ewald(lat, frac @ lat, z, eta=eta, nmax=nmax).cpu().numpy()
    assert nat * (2 * int(10.0 / eta / 4.0) + 1) ** 3 > 2 ** 31
    assert np.max(np.abs(far - usual)) < 1e-7 * (np.max(np.abs(usual)) + 1)
