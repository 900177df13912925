"""Size queries of empty problems (no bands, k points, atoms or projectors) return a size."""

from __future__ import annotations

import pytest


@pytest.mark.parametrize("dt", [0, 1])
def test_size_queries_of_empty_problems(dt):
    from addft_gb300._lib import LIB
    for nk, nb, nG, nat, nh in ((1, 0, 100, 2, 4), (0, 3, 100, 2, 4), (1, 3, 100, 0, 4), (1, 3, 100, 2, 0), (0, 0, 1, 0, 0)):
        assert LIB.addft_nonlocal_gradients_work_bytes(dt, nk, nb, nG, nat, nh) >= 0
    assert LIB.addft_zgemm_df_work_bytes(0, 5, 5) == 0 and LIB.addft_zgemm_df_work_bytes(5, 5, 0) == 0
    full = LIB.addft_nonlocal_gradients_work_bytes(dt, 1, 3, 100, 2, 4)
    assert full >= 2 * 8 * 100 * (16 if dt else 8)
