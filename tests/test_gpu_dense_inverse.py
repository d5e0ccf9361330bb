"""The blocked sweep behind the V-cycle's dense bottom at sizes around its blocks of 64 rows and its update
tiles of 128 x 64: one block, an odd and an even number of blocks, a last block of one row's padding or
almost all of it. Needs a B200.

The inverse is checked against the level's operator: |A inv - I| stays within n eps times the condition
number (at most 1e4 for these levels), 1e-9 asked, and it is symmetric to the last bit.
"""

from __future__ import annotations

import numpy as np
import pytest

from cunibs_b200 import _native
from cunibs_b200.synthetic import sphere_head
from test_gpu_dense_bottom import _csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing, min_rows, max_rows", [(26.0, 4, 64), (15.0, 64, 128), (12.5, 100, 256),
                                                        (9.0, 200, 512), (6.0, 600, 1400), (4.5, 1600, 2600)])
def test_inverse_of_the_bottom_operator(spacing, min_rows, max_rows):
    m = sphere_head(spacing, 90.0, jitter_mm=0.2, seed=1)
    prm = _native.default_params()
    prm.min_coarse_rows = 4
    ctx = _native.Context(m.nodes_mm, m.tet_nodes, m.tet_tags, m.skin_tris, prm)
    try:
        n = ctx.bottom_rows
        assert min_rows <= n <= max_rows
        inv = ctx.array("bottom_inv").reshape(n, n)
        np.testing.assert_array_equal(inv, inv.T)
        prefix, level = ("a", ctx.vcycle_levels) if ctx.vcycle_levels < ctx.n_levels else ("coarse", -1)
        A = _csr(ctx, prefix, level)
        assert np.abs(A @ inv - np.eye(n)).max() <= 1e-9
    finally:
        ctx.close()
