"""Block PCG at sizes around its tiles of 64 rows and at every block width, through the C ABI. Needs a B200.

Each solution satisfies its own stopping test against the exported operator (||b - A x|| <= tol ||b||, twice
that asked: the loop tests a recurrence, 1e-9 against FP64's rounding of the true residual), and a column is
bitwise the one it has in any other block width.
"""

from __future__ import annotations

import numpy as np
import pytest

from cunibs_b200 import _native
from cunibs_b200.synthetic import sphere_head
from test_gpu_dense_bottom import _csr

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("spacing", [24.0, 17.0, 11.0, 7.0, 5.0])
@pytest.mark.parametrize("precision", [_native.PREC_SPLIT, _native.PREC_PLAIN_FP64])
def test_solutions_and_widths(spacing, precision):
    m = sphere_head(spacing, 90.0, jitter_mm=0.2, seed=2)
    prm = _native.default_params()
    prm.min_coarse_rows = 4
    ctx = _native.Context(m.nodes_mm, m.tet_nodes, m.tet_tags, m.skin_tris, prm)
    try:
        A = _csr(ctx, "a", 0)
        n = A.shape[0]
        b = np.random.default_rng(4).standard_normal((n, 16))
        x16, it, rel = ctx.solve(b, 16, 16, precision=precision, tolerance=TOL)
        assert (rel <= TOL).all() and (it > 0).all()
        r = b - A @ x16
        assert (np.linalg.norm(r, axis=0) <= 2 * TOL * np.linalg.norm(b, axis=0)).all()
        for k, width in ((1, 1), (2, 2), (3, 4), (4, 4), (7, 8), (8, 8)):
            cols = np.empty((n, width))
            cols[:, :k] = b[:, 3:3 + k]
            cols[:, k:] = b[:, 2 + k:3 + k]  # a partial block repeats its last column
            xk, itk, _ = ctx.solve(cols, k, width, precision=precision, tolerance=TOL)
            np.testing.assert_array_equal(xk[:, :k], x16[:, 3:3 + k])
            np.testing.assert_array_equal(itk[:k], it[3:3 + k])
        # A warm start from the solution stops at once and keeps it.
        xw, itw, _ = ctx.solve(b, 16, 16, precision=precision, tolerance=1e-8, x0=x16)
        assert (itw <= 1).all() and np.linalg.norm(xw - x16) <= 1e-8 * np.linalg.norm(x16)
    finally:
        ctx.close()


@pytest.mark.parametrize("spacing", [4.2, 3.8, 3.0])
@pytest.mark.parametrize("precision", [_native.PREC_SPLIT, _native.PREC_PLAIN_FP64])
def test_groups_of_tiles_leave_the_sums_as_they_are(spacing, precision):
    """More than 592 tiles of 64 rows: blocks of one, two and four columns hold several groups, 16 columns one."""
    m = sphere_head(spacing, 90.0, jitter_mm=0.2, seed=2)
    ctx = _native.Context(m.nodes_mm, m.tet_nodes, m.tet_tags, m.skin_tris, _native.default_params())
    try:
        b = np.random.default_rng(5).standard_normal((ctx.array("a_ptr", 0).shape[0] - 1, 16))
        x16, it, rel = ctx.solve(b, 16, 16, precision=precision, tolerance=TOL)
        assert (rel <= TOL).all()
        for k in (1, 2, 4):
            xk, itk, _ = ctx.solve(np.ascontiguousarray(b[:, :k]), k, k, precision=precision, tolerance=TOL)
            np.testing.assert_array_equal(xk, x16[:, :k])
            np.testing.assert_array_equal(itk, it[:k])
    finally:
        ctx.close()


@pytest.mark.parametrize("spacing", [11.0, 5.2, 4.2])
@pytest.mark.parametrize("precision", [_native.PREC_SPLIT, _native.PREC_PLAIN_FP64])
def test_launch_modes_give_the_same_bits(spacing, precision, monkeypatch):
    """Programmatic launches on, off and by the rule (on up to 256 rows and columns an SM: 2k rows at 16
    columns, 21k at one; off at 21k and 45k at two)."""
    m = sphere_head(spacing, 90.0, jitter_mm=0.2, seed=2)
    got = {}
    for mode in ("0", "1", None):
        if mode is None:
            monkeypatch.delenv("CUNIBS_PROGRAMMATIC_LAUNCH", raising=False)
        else:
            monkeypatch.setenv("CUNIBS_PROGRAMMATIC_LAUNCH", mode)
        ctx = _native.Context(m.nodes_mm, m.tet_nodes, m.tet_tags, m.skin_tris, _native.default_params())
        try:
            b = np.random.default_rng(6).standard_normal((ctx.array("a_ptr", 0).shape[0] - 1, 16))
            got[mode] = [ctx.solve(np.ascontiguousarray(b[:, :k]), k, k, precision=precision, tolerance=TOL)[:2]
                         for k in (1, 2, 16)]
        finally:
            ctx.close()
    for mode in ("1", None):
        for (x, it), (x0, it0) in zip(got[mode], got["0"]):
            np.testing.assert_array_equal(x, x0)
            np.testing.assert_array_equal(it, it0)
