"""The conductivity study's component tables, built in one pass for all tissues. Needs a B200.

With one, some and all ten perturbed tissues (two to eleven tables), ragged node counts and one or two
placements, a draw's field is that of a context assembled with the draw's own table: both are solved to
1e-10 and stored in FP32 (6e-8 an entry), so 1e-6 in relative L2 leaves room for the operators' conditioning.
"""

from __future__ import annotations

import numpy as np
import pytest

from cunibs_b200 import Placement, Subject
from cunibs_b200.synthetic import figure8_coil, sphere_head
from cunibs_b200.uq import nominal_sigma_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tags,n_sites,spacing", [(1, 1, 9.0), (4, 2, 8.0), (10, 1, 7.5), (10, 3, 9.0)])
def test_a_draw_is_its_own_tables_solve(n_tags, n_sites, spacing):
    mesh = sphere_head(spacing, 90.0, jitter_mm=0.2, seed=5)
    mesh.tet_tags[:] = np.arange(len(mesh.tet_tags)) % 10 + 1  # every tissue, in every row
    coil = figure8_coil(32)
    c = np.array([[0.0, 0.0, 90.0], [20.0, 0.0, 87.7], [0.0, -20.0, 87.7]])[:n_sites]
    h = c + [0.0, 50.0, 0.0]
    d = [4.0] * n_sites
    nominal = nominal_sigma_table()
    tags = tuple(range(1, n_tags + 1))
    draw = nominal[list(tags)] * np.exp(0.2 * np.random.default_rng(6).standard_normal(n_tags))
    subj = Subject(mesh, tolerance=1e-10)
    ref = Subject(mesh, tolerance=1e-10)
    try:
        subj.context.sigma_begin(coil, c, h, d, 1e6, nominal, tags, magnitude=True, recovery="raw")
        got = subj.context.sigma_draw(draw)["magnE"].astype(np.float64)
        subj.context.sigma_end()
        table = nominal.copy()
        table[list(tags)] = draw
        ref.context.set_conductivity(table)
        for i in range(n_sites):
            want = ref.simulate(coil, Placement(c[i], h[i]), magnitude=True, recovery="raw").magnE.astype(np.float64)
            assert np.linalg.norm(got[i] - want) <= 1e-6 * np.linalg.norm(want)
    finally:
        subj.free()
        ref.free()
