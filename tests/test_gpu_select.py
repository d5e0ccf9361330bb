"""Element selection on the GPU (cunibs_context_select, adm.resolve_target) against NumPy on the exported
mesh: the same elements in the same order, the same weights and barycentre. Needs a B200."""

from __future__ import annotations

import numpy as np
import pytest

from cunibs_b200 import Subject, adm, metrics
from cunibs_b200.synthetic import EIGHT_SHELLS, sphere_head

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0.0, 0.2])
def subject(request):
    # Without jitter the lattice is symmetric: several elements are equally near to its points of symmetry.
    with Subject(sphere_head(9.0, 90.0, EIGHT_SHELLS, jitter_mm=request.param, seed=4)) as s:
        yield s


def _expected(ctx, target):
    bary, tags, vols = ctx.array("bary").reshape(-1, 3), ctx.array("tet_tags"), ctx.array("vols")
    ids = np.flatnonzero(metrics.region_mask(tags, target.region)).astype(np.int32)
    d2 = ((bary[ids] - target.position_mm) ** 2).sum(1)
    if target.radius_mm <= 0.0:
        return ids[[int(np.argmin(d2))]], bary, vols
    within = d2 <= target.radius_mm ** 2
    return ids[within if within.any() else d2 == d2.min()], bary, vols


@pytest.mark.parametrize("region", ["gray_matter", "scalp", "all"])
@pytest.mark.parametrize("radius", [-1.0, 0.0, 1e-9, 4.0, 25.0, 500.0, float("inf")])
def test_selection_matches_numpy(subject, region, radius):
    rng = np.random.default_rng(2)
    for p in [np.zeros(3), np.array([0.0, 0.0, 62.0]), np.array([1e4, 0.0, 0.0]), *rng.uniform(-95.0, 95.0, (4, 3))]:
        target = adm.Target(p, region=region, radius_mm=radius)
        sel, bary, vols = _expected(subject.context, target)
        got = adm.resolve_target(subject, target)
        assert got.elem_idx.dtype == np.int32
        np.testing.assert_array_equal(got.elem_idx, sel)
        w = vols[sel] / vols[sel].sum()
        np.testing.assert_array_equal(got.weights, w)
        np.testing.assert_array_equal(got.barycenter_mm, w @ bary[sel])


def test_absent_tissue_is_refused(subject):
    with pytest.raises(ValueError, match="contains no elements"):
        adm.resolve_target(subject, adm.Target([0.0, 0.0, 0.0], region="muscle"))
