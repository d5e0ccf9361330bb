"""The reciprocity field's kernel at grids around its tiles of 512 points and node counts around its stages of
128 nodes and runs of 1024, one to three directions, against the sum in FP64. Needs a B200.

Each operation rounds in FP32 (u = 2^-24): the difference g - r is off by u (|g - c| + |r - c|) from the tile's
centre c, which changes 1/|g - r|^3 by three times that over |g - r|, and the products and the sums over
a stage's nodes add their own few u: 16 u (|g - r| + 2 L) |W| / |g - r|^3 a pair, L half the grid's diagonal.
"""

from __future__ import annotations

import time

import numpy as np
import pytest
import torch

from cunibs_b200 import Subject, adm
from cunibs_b200.synthetic import sphere_head

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[30.0, 14.0, 7.0])
def adjoints(request):
    subj = Subject(sphere_head(request.param, 90.0, jitter_mm=0.2, seed=4), tolerance=1e-9)
    focus = [3.0, 2.0, 60.0]
    yield [adm.solve_adjoint(subj, adm.resolve_target(subj, adm.Target(focus, d, radius_mm=20.0)))
           for d in ((0.0, 1.0, 0.0), None)]
    subj.free()


def _check(adj, origin, sp, shape):
    grid = adm.Grid(origin_m=origin * 1e-3, spacing_m=sp * 1e-3, shape=shape)
    ijk = np.stack(np.meshgrid(*(np.arange(n) for n in shape), indexing="ij"), axis=-1).reshape(-1, 3)
    pts = (origin + ijk * sp) * 1e-3
    half = 0.5 * np.linalg.norm((np.array(shape) - 1) * sp) * 1e-3
    q = adm.sample_qfield(adj, grid).q
    w_all, nodes = adj.node_weights, adj.subject.context.array("nodes_mm").reshape(-1, 3) * 1e-3
    assert q.shape == (len(w_all), *shape, 3)
    for d, w in enumerate(w_all):
        got = q[d].reshape(-1, 3).astype(np.float64)
        for i in range(0, len(pts), 256):
            diff = pts[i:i + 256, None] - nodes[None]
            r = np.linalg.norm(diff, axis=2)
            want = 1e-7 * (np.cross(w[None], diff) / r[..., None] ** 3).sum(1)
            bound = 16 * 2.0**-24 * 1e-7 * ((r + 2 * half) * np.linalg.norm(w, axis=1) / r**3).sum(1)
            assert (np.abs(got[i:i + 256] - want).max(1) <= bound).all()


@pytest.mark.parametrize("gap_mm", [0.05, 0.6, 2.0])
def test_a_point_beside_a_node(adjoints, gap_mm):
    """Nodes nearer than an eighth of the tile's half diagonal take their own cross product."""
    for adj in adjoints:
        node = adj.subject.context.array("nodes_mm").reshape(-1, 3)[-1]
        _check(adj, node - [9.0, 12.0, 6.0] + [gap_mm, 0.0, 0.0], np.full(3, 3.0), (8, 8, 8))


@pytest.mark.parametrize("shape, spacing", [((1, 1, 1), (3, 3, 3)), ((1, 1, 40), (3, 3, 3)), ((8, 8, 8), (3, 3, 3)),
                                           ((9, 8, 8), (2, 3, 4)), ((33, 2, 1), (5, 1, 1)), ((23, 17, 11), (3, 3, 3))])
def test_field_against_the_sum_in_64_bits(adjoints, shape, spacing):
    for adj in adjoints:
        _check(adj, np.array([-21.0, -19.5, 80.3]), np.array(spacing, np.float64), shape)


def test_sampling_is_over_when_the_call_returns(adjoints):
    """A failure of the field's kernels is this call's, and its time too: next to nothing is left on the device."""
    grid = adm.Grid(origin_m=np.array([-0.09, -0.09, 0.0]), spacing_m=np.full(3, 3e-3), shape=(60, 60, 60))
    left = []
    for _ in range(6):
        torch.cuda.synchronize()
        times = [time.perf_counter()]
        adm.sample_qfield(adjoints[1], grid)
        times.append(time.perf_counter())
        torch.cuda.synchronize()
        times.append(time.perf_counter())
        left.append((times[2] - times[1]) / (times[2] - times[0]))
    assert np.median(left[1:]) < 0.2
