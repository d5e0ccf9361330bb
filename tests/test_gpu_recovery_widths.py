"""The harmonic recovery at every block width against the oracle's mirror of its arithmetic, bit for bit: one
column or pairs a thread, few threads (eight patch entries in flight) or many (two). Needs a B200."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from cunibs_b200 import _native
from cunibs_b200.synthetic import sphere_head
from oracle import Oracle

pytestmark = pytest.mark.gpu


# Widths on the near side of the limit of 2048 threads an SM, and beyond it.
@pytest.mark.parametrize("spacing, few, many", [(12.0, (1, 2, 3, 8, 16), ()), (5.0, (1, 8), (9, 16))])
def test_harmonic_apply_bit_exact(spacing, few, many):
    mesh = sphere_head(spacing, 90.0, jitter_mm=0.2, seed=5)
    orc = Oracle(mesh)
    ctx = _native.Context(mesh.nodes_mm, mesh.tet_nodes, mesh.tet_tags, mesh.skin_tris)
    try:
        rng = np.random.default_rng(8)
        limit = 2048 * torch.cuda.get_device_properties(0).multi_processor_count
        for k in few + many:
            threads = ctx.recovery("harmonic")["n_slots"] * (k if k % 2 else k // 2)
            assert (threads < limit) == (k in few)
            v = rng.standard_normal((k, ctx.n_nodes))
            v[:, ctx.ground_node] = 0.0
            dadt = rng.standard_normal((k, ctx.n_nodes, 3)).astype(np.float32)
            got = ctx.recover("harmonic", v=v, dadt_nodes=dadt)
            want = orc.recovery_apply("harmonic", v=v, dadt_nodes=dadt)
            for a, b, name in zip(got, want, ("E_slots", "E", "magnE")):
                np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32), err_msg=f"{name} k={k}")
    finally:
        ctx.close()
