"""The work that users have this framework do, as cases that can be timed and compared.

A case is one call of a public entry point on a synthetic sphere head (a jittered Kuhn lattice of
radius 90 mm, five shells or the ten-tissue model) with a figure-8 coil of point dipoles:

* ``simulate``: one placement, ``Subject.simulate``;
* ``sweep``: many placements, ``Subject.iter_simulate``;
* ``device``: one block with its fields left on the GPU, ``fem.solve_placements_block``;
* ``guided``: blocks two deep from a learned initial guess, device buffers in and out;
* ``study``: a conductivity Monte Carlo, ``Subject.iter_simulate_conductivity_uq``;
* ``field``: adjoint solves and the reciprocity field on a grid, ``adm.solve_adjoint`` and ``sample_qfield``;
* ``optimize``: the coil search over scalp positions and rotations, ``adm.optimize``;
* ``open``: a new head, from its arrays to its first result.

``listed`` gives the named cases, ``draw`` more of the same ranges (lattice spacing 2.63 to 10 mm:
18 thousand to 1 million tetrahedra; 16 to 2048 dipoles a wing; 1 to 24 placements; every recovery
mode and precision). Iteration counts and residuals are not among the outputs: they say how a result
was reached. The results are the fields, the potential and the gray-matter metrics.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from cunibs_b200 import Coil, ConductivityUQConfig, HeadMesh, Placement, Subject, adm, fem
from cunibs_b200.synthetic import EIGHT_SHELLS, EYE_CAP, FIVE_SHELLS, MUSCLE_CAP, cap_placements, figure8_coil, sphere_head

RADIUS_MM = 90.0
JITTER_MM = 0.2
DIDT = 1e6
FOCUS_MM = (0.0, 0.0, 62.0)  # target of the reciprocity cases: cortex below the vertex


def listed() -> list[dict]:
    base = dict(tissues=5, wing=512, coil="flat", sites=1, recovery="harmonic", precision="split", tolerance=1e-6)
    head = dict(base, spacing_mm=2.63, tissues=10, wing=2048, tolerance=1e-8)  # 1.0M tetrahedra
    return [
        # The smallest call: one placement on a coarse head (85k tetrahedra), where launches and waits count.
        dict(base, name="simulate-coarse", kind="simulate", spacing_mm=6.0, wing=128, magnitude=True),
        # One placement on an ordinary head (0.68M tetrahedra) with the default options.
        dict(base, name="simulate-head", kind="simulate", spacing_mm=3.0),
        # The headline workload's sweep: 24 placements on the 1M-tetrahedron ten-tissue head, metrics only.
        dict(head, name="sweep-1M", kind="sweep", sites=24),
        # A ragged sweep (8 + 5 placements) of a bent coil that keeps its fields on the host.
        dict(base, name="sweep-ragged", kind="sweep", spacing_mm=4.0, wing=200, coil="bent", sites=13,
             recovery="spr_tissue", magnitude=True, nodal=True),
        # The plain method: FP64 throughout, the raw field, tolerance 1e-10; three placements in a block of four.
        dict(base, name="plain-fp64", kind="sweep", spacing_mm=3.0, sites=3, recovery="raw", precision="plain",
             tolerance=1e-10, vectors=True, potential=True),
        # FP64 refinement around an FP32 solve, nodal averages over all tissues.
        dict(base, name="sweep-mixed", kind="sweep", spacing_mm=4.0, sites=16, recovery="spr_global",
             precision="mixed", tolerance=1e-8),
        # A block of 8 on the 1M head with every field left on the GPU for the caller's own post-processing.
        dict(head, name="device-1M", kind="device", sites=8, nodal=True, potential=True),
        # Sweeping with the learned initial guess, the headline arm of the benchmark: 4 blocks of 8.
        dict(head, name="guided-1M", kind="guided", sites=32),
        # Conductivity uncertainty: 4 placements, 12 draws of all ten tissues.
        dict(head, name="study", kind="study", spacing_mm=3.0, wing=512, sites=4, draws=12, tolerance=1e-8),
        # Reciprocity of a magnitude target: three adjoint solves and the field on a 3 mm grid over the vertex.
        dict(head, name="field-1M", kind="field", reach_mm=110, tolerance=1e-9),
        # Planning a session on an ordinary head: 40 scalp positions, one field direction.
        dict(base, name="optimize", kind="optimize", spacing_mm=4.0, sites=40, tolerance=1e-9),
        # A new subject: set-up of a 0.68M-tetrahedron head and its first result.
        dict(base, name="open-head", kind="open", spacing_mm=3.0),
    ]


def draw(rng) -> dict:
    kind = rng.choice(["simulate", "sweep", "sweep", "device", "guided", "study", "field", "optimize", "open"])
    case = dict(
        kind=kind,
        spacing_mm=round(math.exp(rng.uniform(math.log(2.63), math.log(10.0))), 3),
        tissues=rng.choice([5, 10]),
        wing=int(math.exp(rng.uniform(math.log(16), math.log(2048)))),
        coil=rng.choice(["flat", "flat", "bent"]),
        sites=1,
        recovery="harmonic",
        precision="split",
        tolerance=rng.choice([1e-6, 1e-7, 1e-8]),
    )
    if kind in ("simulate", "open"):
        case.update(recovery=rng.choice(fem.RECOVERY_MODES), magnitude=rng.random() < 0.5)
    elif kind == "sweep":
        case.update(sites=rng.randint(1, 24), recovery=rng.choice(fem.RECOVERY_MODES),
                    precision=rng.choice(["split", "split", "plain", "mixed"]), potential=rng.random() < 0.3)
    elif kind == "device":
        case.update(sites=rng.randint(1, 8), recovery=rng.choice(fem.RECOVERY_MODES), potential=rng.random() < 0.5)
    elif kind == "guided":
        case.update(sites=8 * rng.randint(1, 4), tolerance=1e-8)
    elif kind == "study":
        case.update(sites=rng.randint(1, 4), draws=rng.randint(2, 12), recovery=rng.choice(["raw", "harmonic"]))
    elif kind == "field":
        case.update(reach_mm=rng.randint(60, 110), tolerance=1e-9, directed=rng.random() < 0.5)
    else:
        case.update(sites=rng.randint(2, 40), tolerance=1e-9)
    return case


# --- inputs ---------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=24)
def _lattice(spacing_mm: float, tissues: int) -> HeadMesh:
    shells, caps = (FIVE_SHELLS, ()) if tissues == 5 else (EIGHT_SHELLS, (EYE_CAP, MUSCLE_CAP))
    return sphere_head(spacing_mm, RADIUS_MM, shells=shells, caps=caps)


def _head(case: dict, seed: int) -> HeadMesh:
    """The case's lattice with this seed's node jitter."""
    base = _lattice(case["spacing_mm"], case["tissues"])
    jitter = np.random.default_rng(seed).uniform(-JITTER_MM, JITTER_MM, base.nodes_mm.shape)
    return HeadMesh(base.nodes_mm + jitter, base.tet_nodes, base.tet_tags, base.skin_tris)


def _coil(case: dict) -> Coil:
    """A figure-8 coil; "bent" tilts each wing 10 degrees towards the head (moments off the coil axis)."""
    flat = figure8_coil(case["wing"])
    if case["coil"] == "flat":
        return flat
    x, y, z = flat.positions_m.T
    mz = flat.moments[:, 2]
    c, s, side = math.cos(math.radians(10)), math.sin(math.radians(10)), np.sign(x)
    return Coil(positions_m=np.stack([x * c, y, z + np.abs(x) * s], 1),
                moments=np.stack([-side * mz * s, np.zeros_like(mz), mz * c], 1), name="bent figure8")


def _sites(case: dict, seed: int) -> list[Placement]:
    rng = np.random.default_rng(seed + 1)
    poses = cap_placements(RADIUS_MM, case["sites"], 40.0, seed=seed)
    if case["kind"] == "optimize":  # candidate positions over the target, within about 30 mm
        u = rng.uniform(-1.0, 1.0, (case["sites"], 2)) * 30.0
        c = np.concatenate([u, np.full((case["sites"], 1), RADIUS_MM)], axis=1)
        c *= RADIUS_MM / np.linalg.norm(c, axis=1, keepdims=True)
        poses = [(p, p + np.array([0.0, 50.0, 0.0])) for p in c]
    distance = 4.0 if case["kind"] in ("guided", "optimize") else None
    return [Placement(c, h, rng.uniform(2.0, 8.0) if distance is None else distance) for c, h in poses]


def _target(case: dict) -> adm.Target:
    one = case["kind"] == "optimize" or case.get("directed", False)
    return adm.Target(FOCUS_MM, direction=(0.0, 1.0, 0.0) if one else None, radius_mm=5.0)


def _grid(case: dict, seed: int) -> adm.Grid:
    """A 3 mm grid about the vertex that holds a coil at any rotation on positions within 30 mm of it:
    ``reach_mm`` to each side, half as much above as below."""
    side = int(2 * case["reach_mm"] / 3) + 1
    low = np.array([-case["reach_mm"], -case["reach_mm"], RADIUS_MM - case["reach_mm"]])
    shift = np.random.default_rng(seed).uniform(-1.0, 1.0, 3)
    return adm.Grid(origin_m=(low + shift) * 1e-3, spacing_m=np.full(3, 3e-3), shape=(side, side, 3 * side // 4))


def prepare(case: dict, seed: int) -> dict:
    mesh, coil, sites = _head(case, seed), _coil(case), _sites(case, seed)
    state = dict(case=case, coil=coil, sites=sites, seed=seed)
    if case["kind"] == "open":
        return dict(state, mesh=mesh)
    subject = Subject(mesh, tolerance=case["tolerance"], precision=case["precision"])
    ctx = subject.context
    state["subject"] = subject
    if case["kind"] == "field":
        state["grid"] = _grid(case, seed)
    if case["kind"] == "study":
        state["config"] = ConductivityUQConfig(n_samples=case["draws"], seed=seed)
    if case["kind"] == "guided":
        from cunibs_b200.warmstart import train_warm_start

        # A small training set (the benchmark takes 8192 solves), so that the inputs are made quickly.
        state["model"] = train_warm_start(ctx, coil, n_train=192, rank=64, epochs=60, seed=3)
        f64 = dict(dtype=torch.float64, device="cuda")
        state["pos"], state["mom"] = torch.tensor(coil.positions_m, **f64), torch.tensor(coil.moments, **f64)
        blocks = [sites[i:i + 8] for i in range(0, len(sites), 8)]
        state["blocks"] = [
            dict(centers=torch.tensor(np.stack([s.center_mm for s in b]), **f64),
                 handles=torch.tensor(np.stack([s.handle_mm for s in b]), **f64),
                 dists=torch.tensor([s.distance_mm for s in b], **f64),
                 out=dict(transforms=torch.empty(len(b), 16, **f64), summary=torch.empty(len(b), 16, **f64),
                          magnE=torch.empty(len(b), ctx.n_tets, dtype=torch.float32, device="cuda"),
                          v=torch.empty(len(b), ctx.n_nodes, **f64)))
            for b in blocks]
        torch.cuda.synchronize()
    return state


# --- one pass -------------------------------------------------------------------------------------


def _metrics(summary) -> np.ndarray:
    """A result's gray-matter metrics as one row."""
    return np.concatenate([[summary["peak_magnE"]], summary["peak_location_mm"], summary["center_of_gravity_mm"],
                           [summary["region_volume_m3"]], list(summary["focality_m3"].values()),
                           list(summary["distribution"].values())])


def _outputs(results) -> dict:
    out = dict(metrics=np.stack([_metrics(r.summary) for r in results]),
               transform=np.stack([r.transform for r in results]))
    for name in ("magnE", "E", "v", "E_slots"):
        if getattr(results[0], name) is not None:
            out[name] = [getattr(r, name) for r in results]
    return out


def _retain(case: dict) -> dict:
    return {k: True for k in ("magnitude", "vectors", "potential", "nodal") if case.get(k)}


def run(state: dict):
    case, coil, sites = state["case"], state["coil"], state["sites"]
    kind = case["kind"]
    if kind == "open":
        with Subject(state["mesh"], tolerance=case["tolerance"], precision=case["precision"]) as subject:
            return _outputs([subject.simulate(coil, sites[0], DIDT, recovery=case["recovery"], **_retain(case))])
    subject = state["subject"]
    if kind == "simulate":
        return _outputs([subject.simulate(coil, sites[0], DIDT, recovery=case["recovery"], **_retain(case))])
    if kind == "sweep":
        return _outputs(list(subject.iter_simulate(coil, sites, DIDT, recovery=case["recovery"], **_retain(case))))
    if kind == "device":
        found = fem.solve_placements_block(
            subject.context, coil.positions_m, coil.moments, [(s.center_mm, s.handle_mm, s.distance_mm) for s in sites],
            DIDT, recovery=case["recovery"], nodal=bool(case.get("nodal")) and case["recovery"] != "raw",
            potential=bool(case.get("potential")))
        return [{k: r[k] for k in ("transform", "E", "magnE", "v", "E_slots") if k in r} for r in found]
    if kind == "guided":
        return _guided(state, subject.context, coil)
    if kind == "study":
        found = subject.iter_simulate_conductivity_uq(coil, sites, state["config"], DIDT, recovery=case["recovery"])
        return [dict(peak=r.peak_samples, focality=r.focality_samples, location=r.peak_location_samples) for r in found]
    if kind == "field":
        adjoint = adm.solve_adjoint(subject, adm.resolve_target(subject, _target(case)), tolerance=case["tolerance"])
        return dict(q=adm.sample_qfield(adjoint, state["grid"]).q)
    best = adm.optimize(subject, coil, _target(case), np.stack([s.center_mm for s in sites]), didt=DIDT)
    return dict(objective=best.center_objective, handles=best.center_handle_mm, contacts=best.centers_mm,
                best=best.best_E)


def _guided(state: dict, ctx, coil: Coil) -> list:
    """The blocks two deep, as ``iter_simulate`` runs them, with device buffers on both sides."""
    blocks = state["blocks"]

    def submit(b):
        return ctx.submit_block_device(state["pos"].data_ptr(), state["mom"].data_ptr(), coil.n_dipoles,
                                       b["centers"].data_ptr(), b["handles"].data_ptr(), b["dists"].data_ptr(),
                                       b["dists"].numel(), DIDT, tolerance=state["case"]["tolerance"],
                                       recovery="harmonic", warm_start=True)

    tickets = [submit(blocks[0])]
    for i, b in enumerate(blocks):
        if i + 1 < len(blocks):
            tickets.append(submit(blocks[i + 1]))
        ctx.finish_block_device(tickets[i], {k: t.data_ptr() for k, t in b["out"].items()})
    return [b["out"] for b in blocks]


# --- what a pass cannot do without, and how exact it is ----------------------------------------------


def _sizes(case: dict) -> tuple[float, float, float]:
    """(tetrahedra, nodes, stiffness entries) of the lattice, from its volume: 6 tetrahedra and one
    node a cell, 15 entries a row."""
    cells = 4.0 / 3.0 * math.pi * (RADIUS_MM / case["spacing_mm"]) ** 3
    return 6.0 * cells, 1.06 * cells, 15.9 * cells


def _grid_points(case: dict) -> float:
    if case["kind"] == "field":
        return float(_grid(case, 0).n_points)
    return (2 * (30 + 72 + 8) / 3.0 + 1) ** 2 * 60  # the optimiser's own grid: the positions and the coil's reach


def work(case: dict) -> dict:
    tets, nodes, nnz = _sizes(case)
    digits = -math.log10(case["tolerance"])
    kind = case["kind"]

    def solve(k: float, runs: float = 1.0) -> tuple[float, float]:
        # A Krylov method reads its FP64 operator and its residual, direction and solution once for
        # each digit that it gains, at best.
        return runs * digits * (12.0 * nnz + 3 * 8.0 * nodes * k), runs * digits * 2.0 * nnz * k

    def recover(k: float) -> tuple[float, float]:
        # Every element's corners and |E| once a placement, the operator once a block.
        return 16.0 * tets + 16.0 * nnz + (4.0 * tets + 20.0 * nodes) * k, 6.0 * nnz * k

    n = case["sites"]
    blocks = -(-n // 8)
    total = [0.0, 0.0]
    parts: list[tuple[float, float]] = []
    if kind in ("simulate", "sweep", "device", "guided", "open"):
        parts += [solve(n / blocks, blocks), tuple(blocks * v for v in recover(n / blocks))]
    if kind == "open":  # the mesh in, the operator, its hierarchy and the recovery weights out
        parts.append((40.0 * tets + 24.0 * nodes + 3 * 20.0 * nnz, 16 * 12.0 * tets))
    if kind == "study":
        parts += [solve(n, 1.0 + case["draws"]), tuple((1 + case["draws"]) * v for v in recover(n))]
    if kind in ("field", "optimize"):
        sets = 1 if kind == "optimize" or case.get("directed") else 3
        points = _grid_points(case)
        # Each (grid point, node) pair: a difference, a distance and its inverse cube (8 operations), then a
        # cross product added to each direction's field (9 multiply-adds).
        parts += [solve(sets), (24.0 * nodes * sets + 12.0 * points * sets, points * nodes * (8.0 + 18.0 * sets))]
    for b, f in parts:
        total[0] += b
        total[1] += f
    return dict(bytes=total[0], flops=total[1])


def tolerance(case: dict) -> dict:
    """About four times what was measured between two correct paths: the coil's dipole sum at every
    node against its table (5e-7 relative in the fields, 5e-6 at single values, FP32), and a solve
    against one to a thirtieth of its tolerance (0.6 of the tolerance relative, ten times that at single
    values)."""
    if case["kind"] == "field":
        # Grid points as near as a tenth of a millimetre to a node: FP32 coordinates leave 2e-5 against 64 bits.
        return dict(rel=8e-5, max=5e-3)
    if case["kind"] == "optimize":
        return dict(rel=1e-5, max=1e-4)  # FP32 sums of the sampled field, and an angle refined on them
    if case["kind"] == "study":
        return dict(rel=3e-4, max=1e-3)  # the focality volume counts whole elements (8e-5 and 3e-4 seen)
    solve = 2.5 * case["tolerance"]
    return dict(rel=2e-6 + solve, max=2e-5 + 20 * solve)


# --- the same results in 64 bits -------------------------------------------------------------------

_SIGMA = (0.0, 0.126, 0.275, 1.654, 0.010, 0.465, 0.5, 0.008, 0.025, 0.6, 0.16)
_CUDA = dict(dtype=torch.float64, device="cuda")


def _spread(v: np.ndarray) -> np.ndarray:
    """The low 21 bits of each value, three places apart."""
    out = np.zeros_like(v)
    for b in range(21):
        out |= ((v >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return out


class _Head64:
    """A head in result order (nodes by Morton key, elements by their lowest node), with its P1
    operator and grounded stiffness in 64 bits."""

    def __init__(self, mesh: HeadMesh) -> None:
        pts = np.asarray(mesh.nodes_mm, np.float64)
        lo = pts.min(0)
        span = np.maximum(pts.max(0) - lo, 1e-12)
        cell = ((pts - lo) / span * 2097151.0).astype(np.uint64)
        key = _spread(cell[:, 0]) | (_spread(cell[:, 1]) << np.uint64(1)) | (_spread(cell[:, 2]) << np.uint64(2))
        perm = np.argsort(key, kind="stable")
        inverse = np.empty_like(perm)
        inverse[perm] = np.arange(perm.size)
        tets = inverse[mesh.tet_nodes]
        order = np.argsort(tets.min(1), kind="stable")
        self.nodes, self.tets, self.tags = pts[perm], tets[order], np.asarray(mesh.tet_tags)[order]
        self.skin = inverse[mesh.skin_tris]
        self.n = pts.shape[0]
        self.ground = int(np.argmin(self.nodes[:, 2]))
        corner = torch.tensor(self.nodes * 1e-3, **_CUDA)[torch.tensor(self.tets, device="cuda")]  # (M, 4, 3)
        edges = corner[:, 1:] - corner[:, :1]
        self.vols = torch.linalg.det(edges).abs() / 6.0
        inner = torch.linalg.inv(edges).transpose(1, 2)  # rows: gradients of corners 1..3
        self.grad = torch.cat([-inner.sum(1, keepdim=True), inner], dim=1)
        self.bary = corner.mean(1) * 1e3
        self.dtets = torch.tensor(self.tets, device="cuda")
        self.dtags = torch.tensor(self.tags, device="cuda", dtype=torch.int64)

    def conductivity(self, table) -> torch.Tensor:
        return torch.tensor(np.asarray(table, np.float64), **_CUDA)[self.dtags]

    def stiffness(self, sigma: torch.Tensor):
        local = torch.einsum("eia,eja->eij", self.grad, self.grad) * (self.vols * sigma)[:, None, None]
        i = self.dtets[:, :, None].expand(-1, 4, 4).reshape(-1)
        j = self.dtets[:, None, :].expand(-1, 4, 4).reshape(-1)
        free = (i != self.ground) & (j != self.ground)
        at = torch.stack([torch.cat([i[free], torch.tensor([self.ground], device="cuda")]),
                          torch.cat([j[free], torch.tensor([self.ground], device="cuda")])])
        val = torch.cat([local.reshape(-1)[free], torch.ones(1, **_CUDA)])
        a = torch.sparse_coo_tensor(at, val, (self.n, self.n)).coalesce()
        diag = torch.zeros(self.n, **_CUDA).index_add_(0, a.indices()[0], a.values() * (a.indices()[0] == a.indices()[1]))
        return a.to_sparse_csr(), diag

    def solve(self, sigma: torch.Tensor, rhs: torch.Tensor) -> torch.Tensor:
        """K v = rhs (n, k) with v = 0 at the ground node, by conjugate gradients to 1e-13."""
        a, diag = self.stiffness(sigma)
        b = rhs.clone()
        b[self.ground] = 0.0
        x, r = torch.zeros_like(b), b.clone()
        z = r / diag[:, None]
        p, rz = z.clone(), (r * z).sum(0)
        limit = 1e-13 * b.norm(dim=0)
        for it in range(20000):
            ap = a @ p
            alpha = rz / (p * ap).sum(0).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * ap
            if it % 50 == 49 and bool((r.norm(dim=0) <= limit).all()):
                break
            z = r / diag[:, None]
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        return x

    def normals(self) -> np.ndarray:
        p, tri = self.nodes, self.skin
        face = np.cross(p[tri[:, 1]] - p[tri[:, 0]], p[tri[:, 2]] - p[tri[:, 0]])

        def spread(f):
            node = np.zeros_like(p)
            for c in range(3):
                np.add.at(node, tri[:, c], f)
            return node

        def unit(v):
            n = np.linalg.norm(v, axis=1, keepdims=True)
            return v / np.where(n > 0, n, 1.0)

        return unit(unit(spread(unit(spread(face)[tri].sum(1))))[tri].sum(1))

    def place(self, sites: list[Placement]) -> np.ndarray:
        """Coil-to-head affines (mm): the nearest skin point, the smoothed normal there, the handle in its plane."""
        tri = self.nodes[self.skin]
        normals = self.normals()
        out = np.zeros((len(sites), 4, 4))
        for k, s in enumerate(sites):
            q = _closest(s.center_mm, tri)
            at = int(np.argmin(((q - s.center_mm) ** 2).sum(1)))
            n, contact = normals[at], q[at]
            z = -n
            y = s.handle_mm - contact
            y = y / np.linalg.norm(y)
            y = y - z * (y @ z)
            y = y / np.linalg.norm(y)
            out[k, :3, 0], out[k, :3, 1], out[k, :3, 2] = np.cross(y, z), y, z
            out[k, :3, 3] = contact + s.distance_mm * n
            out[k, 3, 3] = 1.0
        return out

    def dadt(self, coil: Coil, frames: np.ndarray) -> torch.Tensor:
        """dA/dt at the nodes (k, n, 3)."""
        nodes = torch.tensor(self.nodes * 1e-3, **_CUDA)
        out = []
        for t in frames:
            s = torch.tensor(coil.positions_m @ t[:3, :3].T + t[:3, 3] * 1e-3, **_CUDA)
            m = torch.tensor(coil.moments @ t[:3, :3].T, **_CUDA)
            out.append(DIDT * 1e-7 * _dipole_field(nodes, s, m[None])[0])
        return torch.stack(out)

    def rhs(self, sigma: torch.Tensor, dadt: torch.Tensor) -> torch.Tensor:
        mean = dadt[:, self.dtets].mean(2)  # (k, M, 3)
        corner = -torch.einsum("kea,eia->eik", mean, self.grad) * (self.vols * sigma)[:, None, None]
        return torch.zeros(self.n, dadt.shape[0], **_CUDA).index_add_(0, self.dtets.reshape(-1),
                                                                    corner.reshape(-1, dadt.shape[0]))

    def fields(self, v: torch.Tensor, dadt: torch.Tensor) -> torch.Tensor:
        """E = -grad v - dA/dt per element (k, M, 3)."""
        return -torch.einsum("eik,eia->kea", v[self.dtets], self.grad) - dadt[:, self.dtets].mean(2)

    def metrics(self, e: torch.Tensor) -> np.ndarray:
        """The gray-matter metrics row of one placement's field."""
        gm = self.dtags == 2
        m, w, b = e.norm(dim=1)[gm].cpu().numpy(), self.vols[gm].cpu().numpy(), self.bary[gm].cpu().numpy()
        order = np.argsort(m, kind="stable")
        cum = np.cumsum(w[order])
        q = np.array([np.float32(p / 100) for p in (50.0, 95.0, 99.0, 99.9)], np.float64)
        pct = np.interp(q, (cum - 0.5 * w[order]) / cum[-1], m[order])
        mean = (w * m).sum() / w.sum()
        std = math.sqrt((w * (m - mean) ** 2).sum() / w.sum())
        foc = [w[m >= f * pct[-1]].sum() for f in (0.5, 0.75)]
        return np.concatenate([[m.max()], b[int(np.argmax(m))], ((w * m)[:, None] * b).sum(0) / (w * m).sum(), [w.sum()],
                               foc, [mean, std], pct])


def _dipole_field(points: torch.Tensor, sources: torch.Tensor, moments: torch.Tensor) -> torch.Tensor:
    """sum_j m_j x (r - s_j) / |r - s_j|^3 for every set of moments: (sets, n, 3). The cross product
    is split into products of one (points, sources) matrix with the moments and with m x s."""
    sets = moments.shape[0]
    center = points.mean(0)
    p, s = points - center, sources - center
    cols = torch.cat([moments.permute(1, 0, 2).reshape(-1, sets * 3),
                      torch.linalg.cross(moments, s[None].expand_as(moments)).permute(1, 0, 2).reshape(-1, sets * 3)], 1)
    out = torch.empty(sets, p.shape[0], 3, **_CUDA)
    step = max(256, int(2.5e8 // max(1, s.shape[0])))
    for i in range(0, p.shape[0], step):
        c = p[i:i + step]
        d2 = (c[:, :1] - s[None, :, 0]).square_()
        for a in (1, 2):
            d2 += (c[:, a:a + 1] - s[None, :, a]).square_()
        acc = d2.pow_(-1.5) @ cols
        first, second = acc[:, :sets * 3].reshape(-1, sets, 3), acc[:, sets * 3:].reshape(-1, sets, 3)
        out[:, i:i + step] = (torch.linalg.cross(first, c[:, None].expand_as(first)) - second).permute(1, 0, 2)
    return out


def _closest(p: np.ndarray, tri: np.ndarray) -> np.ndarray:
    """The closest point of every triangle (S, 3, 3) to p: the plane's foot where it falls inside,
    else the nearest of the three edges' closest points."""
    a, b, c = tri[:, 0], tri[:, 1], tri[:, 2]
    n = np.cross(b - a, c - a)
    n2 = (n * n).sum(1, keepdims=True)
    foot = p - n * (((p - a) * n).sum(1, keepdims=True) / n2)
    inside = np.ones(tri.shape[0], bool)
    best, where = np.full(tri.shape[0], np.inf), np.empty_like(a)
    for u, v in ((a, b), (b, c), (c, a)):
        inside &= (np.cross(v - u, foot - u) * n).sum(1) >= 0
        t = np.clip(((p - u) * (v - u)).sum(1) / ((v - u) ** 2).sum(1), 0.0, 1.0)
        q = u + t[:, None] * (v - u)
        d = ((q - p) ** 2).sum(1)
        where[d < best] = q[d < best]
        best = np.minimum(best, d)
    where[inside] = foot[inside]
    return where


def exact(case: dict, seed: int):
    """The potential, the raw field and its metrics, and the reciprocity field, in 64 bits. The recovered
    fields and their metrics have none here: their patch fits choose among rungs by thresholds."""
    kind, raw = case["kind"], case["recovery"] == "raw"
    if kind == "optimize" or (kind == "study" and not raw):
        return None
    head, coil, sites = _Head64(_head(case, seed)), _coil(case), _sites(case, seed)
    if kind == "field":
        return dict(q=_exact_field(case, head, _grid(case, seed)))
    frames = head.place(sites)
    sigma = head.conductivity(_SIGMA)
    dadt = head.dadt(coil, frames)
    if kind == "study":
        return _exact_study(case, seed, head, dadt)
    v = head.solve(sigma, head.rhs(sigma, dadt))
    e = head.fields(v, dadt) if raw else None
    if kind == "device":
        return [dict(transform=frames[k], E=e[k] if raw else None, magnE=e[k].norm(dim=1) if raw else None,
                     v=v[:, k] if case.get("potential") else None) for k in range(len(sites))]
    if kind == "guided":
        return [dict(transforms=frames[i:i + 8].reshape(-1, 16), v=v[:, i:i + 8].T) for i in range(0, len(sites), 8)]
    out = dict(transform=frames, metrics=np.stack([head.metrics(x) for x in e]) if raw else None)
    if case.get("potential"):
        out["v"] = list(v.T)
    if raw and case.get("vectors"):
        out["E"] = list(e)
    if raw and case.get("magnitude"):
        out["magnE"] = [x.norm(dim=1) for x in e]
    return out


def _exact_study(case: dict, seed: int, head: _Head64, dadt: torch.Tensor) -> list:
    from cunibs_b200 import uq

    tags = tuple(int(t) for t in np.unique(head.tags))
    draws = uq.sample_conductivities(ConductivityUQConfig(n_samples=case["draws"], seed=seed), tags)  # inputs
    rows = np.empty((dadt.shape[0], case["draws"], 16))
    for i, d in enumerate(draws):
        table = np.array(_SIGMA)
        table[list(tags)] = d
        sigma = head.conductivity(table)
        v = head.solve(sigma, head.rhs(sigma, dadt))
        for k, e in enumerate(head.fields(v, dadt)):
            rows[k, i] = head.metrics(e)
    return [dict(peak=r[:, 0], location=r[:, 1:4], focality=r[:, 8]) for r in rows]


def _exact_field(case: dict, head: _Head64, grid: adm.Grid) -> torch.Tensor:
    target = _target(case)
    gm = np.flatnonzero(head.tags == 2)
    d2 = ((head.bary[torch.tensor(gm, device="cuda")].cpu().numpy() - target.position_mm) ** 2).sum(1)
    within = d2 <= max(target.radius_mm ** 2, d2.min())
    at = torch.tensor(gm[within], device="cuda")
    weight = torch.zeros(head.tets.shape[0], **_CUDA)
    weight[at] = head.vols[at] / head.vols[at].sum()
    dirs = torch.eye(3, **_CUDA) if target.direction is None else torch.tensor(target.direction, **_CUDA)[None]
    sigma = head.conductivity(_SIGMA)
    corner = torch.einsum("da,eia->eid", dirs, head.grad) * weight[:, None, None]
    rhs = torch.zeros(head.n, dirs.shape[0], **_CUDA).index_add_(0, head.dtets.reshape(-1), corner.reshape(-1, dirs.shape[0]))
    lam = head.solve(sigma, rhs)
    w = torch.einsum("eid,eia->dea", lam[head.dtets], head.grad) * (head.vols * sigma)[None, :, None]
    w -= weight[None, :, None] * dirs[:, None, :]
    nodal = torch.zeros(dirs.shape[0], head.n, 3, **_CUDA)
    nodal.index_add_(1, head.dtets.reshape(-1), (0.25 * w)[:, :, None].expand(-1, -1, 4, -1).reshape(dirs.shape[0], -1, 3))
    axes = [grid.origin_m[a] + grid.spacing_m[a] * np.arange(grid.shape[a]) for a in range(3)]
    points = torch.tensor(np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3), **_CUDA)
    q = 1e-7 * _dipole_field(points, torch.tensor(head.nodes * 1e-3, **_CUDA), nodal)
    return q.reshape(dirs.shape[0], *grid.shape, 3)
