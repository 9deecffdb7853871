"""ParticleHandler2D on the GPU against the oracle.

Cell indices, per-cell counts, positions and barycentric coordinates are compared bit
for bit (the oracle orders particles by cell exactly as the engine does); the
projected node velocity within a tolerance (its sums are associated differently).
"""
import numpy as np
import pytest
import torch

import gpupfem2_gb300 as g
from gpupfem2_gb300 import meshgen as mg
from oracle import oracle as O
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "l0", "l1", "l2", "u", "v", "cell")


def _mesh(nx=32, ny=8, lx=4.0, ly=1.0):
    xy, tri = mg.channel(nx, ny, lx, ly)
    return xy, tri, g.Mesh2D.from_arrays(xy, tri)


def _field(xy, t=0.0):
    x, y = xy[:, 0], xy[:, 1]
    ux = 1.0 + 0.5 * np.sin(2 * np.pi * y + t)
    uy = 0.3 * np.cos(np.pi * x) * np.sin(np.pi * y)
    return ux, uy


def _assert_same(P, R, keys=KEYS):
    assert P["cell"].size == R["cell"].size
    for k in keys:
        assert np.array_equal(P[k], R[k]), k


@pytest.mark.parametrize("level", [1, 2, 3, 4])
def test_seed_bitwise(cuda, level):
    xy, tri, m = _mesh()
    ph = g.ParticleHandler2D(m, level)
    ph.seed()
    _assert_same(ph.download(), O.seed(xy, tri, level))


@pytest.mark.parametrize("level,dt", [(2, 0.05), (3, 0.2), (4, 0.12)])
def test_advect_locate_reseed_bitwise(cuda, level, dt):
    xy, tri, m = _mesh()
    area, invJ = O.mesh_geometry(xy, tri)
    off, idx = O.neighbors(xy.shape[0], tri)
    ph = g.ParticleHandler2D(m, level, capacity_factor=3.0)
    ph.seed()
    R = O.seed(xy, tri, level)
    deleted = added = 0
    for step in range(4):
        ux, uy = _field(xy, 0.7 * step)
        tux, tuy = torch.tensor(ux, device="cuda"), torch.tensor(uy, device="cuda")
        ph.advect(tux, tuy, dt, 3)
        R, nd, na = O.advect(R, xy, tri, invJ, off, idx, ux, uy, dt, 3, level, cap=3 * R["cell"].size)
        deleted += nd
        added += na
        P = ph.download()
        _assert_same(P, R)
    assert deleted > 0 and added > 0  # the outlet deletes, the inlet reseeds


def test_projection_and_correction(cuda):
    xy, tri, m = _mesh()
    area, invJ = O.mesh_geometry(xy, tri)
    off, idx = O.neighbors(xy.shape[0], tri)
    ph = g.ParticleHandler2D(m, 3)
    ph.seed()
    ux, uy = _field(xy)
    tux, tuy = torch.tensor(ux, device="cuda"), torch.tensor(uy, device="cuda")
    ph.init_velocity(tux, tuy)
    R = O.seed(xy, tri, 3)
    R["u"], R["v"] = O.correct_velocity(R, tri, ux, uy)
    _assert_same(ph.download(), R)
    ph.advect(tux, tuy, 0.1, 3)
    R, _, _ = O.advect(R, xy, tri, invJ, off, idx, ux, uy, 0.1, 3, 3)
    px = torch.empty_like(tux)
    py = torch.empty_like(tux)
    ph.project(px, py)
    ox, oy = O.project(R, tri, xy.shape[0])
    # per-cell partial sums, then per-node sums: a different association than the
    # oracle's particle-order accumulation
    assert rel_err(px.cpu().numpy(), ox) < 1e-13 and rel_err(py.cpu().numpy(), oy) < 1e-13
    nx, ny = ux * 1.1, uy - 0.2
    ph.correct(torch.tensor(nx, device="cuda"), torch.tensor(ny, device="cuda"), tux, tuy)
    R["u"], R["v"] = O.correct_velocity(R, tri, nx, ny, ux, uy)
    _assert_same(ph.download(), R)
    # projection after a correction uses the corrected velocities
    ph.project(px, py)
    ox, oy = O.project(R, tri, xy.shape[0])
    assert rel_err(px.cpu().numpy(), ox) < 1e-13


def test_upload_round_trip_and_order(cuda):
    xy, tri, m = _mesh(16, 4)
    R = O.seed(xy, tri, 2)
    perm = np.random.default_rng(1).permutation(R["cell"].size)
    shuffled = {k: v[perm] for k, v in R.items()}
    ph = g.ParticleHandler2D(m, 2)
    ph.upload(shuffled)
    P = ph.download()
    order = np.argsort(shuffled["cell"], kind="stable")
    _assert_same(P, {k: v[order] for k, v in shuffled.items()})


def test_capacity_overflow_is_reported(cuda):
    xy, tri, m = _mesh(16, 4)
    ph = g.ParticleHandler2D(m, 2, capacity_factor=1.1)
    R = O.seed(xy, tri, 2)
    big = {k: np.concatenate([v, v]) for k, v in R.items()}
    with pytest.raises(g.Pf2Error) as e:
        ph.upload(big)
    assert e.value.status == g.OVERFLOW


@pytest.mark.parametrize("level", [1, 2, 3, 4])
def test_sub_cells_at_their_borders_bitwise(cuda, level):
    """The occupied sub-cell is found in FP32 where that is certain: particles on the borders between
    sub-cells, a rounding beside them, and on either side of the band in which the FP64 rule
    decides (1e-5 in level units), at rest.  Which sub-cells the next sort reseeds, and so every
    particle, is the oracle's bit for bit."""
    xy, tri, m = _mesh(64, 32)
    area, invJ = O.mesh_geometry(xy, tri)
    off, idx = O.neighbors(xy.shape[0], tri)
    eps = np.array([0.0, 1e-16, 1e-12, 1e-9, 1e-7, 1e-6, 2.4e-6, 4e-6, 9e-6, 1.1e-5, 3e-5, 1e-4])
    eps = np.concatenate([eps, -eps[1:]]) / level
    rng = np.random.default_rng(level)
    per = 3
    nc = tri.shape[0]
    cell = np.repeat(np.arange(nc, dtype=np.int32), per)
    i, j = rng.integers(0, level + 1, cell.size), rng.integers(0, level + 1, cell.size)
    a = i / level + rng.choice(eps, cell.size)
    b = np.where(rng.random(cell.size) < 0.5, j / level + rng.choice(eps, cell.size), rng.random(cell.size))
    third = rng.random(cell.size) < 0.34  # (the third coordinate on a border instead)
    b = np.where(third, 1.0 - a - (j / level + rng.choice(eps, cell.size)), b)
    inside = (a >= 0) & (b >= 0) & (1.0 - a - b >= 0)
    l0, l1 = np.where(inside, a, 0.3), np.where(inside, b, 0.4)
    l2 = (1.0 - l0) - l1
    P = xy[tri[cell]]
    x = P[:, 0, 0] * l0 + P[:, 1, 0] * l1 + P[:, 2, 0] * l2
    y = P[:, 0, 1] * l0 + P[:, 1, 1] * l1 + P[:, 2, 1] * l2
    zero = np.zeros(cell.size)
    R = dict(x=x, y=y, l0=l0, l1=l1, l2=l2, u=zero, v=zero.copy(), cell=cell)
    ph = g.ParticleHandler2D(m, level, capacity_factor=6.0)
    ph.upload(R)
    still = np.zeros(xy.shape[0])
    t = torch.zeros(xy.shape[0], dtype=torch.float64, device="cuda")
    ph.advect(t, t, 0.1, 1)
    R, _, _ = O.advect(R, xy, tri, invJ, off, idx, still, still, 0.1, 1, level, cap=8 * level * level * nc)
    _assert_same(ph.download(), R)


def test_large_sets_project_again_after_a_correction(cuda):
    """From half a million particles on a correction forms the nodes' change in the place of the
    projection's partial sums: the velocities are the oracle's bit for bit, and projections after it
    are those of a handle that never corrected."""
    xy, tri, m = _mesh(256, 64)
    ph = g.ParticleHandler2D(m, 4)
    ph.seed()
    ux, uy = _field(xy)
    tux, tuy = torch.tensor(ux, device="cuda"), torch.tensor(uy, device="cuda")
    ph.init_velocity(tux, tuy)
    px, py, qx, qy = (torch.empty_like(tux) for _ in range(4))
    ph.project(px, py)
    nx, ny = ux * 1.1, uy - 0.2
    ph.correct(torch.tensor(nx, device="cuda"), torch.tensor(ny, device="cuda"), tux, tuy)
    R = O.seed(xy, tri, 4)
    R["u"], R["v"] = O.correct_velocity(R, tri, ux, uy)
    R["u"], R["v"] = O.correct_velocity(R, tri, nx, ny, ux, uy)
    P = ph.download()
    assert P["cell"].size >= 1 << 19
    _assert_same(P, R)
    other = g.ParticleHandler2D(m, 4)
    other.upload(P)
    for _ in range(2):
        ph.project(px, py)
        other.project(qx, qy)
        assert torch.equal(px, qx) and torch.equal(py, qy)
