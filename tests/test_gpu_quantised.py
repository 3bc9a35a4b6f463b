"""The quantised traversal (flat and two-level triangle BVHs from 256 interior
nodes on) against the oracle's exact one, bit for bit, on the rays its grid has
to be conservative for: origins far from the grid, axis-parallel and nearly
parallel directions, unnormalised ones, rays along box planes, finite and
negative intervals; and instances whose hits tie."""
import numpy as np
import pytest

import oracle
from test_gpu_trace import check_closest
from yaoray_b200 import _lib, accel, scenes
from yaoray_b200.accel import SceneGeometry

pytestmark = pytest.mark.gpu


def grid_mesh(n: int, size: float, flat: bool, seed: int = 4):
    """An n x n sheet of two-triangle cells, level (every box flat) or rough."""
    rng = np.random.default_rng(seed)
    x, z = np.meshgrid(np.linspace(0, size, n + 1), np.linspace(0, size, n + 1), indexing="ij")
    y = np.zeros_like(x) if flat else rng.uniform(0, size / 20, x.shape)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a, b, c, d = i * (n + 1) + j, (i + 1) * (n + 1) + j, (i + 1) * (n + 1) + j + 1, i * (n + 1) + j + 1
    tris = np.concatenate([np.stack([a, b, c], -1).reshape(-1, 3), np.stack([a, c, d], -1).reshape(-1, 3)])
    return np.stack([x, y, z], -1).reshape(-1, 3).astype(np.float32), tris.astype(np.uint32)


def rays_for(geom, n: int = 40_000, seed: int = 1, snap: bool = True) -> np.ndarray:
    """Rays at random vertices of the scene, in every form listed above."""
    rng = np.random.default_rng(seed)
    pos = geom.positions.astype(np.float64)
    lo, hi = pos.min(0), pos.max(0)
    size = float((hi - lo).max())
    target = pos[rng.integers(0, len(pos), n)] + rng.normal(size=(n, 3)) * size * 0.01
    form = np.arange(n) % 10
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    axis = rng.integers(0, 3, n)
    par = form < 4  # parallel to an axis: exact zeros of both signs, or tiny components
    keep = np.arange(3)[None, :] == axis[:, None]
    small = np.where(form == 2, 1e-30, np.where(form == 3, 1e-9, 0.0))[:, None]
    d = np.where(par[:, None] & ~keep, small * rng.choice([-1.0, 1.0], (n, 3)), np.where(par[:, None], np.sign(d), d))
    dist = size * np.select([form == 4, form == 5, form == 6], [40.0, 3e3, 1e6], rng.uniform(0.1, 2.0, n))
    origin = target - d * dist[:, None]
    if snap:  # on the planes of boxes
        at = form == 1
        origin[at] = np.where(keep[at], origin[at], pos[rng.integers(0, len(pos), at.sum())])
    scale = np.where(form == 7, 10.0 ** rng.uniform(-6, 6, n), 1.0)
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = origin
    rays[:, 3] = np.where(form == 8, -size, scenes.RAY_T_MIN)
    rays[:, 4:7] = d * scale[:, None]
    rays[:, 7] = np.where(form == 9, dist * rng.uniform(0.5, 1.5, n), np.inf)
    return rays


def compare(cuda, geom, bvh, rays):
    import torch

    dev = accel.DeviceAccelerator(geom, bvh)
    r = torch.from_numpy(rays).to(cuda)
    inst = torch.empty(rays.shape[0], dtype=torch.int32, device=cuda)
    hits = dev.intersect(r, instances=inst)
    occ = dev.intersect(r, any_hit=True)
    dev.check()
    exp, _ = oracle.OracleScene(geom, bvh).trace(rays, stats=False)
    check_closest(hits, inst, exp, np.where(exp["hit"] != 0, exp["instance"], -1))
    assert np.array_equal(occ.cpu().numpy().astype(bool), exp["hit"].astype(bool))
    assert exp["hit"].any() and not exp["hit"].all()


@pytest.mark.parametrize("case", ["spheres", "flat", "rough", "offset", "small", "anisotropic"])
def test_flat_hits_are_the_oracles(cuda, case):
    if case == "spheres":
        g = scenes.traversal_scene(seed=3, spheres=6)
    elif case == "small":  # about 256 interior nodes
        g = SceneGeometry.from_meshes([grid_mesh(20, 3.0, False)])
    else:
        p, t = grid_mesh(60, 30.0, case != "rough")
        if case == "offset":
            p = p + np.float32(5.0e4)
        if case == "anisotropic":
            p = p * np.array([1.0, 1.0, 1e-3], np.float32)
        g = SceneGeometry.from_meshes([(p, t), (p + np.array([0, 2, 0], np.float32), t)])
    compare(cuda, g, accel.build_bvh(g), rays_for(g))


@pytest.mark.parametrize("case", ["spread", "tied"])
def test_two_level_hits_are_the_oracles(cuda, case):
    """Spread: meshes of very different sizes, so that rays start hundreds of
    extents from a BLAS's grid. Tied: level sheets that overlap in one plane,
    where an equal t goes to the instance visited first."""
    rng = np.random.default_rng(8)
    g = SceneGeometry.from_meshes([grid_mesh(24, 4.0, case == "tied"), grid_mesh(16, 4.0, case == "tied", 9)])
    inst = np.zeros(40, _lib.INSTANCE_DTYPE)
    for k in range(inst.size):
        m = np.eye(4)
        if case == "spread":
            m[:3, :3] = np.linalg.qr(rng.normal(size=(3, 3)))[0] * 10.0 ** rng.uniform(-2, 1)
            m[:3, 3] = rng.uniform(-40, 40, 3)
        else:
            m[:3, 3] = (rng.integers(0, 6), 0.0, rng.integers(0, 6))
        inst[k]["primitive"] = k % 2
        inst[k]["object_to_world"] = m.T.reshape(16)
    g = SceneGeometry(g.positions, g.indices, g.primitives, instances=inst)
    bvh = accel.build_two_level_bvh(g)
    rays = rays_for(SceneGeometry(np.concatenate([g.positions * s for s in (1, 3)]), g.indices, g.primitives),
                    snap=False)
    compare(cuda, g, bvh, rays)
