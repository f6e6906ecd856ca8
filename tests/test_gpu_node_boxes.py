"""The node test (traverse.cuh: test_node) where its rounding bound matters: rays with zero and tiny direction
components, along box faces, from far away, in scenes far from the origin and of extreme scale. A box missed shows as
a hit lost against a brute-force f64 Moeller-Trumbore test of every triangle."""
import numpy as np
import pytest

from rtcuda import PtSession, abi, scenes
from rtcuda.scene import Scene, affine, matte

pytestmark = pytest.mark.gpu


def brute(pos, rays):
    """Closest t in f64 and how far the hit is from its triangle's edges (the least barycentric)."""
    v = pos.astype(np.float64).reshape(-1, 3, 3)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    t_best, edge = np.full(rays.shape[1], np.inf), np.zeros(rays.shape[1])
    for i in range(rays.shape[1]):
        o, d = rays[0, i, :3].astype(np.float64), rays[1, i, :3].astype(np.float64)
        with np.errstate(all="ignore"):
            h = np.cross(d, e2)
            inv = 1.0 / (h * e1).sum(1)
            s = o - v[:, 0]
            b1 = (s * h).sum(1) * inv
            q = np.cross(s, e1)
            b2 = (q @ d) * inv
            t = (q * e2).sum(1) * inv
        m = np.minimum(np.minimum(b1, b2), 1.0 - b1 - b2)
        ok = (m > 0) & (t > 0) & np.isfinite(t)
        if ok.any():
            k = np.argmin(np.where(ok, t, np.inf))
            t_best[i], edge[i] = t[k], m[k]
    return t_best, edge


def awkward_rays(n, rng, centre, scale, far):
    """Rays aimed at points of the cloud; by thirds: general, one zero or tiny component, two of them."""
    target = centre + scale * rng.uniform(-0.5, 0.5, (n, 3))
    d = rng.normal(size=(n, 3))
    kind = np.arange(n) % 3
    for i in range(n):
        for a in rng.permutation(3)[:kind[i]]:
            d[i, a] = rng.choice([0.0, -0.0, 1e-30, -1e-22, 1e-12])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    planes = np.zeros((2, n, 4), np.float32)
    planes[0, :, :3] = target - far * scale * d
    planes[1, :, :3] = d
    planes[1, :, 3] = np.inf
    return planes


@pytest.mark.parametrize("centre,scale,far", [
    ((0, 0, 0), 1.0, 2.0), ((0, 0, 0), 1.0, 3e3), ((1000.0, -500.0, 2000.0), 4.0, 2.0),
    ((0, 0, 0), 1e-5, 2.0), ((0, 0, 0), 1e7, 2.0)])
@pytest.mark.parametrize("instanced", [False, True])
def test_no_hit_is_lost(centre, scale, far, instanced):
    if instanced and scale < 1e-2:
        pytest.skip("a transform of determinant below 1e-6 inverts to the identity, as Matrix4::inverse has it")
    rng = np.random.default_rng(11)
    c = np.asarray(centre, np.float64)
    pos = scenes.triangle_cloud_mesh(3000, seed=5)[0].astype(np.float64)
    world = (c + scale * pos).astype(np.float32)
    idx = np.arange(len(pos), dtype=np.uint32).reshape(-1, 3)
    s = Scene(8, 8)
    mat = s.add_material(matte((0.5, 0.5, 0.5)))
    if instanced:
        s.add_instance(s.add_mesh(pos.astype(np.float32), idx), mat, affine(np.eye(3) * scale, c))
    else:
        s.add_instance(s.add_mesh(world, idx), mat)
    rays = awkward_rays(600, rng, c, scale, far)
    with PtSession(s, abi.make_params(max_depth=4, max_paths=64)) as g:
        prim, _, t = g.intersect(rays)
        blocked = g.intersect(rays, any_hit=True)[0]
    want, edge = brute(world, rays)
    # The f32 hit test resolves a triangle's edges to the rounding of the coordinates it is given: a triangle of the
    # cloud is about 0.03 * scale wide, coordinates are about |centre| + far * scale and carry 2^-24 of that.
    size = np.abs(c).max() + (far + 1.0) * scale
    margin = 16 * size * 2.0 ** -24 / (0.03 * scale) + 1e-5
    clear = np.isfinite(want) & (edge > margin)
    assert clear.sum() > 60
    assert (prim[clear] != 0xFFFFFFFF).all()
    assert blocked[clear].all()
    # Never behind the closest hit by more than the same rounding along the ray (a nearer edge hit may be taken).
    assert (t[clear] <= want[clear] + 64 * size * 2.0 ** -24).all()


@pytest.mark.parametrize("far", [1e15, 5e16, 1e18, 1e22, 1e30])
def test_a_far_instance_hides_nothing(far):
    """One instance far away makes the top node's grid step huge: plane distances overflow along the axes on which a
    ray hardly moves, and no box the ray is in may be lost by that."""
    pos = scenes.triangle_cloud_mesh(3000, seed=5)[0].astype(np.float32)
    idx = np.arange(len(pos), dtype=np.uint32).reshape(-1, 3)
    s = Scene(8, 8)
    mat = s.add_material(matte((0.5, 0.5, 0.5)))
    cloud = s.add_mesh(pos, idx)
    s.add_instance(cloud, mat)
    for sign in (1.0, -1.0):
        s.add_instance(cloud, mat, affine(np.eye(3), (sign * far, -sign * far, sign * far)))
    rng = np.random.default_rng(2)
    rays = awkward_rays(600, rng, np.zeros(3), 1.0, 2.0)
    axis = np.zeros((2, 300, 4), np.float32)
    axis[0, :, :3] = pos.reshape(-1, 3, 3)[rng.integers(0, 3000, 300)].mean(1)
    axis[1, :, 3] = np.inf
    for i in range(300):
        a, sign = i % 3, 1.0 if i % 2 else -1.0
        axis[0, i, a], axis[1, i, a] = -3.0 * sign, sign
    rays = np.concatenate([rays, axis], axis=1)
    with PtSession(s, abi.make_params(max_depth=4, max_paths=64)) as g:
        prim, inst, t = g.intersect(rays)
        blocked = g.intersect(rays, any_hit=True)[0]
    want, edge = brute(pos, rays)
    clear = np.isfinite(want) & (edge > 16 * 3.5 * 2.0 ** -24 / 0.03 + 1e-5)
    assert clear[:600].sum() > 60 and clear[600:].sum() > 200
    assert (prim[clear] != 0xFFFFFFFF).all() and (inst[clear] == 0).all()
    assert blocked[clear].all()
    assert (t[clear] <= want[clear] + 64 * 3.5 * 2.0 ** -24).all()


@pytest.mark.parametrize("length", [1e-28, 1e-25, 1e-21, 1e-12, 1e12, 1e25, 1e30])
@pytest.mark.parametrize("instanced", [False, True])
def test_directions_of_any_length(length, instanced):
    """Directions are used as given: a ray of any length meets what the unit ray meets, at t over its length. Two in
    three have components a hundred million times below the largest, or none."""
    pos = scenes.triangle_cloud_mesh(3000, seed=5)[0].astype(np.float32)
    idx = np.arange(len(pos), dtype=np.uint32).reshape(-1, 3)
    s = Scene(8, 8)
    mat = s.add_material(matte((0.5, 0.5, 0.5)))
    if instanced:
        s.add_instance(s.add_mesh(pos, idx), mat, affine(np.eye(3) * 3.0, (1.0, 2.0, 3.0)))
        world = (pos.astype(np.float64) * 3.0 + (1.0, 2.0, 3.0)).astype(np.float32)
    else:
        s.add_instance(s.add_mesh(pos, idx), mat)
        world = pos
    rng = np.random.default_rng(4)
    centre, scale = (np.array([1.0, 2.0, 3.0]), 3.0) if instanced else (np.zeros(3), 1.0)
    rays = awkward_rays(600, rng, centre, scale, 2.0)
    d = rays[1, :, :3].astype(np.float64)
    d[np.abs(d) < 1e-8] = 0.0
    tiny = (d == 0.0) & (rng.uniform(size=d.shape) < 0.5)
    d = (d + tiny * 1e-9) * length
    rays[1, :, :3] = d
    with PtSession(s, abi.make_params(max_depth=4, max_paths=64)) as g:
        prim, _, t = g.intersect(rays)
        blocked = g.intersect(rays, any_hit=True)[0]
    unit = rays.astype(np.float64)
    unit[1, :, :3] /= length
    want, edge = brute(world, unit)
    size = np.abs(centre).max() + 3.0 * scale
    clear = np.isfinite(want) & (edge > 16 * size * 2.0 ** -24 / (0.03 * scale) + 1e-5)
    assert clear.sum() > 60
    assert (prim[clear] != 0xFFFFFFFF).all()
    assert blocked[clear].all()
    assert (t[clear].astype(np.float64) * length <= want[clear] + 64 * size * 2.0 ** -24).all()
