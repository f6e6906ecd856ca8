"""TLAS leaves of one item each, in both builders: counts around a wide node's eight children, instances in one place
(no split of their centroids exists, so that the builders halve them by their own orders), dense overlap. The device's tree has the host's size and finds the same hits, and
both agree with the f64 oracle."""
import numpy as np
import pytest

import oracle
from rtcuda import PtSession, abi, scenes
from rtcuda.scene import Scene, affine, matte

pytestmark = pytest.mark.gpu


def _scene(n, spread, seed=3):
    rng = np.random.default_rng(seed)
    s = Scene(8, 8)
    mats = [s.add_material(matte((0.5, 0.5, 0.5), id=k)) for k in range(3)]
    meshes = [s.add_mesh(*scenes.unit_cube()), s.add_mesh(*scenes.triangle_cloud_mesh(200, seed=1))]
    rot = scenes.random_rotations(rng, n)
    at = spread * rng.uniform(-1, 1, (n, 3))
    for k in range(n):
        s.add_instance(meshes[k % 2], mats[k % 3], affine(rot[k] * rng.uniform(0.3, 1.0), at[k]))
    return s, at


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 65, 300])
@pytest.mark.parametrize("spread", [0.0, 0.5, 10.0])
def test_builders_agree_and_match_oracle(n, spread):
    s, at = _scene(n, spread)
    rng = np.random.default_rng(8)
    rays = scenes.triangle_cloud_rays(4096, seed=7)
    rays[0, :, :3] *= 1.0 + spread
    rays[1, :, :3] = 0.0
    target = at[rng.integers(0, n, 4096)] + rng.uniform(-0.6, 0.6, (4096, 3))
    d = target - rays[0, :, :3]
    rays[1, :, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    got = {}
    for build in ("device", "host"):
        with PtSession(s, abi.make_params(max_depth=4, max_paths=64, bvh_build=build)) as g:
            prim, inst, t = g.intersect(rays)
            blocked = g.intersect(rays, any_hit=True)[0]
            got[build] = (prim, inst, t, blocked, g.stats()["tlas_nodes"])
    a, b = got["device"], got["host"]
    if spread > 0:
        assert a[4] == b[4]
    else:  # boxes of one centroid have no SAH split: halves by the builders' own orders
        assert abs(a[4] - b[4]) <= 1 + 0.01 * b[4]
    assert np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])
    op, oi, ot, _ = oracle.OracleScene(s).intersect(rays)
    hit = op != 0xFFFFFFFF
    assert hit.sum() > 200
    # Rays that graze an edge may differ in f32; t of the others to f32 rounding of the object-space coordinates.
    same = (a[0] != 0xFFFFFFFF) == hit
    assert same.mean() > 0.999
    both = hit & (a[0] != 0xFFFFFFFF)
    assert (np.abs(a[2][both] - ot[both]) <= 1e-4 * (1.0 + ot[both])).mean() > 0.999
    assert (a[3] == hit).mean() > 0.999


@pytest.mark.parametrize("presence", [1.0, 0.5])
@pytest.mark.parametrize("tris", [1, 2, 3, 5, 17, 63, 64, 65, 300])
def test_small_meshes_build_alike(tris, presence):
    """Meshes around the small-mesh limit (leaves of two instead of four, four in scenes with cutouts)."""
    s = Scene(8, 8)
    mat = s.add_material(matte((0.5, 0.5, 0.5), presence=presence))
    pos, idx = scenes.triangle_cloud_mesh(tris, seed=tris)
    s.add_instance(s.add_mesh(pos * 4.0, idx), mat)
    s.add_instance(s.add_mesh(*scenes.unit_cube()), mat, affine(np.eye(3), (3.0, 0.0, 0.0)))
    rays = scenes.triangle_cloud_rays(4096, seed=7)
    rays[0, :, :3] *= 3.0
    target = pos.reshape(-1, 3, 3)[np.arange(4096) % tris].mean(1) * 4.0
    d = target - rays[0, :, :3]
    rays[1, :, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    got = {}
    for build in ("device", "host"):
        with PtSession(s, abi.make_params(max_depth=4, max_paths=64, bvh_build=build)) as g:
            st = g.stats()
            got[build] = g.intersect(rays) + (st["blas_nodes"], st["tlas_nodes"])
    a, b = got["device"], got["host"]
    assert a[3:] == b[3:]
    assert np.array_equal(a[2], b[2])
    op, _, ot, _ = oracle.OracleScene(s).intersect(rays)
    hit = op != 0xFFFFFFFF
    assert hit.sum() > 2000 and ((a[0] != 0xFFFFFFFF) == hit).mean() > 0.999
    both = hit & (a[0] != 0xFFFFFFFF)
    assert (np.abs(a[2][both] - ot[both]) <= 1e-4 * (1.0 + ot[both])).mean() > 0.999


@pytest.mark.parametrize("offsets", [
    [(0, 0, 0), (1, 0, 0)], [(1, 0, 0), (0, 0, 0)], [(0, 0, 0), (0, 0, 0)], [(0, 0, 0), (0, 0, 1e-7)],
    [(0, 1e-13, 0), (0, 0, 0)], [(2, 1, 0), (0, 1, 2), (1, 1, 1)]])
def test_pairs_part_alike(offsets):
    """Two items left to part take no SAH sweep: either order along the widest axis, one place, centroids within f32 of
    one another."""
    s = Scene(8, 8)
    mat = s.add_material(matte((0.5, 0.5, 0.5)))
    cube = s.add_mesh(*scenes.unit_cube())
    for at in offsets:
        s.add_instance(cube, mat, affine(np.eye(3), at))
    rays = scenes.triangle_cloud_rays(2048, seed=7)
    rays[0, :, :3] *= 3.0
    d = np.asarray(offsets)[np.arange(2048) % len(offsets)] - rays[0, :, :3]
    rays[1, :, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    got = {}
    for build in ("device", "host"):
        with PtSession(s, abi.make_params(max_depth=4, max_paths=64, bvh_build=build)) as g:
            got[build] = g.intersect(rays) + (g.stats()["tlas_nodes"],)
    assert got["device"][3] == got["host"][3]
    assert np.array_equal(got["device"][2], got["host"][2])
    assert np.isfinite(got["host"][2]).all()


def test_large_mesh_instanced_densely():
    """A BLAS and a TLAS whose host trees are collapsed on all threads, the instances split along the BLAS's second
    level: the builders agree on the trees' sizes and on every hit."""
    rng = np.random.default_rng(5)
    s = Scene(8, 8)
    mat = s.add_material(matte((0.5, 0.5, 0.5)))
    mesh = s.add_mesh(*scenes.triangle_cloud_mesh(150_000, seed=9))
    at = rng.normal(size=(1500, 3)) * 0.1
    rot = scenes.random_rotations(rng, len(at))
    for k in range(len(at)):
        s.add_instance(mesh, mat, affine(rot[k], at[k]))
    rays = scenes.triangle_cloud_rays(2048, seed=7)
    got = {}
    for build in ("device", "host"):
        with PtSession(s, abi.make_params(max_depth=4, max_paths=64, bvh_build=build)) as g:
            st = g.stats()
            got[build] = g.intersect(rays) + (st["blas_nodes"], st["tlas_nodes"])
    a, b = got["device"], got["host"]
    assert a[3:] == b[3:] and a[3] > 16_384 and a[4] > 16_384
    assert np.array_equal(a[2], b[2])
    assert np.isfinite(a[2]).mean() > 0.5
