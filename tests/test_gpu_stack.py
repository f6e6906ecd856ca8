"""The traversal stack: its entries in shared memory, the step to local memory and deep ones. The scene is a ladder of
instances, each 1.2 times as far and as large as the one before, which a ray along it enters one by one: its boxes all
lie on the ray, and a nearest-first walk stacks a node's farther children at every level before it tests anything. All
but the last instance are hollow (two slivers in opposite corners), so the ray comes back for every entry. The depths
were counted on the host builder's tree: 17 entries for 20 instances, 27 for 40, 141 for 200, 256 for 400."""
import numpy as np
import pytest

from rtcuda import PtSession, abi, scenes
from rtcuda.scene import Scene, affine, matte

pytestmark = pytest.mark.gpu


def _hollow():
    p = []
    for s in (-1.0, 1.0):
        c = np.full(3, 0.5 * s)
        p += [c, c - (s * 0.02, 0.0, 0.0), c - (0.0, s * 0.02, s * 0.02)]
    return np.array(p), np.arange(6).reshape(2, 3)


def _ladder(n, presence=1.0):
    s = Scene(8, 8)
    hollow, cube = s.add_mesh(*_hollow()), s.add_mesh(*scenes.unit_cube())
    mat = s.add_material(matte((0.5, 0.5, 0.5), presence=presence))
    for k, x in enumerate(1.2 ** np.arange(n)):
        s.add_instance(hollow if k < n - 1 else cube, mat, affine(np.eye(3) * 0.3 * x, (x, 0.0, 0.0)))
    return s


def _rays(n):
    rng = np.random.default_rng(n)
    r = np.zeros((2, 256, 4), np.float32)
    r[0, :, 1:3] = rng.uniform(-0.02, 0.02, (256, 2))
    r[1, :, 0] = 1.0
    r[1, :, 1:3] = rng.uniform(-0.05, 0.05, (256, 2))
    r[1, :, 3] = 1e38
    return r


@pytest.mark.parametrize("build", ["device", "host"])
@pytest.mark.parametrize("n", [1, 20, 28, 32, 36, 60, 200, 400])
def test_every_entry_comes_back(n, build):
    s, rays = _ladder(n), _rays(n)
    with PtSession(s, abi.make_params(max_depth=4, max_paths=64, bvh_build=build)) as g:
        prim, inst, t = g.intersect(rays)
        blocked = g.intersect(rays, any_hit=True)[0]
        trans = g.transmittance(rays)
    assert (inst == n - 1).all()
    # The last cube's near face; t to the rounding of object-space coordinates, which start about 4 before a face at 0.5.
    np.testing.assert_allclose(t, 0.85 * 1.2 ** (n - 1), rtol=1e-5)
    assert blocked.all()
    assert (trans == 0.0).all()


@pytest.mark.parametrize("n", [20, 32, 60, 200, 400])
def test_transmittance_visits_every_entry(n):
    """Cutouts attenuate and do not end the walk: through both faces of the last cube, in no order of distance."""
    with PtSession(_ladder(n, presence=0.5), abi.make_params(max_depth=4, max_paths=64)) as g:
        trans = g.transmittance(_rays(n))
    np.testing.assert_allclose(trans, 0.25, rtol=1e-6)
