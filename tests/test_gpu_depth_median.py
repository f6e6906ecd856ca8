"""The denoiser's depth scale is the median positive depth, selected on the device: even and odd counts, one pixel,
none, ties, zeros and negative depths among them, values over the whole float range. The selected depth itself is
compared bit for bit with a sort; the filter is checked on films besides."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import denoise_oracle  # noqa: E402  (the checker)

from rtcuda.backend import denoise_film, depth_median  # noqa: E402

pytestmark = pytest.mark.gpu


def _film(w, h, depth):
    rng = np.random.default_rng(w * h)
    f = {k: rng.uniform(0.1, 1.0, (h, w, 3)) for k in ("beauty", "diffuse", "specular", "albedo")}
    n = rng.normal(size=(h, w, 3)) * 0.02 + np.array([0.0, 0.0, 1.0])
    f["normal"] = n / np.linalg.norm(n, axis=2, keepdims=True)
    f["depth"] = depth.reshape(h, w, 1)
    f["id"] = np.zeros((h, w, 2))
    return {k: v.astype(np.float32) for k, v in f.items()}


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (7, 5), (64, 33), (523, 401)])
@pytest.mark.parametrize("kind", ["near", "none", "ties", "mixed", "range"])
def test_filter_follows_the_median_depth(w, h, kind):
    rng = np.random.default_rng(len(kind) + w)
    n = w * h
    depth = {"near": 5.0 + rng.uniform(0, 1, n), "none": -rng.uniform(0, 1, n), "ties": rng.integers(3, 6, n) * 1.0,
             "mixed": np.where(rng.uniform(size=n) < 0.6, 0.0, rng.uniform(2, 3, n)),
             "range": np.exp(rng.uniform(-60, 60, n))}[kind]
    film = _film(w, h, depth)
    want = denoise_oracle.denoise({k: v.astype(np.float64) for k, v in film.items()})
    # As in test_gpu_film: f32 weights of fast exponentials. Coarser than a rank of the median or its low bits, which
    # test_median_is_the_sorted_one holds.
    np.testing.assert_allclose(denoise_film(film), want, rtol=2e-3, atol=2e-3)


def test_three_pixels_follow_their_middle_depth():
    """Two near depths, whose difference the filter sees through exp(-50 (dz / median)^2), and one far away: a scale of
    another rank changes the result by far more than the tolerance."""
    for a, b, c in ((1.0, 1.05, 40.0), (1.0, 1.05, 1e-3), (3.0, 3.2, 5.0)):
        depth = np.float32([a, b, c])
        film = _film(3, 1, depth)
        film["normal"][:] = (0.0, 0.0, 1.0)
        want = denoise_oracle.denoise({k: v.astype(np.float64) for k, v in film.items()})
        np.testing.assert_allclose(denoise_film(film), want, rtol=2e-4, atol=2e-4)


@pytest.mark.parametrize("n", [1, 2, 3, 64, 1000, 1001, 65_537, 1_000_003])
@pytest.mark.parametrize("kind", ["low bits", "range", "subnormal", "ties", "mixed", "none", "special"])
def test_median_is_the_sorted_one(n, kind):
    """Bit for bit, with depths that differ in the low ten bits alone (the third pass), in the middle eleven, in all;
    subnormals, infinities and NaN."""
    rng = np.random.default_rng(n + len(kind))
    one = np.float32(1.0).view(np.uint32)
    bits = {"low bits": one + rng.integers(0, 1024, n), "range": rng.integers(1, 0x7F800000, n),
            "subnormal": rng.integers(1, 0x00800000, n), "ties": one + 1024 * rng.integers(0, 3, n),
            "mixed": rng.integers(0, 0xFF800000, n), "none": 0x80000000 + rng.integers(0, 0x7F800000, n),
            "special": rng.choice([0, 1, one, 0x7F7FFFFF, 0x7F800000, 0x7FC00000, 0x80000000, 0xFF800000], n)}[kind]
    depth = bits.astype(np.uint32).view(np.float32)
    positive = np.sort(depth[depth > 0])
    want = positive[len(positive) // 2] if len(positive) else np.float32(0.0)
    assert depth_median(depth).view(np.uint32) == want.view(np.uint32)
