"""The denoiser's depth scale is the median positive depth, selected on the device: even and odd counts, one pixel,
none, ties, zeros and negative depths among them, values over the whole float range."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import denoise_oracle  # noqa: E402  (the checker)

from rtcuda.backend import denoise_film  # noqa: E402

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
    # As in test_gpu_film: f32 weights of fast exponentials. A median off by one rank would change the depth weight of
    # every tap in the "near" films by far more (1 part in n of a scale whose square enters the exponent times 50).
    np.testing.assert_allclose(denoise_film(film), want, rtol=2e-3, atol=2e-3)


def test_scale_is_exact():
    """Two depths whose difference the filter sees through exp(-50 (dz / median)^2): the weight gives the median back."""
    for a, b, c in ((1.0, 1.05, 40.0), (1.0, 1.05, 1e-3), (3.0, 3.2, 5.0)):
        depth = np.float32([a, b, c])
        film = _film(3, 1, depth)
        film["normal"][:] = (0.0, 0.0, 1.0)
        want = denoise_oracle.denoise({k: v.astype(np.float64) for k, v in film.items()})
        np.testing.assert_allclose(denoise_film(film), want, rtol=2e-4, atol=2e-4)
