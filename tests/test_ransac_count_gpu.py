"""Inlier counts from staged coordinates (packed f32, undecided homography tests in f64)
against the CPU oracle: around the ends of a warp's pass and of the staged part, with
residuals spread over the threshold, strong perspective, large and non-finite coordinates."""
import numpy as np
import pytest

import oracle as O
import psift

pytestmark = pytest.mark.gpu


def _matches(n, seed, scale=1.0, spread=3.0, persp=1e-4):
    """A homography's correspondences (coordinates to 2000 * scale), 60 % of them with
    residuals uniform in +-2 * spread pixels, the rest anywhere."""
    rng = np.random.default_rng(seed)
    m = np.zeros(n, psift.MATCH_DTYPE)
    q = rng.uniform(0, 2000, (n, 2))
    w = 1 + persp * q[:, 0] - 0.5 * persp * q[:, 1]
    t = np.stack([(0.9 * q[:, 0] - 0.2 * q[:, 1] + 40) / w, (0.15 * q[:, 0] + 1.1 * q[:, 1] - 30) / w], 1)
    t += rng.uniform(-2 * spread, 2 * spread, (n, 2)) / scale * rng.choice([0.1, 1.0], (n, 1))
    far = rng.random(n) < 0.4
    t[far] = rng.uniform(0, 2000, (int(far.sum()), 2))
    q, t = (q * scale).astype(np.float32), (t * scale).astype(np.float32)
    m["query_index"] = np.arange(n)
    m["target_index"] = np.arange(n)
    m["query_x"], m["query_y"], m["target_x"], m["target_y"] = q[:, 0], q[:, 1], t[:, 0], t[:, 1]
    m["displacement_x"], m["displacement_y"] = (t - q)[:, 0], (t - q)[:, 1]
    m["ratio"] = rng.uniform(0.3, 0.8, n)
    return m


def _same(m, thr):
    for fn, oracle in ((psift.Homography.estimate, lambda: O.homography_ransac(m, thr, None)),
                       (psift.Homography.estimate_similarity,
                        lambda: O.similarity_ransac(m, thr, O.DEFAULT_SIMILARITY_RANSAC_SEED))):
        mask, ref = oracle()
        inl, model = fn(m, psift.RansacOptions(thr, None))
        np.testing.assert_array_equal(inl["query_index"], m["query_index"][mask])
        assert (model is None) == (ref is None)
        if model is not None:
            k = 9 if len(np.ravel(model)) == 9 else 5  # rotation_deg: atan2f may differ by an ulp
            np.testing.assert_array_equal(np.ravel(model)[:k], np.ravel(ref)[:k])


@pytest.mark.parametrize("n", [63, 64, 65, 127, 511, 513, 1000, 9023, 9024, 9025, 9600])
def test_sizes(n):
    _same(_matches(n, n), 3.0)


@pytest.mark.parametrize("scale,thr", [(1.0, 0.5), (1.0, 40.0), (1e-3, 0.5), (200.0, 3.0), (1e4, 3.0), (1e13, 1e12)])
def test_scales_and_thresholds(scale, thr):
    _same(_matches(700, 5, scale, thr), thr)


@pytest.mark.parametrize("persp", [-2e-3, 3e-3])
def test_perspective_through_infinity(persp):
    _same(_matches(900, 6, persp=persp), 3.0)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38])
def test_a_non_finite_or_huge_coordinate(value):
    m = _matches(600, 7)
    m["target_x"][17] = value
    _same(m, 3.0)
