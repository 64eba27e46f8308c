"""The homography counts' f32 test out of its range (coordinates from 1e15): every match is
decided in f64, also where the f32 values of w, U and V are all exactly zero."""
import numpy as np
import pytest

import oracle as O
import psift

pytestmark = pytest.mark.gpu


def _matches(n, seed, share):
    """Queries on the f32 lattice around (2^53, 0), `share` of them at that point: in f32 a
    homography's last column is often the first one times -2^53, which maps the point to 0."""
    rng = np.random.default_rng(seed)
    m = np.zeros(n, psift.MATCH_DTYPE)
    k = rng.integers(-3, 4, (n, 2))
    q = np.stack([2.0 ** 53 + np.where(k[:, 0] > 0, k[:, 0] * 2.0 ** 30, k[:, 0] * 2.0 ** 29), k[:, 1] * 2.0 ** 29], 1)
    q[rng.random(n) < share] = (2.0 ** 53, 0.0)
    q, t = q.astype(np.float32), rng.uniform(0, 2000, (n, 2)).astype(np.float32)
    m["query_index"] = m["target_index"] = np.arange(n)
    m["query_x"], m["query_y"], m["target_x"], m["target_y"] = q[:, 0], q[:, 1], t[:, 0], t[:, 1]
    m["displacement_x"], m["displacement_y"] = (t - q)[:, 0], (t - q)[:, 1]
    m["ratio"] = rng.uniform(0.3, 0.8, n)
    return m


@pytest.mark.parametrize("n", [128, 640])
@pytest.mark.parametrize("share", [0.2, 0.5])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_counts_beyond_the_f32_range_equal_the_oracle(n, share, seed):
    m = _matches(n, seed, share)
    mask, ref = O.homography_ransac(m, 3.0, None)
    inl, model = psift.Homography.estimate(m, psift.RansacOptions(3.0, None))
    np.testing.assert_array_equal(inl["query_index"], m["query_index"][mask])
    np.testing.assert_array_equal(np.ravel(model), np.ravel(ref))
