"""Points of more observations than a solve takes: their lists are ordered in J^T J and the SVD
algorithms, and a solve refuses them."""
import dataclasses

import numpy as np
import pytest

import oracle
from uncertaintyte_b200 import native, scenes

pytestmark = pytest.mark.gpu

LIMIT = 12288


@pytest.mark.parametrize("cams,heavy", [(1, [LIMIT]), (2, [LIMIT + 1]), (5, [30000]), (7, [20000, 3, 13000, 12288])])
def test_jtj_of_long_lists(cams, heavy):
    """Either side of the limit, several long lists among short ones; twice the same bytes. Sums of n
    terms: n eps of the largest sum of magnitudes."""
    rng = np.random.default_rng(cams)
    counts = np.concatenate([heavy, rng.integers(0, 9, 300)])
    op = rng.permutation(np.repeat(np.arange(len(counts)), counts))
    obs, points = len(op), len(counts)
    oc = rng.integers(0, cams, obs)
    cols = np.empty((obs, 2, 12), dtype=np.int32)
    cols[:, :, :9] = (9 * oc)[:, None, None] + np.arange(9)
    cols[:, :, 9:] = (9 * cams + 3 * op)[:, None, None] + np.arange(3)
    vals = rng.standard_normal(24 * obs)
    rows = (12 * np.arange(2 * obs + 1)).astype(np.int32)
    num_cols = 9 * cams + 3 * points
    r, c, v = native.jtj_crs(2 * obs, num_cols, rows, cols.reshape(-1), vals, cams)
    ro, co, vo = oracle.jtj(2 * obs, num_cols, rows, cols.reshape(-1), vals)
    np.testing.assert_array_equal(r, ro)
    np.testing.assert_array_equal(c, co)
    np.testing.assert_allclose(v, vo, rtol=0, atol=2 * obs * 2.2e-16 * np.abs(vo).max())
    np.testing.assert_array_equal(native.jtj_crs(2 * obs, num_cols, rows, cols.reshape(-1), vals, cams)[2], v)


def test_a_solve_refuses_a_long_list_and_goes_on():
    sc = scenes.make_sized_scene(6, 30, 4, seed=3)
    good = scenes.scene_jacobian(sc)
    order = np.concatenate([np.arange(len(sc.obs_cam)), np.full(50000, int(np.flatnonzero(sc.obs_pt == 5)[0]))])
    n = len(order)
    bad = dataclasses.replace(good, num_obs=n, num_rows=2 * n, rows=(12 * np.arange(2 * n + 1)).astype(np.int32),
                              cols=good.cols.reshape(-1, 24)[order].reshape(-1).copy(),
                              values=good.values.reshape(-1, 24)[order].reshape(-1).copy())
    with native.Context(0) as ctx:
        first = native.compute_covariances(good, ctx)[:2]
        for algorithm in (2, 3):  # the Taylor expansion, the SVD of the Schur complement
            with pytest.raises(native.UncError) as e:
                native.compute_covariances(bad, ctx, algorithm=algorithm)
            assert e.value.status == -8
        for a, b in zip(native.compute_covariances(good, ctx)[:2], first):
            np.testing.assert_array_equal(a, b)
