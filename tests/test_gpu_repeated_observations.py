"""Points that a camera observes many times over: the Schur complement takes every repetition, in
lists up to the longest that is accepted, and the work grows with the number of terms alone."""
import dataclasses

import numpy as np
import pytest

from conftest import block_rel_err
from uncertaintyte_b200 import native, scenes

pytestmark = pytest.mark.gpu

LIMIT = 12288  # observations of one point


def _from_blocks(sc, order, scale=None):
    """The Jacobian of the observations `order` (indices, repeats allowed), rows scaled."""
    jac = scenes.scene_jacobian(sc)
    cols, vals = jac.cols.reshape(-1, 24)[order], jac.values.reshape(-1, 24)[order].copy()
    if scale is not None:
        vals *= np.asarray(scale)[:, None]
    n = len(order)
    return dataclasses.replace(jac, num_obs=n, num_rows=2 * n, rows=(12 * np.arange(2 * n + 1)).astype(np.int32),
                               cols=cols.reshape(-1).copy(), values=vals.reshape(-1).copy(), lam=1e-5)


def _repeated(sc, point, counts, seed=0):
    """Multiplicities of every observation: counts (by the point's observations), 1 elsewhere."""
    m = np.ones(len(sc.obs_cam), dtype=int)
    m[np.flatnonzero(sc.obs_pt == point)] = counts
    return m, np.random.default_rng(seed).permutation(np.repeat(np.arange(len(m)), m))


def _check(sc, m, order):
    """m equal observations are one with its rows scaled by sqrt(m). The sums of up to 12288 terms
    err by 12288 eps = 2.7e-12 of ||Z|| <= trace = 9 per camera, divided by lambda = 1e-5."""
    one, _, _ = native.compute_covariances(_from_blocks(sc, np.arange(len(m)), np.sqrt(m)), precision="fp64")
    many, _, _ = native.compute_covariances(_from_blocks(sc, order), precision="fp64")
    assert block_rel_err(many, one, 45) < 2.7e-7 * 9 * len(sc.cams)


def _free_point(sc, cams):
    seen = np.bincount(sc.obs_pt, minlength=len(sc.points))
    return next(p for p in range(len(sc.points)) if seen[p] >= cams and p not in scenes.farthest_triple(sc.points))


@pytest.mark.parametrize("counts", [(2, 1), (33, 32, 31), (240, 241, 1), (1, 4000, 1), (3000, 3000, 3000),
                                    (9000, 1, 2000), (LIMIT - 2, 1, 1)])
def test_one_point_seen_many_times_by_few_cameras(counts):
    """Runs on either side of a warp's width and of the staging buffer; partners of one observation
    past the 8192 that a chunk takes, a camera's run across the two pieces; the longest list."""
    sc = scenes.make_sized_scene(6, 40, 5, seed=11)
    point = _free_point(sc, len(counts))
    idx = np.flatnonzero(sc.obs_pt == point)
    keep = np.sort(np.concatenate([np.flatnonzero(sc.obs_pt != point), idx[:len(counts)]]))
    sc = scenes.Scene(sc.cams, sc.points, sc.obs_cam[keep], sc.obs_pt[keep])
    _check(sc, *_repeated(sc, point, counts))


def test_every_point_seen_several_times():
    """Runs of 1 to 40 in lists of some hundred partners, at every point of a scene."""
    sc = scenes.make_sized_scene(30, 12, 10, seed=5)
    m = np.random.default_rng(2).integers(1, 41, len(sc.obs_cam))
    order = np.random.default_rng(3).permutation(np.repeat(np.arange(len(m)), m))
    _check(sc, m, order)


def test_lists_longer_than_the_limit_are_refused():
    sc = scenes.make_sized_scene(6, 40, 5, seed=11)
    point = _free_point(sc, 3)
    at = np.flatnonzero(sc.obs_pt == point)
    with native.Context(0) as ctx:
        for total, status in ((LIMIT, 0), (LIMIT + 1, -8), (LIMIT, 0)):
            counts = np.full(len(at), total // len(at))
            counts[0] += total - counts.sum()
            _, order = _repeated(sc, point, counts)
            if status == 0:
                native.compute_covariances(_from_blocks(sc, order), ctx)
            else:
                with pytest.raises(native.UncError) as e:
                    native.compute_covariances(_from_blocks(sc, order), ctx)
                assert e.value.status == status
