"""Which points' 3 x 3 blocks are singular: a point seen along one ray always is, whichever point of a
scene it is and however its last pivot rounds; a point of two cameras never."""
import numpy as np
import pytest

import oracle
from conftest import block_rel_err
from uncertaintyte_b200 import native, scenes

pytestmark = pytest.mark.gpu


def _scene(seed):
    sc = scenes.make_scene("tiny", seed=seed)
    free = [p for p in range(len(sc.points)) if p not in scenes.farthest_triple(sc.points)]
    return sc, free


def _with_observations(sc, point, keep):
    """The scene with `point` seen by the observations keep(its observations) alone."""
    idx = np.flatnonzero(sc.obs_pt == point)
    order = np.sort(np.concatenate([np.flatnonzero(sc.obs_pt != point), keep(idx)]))
    return scenes.scene_jacobian(scenes.Scene(sc.cams, sc.points, sc.obs_cam[order], sc.obs_pt[order]))


@pytest.mark.parametrize("repeats", [1, 2, 7])
@pytest.mark.parametrize("seed", range(4))
def test_every_point_seen_by_one_camera_is_refused(seed, repeats):
    sc, free = _scene(seed)
    with native.Context(0) as ctx:
        for point in free[:16]:
            jac = _with_observations(sc, point, lambda idx: np.repeat(idx[:1], repeats))
            with pytest.raises(native.UncError) as e:
                native.compute_covariances(jac, ctx)
            assert e.value.status == -6, point


def test_a_point_seen_once_is_refused_in_a_batch():
    sc, free = _scene(1)
    good = scenes.scene_jacobian(sc)
    b = native.Batch(0)
    for point in free[:6]:
        bad = _with_observations(sc, point, lambda idx: idx[:1])
        assert [status for *_, status in b.compute([good, bad, good])] == [0, -6, 0], point
    b.close()


def test_points_of_two_cameras_are_accepted():
    """lambda = 1e-5 and scaled blocks with eigenvalues above 1e-2: rounding moves Z by some 1e-14 and
    the blocks by 1e-9 of their size; 1e-7."""
    sc, free = _scene(2)
    with native.Context(0) as ctx:
        for point in free[:8]:
            jac = _with_observations(sc, point, lambda idx: idx[[0, -1]])
            jac.lam = 1e-5
            cam, pt, _ = native.compute_covariances(jac, ctx, precision="fp64")
            ref = oracle.compute(jac, lam=jac.lam)
            assert block_rel_err(cam, ref["cam"], 45) < 1e-7 and block_rel_err(pt, ref["pt"], 6) < 1e-7
