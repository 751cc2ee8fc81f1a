"""One context that changes how it evaluates one size: the captured inverse depends on the precision
(its last product on int8 slices above N = 3584) and on the evaluation of the series (a copy of X)."""
import numpy as np
import pytest

from uncertaintyte_b200 import native, scenes

pytestmark = pytest.mark.gpu

MODES = [("mixed", "powers"), ("fp64", "powers"), ("mixed", "sequential"), ("fp64", "sequential"), ("mixed4", "powers")]


@pytest.mark.parametrize("cams", [398, 399])
def test_modes_of_one_size_in_one_context(cams):
    """N = 3582 (tile tasks) and 3591 (recursive, T^T T by int8): five modes in turns, each three times
    (direct, captured, replayed), give the bytes of a context of their own."""
    jac = scenes.scene_jacobian(scenes.make_sized_scene(cams, 10, 4, seed=7))
    jac.lam = 1e-5
    own = {}
    for mode in MODES:
        with native.Context(0) as c:
            own[mode] = native.compute_covariances(jac, c, precision=mode[0], taylor=mode[1])[:2]
    with native.Context(0) as c:
        for _ in range(3):
            for mode in MODES:
                cam, pt, _ = native.compute_covariances(jac, c, precision=mode[0], taylor=mode[1])
                np.testing.assert_array_equal(cam, own[mode][0], err_msg=str(mode))
                np.testing.assert_array_equal(pt, own[mode][1], err_msg=str(mode))
