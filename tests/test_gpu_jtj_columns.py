"""J^T J of rows whose columns name no camera or point of the scene: a layout error."""
import numpy as np
import pytest

from uncertaintyte_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cam,pt", [(10 ** 6, None), (3, None), (None, 40), (None, 10 ** 6), (None, -1), (-1, None)])
def test_columns_out_of_range(cam, pt):
    cams, points = 3, 40
    sc = scenes.make_sized_scene(cams, 14, 3, seed=2)
    keep = sc.obs_pt < points
    jac = scenes.scene_jacobian(scenes.Scene(sc.cams, sc.points[:points], sc.obs_cam[keep], sc.obs_pt[keep]))
    cols = jac.cols.copy().reshape(-1, 2, 12)
    if cam is not None:
        cols[5, :, :9] = 9 * cam + np.arange(9)
    if pt is not None:
        cols[5, :, 9:] = 9 * cams + 3 * pt + np.arange(3)
    with pytest.raises(native.UncError) as e:
        native.jtj_crs(jac.num_rows, jac.num_cols, jac.rows, cols.reshape(-1), jac.values, cams)
    assert e.value.status == -2
    native.jtj_crs(jac.num_rows, jac.num_cols, jac.rows, jac.cols, jac.values, cams)
