"""Eigen-decompositions of blocks that hold a NaN: every output of the block is written, and is no
number; nothing of an earlier call shows through."""
import numpy as np
import pytest

from uncertaintyte_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", range(1, 10))
def test_a_nan_block_gives_nans_in_every_place(dim):
    iu = np.triu_indices(dim)
    blocks = np.stack([np.diag(np.arange(1.0, dim + 1))] * 40)
    for at in ((0, 0), (dim - 1, dim - 1), (0, dim - 1)):
        bad = blocks.copy()
        bad[17, at[0], at[1]] = bad[17, at[1], at[0]] = np.nan
        native.block_eigen((1000.0 * blocks)[:, iu[0], iu[1]].reshape(-1), dim, sub_offset=0, sub_dim=dim)
        vals, vecs = native.block_eigen(bad[:, iu[0], iu[1]].reshape(-1), dim, sub_offset=0, sub_dim=dim)
        assert not np.isin(vals[17], 1000.0 * np.arange(1, dim + 1)).any()
        assert np.isnan(vals[17]).any() and np.isnan(vals[17][~np.isin(vals[17], np.arange(1, dim + 1))]).all()
        assert (np.abs(vecs[17][~np.isnan(vecs[17])]) <= 1).all()
        good = np.arange(40) != 17
        np.testing.assert_array_equal(vals[good], np.tile(np.arange(dim, 0, -1.0), (39, 1)))
