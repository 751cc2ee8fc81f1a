"""The int8 slices of rows whose largest entry has no ordinary exponent: subnormal, infinite, not a
number. What such a row gets stays in its own row of the product."""
import numpy as np
import pytest

from uncertaintyte_b200 import native

pytestmark = pytest.mark.gpu

ROW = 7


def _operands(n):
    rng = np.random.default_rng(n)
    P, X = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    return P + P.T, X + X.T


def _product(P, X, slices=5):
    import torch
    n = len(P)
    p, x = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (P, X))
    c = torch.full((n, n), 5.0, dtype=torch.float64, device="cuda")
    native.gemm_mixed_device(n, p.data_ptr(), x.data_ptr(), n, c.data_ptr(), slices)
    torch.cuda.synchronize()
    return c.cpu().numpy().T  # column-major


@pytest.mark.parametrize("n", [200, 1100, 4200])
@pytest.mark.parametrize("slices", [3, 5])
def test_a_subnormal_row_has_the_digits_of_the_same_row_scaled(n, slices):
    """Entries k 2^-1074 with a largest one in [2^-1025, 2^-1022): exact, so the row's digits are those
    of the row times 2^200, and its products theirs times 2^-200 (X is scaled up to keep them normal)."""
    P, X = _operands(n)
    X *= 2.0 ** 400
    k = np.random.default_rng(1).integers(-2 ** 50, 2 ** 50, n)
    k[3] = 2 ** 50 + 12345  # the largest
    out = []
    for power in (-1074, -874):
        P[ROW] = P[:, ROW] = np.ldexp(k.astype(float), power)
        out.append(_product(P, X, slices))
    np.testing.assert_array_equal(out[0][ROW], out[1][ROW] * 2.0 ** -200)
    others = np.arange(n) != ROW
    np.testing.assert_array_equal(out[0][others], out[1][others])
    assert np.abs(out[1][ROW]).max() > 0


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [200, 1100, 4200])
def test_a_row_that_is_not_finite_leaves_the_others_alone(n, value):
    """Row 7 alone holds the value; its own products are not defined, except that a NaN is passed over."""
    P, X = _operands(n)
    P[ROW, ROW] = 0.0
    want = _product(P, X)
    P[ROW, ROW] = value
    got = _product(P, X)
    others = np.arange(n) != ROW
    np.testing.assert_array_equal(got[others], want[others])
    if np.isnan(value):
        np.testing.assert_array_equal(got[ROW], want[ROW])
