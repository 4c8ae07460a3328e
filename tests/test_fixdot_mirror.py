"""The line operators in mirror form on mirrored lines (chorus-mhd_gb300/csrc/fixdot.cuh, on the
host): the result is the mirrored result to the bit, since both rows of a pair come from the same
sums and are rounded alike.  (The middle row of a derivative, the rounding of one odd sum, is left
out.)  Lines of few significant bits among them, whose sums and limbs end in ties."""
import numpy as np
import pytest

from test_fixdot import MIRROR, apply_mirror, driver  # noqa: F401


@pytest.mark.parametrize("name,C,sigma", MIRROR, ids=[o[0] for o in MIRROR])
def test_mirrored_lines(driver, tmp_path, name, C, sigma):  # noqa: F811
    rng = np.random.default_rng(sum(map(ord, name)) + 2)
    NO, NI = C.shape
    n = 3000
    X = [rng.uniform(-1, 1, (n, NI)), rng.uniform(1, 2, (n, NI)),
         rng.integers(-2 ** 12, 2 ** 12, (n, NI)) * 2.0 ** -12,
         rng.uniform(-1, 1, (n, NI)).astype(np.float32).astype(np.float64),
         1 + rng.integers(-64, 64, (n, NI)) * 2.0 ** rng.integers(-35, -27, (n, 1))]  # limbs of half a unit
    X = np.concatenate(X)
    Y = apply_mirror(driver, tmp_path, C, X, sigma)[0]
    Z = apply_mirror(driver, tmp_path, C, X[:, ::-1], sigma)[0][:, ::-1] * sigma
    rows = np.arange(NO) != (NO // 2 if sigma < 0 and NO % 2 else -1)
    assert np.array_equal(Y[:, rows], Z[:, rows])
