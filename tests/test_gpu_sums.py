"""Sums of floats and float-to-double conversions that the kernels make without FP64
instructions: as exact as in FP64 under cancellation, with subnormals, infinities,
NaN and sums beyond the float range.

Tolerance of a sum: rounded to FP64 three times, 3 x 2^-53 of it, and 2^-69 of the
largest term for the errors that are collected without compensation (16 of 2^-73).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows():
    rng = np.random.default_rng(5)
    x = (rng.standard_normal((4000, 16)) * 10.0 ** rng.uniform(-12, 12, (4000, 16))).astype(np.float32)
    x[:2000, 8:] = -x[:2000, 7::-1] * np.float32(1.0 + 2.0 ** -20)  # strong cancellation
    tiny = (rng.standard_normal((200, 16)) * 1e-39).astype(np.float32)
    mixed = np.concatenate([tiny[:, :8], (rng.standard_normal((200, 8)) * 1e-36).astype(np.float32)], axis=1)
    big = (np.abs(rng.standard_normal((50, 16))) * 0.5e38).astype(np.float32)
    odd = np.ones((6, 16), np.float32)
    odd[0, 3] = np.inf
    odd[1, 3] = -np.inf
    odd[2, 3] = np.nan
    odd[3, 3], odd[3, 9] = np.inf, -np.inf
    odd[4] = 0.0
    odd[5] = -0.0
    return np.ascontiguousarray(np.concatenate([x, tiny, mixed, big, odd]))


def test_sums_and_widening():
    from effmass_gb300 import build
    from effmass_gb300._lib import load
    build.build()
    x = _rows()
    got, wide = np.empty(len(x)), np.empty(x.shape)
    assert load().hpsi_selftest_sums(x.ctypes.data, len(x), got.ctypes.data, wide.ctypes.data) == 0
    nan = np.isnan(x)
    assert np.array_equal(wide[~nan].view(np.uint64), x[~nan].astype(np.float64).view(np.uint64))
    assert np.isnan(wide[nan]).all()
    for r, g in zip(x.astype(np.float64), got):
        if np.isfinite(r).all():
            want = math.fsum(r)
            assert abs(g - want) <= 3 * 2.0 ** -53 * abs(want) + 2.0 ** -69 * np.abs(r).max(), (g, want)
        else:
            with np.errstate(invalid="ignore"):
                want = r.sum()
            assert (np.isnan(g) and np.isnan(want)) or g == want
