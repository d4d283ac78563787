"""Argument checks of the stage functions that come before any CUDA call."""

import ctypes

import pytest

TOO_MANY = (1 << 31) + 1  # the functions index points in 32 bits


@pytest.fixture(scope="module")
def lib():
    from direbm_gb300 import _lib
    from direbm_gb300.build import build

    return _lib.load(build())


def _buffer():
    return ctypes.create_string_buffer(64)  # never read: the counts are refused first


def test_more_points_than_indices_are_refused(lib):
    b = _buffer()
    a = ctypes.addressof(b)
    f = ctypes.c_float
    calls = [
        lambda: lib.dbm_refine_control_points_f32(a, 1, a, a, a, TOO_MANY, f(1.0), 4, a, None),
        lambda: lib.dbm_resample_f32(a, a, a, TOO_MANY, a, 1, f(1.0), a, 0, f(1e-6), a, a, None),
        lambda: lib.dbm_resample_f32(a, a, a, 1, a, TOO_MANY, f(1.0), a, 0, f(1e-6), a, a, None),
        lambda: lib.dbm_resample_f32(a, a, a, 1, a, (1 << 32) + 1, f(1.0), a, 0, f(1e-6), a, a, None),
    ]
    for call in calls:
        assert call() == 1  # DBM_ERR_INVALID
        assert b"bad arguments" in lib.dbm_last_error()
