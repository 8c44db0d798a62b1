"""Which kernel takes few query rows in several row blocks (fa8::decode_takes): the faster one, at points where
both were timed on a B200 (us) and differ by more than a few per cent."""
import ctypes

import pytest

from cutlass_flash_atten_fp8_b200 import _lib


def taken(slices, rows, Sk, D):
    f = _lib.load()._ZN3fa812decode_takesElliii
    f.restype, f.argtypes = ctypes.c_bool, [ctypes.c_int64, ctypes.c_int64] + 3 * [ctypes.c_int]
    return f(slices, rows, Sk, D, 148)


@pytest.mark.parametrize("D,rows,slices,Sk,decode_us,prefill_us", [
    (64, 24, 64, 8192, 28.3, 61.7), (64, 56, 16, 1024, 8.1, 12.3), (64, 56, 148, 8192, 92.9, 63.2), (128, 24, 64, 8192, 55.5, 73.3),
    (128, 24, 148, 8192, 102.9, 74.4), (128, 56, 32, 8192, 52.2, 72.2), (128, 56, 64, 1024, 16.6, 13.8), (160, 16, 32, 8192, 53.3, 64.8),
    (160, 16, 64, 1024, 15.8, 14.0), (160, 16, 64, 8192, 102.6, 65.8), (160, 32, 32, 1024, 15.7, 13.9), (192, 32, 16, 8192, 45.0, 65.6),
    (192, 56, 16, 1024, 16.4, 14.1), (224, 16, 64, 1024, 16.9, 14.6), (224, 56, 32, 8192, 196.1, 68.3), (256, 16, 32, 8192, 47.2, 69.8),
    (256, 32, 32, 1024, 15.8, 14.5), (256, 32, 64, 8192, 155.9, 70.8), (256, 56, 4, 8192, 39.4, 68.7)])
def test_the_faster_kernel_takes_the_call(D, rows, slices, Sk, decode_us, prefill_us):
    assert taken(slices, rows, Sk, D) == (decode_us < prefill_us)


def test_the_range():
    assert all(taken(n, rows, 1, 64) for n in (1, 10 ** 6) for rows in (1, 16))          # one block of rows
    assert all(taken(n, 8, 10 ** 6, 256) for n in (1, 10 ** 6))
    assert not taken(1, 64, 10 ** 6, 64) and taken(1, 63, 10 ** 6, 64)
    assert taken(2 ** 28 - 1, 1, 64, 64) and not taken(2 ** 28, 1, 64, 64)              # the largest grid
