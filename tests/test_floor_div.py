"""The tap position of the general accumulation, floor((float)v / s), without a
division: a model of merge.cu's floor_div_f in FP32 arithmetic (the fused
multiply-add evaluated exactly), against the division, over every output
position of a large frame and its surroundings at scales on and off the binary
grid."""
import numpy as np
import pytest


def floor_div_f(v, s):
    s = np.float32(s)
    fv = v.astype(np.float32)
    c = np.rint(fv * (np.float32(1) / s))
    # fma(-c, s, fv): the product of two 24-bit mantissas and the sum are exact in 64 bits at these sizes
    e = (fv.astype(np.float64) - c.astype(np.float64) * np.float64(s)).astype(np.float32)
    near = (e < 0) & (e > np.abs(c) * s * np.float32(-(2.0 ** -22)))
    q = np.where(e < 0, c - np.float32(1), c)
    return np.where(near, np.floor(fv / s), q).astype(np.int64)


@pytest.mark.parametrize("s", [0.25, 0.5, 0.7, 0.9, 1.0, 1.1, 1.2, 1.25, 1.3, 1.5, 1.7, 2.0, 2.2, 2.5, 3.0, 3.3, 4.0, 4.7, 5.0, 6.0, 7.0, 7.9, 8.0])
def test_floor_div_equals_division(s):
    v = np.arange(-70000, 240000, dtype=np.int64)
    assert np.array_equal(floor_div_f(v, s), np.floor(v.astype(np.float32) / np.float32(s)).astype(np.int64))
    if float(s).is_integer():
        assert np.array_equal(floor_div_f(v, s), v // int(s))


def test_floor_div_random_scales():
    rng = np.random.default_rng(5)
    v = rng.integers(-70000, 240000, 20000)
    for s in rng.uniform(0.2, 8.0, 300).astype(np.float32):
        assert np.array_equal(floor_div_f(v, s), np.floor(v.astype(np.float32) / s).astype(np.int64)), s
