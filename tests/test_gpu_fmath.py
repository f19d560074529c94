"""The kernels' logarithm and power against their host twins bit for bit:
log2 over every mantissa (its division is the device's own), every exponent
and the special values, exp2 through the power over its whole range and its
subnormal results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32)) or bool(
        np.all((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))))


def test_every_mantissa(orc, ctx):
    m = np.arange(1 << 23, dtype=np.uint32)
    for e in (126, 127):  # [0.5, 1) and [1, 2): the opacities' range and the footprints'
        x = (m | np.uint32(e << 23)).view(np.float32)
        y = np.full_like(x, 0.75)
        assert _same(ctx.fmath_eval(x, y), orc.fmath_eval(x, y))


def test_exponents_and_specials(orc, ctx):
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint32).view(np.float32),
                        np.array([0.0, -0.0, 1.0, np.inf, -np.inf, np.nan, 1e-45, 1.17549435e-38],
                                 np.float32)])
    y = np.concatenate([rng.uniform(-160, 160, 1 << 20).astype(np.float32),
                        np.array([0.0, 1.0, -126.0, -126.5, 127.0, 127.9, 128.0, -151.0], np.float32)])
    two = np.full_like(y, 2.0)
    assert _same(ctx.fmath_eval(x, y), orc.fmath_eval(x, y))
    assert _same(ctx.fmath_eval(two, y), orc.fmath_eval(two, y))
