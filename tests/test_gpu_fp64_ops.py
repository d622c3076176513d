"""The FP64 operations of uns_fp64.cuh (register FMAs, integer-pipe division,
square root, comparisons, scalings) against the host's IEEE operations, bit
for bit: random operands over the fast route's exponent range and beyond it,
significands at the ends of their range and one unit apart, exact quotients
and squares and their neighbours, zeros, subnormals, infinities and NaN."""
import ctypes as C

import numpy as np
import pytest

from unsflow2d_gb300 import abi

pytestmark = pytest.mark.gpu
D = C.POINTER(C.c_double)

OPS = {"add": np.add, "sub": np.subtract, "mul": np.multiply, "div": np.divide, "sqrt": lambda a, b: np.sqrt(a),
       "half": lambda a, b: 0.5 * a, "twice": lambda a, b: 2.0 * a, "lt": lambda a, b: (a < b).astype(float),
       "le": lambda a, b: (a <= b).astype(float), "sign": lambda a, b: (a > 0).astype(float) - (a < 0).astype(float),
       "mul_digits": np.multiply, "narrow": lambda a, b: a.astype(np.float32).astype(float),
       "widen": lambda a, b: a.astype(np.float32).astype(float)}


def _operands(op):
    rng = np.random.default_rng(11)
    n = 1 << 20
    one, last = np.uint64(1), np.uint64((1 << 52) - 1)
    m = rng.integers(0, 1 << 52, (2, n), dtype=np.uint64)
    e = rng.integers(760, 1287, (2, n)).astype(np.uint64)  # across both ends of the fast route
    e[:, : n // 4] = rng.integers(1018, 1030, (2, n // 4))
    k = n // 16
    m[0, :k] = 0
    m[1, k:2 * k] = 0
    m[0, 2 * k:3 * k] = last
    m[1, 3 * k:4 * k] = last
    m[0, 4 * k:5 * k] = (m[1, 4 * k:5 * k] + one) & last
    m[0, 5 * k:6 * k] = (m[1, 5 * k:6 * k] - one) & last
    m[1, 6 * k:7 * k] |= np.uint64((1 << 29) - 1)
    m[1, 7 * k:8 * k] &= ~np.uint64((1 << 29) - 1)
    s = rng.integers(0, 2, (2, n)).astype(np.uint64) << np.uint64(63)
    a, b = (s | (e << np.uint64(52)) | m).view(np.float64)
    if op == "div":  # products, and their neighbours, over a factor
        q = rng.standard_normal(2 * k) * b[8 * k:10 * k]
        a[8 * k:10 * k] = q
        a[9 * k:10 * k] = np.nextafter(q[k:], np.inf)
    if op == "sqrt":
        a = np.abs(a)
        r = np.abs(rng.standard_normal(2 * k))
        a[8 * k:10 * k] = r * r
        a[9 * k:10 * k] = np.nextafter(a[9 * k:10 * k], rng.choice([0.0, np.inf], k))
    if op in ("narrow", "widen"):  # FP32's exponent range, its ends and rounding ties
        e[0] = rng.integers(860, 1170, n).astype(np.uint64)
        m[0, : n // 2] &= ~np.uint64((1 << 28) - 1)
        a = (s[0] | (e[0] << np.uint64(52)) | m[0]).view(np.float64)
    if op in ("lt", "le"):
        b[8 * k:9 * k] = a[8 * k:9 * k]
        b[9 * k:10 * k] = np.nextafter(a[9 * k:10 * k], np.inf)
    special = np.array([0.0, -0.0, 1.0, -1.0, 2.0, 4.0, np.finfo(float).max, -np.finfo(float).max, np.finfo(float).tiny,
                        5e-324, -5e-324, 1e-310, np.inf, -np.inf, np.nan, -np.nan, 2.0 ** -255, 2.0 ** -256, 2.0 ** 256, 2.0 ** 257,
                        np.nextafter(2.0 ** 257, 0), 2.0 ** 1023, 2.0 ** -1021, 2.0 ** -1022, 3.5])
    x, y = np.meshgrid(special, special)
    return np.concatenate([a, x.ravel(), special]), np.concatenate([b, y.ravel(), rng.standard_normal(len(special))])


@pytest.mark.parametrize("op", list(OPS))
def test_operation_equals_ieee(op):
    lib = abi.gpu_lib()
    lib.uns_selftest_fp64.argtypes = [C.c_int, D, D, D, C.c_int]
    a, b = (np.ascontiguousarray(x) for x in _operands(op))
    out = np.zeros_like(a)
    p = [x.ctypes.data_as(D) for x in (a, b, out)]
    assert lib.uns_selftest_fp64(list(OPS).index(op), *p, len(a)) == 0
    with np.errstate(all="ignore"):
        ref = OPS[op](a, b)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(out), nan)
    bad = np.flatnonzero((out.view(np.uint64) != ref.view(np.uint64)) & ~nan)
    assert len(bad) == 0, [(float(a[i]).hex(), float(b[i]).hex(), float(out[i]).hex(), float(ref[i]).hex()) for i in bad[:8]] + [len(bad)]
