"""The branch-free FP64 exp, tanh and square roots of csrc/fastmath.cuh.

CPU: the exponentials' operations (Cody-Waite reduction against ln 2; the
degree-13 Taylor polynomial in Estrin form, or the degree-9 interpolant of the
form for [-1.5, 0]; the exponent-field scale) are emulated with exact fused
multiply-adds, with the constants read from the header, and held against libm
or its 80-bit form: within 1 ulp, 2^-52 relative on [-1.5, 0].  GPU: the
device functions (hdnnp_debug_math) against numpy's results: exp and 1/sqrt
within 2 ulp, sqrt within 1 ulp, exp on [-1.5, 0] within 2^-52 and tanh on
[0, 1] (u times a polynomial in u^2) within 4e-16 relative.  These replace the
library calls of the reference's intrinsics exp, tanh and sqrt
(symmetryFunctions.f90:201-327) in the symmetry-function kernels.
"""
import math
import os
import re
import struct
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "high-dimensional-neural-network-potential_b200", "csrc", "fastmath.cuh")


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _exp_constants():
    src = open(HEADER).read()
    body = src[src.index("double exp_clamped(double x)"):]
    body = body[: body.index("\n}\n")]
    named = dict(re.findall(r"constexpr double (\w+) = ([0-9.eE+-]+);", body))
    pairs = re.findall(r"fma\(([0-9.eE+-]+), r, ([0-9.eE+-]+)\)", body)
    return {k: float(v) for k, v in named.items()}, [(float(a), float(b)) for a, b in pairs]


def _exp_emulated(x, K, Q):
    x = min(max(x, -708.0), 709.0)
    t = _fma(x, K["kLog2e"], K["kShift"])
    k = struct.unpack("<q", struct.pack("<d", t))[0] & 0xFFFFFFFF
    k = k - (1 << 32) if k >= (1 << 31) else k
    kd = t - K["kShift"]
    r = _fma(kd, -K["kLn2Hi"], x)
    r = _fma(kd, -K["kLn2Lo"], r)
    r2 = r * r
    r4 = r2 * r2
    r8 = r4 * r4
    q = [r] + [_fma(a, r, b) for a, b in Q]  # q0 .. q6
    s0 = _fma(q[1], r2, q[0])
    s1 = _fma(q[3], r2, q[2])
    s2 = _fma(q[5], r2, q[4])
    t0 = _fma(s1, r4, s0)
    t1 = _fma(q[6], r4, s2)
    p = 1.0 + _fma(t1, r8, t0)
    return p * math.ldexp(1.0, k)


def test_exp_emulation_within_one_ulp():
    K, Q = _exp_constants()
    assert set(K) == {"kLog2e", "kLn2Hi", "kLn2Lo", "kShift"} and len(Q) == 6
    # the coefficients are 1/n! for n = 2..13
    assert all(abs(b - 1 / math.factorial(2 * i + 2)) <= 1e-16 / math.factorial(2 * i + 2) for i, (a, b) in enumerate(Q))
    rng = np.random.default_rng(7)
    xs = np.concatenate([-rng.random(600) * 5.0, -rng.random(200) * 700.0, rng.random(100) * 50.0, [0.0, -1e-300, -708.0]])
    worst = 0.0
    for x in xs:
        ref = math.exp(float(x))
        worst = max(worst, abs(_exp_emulated(float(x), K, Q) - ref) / math.ulp(ref))
    assert worst <= 1.0, worst


@pytest.mark.gpu
def test_device_functions_against_libm(pkg):
    from hdnnp_b200 import engine

    rng = np.random.default_rng(11)
    # exp: the symmetry functions' arguments -eta R (R up to 3 rc^2) and wide ranges
    x = np.concatenate([-rng.random(20000) * 5.0, -rng.random(20000) * 700.0, rng.random(2000) * 700.0, [0.0, -708.0]])
    y = engine.debug_math(0, x)
    ulp = np.abs(y - np.exp(x)) / np.spacing(np.exp(x))
    assert ulp.max() <= 2.0, ulp.max()
    # tanh of u = 1 - r/rc in [0, 1]
    u = np.concatenate([rng.random(40000), np.linspace(0.0, 1.0, 1001), [1e-12, 1e-6]])
    t = engine.debug_math(1, u)
    assert np.abs(t - np.tanh(u)).max() <= 6e-16
    big = u > 0.2
    assert (np.abs(t[big] - np.tanh(u[big])) / np.tanh(u[big])).max() <= 3e-15
    # square roots of squared distances (0 included: sqrt 0 = 0)
    r2 = np.concatenate([rng.random(40000) * 1000.0, rng.random(2000) * 1e-6, [0.0, 144.0]])
    s = engine.debug_math(2, r2)
    assert np.all(np.abs(s - np.sqrt(r2)) <= np.spacing(np.sqrt(r2)))
    pos = r2 > 0
    ir = engine.debug_math(3, r2[pos])
    ref = 1.0 / np.sqrt(r2[pos])
    assert (np.abs(ir - ref) / np.spacing(ref)).max() <= 2.0
    # bad selector
    with pytest.raises(engine.HdnnpError):
        engine.debug_math(7, x[:4])


def _table(name):
    src = open(HEADER).read()
    body = src[src.index(f"__constant__ double {name}["):]
    return [float(v) for v in re.findall(r"-?[0-9.]+(?:e[+-]?[0-9]+)?", body[body.index("{"): body.index("}")])]


def _exp_small_emulated(x, c):
    t = _fma(x, c[0], c[1])
    kd = t - c[1]
    r = _fma(kd, -c[2], x)
    r2 = r * r
    a, b = c[11], c[12]
    for n in (9, 7, 5, 3):
        a = _fma(a, r2, c[n])
    for n in (10, 8, 6, 4):
        b = _fma(b, r2, c[n])
    return math.ldexp(1.0 + _fma(_fma(b, r, a), r2, r), int(kd))


def _bounded_arguments(lo, n, seed):
    """[lo, 0] with both ends and the borders of the reduction."""
    rng = np.random.default_rng(seed)
    k = np.arange(0.5, -lo / math.log(2.0)) * math.log(2.0)
    x = np.concatenate([lo * rng.random(n), -rng.random(n // 10) * 1e-3, [lo, 0.0, -1e-300], -k, -k * (1 + 1e-15),
                        -k * (1 - 1e-15)])
    return x[x >= lo]


def test_exp_small_emulation():
    """Reduction (error of ln 2 in one double, rounding of r), the last terms
    of the polynomial and the last addition: below 2^-52 relative."""
    c = _table("kExpSmall")
    assert len(c) == 13
    for x in _bounded_arguments(-1.5, 3000, 3):
        ref = Fraction(*np.exp(np.longdouble(x)).as_integer_ratio())
        assert abs(Fraction(_exp_small_emulated(float(x), c)) - ref) <= ref / 2**52, x


def test_exp_neg_coefficients():
    """exp_neg's table holds exp_clamped's constants and 1/n!, n = 2..13."""
    K, Q = _exp_constants()
    c = _table("kExpNeg")
    assert c[:4] == [K["kLog2e"], K["kShift"], K["kLn2Hi"], K["kLn2Lo"]]
    assert c[4:] == [v for a, b in Q for v in (b, a)]


@pytest.mark.gpu
def test_device_bounded_functions(pkg):
    """The forms without range tests: exp on [-1.5, 0] below 2^-52 relative,
    exp on [-700, 0] within 2 ulp; tanh on [0, 1] within 4e-16 relative (the
    two last roundings of the polynomial, the product and the interpolation,
    also as u -> 0)."""
    from hdnnp_b200 import engine

    def err(y, ref):
        return np.abs((y.astype(np.longdouble) - ref) / ref).astype(float).max()

    x = _bounded_arguments(-1.5, 100000, 4)
    assert err(engine.debug_math(4, x), np.exp(x.astype(np.longdouble))) <= 2.0**-52
    x = _bounded_arguments(-700.0, 100000, 5)
    y = engine.debug_math(5, x)
    assert (np.abs(y - np.exp(x)) / np.spacing(np.exp(x))).max() <= 2.0
    rng = np.random.default_rng(6)
    u = np.concatenate([rng.random(100000), 10.0 ** -rng.uniform(0, 12, 2000), [1.0, 1e-300]])
    assert err(engine.debug_math(1, u), np.tanh(u.astype(np.longdouble))) <= 4e-16
    assert engine.debug_math(1, np.zeros(1))[0] == 0.0
