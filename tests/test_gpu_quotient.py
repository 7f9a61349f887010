"""The plain FP64 form's branch-free quotients, square roots and WENO5-Z
interpolations (emergence_b200/csrc/quotient.cuh) against the compiler's
correctly rounded operations, bit for bit, on the GPU (needs a B200). A result
counts where the operands' range flag is clear; inside the documented ranges
the flag of a quotient must be clear."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "quotient_check.cu")
OUT = os.path.join(HERE, "native", "_build", "libquotient_check.so")
DEPS = [SRC] + [os.path.join(HERE, "..", "emergence_b200", "csrc", f) for f in ("physics.cuh", "quotient.cuh")]


def _lib():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", "-fmad=false", SRC, "-o", OUT], check=True)
    lib = C.CDLL(OUT)
    lib.quotient_check.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t]
    lib.weno_check.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t]
    lib.square_check.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t]
    return lib


def _ulps(x, k):
    """x moved by k units in the last place (x > 0)."""
    return (x.view(np.int64) + k).view(np.float64)


def _mantissas(rng, n):
    """[1, 2) with the values that decide roundings over-represented."""
    m = 1.0 + rng.random(n)
    pick = rng.integers(0, 6, n)
    k = rng.integers(0, 40, n)
    m = np.where(pick == 0, _ulps(np.full(n, 2.0), -k - 1), m)         # just below a power of two
    m = np.where(pick == 1, _ulps(np.full(n, 1.0), k), m)              # at or just above one
    m = np.where(pick == 2, 1.0 + rng.integers(0, 64, n) / 64.0, m)    # few bits
    return m


def _operands(rng, n, kind):
    b = _mantissas(rng, n) * 2.0 ** rng.integers(-99, 99, n)
    if kind == "any":
        a = _mantissas(rng, n) * 2.0 ** rng.integers(-899, 899, n)
    elif kind == "exact":      # quotients that are representable, and their neighbours
        a = b * (1.0 + rng.integers(0, 1 << 20, n) / float(1 << 20))
        a = _ulps(a, rng.integers(-2, 3, n))
    else:                      # quotients next to the midpoint of two doubles
        q = 1.0 + rng.random(n)
        a = _ulps(b * q + 0.5 * b * np.spacing(q), rng.integers(-2, 3, n))
    return a * rng.choice([-1.0, 1.0], n), b


def _check(a, b):
    out = np.empty((a.size, 10))
    assert _lib().quotient_check(a.ctypes.data, b.ctypes.data, out.ctypes.data, a.size) == 0
    return out


def _same(x, y):
    return x.view(np.int64) == y.view(np.int64)


@pytest.mark.parametrize("kind", ["any", "exact", "midpoint"])
def test_quotients_round_as_ieee_division(kind):
    rng = np.random.default_rng(20261204)
    a, b = (np.ascontiguousarray(x) for x in _operands(rng, 1 << 21, kind))
    a[:4] = [0.0, -0.0, 1.0, -1.0]
    b[:6] = [3.0, 7.0, 1.0 - 2.0 ** -53, 2.0 - 2.0 ** -52, 1.0, 2.0 ** 99]
    o = _check(a, b)
    assert not o[:, 2].any() and not o[:, 5].any()  # every operand lies inside the ranges
    assert _same(o[:, 0].copy(), o[:, 1].copy()).all()
    assert _same(o[:, 3].copy(), o[:, 4].copy()).all()
    assert _same(o[:, 6].copy(), 1.0 / b).all()


def test_operands_outside_the_ranges_are_flagged():
    x = np.array([0.0, -1.0, np.inf, -np.inf, np.nan, 2.0 ** -101, 2.0 ** 100, 5e-324])
    o = _check(np.ones_like(x), x)
    assert o[:, 2].all() and o[:, 8].all()
    y = np.array([np.inf, -np.inf, np.nan, 2.0 ** -901, 2.0 ** 900, 5e-324, -5e-324])
    assert _check(y, np.ones_like(y))[:, 2].all()


def test_square_roots_round_as_ieee_square_roots():
    rng = np.random.default_rng(20261205)
    n = 1 << 20
    g = _mantissas(rng, n) * 2.0 ** rng.integers(-48, 48, n)
    x = np.concatenate([(1.0 + rng.random(n)) * 2.0 ** rng.integers(-99, 99, n),
                        _mantissas(rng, n) * 2.0 ** rng.integers(-99, 99, n),
                        _ulps(g * g, rng.integers(-2, 3, n)),                          # squares and their neighbours
                        _ulps(g * g + g * np.spacing(g), rng.integers(-2, 3, n))])     # squares of midpoints
    o = _check(np.ones_like(x), np.ascontiguousarray(x))
    ok = o[:, 8] == 0.0
    assert _same(o[ok, 7].copy(), o[ok, 9].copy()).all()
    # roots within 2^-18 of a midpoint are left to the compiler's; the others are 1 − 2^-16 of random operands
    assert ok[:n].mean() > 0.999


def _hard_numerators(b):
    """For b = B·2^-52, B odd: a whose quotient is as close to the midpoint of two
    doubles as any by b, A·2^53 or A·2^54 = ±1 modulo B (A·2^-52 = a in [1, 2))."""
    out = []
    for x in b:
        B = int(x * 2.0 ** 52)
        for shift in (53, 54):
            A = pow(pow(2, shift, B), -1, B)
            out += [(float(A0) * 2.0 ** -52, x) for A0 in (A, B - A) if 2 ** 52 <= A0 < 2 ** 53 and (A0 < B) == (shift == 54)]
            # a ≥ b: the residues above B
            out += [(float(A0) * 2.0 ** -52, x) for A0 in (A + B, 2 * B - A) if shift == 53 and A0 < 2 ** 53]
    return out


def test_square_denominators_round_as_ieee_division():
    """recip_sq is not a correctly rounded reciprocal, so what decides are denominators
    next below a power of two and, by any denominator, the quotients next to a midpoint."""
    rng = np.random.default_rng(20261210)
    k = np.concatenate([np.arange(1, 6145, 2), 2 * rng.integers(0, 1 << 15, 4000) + 1]       # next to 2
                       + [2 * rng.integers(0, 1 << m, 20000) + 1 for m in (19, 24, 29, 33, 50)])
    near = 2.0 - np.arange(1, 6145) * 2.0 ** -52
    pairs = np.array(_hard_numerators(2.0 - k.astype(np.float64) * 2.0 ** -52) + [(2.0, x) for x in near] +
                     [(1.0, x) for x in near] + [(1.0 + rng.random(), x) for x in near])
    assert len(pairs) > 100000
    a, b = pairs[:, 0] * rng.choice([-1.0, 1.0], len(pairs)), pairs[:, 1]
    for lo, hi in ((-1, 1), (-132, 499)):  # the range of the smoothness indicators
        a = np.concatenate([a, pairs[:, 0] * 2.0 ** rng.integers(-400, 400, len(pairs))])
        b = np.concatenate([b, pairs[:, 1] * 2.0 ** rng.integers(lo, hi, len(pairs))])
    for kind in ("any", "exact", "midpoint"):
        x, y = _operands(rng, 1 << 20, kind)
        a, b = np.concatenate([a, x]), np.concatenate([b, y])
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    out = np.empty((a.size, 2))
    assert _lib().square_check(a.ctypes.data, b.ctypes.data, out.ctypes.data, a.size) == 0
    assert _same(out[:, 0].copy(), out[:, 1].copy()).all()


def test_stencils_with_denominators_next_to_a_power_of_two():
    rng = np.random.default_rng(20261211)
    n = 1 << 17
    # ramps of slope d, bent a little: beta_k near d², just below a power of two
    d = np.sqrt(2.0 ** rng.integers(-20, 20, n) * (1.0 - 2.0 ** rng.uniform(-60, -47, n)))
    v = d[:, None] * (np.arange(6) + rng.integers(-8, 8, (n, 1))) + (d * 2.0 ** rng.uniform(-60, -54, n))[:, None] * rng.normal(size=(n, 6))
    # values that differ by a few units in the last place: beta_k a few bits each
    w = _ulps(np.repeat(1.0 + rng.random((n, 1)), 6, axis=1), rng.integers(-40, 41, (n, 6)))
    v = np.ascontiguousarray(np.concatenate([v, w]))
    out = np.empty((2 * n, 5))
    assert _lib().weno_check(v.ctypes.data, out.ctypes.data, 2 * n) == 0
    assert not out[:, 4].any()
    assert _same(out[:, 0].copy(), out[:, 2].copy()).all() and _same(out[:, 1].copy(), out[:, 3].copy()).all()


def test_interpolations_round_as_the_plain_ones():
    rng = np.random.default_rng(20261206)
    n = 1 << 20
    v = rng.normal(size=(n, 6)) * 10.0 ** rng.uniform(-8, 8, (n, 1))
    smooth = 1.0 + 10.0 ** rng.uniform(-16, 0, (n, 1)) * np.sin(np.arange(6) * rng.uniform(0, 1, (n, 1)) + rng.random((n, 1)))
    step = np.where(np.arange(6) < rng.integers(0, 7, (n, 1)), rng.random((n, 1)), rng.random((n, 1)))
    flat = np.repeat(rng.normal(size=(n, 1)), 6, axis=1)
    flat[: n // 4] = 0.0
    wild = np.where(rng.random((n, 6)) < 0.3, 10.0 ** rng.uniform(-320, 308, (n, 6)), rng.normal(size=(n, 6)))
    wild[rng.random((n, 6)) < 0.02] = np.inf
    wild[rng.random((n, 6)) < 0.02] = np.nan
    faint = rng.normal(size=(n, 6)) * 10.0 ** rng.uniform(-268, -8, (n, 1))  # far ahead of a front
    for name, s in (("faint", faint), ("random", v), ("smooth", smooth), ("step", step), ("flat", flat), ("wild", wild)):
        s = np.ascontiguousarray(s)
        out = np.empty((n, 5))
        assert _lib().weno_check(s.ctypes.data, out.ctypes.data, n) == 0
        ok = out[:, 4] == 0.0
        assert _same(out[ok, 0].copy(), out[ok, 2].copy()).all(), name
        assert _same(out[ok, 1].copy(), out[ok, 3].copy()).all(), name
        if name != "wild":
            assert ok.all(), (name, (~ok).sum())
