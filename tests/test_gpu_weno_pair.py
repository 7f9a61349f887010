"""The paired WENO5-Z interpolations of the fast and mixed forms
(weno5z_pair_f, weno5z_pair_m in emergence_b200/csrc/physics.cuh) against the
plain interpolation on the same stencils (needs a B200).

An undivided difference of the stencil is formed to a few units u of rounding
of the values it is formed from (u·max|v| in FP64; u·range in the mixed form,
whose differences are taken in FP64 and rounded to FP32). A weight is off by
that over the difference, the candidates it weighs differ by a few times the
difference, so the interpolant is off by a moderate multiple of u·max|v| (or
u·range) whatever the stencil: 256 units are allowed."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "weno_pair_check.cu")
OUT = os.path.join(HERE, "native", "_build", "libweno_pair_check.so")
DEPS = [SRC, os.path.join(HERE, "..", "emergence_b200", "csrc", "physics.cuh")]


def _run(v):
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", "-fmad=true", "-use_fast_math", SRC, "-o", OUT], check=True)
    lib = C.CDLL(OUT)
    lib.pair_check.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t]
    v = np.ascontiguousarray(v)
    out = np.empty((len(v), 6))
    assert lib.pair_check(v.ctypes.data, out.ctypes.data, len(v)) == 0
    return out


def _stencils(kind, rng, n):
    if kind == "random":
        return rng.normal(size=(n, 6)) * 10.0 ** rng.uniform(-6, 6, (n, 1))
    if kind == "smooth":
        return 1.0 + 10.0 ** rng.uniform(-16, 0, (n, 1)) * np.sin(np.arange(6) * rng.uniform(0, 1, (n, 1)) + rng.random((n, 1)))
    if kind == "step":
        return np.where(np.arange(6) < rng.integers(0, 7, (n, 1)), rng.random((n, 1)), rng.random((n, 1)))
    return np.repeat(rng.normal(size=(n, 1)), 6, axis=1) * (rng.random((n, 1)) < 0.7)  # flat, zeros among them


@pytest.mark.parametrize("kind", ["random", "smooth", "step", "flat"])
def test_pairs_match_the_plain_interpolation(kind):
    rng = np.random.default_rng(20261208)
    v = _stencils(kind, rng, 1 << 19)
    o = _run(v)
    size, span = np.abs(v).max(axis=1), v.max(axis=1) - v.min(axis=1)
    for side in (0, 1):
        fast, mixed = np.abs(o[:, side] - o[:, 4 + side]), np.abs(o[:, 2 + side] - o[:, 4 + side])
        assert (fast <= 256 * 2.0 ** -53 * size).all(), float((fast / np.maximum(size, 1e-300)).max())
        lim = 256 * 2.0 ** -24 * span + 256 * 2.0 ** -53 * size
        assert (mixed <= lim).all(), float((mixed / np.maximum(lim, 1e-300)).max())


def test_values_beyond_the_sixth_powers_range_take_the_other_path():
    rng = np.random.default_rng(20261209)
    v = rng.normal(size=(1 << 16, 6)) * 10.0 ** rng.uniform(18, 45, (1 << 16, 1))
    o = _run(v)
    size = np.abs(v).max(axis=1)
    for side in (0, 1):
        assert (np.abs(o[:, side] - o[:, 4 + side]) <= 256 * 2.0 ** -53 * size).all()
    assert not np.isfinite(_run(np.array([[1.0, 2.0, np.nan, 3.0, 4.0, 5.0]]))[0, :2]).any()
