"""The division-free admissibility test that the sweep's positivity limiter
tries first (surely_admissible of emergence_b200/csrc/physics.cuh, ideal gas) never
accepts a state that the reference's test (to_prim then admissible,
C/system.rs:197-203,404-407) rejects, so the limiter decides exactly as the
reference does. The function itself, compiled for the host (no GPU), over states
spread across the admissibility boundary."""
import ctypes as C
import os
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "admissible_host.cpp")
OUT = os.path.join(HERE, "native", "_build", "libadmissible_host.so")
DEPS = [SRC, os.path.join(HERE, "..", "emergence_b200", "csrc", "physics.cuh")]


def surely_admissible(a):
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-Wno-unknown-pragmas",
                        "-I", cuda_inc, SRC, "-o", OUT], check=True)
    a = np.ascontiguousarray(a, dtype=np.float64)
    out = np.zeros(len(a), dtype=np.uint8)
    lib = C.CDLL(OUT)
    lib.admissible_check(C.c_void_p(a.ctypes.data), C.c_size_t(len(a)), C.c_void_p(out.ctypes.data))
    return out.astype(bool)


def reference_admissible(a, gamma):
    with np.errstate(all="ignore"):
        rho = a[:, 0]
        vx, vy, vz = a[:, 1] / rho, a[:, 2] / rho, a[:, 3] / rho
        ein = a[:, 4] / rho - 0.5 * (vx * vx + vy * vy + vz * vz)
        v = 1.0 / rho
        p = (gamma - 1.0) * (ein - 0.0) / (v - 0.0) - gamma * 0.0
        return np.isfinite(rho) & np.isfinite(p) & (rho > 0) & (1.0 / rho > 0.0) & (p + 0.0 > 0)


def states(n, rng, rel):
    """Conserved states whose 2ρE − |ρu|² is rel·(2ρE + |ρu|²)-ish."""
    rho = 10.0 ** rng.uniform(-6, 6, n)
    m = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-6, 6, (n, 1))
    m2 = (m * m).sum(axis=1)
    E = m2 / (2 * rho) * (1 + rel)
    a = np.column_stack([rho, m, E])
    return a


def test_fast_test_never_accepts_what_the_reference_rejects():
    rng = np.random.default_rng(20261203)
    for gamma in (1.4, 5.0 / 3.0, 1.1, 50.0):
        for rel in (rng.uniform(-1e-9, 1e-9, 200000), rng.uniform(-1e-13, 1e-13, 200000),
                    rng.uniform(-1.0, 1.0, 200000), 10.0 ** rng.uniform(-16, 2, 200000)):
            a = states(len(rel), rng, rel)
            fast, ref = surely_admissible(a), reference_admissible(a, gamma)
            assert not np.any(fast & ~ref), int(np.sum(fast & ~ref))


def test_fast_test_accepts_ordinary_states():
    rng = np.random.default_rng(7)
    rho = rng.uniform(0.1, 10, 100000)
    u = rng.uniform(-3, 3, (100000, 3))
    p = rng.uniform(0.01, 10, 100000)
    E = p / 0.4 + 0.5 * rho * (u * u).sum(axis=1)
    a = np.column_stack([rho, rho[:, None] * u, E])
    assert surely_admissible(a).mean() > 0.999


def test_fast_test_rejects_extremes_and_non_finite_values():
    a = np.array([[1.0, 0, 0, 0, 1.0],          # ordinary
                  [0.0, 0, 0, 0, 1.0],          # ρ = 0
                  [-1.0, 0, 0, 0, 1.0],         # ρ < 0
                  [1.0, 2.0, 0, 0, 1.0],        # p < 0
                  [np.nan, 0, 0, 0, 1.0],
                  [1.0, 0, 0, 0, np.inf],
                  [1e-200, 0, 0, 0, 1e-200]])   # outside the bounded range: left to the full test
    assert list(surely_admissible(a)) == [True, False, False, False, False, False, False]


def test_fast_test_bounds():
    """2^±332 on ρ, E and |ρu|: beyond them the test leaves the state to the full one."""
    lo, hi = 2.0 ** -332, 2.0 ** 332
    below = np.nextafter
    ok = np.array([[lo, 0, 0, 0, 1.0], [1.0, 0, 0, 0, lo], [below(hi, 0), 0, 0, 0, 1.0], [below(hi, 0), 0, 0, 0, below(hi, 0)],
                   [below(hi, 0), 0, -below(hi, 0), 0, below(hi, 0)]])
    out = np.array([[below(lo, 0), 0, 0, 0, 1.0], [1.0, 0, 0, 0, below(lo, 0)], [hi, 0, 0, 0, 1.0], [1.0, 0, 0, 0, hi],
                    [1.0, hi, 0, 0, 1.0], [1.0, 0, -hi, 0, 1.0], [1.0, 0, 0, np.nan, 1.0], [1.0, 0, 0, -np.inf, 1.0]])
    assert surely_admissible(ok).all() and not surely_admissible(out).any()
