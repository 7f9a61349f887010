"""Downloads into pageable memory go through a pinned buffer emptied by several
host threads above 8 MB (emergence_b200/csrc/host_copy.cu): the same bytes as a
direct copy into pinned memory, at sizes around the threshold and the 2 MB
slots, and from two handles at once (needs a B200)."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from emergence_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _solver(n, seed):
    from emergence_b200 import GpuSolver
    s, mesh, u, bc = W.explosion(n, 0.3, seed=seed)
    return GpuSolver(s, mesh, u, bc=bc), mesh, u


# bytes: 8 below the threshold, a plain copy; 32 above, four slots and a rest; sixteen
# slots less 32 and plus 8 bytes; four slots and a bit; more than two rounds of them
@pytest.mark.parametrize("n,staged", [((209703, 1, 1), False), ((209704, 1, 1), True), ((838848, 1, 1), True),
                                      ((838849, 1, 1), True), ((500, 403, 1), True), ((128, 111, 119), True)])
def test_pageable_download_equals_the_pinned_one(n, staged):
    import torch
    g, mesh, u = _solver(n, 3)
    assert (mesh.len() * 40 >= 8 << 20) == staged
    pin = torch.empty((mesh.len(), 5), dtype=torch.float64, pin_memory=True).numpy()
    g.download(out=pin)
    out = np.full((mesh.len(), 5), np.nan)
    assert np.array_equal(g.download(out=out), pin)
    assert np.array_equal(mesh.interior(out), mesh.interior(u))


def test_two_handles_download_at_once():
    pairs = [_solver((64, 64, 64), k) for k in (1, 2)]
    bad = []

    def run(g, mesh, u):
        for _ in range(5):
            if not np.array_equal(mesh.interior(g.download()), mesh.interior(u)):
                bad.append(1)

    t = [threading.Thread(target=run, args=p) for p in pairs]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not bad


def test_released_buffer_comes_back():
    from emergence_b200.solver import release_memory
    g, mesh, u = _solver((64, 64, 64), 5)
    a = g.download()
    release_memory()
    assert np.array_equal(g.download(), a)


RESET = """
import ctypes
import numpy as np
from emergence_b200 import GpuAmr, GpuBatch1D, workloads as W

def results():
    sys_, n, dx, u, _ = W.riemann_batch(ninst=1024, nmax=2048)
    b = GpuBatch1D(sys_, n, dx, u)
    a = GpuAmr(*W.shock_bubble(dim=2, base=4, levels=2))
    a.step(a.dt_cfl())
    out = b.download(), a.download()
    assert out[0].nbytes > 2 * (8 << 20)  # staged
    b.close(), a.close()
    return out

first = results()
assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0
assert all(np.array_equal(x, y) for x, y in zip(first, results()))
print("same")
"""


def test_downloads_outlive_a_device_reset():
    """The page-locked buffer is the process's: after the context it was locked in
    has gone, the next download locks it again."""
    root = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")
    r = subprocess.run([sys.executable, "-c", RESET], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
