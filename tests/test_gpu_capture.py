"""The allocation-free step, whose kernels are dependent launches, on the streams a
caller may give it: the legacy and the per-thread default stream, and inside a
stream capture, between the caller's own kernels and after the join of a side
stream (needs a B200)."""
import ctypes as C

import numpy as np
import pytest

from emergence_b200 import _abi
from emergence_b200 import workloads as W
from emergence_b200.physics import FluxMode, Precision
from emergence_b200.solver import _c_bcs, _c_eos, _c_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [Precision.F64, Precision.Mixed, Precision.F64Fast])
@pytest.mark.parametrize("n", [(48, 48, 1), (400, 1, 1), (20, 24, 18)])
def test_steps_agree_on_every_stream_and_in_a_capture(n, precision):
    import torch
    s, mesh, u, bc = W.explosion(n, 0.3)
    args = _c_mesh(mesh), _c_eos(s.eos), _c_bcs(bc), _abi.EmgOpts(0.5, 1e-3, FluxMode.Weno, 1, precision, 0)
    dt = 0.1 * min(mesh.dx[d] for d in range(3) if n[d] > 1)
    start = torch.from_numpy(np.ascontiguousarray(u.T)).cuda()
    bufs = [torch.empty_like(start) for _ in range(3)]

    def steps(first, stream):
        m, e, b, o = args
        for a, z in zip([first] + bufs, bufs):
            _abi.check(_abi.lib().emg_uniform_step_noalloc(C.byref(m), C.byref(e), b, C.byref(o), a.data_ptr(),
                                                           z.data_ptr(), dt, stream))
        return bufs[-1]

    torch.cuda.synchronize()
    want = steps(start, 0).clone()  # legacy default stream
    torch.cuda.synchronize()
    steps(start, 2)  # cudaStreamPerThread
    torch.cuda.synchronize()
    assert torch.equal(bufs[-1], want)

    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=main):
        side.wait_stream(main)
        with torch.cuda.stream(side):
            copy = start * 1.0
        main.wait_stream(side)
        result = steps(copy, main.cuda_stream) * 1.0
    for _ in range(3):
        for b in bufs + [result]:
            b.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(result, want)
