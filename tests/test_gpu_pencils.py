"""The uniform sweeps tile the pencils of a whole cross-section one row after
another (uniform.cu sweep_grid, five.cu plan): cross-sections whose rows are no
multiple of the tile, smaller than one tile, and of one more or one less pencil
than a tile, against the CPU oracle bit for bit (needs a B200)."""
import numpy as np
import pytest

from emergence_b200 import workloads as W
from emergence_b200.physics import FluxMode
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(9, 3, 11), (7, 31, 5), (6, 33, 3), (40, 2, 2), (5, 17, 2), (12, 8, 4), (50, 33, 1), (2, 70, 1), (31, 1, 1)]


@pytest.mark.parametrize("n", SHAPES)
@pytest.mark.parametrize("mode", [FluxMode.Weno, FluxMode.Hybrid])
def test_ragged_cross_sections(n, mode):
    from emergence_b200 import GpuSolver
    s, mesh, u, bc = W.explosion(n, 0.3)
    g, o = GpuSolver(s, mesh, u, bc=bc, mode=mode), O.OracleSolver(s, mesh, u, bc=bc, mode=mode)
    for _ in range(2):
        dt = o.dt_cfl()
        assert g.dt_cfl() == dt
        g.step(dt)
        o.step(dt)
    assert np.array_equal(mesh.interior(g.download()), mesh.interior(o.download()))
    assert g.counters() == o.counters()


@pytest.mark.parametrize("n", [5, 9, 13])
def test_ragged_cross_sections_of_the_five_equation_sweep(n):
    from emergence_b200.five import GpuFiveSolver
    s, mesh, u, bc = W.two_phase_shock_bubble(n)
    g, o = GpuFiveSolver(s, mesh, u, bc=bc), O.FiveOracleSolver(s, mesh, u, bc=bc)
    dt = o.dt_cfl()
    assert g.dt_cfl() == dt
    g.step(dt)
    o.step(dt)
    assert np.array_equal(mesh.interior(g.download()), mesh.interior(o.download()))
