"""The composed ghost fill (one launch for all axes, uniform.cu
ghost_all_kernel) against the CPU oracle's fill axis by axis, every padded cell
bit for bit: each copying boundary kind beside each other one, walls whose
momenta flip once or twice in edges and corners, periodic axes shorter than
their ghost layers (needs a B200)."""
import numpy as np
import pytest

from emergence_b200 import workloads as W
from emergence_b200.physics import Bc
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

FAR = W.explosion((8, 1, 1), 0.3)[0].to_cons(np.array([0.7, 0.2, -0.1, 0.3, 0.6]))
D = Bc.dirichlet(FAR)
P, X, R = Bc.Periodic, Bc.Outflow, Bc.Reflect
SIDES = {
    "walls": [[R, R], [R, R], [R, R]],
    "mixed": [[D, X], [R, D], [X, R]],
    "far": [[D, D], [D, R], [R, D]],
    "periodic": [[P, P], [R, X], [P, P]],
}


@pytest.mark.parametrize("name", list(SIDES))
@pytest.mark.parametrize("n", [(9, 7, 8), (6, 11, 6), (13, 9, 1), (1, 8, 10)])
def test_every_ghost_cell_matches_the_axis_by_axis_fill(name, n):
    from emergence_b200 import GpuSolver
    s, mesh, u, _ = W.explosion(n, 0.3, noise=0.3)
    ui = mesh.interior(u)
    rng = np.random.default_rng(1)
    ui[..., 1:4] = 0.02 * rng.uniform(-1.0, 1.0, ui[..., 1:4].shape)  # momenta of every sign, pressures stay positive
    bc = SIDES[name]
    g, o = GpuSolver(s, mesh, u, bc=bc), O.OracleSolver(s, mesh, u, bc=bc)
    for _ in range(2):
        dt = o.dt_cfl()
        g.step(dt)
        o.step(dt)
        assert np.array_equal(g.download(), o.download())


@pytest.mark.parametrize("n", [(4, 9, 1), (9, 3, 5)])
def test_periodic_axes_shorter_than_the_ghost_layers(n):
    from emergence_b200 import GpuSolver
    s, mesh, u, _ = W.explosion(n, 0.3, noise=0.3)
    bc = [[P, P]] * 3
    g, o = GpuSolver(s, mesh, u, bc=bc), O.OracleSolver(s, mesh, u, bc=bc)
    dt = o.dt_cfl()
    g.step(dt)
    o.step(dt)
    assert np.array_equal(g.download(), o.download())
