"""The 2D cell pass bit for bit with the oracle on both sides of its dispatch (4256
blocks of 32x4 cells, all roles counted), at ragged rows."""
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import Solver, initial_conditions
from oracle.oracle import Oracle
from tests.golden_io import same

GAS = [dict(gamma=1.4, M=0.02896, mu=1.8e-5), dict(gamma=1.67, M=0.004, mu=1.99e-5)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,ceq", [((703, 256), True), ((703, 259), True), ((677, 401), False)])
def test_gpu_plain2d_on_both_sides_of_the_dispatch(n, ceq):
    cfg = abi.make_config(2, n, dx=(1 / 700, 1 / 300), dt=1e-7, species=GAS, visc=True, ceq=ceq, buoyancy=True)
    U = initial_conditions(cfg, abi.IC_RANDOM_SMOOTH, 3)
    o, g = Oracle(cfg), Solver(cfg)
    for x in (o, g):
        x.set_state(U)
        x.apply_bcs()
    assert same(g.compute_rhs(), o.compute_rhs())
    o.rk_step(1)
    g.rk_step(1)
    assert same(g.get_state(), o.get_state())
