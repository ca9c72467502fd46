"""The 3D mixed kernels at the edges of their launch plan: fewer planes than a
block can march, a remainder, tiles of one column or row beyond a multiple (grids
of one or two planes have no finite reference: their ghosts mirror ghosts).  Against the FP64 oracle by the bar of tests/accuracy.py."""
import numpy as np
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import initial_conditions
from tests.accuracy import check_fields, run_pair

pytestmark = pytest.mark.gpu

GAS = [dict(gamma=1.4, M=0.02896, mu=1.8e-5), dict(gamma=1.67, M=0.004, mu=1.99e-5)]


@pytest.mark.parametrize("n", [(32, 8, 3), (63, 15, 17), (33, 20, 18), (64, 64, 40)])
@pytest.mark.parametrize("ceq", [False, True])
def test_mixed_launch_plan_edges(n, ceq):
    cfg = abi.make_config(3, n, dx=(1 / 64,) * 3, dt=2e-7, species=GAS, visc=True, ceq=ceq,
                          mode=abi.MODE_MIXED)
    U0 = initial_conditions(cfg, abi.IC_MIXING_3D, 3, p_ambient=1e5, T_ambient=300.0, nkernels=3)
    U, Ur, Up = run_pair(cfg, U0, 2)
    assert np.isfinite(U).all()
    check_fields(cfg, U, Ur, Up, U0)
