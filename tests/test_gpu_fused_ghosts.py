"""The fused ghost fill of the 3D mixed stages (k_mfill3_shell) with the hydrostatic
energy extrapolation on the low and the high face of each axis, at 3 cells an axis and
more, against the separate passes: bit for bit."""
import numpy as np
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import Solver, initial_conditions
from tests.golden_io import same

pytestmark = pytest.mark.gpu

GAS = [dict(gamma=1.4, M=0.02896, mu=1.8e-5), dict(gamma=1.67, M=0.004, mu=1.99e-5)]
P = ("periodic", "periodic")
# (low, high) face of x, y, z; the axis filled last is the last one that is not periodic
FACES = [(("outflow", "noslip"), ("noslip", "reflective"), ("hydrostatic", "hydrostatic")),
         (P, ("outflow", "reflective"), ("hydrostatic", "noslip")),
         (("reflective", "noslip"), P, ("outflow", "hydrostatic")),
         (P, ("hydrostatic", "hydrostatic"), P),
         (("noslip", "outflow"), ("reflective", "hydrostatic"), P),
         (("hydrostatic", "outflow"), P, P),
         (("outflow", "hydrostatic"), P, P)]


@pytest.mark.parametrize("n", [(37, 18, 11), (3, 9, 10), (35, 3, 8), (8, 7, 3), (3, 3, 3)])
@pytest.mark.parametrize("faces", FACES)
def test_fused_hydrostatic_fill_matches_separate_passes(faces, n, monkeypatch):
    cfg = abi.make_config(3, n, dx=(1 / 32,) * 3, dt=2e-7, species=GAS, visc=True, ceq=True,
                          periodic=tuple(f == P for f in faces),
                          bcs=tuple("outflow" if t == "periodic" else t for f in faces for t in f),
                          mode=abi.MODE_MIXED)
    U = initial_conditions(cfg, abi.IC_MIXING_3D, 3, p_ambient=1e5, T_ambient=300.0, nkernels=3)
    out = []
    for unfused in (False, True):
        if unfused:
            monkeypatch.setenv("FST_MIXED_UNFUSED", "1")
        s = Solver(cfg)
        s.set_state(U)
        s.set_profiling(True)
        s.rk_step(3)
        assert ("mfill3d_shell" in s.kernel_times()) != unfused
        out.append(s.get_state())
        s.rk_step(1)  # the ghosts of the state itself again, after a read
        out.append(s.get_state())
        s.close()
    assert np.isfinite(out[0]).all()
    assert same(out[0], out[2]) and same(out[1], out[3])
