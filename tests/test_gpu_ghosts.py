"""The one-launch ghost fill (fst_bc_dev.cuh GhostRule) and its fused form in the
3D mixed stages: every mix of boundary types and periodic axes, at the least
extents it takes (3 cells) and below them (the fills one after another)."""
import itertools

import numpy as np
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import Solver, initial_conditions
from oracle.oracle import Oracle
from tests.golden_io import same

pytestmark = pytest.mark.gpu

GAS = [dict(gamma=1.4, M=0.02896, mu=1.8e-5), dict(gamma=1.67, M=0.004, mu=1.99e-5)]
KINDS = ("periodic", "outflow", "reflective", "noslip", "hydrostatic")


def _config(nd, n, kinds, mode=abi.MODE_PLAIN_FP64, ceq=True):
    per = tuple(k == "periodic" for k in kinds) + (False,) * (3 - nd)
    lo = ["outflow" if k == "periodic" else k for k in kinds]
    # another type on the high face of a non-periodic axis
    hi = ["outflow" if k == "periodic" else KINDS[1 + (KINDS.index(k)) % 3] for k in kinds]
    bcs = [t for p in zip(lo, hi) for t in p] + ["outflow"] * (6 - 2 * nd)
    return abi.make_config(nd, n, dx=(1 / 32,) * nd, dt=2e-7, species=GAS, visc=True, ceq=ceq,
                           periodic=per, bcs=tuple(bcs), mode=mode)


@pytest.mark.parametrize("nd,n", [(2, (3, 3)), (2, (5, 9)), (2, (2, 7)), (3, (3, 3, 3)), (3, (7, 4, 5)),
                                  (3, (2, 4, 3))])
def test_fill_matches_oracle(nd, n):
    rng = np.random.default_rng(1)
    for kinds in itertools.product(KINDS, repeat=nd):
        cfg = _config(nd, n, kinds)
        U = np.asfortranarray(rng.uniform(0.5, 2.0, abi.dims(cfg)))
        U[..., :nd] -= 1.25
        o, g = Oracle(cfg), Solver(cfg)
        for x in (o, g):
            x.set_state(U)
            x.apply_bcs()
        assert same(g.get_state(), o.get_state()), kinds
        g.close()


@pytest.mark.parametrize("kinds", [("periodic", "reflective", "noslip"), ("noslip", "periodic", "outflow"),
                                   ("reflective", "noslip", "periodic"), ("hydrostatic", "outflow", "periodic")])
@pytest.mark.parametrize("ceq", [False, True])
def test_fused_fill_matches_separate_passes(kinds, ceq, monkeypatch):
    n = (37, 18, 11)
    cfg = _config(3, n, kinds, abi.MODE_MIXED, ceq)
    U = initial_conditions(cfg, abi.IC_MIXING_3D, 3, p_ambient=1e5, T_ambient=300.0, nkernels=3)
    out = []
    for unfused in (False, True):
        if unfused:
            monkeypatch.setenv("FST_MIXED_UNFUSED", "1")
        s = Solver(cfg)
        s.set_state(U)
        s.rk_step(3)
        out.append(s.get_state())
        s.rk_step(1)  # the ghosts of the state itself again, after a read
        out.append(s.get_state())
    assert np.isfinite(out[0]).all()
    assert same(out[0], out[2]) and same(out[1], out[3])
