"""The 3D noise removal bit for bit with the oracle: at partial tiles, with every
combination of filtered variables left to visit, and with values at which the quotients
and the doubled centre leave the fast arithmetic's range."""
import itertools

import numpy as np
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import Solver, initial_conditions
from oracle.oracle import Oracle
from tests.test_noise import _same_bits

pytestmark = pytest.mark.gpu


def run(cfg, U, mode, nt):
    o, s = Oracle(cfg), Solver(cfg)
    for x in (o, s):
        x.set_state(U)
        x.noise_filter(1e-3, 0.1, 0.0, nt, mode)
    assert _same_bits(s.get_state(), o.get_state())
    return U, o.get_state()


def config(n):
    return abi.make_config(3, n, dx=(1 / n[0], 0.9 / n[1], 1.3 / n[2]), dt=1e-4,
                           species=[dict(gamma=1.4, M=1.0, mu=1e-3)], R=1.0)


@pytest.mark.parametrize("n", [(7, 9, 16), (17, 8, 5), (8, 8, 8), (25, 16, 9)])
@pytest.mark.parametrize("rough", [c for m in (1, 2, 3) for c in itertools.combinations(range(3), m)])
def test_variables_left_to_visit(n, rough):
    cfg = config(n)
    U = np.array(initial_conditions(cfg, abi.IC_RANDOM_SMOOTH, 2), order="F")
    U[..., :3] = 0.5
    rng = np.random.default_rng(3)
    for v in rough:
        U[..., v] += 0.05 * rng.standard_normal(U.shape[:3])
    U, V = run(cfg, U, 1, 2)
    for v in range(3):
        assert (U[..., v] != V[..., v]).any() == (v in rough)


@pytest.mark.parametrize("n,mode", [((18, 11, 10), 1), ((9, 17, 8), 2)])
@pytest.mark.parametrize("scale", [1.0, 1e-300, 5e-324 * 1e16])
def test_values_out_of_the_fast_range(n, mode, scale):
    cfg = config(n)
    rng = np.random.default_rng(6)
    U = np.array(initial_conditions(cfg, abi.IC_RANDOM_SMOOTH, 2), order="F")
    v = 0 if mode == 1 else 3
    U[..., v] = (1 + 0.05 * rng.standard_normal(U.shape[:3])) * scale
    at = [tuple(rng.integers(3, 3 + m) for m in n) for _ in range(9)]
    for p, x in zip(at, (1.5e308, -1.2e308, 9.1e307, 5e-324, -3e-310, 0.0, -0.0, np.inf, np.nan)):
        U[p + (v,)] = x
    run(cfg, U, mode, 1)
