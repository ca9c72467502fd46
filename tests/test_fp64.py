"""The integer-pipe FP64 arithmetic (csrc/fst_fp64.cuh) and the marching WENO5
flux built on it (csrc/fst_flux_dev.cuh): the operations against the CPU's IEEE
arithmetic on the host, the flux against the oracle bit for bit at the edges of
its launch plan (line chunks of 32, segments) and of its value range."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import Solver, initial_conditions
from oracle.oracle import Oracle
from tests.golden_io import same

HERE = os.path.dirname(os.path.abspath(__file__))


def test_operations_round_as_ieee(tmp_path):
    so = str(tmp_path / "fp64_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    os.path.join(HERE, "cpp", "fp64_check.cpp"), "-o", so], check=True)
    fn = C.CDLL(so).fp64_check
    fn.restype, fn.argtypes = C.c_longlong, [C.c_longlong, C.c_uint64]
    assert fn(2_000_000, 20240607) == 0


GAS = [dict(gamma=1.4, M=0.02896, mu=1.8e-5), dict(gamma=1.67, M=0.004, mu=1.99e-5),
       dict(gamma=1.3, M=0.044, mu=1.5e-5), dict(gamma=1.32, M=0.016, mu=1.1e-5),
       dict(gamma=1.4, M=0.002, mu=0.9e-5), dict(gamma=1.35, M=0.03, mu=1.0e-5)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,ns,dx", [
    ((1, 1, 1), 1, 0.25), ((31, 3, 2), 2, 1 / 31), ((32, 33, 5), 5, 1 / 32), ((63, 2, 34), 6, 0.1),
    ((7, 65, 3), 3, 1 / 64), ((1, 1), 1, 0.25), ((33, 31), 2, 1 / 33), ((64, 130), 4, 1 / 64)])
@pytest.mark.parametrize("extremes", [False, True])
def test_gpu_flux_plan_edges_and_value_range(n, ns, dx, extremes):
    nd = len(n)
    cfg = abi.make_config(nd, n, dx=(dx,) * nd, dt=1e-6, species=GAS[:ns], visc=True, ceq=nd == 3)
    U = initial_conditions(cfg, abi.IC_RANDOM_SMOOTH, 3)
    if extremes:
        # tiny, huge, zero and non-finite momenta and one energy: the stencils around
        # them leave the fast path's range
        rng = np.random.default_rng(5)
        I = U[3:-3, 3:-3, 3:-3] if nd == 3 else U[3:-3, 3:-3]
        for v, x in ((0, 1e-70), (1, -1e-61), (0, 0.0), (1, 3e47), (0, 1e160), (0, np.inf), (1, np.nan),
                     (nd, 2e45), (1, 5e-324), (0, -0.0)):
            at = tuple(rng.integers(0, s) for s in I.shape[:3])
            I[at + (v,)] = x
    o, g = Oracle(cfg), Solver(cfg)
    for x in (o, g):
        x.set_state(U)
        x.apply_bcs()
    assert same(g.compute_rhs(), o.compute_rhs())
    o.rk_step(2)
    g.rk_step(2)
    assert same(g.get_state(), o.get_state())
