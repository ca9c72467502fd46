"""The mixed path's FP64 <-> FP32 conversions (csrc/fst_conv.cuh) on the host, against
NumPy, at the edges of their ranges; on the GPU, a state beyond the FP32 range takes
the general equation of state."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fiesta_gb300 import abi
from fiesta_gb300.solver import Solver, initial_conditions

HERE = os.path.dirname(os.path.abspath(__file__))


def test_conversions(tmp_path):
    so = str(tmp_path / "conv_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    os.path.join(HERE, "cpp", "conv_check.cpp"), "-o", so], check=True)
    r = np.random.default_rng(11)
    n = 400_000
    ex = r.integers(0, 2048, n).astype(np.uint64)
    ex[: n // 2] = r.integers(890, 1160, n // 2)  # the FP32 range and its edges
    m = r.integers(0, 1 << 52, n, dtype=np.uint64)
    m[::5] |= np.uint64((1 << 52) - (1 << 28))     # rounds into the exponent
    m[1::5] = (m[1::5] >> np.uint64(29) << np.uint64(29)) | np.uint64(1 << 28)  # ties
    m[2::5] &= ~np.uint64((1 << 29) - 1)           # exact
    x = (r.integers(0, 2, n).astype(np.uint64) << np.uint64(63) | ex << np.uint64(52) | m).view(np.float64)
    x[:6] = 0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324
    y = r.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)
    y[:6] = 0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45
    out = [np.empty(n, t) for t in (np.float32, np.float64) + (np.float32,) * 4]
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    C.CDLL(so).conv_check(C.c_longlong(n), p(x), p(y), *map(p, out))
    f, d, h, l, hr, lr = out

    e = (x.view(np.uint64) >> np.uint64(52)) & np.uint64(2047)
    # nearest, ties away: half a unit added to the mantissa, the rest cut off
    near = ((x.view(np.uint64) + np.uint64(1 << 28)) >> np.uint64(29) << np.uint64(29)).view(np.float64)
    with np.errstate(over="ignore", invalid="ignore"):
        want = np.where(e < 897, np.copysign(np.float32(0), x), np.where(e > 1150, np.copysign(np.inf, x), near)).astype(np.float32)
    want[np.isnan(x)] = np.nan
    bits = lambda a: np.where(np.isnan(a), np.uint32(0x7FC00000), a.view(np.uint32))
    assert np.array_equal(bits(f), bits(want)) and np.array_equal(bits(h), bits(want))
    tiny = np.abs(y) < np.float32(2.0 ** -126)
    with np.errstate(invalid="ignore"):
        wd = np.where(tiny, np.copysign(0.0, y), y.astype(np.float64))
    assert np.array_equal(np.isnan(d), np.isnan(y)) and np.array_equal(d[~np.isnan(y)].view(np.uint64), wd[~np.isnan(y)].view(np.uint64))

    ok = e < 1151
    assert np.array_equal(h[ok].view(np.uint32), hr[ok].view(np.uint32)) and np.array_equal(l[ok], lr[ok])
    none = (e < 921) | (e > 1150)
    assert np.all(l[none] == 0)
    # x with its 6 lowest bits cut, less h (exact in FP64); the host does not flush denormals
    s = ~none & np.isfinite(h)
    cut = (x.view(np.uint64) >> np.uint64(6) << np.uint64(6)).view(np.float64)
    assert np.array_equal(l[s], (cut[s] - h[s].astype(np.float64)).astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("ns", [1, 3, 5, 6])
def test_gpu_state_beyond_fp32(ns):
    """One cell out of the FP32 range spoils itself and what its stencils reach, not the
    cells that share its warp."""
    gas = [dict(gamma=1.4 - 0.02 * s, M=0.029 + 0.002 * s, mu=1.8e-5) for s in range(ns)]
    n = (40, 9, 7)
    cfg = abi.make_config(3, n, dx=(1 / 40, 1 / 9, 1 / 7), dt=1e-7, species=gas, visc=True, ceq=False,
                          mode=abi.MODE_MIXED)
    U = initial_conditions(cfg, abi.IC_RANDOM_SMOOTH, 3)
    V = np.array(U, order="F")
    V[4, 4, 4, 0], V[4, 4, 4, 3] = 1e39, np.inf
    res = []
    for u in (U, V):
        s = Solver(cfg)
        s.set_state(u)
        s.rk_step(1)
        res.append(s.get_state())
    far = np.s_[20:34, 3:-3, 3:-3]
    assert np.isfinite(res[0][far]).all()
    assert np.array_equal(res[0][far], res[1][far])
    assert not np.isfinite(res[1][4, 4, 4]).all()
