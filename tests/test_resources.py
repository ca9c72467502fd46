"""What ptxas reports for the kernels whose speed hangs on it: registers (warps in
flight).  Compiles the units here; no GPU."""
import os
import re
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

from fiesta_gb300 import build

pytestmark = pytest.mark.skipif(shutil.which(build.NVCC) is None, reason="nvcc not found")
EXTRA = dict(build.UNITS)


def _ptxas(unit, tmp):
    """ptxas -v of a unit: [(mangled kernel name, registers)] and the whole text."""
    r = subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "--extended-lambda", "-Xptxas", "-v",
                        *EXTRA[unit], "-I", build.CSRC, "-c", os.path.join(build.CSRC, unit), "-o",
                        os.path.join(tmp, unit + ".o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    regs = re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", r.stderr, re.S)
    return [(name, int(n)) for name, n in regs], r.stderr


def _resident(regs, threads):
    """Threads of such blocks that an SM's 65,536 registers hold."""
    return 65536 // (-(-regs // 8) * 8 * threads) * threads


def test_2d_tile_keeps_its_warps(tmp_path):
    """Both faces' reconstructions side by side raise the tile's registers; the launch
    bounds hold 1024 threads an SM for every variable count, with learned routing too."""
    units = ["fst_mixed.cu", "fst_batch_w16.cu", "fst_batch_w32.cu", "fst_batch_w64.cu"]
    with ThreadPoolExecutor(len(units)) as ex:
        found = [k for regs, _ in ex.map(lambda u: _ptxas(u, str(tmp_path)), units) for k in regs]
    seen = 0
    for name, regs in found:
        single = re.search(r"k_mrhs2dILi(\d+)ELb[01]E", name)
        batch = re.search(r"k_brhsILi(\d+)ELi(\d+)ELi(\d+)E", name)
        if not (single or batch):
            continue
        seen += 1
        threads = 256 if single else int(batch.group(2)) * int(batch.group(3))
        assert _resident(regs, threads) >= 1024, (name, regs)
    assert seen == 14 + 48  # 7 variable counts with and without routing; 6 counts, 8 shapes


def _primitive_passes(tmp):
    """[(is k_bprim, species or 0 for any number, registers)] of the 2D primitive passes."""
    out = []
    for name, regs in _ptxas("fst_batch.cu", tmp)[0] + _ptxas("fst_mixed.cu", tmp)[0]:
        m = re.search(r"(k_bprimI|k_mprimILi2E)Li(\d+)E", name)
        if m:
            out.append((m.group(1) == "k_bprimI", int(m.group(2)), regs))
    return out


def test_any_species_primitive_pass_keeps_its_warps(tmp_path):
    """The passes whose species count is not known at compile time: their loops are not
    unrolled 16 times."""
    found = [(batch, regs) for batch, ns, regs in _primitive_passes(str(tmp_path)) if ns == 0]
    assert len(found) == 2
    for batch, regs in found:
        assert _resident(regs, 256) >= (768 if batch else 1024), (batch, regs)


def test_primitive_passes_keep_their_warps(tmp_path):
    """The passes of 1 to 5 species."""
    found = [(batch, ns, regs) for batch, ns, regs in _primitive_passes(str(tmp_path)) if ns > 0]
    assert len(found) == 10
    for batch, ns, regs in found:
        assert _resident(regs, 256) >= (768 if batch else 1024), (batch, ns, regs)
