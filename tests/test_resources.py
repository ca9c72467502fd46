"""What the kernels' speed hangs on and no result shows: the registers and spills that
ptxas reports, constant memory.  Compiles the units here; no GPU."""
import os
import re
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

from fiesta_gb300 import build

pytestmark = pytest.mark.skipif(shutil.which(build.NVCC) is None, reason="nvcc not found")
EXTRA = dict(build.UNITS)


UNITS = ["fst_mixed.cu", "fst_batch.cu", "fst_batch_w16.cu", "fst_batch_w32.cu", "fst_batch_w64.cu"]


@pytest.fixture(scope="module")
def ptxas(tmp_path_factory):
    """What ptxas -v says of the units: {unit: (its text, [(mangled kernel, registers, bytes spilled)])}."""
    tmp = str(tmp_path_factory.mktemp("ptxas"))

    def compile(unit):
        r = subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "--extended-lambda", "-Xptxas", "-v",
                            *EXTRA[unit], "-I", build.CSRC, "-c", os.path.join(build.CSRC, unit), "-o",
                            os.path.join(tmp, unit + ".o")], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-2000:]
        found = re.findall(r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores.*?Used (\d+) registers",
                           r.stderr, re.S)
        return r.stderr, [(name, int(regs), int(spill)) for name, spill, regs in found]

    with ThreadPoolExecutor(len(UNITS)) as ex:
        return dict(zip(UNITS, ex.map(compile, UNITS)))


def _resident(regs, threads):
    """Threads of such blocks that an SM's 65,536 registers hold."""
    return 65536 // (-(-regs // 8) * 8 * threads) * threads


def _tiles(ptxas):
    """[(kernel, variables, threads a block, registers, bytes spilled)] of the 2D tile."""
    for _, kernels in ptxas.values():
        for name, regs, spill in kernels:
            m = re.search(r"(k_mrhs2d|k_brhs)ILi(\d+)EL([ib])(\d+)EL?i?(\d+)?", name)
            if m:
                threads = 256 if m.group(1) == "k_mrhs2d" else int(m.group(4)) * int(m.group(5))
                yield name, m.group(1) == "k_mrhs2d", int(m.group(2)), threads, regs, spill


def test_2d_tile_keeps_its_warps(ptxas):
    """The launch bounds hold 1024 threads an SM for every variable count, with learned
    routing too (but for the form of more than 9 variables for grids that need no more than
    two blocks an SM)."""
    tiles = [t for t in _tiles(ptxas) if not re.search(r"k_mrhs2dILi20ELb[01]ELi2E", t[0])]
    assert len(tiles) == 14 + 48  # 7 variable counts with and without routing; 6 counts, 8 shapes
    for name, _, _, threads, regs, _ in tiles:
        assert _resident(regs, threads) >= 1024, (name, regs)


def test_2d_tile_of_many_variables_does_not_spill(ptxas):
    """Both faces' reconstructions side by side need registers that single runs of 7 to 9
    variables, or with learned routing, do not have: one face after the other there."""
    for name, single, nv, _, _, spill in _tiles(ptxas):
        if single and nv <= 9 and (nv >= 7 or "Lb1E" in name):
            assert spill == 0, (name, spill)


def _primitive_passes(ptxas):
    """[(is k_bprim, species or 0 for any number, registers)] of the 2D primitive passes."""
    for _, kernels in ptxas.values():
        for name, regs, _ in kernels:
            m = re.search(r"(k_bprimI|k_mprimILi2E)Li(\d+)E", name)
            if m:
                yield m.group(1) == "k_bprimI", int(m.group(2)), regs


def test_any_species_primitive_pass_keeps_its_warps(ptxas):
    """The passes whose species count is not known at compile time: their loops are not
    unrolled 16 times."""
    found = [(batch, regs) for batch, ns, regs in _primitive_passes(ptxas) if ns == 0]
    assert len(found) == 2
    for batch, regs in found:
        assert _resident(regs, 256) >= (768 if batch else 1024), (batch, regs)


def test_primitive_passes_keep_their_warps(ptxas):
    """The passes of 1 to 5 species."""
    found = [(batch, ns, regs) for batch, ns, regs in _primitive_passes(ptxas) if ns > 0]
    assert len(found) == 10
    for batch, ns, regs in found:
        assert _resident(regs, 256) >= (768 if batch else 1024), (batch, ns, regs)


def test_no_unit_has_constant_memory():
    """A __constant__ variable costs every launch of every kernel of its unit 0.1 us."""
    for name in os.listdir(build.CSRC):
        with open(os.path.join(build.CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        assert "__constant__" not in code, name
