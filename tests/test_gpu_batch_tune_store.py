"""Which stored choices of the ensemble autotuner are reused."""
import json
import re

import pytest

from fiesta_gb300.batch import Batch, rt_ensemble

pytestmark = pytest.mark.gpu


def _tuned(cfgs, states, path):
    b = Batch(cfgs)
    for c, U in enumerate(states):
        b.set_state(c, U)
    shape = b.tune(path)
    with open(path) as f:
        return shape, json.load(f)["entries"]


def test_choice_of_another_tile_kernel_is_not_reused(tmp_path):
    cfgs, states = rt_ensemble(ncases=2, nmin=24, nmax=40, seed=3)
    path = str(tmp_path / "tune.json")
    _, (entry,) = _tuned(cfgs, states, path)
    # the entry of a kernel without a version in its key, and of an earlier version: a shape
    # and a time of their own
    bare = re.sub(r"\|tile=\d+", "", entry["key"])
    old = [dict(entry, key=k, tile_width=64, tile_height=4, blocks_per_sm=1, best_ms=1e-6, candidates=1)
           for k in (bare, bare + "|tile=1")]
    with open(path, "w") as f:
        f.write('{"entries": [\n' + ",\n".join("  " + json.dumps(e) for e in old) + "\n]}\n")
    shape, entries = _tuned(cfgs, states, path)
    assert [e["key"] for e in entries] == [bare, bare + "|tile=1", entry["key"]]  # the others stay
    assert entries[2]["best_ms"] > 1e-6 and entries[2]["candidates"] > 8
    assert shape == tuple(entries[2][k] for k in ("tile_width", "tile_height", "blocks_per_sm"))


def test_buoyancy_has_its_own_choice(tmp_path):
    """The switch adds loads and work to the tile."""
    cfgs, states = rt_ensemble(ncases=2, nmin=24, nmax=40, seed=3)
    path = str(tmp_path / "tune.json")
    assert len(_tuned(cfgs, states, path)[1]) == 1
    for cfg in cfgs:
        cfg.buoyancy = 0
    assert len(_tuned(cfgs, states, path)[1]) == 2
