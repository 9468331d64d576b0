"""Replayed builds, whose graph has two branches, before and after the tuning changes (the graph is recorded again): every buffer as in
the first build, launched one kernel after another; small builds (one block sorts them) and larger ones."""
import numpy as np
import pytest

from sesdf_gb300 import SesBuild, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["full", "exterior"])
@pytest.mark.parametrize("n", [700, 8192, 8193])
def test_replays(n, mode):
    atoms = synth.globule(n, 91)
    with SesBuild(atoms, 1.4, mode) as g:
        g.build()
        want = g.fetch()
        knobs = g.tuning()
        for change in ({}, {"probe_warps": 2, "probe_queue": 1}, {"neighbor_warps": 4, "visibility_warps": 2}, knobs):
            g.set_tuning(**change)
            for _ in range(3):
                g.build()
            got = g.fetch()
            assert got.keys() == want.keys()
            for k in want:
                assert k == "counts" or np.array_equal(got[k], want[k], equal_nan=want[k].dtype.kind == "f"), (k, change)
            assert [got["counts"][k] for k in ("probes", "segments", "tori", "pairs")] == [want["counts"][k] for k in ("probes", "segments", "tori", "pairs")]
