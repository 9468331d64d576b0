"""Builds whose head runs in one block (up to 8192 atoms of one molecule) against the general path, which a batch takes:
sizes at the edges of its items per thread, of a warp and of the largest size, atoms in one cell and far apart (a grid that is
coarsened to the counters), atoms outside the reference grid, and both modes; buffer for buffer, bit for bit."""
import numpy as np
import pytest

import canon
from sesdf_gb300 import SesBatch, SesBuild, synth
from test_gpu_batch import compare

pytestmark = pytest.mark.gpu


def sparse(n, span, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.uniform(-span, span, (n, 3)), rng.uniform(1.1, 2.0, (n, 1))], 1).astype(np.float32)


def line(n):
    x = 1.5 * np.arange(n, dtype=np.float32)
    return np.stack([x, np.zeros(n, np.float32), np.zeros(n, np.float32), np.full(n, 1.6, np.float32)], 1)


SETS = {
    "edges": lambda: [synth.globule(n, 3000 + n) for n in (1, 2, 31, 33, 511, 1024, 2047, 2048, 2049)],
    "larger": lambda: [synth.globule(n, 3000 + n) for n in (4095, 4097, 8191, 8192, 8193)],
    "sparse": lambda: [sparse(600, 60.0, 1), sparse(3000, 900.0, 2), sparse(8192, 250.0, 3), line(5000)],
}


@pytest.mark.parametrize("mode", ["full", "exterior"])
@pytest.mark.parametrize("name", sorted(SETS))
def test_front_matches_general(name, mode):
    mols = SETS[name]()
    with SesBatch(mols, 1.4, mode) as g:
        g.build()
        compare(g, mols, mode)


@pytest.mark.parametrize("mode", ["full", "exterior"])
@pytest.mark.parametrize("n", [700, 5000, 12000])
def test_moved_atoms_and_replay(n, mode):
    # the recorded build (with the probes' neighbours beside the segments or tori) sees new positions and other
    # radii on each pass, some outside the grid of the first ones
    a, b = synth.globule(n, 71), synth.globule(n, 72)
    b[:, 3] *= 1.1
    b[:5, :3] += 40.0
    names = ["atoms", "perm", "probe_pos", "probe_ids"]
    names += ["sectors", "segments"] if mode == "full" else ["tori_pos", "tori_axis", "tori_vs"]
    with SesBuild(a, 1.4, mode) as g, SesBuild(a, 1.4, mode, graph=False) as h:
        for atoms in (a, b, a):
            out = []
            for k in (g, h):
                k.set_atoms(atoms)
                k.build()
                out.append(k.fetch(analysis=True))
            x, y = out
            for k in names:
                assert np.array_equal(x[k], y[k], equal_nan=True), k
            q = x["counts"]["singular_probes"]
            assert np.array_equal(canon.written_probe_nbrs(x["probe_nbrs"], x["probe_ids"], q),
                                  canon.written_probe_nbrs(y["probe_nbrs"], y["probe_ids"], q))
