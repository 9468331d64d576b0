"""Probe candidates left open by float32, settled with four lanes per triplet up to 24,576 of them and by a thread each
beyond: both sides of the line against the oracle, with atom lists of one and of several steps of 32 neighbours, and clusters whose
triplets are degenerate (no solution, coplanar, equal distances)."""
import numpy as np
import pytest

from cases import hand_cases
from oracle import oracle
from sesdf_gb300 import SesBuild, synth
from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def lattice(n, spacing, r):
    g = np.arange(n, dtype=np.float32) * spacing
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return np.concatenate([xyz, np.full((len(xyz), 1), r, np.float32)], 1)


CASES = {
    "few": (lambda: synth.globule(700, 8101), 1.4),
    "long lists": (lambda: synth.globule(900, 8102), 2.4),
    "short lists": (lambda: synth.globule(900, 8103), 0.6),
    "cluster": (lambda: hand_cases()["cluster40"], 1.4),
    "lattice": (lambda: lattice(5, 3.7, 1.7) + np.random.default_rng(4).normal(0, 1e-4, (125, 4)).astype(np.float32) * [1, 1, 1, 0], 1.4),
}


@pytest.mark.parametrize("mode", ["full", "exterior"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_open_candidates(name, mode):
    make, rp = CASES[name]
    atoms = np.asarray(make(), np.float32)
    with SesBuild(atoms, rp, mode) as g:
        g.build()
        out = g.fetch()
        box = g.box
    compare(atoms, out, oracle.run(atoms, rp, mode, box=box), mode)


def test_many_open_candidates_match_small_builds():
    # 20 copies of one molecule side by side leave more candidates open than the line; a copy alone leaves fewer
    from sesdf_gb300 import SesBatch
    from test_gpu_batch import compare as same
    mols = [synth.globule(11000, 8104)] * 20
    with SesBatch(mols, 1.4, "full") as b:
        b.build()
        same(b, mols[:1], "full")
