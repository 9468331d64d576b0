"""A batch that leaves more probe candidates open than four lanes each are given for (24,576): by count, and every molecule of it as its
own build, which leaves fewer, has it."""
import numpy as np
import pytest

from sesdf_gb300 import SesBatch, SesBuild, synth

pytestmark = pytest.mark.gpu
SOLVE, LINE = 4, 24_576  # place of the candidates' count in the double-precision decisions


def test_more_open_candidates_than_the_line():
    mols = [synth.globule(11000, 8104)] * 10 + [synth.globule(11000, 8105)] * 10
    with SesBatch(mols, 1.4, "full") as b:
        b.build()
        assert b.counts()["fp64_decisions"][SOLVE] > LINE
        got = [b.molecule(m) for m in range(len(mols))]
    for first in (0, 10):
        with SesBuild(mols[first], 1.4, "full") as g:
            g.build()
            want = g.fetch(analysis=False)
            assert 0 < g.counts()["fp64_decisions"][SOLVE] < LINE
        for m in range(first, first + 10):
            for k in ("probe_pos", "probe_ids", "segments", "sectors", "full"):
                assert np.array_equal(got[m][k], want[k]), (m, k)
