"""Neighbour lists around the sizes at which the probe search changes: up to 64 neighbours (touch masks in shared memory),
65 to 128 (masks in global memory) and more (every neighbour tried), lists cut at the capacity, steps of the visibility test with
17 to 20 circles, against the oracle; and a first build whose mask buffer is too small."""
import numpy as np
import pytest

from oracle import oracle
from sesdf_gb300 import SesBuild, synth
from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["full", "exterior"])
@pytest.mark.parametrize("n,rp,slots,least,most", [(900, 1.9, 128, 63, 66), (900, 2.6, 128, 64, 65), (1200, 2.9, 288, 127, 129),
                                                   (1200, 2.9, 128, 64, 128), (1200, 3.3, 288, 128, 140), (700, 2.6, 72, 64, 72),
                                                   (700, 2.6, 64, 60, 64), (400, 0.4, 128, 16, 20)])
def test_list_lengths(n, rp, slots, least, most, mode):
    atoms = synth.globule(n, 8200)
    o = oracle.run(atoms, rp, mode, max_nbr=slots)
    lengths = np.diff(o["noff"])
    assert lengths.max() >= least and ((lengths >= least) & (lengths <= most)).any()
    with SesBuild(atoms, rp, mode, max_neighbor_per_atom=slots) as g:
        g.build()
        out = g.fetch()
    compare(atoms, out, o, mode)


def test_wide_masks_from_minimal_capacities():
    atoms = synth.globule(900, 8200)
    with SesBuild(atoms, 2.6, "full", min_capacity=True) as g:
        g.build()
        out = g.fetch()
    assert out["counts"]["rebuilds"] > 0
    compare(atoms, out, oracle.run(atoms, 2.6, "full"), "full")
