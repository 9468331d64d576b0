"""Signed distance with one lane and with two lanes a query: either side of the number of queries where that changes, and a
multiple of it, the values and gradients of the same queries in smaller numbers."""
import numpy as np
import pytest

from sesdf_gb300 import SesBuild, synth
from test_gpu_sdf_tile import evaluate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [167_999, 168_000, 1_048_577])
def test_one_and_two_lanes(m):
    atoms = synth.globule(300, 71)
    q = synth.queries(atoms, m, 72)
    w = np.zeros(m, np.float32)
    part = np.random.default_rng(73).permutation(m)[:20_000]
    w[part] = np.random.default_rng(74).standard_normal(len(part)).astype(np.float32)
    with SesBuild(atoms, 1.4, "full") as g:
        g.build()
        got, kind, grad = evaluate(g, q, w)
        want, wkind, wgrad = evaluate(g, q[part], w[part])
    assert np.array_equal(got[part], want) and np.array_equal(kind[part], wkind)
    assert np.linalg.norm(grad - wgrad) <= 1e-4 * np.linalg.norm(wgrad)
