"""Queries as near to several probes as to the first of them: the gradient goes to one of the nearest, the same one whether the query
comes alone, among thousands (tiles of any number of lanes) or by the general search, and on every call."""
import numpy as np
import pytest

from cases import hand_cases
from sesdf_gb300 import SesBuild
from sesdf_gb300.api import aabb
from test_gpu_sdf_tile import evaluate

pytestmark = pytest.mark.gpu


def rings(n):
    # octahedra side by side, 4 A between their atoms: eight probes each around a common centre
    one = hand_cases()["octahedron"] * np.float32([1.0 / 3.0, 1.0 / 3.0, 1.0 / 3.0, 1.0]) * np.float32([2.0, 2.0, 2.0, 1.0])
    g = np.arange(n, dtype=np.float32) * np.float32(16.0)
    at = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 1, 3)
    a = np.tile(one, (n ** 3, 1, 1))
    a[:, :, :3] += at
    return a.reshape(-1, 4), at.reshape(-1, 3)


def test_ties_go_to_the_same_probe():
    # enough atoms that a query alone takes the general search; the order of the atoms, which decides, follows the box
    atoms, centres = rings(13)
    centres = centres[::37]
    far = np.float32([[*(atoms[:, :3].max(0) + 100.0), 1.5]])
    both = np.concatenate([atoms, far])
    t = np.linspace(1.0, 3.0, 9, dtype=np.float32)[:, None]
    # on the planes and the axes of symmetry
    ways = np.float32([[0, 0, 1], [0, 0, -1], [1, 0, 0], [-1, 0, 0], [1, 1, 0], [1, -1, 0], [0, 1, 1], [0, -1, 1], [-1, 0, 1]])
    local = (ways[:, None, :] * t[None]).reshape(-1, 3)
    q = (centres[:, None, :] + local[None]).reshape(-1, 3).astype(np.float32)
    for box in (None, aabb(atoms)):
        with SesBuild(both, 1.4, "full", box=box) as g:
            g.build()
            value, kind, _ = evaluate(g, q)
            probes = g.fetch(analysis=False)["probe_pos"][:, :3].astype(np.float64)
            own = np.stack([probes[np.argsort(np.linalg.norm(probes - c, axis=1))[:16]] for c in centres])
            d = np.sort(np.linalg.norm(q.reshape(len(centres), -1, 1, 3) - own[:, None], axis=3), axis=2).reshape(len(q), -1)
            tied = np.where((kind == 5) & (d[:, 1] - d[:, 0] < 1e-9))[0]
            assert len(tied) > 100
            for k in tied[:: len(tied) // 24]:
                weight = np.zeros(len(q), np.float32)
                weight[k] = 1.0
                got, gkind, want = evaluate(g, q[k:k + 1], weight[k:k + 1])
                assert got[0] == value[k] and gkind[0] == kind[k]
                assert np.count_nonzero(np.abs(want).sum(1)) in (1, 2, 3)  # by symmetry an atom's term may be zero
                for first, many in ((0, len(q)), (k - k % 2, 2), (k - k % 100, 100), (0, len(q))):
                    _, _, grad = evaluate(g, q[first:first + many], weight[first:first + many])
                    assert np.array_equal(grad, want), (k, many)
