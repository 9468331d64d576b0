"""Signed distance on the lines through two atom centres, and at the centres: all points of the circle of such a pair are as near,
and it counts if one of them is accessible. Both searches give the same values, with up to dozens of centres close to the query,
and those of the FP64 oracle a little off the line (the distance changes by no more than its argument does). Not so in the
lattice, four of whose spheres meet in a point: a build lists no vertex there, and off the line the nearest point may be one."""
import numpy as np
import pytest

from cases import hand_cases
from oracle import oracle
from sesdf_gb300 import SesBuild, synth
from sesdf_gb300.api import aabb
from test_gpu_sdf_tile import FAR, evaluate

pytestmark = pytest.mark.gpu
STEP, TOL = 1e-3, 1e-4  # off the line; of a value against the oracle


def lattice(n, spacing, r):
    g = np.arange(n, dtype=np.float32) * np.float32(spacing)
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return np.concatenate([xyz, np.full((len(xyz), 1), r, np.float32)], 1)


def crowd(seed):
    rng = np.random.default_rng(seed)
    near = np.c_[rng.normal(0.0, 0.45, (24, 3)), rng.uniform(1.2, 1.9, 24)]
    return np.concatenate([near, synth.globule(60, seed) + np.float32([3, 0, 0, 0])]).astype(np.float32)


MOLECULES = {"globule": lambda: synth.globule(600, 22), "lattice": lambda: lattice(5, 3.0, 1.2), "crowd": lambda: crowd(3),
             "stack": lambda: hand_cases()["stack"], "pair": lambda: hand_cases()["pair"]}


@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_on_the_axis_of_circles(name):
    atoms = MOLECULES[name]()
    both = np.concatenate([atoms, FAR + np.float32([*atoms[:, :3].mean(0), 0.0])])
    d = np.linalg.norm(atoms[:, None, :3] - atoms[None, :, :3], axis=2)
    i, j = np.where(np.triu((d < 6.2) & (d > 0.0), 1))
    p, v = atoms[i, :3], atoms[j, :3] - atoms[i, :3]
    q = np.concatenate([p + v * np.float32(0.5), p + v * np.float32(0.37), p - v * np.float32(0.25), atoms[:, :3]])
    u = np.random.default_rng(9).normal(size=q.shape)
    off = q + STEP * u / np.linalg.norm(u, axis=1)[:, None]
    with SesBuild(both, 1.4, "full", max_neighbor_per_atom=288) as tile, \
            SesBuild(both, 1.4, "full", box=aabb(atoms), max_neighbor_per_atom=288) as general:
        tile.build()
        general.build()
        assert tile.counts()["outside_atoms"] == 0 and general.counts()["outside_atoms"] == 1
        got, _, _ = evaluate(tile, q)
        want, _, _ = evaluate(general, q)
    exact, _, _ = oracle.sdf(oracle.run(atoms, 1.4, "full"), off.astype(np.float32))
    moved = np.linalg.norm(off.astype(np.float32).astype(np.float64) - q, axis=1)
    assert np.array_equal(got, want)
    assert name == "lattice" or np.all(np.abs(got - exact) <= moved + TOL)
