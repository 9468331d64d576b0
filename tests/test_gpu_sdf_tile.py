"""The tile search of the signed distance against the general search, and against itself in other tiles.

A context whose box leaves an atom outside takes the general search for every query (the tile search needs
every atom inside the grid), so that the same molecule, with one more atom far from everything, gives the
general search's values: the tile search's have to be the same float32 numbers, and so do its gradients to the
rounding of their float32 sums. Query counts around the numbers of lanes a query gets (1 to 32) and of queries
a tile holds; probe radii from small to larger than the band; radii and coordinates far from a protein's; points
that are not numbers, far away, at atom centres and on probes."""
import numpy as np
import pytest

from cases import hand_cases
from sesdf_gb300 import SesBuild, synth
from sesdf_gb300.api import aabb

pytestmark = pytest.mark.gpu
FAR = np.array([[400.0, 0.0, 0.0, 1.5]], np.float32)


def evaluate(g, q, gq=None):
    import torch
    dq = torch.from_numpy(np.ascontiguousarray(q, np.float32)).cuda()
    out = torch.empty(len(q), dtype=torch.float32, device="cuda")
    kind = torch.empty(len(q), dtype=torch.int32, device="cuda")
    g.sdf(dq.data_ptr(), len(q), out.data_ptr(), kind.data_ptr())
    grad = None
    if gq is not None:
        dg = torch.from_numpy(np.ascontiguousarray(gq, np.float32)).cuda()
        ga = torch.empty((g.atoms.shape[0], 4), dtype=torch.float32, device="cuda")
        g.sdf_backward(dq.data_ptr(), len(q), dg.data_ptr(), ga.data_ptr())
        grad = ga.cpu().numpy()
    torch.cuda.synchronize()
    return out.cpu().numpy(), kind.cpu().numpy(), grad


def molecules():
    shrunk = synth.globule(400, 21)
    shrunk[:, 3] *= 0.5
    coarse = synth.globule(600, 22)
    coarse *= np.float32(3.0)  # beads of 5 A
    moved = synth.globule(700, 23)
    moved[:, :3] += np.float32([150.0, -90.0, 60.0])
    dense = synth.globule(900, 24)
    dense[:, :3] *= np.float32(0.6)
    out = {"globule": (synth.globule(1500, 20), 1.4), "small_radii": (shrunk, 1.4), "beads": (coarse, 1.4), "moved": (moved, 1.2),
           "dense": (dense, 1.4), "coarse_probe": (synth.globule(800, 25), 2.4), "large_probe": (synth.globule(500, 26), 3.6)}
    for name in ("single", "pair", "collinear", "octahedron", "stack"):
        out[name] = (hand_cases()[name], 1.4)
    return out


@pytest.mark.parametrize("name", sorted(molecules()))
def test_tile_search_gives_the_general_search(name):
    atoms, rp = molecules()[name]
    atoms = np.concatenate([atoms, FAR + np.float32([*atoms[:, :3].mean(0), 0.0])])
    plain = 3000
    q = np.concatenate([synth.queries(atoms[:-1], plain, 31), atoms[:40, :3], atoms[:40, :3] + np.float32(1e-3),
                        (atoms[:40, :3] + atoms[1:41, :3][: len(atoms[:40])]) * np.float32(0.5) if len(atoms) > 41 else atoms[:0, :3],
                        np.float32([[np.nan, 0, 0], [np.inf, 0, 0], [1e6, 1e6, -1e6], [0, 1e30, 0]])])
    rng = np.random.default_rng(5)
    with SesBuild(atoms, rp, "full", max_neighbor_per_atom=288) as tile, \
            SesBuild(atoms, rp, "full", box=aabb(atoms[:-1]), max_neighbor_per_atom=288) as general:
        tile.build()
        general.build()
        assert tile.counts()["outside_atoms"] == 0 and general.counts()["outside_atoms"] == 1
        assert tile.counts()["truncated_atoms"] == 0
        probes = tile.fetch(analysis=False)["probe_pos"]
        if len(probes):
            q = np.concatenate([q, probes[:200, :3], probes[:200, :3] + rng.normal(0, 1e-4, (len(probes[:200]), 3)).astype(np.float32)])
        gq = rng.standard_normal(len(q)).astype(np.float32)
        gq[plain:] = 0.0  # a gradient is defined where one primitive is nearest
        got, kind, grad = evaluate(tile, q, gq)
        want, wkind, wgrad = evaluate(general, q, gq)
    assert np.array_equal(got, want)
    assert np.mean(kind == wkind) > 0.999  # equal distances may go by the atoms' order, which the box changes
    # float32 sums in any order; a probe near the plane of its atoms moves by thousands of their steps
    assert np.linalg.norm(grad - wgrad) <= 1e-4 * max(np.linalg.norm(wgrad), 1e-6)


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 127, 2433, 4999, 38913, 77825])
def test_values_do_not_depend_on_the_tile(m):
    """Any number of queries, in any order: the same value for each."""
    atoms = synth.globule(1200, 41)
    q = synth.queries(atoms, 80000, 42)
    order = np.random.default_rng(m).permutation(len(q))[:m]
    with SesBuild(atoms, 1.4, "full") as g:
        g.build()
        want, wkind, _ = evaluate(g, q)
        got, kind, _ = evaluate(g, q[order])
    assert np.array_equal(got, want[order])
    assert np.array_equal(kind, wkind[order])


@pytest.mark.parametrize("n,few", [(20000, 1), (50000, 4), (60000, 300), (100000, 2000)])
def test_few_queries_alone_as_among_many(n, few):
    import torch
    # few queries take the general search alone, many take tiles: the same bits for each query, and the same
    # gradient up to the order of its sums where the others have no weight
    atoms = synth.globule(n, 4200 + few)
    rng = np.random.default_rng(few)
    many = 8000
    k = rng.integers(0, n, many)
    d = rng.normal(size=(many, 3))
    q = atoms[k, :3] + d / np.linalg.norm(d, axis=1)[:, None] * (atoms[k, 3:] + rng.uniform(-0.5, 1.5, (many, 1)))
    q[1::97] += 500.0  # out of reach
    q = torch.tensor(q.astype(np.float32), device="cuda")
    w = torch.zeros(many, device="cuda")
    w[:few] = torch.rand(few, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    out, kind, grad = {}, {}, {}
    with SesBuild(atoms, 1.4, "full") as g:
        g.build()
        for m in (few, many):
            out[m] = torch.empty(m, device="cuda")
            kind[m] = torch.empty(m, dtype=torch.int32, device="cuda")
            grad[m] = torch.empty(n, 4, device="cuda")
            g.sdf(q.data_ptr(), m, out[m].data_ptr(), kind[m].data_ptr(), s)
            g.sdf_backward(q.data_ptr(), m, w.data_ptr(), grad[m].data_ptr(), s)
        torch.cuda.synchronize()
    assert torch.equal(out[few], out[many][:few]) and torch.equal(kind[few], kind[many][:few])
    # one query adds to a row once; a row sums at most `few` terms of size at most 1
    assert torch.allclose(grad[few], grad[many], rtol=0, atol=few * 2.0 ** -22)


@pytest.mark.parametrize("width,height", [(1, 1), (61, 100), (62, 100), (245, 200), (246, 200), (328, 299), (328, 300), (447, 439),
                                          (447, 441)])
def test_image_by_rays_per_warp(width, height):
    # the number of pixels of a warp changes between these sizes; the general search takes a ray's points one by one
    import torch
    atoms = np.concatenate([synth.globule(300, 33), FAR])
    lo, hi = atoms[:-1, :3].min(0), atoms[:-1, :3].max(0)
    centre, rad = 0.5 * (lo + hi).astype(np.float64), 0.5 * float(np.linalg.norm(hi - lo)) + 4.0
    cam = {"eye": centre + [0, -3.0 * rad, 0], "forward": [0, 1, 0], "right": [1, 0, 0], "up": [0, 0, 1], "tan_half_fov": 0.36,
           "t_near": rad, "t_far": 5.0 * rad, "eps": 1e-3, "normal_step": 1e-2, "width": width, "height": height, "max_steps": 128}
    images = []
    for box in (None, aabb(atoms[:-1])):
        with SesBuild(atoms, 1.4, "full", box=box) as g:
            g.build()
            depth = torch.full((height, width), -1.0, device="cuda")
            normals = torch.full((height, width, 3), -1.0, device="cuda")
            g.render(cam, depth.data_ptr(), normals.data_ptr(), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            images.append((depth.cpu().numpy(), normals.cpu().numpy()))
    assert width == 1 or np.isfinite(images[0][0]).any()
    assert np.array_equal(images[0][0], images[1][0])
    assert np.array_equal(images[0][1], images[1][1], equal_nan=True)
