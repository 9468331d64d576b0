"""Builds whose signed distance and image take the general search alone: truncated neighbour lists, atoms outside the box,
spheres of tens of A; and arcs in more pieces than their buffer holds, which only the device finds out. The values are
those of the general search on the same molecule with an atom outside its box, and nothing is launched for tiles."""
import numpy as np
import pytest

from cases import hand_cases
from sesdf_gb300 import SesBuild, api, synth
from sesdf_gb300.api import aabb
from test_gpu_sdf_tile import evaluate

pytestmark = pytest.mark.gpu


def camera(atoms, width, height):
    lo, hi = atoms[:, :3].min(0), atoms[:, :3].max(0)
    centre, rad = 0.5 * (lo + hi).astype(np.float64), 0.5 * float(np.linalg.norm(hi - lo)) + 30.0
    return {"eye": centre + [0, -3.0 * rad, 0], "forward": [0, 1, 0], "right": [1, 0, 0], "up": [0, 0, 1], "tan_half_fov": 0.36,
            "t_near": rad, "t_far": 5.0 * rad, "eps": 1e-3, "normal_step": 1e-2, "width": width, "height": height, "max_steps": 2000}


def image(g, cam):
    import torch
    depth = torch.full((cam["height"], cam["width"]), -1.0, device="cuda")
    normals = torch.full((cam["height"], cam["width"], 3), -1.0, device="cuda")
    g.render(cam, depth.data_ptr(), normals.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return depth.cpu().numpy(), normals.cpu().numpy()


def launches(call):
    lib = api.load_library()
    before = lib.sesgb_launch_count()
    call()
    return lib.sesgb_launch_count() - before


def pairs(n):
    # 64 pieces for the circle of two spheres of 15 A, more than 16 an atom
    g = np.arange(8, dtype=np.float32) * 80.0
    c = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[: n // 2]
    a = np.concatenate([np.c_[c, np.full(n // 2, 13.0)], np.c_[c + np.float32([6.0, 1.0, 2.0]), np.full(n // 2, 13.5)]])
    return a.astype(np.float32)


MOLECULES = {"pieces do not fit": (lambda: pairs(800), 1.4), "beads": (lambda: synth.globule(400, 61) * np.float32(13.0), 2.0)}


@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_values_are_those_of_the_general_search(name):
    make, rp = MOLECULES[name]
    atoms = make()
    far = np.float32([[*(atoms[:, :3].max(0) + 2000.0), 1.5]])
    both = np.concatenate([atoms, far])
    rng = np.random.default_rng(8)
    k = rng.integers(0, len(atoms), 3000)
    d = rng.normal(size=(3000, 3))
    q = (atoms[k, :3] + d / np.linalg.norm(d, axis=1)[:, None] * (atoms[k, 3:] + rng.uniform(-0.9 * rp, 1.5, (3000, 1)))).astype(np.float32)
    gq = rng.standard_normal(len(q)).astype(np.float32)
    cam = camera(atoms, 70, 50)
    out = []
    for box in (None, aabb(atoms)):
        with SesBuild(both, rp, "full", box=box, max_neighbor_per_atom=288) as g:
            g.build()
            assert g.counts()["outside_atoms"] == (box is not None) and g.counts()["truncated_atoms"] == 0
            out.append((evaluate(g, q, gq), image(g, cam)))
    ((got, kind, grad), im), ((want, wkind, wgrad), wim) = out
    assert np.array_equal(got, want) and np.mean(kind == wkind) > 0.999
    assert len(np.unique(kind)) > 3
    assert np.linalg.norm(grad - wgrad) <= 1e-4 * np.linalg.norm(wgrad)
    assert np.isfinite(im[0]).any() and np.array_equal(im[0], wim[0]) and np.array_equal(im[1], wim[1], equal_nan=True)


def test_general_builds_launch_nothing_for_tiles():
    # without truncated lists one kernel more for the arcs, of queries and of an image, and one for the image's tiles
    import torch
    atoms = synth.globule(1500, 62)
    cam = camera(atoms, 16, 16)
    q = torch.from_numpy(synth.queries(atoms, 1000, 3)).cuda()
    out, grad = torch.empty(1000, device="cuda"), torch.empty(1500, 4, device="cuda")
    counts = []
    for slots in (16, 128):
        with SesBuild(atoms, 1.4, "full", max_neighbor_per_atom=slots) as g:
            g.build()
            assert (g.counts()["truncated_atoms"] > 0) == (slots == 16)
            counts.append([launches(lambda: g.sdf(q.data_ptr(), 1000, out.data_ptr())),
                           launches(lambda: g.sdf_backward(q.data_ptr(), 1000, out.data_ptr(), grad.data_ptr())),
                           launches(lambda: image(g, cam))])
            torch.cuda.synchronize()
    # (the scan of the general search's fewer cells may be a launch shorter too)
    assert all(t - g >= less for g, t, less in zip(*counts, (1, 1, 2)))


@pytest.mark.parametrize("n,few,many", [(12_500, (1, 1), (2, 1)), (65_000, (35, 35), (36, 35))])
def test_images_of_few_pixels(n, few, many):
    # either side of the number of pixels from which an image takes tiles: bits of the general search, and the kernels launched
    atoms = synth.assembly(n // 2500, 2500)[: n - 1]
    both = np.concatenate([atoms, np.float32([[*(atoms[:, :3].max(0) + 50.0), 1.5]])])
    images, counts = [], []
    for box in (None, aabb(atoms)):
        with SesBuild(both, 1.4, "full", box=box) as g:
            g.build()
            for w, h in (few, many):
                cam = camera(atoms, w, h)
                if w < 3:  # at an atom
                    cam.update(eye=atoms[0, :3] + [0, -3.0 * cam["t_near"], 0], tan_half_fov=1e-4)
                image(g, cam)
                counts.append(launches(lambda: images.append(image(g, cam))))
    for k in range(2):
        assert np.array_equal(images[k][0], images[2 + k][0]) and np.array_equal(images[k][1], images[2 + k][1], equal_nan=True)
    assert np.isfinite(images[1][0]).any()
    assert counts[0] <= counts[2] and counts[1] >= counts[3] + 2


@pytest.mark.parametrize("name", ["single", "pair", "triangle", "collinear", "octahedron", "stack", "tangent"])
def test_tiles_of_a_few_atoms(name):
    # so many queries and pixels that molecules of a few atoms take tiles too: bits of the general search
    atoms = hand_cases()[name]
    both = np.concatenate([atoms, np.float32([[200.0, 0.0, 0.0, 1.5]])])
    rng = np.random.default_rng(11)
    m = 30_000
    k = rng.integers(0, len(atoms), m)
    q = (atoms[k, :3] + rng.normal(size=(m, 3)) * 2.0).astype(np.float32)
    q[:2000:7] = atoms[k[:2000:7], :3]
    q[1:2000:7] = 0.5 * (atoms[k[1:2000:7], :3] + atoms[k[2:2001:7], :3])
    cam = camera(atoms, 270, 270)
    out = []
    for box in (None, aabb(atoms)):
        with SesBuild(both, 1.4, "full", box=box) as g:
            g.build()
            out.append((evaluate(g, q), image(g, cam)))
    ((got, kind, _), im), ((want, wkind, _), wim) = out
    assert np.array_equal(got, want) and np.mean(kind == wkind) > 0.999
    assert np.array_equal(im[0], wim[0]) and np.array_equal(im[1], wim[1], equal_nan=True)
