"""The cavity raster decides most voxels in float32 and the ones within its error of a sphere by the double-precision
test: grids with voxel centres exactly on spheres, far from the origin, coarse and very coarse voxels, more components
than one warp's words, against the host labelling voxel for voxel."""
import numpy as np
import pytest

from test_cavities import shell
from test_gpu_cavities import both, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0.0, 1000.0, -5e4])
@pytest.mark.parametrize("h", [0.25, 0.5, 1.0])
def test_centres_on_the_sphere(shift, h):
    # radii and spacings are multiples of the voxel (1.6 + 1.4 = 3.0 up to float32): rims touch voxel centres
    g = np.arange(3) * 5.0
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) + shift
    atoms = np.concatenate([xyz, np.full((27, 1), 1.6)], 1).astype(np.float32)
    got, want, _ = both(atoms, "full", h)
    check(got, want)


@pytest.mark.parametrize("h", [3.0, 7.0, 100.0])
def test_voxels_larger_than_atoms(h):
    rng = np.random.default_rng(5)
    atoms = np.concatenate([rng.uniform(-30, 30, (200, 3)), rng.uniform(1.2, 2.0, (200, 1))], 1).astype(np.float32)
    got, want, _ = both(atoms, "full", h)
    check(got, want)


@pytest.mark.parametrize("n,h", [(1, 0.2), (2, 0.4), (5, 0.35), (33, 0.7)])
def test_many_components(n, h):
    # n closed shells in a row: the inside of each is a component of its own
    one = shell()
    atoms = np.concatenate([one + np.array([60.0 * i, 0, 0, 0], np.float32) for i in range(n)]).astype(np.float32)
    got, want, _ = both(atoms, "full", h)
    check(got, want)
    assert len(got["cavities"]) >= n
