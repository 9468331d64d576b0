"""The work that users of this package have it do, as cases that can be timed and compared.

Every case goes through the package's public entry points (`SesBuild`, `SesBatch`, the torch binding) on seeded
protein-like molecules of this repository's own generator: `listed()` the cases, `draw()` one more of the same ranges,
`prepare()` what a program has in hand before the call (atoms on the device, a built context with its buffers),
`run()` one call and its outputs, `work()` the bytes and operations the call cannot do without, `exact()` the
outputs in double precision, from plain torch.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from sesdf_gb300 import SesBatch, SesBuild, render, synth, torch_sdf
from sesdf_gb300.api import FullData

GLOBULE_MOST = 50_000  # larger molecules are assemblies of globules


def listed():
    return [
        # a small protein, rebuilt from host coordinates as bcs::Sesdf::build does: launches and latency
        {"name": "globule_2k_host", "kind": "build", "atoms": 2000, "mode": "full", "probe": 1.4, "slots": 0, "host": True},
        # an ordinary structure of the PDB's size, exterior surface only, coordinates on the device
        {"name": "globule_11638_exterior", "kind": "build", "atoms": 11638, "mode": "exterior", "probe": 1.4, "slots": 0, "host": False},
        # the benchmark's molecule: a 100,000-atom assembly, full surface
        {"name": "assembly_100k", "kind": "build", "atoms": 100_000, "mode": "full", "probe": 1.4, "slots": 0, "host": False},
        # the largest build: a capsid-like shell of a million atoms
        {"name": "shell_1m", "kind": "build", "atoms": 1_000_000, "mode": "full", "probe": 1.4, "slots": 0, "host": False},
        # a coarse probe: the reference's second configuration (2.4 A, 288 neighbour slots), lists of ~75 neighbours
        {"name": "globule_6007_probe24", "kind": "build", "atoms": 6007, "mode": "full", "probe": 2.4, "slots": 288, "host": False},
        # a library of structures of uneven size in one batch
        {"name": "batch_64", "kind": "batch", "molecules": 64, "least": 500, "most": 20_000, "frames": False, "mode": "full", "probe": 1.4},
        # a handful of points against a small molecule (docking, collision): the latency of a query call
        {"name": "sdf_2k_4999", "kind": "sdf", "atoms": 2000, "queries": 4999, "probe": 1.4},
        # a dense sampling of the field around a protein
        {"name": "sdf_20k_1m", "kind": "sdf", "atoms": 20_000, "queries": 1_000_000, "probe": 1.4},
        # one training step on the signed distance: build, values, gradient with respect to atoms and radii
        {"name": "sdf_train_20k_200k", "kind": "sdf_train", "atoms": 20_000, "queries": 200_000, "probe": 1.4},
        # the surface area per atom and its gradient (solvation terms), one step of a minimiser
        {"name": "area_20k", "kind": "area", "atoms": 20_000, "probe": 1.4},
        # a depth and normal image of a protein
        {"name": "image_20k_512", "kind": "image", "atoms": 20_000, "width": 512, "height": 512, "probe": 1.4},
        # pockets and cavities of a protein on a 0.5 A grid
        {"name": "cavities_20k", "kind": "cavities", "atoms": 20_000, "voxel": 0.5, "probe": 1.4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "batch", "sdf", "sdf", "sdf_train", "area", "image", "cavities"])
    probe = rng.choice([1.4, 1.4, 1.4, 1.2, 1.6])
    if kind == "build":
        case = {"kind": kind, "atoms": _log(rng, 500, 200_000), "mode": rng.choice(["full", "exterior"]), "probe": probe, "slots": 0,
                "host": rng.random() < 0.3}
        if rng.random() < 0.2:
            case.update(atoms=_log(rng, 500, 20_000), probe=2.4, slots=288)
        return case
    if kind == "batch":
        if rng.random() < 0.4:  # MD-like frames of one molecule
            n = _log(rng, 1000, 20_000)
            return {"kind": kind, "molecules": rng.randint(3, 16), "least": n, "most": n, "frames": True,
                    "mode": rng.choice(["full", "exterior"]), "probe": probe}
        return {"kind": kind, "molecules": rng.randint(2, 64), "least": 500, "most": _log(rng, 2000, 20_000), "frames": False,
                "mode": rng.choice(["full", "exterior"]), "probe": probe}
    n = _log(rng, 500, 20_000)
    if kind == "sdf":
        return {"kind": kind, "atoms": n, "queries": _log(rng, 1000, 900_000), "probe": probe}
    if kind == "sdf_train":
        return {"kind": kind, "atoms": n, "queries": _log(rng, 1000, 200_000), "probe": probe}
    if kind == "image":
        return {"kind": kind, "atoms": n, "width": rng.randint(64, 512), "height": rng.randint(64, 512), "probe": probe}
    if kind == "cavities":
        return {"kind": kind, "atoms": n, "voxel": rng.choice([0.4, 0.5, 0.7]), "probe": probe}
    return {"kind": kind, "atoms": n, "probe": probe}


# ---- inputs ---------------------------------------------------------------------------------------------------

def _grid_position(atoms, rp):
    """Float32 position of every atom in the reference grid, in cells, and the grid's size."""
    f = np.float32
    lo, hi = (atoms[:, :3] - atoms[:, 3:]).min(0), (atoms[:, :3] + atoms[:, 3:]).max(0)
    origin = (lo - f(3.48)) - f(rp)
    size = 1 << max(0, (int(math.floor(math.log2(len(atoms)))) - 1).bit_length())
    cell = np.abs(((hi + f(3.48)) + f(rp)) - origin) / f(size)
    return (atoms[:, :3] - origin) / cell, size


def _off_boundaries(atoms, rp):
    """Atoms a rounding away from a cell boundary of the reference grid moved by 0.002 A: the order of the outputs
    follows the cells, and is then the same in any arithmetic."""
    for _ in range(20):
        q, _ = _grid_position(atoms, rp)
        near = np.abs(q - np.round(q)) < 2e-5
        if not near.any():
            break
        atoms[:, :3][near] += np.float32(0.002)
    return atoms


def _molecule(n, seed, rp):
    if n <= GLOBULE_MOST:
        return _off_boundaries(synth.globule(n, 7919 * seed + 11), rp)
    per = 5000
    parts = -(-n // per)
    make = synth.shell if n >= 500_000 else synth.assembly
    return _off_boundaries(np.ascontiguousarray(make(parts, per, 7919 * seed + 11)[:n]), rp)


def _batch(case, seed):
    if case["frames"]:
        base = synth.globule(case["least"], 7919 * seed + 11)
        mols = [synth.jitter(base, 0.3, 7919 * seed + f) for f in range(case["molecules"])]
    else:  # sizes spread evenly over their logarithm, in no order
        m = case["molecules"]
        steps = np.random.default_rng(m).permutation(m) + 0.5
        sizes = (case["least"] * (case["most"] / case["least"]) ** (steps / m)).astype(int)
        mols = [synth.globule(int(n), 7919 * seed + 13 * k) for k, n in enumerate(sizes)]
    return [_off_boundaries(m, case["probe"]) for m in mols]


def _queries(case, seed, atoms):
    q = synth.queries(atoms, case["queries"], 7919 * seed + 5)
    if len(q) != case["queries"]:
        raise RuntimeError("fewer query points than asked for")
    return torch.from_numpy(q).cuda()


def _weights(m, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(m, generator=g).cuda()


class _Device:
    """Device memory of a build as the array interface that torch reads. A tensor made of it holds this object, and
    with it the build that owns the memory."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 3}


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _view(state, name, ptr, count, width, kind):
    """Device memory at ptr as a tensor; the tensor of the last call where it is the same memory."""
    key, t = state.get(name, (None, None))
    if key != (ptr, count):
        t = torch.as_tensor(_Device(state["build"], ptr, (count, width), kind), device="cuda")
        state[name] = ((ptr, count), t)
    return t


# Output buffers: field, its count, values a row, type, and rows per atom that are returned. How many rows a build
# writes depends on the molecule; the outputs are the buffers up to a number of rows that depends on the atom count
# alone (well within the capacities that a context starts with), the rows past the counts being zero.
_FULL = {"atoms": ("atoms", "atomNb", 4, "<f4", 1), "convex": ("convexPatches", "convexPatchNb", 2, "<i4", 1),
         "sectors": ("sectors", "sectorNb", 4, "<f4", 36), "segments": ("segmentPatches", "segmentPatchNb", 4, "<i4", 6),
         "circles": ("circlePatches", "circlePatchNb", 2, "<i4", 2), "probes": ("concavePatchesPosition", "concavePatchNb", 4, "<f4", 4),
         "probe_ids": ("concavePatchesId", "concavePatchNb", 4, "<i4", 4)}
_EXTERIOR = {"atoms": ("atoms", "atomNb", 4, "<f4", 1), "tori": ("circlePosition", "circlePatchNb", 4, "<f4", 8),
             "axes": ("circleAxis", "circlePatchNb", 4, "<f4", 8), "spheres": ("circleVs", "circlePatchNb", 4, "<f4", 8),
             "probes": ("concavePatchesPosition", "concavePatchNb", 4, "<f4", 4),
             "probe_ids": ("concavePatchesId", "concavePatchNb", 4, "<i4", 4)}
_NEIGHBOURS = 2  # singular probes per atom, 32 slots each


def _buffers(state):
    """Every output buffer of the last build (bcs::Sesdf::getData), as tensors over the library's memory."""
    d = state["build"].data()
    out = {}
    for name, (field, _, width, kind, per) in (_FULL if isinstance(d, FullData) else _EXTERIOR).items():
        out[name] = _view(state, name, getattr(d, field), per * d.atomNb, width, kind)
    out["neighbours"] = _view(state, "neighbours", d.concavePatchesNeighbors, 32 * _NEIGHBOURS * d.atomNb, 4, "<f4")
    return out


def _first_build(state):
    """The first build sizes the context's buffers; what no build of this molecule writes in them is zeroed."""
    b = state["build"]
    b.build_device(state["device_atoms"].data_ptr(), _stream())
    d = b.data()
    counts = b.counts()
    for field, count, _, _, per in (_FULL if isinstance(d, FullData) else _EXTERIOR).values():
        if getattr(d, count) > per * d.atomNb or counts["singular_probes"] > _NEIGHBOURS * d.atomNb:
            raise RuntimeError("more rows in %s than the outputs hold" % field)
    for t in _buffers(state).values():
        t.zero_()
    b.build_device(state["device_atoms"].data_ptr(), _stream())


def prepare(case, seed):
    kind, rp = case["kind"], case["probe"]
    state = {"case": dict(case)}
    if kind == "batch":
        mols = _batch(case, seed)
        state["build"] = b = SesBatch(mols, rp, case["mode"])
        state["device_atoms"] = torch.from_numpy(b.atoms).cuda()
        _first_build(state)
        return state
    atoms = _molecule(case["atoms"], seed, rp)
    if kind == "sdf_train":
        state["atoms"] = torch.from_numpy(atoms).cuda().requires_grad_(True)
        state["queries"] = _queries(case, seed, atoms)
        state["weights"] = _weights(case["queries"], seed)
        return state
    state["device_atoms"] = torch.from_numpy(atoms).cuda()
    state["build"] = b = SesBuild(atoms, rp, case.get("mode", "full"), max_neighbor_per_atom=case.get("slots", 0))
    _first_build(state)
    if kind == "build" and case["host"]:
        state["pinned"] = torch.from_numpy(atoms).pin_memory()
        b.set_host_pointer(state["pinned"].data_ptr())
    elif kind == "sdf":
        state["queries"] = _queries(case, seed, atoms)
        state["sdf"] = torch.empty(case["queries"], device="cuda")
        state["which"] = torch.empty(case["queries"], dtype=torch.int32, device="cuda")
    elif kind == "area":
        state["area"] = torch.empty(case["atoms"], device="cuda")
        state["grad"] = torch.empty((case["atoms"], 4), device="cuda")
    elif kind == "image":
        eye, centre, up, near, far = render.framing(atoms, rp)
        f, r, u = render.camera_basis(eye, centre, up)
        w, h = case["width"], case["height"]
        state["camera"] = dict(eye=eye, forward=f, right=r, up=u, tan_half_fov=math.tan(math.radians(20.0)), t_near=near, t_far=far,
                               eps=1e-3, normal_step=1e-2, width=w, height=h, max_steps=256)
        state["depth"] = torch.empty((h, w), device="cuda")
        state["normals"] = torch.zeros((h, w, 3), device="cuda")
    elif kind == "cavities":
        n, h = case["atoms"], case["voxel"]
        side = int((2.0 * ((3.0 * n / (4.0 * math.pi * 0.045)) ** (1.0 / 3.0) + 1.8 + rp) + 1.0) / h) + 8
        state["component"] = torch.zeros(4 * n, dtype=torch.int32, device="cuda")
        state["grid"] = torch.zeros(side**3, dtype=torch.int32, device="cuda")
    return state


# ---- one pass -------------------------------------------------------------------------------------------------

def _labels(state):
    """The label grid of the last cavities() call (sesgb_cavity_labels of the C interface: it stays on the device)."""
    b = state["build"]
    p, v = ctypes.c_void_p(), ctypes.c_uint64()
    b._check(b._lib.sesgb_cavity_labels(b._h, ctypes.byref(p), ctypes.byref(v)), "cavity_labels")
    return _view(state, "labels", p.value, v.value, 1, "<i4")[:, 0]


def _padded(values, count):
    out = np.zeros(count, values.dtype)
    out[: len(values)] = values
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sdf_train":
        out = torch_sdf.ses_sdf(state["atoms"], state["queries"], case["probe"])
        (grad,) = torch.autograd.grad(out, state["atoms"], state["weights"])
        return {"sdf": out, "grad": grad}
    b = state["build"]
    if kind in ("build", "batch"):
        if case.get("host"):
            b.build(_stream())
        else:
            b.build_device(state["device_atoms"].data_ptr(), _stream())
        return _buffers(state)
    if kind == "sdf":
        b.sdf(state["queries"].data_ptr(), case["queries"], state["sdf"].data_ptr(), state["which"].data_ptr(), _stream())
        return {"sdf": state["sdf"], "which": state["which"]}
    if kind == "area":
        parts = b.ses_area(state["area"].data_ptr(), _stream())
        b.ses_area_backward(state["grad"].data_ptr(), (1.0, 1.0, 1.0), _stream())
        # the parts are float64 sums of float32 patches: they come back with the precision they have
        return {"parts": np.array([parts["convex"], parts["toroidal"], parts["concave"]], np.float32), "area": state["area"],
                "grad": state["grad"]}
    if kind == "image":
        b.render(state["camera"], state["depth"].data_ptr(), state["normals"].data_ptr(), _stream())
        return {"depth": state["depth"], "normals": state["normals"]}
    info = b.cavities(case["voxel"], state["component"].data_ptr(), _stream())
    voxels, border = b.cavity_components(info["components"])
    labels = _labels(state)
    state["grid"][: len(labels)].copy_(labels)  # the program's own grid: the library's goes with the next call
    return {"origin": info["origin"], "dims": np.array(info["dims"]), "exterior": info["exterior"], "cavities": info["cavities"],
            "voxels": _padded(voxels.astype(np.int64), case["atoms"]), "border": _padded(border, case["atoms"]),
            "component": state["component"], "grid": state["grid"]}


def work(case):
    """Per atom of a full build at 1.4 A: 35 neighbours, 20.5 sectors, 1.7 probes (0.7 singular with ~10 neighbours),
    2.6 segments; ~330 pair tests, 17.5 circles against 35 atoms, 37 triplets."""
    kind = case["kind"]
    reach = (case["probe"] + 1.6) ** 3 / 27.0  # neighbours grow with the probe's reach
    if kind == "batch":
        mean = case["least"] if case["least"] == case["most"] else (case["most"] - case["least"]) / math.log(case["most"] / case["least"])
        n = mean * case["molecules"]
    else:
        n = case["atoms"]
    build = {"bytes": n * (570.0 if case.get("mode", "full") == "full" else 360.0), "flops": n * 30e3 * reach * reach}
    if kind in ("build", "batch"):
        return build
    if kind == "sdf":
        return {"bytes": 20.0 * case["queries"] + 16.0 * n, "flops": 8e3 * case["queries"]}
    if kind == "sdf_train":
        return {"bytes": 20.0 * case["queries"] + 32.0 * n, "flops": 17e3 * case["queries"] + build["flops"]}
    if kind == "area":
        return {"bytes": 40.0 * n, "flops": 120e3 * n}
    if kind == "image":
        return {"bytes": 16.0 * case["width"] * case["height"] + 16.0 * n, "flops": 60e3 * case["width"] * case["height"]}
    voxels = n / 0.03 / case["voxel"] ** 3
    return {"bytes": 4.0 * voxels + 16.0 * n, "flops": 20.0 * voxels}


# ---- the same in double precision -----------------------------------------------------------------------------

TOL = float(np.float32(1e-4))


def _rows(total, width, most=4_000_000):
    step = max(1, most // max(1, width))
    for a in range(0, total, step):
        yield slice(a, min(total, a + step))


def _dot(a, b):
    return (a * b).sum(-1)


def _bins(points, cell):
    """Cell lists of points as a padded table (index len(points) = none), and the table's rows around query points."""
    lo = points.min(0).values - cell
    dims = ((points.max(0).values - lo) / cell).floor().long() + 3

    def key(p):
        c = ((p - lo) / cell).floor().long()
        return torch.minimum(c.clamp_min(0), dims - 1)

    def flat(c):
        return (c[..., 2] * dims[1] + c[..., 1]) * dims[0] + c[..., 0]

    k = flat(key(points))
    order = torch.argsort(k, stable=True)
    count = torch.bincount(k, minlength=int(dims.prod()))
    start = count.cumsum(0) - count
    table = torch.full((int(dims.prod()), int(count.max())), len(points), dtype=torch.long, device=points.device)
    table[k[order], torch.arange(len(points), device=points.device) - start[k[order]]] = order
    r = torch.arange(-1, 2, device=points.device)
    around = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)

    def near(p):
        c = key(p)[:, None, :] + around
        ok = ((c >= 0) & (c < dims)).all(-1)
        return torch.where(ok[..., None], table[flat(torch.where(ok[..., None], c, 0))], len(points)).flatten(1)

    return near


class _Surface:
    """The build of one molecule: neighbours, circle statuses, probes."""

    def __init__(self, atoms, rp, mode):
        q, size = _grid_position(atoms, rp)
        p = np.floor(q).astype(np.int64) & (size - 1)
        self.perm = np.argsort((p[:, 2] * size + p[:, 1]) * size + p[:, 0], kind="stable")
        self.atoms = torch.from_numpy(atoms[self.perm]).cuda()
        a = self.atoms.double()
        self.rp, self.n, self.mode = float(np.float32(rp)), len(atoms), mode
        far = torch.full((1, 4), 1e6, dtype=a.dtype, device=a.device)
        a = torch.cat([a, far])  # index n: an atom that is no neighbour of any
        self.c, self.R = a[:, :3], a[:, 3] + self.rp
        self._neighbours()
        self._statuses()
        self._probes()

    def _neighbours(self):
        c, R, n = self.c, self.R, self.n
        near = _bins(c[:n], float(2.0 * R[:n].max() + 0.01))
        found = []
        for s in _rows(n, 800):
            i = torch.arange(s.start, s.stop, device=c.device)
            j = near(c[i])
            d = c[i][:, None] - c[j]
            sum_r = R[i][:, None] + R[j]
            ok = (_dot(d, d) - sum_r * sum_r <= TOL) & (j != i[:, None]) & (j < n)
            found.append(torch.where(ok, j, n).sort(1).values[:, :320])
        self.K = max(int((f < n).sum(1).max()) for f in found)
        self.nb = torch.cat([f[:, : self.K] for f in found])

    def _circle(self, i, j):
        R1, R2 = self.R[i], self.R[j]
        v = self.c[j] - self.c[i]
        d = _dot(v, v)
        t = (R1 * R1 - R2 * R2 + d) / (2.0 * d)
        centre = self.c[i] + v * t[..., None]
        to = self.c[i] - centre
        return centre, v / d.sqrt()[..., None], (R1 * R1 - _dot(to, to)).sqrt(), t, d

    def _statuses(self):
        n, nb = self.n, self.nb
        i, s = ((nb < n) & (nb > torch.arange(n, device=nb.device)[:, None])).nonzero(as_tuple=True)
        j = nb[i, s]
        status = torch.empty(len(i), dtype=torch.int8, device=nb.device)
        for r in _rows(len(i), self.K):
            centre, normal, radius, _, _ = self._circle(i[r], j[r])
            k = nb[i[r]]
            v = centre[:, None] - self.c[k]
            dist = _dot(v, v).sqrt()
            second = _dot(v, normal[:, None])
            sin = (1.0 - (second / dist).square()).sqrt()
            ok = (k < n) & (k != j[r][:, None])
            far = (sin * dist + radius[:, None]).square() + second.square() - self.R[k].square() < TOL
            close = (radius[:, None] - sin * dist).square() + second.square() - self.R[k].square() < TOL
            status[r] = torch.where((far & ok).any(1), 0, torch.where((close & ok).any(1), 1, 2)).to(torch.int8)
        self.i, self.j, self.status = i, j, status
        self.table = torch.zeros_like(nb, dtype=torch.int8)
        self.table[i, s] = status
        if self.mode == "full":  # circle (j, i) is circle (i, j)
            a, t = ((nb < n) & (nb < torch.arange(n, device=nb.device)[:, None])).nonzero(as_tuple=True)
            self.table[a, t] = status[torch.searchsorted(i * (n + 1) + j, nb[a, t] * (n + 1) + a).clamp_max(len(i) - 1)]

    def point(self, i, j, k, side, c=None, R=None):
        """The point at distance R from the centres of i, j and k, on the side of (c_j - c_i) x (c_k - c_i)."""
        c, R = (self.c, self.R) if c is None else (c, R)
        a, b = c[j] - c[i], c[k] - c[i]
        m = torch.linalg.cross(a, b)
        Ri2 = R[i] * R[i]
        p = (_dot(a, a) + Ri2 - R[j] * R[j]) * 0.5
        q = (_dot(b, b) + Ri2 - R[k] * R[k]) * 0.5
        mm = _dot(m, m)
        y = (p[:, None] * torch.linalg.cross(b, m) + q[:, None] * torch.linalg.cross(m, a)) / mm[:, None]
        h2 = Ri2 - _dot(y, y)
        return c[i] + y + m * (side * (h2 / mm).sqrt())[:, None], h2

    def _probes(self):
        n, nb = self.n, self.nb
        part = self.status == 1
        ei, ej = self.i[part], self.j[part]
        got = []
        for r in _rows(len(ei), self.K):
            i, j = ei[r], ej[r]
            k = nb[i]
            ok = (k > j[:, None]) & (k < n) & (self.table[i] == 1)
            v = self.c[j][:, None] - self.c[k]
            sum_r = self.R[j][:, None] + self.R[k]
            e, s = (ok & (_dot(v, v) - sum_r * sum_r <= TOL)).nonzero(as_tuple=True)
            i, j, k = i[e], j[e], k[e, s]
            for u in _rows(len(i), 2 * self.K):
                iu, ju, ku = (x[u].repeat_interleave(2) for x in (i, j, k))
                side = torch.tensor([1.0, -1.0], dtype=self.c.dtype, device=self.c.device).repeat(u.stop - u.start)
                x, h2 = self.point(iu, ju, ku, side)
                o = nb[iu]
                d = self.c[o] - x[:, None]
                free = (_dot(d, d) - self.R[o].square() > 0.0) | (o >= n) | (o == ju[:, None]) | (o == ku[:, None])
                keep = (h2 >= 0.0) & free.all(1)
                got.append([t[keep] for t in (iu, ju, ku, side, x, h2)])
        i, j, k, side, x, h2 = (torch.cat(t) for t in zip(*got))
        singular = h2 - self.rp * self.rp < -TOL
        order = torch.cat([singular.nonzero()[:, 0], (~singular).nonzero()[:, 0]])
        self.pi, self.pj, self.pk, self.side, self.x = (t[order] for t in (i, j, k, side, x))
        self.Q = int(singular.sum())

    # -- outputs of a build
    def probes(self):
        w = self.side.clone()
        w[: self.Q] *= 2.0
        if self.mode == "exterior":  # the index of a singular probe's neighbour block
            w[: self.Q] = 32.0 * torch.arange(self.Q, device=w.device)
        return torch.cat([self.x, w[:, None]], 1)

    def sectors(self):
        i, s = (self.table != 0).nonzero(as_tuple=True)
        v = self.c[self.nb[i, s]] - self.c[i]
        d = _dot(v, v)
        t = (self.R[i].square() - self.R[self.nb[i, s]].square() + d) / (2.0 * d)
        return torch.cat([v / d.sqrt()[:, None], torch.acos((t * d.sqrt() / self.R[i]).clamp(-1.0, 1.0))[:, None]], 1)

    def tori(self):
        n = self.n
        key = self.i * (n + 1) + self.j
        status = self.status.clone()
        for a, b in ((self.pi, self.pj), (self.pi, self.pk), (self.pj, self.pk)):
            at = torch.searchsorted(key, a * (n + 1) + b).clamp_max(len(key) - 1)
            hit = at[(key[at] == a * (n + 1) + b)]
            status[hit[status[hit] == 1]] = 2
        i, j = self.i[status == 2], self.j[status == 2]
        centre, _, radius, t, _ = self._circle(i, j)
        v = self.c[j] - self.c[i]
        rel = v * t[:, None]
        axis = rel / _dot(rel, rel).sqrt()[:, None]
        z = torch.tensor([0.0, 0.0, 1.0], dtype=v.dtype, device=v.device).expand_as(axis)
        ortho = torch.linalg.cross(axis, z)
        ortho = ortho / _dot(ortho, ortho).sqrt()[:, None]
        P = rel + ortho * torch.nan_to_num(radius)[:, None]
        X = P / _dot(P, P).sqrt()[:, None] * (self.R[i] - self.rp)[:, None]
        li, lj = _dot(P, P).sqrt(), _dot(P - v, P - v).sqrt()
        C = v * (li / (lj + li))[:, None]
        dist = _dot(X - C, X - C).sqrt()
        rp = torch.full_like(dist, self.rp)
        return (torch.cat([centre, torch.nan_to_num(radius)[:, None]], 1), torch.cat([axis, rp[:, None]], 1),
                torch.cat([C - rel, dist[:, None]], 1))

    # -- signed distance: every primitive within the best distance so far, hidden ones left out
    def sdf(self, queries, weights=None):
        c, R, n, rp = self.c, self.R, self.n, self.rp
        T = rp + 3.0
        atom_near = _bins(c[:n], float(R[:n].max()) + T)
        probe_near = _bins(self.x, T)
        open_ = torch.cat([(self.table != 0).any(1) | (self.nb >= n).all(1), torch.zeros(1, dtype=torch.bool, device=c.device)])
        px = torch.cat([self.x, torch.full((1, 3), 1e6, dtype=c.dtype, device=c.device)])
        lc, lr = c.clone().requires_grad_(True), R.clone().requires_grad_(True)
        value = torch.empty(len(queries), dtype=c.dtype, device=c.device)
        for r in _rows(len(queries), 0, 4096):
            x = queries[r].double()
            m = len(x)
            near = atom_near(x)
            L = (x[:, None] - c[near]).norm(dim=-1)
            smin = (L - R[near]).min(1).values
            vmin, va = (L - R[near] + rp).min(1)
            va = near.gather(1, va[:, None])[:, 0]
            outside = ~(smin < 0.0)
            pn = probe_near(x)
            best, bp = (x[:, None] - px[pn]).norm(dim=-1).min(1)
            bp = pn.gather(1, bp[:, None])[:, 0]
            probe_d = best
            best = best.clamp_max(T)
            # radial projections on accessible spheres
            q, s = (((L - R[near]).abs() <= best[:, None]) & open_[near] & (~outside & (-smin < T))[:, None]).nonzero(as_tuple=True)
            i = near[q, s]
            on = c[i] + (x[q] - c[i]) / L[q, s][:, None] * R[i][:, None]
            hid = self._hidden(on, i, None)
            ds = torch.where(hid, 1e9, (L[q, s] - R[i]).abs())
            sphere_d = torch.full((m,), 1e9, dtype=c.dtype, device=c.device).scatter_reduce(0, q, ds, "amin")
            best = torch.minimum(best, sphere_d)
            # nearest points of visible circles (i, j), i < j
            cq, ci, cj, cd = [], [], [], []
            for u in _rows(len(q), 2 * self.K):
                qq, ii = q[u], i[u]
                j = self.nb[ii]
                ok = (self.table[ii] != 0) & (j > ii[:, None]) & (j < n)
                ok &= ((x[qq][:, None] - c[j]).norm(dim=-1) - R[j]).abs() <= best[qq][:, None]
                e, s = ok.nonzero(as_tuple=True)
                e_q, e_i, e_j = qq[e], ii[e], j[e, s]
                pt, dist = self._on_circle(x[e_q], e_i, e_j, c, R)
                keep = dist <= best[e_q]
                e_q, e_i, e_j, pt, dist = e_q[keep], e_i[keep], e_j[keep], pt[keep], dist[keep]
                keep = ~self._hidden(pt, e_i, e_j)
                cq.append(e_q[keep]), ci.append(e_i[keep]), cj.append(e_j[keep]), cd.append(dist[keep])
            cq, ci, cj, cd = (torch.cat(t) for t in (cq, ci, cj, cd))
            circle_d = torch.full((m,), 1e9, dtype=c.dtype, device=c.device).scatter_reduce(0, cq, cd, "amin")
            value[r] = torch.where(outside, vmin.clamp_max(3.0), rp - torch.minimum(torch.minimum(best, circle_d), probe_d).clamp_max(T))
            if weights is None:
                continue
            g = weights[r].double()
            inner = ~outside & (-smin < T)
            loss = torch.zeros((), dtype=c.dtype, device=c.device)
            w = (outside & (vmin <= 3.0)).nonzero()[:, 0]
            loss = loss + (g[w] * ((x[w] - lc[va[w]]).norm(dim=-1) - lr[va[w]])).sum()
            least = torch.minimum(torch.minimum(sphere_d, circle_d), probe_d)
            w = (inner & (probe_d <= least) & (probe_d < T)).nonzero()[:, 0]
            b = bp[w]
            pt, _ = self.point(self.pi[b], self.pj[b], self.pk[b], self.side[b], lc, lr)
            loss = loss - (g[w] * (x[w] - pt).norm(dim=-1)).sum()
            first = (ds <= sphere_d[q]) & (sphere_d[q] <= least[q]) & (sphere_d < probe_d)[q] & (sphere_d[q] < T)
            loss = loss - (g[q[first]] * ((x[q[first]] - lc[i[first]]).norm(dim=-1) - lr[i[first]]).abs()).sum()
            first = (cd <= circle_d[cq]) & (circle_d < torch.minimum(sphere_d, probe_d))[cq] & (circle_d[cq] < T)
            _, dist = self._on_circle(x[cq[first]], ci[first], cj[first], lc, lr)
            (loss - (g[cq[first]] * dist).sum()).backward()
        if weights is None:
            return value, None
        grad = torch.empty((n, 4), dtype=c.dtype, device=c.device)
        grad[torch.from_numpy(self.perm).to(c.device)] = torch.cat([lc.grad, lr.grad[:, None]], 1)[:n]
        return value, grad

    def _hidden(self, pt, i, skip):
        out = torch.empty(len(pt), dtype=torch.bool, device=pt.device)
        for u in _rows(len(pt), self.K):
            k = self.nb[i[u]]
            d = pt[u][:, None] - self.c[k]
            h = (_dot(d, d) < self.R[k].square()) & (k < self.n)
            out[u] = (h if skip is None else h & (k != skip[u][:, None])).any(1)
        return out

    def _on_circle(self, x, i, j, c, R):
        v = c[j] - c[i]
        d = _dot(v, v)
        t = (R[i].square() - R[j].square() + d) / (2.0 * d)
        r = (R[i].square() - t * t * d).clamp_min(0.0).sqrt()
        n = v / d.sqrt()[:, None]
        w = x - (c[i] + v * t[:, None])
        h = _dot(w, n)
        flat = w - h[:, None] * n
        rho = _dot(flat, flat).sqrt()
        return x - w + flat * (r / rho)[:, None], (h * h + (rho - r).square()).sqrt()

    # -- area: Gauss-Bonnet on the three 120 degree lunes of every region {y . w <= c}, gradient by autograd
    def area(self):
        n, nb, rp = self.n, self.nb, self.rp
        lc, lr = self.c.clone().requires_grad_(True), self.R.clone().requires_grad_(True)
        per_atom = torch.zeros(n + 1, dtype=lc.dtype, device=lc.device)
        parts = [0.0, 0.0, 0.0]
        open_ = (self.table != 0).any(1) | (nb >= n).all(1)
        for u in _rows(n, self.K * self.K, 1_500_000):
            i = torch.arange(u.start, u.stop, device=nb.device)[open_[u]]
            j = nb[i]
            v = lc[j] - lc[i][:, None]
            d = _dot(v, v).sqrt()
            Ri, Rj = lr[i][:, None], lr[j]
            cons = torch.where(j < n, (Ri * Ri - Rj * Rj + d * d) / (2.0 * d * Ri), 2.0)
            U, angle = _region(v / d[..., None], cons)
            convex = (lr[i] - rp).square() * U
            torus = torch.where((j > i[:, None]) & (j < n) & (angle > 0.0), _torus(d, Ri, Rj, rp) * angle, 0.0)
            (convex.sum() + torus.sum()).backward()
            with torch.no_grad():
                per_atom.index_add_(0, i, convex + 0.5 * torus.sum(1))
                per_atom.index_add_(0, j.flatten(), 0.5 * torus.flatten())
                parts[0] += float(convex.sum())
                parts[1] += float(torus.sum())
        # the surface's primitives are the stored positions of the probes, which follow their atoms by |x - c| = R
        stored = self.x.float().double()
        x = stored.clone().requires_grad_(True)
        idx = torch.full((len(x), 32), len(x), dtype=torch.long, device=nb.device)
        if self.Q:
            near = _bins(stored[: self.Q], 2.0 * rp + 0.01)
            for u in _rows(self.Q, 2000):
                o = near(stored[u])
                me = torch.arange(u.start, u.stop, device=nb.device)[:, None]
                p = torch.cat([stored[: self.Q], stored.new_full((1, 3), 1e6)])
                ok = ((stored[u][:, None] - p[o]).norm(dim=-1) < 2.0 * rp) & (o != me) & (o < self.Q)
                idx[u] = torch.nn.functional.pad(torch.where(ok, o, len(x)).sort(1).values, (0, 32), value=len(x))[:, :32]
        ids = torch.stack([self.pi, self.pj, self.pk], 1)
        for u in _rows(len(x), 35 * 35, 1_500_000):
            v = lc[ids[u]] - x[u][:, None]
            v = v / _dot(v, v).sqrt()[..., None]
            e = torch.linalg.cross(v, v.roll(-1, 1))
            side = torch.sign(_dot(e, v.roll(-2, 1)))
            w = -side[..., None] * e / _dot(e, e).sqrt()[..., None]
            most = max(1, int((idx[u] < len(x)).sum(1).max()))
            o = idx[u][:, :most]
            D = torch.cat([x, x.detach().new_full((1, 3), 1e6)])[o] - x[u][:, None]
            l = _dot(D, D).sqrt()
            ok = (o < len(x)) & (l < 2.0 * rp)
            U, _ = _region(torch.cat([w, D / l[..., None]], 1), torch.cat([torch.zeros_like(side), torch.where(ok, l / (2.0 * rp), 2.0)], 1))
            patch = rp * rp * U
            patch.sum().backward()
            with torch.no_grad():
                per_atom.index_add_(0, ids[u].flatten(), (patch / 3.0).repeat_interleave(3))
                parts[2] += float(patch.sum())
        arm = stored[:, None] - self.c[ids]
        lam = torch.linalg.solve(arm.transpose(1, 2), x.grad)
        gc, gr = lc.grad, lr.grad
        gc.index_add_(0, ids.flatten(), (lam[..., None] * arm).flatten(0, 1))
        gr.index_add_(0, ids.flatten(), (lam * self.R[ids]).flatten())
        out, grad = per_atom.new_empty(n), per_atom.new_empty((n, 4))
        perm = torch.from_numpy(self.perm).to(out.device)
        out[perm] = per_atom[:n]
        grad[perm] = torch.cat([gc, gr[:, None]], 1)[:n]
        return np.array(parts), out, grad


def _torus(d, Ri, Rj, rp):
    """Area per unit angle of the torus of two spheres between its contact circles, trimmed at its axis."""
    hi = (Ri * Ri - Rj * Rj + d * d) / (2.0 * d)
    hj = d - hi
    rho = (Ri * Ri - hi * hi).clamp_min(1e-30).sqrt()
    F = rho * (torch.atan2(hj, rho) + torch.atan2(hi, rho)) - rp * (hj / Rj + hi / Ri)
    cut = (rho < rp) & (hi > 0.0) & (hj > 0.0)
    k = torch.where(cut, rho / rp, 0.5)
    return rp * (F - torch.where(cut, 2.0 * rho * torch.acos(k) - 2.0 * rp * (1.0 - k * k).sqrt(), 0.0))


def _turn(w, c, s, e1, e2, phi):
    """Angle of the boundary's tangent at phi against a frame field of the sphere."""
    a = torch.tensor([0.32140077, 0.55410134, 0.76790185], dtype=w.dtype, device=w.device)
    y = w * c[..., None] + (e1 * phi.cos()[..., None] + e2 * phi.sin()[..., None]) * s[..., None]
    t = e1 * phi.sin()[..., None] - e2 * phi.cos()[..., None]
    xi = a - y * _dot(a.expand_as(y), y)[..., None]
    return torch.atan2(_dot(torch.linalg.cross(xi, t), y), _dot(xi, t))


def _region(w, c):
    """Area of {y . w_m <= c_m} on the unit sphere for a batch of regions, and the boundary angle of every circle."""
    B, M = c.shape
    tau = 2.0 * math.pi
    area, angle = 0.0, torch.zeros_like(c)
    ax = w.detach().abs()
    unit = torch.nn.functional.one_hot(ax.argmin(-1), 3).to(w.dtype)
    for lune in range(3):
        al, be = tau * lune / 3.0, tau * (lune + 1) / 3.0
        pair = torch.tensor([[math.sin(al), -math.cos(al), 0.0], [-math.sin(be), math.cos(be), 0.0]], dtype=w.dtype, device=w.device)
        W = torch.cat([w, pair.expand(B, 2, 3)], 1)
        C = torch.cat([c, c.new_zeros(B, 2)], 1)
        un = torch.cat([unit, torch.tensor([0.0, 0.0, 1.0], dtype=w.dtype, device=w.device).expand(B, 2, 3)], 1)
        live = C < 1.0
        S = torch.where(live, (1.0 - C) * (1.0 + C), 1.0).clamp_min(1e-30).sqrt()
        e1 = torch.linalg.cross(W, un)
        e1 = e1 / _dot(e1, e1).sqrt()[..., None]
        e2 = torch.linalg.cross(W, e1)
        # cut of circle m by cap n
        p1, p2 = e1 @ W.transpose(1, 2), e2 @ W.transpose(1, 2)
        rhs = C[:, None, :] - C[:, :, None] * (W @ W.transpose(1, 2))
        b = S[:, :, None] * (p1 * p1 + p2 * p2).clamp_min(1e-300).sqrt()
        other = live[:, None, :] & ~torch.eye(M + 2, dtype=torch.bool, device=c.device)
        cut = other & (b > rhs.abs())
        gone = (other & ~cut & (rhs < 0.0)).any(2) | ~live
        delta = torch.atan2(torch.where(cut, (b - rhs) * (b + rhs), 1.0).sqrt(), torch.where(cut, rhs, 1.0))
        start = torch.where(cut, torch.remainder(torch.atan2(p2, p1) - delta, tau), 1e9)
        end = torch.where(cut, start + 2.0 * delta, -1e9)
        order = start.argsort(2)
        st, en = start.gather(2, order), end.gather(2, order)
        st, en = torch.cat([st, torch.where(st < 1e8, st + tau, 1e9)], 2), torch.cat([en, torch.where(en > -1e8, en + tau, -1e9)], 2)
        # the second turn's starts are sorted after the first's
        o2 = st.argsort(2)
        st, en = st.gather(2, o2), en.gather(2, o2)
        top, _ = torch.cummax(en, 2)
        gap = st[:, :, 1:] - top[:, :, :-1]
        good = (gap > 0.0) & (st[:, :, 1:] < 1e8) & (st[:, :, 1:] >= tau) & ~gone[..., None]
        whole = ~gone & ~cut.any(2)
        m = good.nonzero(as_tuple=True)
        a, g = top[:, :, :-1][m], gap[m]
        args = [t[m[0], m[1]] for t in (W, C, S, e1, e2)]
        turn = _turn(*args, a) - _turn(*args, a + g)
        per = torch.zeros_like(C).index_put((m[0], m[1]), C[m[0], m[1]] * g + turn, accumulate=True)
        total = (per + torch.where(whole, C * tau, 0.0)).sum(1)
        total = torch.remainder(total, tau)
        total = torch.where(total > 5.0 * math.pi / 3.0, total - tau, total)
        area = area + torch.where((c > -1.0).all(1), total.clamp_min(0.0), 0.0)
        phi = torch.zeros_like(C).index_put((m[0], m[1]), g, accumulate=True) + torch.where(whole, tau, 0.0)
        angle = angle + phi[:, :M]
    return area, angle


def exact(case, seed):
    kind, rp = case["kind"], case["probe"]
    if kind == "image":
        return None  # a marched ray ends within eps of the surface: no one value
    if kind == "batch":
        mols = _batch(case, seed)
    elif case["atoms"] > GLOBULE_MOST * 4:
        return None  # over 20 s
    else:
        mols = [_molecule(case["atoms"], seed, rp)]
    if kind == "cavities":
        a = mols[0].astype(np.float64)
        lo = (a[:, :3] - (a[:, 3:] + float(np.float32(rp)))).min(0) - 2 * case["voxel"]
        return {"origin": lo}
    mode = case.get("mode", "full")
    built = [_Surface(m, rp, mode) for m in mols]
    if kind in ("build", "batch"):
        n = sum(s.n for s in built)
        out = {"atoms": [s.atoms.double() for s in built], "probes": [s.probes() for s in built]}
        if mode == "full":
            out["sectors"] = [s.sectors() for s in built]
        else:
            out["tori"], out["axes"], out["spheres"] = zip(*(s.tori() for s in built))
        rows = _FULL if mode == "full" else _EXTERIOR
        out = {k: torch.cat(list(v)) for k, v in out.items()}
        return {k: torch.nn.functional.pad(v, (0, 0, 0, rows[k][4] * n - len(v))) for k, v in out.items()}
    s = built[0]
    if kind == "area":
        parts, area, grad = s.area()
        return {"parts": parts, "area": area, "grad": grad}
    value, grad = s.sdf(_queries(case, seed, mols[0]), _weights(case["queries"], seed) if kind == "sdf_train" else None)
    return {"sdf": value} if kind == "sdf" else {"sdf": value, "grad": grad}
