"""Performance cases of the neighbour-list engine.

Each case is one piece of work a program has the package do, called through its
public functions.  The families (``work`` key of a case):

host      ``neighbour_list`` on numpy arrays, numpy arrays back: an interactive or
          ASE-driven script on a small cell.
list      ``neighbour_list`` on positions that live on the GPU, results left there:
          molecular dynamics and machine-learned potentials, from a thousand atoms
          to a million, dense, layered and dilute.
batch     ``NeighbourListBatch.run``: a data set of small systems rebuilt together.
grad      ``neighbour_list_autograd`` forward and backward: training on forces and
          stresses.
lj        ``lennard_jones``: one force evaluation of a large pair-potential run.
verlet    ``VerletList.update`` between rebuilds: a stored list with a skin.
triplets  ``first_neighbours`` + ``triplet_list`` on a device list: the angular terms
          of three-body potentials.
matrix    ``neighbour_matrix``: the padded list that graph networks read.

A system is made on the GPU from the seed alone: ``uniform`` random positions,
or an ``fcc`` / ``cubic`` lattice with Gaussian jitter, at a number density, in
a sheared cell with the given periodicity; ``vacuum`` stretches the cell along
z around a slab of atoms.  Lattice sites fill the cell plane by plane, so a
count that is no full lattice leaves the last plane ragged.
"""

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("matscipy-neighbours_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from matscipy_neighbours import (first_neighbours, lennard_jones, neighbour_list,  # noqa: E402
                                 neighbour_matrix, triplet_list)
from matscipy_neighbours.autograd import neighbour_list_autograd  # noqa: E402
from matscipy_neighbours.batch import NeighbourListBatch  # noqa: E402
from matscipy_neighbours.verlet import VerletList  # noqa: E402

_PAIR_BYTES = {"i": 4, "j": 4, "d": 8, "D": 24, "S": 12}
_FCC = 4.0 / 3.6 ** 3      # atoms per A^3 of the fcc metal (lattice constant 3.6 A)


def listed():
    return [
        # One molecule or primitive cell at a time from a script: all of it is
        # latency (argument handling, launches, copies).
        dict(name="host_100", work="host", n=100, place="uniform", density=0.1, rc=4.0,
             cut="scalar", pbc="TTT", shear=0.0, vacuum=1.0, quantities="ijdDS"),
        # The small MD cell: 1,000 atoms, every step a fresh list.
        dict(name="list_1000", work="list", n=1000, place="uniform", density=1.0, rc=2.5,
             cut="scalar", pbc="TTT", shear=0.0, vacuum=1.0, quantities="ijdDS"),
        # An ordinary liquid at a water-like density, a count that is no round
        # number, as a graph network asks for it (edges and shifts).
        dict(name="list_10007", work="list", n=10007, place="uniform", density=0.1, rc=5.0,
             cut="scalar", pbc="TTT", shear=0.05, vacuum=1.0, quantities="ijDS"),
        # The bulk metal of the benchmark: a million atoms, everything returned.
        dict(name="list_fcc_1M", work="list", n=1048576, place="fcc", density=_FCC, rc=5.0,
             cut="scalar", pbc="TTT", shear=0.2, vacuum=1.0, quantities="ijdDS"),
        # A layer in vacuum with a cutoff per pair of species.
        dict(name="list_slab_200k", work="list", n=200000, place="uniform", density=0.03125,
             rc=4.0, cut="type", pbc="TTF", shear=0.0, vacuum=10.0, quantities="ijdD"),
        # A dilute gas: most cells empty, about two neighbours per atom.
        dict(name="list_gas_200k", work="list", n=200000, place="uniform", density=0.0185185,
             rc=3.0, cut="scalar", pbc="TTT", shear=0.0, vacuum=1.0, quantities="ijdDS"),
        # A training set of small periodic and open systems, rebuilt per step.
        dict(name="batch_4096", work="batch", nsys=4096, nmin=8, nmax=512, density=0.08,
             rmin=3.0, rmax=6.0, quantities="ijdDS"),
        # A training step through distances on a jittered lattice.
        dict(name="grad_132651", work="grad", n=132651, place="cubic", density=2.8 ** -3, rc=6.0,
             cut="scalar", pbc="TTT", shear=0.1, vacuum=1.0, quantities="ijDdS"),
        # One force call of a million-atom Lennard-Jones crystal in an open box.
        dict(name="lj_1M", work="lj", n=1000000, place="fcc", density=4.0 / 1.6 ** 3, rc=2.5,
             cut="scalar", pbc="FFF", shear=0.0, vacuum=1.0, quantities=""),
        # A step between two rebuilds of the stored list.
        dict(name="verlet_fcc_1M", work="verlet", n=1048576, place="fcc", density=_FCC, rc=5.0,
             cut="scalar", pbc="TTT", shear=0.2, vacuum=1.0, quantities="ijdDS", skin=0.5),
        # Angular terms inside a shorter cutoff than the list's.
        dict(name="triplets_132651", work="triplets", n=132651, place="cubic",
             density=2.8 ** -3, rc=6.0, cut="scalar", pbc="TTT", shear=0.1, vacuum=1.0,
             quantities="id", rc3=3.5),
        # The padded matrix of a metal for a graph network.
        dict(name="matrix_131072", work="matrix", n=131072, place="fcc", density=_FCC, rc=5.0,
             cut="scalar", pbc="TTT", shear=0.2, vacuum=1.0, quantities="jD", width=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["host", "list", "list", "list", "list", "batch", "grad", "lj", "verlet",
                       "triplets", "matrix"])
    if kind == "batch":
        nmin = rng.choice([2, 8, 20])
        return dict(work="batch", nsys=int(_log(rng, 48, 4096)), nmin=nmin,
                    nmax=int(nmin * _log(rng, 4, 512 / nmin)), density=rng.uniform(0.04, 0.1),
                    rmin=rng.uniform(1.5, 3.0), rmax=rng.uniform(3.0, 5.5),
                    quantities=rng.choice(["ijdDS", "ijdD", "ijDS", "ijd"]))
    lo, hi = {"host": (20, 3000), "list": (500, 1048576), "grad": (2000, 200000),
              "lj": (4000, 1000000), "verlet": (4000, 1048576), "triplets": (2000, 200000),
              "matrix": (2000, 262144)}[kind]
    n = int(_log(rng, lo, hi)) | 1
    place = rng.choice(["uniform", "fcc", "cubic"])
    if kind in ("lj", "triplets", "matrix"):
        place = rng.choice(["fcc", "cubic"])   # no two atoms (nearly) on top of each other
    density = _log(rng, 0.02, 1.0)
    want = _log(rng, 1.5, 65.0) if kind in ("host", "list") else _log(rng, 14.0, 55.0)
    c = dict(work=kind, n=n, place=place, density=density,
             rc=(want / (4.0 / 3.0 * math.pi * density)) ** (1.0 / 3.0),
             cut=rng.choice(["scalar", "scalar", "atom", "type"]) if kind in ("host", "list")
             else "scalar",
             pbc=rng.choice(["TTT", "TTT", "TTF", "FFF", "TFT"]),
             shear=rng.choice([0.0, 0.0, 0.1, 0.3]),
             vacuum=rng.choice([1.0, 1.0, 3.0, 10.0]) if kind in ("host", "list") else 1.0,
             quantities={"grad": "ijDdS", "lj": "", "triplets": "id", "matrix": "jD"}.get(
                 kind, rng.choice(["ijdDS", "ijdDS", "ijdD", "ijDS", "ijd", "ij"])))
    if kind == "verlet":
        c["skin"] = c["rc"] * rng.uniform(0.05, 0.12)
    if kind == "triplets":
        c["rc3"] = c["rc"] * rng.uniform(0.5, 0.75)
    if kind == "matrix":
        c["width"] = int(1.6 * want) + 16
    return c


# -- inputs ------------------------------------------------------------------

def _gen(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _dims(case):
    """Sites along each axis and sites per lattice cell."""
    per = 4 if case["place"] == "fcc" else 1
    cells = -(-case["n"] // per)
    nx = max(1, math.ceil(cells ** (1.0 / 3.0) - 1e-9))
    ny = max(1, math.ceil(math.sqrt(cells / nx) - 1e-9))
    return nx, ny, -(-cells // (nx * ny)), per


def _system(case, seed, device):
    """Positions (device tensor), cell, pbc, cutoff and types of one system.
    The structure is the case's own; the seed says where it sits in the cell
    (shifted along every axis, wrapped on periodic ones) and which atom is the
    first, so that every seed has other numbers and the same number of pairs."""
    n, g, at = case["n"], _gen(20011, device), np.random.default_rng(seed)
    f64 = dict(dtype=torch.float64, device=device)
    pbc = np.array([c == "T" for c in case["pbc"]])
    shift = at.uniform(0.0, 1.0, 3)
    roll = int(at.integers(0, n))
    if case["place"] == "uniform":
        slab = (n / case["density"] / case["vacuum"] ** 2) ** (1.0 / 3.0)
        edge = np.array([slab * case["vacuum"]] * 2 + [slab])  # a slab as wide as the cell is high
        frac = torch.rand((n, 3), generator=g, **f64)
        edge *= 1.0 + 1e-9    # not a whole number of cutoffs wide to the last bit
        jitter = None
    else:
        nx, ny, nz, per = _dims(case)
        a = (per / case["density"]) ** (1.0 / 3.0)
        edge = a * np.array([nx, ny, nz], dtype=float)
        site = torch.arange(n, device=device)
        unit = site // per
        base = torch.tensor([[0.0, 0.0, 0.0], [0.5, 0.5, 0.0], [0.5, 0.0, 0.5],
                             [0.0, 0.5, 0.5]], **f64)[site % per]
        xyz = torch.stack([unit % nx, (unit // nx) % ny, unit // (nx * ny)], dim=1).to(torch.float64)
        frac = (xyz + base + 0.25) / torch.tensor([nx, ny, nz], **f64)
        # thermal displacements: some three hundredths of the lattice constant
        jitter = torch.randn((n, 3), generator=g, **f64) * (0.03 * a)
    s = case["shear"] * edge[0]
    cell = np.array([[edge[0], 0.0, 0.0], [s, edge[1], 0.0], [0.5 * s, 0.0, edge[2]]])
    # open axes: a vacuum around the slab, else room for the shift
    wide = np.array([1.0, 1.0, case["vacuum"]])
    wide = np.where(pbc | (wide > 1.0), wide, 1.02)
    cell *= wide[:, None]
    wide, shift = torch.from_numpy(wide).to(device), torch.from_numpy(shift).to(device)
    per = torch.from_numpy(pbc).to(device)
    frac = frac / wide + shift * torch.where(per, 1.0, 1.0 - 1.0 / wide)
    frac = torch.where(per, frac - torch.floor(frac), frac)
    ct = torch.from_numpy(cell).to(device)
    pos = frac @ ct
    if jitter is not None:
        if not pbc.all():          # open axes: the jittered atoms stay in the box
            f = jitter @ torch.linalg.inv(ct)
            room = 0.2 / torch.tensor([nx, ny, nz], **f64) / wide
            jitter = torch.where(per, f, torch.maximum(torch.minimum(f, room), -room)) @ ct
        pos = pos + jitter
    rc, types, moved = float(case["rc"]), None, None
    cutoff = rc
    if case["cut"] == "atom":     # radii: the widest pair reaches rc
        cutoff = rc * (0.25 + 0.25 * torch.rand(n, generator=g, **f64))
        cutoff = cutoff.roll(roll).cpu().numpy()
    elif case["cut"] == "type":
        types = torch.randint(0, 2, (n,), generator=g, device=device).to(torch.int32)
        types = types.roll(roll).cpu().numpy()
        cutoff = rc * np.array([[0.5, 0.75], [0.75, 1.0]])
    if "skin" in case:            # some steps later: displaced by less than half the skin
        moved = pos + (torch.rand((n, 3), generator=g, **f64) - 0.5) * (0.5 * case["skin"])
        moved = moved.roll(roll, 0).contiguous()
    return dict(positions=pos.roll(roll, 0).contiguous(), cell=cell, pbc=pbc, cutoff=cutoff,
                numbers=types, moved=moved)


def _batch_systems(case, seed):
    """Small systems, sizes log-uniform, each with its own triclinic cell and
    periodicity and a radius per atom; placed by the seed as in _system."""
    rng, at = np.random.default_rng(20011), np.random.default_rng(seed)
    out = []
    for _ in range(case["nsys"]):
        n = int(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1))))
        n = min(max(n, case["nmin"]), case["nmax"])
        e = rng.uniform(8.0, 25.0, 3)
        al, be, ga = np.radians(rng.uniform(75.0, 105.0, 3))
        cx, cy = math.cos(be), (math.cos(al) - math.cos(be) * math.cos(ga)) / math.sin(ga)
        cell = np.array([[e[0], 0.0, 0.0], [e[1] * math.cos(ga), e[1] * math.sin(ga), 0.0],
                         [e[2] * cx, e[2] * cy, e[2] * math.sqrt(1.0 - cx * cx - cy * cy)]])
        cell *= (n / case["density"] / abs(np.linalg.det(cell))) ** (1.0 / 3.0)
        cell *= max(1.0, 8.0 / np.linalg.norm(cell, axis=1).min())
        pbc = rng.integers(0, 2, 3).astype(bool)
        frac, radii = rng.uniform(0.0, 1.0, (n, 3)), rng.uniform(case["rmin"], case["rmax"], n)
        wide, roll = np.where(pbc, 1.0, 1.02), int(at.integers(0, n))
        cell *= wide[:, None]
        frac = frac / wide + at.uniform(0.0, 1.0, 3) * np.where(pbc, 1.0, 1.0 - 1.0 / wide)
        frac = np.where(pbc, frac - np.floor(frac), frac)
        out.append(dict(positions=np.roll(frac @ cell, roll, axis=0), cell=cell, pbc=pbc,
                        cutoff=np.roll(radii, roll)))
    first = int(at.integers(0, len(out)))
    return out[first:] + out[:first]


# -- one pass ----------------------------------------------------------------

def _device_list(quantities, s):
    return neighbour_list(quantities, positions=s["positions"], cell=s["cell"], pbc=s["pbc"],
                          cutoff=s["cutoff"], numbers=s["numbers"], array_namespace=torch)


def _upstream(case, seed, npairs, device):
    """The gradients a model hands back for D and d."""
    g = _gen(seed + 104729, device)
    return (torch.randn((npairs, 3), generator=g, dtype=torch.float64, device=device),
            torch.randn(npairs, generator=g, dtype=torch.float64, device=device))


def prepare(case, seed):
    kind = case["work"]
    if kind == "batch":
        return dict(case=case, batch=NeighbourListBatch(_batch_systems(case, seed),
                                                        case["quantities"]))
    s = _system(case, seed, "cuda")
    s["case"] = case
    if kind == "host":
        s["positions"] = s["positions"].cpu().numpy()
    elif kind == "verlet":
        s["list"] = VerletList(case["rc"], case["skin"], s["cell"], s["pbc"], case["quantities"])
        s["list"].update(s["positions"])
    elif kind == "grad":
        npairs = _device_list("i", s).shape[0]
        s["gD"], s["gd"] = _upstream(case, seed, npairs, s["positions"].device)
        s["positions"].requires_grad_(True)
        s["cell_t"] = torch.from_numpy(s["cell"]).cuda().requires_grad_(True)
    elif kind == "triplets":
        s["i"], s["d"] = _device_list("id", s)
    return s


def run(state):
    case = state["case"]
    kind = case["work"]
    if kind == "host":
        return neighbour_list(case["quantities"], positions=state["positions"],
                              cell=state["cell"], pbc=state["pbc"], cutoff=state["cutoff"],
                              numbers=state["numbers"])
    if kind == "list":
        return _device_list(case["quantities"], state)
    if kind == "batch":
        state["batch"].run()
        out = state["batch"].results()
        for t in out:           # views of the batch's own buffers: they keep it alive
            t.batch = state["batch"]
        return out
    if kind == "grad":
        i, j, D, d, S = neighbour_list_autograd(state["positions"], state["cell_t"],
                                                state["pbc"], state["cutoff"])
        gr, gc = torch.autograd.grad((D, d), (state["positions"], state["cell_t"]),
                                     (state["gD"], state["gd"]))
        return D.detach(), d.detach(), gr, gc
    if kind == "lj":
        return lennard_jones(state["positions"], state["cutoff"], cell=state["cell"],
                             pbc=state["pbc"])
    if kind == "verlet":
        return state["list"].update(state["moved"])
    if kind == "triplets":
        seed = first_neighbours(case["n"], state["i"])
        return (seed,) + tuple(triplet_list(seed, state["d"], case["rc3"]))
    return neighbour_matrix(positions=state["positions"], cell=state["cell"], pbc=state["pbc"],
                            cutoff=state["cutoff"], max_neighbours=case["width"],
                            array_namespace=torch)


# -- what a pass cannot do without --------------------------------------------

def _pairs(case, rc=None):
    """Expected directed pairs: the density's sphere, less what open faces cut
    off, at the mean cubed cutoff of the pairs."""
    rc = case["rc"] if rc is None else rc
    n = case["n"]
    r3 = {"scalar": 1.0, "type": (0.5 ** 3 + 2 * 0.75 ** 3 + 1.0) / 4.0,
          "atom": 0.4375}[case["cut"]] * rc ** 3
    per = case["density"] * 4.0 / 3.0 * math.pi * r3
    if case["place"] == "uniform":
        slab = (n / case["density"] / case["vacuum"] ** 2) ** (1.0 / 3.0)
        edge = [slab * case["vacuum"]] * 2 + [slab]
    else:
        nx, ny, nz, sites = _dims(case)
        a = (sites / case["density"]) ** (1.0 / 3.0)
        edge = [a * nx, a * ny, a * nz]
    for k in range(3):
        if case["pbc"][k] == "F" or (k == 2 and case["vacuum"] > 1.0):
            per *= max(0.3, 1.0 - 0.375 * rc / edge[k])
    return n * per


def work(case):
    kind = case["work"]
    if kind == "batch":
        lo, hi = case["nmin"], case["nmax"]
        n = case["nsys"] * (hi - lo) / max(math.log(hi / lo), 1e-9)
        r = 0.5 * (case["rmin"] + case["rmax"])
        r3 = (2 * r) ** 3 + 6 * r * (case["rmax"] - case["rmin"]) ** 2 / 6.0
        # half of the axes are open and the boxes are about as wide as the
        # cutoff: three fifths of the neighbours of the full sphere are there
        pairs = 0.6 * n * case["density"] * 4.0 / 3.0 * math.pi * r3
        return {"bytes": pairs * sum(_PAIR_BYTES[q] for q in case["quantities"]) + 32.0 * n,
                "flops": 12.0 * pairs}
    n, pairs = case["n"], _pairs(case)
    per = sum(_PAIR_BYTES[q] for q in case["quantities"])
    atom = 24.0 + {"scalar": 0.0, "atom": 8.0, "type": 4.0}[case["cut"]]
    if kind == "grad":
        # the list out; then i, j, S, D, d and both gradients in
        return {"bytes": pairs * (52.0 + 84.0) + 2 * 24.0 * n, "flops": 40.0 * pairs}
    if kind == "lj":
        return {"bytes": 56.0 * n, "flops": 30.0 * pairs}
    if kind == "verlet":
        stored = _pairs(case, case["rc"] + case["skin"])
        return {"bytes": 20.0 * stored + per * pairs + 2 * 24.0 * n, "flops": 20.0 * stored}
    if kind == "triplets":
        m = _pairs(case, case["rc3"]) / n
        return {"bytes": 12.0 * pairs + 4.0 * n + 8.0 * n * m * max(m - 1.0, 1.0),
                "flops": pairs}
    if kind == "matrix":
        return {"bytes": n * (28.0 * case["width"] + 28.0), "flops": 12.0 * pairs}
    return {"bytes": per * pairs + atom * n, "flops": 12.0 * pairs}


# -- the same in plain torch ---------------------------------------------------

def _grid(cell, rc):
    """Cells and scanned cells per axis of a grid with cells at least rc wide."""
    vol = abs(np.linalg.det(cell))
    width = np.array([vol / np.linalg.norm(np.cross(cell[(k + 1) % 3], cell[(k + 2) % 3]))
                      for k in range(3)])
    n = np.maximum(np.floor(width / rc).astype(int), 1)
    return n, np.ceil(rc * n / width).astype(int)


def _pairs_of(pos, cell, pbc, cutoff, types=None):
    """All pairs (i, j, S, D) of one system in the package's documented order:
    by i, then by neighbour cell (z, y, x), then by j."""
    dev = pos.device
    n = pos.shape[0]
    radii = matrix = None
    if np.ndim(cutoff) == 1:
        radii, rc = torch.from_numpy(cutoff).to(dev), float(2.0 * cutoff.max())
    elif np.ndim(cutoff) == 2:
        matrix, rc = torch.from_numpy(cutoff).to(dev), float(cutoff.max())
        types = torch.from_numpy(types).to(dev).long()
    else:
        rc = float(cutoff)
    nc, ns = _grid(cell, rc)
    ct = torch.from_numpy(cell).to(dev)
    nct = torch.from_numpy(nc).to(dev)
    per = torch.from_numpy(np.asarray(pbc)).to(dev)
    raw = torch.floor((pos @ torch.linalg.inv(ct)) * nct).long()
    home = torch.where(per, raw % nct, torch.minimum(raw.clamp(min=0), nct - 1))
    image = torch.where(per, torch.div(raw, nct, rounding_mode="floor"), torch.zeros_like(raw))
    lin = home[:, 0] + nct[0] * (home[:, 1] + nct[1] * home[:, 2])
    scan = torch.from_numpy(np.array([[x, y, z] for z in range(-ns[2], ns[2] + 1)
                                      for y in range(-ns[1], ns[1] + 1)
                                      for x in range(-ns[0], ns[0] + 1)])).to(dev)

    def target(off):
        """Folded neighbour cells at offset(s) `off`: index, image, inside."""
        t = home + off
        m = torch.where(per, torch.div(t, nct, rounding_mode="floor"), torch.zeros_like(t))
        t = t - m * nct
        ok = ((t >= 0) & (t < nct)).all(dim=-1)
        return t[..., 0] + nct[0] * (t[..., 1] + nct[1] * t[..., 2]), m, ok

    def within(i, j, m, zero):
        """The candidates inside their cutoff, as (i, j, S)."""
        S = image[i] - image[j] + m
        D = pos[j] - pos[i] + S.to(torch.float64) @ ct
        r2 = (D * D).sum(dim=1)
        good = (r2 < rc * rc) & ~(zero & (i == j))
        if radii is not None:
            good &= r2 < (radii[i] + radii[j]) ** 2
        elif matrix is not None:
            good &= r2 < matrix[types[i], types[j]] ** 2
        return i[good].int(), j[good].int(), S[good].int()

    keep = []
    if n <= 1024:                  # every (offset, i, j) at once
        key, m, ok = target(scan[:, None, :])
        v, i, j = torch.nonzero(ok[:, :, None] & (key[:, :, None] == lin), as_tuple=True)
        keep.append(within(i, j, m[v, i], (scan[v] == 0).all(dim=1)))
    else:                          # one offset at a time over the sorted cells
        order = torch.argsort(lin, stable=True)
        sorted_lin = lin[order]
        for off in scan:
            key, m, ok = target(off)
            b = torch.searchsorted(sorted_lin, key)
            ln = torch.where(ok, torch.searchsorted(sorted_lin, key, right=True) - b, 0)
            i = torch.repeat_interleave(torch.arange(n, device=dev), ln)
            j = order[(b - torch.cumsum(ln, 0) + ln)[i] + torch.arange(i.numel(), device=dev)]
            keep.append(within(i, j, m[i], bool((off == 0).all())))
    i, j, S = (torch.cat(v) for v in zip(*keep))
    by_i = torch.argsort(i, stable=True)
    i, j, S = i[by_i], j[by_i], S[by_i]
    return i, j, S, pos[j.long()] - pos[i.long()] + S.to(torch.float64) @ ct


def _picked(quantities, i, j, S, D):
    d = (D * D).sum(dim=1).sqrt()
    return tuple({"i": i, "j": j, "S": S, "D": D, "d": d}[q] for q in quantities)


def exact(case, seed):
    kind = case["work"]
    if kind == "triplets":
        return None     # whole numbers only
    if kind == "batch":
        parts = [_pairs_of(torch.from_numpy(s["positions"]).cuda(), s["cell"], s["pbc"],
                           s["cutoff"]) for s in _batch_systems(case, seed)]
        return _picked(case["quantities"], *(torch.cat(v) for v in zip(*parts)))
    s = _system(case, seed, "cuda")
    pos, cell, pbc, cutoff, types = (s["positions"], s["cell"], s["pbc"], s["cutoff"],
                                     s["numbers"])
    if kind == "verlet":
        i, j, S, _ = _pairs_of(pos, cell, pbc, case["rc"] + case["skin"])
        new = s["moved"]
        D = new[j.long()] - new[i.long()] + S.to(torch.float64) @ torch.from_numpy(cell).to(pos.device)
        near = (D * D).sum(dim=1) < case["rc"] ** 2
        return _picked(case["quantities"], i[near], j[near], S[near], D[near])
    i, j, S, D = _pairs_of(pos, cell, pbc, cutoff, types)
    n = case["n"]
    if kind == "grad":
        d = (D * D).sum(dim=1).sqrt()
        gD, gd = _upstream(case, seed, i.numel(), pos.device)
        g = gD + (gd / d)[:, None] * D
        gr = torch.zeros_like(pos)
        gr.index_add_(0, j.long(), g)
        gr.index_add_(0, i.long(), -g)
        return D, d, gr, S.to(torch.float64).T @ g
    if kind == "lj":
        s6 = (1.0 / (D * D).sum(dim=1)) ** 3
        f = torch.zeros_like(pos)
        f.index_add_(0, i.long(), (-24.0 * s6 * (2.0 * s6 - 1.0) / (D * D).sum(dim=1))[:, None] * D)
        return (2.0 * (s6 * s6 - s6)).sum(), f
    if kind == "matrix":
        K = case["width"]
        count = torch.bincount(i.long(), minlength=n)
        slot = torch.arange(i.numel(), device=pos.device) - (torch.cumsum(count, 0) - count)[i.long()]
        idx = torch.zeros((n, K), dtype=torch.int32, device=pos.device)
        dist = torch.zeros((n, K, 3), dtype=torch.float64, device=pos.device)
        idx[i.long(), slot] = j
        dist[i.long(), slot] = D
        return idx, dist, count.int()
    return _picked(case["quantities"], i, j, S, D)
