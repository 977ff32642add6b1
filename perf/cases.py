"""Performance cases: what a user of this package has it compute, through its public entry points.

Three kinds of case:
  search   one receptor, one ligand with its conformers and rotations: Receptor.search (host
           buffers) or Receptor.search_device (device buffers, optionally graph replay);
  serve    a burst of docking requests of uneven size through one Server;
  cluster  the diverse-conformer selection that precedes docking.

Inputs are synthetic and seeded: receptor atoms uniform in a cube, soft-core capped
Lennard-Jones grids at eight probe radii and a capped Coulomb grid, a compact ligand whose atoms
use some of the eight radius classes, conformers perturbed by up to 0.5 A per axis, uniform
quaternions.
"""
import math

import numpy as np
import torch

from cdocker_b200 import CDK_FORM_BF16X3, CDK_FORM_FP16X2, CDK_FORM_FP32, Receptor
from cdocker_b200.conformers import cluster_conformers
from cdocker_b200.serving import Server

FORMS = {"fp32": CDK_FORM_FP32, "bf16x3": CDK_FORM_BF16X3, "fp16x2": CDK_FORM_FP16X2}
SPACING = 0.5
PROBES = np.linspace(1.2, 2.2, 8).astype(np.float32)
# receptor atoms and cube edge (A) per grid edge
RECEPTORS = {32: (400, 16.0), 64: (2500, 32.0), 96: (6000, 48.0), 128: (12000, 64.0)}


def _search(name, n, form, atoms, confs, rots, classes=8, device=False, graphs=False):
    return {"name": name, "kind": "search", "n": n, "form": form, "atoms": atoms, "confs": confs,
            "rots": rots, "classes": classes, "device": device, "graphs": graphs}


def listed():
    return [
        # one small ligand against a small site, the size of a first try or a unit of a screen
        _search("search 32 fp32", 32, "fp32", 24, 1, 500),
        # the smallest call: a fragment with a few refinement rotations; latency and launches
        _search("search 64 fp16x2 smallest", 64, "fp16x2", 11, 1, 61, classes=3),
        # the default form at production grid size, a few conformers of one ligand
        _search("search 64 fp32", 64, "fp32", 40, 5, 1000),
        # the batch that a docking run repeats per ligand: inputs resident, graph replay
        _search("search 64 fp16x2 batch", 64, "fp16x2", 40, 100, 1000, device=True, graphs=True),
        # the same grid in the more precise tensor-core form, from host buffers
        _search("search 64 bf16x3", 64, "bf16x3", 40, 20, 1000),
        # a ligand past the 96 atoms of the direct plane path (peptides, macrocycles)
        _search("search 64 bf16x3 large ligand", 64, "bf16x3", 100, 1, 1000),
        # a mid-size site, odd counts that fill no tile
        _search("search 96 fp32 ragged", 96, "fp32", 31, 3, 333, classes=6),
        _search("search 96 fp16x2 ragged", 96, "fp16x2", 80, 7, 301),
        # the largest grid, in the default and in the fast form
        _search("search 128 fp32", 128, "fp32", 60, 1, 1000),
        _search("search 128 fp16x2", 128, "fp16x2", 60, 4, 1000, device=True),
        # a burst of requests of uneven ligand, conformer and rotation counts on one receptor
        {"name": "serve 96 fp16x2", "kind": "serve", "n": 96, "form": "fp16x2", "requests": 6,
         "most_atoms": 80, "most_rots": 2000},
        # 1,000 random conformers reduced to at most 100 diverse ones before docking
        {"name": "cluster 1000", "kind": "cluster", "confs": 1000, "atoms": 40, "centers": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["serve", "cluster"])
    if kind == "cluster":
        return {"kind": kind, "confs": _log_int(rng, 60, 1500), "atoms": rng.randint(12, 70),
                "centers": rng.randint(20, 120)}
    n = rng.choice([32, 64, 64, 96, 128])
    form = rng.choice(["fp32", "fp32", "fp16x2", "bf16x3"])
    if kind == "serve":
        return {"kind": kind, "n": n, "form": form, "requests": rng.randint(2, 8),
                "most_atoms": rng.randint(20, 80),
                "most_rots": _log_int(rng, 60, 3000 * 96 // n if n <= 96 else 1000)}
    # rotations such that no drawn case runs longer than the largest listed one
    most = {32: 40000, 64: 20000, 96: 6000, 128: 2500}[n]
    rots = _log_int(rng, 40, most)
    confs = max(1, min(rots // 8, _log_int(rng, 1, 60)))
    atoms = _log_int(rng, 8, 128 if form == "fp32" and n > 32 else 90)
    return {"kind": kind, "n": n, "form": form, "atoms": atoms, "confs": confs,
            "rots": max(1, rots // confs), "classes": rng.randint(2, 8),
            "device": rng.random() < 0.4, "graphs": rng.random() < 0.2}


def _receptor_grids(n, rng):
    """[9, n, n, n] float32: eight capped soft-core Lennard-Jones grids, one Coulomb grid.
    Evaluated on the GPU in blocks of 16^3 points with the atoms within 12 A of each."""
    atoms, edge = RECEPTORS[n]
    xyz = rng.uniform(0.0, edge, (atoms, 3)).astype(np.float32)
    origin = edge / 2 - (n - 1) * SPACING / 2
    dev = torch.device("cuda")
    x = torch.from_numpy(xyz).to(dev)
    par = np.stack([rng.uniform(1.5, 2.0, atoms), np.sqrt(rng.uniform(0.05, 0.2, atoms)),
                    332.0716 * rng.normal(0.0, 0.3, atoms)]).astype(np.float32)
    radius, root_eps, charge = torch.from_numpy(par).to(dev)
    out = torch.empty(9, n, n, n, device=dev)
    axis = origin + SPACING * torch.arange(n, device=dev)
    for bx in range(0, n, 16):
        for by in range(0, n, 16):
            for bz in range(0, n, 16):
                lo = origin + SPACING * np.array([bx, by, bz])
                near = np.all((xyz > lo - 12.0) & (xyz < lo + 7.5 + 12.0), axis=1)
                at = torch.from_numpy(np.nonzero(near)[0]).to(dev)
                a = x[at]
                d2 = ((axis[bx:bx + 16, None] - a[:, 0]).square()[:, None, None]
                      + (axis[by:by + 16, None] - a[:, 1]).square()[None, :, None]
                      + (axis[bz:bz + 16, None] - a[:, 2]).square()[None, None, :])
                se = torch.where(d2 <= 144.0, root_eps[at], 0.0)
                box = out[:, bx:bx + 16, by:by + 16, bz:bz + 16]
                for v, probe in enumerate(PROBES):
                    r2 = (radius[at] + float(probe)).square()
                    s6 = (r2 / torch.maximum(d2, 0.25 * r2)).pow(3)
                    box[v] = (se * (s6 * s6 - 2.0 * s6)).sum(-1).clamp(max=3.0)
                q = torch.where(d2 <= 144.0, charge[at], 0.0)
                box[8] = (q / (4.0 * d2.clamp(min=0.25))).sum(-1).clamp(-40.0, 40.0)
    return out.cpu().numpy()


def _quaternions(count, rng):
    q = rng.normal(size=(count, 4))
    return (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)


def _ligand(atoms, confs, rots, classes, rng):
    """Coordinates [confs, atoms, 3], charges, epsilons, radius classes 0..7, quaternions."""
    radius = 4.0 * (atoms / 24) ** (1 / 3)
    v = rng.normal(size=(atoms, 3))
    base = v / np.linalg.norm(v, axis=1, keepdims=True) * radius * rng.uniform(size=(atoms, 1)) ** (1 / 3)
    used = np.sort(rng.choice(8, classes, replace=False))
    cls = used[np.concatenate([np.arange(min(classes, atoms)),
                               rng.integers(0, classes, max(0, atoms - classes))])]
    charge = rng.normal(0.0, 0.3, atoms)
    return {"coor": (base + rng.uniform(-0.5, 0.5, (confs, atoms, 3))).astype(np.float32),
            "charge": (charge - charge.mean()).astype(np.float32),
            "eps": rng.uniform(0.02, 0.2, atoms).astype(np.float32),
            "cls": cls, "quats": _quaternions(confs * rots, rng).reshape(confs, rots, 4)}


def _search_inputs(case, seed):
    rng = np.random.default_rng([seed, 1])
    grids = _receptor_grids(case["n"], rng)
    lig = _ligand(case["atoms"], case["confs"], case["rots"], case["classes"], rng)
    used = np.unique(lig["cls"])  # only the grids that the ligand's atoms use, then elec
    lig["slot"] = np.searchsorted(used, lig["cls"]).astype(np.int32)
    return np.ascontiguousarray(np.concatenate([grids[used], grids[8:]])), lig


def _serve_inputs(case, seed):
    rng = np.random.default_rng([seed, 2])
    grids = _receptor_grids(case["n"], rng)
    size = np.random.default_rng(7)  # the requests' sizes belong to the case
    requests = []
    for _ in range(case["requests"]):
        rots = int(size.integers(max(1, case["most_rots"] // 10), case["most_rots"] + 1))
        confs = int(size.integers(1, min(60, rots) + 1))
        atoms = int(size.integers(10, case["most_atoms"] + 1))
        lig = _ligand(atoms, confs, max(1, rots // confs), 8, rng)
        lig["slot"] = lig["cls"].astype(np.int32)
        requests.append(lig)
    return grids, requests


def _conformers(case, seed):
    """Random-rotor conformers of a chain of 1.5 A bonds, each randomly placed; energies."""
    rng = np.random.default_rng([seed, 3])
    confs, atoms = case["confs"], case["atoms"]
    step = rng.normal(size=(atoms, 3))
    step = 1.5 * step / np.linalg.norm(step, axis=1, keepdims=True) + np.array([0.8, 0.0, 0.0])
    x = np.repeat(np.cumsum(step, 0)[None], confs, 0)
    for r in np.sort(rng.choice(np.arange(1, atoms - 2), min(6, atoms - 3), replace=False)):
        ax = x[:, r + 1] - x[:, r]
        ax = (ax / np.linalg.norm(ax, axis=1, keepdims=True))[:, None]
        t = rng.uniform(-np.pi, np.pi, confs)[:, None, None]
        p = x[:, r + 1:] - x[:, r + 1:r + 2]
        x[:, r + 1:] = (x[:, r + 1:r + 2] + p * np.cos(t) + np.cross(ax, p) * np.sin(t)
                        + ax * (p * ax).sum(-1, keepdims=True) * (1 - np.cos(t)))
    energy = 5.0 * np.sqrt(((x - x.mean(1, keepdims=True)) ** 2).sum(-1).mean(1)) + rng.normal(size=confs)
    rot = _rotation_matrices(torch.from_numpy(_quaternions(confs, rng).astype(np.float64))).numpy()
    return x @ rot.transpose(0, 2, 1) + rng.uniform(-10, 10, (confs, 1, 3)), energy


class _Service:
    """A server and its receptor, closed in that order."""

    def __init__(self, grids, form, requests):
        self.requests = requests
        self.receptor = Receptor(grids, SPACING, form=form)
        self.server = Server(self.receptor, arena_bytes=1 << 28, max_box=32, max_atoms=96,
                             wave_rotations=512)

    def __del__(self):
        self.server.close()
        self.receptor.close()


def prepare(case, seed):
    if case["kind"] == "cluster":
        coords, energies = _conformers(case, seed)
        return {"coords": coords, "energies": energies, "centers": case["centers"]}
    if case["kind"] == "serve":
        grids, requests = _serve_inputs(case, seed)
        return _Service(grids, FORMS[case["form"]], requests)
    grids, lig = _search_inputs(case, seed)
    s = {"lig": lig, "receptor": Receptor(grids, SPACING, form=FORMS[case["form"]],
                                          use_graphs=int(case["graphs"]))}
    if case["device"]:
        count = case["confs"] * case["rots"]
        s["dev"] = [torch.from_numpy(lig[k]).cuda() for k in ("coor", "charge", "eps", "slot", "quats")]
        s["out"] = [torch.empty(count, dtype=torch.float32, device="cuda"),
                    torch.empty(count, 3, dtype=torch.int32, device="cuda")]
    return s


def run(state):
    if isinstance(state, _Service):
        tickets = [state.server.submit(r["coor"], r["charge"], r["eps"], r["slot"], r["quats"])
                   for r in state.requests]
        done = [state.server.poll(t) for t in tickets]
        return [{"minE": e, "idx": i} for e, i, _ in done]
    if "coords" in state:
        centers = np.full(state["centers"], -1, np.int32)  # as many as asked for, or fewer
        got = cluster_conformers(state["coords"], state["energies"], 1.5, state["centers"])
        centers[:len(got)] = got
        return centers
    lig = state["lig"]
    if "dev" in state:
        coor, charge, eps, slot, quats = (t.data_ptr() for t in state["dev"])
        min_e, idx = state["out"]
        confs, atoms, _ = lig["coor"].shape
        state["receptor"].search_device(atoms, confs, coor, charge, eps, slot, lig["quats"].shape[1],
                                        quats, min_e.data_ptr(), idx.data_ptr())
    else:
        min_e, idx = state["receptor"].search(lig["coor"], lig["charge"], lig["eps"], lig["slot"],
                                              lig["quats"])
    return {"minE": min_e, "idx": idx}


def _work_search(n, k, atoms, confs, rots):
    points = n ** 3
    # per rotation: k forward and one inverse real FFT, the conjugate products and their sum
    flops = confs * rots * ((k + 1) * 2.5 * points * math.log2(points) + k * 4.0 * points)
    return 4.0 * k * points + confs * atoms * 12.0 + atoms * 12.0 + confs * rots * 32.0, flops


def work(case):
    if case["kind"] == "cluster":
        c, a = case["confs"], case["atoms"]
        return {"bytes": c * a * 24.0 + c * 8.0, "flops": c * (c - 1) / 2 * (18.0 * a + 300.0)}
    if case["kind"] == "serve":
        size = np.random.default_rng(7)
        total = [4.0 * 9 * case["n"] ** 3, 0.0]
        for _ in range(case["requests"]):
            rots = int(size.integers(max(1, case["most_rots"] // 10), case["most_rots"] + 1))
            confs = int(size.integers(1, min(60, rots) + 1))
            atoms = int(size.integers(10, case["most_atoms"] + 1))
            b, f = _work_search(case["n"], 9, atoms, confs, max(1, rots // confs))
            total = [total[0] + b - 4.0 * 9 * case["n"] ** 3, total[1] + f]
        return {"bytes": total[0], "flops": total[1]}
    k = min(case["classes"], case["atoms"]) + 1
    b, f = _work_search(case["n"], k, case["atoms"], case["confs"], case["rots"])
    return {"bytes": b, "flops": f}


def _rotation_matrices(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([
        w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y),
        2 * (x * y + w * z), w * w - x * x + y * y - z * z, 2 * (y * z - w * x),
        2 * (x * z - w * y), 2 * (y * z + w * x), w * w - x * x - y * y + z * z,
    ], -1).reshape(*q.shape[:-1], 3, 3)


def _exact_minima(grids, lig):
    """Minimum correlation energy of every rotation in 64 bits: trilinear spread of the rotated
    atoms, FFT correlation with the receptor grids, minimum over the translation window."""
    dev = torch.device("cuda")
    k, n = grids.shape[:2]
    spectra = torch.fft.rfftn(torch.from_numpy(grids).to(dev, torch.float64), dim=(1, 2, 3))
    coor = torch.from_numpy(lig["coor"]).to(dev, torch.float64)
    quats = torch.from_numpy(lig["quats"]).to(dev, torch.float64)
    slot = torch.from_numpy(lig["slot"].astype(np.int64)).to(dev)
    weight = torch.from_numpy(lig["eps"]).to(dev, torch.float64).sqrt()
    charge = torch.from_numpy(lig["charge"]).to(dev, torch.float64)
    count = quats.shape[0] * quats.shape[1]
    rots = quats.reshape(-1, 4)
    conf = torch.arange(count, device=dev) // quats.shape[1]
    best = torch.empty(count, dtype=torch.float64, device=dev)
    chunk = max(1, 2 ** 27 // (k * n ** 3))
    axis = torch.arange(n, device=dev)
    for lo in range(0, count, chunk):
        hi = min(count, lo + chunk)
        b = hi - lo
        x = torch.einsum("bij,baj->bai", _rotation_matrices(rots[lo:hi]), coor[conf[lo:hi]])
        x = x - x.amin(1, keepdim=True)
        cell = (x / SPACING).long()
        frac = x / SPACING - cell
        window = n - (x.amax(1) / SPACING).long() - 2
        fill = torch.zeros(b * k * n ** 3, dtype=torch.float64, device=dev)
        row = torch.arange(b, device=dev)[:, None] * k
        for corner in range(8):
            d = torch.tensor([corner >> 2, corner >> 1 & 1, corner & 1], device=dev)
            w = torch.where(d == 1, frac, 1 - frac).prod(-1)
            c = cell + d
            at = (c[..., 0] * n + c[..., 1]) * n + c[..., 2]
            fill.index_add_(0, ((row + slot) * n ** 3 + at).reshape(-1), (w * weight).reshape(-1))
            fill.index_add_(0, ((row + k - 1) * n ** 3 + at).reshape(-1), (w * charge).reshape(-1))
        f = torch.fft.rfftn(fill.reshape(b, k, n, n, n), dim=(2, 3, 4))
        e = torch.fft.irfftn((f.conj() * spectra).sum(1), s=(n, n, n), dim=(1, 2, 3))
        inside = ((axis < window[:, 0, None])[:, :, None, None] & (axis < window[:, 1, None])[:, None, :, None]
                  & (axis < window[:, 2, None])[:, None, None, :])
        best[lo:hi] = torch.where(inside, e, math.inf).reshape(b, -1).amin(1)
    return best


def exact(case, seed):
    if case["kind"] == "cluster":
        return None  # indices only
    if case["kind"] == "serve":
        grids, requests = _serve_inputs(case, seed)
        return [{"minE": _exact_minima(grids, r), "idx": None} for r in requests]
    return {"minE": _exact_minima(*_search_inputs(case, seed)), "idx": None}
