"""The evaluations, MD steps and training steps that users of this engine run, as measured cases.

Potentials are the ones under tests/golden/potentials (levels 16 to 28); structures are thermally
displaced crystals with vacancies (so atom counts are odd and rows ragged) and synthetic training
configurations.  Rows are built here with torch, so a case's inputs depend on its seed alone.

Results of mixed-precision handles carry FP32's 24 bits in FP64 arrays; such a case returns them as FP32.
"""

import ctypes
import math
import os
import re
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "jax-mtp_b200"))

from mtp_b200 import _lib, synth  # noqa: E402
from mtp_b200.engine import MTPEngine, pinned_empty  # noqa: E402
from mtp_b200.md import DeviceMD  # noqa: E402
from mtp_b200.train import DeviceBatch, predict, weighted_loss  # noqa: E402

DEV = "cuda"
POTENTIALS = {"L16S1": "cfg0_L16_S1", "L16": "cfg1md_L16_S2", "L20": "cfg3_L20_S2", "L24": "cfg2md_L24_S3",
              "L28": "cfg4_L28_S4"}
LATTICES = {"fcc": (3.6, [[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]), "bcc": (2.87, [[0, 0, 0], [.5, .5, .5]])}
SKIN = 0.3


def listed():
    return [
        # one call of a calculator on a small cell from host arrays (relaxation, phonons): latency only
        {"name": "calculator_16_l16_fp64", "kind": "calculator", "pot": "L16", "precision": "fp64", "lattice": "bcc",
         "nx": 2, "ny": 2, "nz": 2, "vacancies": 0.0, "stride": 64},
        # the LAMMPS pair style's force call at the size of the reference's MD input: positions and list in pinned
        # host buffers that stay the same from step to step
        {"name": "pair_2000_l16_fp64", "kind": "pair", "pot": "L16", "precision": "fp64", "lattice": "bcc",
         "nx": 10, "ny": 10, "nz": 10, "vacancies": 0.0, "stride": 64},
        # a 256-atom single-species cell whose rows are on the GPU already
        {"name": "device_256_l16_fp64", "kind": "device", "pot": "L16S1", "precision": "fp64", "lattice": "fcc",
         "nx": 4, "ny": 4, "nz": 4, "vacancies": 0.0, "stride": 64},
        # a mid-size system with vacancies, per-atom virials asked for (stress maps)
        {"name": "device_10k_l20_mixed_vatom", "kind": "device", "pot": "L20", "precision": "mixed", "lattice": "bcc",
         "nx": 17, "ny": 17, "nz": 18, "vacancies": 0.04, "stride": 61, "vatom": True},
        # drop-in FP64 forces of a production-size cell at the headline level
        {"name": "device_31k_l24_fp64", "kind": "device", "pot": "L24", "precision": "fp64", "lattice": "fcc",
         "nx": 20, "ny": 20, "nz": 20, "vacancies": 0.03, "stride": 64},
        # an FP64 evaluation from a host program's packed rows in pinned memory, copies included
        {"name": "rows_108k_l16_fp64", "kind": "rows", "pot": "L16", "precision": "fp64", "lattice": "bcc",
         "nx": 38, "ny": 38, "nz": 38, "vacancies": 0.02, "stride": 60},
        # ten steps of device-resident NVE MD with one list rebuild, replayed graphs
        {"name": "md_131k_l24_mixed", "kind": "md", "pot": "L24", "precision": "mixed", "lattice": "fcc",
         "nx": 32, "ny": 32, "nz": 32, "vacancies": 0.0, "stride": 64, "steps": 10},
        # the headline size: forces of one MD step of a million atoms, mixed precision
        {"name": "device_1m_l24_mixed", "kind": "device", "pot": "L24", "precision": "mixed", "lattice": "fcc",
         "nx": 64, "ny": 64, "nz": 64, "vacancies": 0.0, "stride": 64},
        # the highest level, FP64, as a validation run evaluates it
        {"name": "device_4k_l28_fp64", "kind": "device", "pot": "L28", "precision": "fp64", "lattice": "fcc",
         "nx": 10, "ny": 10, "nz": 10, "vacancies": 0.02, "stride": 80},
        # batched forward of a whole training set (least-squares columns, validation errors)
        {"name": "batch_512_l20_mixed", "kind": "batch", "pot": "L20", "precision": "mixed", "configs": 512,
         "nmin": 16, "nmax": 256},
        # one training step (forward, loss, coefficient gradients) on a mini-batch
        {"name": "train_32_l20", "kind": "train", "pot": "L20", "precision": "fp64", "configs": 32, "nmin": 16,
         "nmax": 256},
        # one training step at the highest level
        {"name": "train_64_l28", "kind": "train", "pot": "L28", "precision": "fp64", "configs": 64, "nmin": 32,
         "nmax": 512},
    ]


def draw(rng):
    lo = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["calculator", "pair", "device", "device", "device", "rows", "md", "batch", "train"])
    if kind in ("batch", "train"):
        pot = rng.choice(["L16", "L20"] if kind == "batch" else ["L16", "L20", "L28"])
        nmin = lo(8, 64)
        return {"kind": kind, "pot": pot, "precision": rng.choice(["fp64", "mixed"]) if kind == "batch" else "fp64",
                "configs": lo(3, 24 if pot == "L28" else 96 if kind == "train" else 256), "nmin": nmin,
                "nmax": nmin + lo(8, 200)}
    pot = {"calculator": ["L16", "L20"], "pair": ["L16", "L20", "L24"]}.get(kind, ["L16", "L20", "L24", "L24"])
    if kind == "device":
        pot = pot + ["L28"]
    case = {"kind": kind, "pot": rng.choice(pot), "precision": rng.choice(["fp64", "mixed"])}
    if kind in ("calculator", "pair") and case["pot"] == "L20":
        case["precision"] = "fp64"          # its random coefficients cancel to a total that FP32 does not resolve
    case["lattice"] = "fcc" if case["pot"] in ("L24", "L28") else rng.choice(["fcc", "bcc"])
    small, large = {"calculator": (2, 4), "pair": (4, 13), "rows": (21, 34), "md": (8, 24), "device": (4, 44)}[kind]
    if case["pot"] == "L28":
        large = 12
    n = lo(small, large)
    for axis in ("nx", "ny", "nz"):
        case[axis] = max(small, min(large, n + rng.randint(-2, 2)))
    case["vacancies"] = 0.0 if kind in ("pair", "calculator") else round(rng.choice([0.0, rng.uniform(0.005, 0.08)]), 4)
    case["stride"] = rng.randint(79, 96) if case["pot"] == "L28" else rng.choice([64, 64, rng.randint(61, 80)])
    if kind == "device" and rng.random() < 0.3:
        case["vatom"] = True
    if kind == "md":
        case["steps"] = rng.randint(1, 10)
    return case


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _path(case):
    return os.path.join(ROOT, "tests", "golden", "potentials", POTENTIALS[case["pot"]] + ".mtp")


_tables = {}


def _potential(case):
    """The .mtp file's tables as numpy arrays."""
    if case["pot"] not in _tables:
        with open(_path(case)) as f:
            text = f.read()
        get = lambda k: re.search(r"^\s*%s = (.*)$" % k, text, re.M).group(1)  # noqa: E731
        nums = lambda s, t: np.array([t(x) for x in re.findall(r"[-+\d.eE]+", s)])  # noqa: E731
        S, R, K = (int(get(k)) for k in ("species_count", "radial_funcs_count", "radial_basis_size"))
        radial = text[text.index("radial_coeffs"):text.index("alpha_moments_count")]
        rows = np.array([nums(r, float) for r in re.findall(r"\{([^}]*)\}", radial)])
        _tables[case["pot"]] = {
            "S": S, "R": R, "K": K, "M": int(get("alpha_moments_count")), "scaling": float(get("scaling")),
            "rmin": float(get("min_dist")), "rmax": float(get("max_dist")), "radial": rows.reshape(S, S, R, K),
            "basic": nums(get("alpha_index_basic"), int).reshape(-1, 4),
            "times": nums(get("alpha_index_times"), int).reshape(-1, 4),
            "map": nums(get("alpha_moment_mapping"), int), "species": nums(get("species_coeffs"), float),
            "moment": nums(get("moment_coeffs"), float)}
    return _tables[case["pot"]]


def _crystal(case, seed):
    """Displaced crystal with vacancies: positions, cell edges, species, and the site grid that rows are built from."""
    p = _potential(case)
    a, basis = LATTICES[case["lattice"]]
    if case["pot"] == "L16S1":
        a = 4.05
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = [case["nx"], case["ny"], case["nz"]]
    cells = torch.cartesian_prod(*[torch.arange(k, device=DEV) for k in n])
    b = torch.tensor(basis, dtype=torch.float64, device=DEV)
    ideal = (cells.double()[:, None] + b[None]).reshape(-1, 3) * a
    x = ideal + 0.06 * torch.randn(ideal.shape, generator=g, device=DEV, dtype=torch.float64)
    types = torch.randint(0, p["S"], (len(x),), generator=g, device=DEV, dtype=torch.int32)
    there = torch.ones(len(x), dtype=torch.bool, device=DEV)
    there[torch.randperm(len(x), generator=g, device=DEV)[:_vacant(case)]] = False
    return x, types, there, cells, b, a, n


def _sites(case):
    return case["nx"] * case["ny"] * case["nz"] * len(LATTICES[case["lattice"]][1])


def _vacant(case):
    return int(_sites(case) * case["vacancies"])


def _rows(case, seed, cutoff):
    """Rows of all periodic images closer than `cutoff`, from the lattice's own neighbour sites."""
    x, types, there, cells, b, a, n = _crystal(case, seed)
    nb, stride = len(b), case["stride"]
    size = torch.tensor(n, device=DEV)
    new = torch.cumsum(there.int(), 0, dtype=torch.int32) - 1
    N = int(there.sum())
    js = torch.full((N, stride), -1, dtype=torch.int32, device=DEV)
    jt, r = torch.full_like(js, -1), torch.zeros((N, stride, 3), dtype=torch.float64, device=DEV)
    counts = torch.zeros(N, dtype=torch.int32, device=DEV)
    reach = range(-int(math.ceil((cutoff + 1) / a)) - 1, int(math.ceil((cutoff + 1) / a)) + 2)
    grid = [(i, j, k) for i in reach for j in reach for k in reach]
    for bi in range(nb):
        mine = torch.arange(len(cells), device=DEV) * nb + bi
        mine, from_cell = mine[there[mine]], cells[there[mine]]
        me = new[mine].long()
        for c in grid:
            for bj in range(nb):
                d = _shift(c, bi, bj, case["lattice"], a)
                if not 0 < sum(v * v for v in d) < (cutoff + 0.75) ** 2:
                    continue
                to = (from_cell + torch.tensor(c, device=DEV)) % size
                j = ((to[:, 0] * n[1] + to[:, 1]) * n[2] + to[:, 2]) * nb + bj
                home = from_cell + torch.tensor(c, device=DEV) - to
                vec = x[j] - x[mine] + home.double() * a
                keep = there[j] & ((vec * vec).sum(1) < cutoff * cutoff) & (counts[me] < stride)
                i, jj, slot = me[keep], j[keep], counts[me[keep]].long()
                js[i, slot], jt[i, slot], r[i, slot] = new[jj], types[jj], vec[keep]
                counts[i] += 1
    return types[there].contiguous(), r, js, jt, counts


def _shift(c, bi, bj, lattice, a):
    basis = LATTICES[lattice][1]
    return [(c[k] + basis[bj][k] - basis[bi][k]) * a for k in range(3)]


def _pair_inputs(case, seed, cutoff):
    """Local and ghost positions, owners and full lists, as an MD code hands them to a pair style."""
    x, types, _, _, _, a, n = _crystal(case, seed)
    edges = torch.tensor(n, device=DEV, dtype=torch.float64) * a
    x = x % edges
    xs, own = [x], [torch.arange(len(x), device=DEV)]
    m = [int(math.ceil(cutoff / float(e))) for e in edges]
    for i in range(-m[0], m[0] + 1):
        for j in range(-m[1], m[1] + 1):
            for k in range(-m[2], m[2] + 1):
                if i or j or k:
                    y = x + torch.tensor([i, j, k], device=DEV, dtype=torch.float64) * edges
                    keep = ((y > -cutoff) & (y < edges + cutoff)).all(1)
                    xs.append(y[keep])
                    own.append(own[0][keep])
    xs, own = torch.cat(xs), torch.cat(own)
    near = torch.cdist(x, xs, compute_mode="donot_use_mm_for_euclid_dist") < cutoff
    near[torch.arange(len(x)), torch.arange(len(x))] = False
    num = near.sum(1)
    width = int(num.max())
    neigh = torch.argsort(~near, dim=1, stable=True)[:, :width].int()
    return xs, types[own], own.int(), neigh, num.int()


_engines = {}


def _engine(case, natoms, nbr):
    """A program's handle for one potential: made once and kept for all of its inputs (the last few are held)."""
    key = (case["pot"], case["precision"], natoms, nbr)
    if key not in _engines:
        while len(_engines) >= 2:
            _engines.pop(next(iter(_engines))).close()
        _engines[key] = MTPEngine(_path(case), natoms, nbr, precision=case["precision"])
    return _engines[key]


def _configs(case, seed):
    """Training configurations and targets on the GPU, rows with every periodic image inside the cutoff."""
    p = _potential(case)
    # sizes belong to the case, structures to the seed
    sizes = np.random.default_rng(case["configs"]).integers(case["nmin"], case["nmax"] + 1, case["configs"])
    structs = [synth.training_batch(1, int(n), int(n), p["S"], seed=[seed, k], a_range=(3.4, 4.2), sigma=0.05)[0]
               for k, n in enumerate(sizes)]
    rows, first = [], 0
    for s in structs:
        x = torch.tensor(s.positions, device=DEV)
        cell = torch.tensor(s.cell, device=DEV)
        t = torch.tensor(s.types, dtype=torch.int32, device=DEV)
        n = [int(math.ceil(p["rmax"] * np.linalg.norm(np.cross(s.cell[(k + 1) % 3], s.cell[(k + 2) % 3])) / s.volume)) + 1
             for k in range(3)]
        im = torch.cartesian_prod(*[torch.arange(-k, k + 1, device=DEV) for k in n]).double() @ cell
        d = x[None, None] + im[None, :, None] - x[:, None, None]
        d2 = (d * d).sum(-1)
        i, _, j = keep = torch.nonzero((d2 < p["rmax"] ** 2) & (d2 > 1e-12), as_tuple=True)
        num = torch.bincount(i, minlength=len(x))
        slot = torch.arange(len(i), device=DEV) - (torch.cumsum(num, 0) - num)[i]
        rows.append((i + first, slot, j + first, t[j], d[keep], num, t))
        first += len(x)
    N, width = first, max(int(r[5].max()) for r in rows)
    i, slot, j, tj, d, num, types = (torch.cat([r[k] for r in rows]) for k in range(7))
    js = torch.full((N, width), -1, dtype=torch.int32, device=DEV)
    jt, r = torch.full_like(js, -1), torch.zeros((N, width, 3), dtype=torch.float64, device=DEV)
    js[i, slot], jt[i, slot], r[i, slot] = j.int(), tj, d
    cfg = torch.cat([torch.full((len(q[6]),), k, dtype=torch.int32, device=DEV) for k, q in enumerate(rows)])
    vol = torch.tensor([s.volume for s in structs], device=DEV, dtype=torch.float64)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *k: torch.randn(*k, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    C = len(structs)
    natoms = torch.bincount(cfg, minlength=C).double()
    targets = (-3 * natoms + rand(C), rand(N, 3), 0.01 * rand(C, 6))
    return DeviceBatch(types, r, js, jt, num.int(), cfg, vol, C), targets


def _coefficients(case, seed):
    """Coefficients part-way through a fit: the file's, moved a little."""
    p = _potential(case)
    g = np.random.default_rng(seed)
    return {k: torch.tensor(p[n] * (1 + 0.05 * g.normal(size=p[n].shape)), device=DEV, dtype=torch.float64)
            for k, n in (("species", "species"), ("basis", "moment"), ("radial", "radial"))}


def prepare(case, seed):
    kind, p = case["kind"], _potential(case)
    if kind in ("batch", "train"):
        batch, targets = _configs(case, seed)
        s = {"case": case, "batch": batch, "targets": targets}
        # the handle of a training program holds its largest batch
        cap = case["configs"] * case["nmax"]
        s["engine"] = _engine(case, cap, 128)
        if kind == "train":
            s["params"] = {k: v.requires_grad_() for k, v in _coefficients(case, seed).items()}
        return s
    if kind == "md":
        x, types, there, _, _, a, n = _crystal(case, seed)
        st = synth.Structure(x[there].cpu().numpy(), np.diag(np.array(n) * a), types[there].cpu().numpy())
        eng = MTPEngine(_path(case), st.natoms, case["stride"], precision=case["precision"])
        md = DeviceMD(eng, st, [55.845] * p["S"], synth.maxwell_boltzmann(st.natoms, 600.0, 55.845, seed), skin=SKIN,
                      stride=case["stride"], rebuild_every=min(10, case["steps"]))
        md.capture()
        return {"case": case, "md": md, "engine": eng}
    if kind == "pair":
        x, sp, own, neigh, num = (t.cpu().numpy() for t in _pair_inputs(case, seed, p["rmax"] + SKIN))
        eng = MTPEngine(_path(case), len(num), case["stride"], cutoff=p["rmax"], precision=case["precision"])
        s = {"case": case, "engine": eng}
        for k, v in (("x", x), ("species", sp), ("owner", own), ("neigh", neigh), ("num", num)):
            s[k] = pinned_empty(v.shape, v.dtype)
            s[k][...] = v
        for k, shape in (("energy", 1), ("forces", (len(num), 3)), ("virial", 6)):
            s[k] = pinned_empty(shape)
        return s
    it, r, js, jt, counts = _rows(case, seed, p["rmax"] + SKIN)
    s = {"case": case, "rows": (it, r, js, jt, counts)}
    if kind == "calculator":
        s["rows"] = tuple(t.cpu().numpy() for t in s["rows"])
        s["engine"] = _engine(case, _sites(case), case["stride"])
    elif kind == "rows":
        s["engine"] = _engine(case, _sites(case), case["stride"])
        s["rows"] = []
        for t in (it, r, js, jt, counts):
            s["rows"].append(pinned_empty(tuple(t.shape), np.float64 if t.is_floating_point() else np.int32))
            torch.from_numpy(s["rows"][-1]).copy_(t)
        for k, shape in (("energy", 1), ("forces", (len(it), 3)), ("virial", 6)):
            s[k] = pinned_empty(shape)
    else:
        s["engine"] = _engine(case, _sites(case), case["stride"])
        s["eatom"] = torch.empty(len(it), dtype=torch.float64, device=DEV)
        s["vatom"] = torch.empty((len(it), 6), dtype=torch.float64, device=DEV) if case.get("vatom") else None
    return s


# ---------------------------------------------------------------------------------------------------------------------
# the passes
# ---------------------------------------------------------------------------------------------------------------------
def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def run(s):
    case, eng = s["case"], s.get("engine")
    kind = case["kind"]
    out = _run(s, case, eng, kind)
    if case["precision"] == "mixed":
        f32 = lambda v: None if v is None else v.float() if torch.is_tensor(v) else np.float32(v)  # noqa: E731
        out = {k: f32(v) for k, v in out.items()}
    return out


def _run(s, case, eng, kind):
    if kind == "calculator":
        return eng.compute(*s["rows"])
    if kind in ("pair", "rows"):
        flags = _lib.EFLAG | _lib.VFLAG
        tail = (flags, _ptr(s["energy"]), _ptr(s["forces"]), _ptr(s["virial"]), None, None)
        if kind == "pair":
            code = _lib.lib().mtp_compute_positions(
                eng.handle, len(s["num"]), len(s["x"]), _ptr(s["x"]), _ptr(s["species"]), _ptr(s["owner"]),
                s["neigh"].shape[1], _ptr(s["neigh"]), _ptr(s["num"]), *tail)
        else:
            it, r, js, jt, counts = s["rows"]
            code = _lib.lib().mtp_compute(eng.handle, len(it), r.shape[1], _ptr(it), _ptr(r), _ptr(js), _ptr(jt),
                                          _ptr(counts), *tail)
        _lib.check(code, eng.handle)
        return {"energy": s["energy"], "forces": s["forces"], "virial": s["virial"]}
    if kind == "device":
        energy, forces, virial = eng.compute_device(*s["rows"], eatom=s["eatom"], vatom=s["vatom"])
        return {"energy": energy, "forces": forces, "virial": virial, "eatom": s["eatom"], "vatom": s["vatom"]}
    if kind == "md":
        md = s["md"]
        md.run(case["steps"], graphs=True)
        return {"x": md.x, "v": md.v, "forces": md.f, "energy": md.energy, "virial": md.virial}
    b = s["batch"]
    if kind == "batch":
        energy, forces, stress = eng.batch_device(b.itypes, b.rijs, b.js, b.jtypes, b.counts, b.cfg, b.volumes, b.nconfig)
        return {"energy": energy, "forces": forces, "stress": stress}
    for v in s["params"].values():
        v.grad = None
    energy, forces, stress = predict(s["params"], eng, b)
    loss = weighted_loss(energy, forces, stress, s["targets"])
    loss.backward()
    return {"loss": loss.detach(), "energy": energy.detach(), "forces": forces.detach(), "stress": stress.detach(),
            **{"grad_" + k: v.grad for k, v in s["params"].items()}}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    p = _potential(case)
    if case["kind"] in ("batch", "train"):
        # mean size; mean density of the three lattices over the range of lattice constants
        N = case["configs"] * (case["nmin"] + case["nmax"]) / 2
        near = 4 / 3 * math.pi * p["rmax"] ** 3 * 0.055
        listed_ = near
    else:
        N = _sites(case) - _vacant(case)
        shells = [math.dist((0, 0, 0), _shift((i, j, k), 0, b, case["lattice"], LATTICES[case["lattice"]][0]))
                  for i in range(-3, 4) for j in range(-3, 4) for k in range(-3, 4)
                  for b in range(len(LATTICES[case["lattice"]][1]))]
        near, listed_ = (sum(0 < d < c for d in shells) * (1 - case["vacancies"]) for c in (p["rmax"], p["rmax"] + SKIN))
    B, P = len(p["basic"]), len({tuple(r[1:]) for r in p["basic"].tolist()})
    # radial functions and powers, basic moments and their reverse, products forward and reverse, the energy sum
    flops = near * (10 * B + 6 * p["R"] * p["K"] + 6 * p["K"] + 2 * P + 75) + 9 * len(p["times"]) + 2 * len(p["map"])
    row = {"pair": 4}.get(case["kind"], 32)     # list entry, or r_ij, owner and species
    read, written = listed_ * row + 8, 32 + 8 + (48 if case.get("vatom") else 0)
    steps = 1
    if case["kind"] == "md":
        steps, read, written = case["steps"], 52 + listed_ * 12, 48
    if case["kind"] == "train":
        flops *= 4                               # forward, then the dual-number reverse of it
    return {"bytes": N * steps * (read + written), "flops": N * steps * flops}


# ---------------------------------------------------------------------------------------------------------------------
# the same values in 64 bits from plain torch
# ---------------------------------------------------------------------------------------------------------------------
def _tensors(p):
    t = lambda a: torch.tensor(a, device=DEV)  # noqa: E731
    depth = np.zeros(p["M"], dtype=int)
    for a, b, _, c in p["times"]:
        depth[c] = max(depth[c], depth[a] + 1, depth[b] + 1)
    d = depth[p["times"][:, 3]]
    monos, of = np.unique(p["basic"][:, 1:], axis=0, return_inverse=True)
    return {"levels": [t(p["times"][d == k]) for k in range(1, depth.max() + 1)], "monos": t(monos),
            "of": t(of.reshape(-1)), "mu": t(p["basic"][:, 0]), "map": t(p["map"])}


def _site_energies(p, q, coef, it, r, jt, mask):
    """E_i of a few atoms' rows; differentiable in r and in the coefficients."""
    d = r.square().sum(-1).sqrt()
    x = (2 * d - (p["rmin"] + p["rmax"])) / (p["rmax"] - p["rmin"])
    cheb = [torch.ones_like(x), x]
    for _ in range(p["K"] - 2):
        cheb.append(2 * x * cheb[-1] - cheb[-2])
    phi = p["scaling"] * (p["rmax"] - d).square().unsqueeze(-1) * torch.stack(cheb, -1)
    phi = phi * mask.unsqueeze(-1)
    f = torch.einsum("nsrk,nsk->nsr", coef["radial"][it.long()[:, None], jt.clamp_min(0).long()], phi)
    u = r / d.unsqueeze(-1)
    power = [torch.ones_like(u)]
    for _ in range(int(q["monos"].max())):
        power.append(power[-1] * u)
    power = torch.stack(power, -1)                                    # [n, s, 3, e]
    mono = power[:, :, 0, q["monos"][:, 0]] * power[:, :, 1, q["monos"][:, 1]] * power[:, :, 2, q["monos"][:, 2]]
    basic = torch.einsum("nsr,nsp->rpn", f, mono)[q["mu"], q["of"]]   # [B, n]
    m = torch.zeros((p["M"], len(it)), dtype=torch.float64, device=DEV)
    m = m.index_copy(0, torch.arange(len(basic), device=DEV), basic)
    for lev in q["levels"]:
        m = m.index_add(0, lev[:, 3], m[lev[:, 0]] * m[lev[:, 1]] * lev[:, 2:3])
    return coef["species"][it.long()] + coef["basis"] @ m[q["map"]]


def _chunks(p, it, r, jt, counts):
    n = len(it)
    size = max(16, min(n, int(1.5e8 / (len(p["times"]) + 40 * r.shape[1]))))
    for lo in range(0, n, size):
        s = slice(lo, min(n, lo + size))
        mask = (jt[s] >= 0) & (torch.arange(r.shape[1], device=DEV)[None] < counts[s, None])
        rr = torch.where(mask.unsqueeze(-1), r[s], torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64, device=DEV))
        mask = mask & (rr.square().sum(-1) < p["rmax"] ** 2)
        yield s, it[s], rr, jt[s], mask


def _forces(js, G, N):
    """F_k = own gradients - gradients of the slots that point at k."""
    there = (js >= 0) & (js < N)
    return G.sum(1).index_add(0, js[there].long(), -G[there])


def _sym(r, g):
    w = torch.einsum("...a,...b->...ab", r, g)
    w = 0.5 * (w + w.transpose(-1, -2))
    return torch.stack([w[..., 0, 0], w[..., 1, 1], w[..., 2, 2], w[..., 0, 1], w[..., 0, 2], w[..., 1, 2]], -1)


def _evaluate(p, coef, it, r, js, jt, counts):
    q = _tensors(p)
    E, G = torch.empty(len(it), dtype=torch.float64, device=DEV), torch.empty_like(r)
    for s, i, rr, t, mask in _chunks(p, it, r, jt, counts):
        rr.requires_grad_()
        e = _site_energies(p, q, coef, i, rr, t, mask)
        G[s] = torch.autograd.grad(e.sum(), rr)[0] * mask.unsqueeze(-1)
        E[s] = e.detach()
    return E, G


def _file_coefficients(p):
    t = lambda a: torch.tensor(a, device=DEV, dtype=torch.float64)  # noqa: E731
    return {"species": t(p["species"]), "basis": t(p["moment"]), "radial": t(p["radial"])}


def exact(case, seed):
    kind, p = case["kind"], _potential(case)
    if kind == "md":
        return None
    if kind in ("batch", "train"):
        b, targets = _configs(case, seed)
        it, r, js, jt, counts = b.itypes, b.rijs, b.js, b.jtypes, b.counts
        coef = _file_coefficients(p) if kind == "batch" else _coefficients(case, seed)
    elif kind == "pair":
        x, sp, own, neigh, num = _pair_inputs(case, seed, p["rmax"] + SKIN)
        it, counts, j = sp[:len(num)], num, neigh.long()
        r, js, jt, coef = x[j] - x[:len(num), None], own[j], sp[j], _file_coefficients(p)
    else:
        it, r, js, jt, counts = _rows(case, seed, p["rmax"] + SKIN)
        coef = _file_coefficients(p)
    E, G = _evaluate(p, coef, it, r, js, jt, counts)
    F = _forces(js, G, len(it))
    if kind not in ("batch", "train"):
        w = -_sym(r, G)
        out = {"energy": E.sum() if kind == "calculator" else E.sum().reshape(1), "forces": F, "virial": w.sum((0, 1))}
        if kind == "calculator":
            return {**out, "energy": float(out["energy"]), "site_energies": E}
        if kind == "device":
            out["eatom"] = E
            if case.get("vatom"):
                there = (js >= 0) & (js < len(it)) & (jt >= 0)
                out["vatom"] = 0.5 * (w.sum(1) + torch.zeros_like(w[:, 0]).index_add(0, js[there].long(), w[there]))
        return out
    cfg = b.cfg.long()
    per = lambda v: torch.zeros((b.nconfig,) + v.shape[1:], dtype=torch.float64, device=DEV).index_add(0, cfg, v)  # noqa: E731
    Ec = per(E)
    Sc = per(_sym(r, G).sum(1))[:, [0, 1, 2, 5, 4, 3]] / b.volumes[:, None]
    if kind == "batch":
        return {"energy": Ec, "forces": F, "stress": Sc}
    leaf = [t.clone().requires_grad_() for t in (Ec, F, Sc)]
    loss = _weighted_loss(*leaf, targets)
    gE, gF, gS = torch.autograd.grad(loss, leaf)
    # the loss gradient is that of sum_i gE E_i + sum_s dr_s . dE_i/dr_s with dr the direction below
    c = gS / b.volumes[:, None]
    C = torch.stack([torch.stack([c[:, 0], c[:, 5] / 2, c[:, 4] / 2], -1),
                     torch.stack([c[:, 5] / 2, c[:, 1], c[:, 3] / 2], -1),
                     torch.stack([c[:, 4] / 2, c[:, 3] / 2, c[:, 2]], -1)], 1)
    dr = gF[:, None] - gF[js.clamp_min(0).long()] + torch.einsum("nab,nsb->nsa", C[cfg], r)
    q = _tensors(p)
    coef = {k: v.requires_grad_() for k, v in coef.items()}
    total = [torch.zeros_like(v) for v in coef.values()]
    for s, i, rr, t, mask in _chunks(p, it, r, jt, counts):
        rr.requires_grad_()
        e = _site_energies(p, q, coef, i, rr, t, mask)
        g = torch.autograd.grad(e.sum(), rr, create_graph=True)[0]
        value = (gE[cfg[s]] * e).sum() + (dr[s] * g * mask.unsqueeze(-1)).sum()
        for a, v in zip(total, torch.autograd.grad(value, list(coef.values()))):
            a += v
    return {"loss": loss.detach(), "energy": Ec, "forces": F, "stress": Sc,
            **{"grad_" + k: v for k, v in zip(coef, total)}}


def _weighted_loss(E, F, S, targets):
    return sum(w * (a - t).square().sum() for w, a, t in zip((1.0, 0.01, 0.001), (E, F, S), targets))
