"""The work that is timed when the framework is measured: what its users have it do.

Each case goes through a public entry point as a user's program calls it: the direct API
(``ANIPotential``), the FeNNol API (``FENNIX``), molecular dynamics (``MDEngine``), the
training-loss gradient (``LossGradient``) and the request loop (``ServingEngine``).  The
systems are the ones of the tests and of the benchmark: periodic water boxes from a few
molecules to 98,304 atoms (cubic and ragged), and gas-phase organic molecules with seven
elements, alone and in batches.

``listed`` names the cases, ``draw`` gives another one of the same ranges, ``prepare``
makes the inputs and the handle a program keeps, ``run`` is one pass, ``work`` counts what
a pass cannot do without, and ``exact`` is the same result in 64 bits from plain torch.
"""

from __future__ import annotations

import functools
import math
from collections import OrderedDict

import numpy as np
import torch

# The ANI-2x layout of the tests and the benchmark.
SPECIES = ("H", "C", "N", "O", "S", "F", "Cl")
NUMBERS = (1, 6, 7, 8, 16, 9, 17)
RC, RCA = 5.2, 3.5
ETA_R, ETA_A, ZETA = 19.7, 12.5, 14.1
R_DIV, A_DIV, SECTIONS, START = 16, 8, 4, 0.9
ALPHA = 0.1
PAIRS = len(SPECIES) * (len(SPECIES) + 1) // 2
RADIAL = len(SPECIES) * R_DIV
ANGULAR = A_DIV * SECTIONS
DIMS = (RADIAL + PAIRS * ANGULAR, 256, 192, 160, 1)

LATTICE = 12.42 / 4.0           # A between water molecules at about 1 g/cm^3
MASSES = {1: 1.008, 8: 15.999}  # Da
KT = 3.166811563e-6 * 627.5096080305927 * 300.0                                          # kcal/mol at 300 K
DA = 1836.1526734252586 * 627.5096080305927 * (2.4188843e-2 / 1000.0) ** 2 / 0.52917721 ** 2  # kcal/mol ps^2/A^2
W_E, W_F = 1.0, 10.0            # weights of the training loss


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # one molecule, one network: geometry optimisation and scans; launches and latency count
        dict(name="molecule_24", kind="point", molecules=1, atoms=24, models=1, precision="f16x3x1"),
        # a small periodic box with the eight-network ensemble of ANI-2x, through FeNNol's API
        dict(name="water_192_ens8_fennix", kind="fennix", nx=4, ny=4, nz=4, models=8, precision="f16x3x1"),
        # conformers scored in one call, ensemble, the form for tight forces; every element present
        dict(name="molecules_256_ens8", kind="point", molecules=256, atoms=0, models=8, precision="f16x3x2"),
        # the direct API's default precision, on a box with no nice number in it
        dict(name="water_6k_fp32_ens8", kind="point", nx=12, ny=13, nz=14, models=8, precision="fp32"),
        # energies, forces and virial (pressure, stress for ASE), the FeNNol API's default precision
        dict(name="water_12k_virial", kind="virial", nx=16, ny=16, nz=16, models=1, precision="bf16x2"),
        # energies without forces: Monte Carlo, scoring
        dict(name="water_12k_energy_ens8", kind="energy", nx=16, ny=16, nz=16, models=8, precision="f16x3x1"),
        # descriptors of a set of molecules for another model
        dict(name="molecules_256_embedding", kind="embedding", molecules=256, atoms=0, models=1, precision="f16x3x1"),
        # a large single point through FeNNol's API: the list is built on every call
        dict(name="water_98k_ens8_fennix", kind="fennix", nx=32, ny=32, nz=32, models=8, precision="f16x3x1"),
        # Langevin dynamics, one network
        dict(name="md_water_12k", kind="md", nx=16, ny=16, nz=16, models=1, precision="f16x3x1", steps=10,
             thermostat="LGV"),
        # the benchmark's dynamics: NVE, the ensemble, 98,304 atoms
        dict(name="md_water_98k_ens8", kind="md", nx=32, ny=32, nz=32, models=8, precision="f16x3x1", steps=8,
             thermostat="NVE"),
        # one training step's gradient: energies and forces of 256 molecules
        dict(name="train_molecules_256", kind="train", molecules=256, atoms=0, models=1, precision="fp32"),
        # a queue of single points of uneven sizes: every batch is a new one
        dict(name="serve_32_points", kind="serve", requests=32, models=1, precision="f16x3x1"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, most):
    """Three sides of a water box, 27 to ``most`` molecules, uneven more often than not."""
    n = _log(rng, 27, most)
    nx, ny = (max(3, min(32, int(round(n ** (1.0 / 3.0) * rng.uniform(0.85, 1.15))))) for _ in range(2))
    return nx, ny, max(3, min(32, n // (nx * ny)))


def draw(rng):
    kind = rng.choice(["point", "point", "fennix", "fennix", "virial", "energy", "embedding", "md", "md", "train",
                       "serve"])
    case = dict(kind=kind, models=rng.choice([1, 1, 2, 5, 8]),
                precision=rng.choice(["f16x3x1", "f16x3x1", "f16x3x2", "bf16x2", "fp32"]))
    if kind == "serve":
        return dict(case, requests=_log(rng, 2, 64), models=1, precision="f16x3x1")
    if kind == "train":
        return dict(case, molecules=_log(rng, 2, 256), atoms=0, models=1, precision="fp32")
    if kind == "embedding" or (kind in ("point", "fennix", "energy") and rng.random() < 0.4):
        many = _log(rng, 1, 512)
        return dict(case, molecules=many, atoms=rng.randint(5, 60) if many == 1 else 0)
    # the FP32 form of large boxes with an ensemble costs more than the largest listed case
    most = 8000 if case["precision"] == "fp32" else 32768
    if kind == "md":
        case.update(steps=rng.randint(4, 10), thermostat=rng.choice(["LGV", "NVE"]))
        most = most // 4 if case["precision"] == "fp32" else most * 7 // 10
    nx, ny, nz = _box(rng, most)
    return dict(case, nx=nx, ny=ny, nz=nz)


# ------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=6)
def _weights(models, bf16, scale):
    """The model: seeded networks with N(0, 1/fan_in) float32 kernels and small biases (rounded to
    BF16 for the form made for models stored in BF16), float64 arrays that float32 represents."""
    out = []
    for m in range(models):
        rng = np.random.default_rng(1000 * m)
        model = {}
        for sym in SPECIES:
            layers = []
            for k, (din, dout) in enumerate(zip(DIMS[:-1], DIMS[1:])):
                w = rng.standard_normal((din, dout), dtype=np.float32) * np.float32(din ** -0.5)
                if k == 3:
                    w = w * np.float32(scale)
                if bf16:
                    w = torch.from_numpy(w).to(torch.bfloat16).to(torch.float32).numpy()
                b = rng.standard_normal(dout, dtype=np.float32) * np.float32(0.05)
                layers.append((w.astype(np.float64), b.astype(np.float64)))
            model[sym] = layers
        out.append(model)
    return out


def _model_of(case):
    # dynamics takes the last layer scaled down, so that forces are of thermal size
    return _weights(case["models"], case["precision"] == "bf16x2", 0.02 if case["kind"] == "md" else 1.0)


def _water(rng, nx, ny, nz):
    """Coordinates, atomic numbers and cell sides of a periodic box of nx x ny x nz waters."""
    sides = (np.array([nx, ny, nz]) * LATTICE).astype(np.float32).astype(np.float64)
    grid = np.stack(np.meshgrid(*(np.arange(k) + 0.5 for k in (nx, ny, nz)), indexing="ij"), -1).reshape(-1, 3)
    o = grid * (sides / np.array([nx, ny, nz])) + rng.uniform(-0.2, 0.2, (grid.shape[0], 3))
    u = rng.standard_normal((grid.shape[0], 3))
    v = rng.standard_normal((grid.shape[0], 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v -= (v * u).sum(1, keepdims=True) * u
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    half = math.radians(104.52) / 2
    h1 = o + 0.9572 * (math.cos(half) * u + math.sin(half) * v)
    h2 = o + 0.9572 * (math.cos(half) * u - math.sin(half) * v)
    xyz = np.stack([o, h1, h2], 1).reshape(-1, 3).astype(np.float32)
    return xyz, np.tile(np.array([8, 1, 1], np.int32), grid.shape[0]), sides


def _chain(rng, n):
    """A bonded random walk of n atoms, no two nearer than 0.9 A."""
    xyz = np.zeros((n, 3))
    k = 1
    while k < n:
        for _ in range(60):
            d = rng.standard_normal(3)
            new = xyz[k - 1] + d * (rng.uniform(1.1, 1.6) / math.sqrt(float(d @ d)))
            away = xyz[:k] - new
            if float((away * away).sum(1).min()) >= 0.81:
                xyz[k] = new
                k += 1
                break
        else:
            k = max(1, k - 4)  # walled in: take some steps back
    z = rng.choice(np.array(NUMBERS, np.int32), size=n, p=(0.50, 0.30, 0.07, 0.08, 0.02, 0.02, 0.01))
    return (xyz - xyz.mean(0)).astype(np.float32), z.astype(np.int32)


def _inputs(case, seed):
    """Coordinates, atomic numbers, atoms of each system and (water) the cell's sides."""
    rng = np.random.default_rng([int(seed), 7])
    if "nx" in case:
        xyz, z, sides = _water(rng, case["nx"], case["ny"], case["nz"])
        return xyz, z, np.array([z.shape[0]], np.int32), sides
    sizes = [case["atoms"]] * case["molecules"] if case["atoms"] else \
        [int(n) for n in np.random.default_rng(case["molecules"]).integers(10, 41, case["molecules"])]
    parts = [_chain(rng, n) for n in sizes]
    return (np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]),
            np.array(sizes, np.int32), None)


def _requests(case, seed):
    """Uneven single points, half of them chains, half periodic boxes, 8 to about 2,000 atoms."""
    rng, sizes = np.random.default_rng([int(seed), 11]), np.random.default_rng(case["requests"])
    out = []
    for _ in range(case["requests"]):
        n = int(round(math.exp(sizes.uniform(math.log(8), math.log(2000)))))
        if sizes.uniform() < 0.5 or n < 24:
            out.append((*_chain(rng, n), None))
        else:
            k = max(2, int(round((n / 3) ** (1 / 3))))
            out.append(_water(rng, k, k, k))
    return out


def _targets(seed, natoms):
    """Reference energies and forces of a training batch."""
    rng = np.random.default_rng([int(seed), 13])
    return rng.standard_normal(len(natoms)) * 0.3 * np.sqrt(natoms), rng.standard_normal((int(natoms.sum()), 3)) * 0.05


def _fennix(case):
    from fennol_b200.fennix import FENNIX
    from fennol_b200.params import weights_to_variables

    sp = list(SPECIES)
    modules = OrderedDict(
        embedding=dict(module_name="ANI_AEV", species_order=sp, graph_angle_key="graph_angle", radial_eta=ETA_R,
                       angular_eta=ETA_A, radial_dist_divisions=R_DIV, angular_dist_divisions=A_DIV, zeta=ZETA,
                       angle_sections=SECTIONS, radial_start=START, angular_start=START),
        energy=dict(module_name="SPECIES_INDEX_NET", species_order=sp, activation="partial(celu,alpha=0.1)",
                    output_dim=1, hidden_neurons=list(DIMS[1:4]), input_key="embedding", squeeze=True))
    prep = OrderedDict(
        graph_filter_angle=dict(module_name="GRAPH_FILTER", cutoff=RCA, graph_key="graph_angle",
                                parent_graph="graph"),
        angle_extension=dict(module_name="GRAPH_ANGULAR_EXTENSION", graph_key="graph_angle"),
        species_indexer=dict(output_key="species_index"))
    return FENNIX(RC, modules, prep, energy_terms=["energy"], precision=case["precision"],
                  variables=weights_to_variables(_model_of(case), "energy"))


def prepare(case, seed):
    from fennol_b200.potential import ANIPotential

    kind = case["kind"]
    if kind == "serve":
        from fennol_b200.serving import ServeRequest, ServingEngine

        pot = ANIPotential(precision=case["precision"], weights=_model_of(case))
        reqs = [ServeRequest(k, "ef", z, x, None if sides is None else np.diag(sides))
                for k, (x, z, sides) in enumerate(_requests(case, seed))]
        return dict(kind=kind, engine=ServingEngine(pot), requests=reqs)
    xyz, z, natoms, sides = _inputs(case, seed)
    cells = None if sides is None else np.diag(sides)[None]
    coords = torch.from_numpy(xyz).cuda()
    if kind == "point":
        pot = ANIPotential(precision=case["precision"], weights=_model_of(case))
        return dict(kind=kind, pot=pot, args=(coords, z, natoms, cells))
    if kind == "train":
        from fennol_b200.training import LossGradient

        pot = ANIPotential(precision=case["precision"], weights=_model_of(case))
        e_ref, f_ref = _targets(seed, natoms)
        return dict(kind=kind, loss=LossGradient(pot, w_e=W_E, w_f=W_F), args=(coords, z, natoms, e_ref, f_ref))
    if kind == "md":
        from fennol_b200.md import MDEngine

        pot = ANIPotential(precision=case["precision"], weights=_model_of(case))
        mass = np.array([MASSES[int(k)] for k in z]) * DA
        v = np.random.default_rng([int(seed), 17]).standard_normal(xyz.shape) * np.sqrt(KT / mass)[:, None]
        eng = MDEngine(pot, xyz.astype(np.float64), z, cells[0], dt_fs=0.5, thermostat=case["thermostat"],
                       temperature=300.0, gamma_ps=1.0, skin=1.0, trigger="stride", seed=int(seed) % (1 << 31),
                       velocities=v)
        start = (eng.x.clone(), eng.v.clone(), eng.ws.forces4.clone())
        return dict(kind=kind, engine=eng, start=start, steps=case["steps"])
    args = dict(species=z, coordinates=coords, natoms=natoms)
    if cells is not None:
        args["cells"] = cells
        if min(sides) >= 2 * RC:
            args["flags"] = {"minimum_image": True}
    return dict(kind=kind, model=_fennix(case), args=args)


# ------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "point":
        e, f = state["pot"].energy_and_forces(*state["args"])
        return {"energy": e, "forces": f}
    if kind == "fennix":
        e, f, out = state["model"].energy_and_forces(**state["args"])
        return {"energy": e, "forces": f, "atomic": out["energy"]}
    if kind == "virial":
        e, f, v, out = state["model"].energy_and_forces_and_virial(**state["args"])
        return {"energy": e, "forces": f, "virial": v, "atomic": out["energy"]}
    if kind == "energy":
        e, out = state["model"].total_energy(**state["args"])
        return {"energy": e, "atomic": out["energy"]}
    if kind == "embedding":
        out = state["model"](**state["args"])
        return {"embedding": out["embedding"], "energy": out["total_energy"], "atomic": out["energy"]}
    if kind == "train":
        terms, grads = state["loss"](*state["args"])
        return {"loss": terms.loss, "energy_loss": terms.energy_loss, "force_loss": terms.force_loss,
                "energy": terms.energy, "forces": terms.forces,
                "grads": {sym: [list(wb) for wb in grads[sym]] for sym in SPECIES}}
    if kind == "md":
        # a short trajectory from a stored configuration
        eng, (x, v, f4) = state["engine"], state["start"]
        eng.x.copy_(x)
        eng.v.copy_(v)
        eng.ws.forces4.copy_(f4)
        eng.step_counter.zero_()
        eng.step_count = 0
        eng.run(state["steps"])
        return {"x": eng.x, "v": eng.v, "forces": eng.ws.forces4[:, :3]}
    results = sorted(state["engine"].run(state["requests"], realtime=False), key=lambda r: r.rid)
    return {"energy": np.array([r.energy for r in results]), "forces": np.concatenate([r.forces for r in results])}


# ------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind, models = case["kind"], case["models"]
    water = "nx" in case
    if kind == "serve":
        atoms, present = case["requests"] * 360, 7  # the mean of the sizes' distribution
    else:
        atoms = 3 * case["nx"] * case["ny"] * case["nz"] if water else case["molecules"] * (case["atoms"] or 25)
        present = 2 if water else 7
    columns = present * R_DIV + present * (present + 1) // 2 * ANGULAR
    network = columns * DIMS[1] + DIMS[1] * DIMS[2] + DIMS[2] * DIMS[3] + DIMS[3]
    # neighbours within both cutoffs of the liquid and of the chains; 2 operations a multiply-add
    near, angular = (59, 17) if water else (15, 8)
    features = near * R_DIV * 4 + angular * (angular - 1) // 2 * (ANGULAR * 2 + 60)
    forces = kind not in ("energy", "embedding")
    flops = atoms * (models * 2 * network * (2 if forces else 1) + features * (3 if forces else 1))
    weights = 4 * models * present * network
    values = atoms * (12 + 4 + 4 + (12 if forces else 0))
    if kind == "embedding":
        values += atoms * DIMS[0] * 4
    if kind == "train":
        # the sweep for the parameters: activations and tangents, forward and twice backward
        flops += atoms * 3 * 2 * 2 * network
        return {"bytes": values + 2 * weights, "flops": flops}
    if kind == "md":
        steps = case["steps"]
        return {"bytes": steps * (atoms * (48 * 2 + 8) + weights), "flops": steps * flops}
    return {"bytes": values + weights, "flops": flops}


# ------------------------------------------------------------------- the same in 64 bits
def _pair_column(device):
    s1, s2 = np.triu_indices(len(SPECIES))
    table = np.zeros((len(SPECIES), len(SPECIES)), np.int64)
    table[s1, s2] = table[s2, s1] = np.arange(s1.shape[0])
    return torch.from_numpy(table).to(device)


def _index_of(z):
    table = np.full(max(NUMBERS) + 1, -1, np.int64)
    table[list(NUMBERS)] = np.arange(len(NUMBERS))
    return table[z]


def _edges(x, lo, hi, sides, centres):
    """Directed pairs (i, j) of one system's centres [centres) within the cutoff, and x_j - x_i."""
    xi, xj = x[centres[0]:centres[1]], x[lo:hi]
    i0 = torch.arange(centres[0], centres[1], device=x.device)
    if sides is None:
        images = [(0, 0, 0)]
    else:
        reps = [0 if s >= 2 * RC else int(math.ceil(RC / s)) + 1 for s in sides]
        images = [(a, b, c) for a in range(-reps[0], reps[0] + 1) for b in range(-reps[1], reps[1] + 1)
                  for c in range(-reps[2], reps[2] + 1)]
        box = torch.tensor(np.asarray(sides), dtype=torch.float64, device=x.device)
        wide = torch.tensor([float(s >= 2 * RC) for s in sides], dtype=torch.float64, device=x.device)
    found = []
    for image in images:
        r = xj[None, :, :] - xi[:, None, :]
        if sides is not None:
            r = r - torch.round(r / box) * box * wide + torch.tensor(image, dtype=torch.float64, device=x.device) * box
        near = (r * r).sum(-1) < RC * RC
        if image == (0, 0, 0):
            near[torch.arange(xi.shape[0], device=x.device), i0 - lo] = False
        a, b = near.nonzero(as_tuple=True)
        found.append((a + centres[0], b + lo, r[a, b]))
    i = torch.cat([f[0] for f in found])
    order = torch.argsort(i, stable=True)
    return i[order], torch.cat([f[1] for f in found])[order], torch.cat([f[2] for f in found])[order]


def _features(i, r, sj, first, n, table):
    """AEV rows of n centres (first, first + 1, ...) from their sorted edges: vectors r, neighbour species sj."""
    dev = r.device
    d = (r * r).sum(-1).sqrt()
    centre = i - first
    shift_r = START + (RC - START) / R_DIV * torch.arange(R_DIV, dtype=torch.float64, device=dev)
    cut = 0.5 * torch.cos(d * (math.pi / RC)) + 0.5
    terms = (0.25 * cut)[:, None] * torch.exp(-ETA_R * (d[:, None] - shift_r) ** 2)
    radial = torch.zeros(n * len(SPECIES), R_DIV, dtype=torch.float64, device=dev)
    radial = radial.index_add(0, centre * len(SPECIES) + sj, terms).reshape(n, RADIAL)
    # pairs of neighbours within the angular cutoff, a before b
    keep = (d.detach() < RCA).nonzero().squeeze(1)
    c = centre[keep]
    count = torch.bincount(c, minlength=n)
    start = torch.cumsum(count, 0) - count
    most = int(count.max()) if keep.numel() else 0
    angular = torch.zeros(n * PAIRS, ANGULAR, dtype=torch.float64, device=dev)
    if most >= 2:
        ta, tb = torch.triu_indices(most, most, 1, device=dev)
        at, k = (tb[None, :] < count[:, None]).nonzero(as_tuple=True)
        a, b = keep[start[at] + ta[k]], keep[start[at] + tb[k]]
        da, db = d[a], d[b]
        cos = 0.95 * (r[a] * r[b]).sum(-1) / (da * db)
        sin = (1 - cos * cos).sqrt()
        z = math.pi / SECTIONS * (torch.arange(SECTIONS, dtype=torch.float64, device=dev) + 0.5)
        shift_a = START + (RCA - START) / A_DIV * torch.arange(A_DIV, dtype=torch.float64, device=dev)
        fa = 0.5 * torch.cos(da * (math.pi / RCA)) + 0.5
        fb = 0.5 * torch.cos(db * (math.pi / RCA)) + 0.5
        f1 = (2.0 * fa * fb)[:, None] * ((1 + cos[:, None] * torch.cos(z) + sin[:, None] * torch.sin(z)) / 2) ** ZETA
        f2 = torch.exp(-ETA_A * (0.5 * (da + db)[:, None] - shift_a) ** 2)
        block = (f2[:, :, None] * f1[:, None, :]).reshape(-1, ANGULAR)
        angular = angular.index_add(0, at * PAIRS + table[sj[a], sj[b]], block)
    return torch.cat([radial, angular.reshape(n, PAIRS * ANGULAR)], 1)


def _networks(rows, si, nets):
    """Mean energy of each row over the models; nets[model][species] = [(W, b), ...]."""
    total = torch.zeros(rows.shape[0], dtype=torch.float64, device=rows.device)
    for s in range(len(SPECIES)):
        at = (si == s).nonzero().squeeze(1)
        if at.numel() == 0:
            continue
        mean = 0
        for net in nets:
            h = rows[at]
            for k, (w, b) in enumerate(net[s]):
                h = h @ w + b
                if k < 3:
                    h = torch.clamp(h, min=0) + ALPHA * torch.expm1(torch.clamp(h, max=0) / ALPHA)
            mean = mean + h[:, 0] / len(nets)
        total = total.index_add(0, at, mean)
    return total


def _device_networks(weights, device, grad=False):
    return [[[tuple(torch.tensor(t, dtype=torch.float64, device=device, requires_grad=grad) for t in wb)
              for wb in model[sym]] for sym in SPECIES] for model in weights]


def _evaluate(xyz, z, natoms, sides, nets, device, want="forces"):
    """Energies, forces, virials and atomic energies; with want="rows" the AEV rows too."""
    table = _pair_column(device)
    x = torch.from_numpy(np.asarray(xyz, np.float64)).to(device)
    si = torch.from_numpy(_index_of(z)).to(device)
    n = x.shape[0]
    bounds = np.concatenate([[0], np.cumsum(natoms)])
    atomic = torch.zeros(n, dtype=torch.float64, device=device)
    forces = torch.zeros_like(x)
    virial = torch.zeros(len(natoms), 3, 3, dtype=torch.float64, device=device)
    rows = []
    for b in range(len(natoms)):
        lo, hi = int(bounds[b]), int(bounds[b + 1])
        step = max(32, min(2048, int(4e7) // max(hi - lo, 1)))
        for c0 in range(lo, hi, step):
            c1 = min(hi, c0 + step)
            i, j, r = _edges(x, lo, hi, sides, (c0, c1))
            r = r.detach().requires_grad_(want == "forces")
            row = _features(i, r, si[j], c0, c1 - c0, table)
            e = _networks(row, si[c0:c1], nets)
            atomic[c0:c1] = e.detach()
            if want == "rows":
                rows.append(row)
            if want == "forces" and i.numel():
                (g,) = torch.autograd.grad(e.sum(), r)
                forces.index_add_(0, i, g)
                forces.index_add_(0, j, -g)
                virial[b] += r.detach().T @ g
    system = torch.from_numpy(np.repeat(np.arange(len(natoms)), natoms)).to(device)
    energy = torch.zeros(len(natoms), dtype=torch.float64, device=device).index_add(0, system, atomic)
    return energy, forces, virial, atomic, rows


def _training(xyz, z, natoms, e_ref, f_ref, weights, device):
    """The loss, its terms and its gradient by differentiating twice."""
    table = _pair_column(device)
    x = torch.from_numpy(np.asarray(xyz, np.float64)).to(device)
    si = torch.from_numpy(_index_of(z)).to(device)
    nets = _device_networks(weights, device, grad=True)
    bounds = np.concatenate([[0], np.cumsum(natoms)])
    parts = [_edges(x, int(bounds[b]), int(bounds[b + 1]), None, (int(bounds[b]), int(bounds[b + 1])))
             for b in range(len(natoms))]
    i, j = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    r = torch.cat([p[2] for p in parts]).requires_grad_(True)
    atomic = _networks(_features(i, r, si[j], 0, x.shape[0], table), si, nets)
    (g,) = torch.autograd.grad(atomic.sum(), r, create_graph=True)
    forces = torch.zeros_like(x).index_add(0, i, g).index_add(0, j, -g)
    system = torch.from_numpy(np.repeat(np.arange(len(natoms)), natoms)).to(device)
    energy = torch.zeros(len(natoms), dtype=torch.float64, device=device).index_add(0, system, atomic)
    le = W_E * ((energy - torch.from_numpy(e_ref).to(device)) ** 2).mean()
    lf = W_F * ((forces - torch.from_numpy(f_ref).to(device)) ** 2).mean()
    flat = [t for layers in nets[0] for wb in layers for t in wb]
    grads = iter(torch.autograd.grad(le + lf, flat, allow_unused=True, materialize_grads=True))
    le, lf = float(le.detach()), float(lf.detach())
    return {"loss": le + lf, "energy_loss": le, "force_loss": lf, "energy": energy.detach(), "forces": forces.detach(),
            "grads": {sym: [[next(grads), next(grads)] for _ in range(4)] for sym in SPECIES}}


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind, weights = case["kind"], _model_of(case)
    if kind == "md":
        return None  # the noise is the framework's own stream, and a trajectory amplifies what it is given
    if kind == "serve":
        nets = _device_networks(weights, device)
        done = [_evaluate(x, z, [len(z)], sides, nets, device) for x, z, sides in _requests(case, seed)]
        return {"energy": torch.cat([d[0] for d in done]), "forces": torch.cat([d[1] for d in done])}
    xyz, z, natoms, sides = _inputs(case, seed)
    if kind == "train":
        e_ref, f_ref = _targets(seed, natoms)
        return _training(xyz, z, natoms, e_ref, f_ref, weights, device)
    want = {"energy": "energy", "embedding": "rows"}.get(kind, "forces")
    energy, forces, virial, atomic, rows = _evaluate(xyz, z, natoms, sides, _device_networks(weights, device), device,
                                                     want)
    if kind == "point":
        return {"energy": energy, "forces": forces}
    if kind == "fennix":
        return {"energy": energy, "forces": forces, "atomic": atomic}
    if kind == "virial":
        return {"energy": energy, "forces": forces, "virial": virial, "atomic": atomic}
    if kind == "energy":
        return {"energy": energy, "atomic": atomic}
    return {"embedding": torch.cat(rows), "energy": energy, "atomic": atomic}
