"""GPU parity of the AEV, energies and forces against the FP64 oracle.

Tolerances (from the error budget of the path): force RMSE <= 0.05
kcal/mol/A and |dE|/N <= 1e-4 kcal/mol/atom against the FP64 oracle;
AEV features within 2e-5 absolute + 1e-4 relative (float32 kernel)."""

from pathlib import Path

import numpy as np
import pytest
import torch

from fennol_b200.params import AEVConfig, MLPConfig, init_weights
from fennol_b200.potential import ANIPotential, HARTREE_TO_KCALMOL
from fennol_b200.systems import molecule_batch, water_box
from oracle import ani_ref

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).parent / "golden"
CFG, MCFG = AEVConfig(), MLPConfig()
FORCE_RMSE_TOL = 0.05   # kcal/mol/A
ENERGY_TOL = 1e-4       # kcal/mol/atom


def errors(e, f, ref_e, ref_f, natoms):
    de = np.abs(np.asarray(e) - ref_e) * HARTREE_TO_KCALMOL / np.asarray(natoms)
    rmse = np.sqrt(np.mean((np.asarray(f) - ref_f) ** 2)) * HARTREE_TO_KCALMOL
    return float(de.max()), float(rmse)


@pytest.fixture(scope="module")
def pot32(cuda_device):
    return ANIPotential(precision="fp32", device=cuda_device, seed=0)


def test_golden_water64_energy_forces(pot32):
    d = np.load(GOLDEN / "water64.npz")
    e, f = pot32.energy_and_forces(d["coordinates"], d["species"], [192], d["cell"][None])
    de, rmse = errors(e.cpu().numpy(), f.cpu().numpy(), d["energy"], d["forces"], [192])
    assert de <= ENERGY_TOL and rmse <= FORCE_RMSE_TOL, (de, rmse)
    # much tighter in practice for the float32 form
    assert rmse < 5e-3


def test_aev_rows_match_oracle(pot32, cuda_device):
    d = np.load(GOLDEN / "water64.npz")
    pot32.energy_and_forces(d["coordinates"], d["species"], [192], d["cell"][None])
    layout, g, ws = next(iter(pot32._cache.values()))
    rows = ws.x.float().cpu().numpy()[layout.atom_row_host[:8], :1008]
    np.testing.assert_allclose(rows, d["aev_rows"], rtol=1e-4, atol=2e-5)


def test_golden_molecules(pot32):
    d = np.load(GOLDEN / "molecules6.npz")
    e, f = pot32.energy_and_forces(d["coordinates"], d["species"], d["natoms"])
    de, rmse = errors(e.cpu().numpy(), f.cpu().numpy(), d["energy"], d["forces"], d["natoms"])
    assert de <= ENERGY_TOL and rmse <= FORCE_RMSE_TOL, (de, rmse)


@pytest.mark.parametrize("n_side,seed", [(8, 1), (12, 2)])
def test_water_boxes_vs_fp64(pot32, n_side, seed):
    s = water_box(n_side, seed=seed)
    r = ani_ref.energy_and_forces(s.coordinates, s.species, [s.natoms], pot32.weights, CFG, MCFG,
                                  cells=s.cell[None])
    e, f = pot32.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    de, rmse = errors(e.cpu().numpy(), f.cpu().numpy(), r["energy"], r["forces"], [s.natoms])
    assert de <= ENERGY_TOL and rmse <= FORCE_RMSE_TOL, (de, rmse)


def test_net_force_vanishes(pot32):
    s = water_box(8, seed=3)
    _, f = pot32.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    net = f.double().sum(0).cpu().numpy() * HARTREE_TO_KCALMOL
    assert np.abs(net).max() < 1e-2


def test_ensemble_mean(cuda_device):
    W = init_weights(CFG, MCFG, seed=7, n_models=3)
    pot = ANIPotential(precision="fp32", device=cuda_device, weights=W)
    mols = molecule_batch(5, seed=12)
    xyz = np.concatenate([m.coordinates for m in mols])
    sp = np.concatenate([m.species for m in mols])
    nat = [m.natoms for m in mols]
    r = ani_ref.energy_and_forces(xyz, sp, nat, W, CFG, MCFG)
    e, f = pot.energy_and_forces(xyz, sp, nat)
    de, rmse = errors(e.cpu().numpy(), f.cpu().numpy(), r["energy"], r["forces"], nat)
    assert de <= ENERGY_TOL and rmse <= FORCE_RMSE_TOL, (de, rmse)


def test_batched_equals_alone(pot32):
    """Each system's result is the same alone and inside a mixed batch."""
    box = water_box(6, seed=4)
    mols = molecule_batch(4, seed=13)
    systems = [mols[0], box, mols[1], mols[2], mols[3]]
    cells = [None, box.cell, None, None, None]
    xyz = np.concatenate([s.coordinates for s in systems])
    sp = np.concatenate([s.species for s in systems])
    nat = [s.natoms for s in systems]
    e_mix, f_mix = pot32.energy_and_forces(xyz, sp, nat, cells)
    e_mix, f_mix = e_mix.cpu().numpy().copy(), f_mix.cpu().numpy().copy()
    off = np.concatenate([[0], np.cumsum(nat)])
    for b, s in enumerate(systems):
        c = None if cells[b] is None else cells[b][None]
        e, f = pot32.energy_and_forces(s.coordinates, s.species, [s.natoms], c)
        assert abs(float(e[0]) - e_mix[b]) * HARTREE_TO_KCALMOL / s.natoms < 1e-6
        np.testing.assert_allclose(f.cpu().numpy(), f_mix[off[b]:off[b + 1]], atol=2e-5)


def test_staged_adjoint_matches_unstaged(cuda_device):
    """fennol_aev_backward_staged (reading the staging saved by
    fennol_aev_forward_staged) gives the forces of fennol_aev_backward, and
    the staged forward writes the same AEV rows as the plain one."""
    from fennol_b200 import _lib
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr, _ptr

    pot = ANIPotential(precision="bf16x2", device=cuda_device, seed=0, bf16_weights=True)
    s = water_box(6, seed=31)
    x = torch.tensor(s.coordinates, dtype=torch.float32, device=cuda_device)
    pot.energy_and_forces(x, s.species, [s.natoms], s.cell[None])
    lay, g, ws = next(iter(pot._cache.values()))
    st = torch.cuda.current_stream().cuda_stream
    lp = C_ptr(pot.params)
    args = (ws.xyzs.data_ptr(), lay.n, lay.t_atom_sys.data_ptr(), lay.t_cell.data_ptr(), g.rad_j.data_ptr(),
            g.rad_s.data_ptr(), g.rad_n.data_ptr(), g.cap_r, lp, lay.t_atom_row.data_ptr())
    rows = lay.t_atom_row.long()
    call("fennol_aev_forward", *args, ws.aev_kind, ws.x.data_ptr(), _ptr(ws.x_lo), ws.x.shape[1],
         ws.status.data_ptr(), st)
    x_plain = ws.x[rows].clone()
    call("fennol_aev_forward_staged", *args, ws.aev_kind, ws.x.data_ptr(), _ptr(ws.x_lo), ws.x.shape[1],
         g.aev_stage.data_ptr(), g.aev_stage.numel(), ws.status.data_ptr(), st)
    assert torch.equal(ws.x[rows], x_plain)
    ws.dx.normal_()  # any dE/dAEV rows
    f = []
    for name, extra in (("fennol_aev_backward", ()), ("fennol_aev_backward_staged", (g.aev_stage.data_ptr(),))):
        ws.forces4.zero_()
        call(name, *args, ws.dx.data_ptr(), ws.dx.shape[1], ws.forces4.data_ptr(), *extra,
             ws.status.data_ptr(), st)
        f.append(ws.forces4[:lay.n, :3].cpu().numpy().copy())
    assert int(ws.status[_lib.ST_ANG_OVERFLOW]) == 0
    scale = np.abs(f[0]).max()
    np.testing.assert_allclose(f[1], f[0], atol=1e-5 * scale, rtol=0)


@pytest.mark.parametrize("n_h,n_o", [(2, 1), (8, 1), (9, 3), (32, 2), (33, 1), (44, 6)])
def test_crowded_centres_vs_fp64(pot32, n_h, n_o):
    """Clusters in which every atom is an angular neighbour of every other: a
    triplet count at and around multiples of 32, one and several species, more
    neighbours of a species than the pair table holds (32), and rounds in
    which most lanes add to the same neighbour.

    Bound: a triplet's force terms carry about 2e-6 (the power of the angular
    factor) plus the float32 rounding of the sums; up to 49 * 48 of them of
    either sign meet in one force, whose sum of moduli is up to some 50 times
    the largest force: 1e-4 of it."""
    rng = np.random.default_rng(100 * n_h + n_o)
    n = n_h + n_o
    xyz = np.zeros((0, 3))
    while len(xyz) < n:  # a ball of radius 1.7, no two atoms nearer than 0.55
        p = rng.uniform(-1.7, 1.7, 3)
        if p @ p < 1.7 ** 2 and (len(xyz) == 0 or np.linalg.norm(xyz - p, axis=1).min() > 0.55):
            xyz = np.vstack([xyz, p])
    sp = np.array([1] * n_h + [8] * n_o)[rng.permutation(n)]
    xyz = xyz.astype(np.float32).astype(np.float64)
    r = ani_ref.energy_and_forces(xyz, sp, [n], pot32.weights, CFG, MCFG)
    _, f = pot32.energy_and_forces(xyz, sp, [n])
    np.testing.assert_allclose(f.cpu().numpy(), r["forces"], rtol=0, atol=1e-4 * np.abs(r["forces"]).max())


@pytest.mark.parametrize("precision", ["fp32", "bf16", "bf16x2", "f16x3x1"])
@pytest.mark.parametrize("off", [0, 1])
def test_forward_groups_and_staged_virial(cuda_device, precision, off):
    """fennol_aev_forward_groups writes the named column groups as
    fennol_aev_forward does (also at an output off 16 bytes) and no others, and
    the virial adjoint reads its staging: the same arithmetic in another
    instantiation, so a few float32 roundings (1e-6) of the largest value; the
    forces in the order of their atomics (1e-5, as above)."""
    from fennol_b200 import _lib
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr

    pot = ANIPotential(precision=precision, device=cuda_device, seed=0)
    s = water_box(5, seed=33)
    x = torch.tensor(s.coordinates, dtype=torch.float32, device=cuda_device)
    pot.energy_and_forces(x, s.species, [s.natoms], s.cell[None])
    lay, g, ws = next(iter(pot._cache.values()))
    st = torch.cuda.current_stream().cuda_stream
    args = (ws.xyzs.data_ptr(), lay.n, lay.t_atom_sys.data_ptr(), lay.t_cell.data_ptr(), g.rad_j.data_ptr(),
            g.rad_s.data_ptr(), g.rad_n.data_ptr(), g.cap_r, C_ptr(pot.params), lay.t_atom_row.data_ptr())
    rows, d0 = ws.x.shape
    F = pot.aev_cfg.aev_length
    groups = pot.active_groups(lay.species_mask)
    named = np.array([(int(groups[c // 1024]) >> (c // 16 % 64)) & 1 for c in range(F)], bool)
    assert 0 < named.sum() < F
    got = []
    for words in (None, groups):
        bufs = [torch.full((rows * d0 + off,), 7.0, dtype=ws.x.dtype, device=cuda_device) for _ in range(2)]
        lo = bufs[1][off:] if ws.x_lo is not None else None
        out = (ws.aev_kind, bufs[0][off:].data_ptr(), None if lo is None else lo.data_ptr(), d0)
        if words is None:
            call("fennol_aev_forward", *args, *out, ws.status.data_ptr(), st)
        else:
            ws.forces4.fill_(3.0)
            call("fennol_aev_forward_groups", *args, *out, words.ctypes.data, words.size, g.aev_stage.data_ptr(),
                 g.aev_stage.numel(), ws.forces4.data_ptr(), ws.status.data_ptr(), st)
            assert int(torch.count_nonzero(ws.forces4[:lay.n])) == 0
        got.append([b[off:].view(rows, d0)[lay.t_atom_row.long(), :F].float().cpu().numpy() for b in bufs])
    for k, (full, part) in enumerate(zip(*got)):
        np.testing.assert_array_equal(part[:, named], full[:, named])
        assert (part[:, ~named] == 7.0).all()
        assert k == 1 and ws.x_lo is None or (full[:, ~named] == 0.0).all()
    ws.dx.normal_()  # any dE/dAEV rows
    f, v = [], []
    for name, extra in (("fennol_aev_backward_virial", ()),
                        ("fennol_aev_backward_virial_staged", (g.aev_stage.data_ptr(),))):
        ws.forces4.zero_()
        av = torch.zeros((lay.n, 9), device=cuda_device)
        call(name, *args, ws.dx.data_ptr(), ws.dx.shape[1], ws.forces4.data_ptr(), av.data_ptr(), *extra,
             ws.status.data_ptr(), st)
        f.append(ws.forces4[:lay.n, :3].cpu().numpy())
        v.append(av.cpu().numpy())
    assert int(ws.status[_lib.ST_ANG_OVERFLOW]) == 0
    np.testing.assert_allclose(f[1], f[0], atol=1e-5 * np.abs(f[0]).max(), rtol=0)
    np.testing.assert_allclose(v[1], v[0], atol=1e-6 * np.abs(v[0]).max(), rtol=0)


@pytest.mark.parametrize("sizes", [[1], [1024], [1025, 0, 1023], [40000], [7] * 9 + [3000], [33 * 1024 + 1] * 3])
def test_sums_per_system(cuda_device, sizes):
    """Energies and virials summed per system: one and several chunks of 1024, more
    partials than a warp's 32, a warp or a thread per system, empty systems.

    Bound: n float64 additions of either sign round to n 2^-53 of the sum of moduli."""
    from fennol_b200 import _lib
    from fennol_b200._lib import call

    rng = np.random.default_rng(sum(sizes))
    n, nsys = sum(sizes), len(sizes)
    start = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    e = rng.standard_normal(n + 5).astype(np.float32)
    row = rng.permutation(n + 5)[:n].astype(np.int32)
    vir = rng.standard_normal((n, 9)).astype(np.float32)
    dev = [torch.tensor(a, device=cuda_device) for a in (e, row, start, vir)]
    st = torch.cuda.current_stream().cuda_stream
    ws = torch.zeros(int(_lib.load().fennol_energy_workspace_bytes(n, nsys)), dtype=torch.uint8, device=cuda_device)
    for name in ("fennol_energy_reduce", "fennol_energy_reduce_behind_adjoint"):
        energy = torch.zeros(nsys, dtype=torch.float64, device=cuda_device)
        e_atom = torch.zeros(n, dtype=torch.float64, device=cuda_device)
        call(name, dev[0].data_ptr(), dev[1].data_ptr(), n, dev[2].data_ptr(), nsys, 0.5, energy.data_ptr(),
             e_atom.data_ptr(), ws.data_ptr(), ws.numel(), st)
        v = torch.zeros((nsys, 9), dtype=torch.float64, device=cuda_device)
        call("fennol_virial_reduce", dev[3].data_ptr(), n, dev[2].data_ptr(), nsys, 0.5, v.data_ptr(), st)
        np.testing.assert_array_equal(e_atom.cpu().numpy(), 0.5 * e[row].astype(np.float64))
        for b in range(nsys):
            i = slice(start[b], start[b + 1])
            for got, x in ((energy[b:b + 1], e[row[i]][:, None]), (v[b], vir[i])):
                x = 0.5 * x.astype(np.float64)
                err = np.abs(got.cpu().numpy() - x.sum(0))
                assert (err <= (sizes[b] + 1) * 2.0 ** -52 * np.abs(x).sum(0)).all()


@pytest.mark.parametrize("kind,dtype", [(0, torch.float32), (1, torch.bfloat16), (2, torch.bfloat16),
                                        (3, torch.float16)])
@pytest.mark.parametrize("width,ld,off", [(1008, 1024, 0), (4, 4, 0), (1008, 1024, 1), (131, 134, 0), (1100, 1101, 0)])
def test_gather_rows(cuda_device, kind, dtype, width, ld, off):
    """Rows in atom order equal the parts converted and added by torch, aligned or not."""
    from fennol_b200._lib import call

    n, rows = 37, 50
    gen = torch.Generator(device=cuda_device).manual_seed(kind + width)
    parts = [torch.randn(rows * ld + off, generator=gen, device=cuda_device).to(dtype) for _ in range(2)]
    at = torch.randperm(rows, generator=gen, device=cuda_device)[:n].int()
    hi, lo = (p[off:].view(rows, ld) for p in parts)
    want = hi[at.long(), :width].float()
    if kind >= 2:
        want = want + lo[at.long(), :width].float()
    out = torch.full((n, width), 9.0, device=cuda_device)
    call("fennol_aev_gather_rows", hi.data_ptr(), lo.data_ptr() if kind >= 2 else None, kind, ld, at.data_ptr(), n,
         width, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert torch.equal(out, want)
