"""GPU parity of the tcgen05 (tensor-core) species MLP against the FP64 oracle
and the FP32 CUDA-core form.

Tolerances: force RMSE <= 0.05 kcal/mol/A and |dE|/N <= 1e-4 kcal/mol/atom
(max over systems) against the FP64 oracle of the same float32 weights for
the FP16 forms f16x3x1 / f16x3x2 (seeded N(0, 1/fan_in) weights, not
rounded), and for bf16x2 on BF16-exact weights (the BF16 model form).
bf16x3 on arbitrary float weights carries a systematic ~1e-4 kcal/mol/atom
energy bias from the weights' own 16-bit hi+lo representation and is held to
3e-4; the single-product BF16 form is reported against a looser bound."""

import numpy as np
import pytest
import torch

from fennol_b200.params import AEVConfig, MLPConfig, init_weights
from fennol_b200.potential import ANIPotential, HARTREE_TO_KCALMOL, round_weights_bf16
from fennol_b200.systems import molecule_batch, water_box
from oracle import ani_ref

pytestmark = pytest.mark.gpu
CFG, MCFG = AEVConfig(), MLPConfig()


def errors(pot, xyz, sp, nat, cells=None):
    e, f = pot.energy_and_forces(xyz, sp, nat, cells)
    r = ani_ref.energy_and_forces(xyz, sp, nat, pot.weights, CFG, MCFG, cells=cells)
    de = np.max(np.abs(e.cpu().numpy() - r["energy"]) / np.asarray(nat)) * HARTREE_TO_KCALMOL
    rmse = float(np.sqrt(np.mean((f.cpu().numpy() - r["forces"]) ** 2)) * HARTREE_TO_KCALMOL)
    return de, rmse


def _err_word(pot):
    layout, g, ws = next(iter(pot._cache.values()))
    return int(ws.mlp_ws[:4].view(torch.int32)[0])


@pytest.mark.parametrize("n_side", [4, 8])
def test_bf16x3_water_vs_fp64(cuda_device, n_side):
    pot = ANIPotential(precision="bf16x3", device=cuda_device, seed=0)
    s = water_box(n_side, seed=n_side)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert _err_word(pot) == 0
    assert de <= 3e-4 and rmse <= 0.05, (de, rmse)


def test_bf16x2_with_bf16_weights(cuda_device):
    W = round_weights_bf16(init_weights(CFG, MCFG, seed=0))
    pot = ANIPotential(precision="bf16x2", device=cuda_device, weights=W)
    s = water_box(6, seed=3)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert de <= 1e-4 and rmse <= 0.05, (de, rmse)


def test_bf16_single_product_is_coarser(cuda_device):
    pot = ANIPotential(precision="bf16", device=cuda_device, seed=0)
    s = water_box(6, seed=4)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert rmse < 1.0 and de < 0.1, (de, rmse)   # ~0.2 kcal/mol/A expected: outside the budget


def test_bf16x3_molecules_all_species_and_ensemble(cuda_device):
    W = init_weights(CFG, MCFG, seed=5, n_models=3)
    pot = ANIPotential(precision="bf16x3", device=cuda_device, weights=W)
    mols = molecule_batch(30, seed=8)
    xyz = np.concatenate([m.coordinates for m in mols])
    sp = np.concatenate([m.species for m in mols])
    nat = [m.natoms for m in mols]
    de, rmse = errors(pot, xyz, sp, nat)
    assert de <= 3e-4 and rmse <= 0.05, (de, rmse)


def test_bf16x2_ensemble_molecules(cuda_device):
    W = round_weights_bf16(init_weights(CFG, MCFG, seed=6, n_models=4))
    pot = ANIPotential(precision="bf16x2", device=cuda_device, weights=W)
    mols = molecule_batch(30, seed=9)
    xyz = np.concatenate([m.coordinates for m in mols])
    sp = np.concatenate([m.species for m in mols])
    nat = [m.natoms for m in mols]
    de, rmse = errors(pot, xyz, sp, nat)
    assert de <= 1e-4 and rmse <= 0.05, (de, rmse)


def test_tensor_core_matches_fp32_form(cuda_device):
    s = water_box(10, seed=9)
    p32 = ANIPotential(precision="fp32", device=cuda_device, seed=0)
    ptc = ANIPotential(precision="bf16x3", device=cuda_device, seed=0)
    e32, f32 = p32.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    etc, ftc = ptc.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    assert abs(float(e32[0]) - float(etc[0])) * HARTREE_TO_KCALMOL / s.natoms < 3e-4
    rmse = float(torch.sqrt(torch.mean((f32 - ftc) ** 2))) * HARTREE_TO_KCALMOL
    assert rmse < 0.05


# ---- FP16 split forms on the unrounded float32 model --------------------------------

E_BUDGET, F_BUDGET = 1e-4, 0.05   # kcal/mol/atom, kcal/mol/A


@pytest.mark.parametrize("precision", ["f16x3x1", "f16x3x2"])
def test_f16_forms_water64_unrounded(cuda_device, precision):
    """C1: 64 waters, one model with the seeded float32 weights."""
    pot = ANIPotential(precision=precision, device=cuda_device, seed=0)
    s = water_box(4, seed=0)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert _err_word(pot) == 0
    assert de <= E_BUDGET and rmse <= F_BUDGET, (de, rmse)
    if precision == "f16x3x2":
        assert rmse <= 0.03, rmse   # the two-product input gradient: ~0.02 expected


@pytest.mark.parametrize("precision", ["f16x3x1", "f16x3x2"])
def test_f16_forms_water12k_unrounded(cuda_device, precision):
    """The 12,288-atom water box (4096 H2O), one model, float32 weights."""
    pot = ANIPotential(precision=precision, device=cuda_device, seed=0)
    s = water_box(16, seed=1)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert _err_word(pot) == 0
    assert de <= E_BUDGET and rmse <= F_BUDGET, (de, rmse)


def test_f16x3x1_ensemble8_unrounded(cuda_device):
    """8-model ensemble (independent seeds) on a 1536-atom water box."""
    W = init_weights(CFG, MCFG, seed=0, n_models=8)
    pot = ANIPotential(precision="f16x3x1", device=cuda_device, weights=W)
    s = water_box(8, seed=2)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert _err_word(pot) == 0
    assert de <= E_BUDGET and rmse <= F_BUDGET, (de, rmse)


@pytest.mark.parametrize("precision", ["f16x3x1", "f16x3x2"])
def test_f16_forms_molecules_all_species(cuda_device, precision):
    """30 molecules of 10-40 atoms with all seven species, 3-model ensemble:
    small systems, so the per-atom energy error is the max over molecules."""
    W = init_weights(CFG, MCFG, seed=5, n_models=3)
    pot = ANIPotential(precision=precision, device=cuda_device, weights=W)
    mols = molecule_batch(30, seed=8)
    xyz = np.concatenate([m.coordinates for m in mols])
    sp = np.concatenate([m.species for m in mols])
    nat = [m.natoms for m in mols]
    de, rmse = errors(pot, xyz, sp, nat)
    assert de <= E_BUDGET and rmse <= F_BUDGET, (de, rmse)


def test_f16_form_md_scale_model(cuda_device):
    """The MD workloads' model (last layer x 0.02): small weights in the last
    layer exercise the power-of-two gradient scale."""
    from fennol_b200.params import MD_OUTPUT_SCALE
    pot = ANIPotential(precision="f16x3x1", device=cuda_device, seed=0, output_scale=MD_OUTPUT_SCALE)
    s = water_box(6, seed=5)
    de, rmse = errors(pot, s.coordinates, s.species, [s.natoms], s.cell[None])
    assert de <= 1e-6 and rmse <= 5e-3, (de, rmse)


def test_f16_form_matches_fp32_form(cuda_device):
    s = water_box(10, seed=9)
    p32 = ANIPotential(precision="fp32", device=cuda_device, seed=0)
    p16 = ANIPotential(precision="f16x3x2", device=cuda_device, seed=0)
    e32, f32 = p32.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    e16, f16 = p16.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    assert abs(float(e32[0]) - float(e16[0])) * HARTREE_TO_KCALMOL / s.natoms < 2e-5
    rmse = float(torch.sqrt(torch.mean((f32 - f16) ** 2))) * HARTREE_TO_KCALMOL
    assert rmse < 0.03


@pytest.mark.parametrize("precision", ["bf16x2", "f16x3x1", "f16x3x2"])
def test_active_chunks_match_dense(cuda_device, precision):
    """fennol_mlp_energy_grad_active (water: 6 of 16 input chunks active)
    gives the dense call's row energies and its dE/dAEV on the active
    columns; the skipped input columns are zero, so only FP32 rounding of the
    accumulation may differ."""
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr, _ptr

    pot = ANIPotential(precision=precision, device=cuda_device, seed=0, n_models=2,
                       bf16_weights=precision == "bf16x2")
    s = water_box(6, seed=2)
    pot.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    layout, g, ws = next(iter(pot._cache.values()))
    mask = pot.active_chunks(layout.species_mask)
    assert mask == 0b110000001111
    st = torch.cuda.current_stream().cuda_stream
    outs = {}
    for name, m in (("active", mask), ("dense", None)):
        e_rows = torch.zeros_like(ws.e_rows)
        dx = torch.zeros_like(ws.dx)
        args = (pot.precision, layout.rows, layout.ntiles, layout.t_tile_species.data_ptr(),
                layout.t_tile_row.data_ptr(), C_ptr(pot.mlp.struct), ws.x.data_ptr(), _ptr(ws.x_lo))
        tail = (e_rows.data_ptr(), dx.data_ptr(), ws.mlp_ws.data_ptr(), ws.mlp_ws.numel(), st)
        if m is None:
            call("fennol_mlp_energy_grad", *args, *tail)
        else:
            call("fennol_mlp_energy_grad_active", *args, m, *tail)
        torch.cuda.synchronize()
        outs[name] = (e_rows.cpu().numpy(), dx.cpu().numpy())
    assert _err_word(pot) == 0
    cols = np.concatenate([np.arange(64 * c, 64 * c + 64) for c in range(16) if (mask >> c) & 1])
    np.testing.assert_allclose(outs["active"][0], outs["dense"][0], rtol=1e-6, atol=1e-7)
    da, dd = outs["active"][1], outs["dense"][1]
    np.testing.assert_allclose(da[:, cols], dd[:, cols], rtol=1e-5, atol=1e-7 * np.abs(dd).max())
    inactive = np.setdiff1d(np.arange(da.shape[1]), cols)
    assert not da[:, inactive].any()   # never written


def _row_results(pot, layout, ws, x_groups, dx_groups, want_dx=True):
    """Row energies and dE/dAEV of one MLP call on the workspace's AEV rows,
    into buffers filled with a marker."""
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr, _ptr

    e_rows = torch.full_like(ws.e_rows, 7.0)
    dx = torch.full_like(ws.dx, 7.0)
    words = max(len(x_groups) if x_groups is not None else 0, len(dx_groups) if dx_groups is not None else 0)
    call("fennol_mlp_energy_grad_groups", pot.precision, layout.rows, layout.ntiles,
         layout.t_tile_species.data_ptr(), layout.t_tile_row.data_ptr(), C_ptr(pot.mlp.struct), ws.x.data_ptr(),
         _ptr(ws.x_lo), None if x_groups is None else x_groups.ctypes.data,
         None if dx_groups is None else dx_groups.ctypes.data, words, e_rows.data_ptr(),
         dx.data_ptr() if want_dx else None, ws.mlp_ws.data_ptr(), ws.mlp_ws.numel(),
         torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    if pot.precision != 0:
        assert _err_word(pot) == 0
    return e_rows.cpu().numpy(), dx.cpu().numpy()


def _columns(groups):
    return np.array([c for g in range(64 * len(groups)) if (int(groups[g // 64]) >> (g % 64)) & 1
                     for c in range(16 * g, 16 * g + 16)])


@pytest.mark.parametrize("precision", ["fp32", "bf16", "bf16x2", "f16x3x1", "f16x3x2", "bf16x3"])
@pytest.mark.parametrize("molecules", [False, True])
def test_column_groups_match_dense(cuda_device, precision, molecules):
    """The column groups of a species set, the energies-only call and odd sets
    of wanted columns give the dense call's values bit for bit: the columns
    left out are zero in every row, and the order of the other products is the
    same.  The fused forms leave columns that are not wanted as they were."""
    pot = ANIPotential(precision=precision, device=cuda_device, seed=0, n_models=2)
    if molecules:
        mols = molecule_batch(5, seed=11)
        xyz, sp = np.concatenate([m.coordinates for m in mols]), np.concatenate([m.species for m in mols])
        pot.energy_and_forces(xyz, sp, [m.natoms for m in mols])
    else:
        s = water_box(4, seed=2)
        pot.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    layout, g, ws = next(iter(pot._cache.values()))
    groups = pot.active_groups(layout.species_mask)
    ws.x[:, pot.aev_cfg.aev_length:] = 0
    e, dx = _row_results(pot, layout, ws, None, None)
    odd = groups.copy()
    odd[0] &= np.uint64(0xF7FF_FFFF_FBFF_FFFB)  # leaves some out: runs of every length
    for want in (groups, odd):
        e2, dx2 = _row_results(pot, layout, ws, groups, want)
        assert np.array_equal(e2, e)
        cols = _columns(want)
        assert np.array_equal(dx2[:, cols], dx[:, cols])
        if precision not in ("fp32", "bf16x3"):
            assert (dx2[:, np.setdiff1d(np.arange(dx.shape[1]), cols)] == 7.0).all()
    e3, dx3 = _row_results(pot, layout, ws, groups, None, want_dx=False)
    assert np.array_equal(e3, e) and (dx3 == 7.0).all()


@pytest.mark.parametrize("n_side,n_models", [(4, 3), (9, 8), (19, 2), (21, 3)])
def test_shared_tiles_are_the_mean_of_the_models(cuda_device, n_side, n_models):
    """Ensembles whose (tile, model) items the CTAs share out inside tiles
    (fewer items than SMs, some per CTA, many per CTA with a ragged end): the
    row energies and dE/dAEV are the mean of the single-model results.
    float32 sums of at most eight models: 8 half-ulps of the largest term."""
    W = init_weights(CFG, MCFG, seed=3, n_models=n_models)
    s = water_box(n_side, seed=n_side)
    pot = ANIPotential(precision="f16x3x1", device=cuda_device, weights=W)
    pot.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    layout, g, ws = next(iter(pot._cache.values()))
    groups = pot.active_groups(layout.species_mask)
    e, dx = _row_results(pot, layout, ws, groups, groups)
    cols = _columns(groups)
    es, ds = [], []
    for m in range(n_models):
        one = ANIPotential(precision="f16x3x1", device=cuda_device, weights=[W[m]])
        one.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
        lay1, _, ws1 = next(iter(one._cache.values()))
        e1, d1 = _row_results(one, lay1, ws1, groups, groups)
        es.append(e1.astype(np.float64))
        ds.append(d1[:, cols].astype(np.float64))
    used = np.concatenate([np.arange(r, r + 128) for r in layout.t_tile_row.cpu().numpy()])
    tol = 8 * 2.0 ** -24
    em, dm = np.mean(es, 0)[used], np.mean(ds, 0)[used]
    assert np.abs(e[used] - em).max() <= tol * np.abs(es).max()
    assert np.abs(dx[used][:, cols] - dm).max() <= tol * np.abs(ds).max()


@pytest.mark.parametrize("groups", [False, True])
def test_fp32_form_takes_buffers_off_16_bytes(cuda_device, groups):
    """The FP32 form reads four floats at a time only where every array is
    16-byte aligned; on rows and gradients that start one float further on it
    gives the same bits."""
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr

    pot = ANIPotential(precision="fp32", device=cuda_device, seed=0, n_models=3)
    s = water_box(4, seed=2)
    pot.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    layout, g, ws = next(iter(pot._cache.values()))
    words = pot.active_groups(layout.species_mask)
    got = []
    for off in (0, 1):
        x = torch.zeros(ws.x.numel() + 1, device=cuda_device)
        x[off:off + ws.x.numel()] = ws.x.flatten()
        dx = torch.zeros(ws.x.numel() + 1, device=cuda_device)
        e_rows = torch.zeros_like(ws.e_rows)
        call("fennol_mlp_energy_grad_groups", pot.precision, layout.rows, layout.ntiles,
             layout.t_tile_species.data_ptr(), layout.t_tile_row.data_ptr(), C_ptr(pot.mlp.struct),
             x.data_ptr() + 4 * off, None, words.ctypes.data if groups else None,
             words.ctypes.data if groups else None, len(words), e_rows.data_ptr(), dx.data_ptr() + 4 * off,
             ws.mlp_ws.data_ptr(), ws.mlp_ws.numel(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got.append((e_rows.cpu().numpy(), dx[off:off + ws.x.numel()].cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("atoms,models", [(1, 1), (129, 1), (700, 3)])
def test_fp32_half_tiles_match_whole(cuda_device, atoms, models):
    """The FP32 form in half tiles (few row tiles) gives what whole tiles give (the
    same rows repeated until the blocks are many): every element is the same
    chain of FMAs, so the same bits."""
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr

    pot = ANIPotential(precision="fp32", device=cuda_device, seed=4, n_models=models)
    d0, F = pot.mlp.dims[0], pot.aev_cfg.aev_length
    tiles = -(-atoms // 128)
    gen = torch.Generator(device=cuda_device).manual_seed(atoms)
    x1 = torch.zeros((tiles * 128, d0), device=cuda_device)
    x1[:atoms, :F] = torch.rand((atoms, F), generator=gen, device=cuda_device)
    got = []
    for copies in (1, -(-600 // tiles)):
        n = tiles * copies
        x = x1.repeat(copies, 1).contiguous()
        sp = torch.zeros(n, dtype=torch.int32, device=cuda_device)
        row = torch.arange(n, dtype=torch.int32, device=cuda_device) * 128
        e, dx = torch.zeros(n * 128, device=cuda_device), torch.zeros_like(x)
        from fennol_b200 import _lib
        ws = torch.zeros(int(_lib.load().fennol_mlp_workspace_bytes(pot.precision, n * 128, models, C_ptr(pot.mlp.struct))),
                         dtype=torch.uint8, device=cuda_device)
        call("fennol_mlp_energy_grad_groups", pot.precision, n * 128, n, sp.data_ptr(), row.data_ptr(),
             C_ptr(pot.mlp.struct), x.data_ptr(), None, None, None, 0, e.data_ptr(), dx.data_ptr(), ws.data_ptr(),
             ws.numel(), torch.cuda.current_stream().cuda_stream)
        got.append((e[:atoms].cpu().numpy(), dx[:atoms].cpu().numpy()))
    for a, b in zip(*got):
        assert np.abs(a).max() > 0
        np.testing.assert_array_equal(a, b)


def _tile_batch(pot, tiles, columns, seed, species=None):
    """AEV rows of ``tiles`` full row tiles, random in the given columns and zero
    elsewhere, in the form's operand layout; the tiles' species and first rows."""
    dev, d0 = pot.device, pot.mlp.dims[0]
    gen = torch.Generator(device=dev).manual_seed(seed)
    x = torch.zeros((tiles * 128, d0), device=dev)
    x[:, columns] = torch.rand((tiles * 128, len(columns)), generator=gen, device=dev)
    half = torch.float16 if pot.precision_name.startswith("f16") else torch.bfloat16
    hi = x.to(half)
    lo = (x - hi.float()).to(half)
    if species is None:
        species = pot.mlp.n_species
    sp = torch.arange(tiles, dtype=torch.int32, device=dev) % species
    return hi, lo, sp, torch.arange(tiles, dtype=torch.int32, device=dev) * 128


def _tile_results(pot, batch, ws, x_groups=None, dx_groups=None):
    """Row energies and dE/dAEV of a ``_tile_batch``, into buffers filled with a marker."""
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr

    hi, lo, sp, row = batch
    n = sp.numel()
    e = torch.full((n * 128,), 7.0, device=pot.device)
    dx = torch.full(hi.shape, 7.0, device=pot.device)
    words = 0 if x_groups is None and dx_groups is None else pot.mlp.dims[0] // 1024
    call("fennol_mlp_energy_grad_groups", pot.precision, n * 128, n, sp.data_ptr(), row.data_ptr(),
         C_ptr(pot.mlp.struct), hi.data_ptr(), lo.data_ptr(), None if x_groups is None else x_groups.ctypes.data,
         None if dx_groups is None else dx_groups.ctypes.data, words, e.data_ptr(), dx.data_ptr(), ws.data_ptr(),
         ws.numel(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(ws[:4].view(torch.int32)[0]) == 0  # no wait ran out
    return e, dx


def _tile_workspace(pot, tiles):
    from fennol_b200 import _lib
    from fennol_b200.potential import C_ptr

    nb = _lib.load().fennol_mlp_workspace_bytes(pot.precision, tiles * 128, pot.mlp.n_models, C_ptr(pot.mlp.struct))
    return torch.zeros(int(nb), dtype=torch.uint8, device=pot.device)


@pytest.mark.parametrize("precision,wanted,models", [("f16x3x1", 64, 1), ("bf16", 64, 3), ("f16x3x2", 24, 1),
                                                     ("bf16x2", 9, 2)])
def test_short_first_layer_behind_many_dx_runs(cuda_device, precision, wanted, models):
    """A first layer of one column group right behind the 2 to 8 dX runs of the
    item before: its accumulator is announced on the barrier of the run before
    the last, which every epilogue warp must have taken by then.  Same bits as
    with every input column (the others are zero)."""
    pot = ANIPotential(precision=precision, device=cuda_device, seed=2, n_models=models)
    tiles = 3 * torch.cuda.get_device_properties(cuda_device).multi_processor_count + 80
    batch = _tile_batch(pot, tiles, np.arange(16), seed=wanted)
    ws = _tile_workspace(pot, tiles)
    one = np.array([1], np.uint64)
    want = np.array([2 ** wanted - 1], np.uint64)
    e, dx = _tile_results(pot, batch, ws, None, want)
    assert float(dx[:, :16 * wanted].abs().max()) > 0
    for _ in range(20):
        e1, dx1 = _tile_results(pot, batch, ws, one, want)
        assert torch.equal(e1, e) and torch.equal(dx1, dx)


@pytest.mark.parametrize("precision", ["f16x3x1", "bf16x2"])
@pytest.mark.parametrize("extra,models", [(1, 8), (2, 2), (2, 5), (18, 8), (19, 8), (72, 2), (74, 2), (149, 3)])
def test_join_adds_only_what_the_tile_has(cuda_device, precision, extra, models):
    """Tiles beyond a whole number per CTA, seven species and every column of dX
    wanted: shared tiles with fewer items than CTAs (most of them have none of
    the tile), as many, and more.  The scratch holds a marker before the call.
    dE/dAEV and the energies are the mean of the single-model results: float32
    sums of at most eight terms, 8 half-ulps of the largest one."""
    W = init_weights(CFG, MCFG, seed=3, n_models=models)
    if precision == "bf16x2":
        W = round_weights_bf16(W)
    pot = ANIPotential(precision=precision, device=cuda_device, weights=W)
    tiles = torch.cuda.get_device_properties(cuda_device).multi_processor_count + extra
    batch = _tile_batch(pot, tiles, np.arange(CFG.aev_length), seed=extra)
    ws = _tile_workspace(pot, tiles)
    ws[256:] = 0x7F  # 3.4e38 as float32
    e, dx = _tile_results(pot, batch, ws)
    es, ds, em, dm = 0.0, 0.0, 0.0, 0.0
    for m in range(models):
        one = ANIPotential(precision=precision, device=cuda_device, weights=[W[m]])
        e1, d1 = _tile_results(one, batch, _tile_workspace(one, tiles))
        es, ds = max(es, float(e1.abs().max())), max(ds, float(d1.abs().max()))
        em, dm = em + e1.double() / models, dm + d1.double() / models
    tol = 8 * 2.0 ** -24
    assert ds > 0
    assert float((e.double() - em).abs().max()) <= tol * es
    assert float((dx.double() - dm).abs().max()) <= tol * ds


@pytest.mark.parametrize("field", ["b32", "w32"])
def test_fused_form_refuses_biases_off_16_bytes(cuda_device, field):
    """The fused kernel copies biases and the last kernel in bulk, which needs
    16-byte aligned addresses: others are refused before anything is launched."""
    import ctypes

    from fennol_b200 import _lib

    pot = ANIPotential(precision="f16x3x1", device=cuda_device, seed=0)
    batch, ws = _tile_batch(pot, 1, np.arange(16), seed=1, species=1), _tile_workspace(pot, 1)
    _tile_results(pot, batch, ws)
    good = _lib.MLPWeights.from_buffer_copy(pot.mlp.struct)
    for l in ([0, 1, 2] if field == "b32" else [3]):
        getattr(pot.mlp.struct, field)[l] += 4
        with pytest.raises(_lib.FennolError):
            _tile_results(pot, batch, ws)
        ctypes.memmove(ctypes.byref(pot.mlp.struct), ctypes.byref(good), ctypes.sizeof(good))
    _tile_results(pot, batch, ws)


@pytest.mark.parametrize("precision,models", [("fp32", 1), ("fp32", 8), ("f16x3x1", 1), ("f16x3x1", 8), ("bf16x2", 3),
                                              ("bf16x3", 2)])
@pytest.mark.parametrize("molecules,n_side", [(0, 4), (0, 12), (30, 0), (0, 24)])
def test_launch_count_is_what_a_call_launches(cuda_device, precision, models, molecules, n_side):
    """The kernels of one call (the nodes of a graph it is captured in) are the ones
    that mlp_launches counts: one or several models per launch, dX by model and
    its sum, shared tiles and none, with and without forces."""
    import ctypes

    pot = ANIPotential(precision=precision, device=cuda_device, seed=0, n_models=models)
    if molecules:
        mols = molecule_batch(molecules, seed=8)
        xyz, sp = np.concatenate([m.coordinates for m in mols]), np.concatenate([m.species for m in mols])
        pot.energy_and_forces(xyz, sp, [m.natoms for m in mols])
    else:
        s = water_box(n_side, seed=1)
        pot.energy_and_forces(s.coordinates, s.species, [s.natoms], s.cell[None])
    layout, g, ws = next(iter(pot._cache.values()))
    groups = pot.active_groups(layout.species_mask)
    from fennol_b200._lib import call
    from fennol_b200.potential import C_ptr, _ptr

    for want in (True, False):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            call("fennol_mlp_energy_grad_groups", pot.precision, layout.rows, layout.ntiles,
                 layout.t_tile_species.data_ptr(), layout.t_tile_row.data_ptr(), C_ptr(pot.mlp.struct),
                 ws.x.data_ptr(), _ptr(ws.x_lo), groups.ctypes.data, groups.ctypes.data, groups.size,
                 ws.e_rows.data_ptr(), ws.dx.data_ptr() if want else None, ws.mlp_ws.data_ptr(), ws.mlp_ws.numel(),
                 torch.cuda.current_stream().cuda_stream)
        nodes = ctypes.c_size_t()
        rc = ctypes.CDLL("libcudart.so.12").cudaGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None,
                                                              ctypes.byref(nodes))
        assert rc == 0
        assert nodes.value == pot.mlp_launches(layout.ntiles, layout.rows, layout.species_mask, want)
