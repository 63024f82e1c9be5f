"""Training-loss parameter gradients through the hand-written adjoints
(AEV tangent kernel + explicit network sweep) against second-order autograd
of the FP64 oracle and against finite differences of the FP64 loss."""

import numpy as np
import pytest
import torch

from fennol_b200.params import AEVConfig, MLPConfig, init_weights
from fennol_b200.potential import ANIPotential
from fennol_b200.systems import molecule_batch, water_box
from fennol_b200.training import LossGradient, flatten
from oracle import ani_ref

pytestmark = pytest.mark.gpu
CFG, MCFG = AEVConfig(), MLPConfig()
REL_TOL = 2e-4  # relative L2 error of the whole gradient vector against FP64


def batch(n_mol, seed):
    mols = molecule_batch(n_mol, seed=seed)
    xyz = np.concatenate([m.coordinates for m in mols])
    sp = np.concatenate([m.species for m in mols])
    return xyz, sp, np.array([m.natoms for m in mols])


def teacher_targets(xyz, sp, nat, cells=None):
    teacher = init_weights(CFG, MCFG, seed=77)
    r = ani_ref.energy_and_forces(xyz, sp, nat, teacher, CFG, MCFG, cells=cells)
    return r["energy"], r["forces"]


def rel_err(g, g_ref):
    a, b = flatten(g, CFG.species_order), flatten(g_ref, CFG.species_order)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_gradient_matches_second_order_autograd(cuda_device, dtype):
    xyz, sp, nat = batch(24, seed=41)
    W = init_weights(CFG, MCFG, seed=5, bias_std=0.05)
    e_ref, f_ref = teacher_targets(xyz, sp, nat)
    pot = ANIPotential(precision="fp32", device=cuda_device, weights=W)
    terms, g = LossGradient(pot, w_e=1.0, w_f=10.0, dtype=dtype)(xyz, sp, nat, e_ref, f_ref)
    loss_ref, g_ref = ani_ref.loss_and_grads(xyz, sp, nat, W[0], CFG, MCFG, e_ref, f_ref)
    assert abs(terms.loss - loss_ref) <= 1e-4 * loss_ref
    assert rel_err(g, g_ref) < REL_TOL
    for sym in CFG.species_order:
        for (gw, gb), (rw, rb) in zip(g[sym], g_ref[sym]):
            scale = max(np.abs(rw).max(), 1e-30)
            np.testing.assert_allclose(gw, rw, rtol=0, atol=2e-3 * scale)


def test_force_term_alone_and_energy_term_alone(cuda_device):
    """Each seed path on its own (w_e = 0 exercises the tangent kernel only)."""
    xyz, sp, nat = batch(12, seed=43)
    W = init_weights(CFG, MCFG, seed=6, bias_std=0.05)
    e_ref, f_ref = teacher_targets(xyz, sp, nat)
    pot = ANIPotential(precision="fp32", device=cuda_device, weights=W)
    for w_e, w_f in ((0.0, 1.0), (1.0, 0.0)):
        _, g = LossGradient(pot, w_e=w_e, w_f=w_f)(xyz, sp, nat, e_ref, f_ref)
        _, g_ref = ani_ref.loss_and_grads(xyz, sp, nat, W[0], CFG, MCFG, e_ref, f_ref, w_e=w_e, w_f=w_f)
        assert rel_err(g, g_ref) < REL_TOL, (w_e, w_f)


def test_periodic_box_gradient(cuda_device):
    s = water_box(4, seed=12)
    W = init_weights(CFG, MCFG, seed=8, bias_std=0.05)
    e_ref, f_ref = teacher_targets(s.coordinates, s.species, [s.natoms], s.cell[None])
    pot = ANIPotential(precision="fp32", device=cuda_device, weights=W)
    _, g = LossGradient(pot)(s.coordinates, s.species, [s.natoms], e_ref, f_ref, s.cell[None])
    _, g_ref = ani_ref.loss_and_grads(s.coordinates, s.species, [s.natoms], W[0], CFG, MCFG, e_ref, f_ref,
                                      cells=s.cell[None])
    assert rel_err(g, g_ref) < REL_TOL


def test_gradient_entries_match_finite_differences(cuda_device):
    """Central differences of the FP64 loss, step 1e-4, on one entry of every
    kernel and bias of the hydrogen network."""
    xyz, sp, nat = batch(6, seed=45)
    W = init_weights(CFG, MCFG, seed=9, bias_std=0.05)
    e_ref, f_ref = teacher_targets(xyz, sp, nat)
    pot = ANIPotential(precision="fp32", device=cuda_device, weights=W)
    _, g = LossGradient(pot, dtype=torch.float64)(xyz, sp, nat, e_ref, f_ref)
    graph = ani_ref.Graph(xyz, nat, None, None, CFG.radial_cutoff, CFG.angular_cutoff)
    model = W[0]
    h = 1e-4
    for layer in range(4):
        for which in range(2):
            arr = model["H"][layer][which]
            idx = np.unravel_index(int(np.argmax(np.abs(g["H"][layer][which]))), arr.shape)
            orig = arr[idx]
            arr[idx] = orig + h
            lp = ani_ref.loss_value(xyz, sp, nat, model, CFG, MCFG, e_ref, f_ref, graph=graph)
            arr[idx] = orig - h
            lm = ani_ref.loss_value(xyz, sp, nat, model, CFG, MCFG, e_ref, f_ref, graph=graph)
            arr[idx] = orig
            fd = (lp - lm) / (2 * h)
            got = g["H"][layer][which][idx]
            assert abs(fd - got) <= 1e-3 * abs(fd) + 1e-9, (layer, which, fd, got)


def test_replayed_gradient_equals_direct(cuda_device):
    """From the third call on one batch the pass is one CUDA-graph replay;
    its results must equal the direct evaluation at new positions."""
    xyz, sp, nat = batch(16, seed=47)
    W = init_weights(CFG, MCFG, seed=10, bias_std=0.05)
    e_ref, f_ref = teacher_targets(xyz, sp, nat)
    pot = ANIPotential(precision="fp32", device=cuda_device, weights=W)
    lg = LossGradient(pot)
    rng = np.random.default_rng(3)
    for k in range(4):
        x = xyz + rng.normal(scale=0.02, size=xyz.shape)
        terms, g = lg(x, sp, nat, e_ref, f_ref)
        ref_pot = ANIPotential(precision="fp32", device=cuda_device, weights=W, use_graphs=False)
        t2, g2 = LossGradient(ref_pot, use_graphs=False)(x, sp, nat, e_ref, f_ref)
        assert abs(terms.loss - t2.loss) <= 1e-6 * t2.loss, k
        a, b = flatten(g, CFG.species_order), flatten(g2, CFG.species_order)
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b), k
    assert lg._rec is not None  # the later calls replayed the captured pass


@pytest.mark.parametrize("dims", [(20, 12, 8, 4, 1), (19, 7, 5, 3, 1), (1008, 256, 192, 160, 1)])
@pytest.mark.parametrize("rows", [(1, 0, 2), (130, 1, 65), (0, 400, 63)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_network_sweep_at_odd_sizes(cuda_device, dims, rows, dtype):
    """fennol_net_loss_grad on its own, widths that are and are not multiples
    of four, rows at the edges of the 128-row tiles and of the row slices,
    species without rows: no further from double differentiation in float64
    than four times what the same differentiation in float32 is, in units of
    the type's epsilon (rounding of z is amplified by 1 / alpha^2 in the CELU's
    second derivative, for both alike), plus 64 epsilons of the largest entry."""
    import ctypes
    from fennol_b200 import _lib

    rng = np.random.default_rng(int(sum(dims) + 10 * sum(rows)))
    S, alpha = len(rows), float(np.float32(0.1))  # alpha is passed as a float
    pad, ld = [-(-r // 128) * 128 for r in rows], dims[0] + 3
    row0 = np.concatenate([[0], np.cumsum(pad)])[:S].astype(np.int32)
    total = max(sum(pad), 1)
    x64, t64, c64 = (torch.tensor(rng.standard_normal((total, w))).to(dtype).double() for w in (ld, ld, 1))
    net = _lib.NetTrain()
    net.n_species, net.celu_alpha, net.is_double = S, alpha, int(dtype == torch.float64)
    keep, weights = [], []
    for k in range(5):
        net.dims[k] = dims[k]
    for s in range(S):
        layers = []
        for l in range(4):
            w = torch.tensor(rng.standard_normal((dims[l], dims[l + 1])) * dims[l] ** -0.5).to(dtype)
            b = torch.tensor(rng.standard_normal(dims[l + 1]) * 0.1).to(dtype)
            dev = [v.to(cuda_device) for v in (w, b)] + [torch.full_like(v, 9.0, device=cuda_device) for v in (w, b)]
            net.w[l][s], net.b[l][s], net.gw[l][s], net.gb[l][s] = (v.data_ptr() for v in dev)
            keep.append(dev)
            layers.append((w.double(), b.double()))
        weights.append(layers)
    host_rows = np.array(rows, np.int32)
    lib = _lib.load()
    nb = lib.fennol_net_loss_grad_workspace_bytes(ctypes.byref(net), host_rows.ctypes.data)
    ws = torch.empty(max(int(nb), 256), dtype=torch.uint8, device=cuda_device)
    x, t, c = (v.to(dtype).to(cuda_device).contiguous() for v in (x64, t64, c64))
    _lib.call("fennol_net_loss_grad", ctypes.byref(net), row0.ctypes.data, host_rows.ctypes.data, x.data_ptr(),
              t.data_ptr(), ld, c.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    eps = float(torch.finfo(dtype).eps)
    for s in range(S):
        if rows[s] == 0:
            for l in range(4):  # left alone
                assert (keep[4 * s + l][2] == 9.0).all() and (keep[4 * s + l][3] == 9.0).all()
            continue
        at = slice(int(row0[s]), int(row0[s]) + rows[s])

        def differentiated(kind):
            params = [v.detach().to(kind).requires_grad_(True) for wb in weights[s] for v in wb]
            a = x64[at, :dims[0]].to(kind).requires_grad_(True)
            h = a
            for l in range(4):
                h = h @ params[2 * l] + params[2 * l + 1]
                if l < 3:
                    h = ani_ref.celu(h, alpha)
            (ga,) = torch.autograd.grad(h.sum(), a, create_graph=True)
            loss = (c64[at].to(kind) * h).sum() - (ga * t64[at, :dims[0]].to(kind)).sum()
            return [v.double() for v in torch.autograd.grad(loss, params)]

        ref, plain = differentiated(torch.float64), differentiated(torch.float32)
        for l in range(4):
            for k in range(2):
                r = ref[2 * l + k]
                err = float((keep[4 * s + l][2 + k].double().cpu() - r).abs().max())
                own = float((plain[2 * l + k] - r).abs().max()) * eps / 2.0 ** -23
                assert err <= 4 * own + 64 * eps * max(float(r.abs().max()), 1.0), (s, l, k, err, own)


@pytest.mark.parametrize("natoms", [[1], [255, 1], [7, 250, 512]])
def test_loss_seeds(cuda_device, natoms):
    """fennol_loss_seed against plain float64 formulas (block edges at 256 atoms)."""
    from fennol_b200 import _lib

    rng = np.random.default_rng(len(natoms))
    n, B = sum(natoms), len(natoms)
    e, er = rng.standard_normal(B), rng.standard_normal(B)
    f, fr = rng.standard_normal((n, 3)).astype(np.float32), rng.standard_normal((n, 3))
    sys = np.repeat(np.arange(B), natoms).astype(np.int32)
    row = rng.permutation(n + 5)[:n].astype(np.int32)
    d = [torch.tensor(v, device=cuda_device) for v in (e, er, f, fr, sys, row)]
    du = torch.zeros((n, 4), device=cuda_device)
    c = torch.zeros(n + 5, dtype=torch.float64, device=cuda_device)
    terms = torch.zeros(_lib.STATUS_WORDS + 2, dtype=torch.float64, device=cuda_device)
    status = torch.arange(_lib.STATUS_WORDS, dtype=torch.int32, device=cuda_device)
    ws = torch.zeros(_lib.load().fennol_loss_seed_workspace_bytes(n), dtype=torch.uint8, device=cuda_device)
    _lib.call("fennol_loss_seed", d[0].data_ptr(), d[1].data_ptr(), B, d[2].data_ptr(), d[3].data_ptr(), n,
              d[4].data_ptr(), d[5].data_ptr(), 1.5, 10.0, status.data_ptr(), du.data_ptr(), c.data_ptr(), 1,
              terms.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    df = f.astype(np.float64) - fr
    np.testing.assert_allclose(du.cpu().numpy()[:, :3], 20.0 / (3 * n) * df, rtol=1e-6, atol=1e-9)
    np.testing.assert_allclose(c.cpu().numpy()[row], (3.0 / B * (e - er))[sys], rtol=1e-14)
    got = terms.cpu().numpy()
    assert np.array_equal(got[:_lib.STATUS_WORDS], np.arange(_lib.STATUS_WORDS))
    np.testing.assert_allclose(got[_lib.STATUS_WORDS:], [1.5 * np.mean((e - er) ** 2), 10.0 * np.mean(df ** 2)],
                               rtol=1e-12)
