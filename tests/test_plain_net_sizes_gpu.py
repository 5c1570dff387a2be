"""The plain FP32 network at the footprints that decide the backward kernel's
buffers: the accepted maximum (128 encoded columns, seven hidden layers, 80
outputs), and configurations just above and just below the limit of the
two-buffer form.

One tile and a partial one: raw outputs and the parameter gradient against the
FP64 oracle with the bounds of test_field_gpu (1e-4 max(1, |y|); 1e-3 of the
largest |g| of a block), then a training step, its gradient against the FP64
network adjoint of the FP64 loss adjoint at the kernel's own raw outputs,
test_field_gpu's 2e-3.

Several tiles per block (two blocks of 152 SMs, tiles of 64 rows), where the one
grid-gradient buffer is written and read again: the gradient of all rows against
the sum of the gradients of parts with one tile per block. A row's forward pass
has the same bits in both, so the same units are off and only the order of the
FP32 sums differs: at most 38,977 x 8 terms in an entry, 2^-24 sqrt(3e5) = 3.3e-5
of a partial sum no larger than a few times the largest |g|: 1e-4 of it. (The
oracle is no yardstick there: among 17 million hidden units some lie within FP32
rounding of zero, and one that is on in one and off in the other is 1e-3 of the
gradient.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HASH = dict(grid_hash=1, grid_log2_hashmap=9, grid_base_resolution=4, grid_per_level_scale=1.5)
CASES = [
    # feats, levels, mode, sh, bins, hidden, lobes, selection: bytes of the two-buffer form (limit 232,448)
    (8, 15, 1, 1, 1, 7, 16, 1),   # 259,584, 128 encoded columns
    (4, 24, 1, 2, 8, 7, 16, 1),   # 235,008
    (8, 15, 0, 1, 1, 7, 8, 0),    # 239,104
    (8, 15, 0, 1, 1, 6, 16, 1),   # 243,200
    (8, 13, 1, 1, 1, 7, 16, 0),   # 235,008
    (4, 24, 1, 2, 8, 7, 16, 0),   # 222,720: two buffers
]


def make(nmg, torch, case, n):
    feats, levels, mode, sh, bins, hidden, lobes, sel = case
    cfg = nmg.config(nmg.PRESET_HASHGRID, path=nmg.PATH_FP32, grid_features=feats, grid_levels=levels, input_mode=mode,
                     sh_degree=sh, oneblob_bins=bins, hidden_layers=hidden, n_lobes=lobes, selection=sel, **HASH)
    f = nmg.GuidingField(cfg, max_queries=n, max_batch=n)
    rng = np.random.default_rng(19)
    x = rng.random((n, f.info.n_input)).astype(np.float32)
    draw = rng.standard_normal((n, f.info.n_output_padded)).astype(np.float32)
    p = f.get_params(0)
    p[int(f.info.n_mlp_params):] = torch.from_numpy(
        rng.uniform(-0.3, 0.3, int(f.info.n_grid_params)).astype(np.float32)).cuda()
    f.set_params(p)
    offs, w_in = [0], int(f.info.n_encoded_padded)
    for _ in range(hidden):
        offs.append(offs[-1] + 64 * w_in)
        w_in = 64
    offs += [offs[-1] + int(f.info.n_output_padded) * 64, f.n_params]
    return f, rng, x, draw, p.cpu().numpy(), list(zip(offs[:-1], offs[1:]))


def close(g, want, blocks, tol):
    for a, b in blocks:
        assert np.abs(g[a:b] - want[a:b]).max() <= tol * np.abs(want[a:b]).max(), (a, b)


IDS = dict(ids=lambda c: "F%dL%dh%dK%ds%d" % (c[0], c[1], c[5], c[6], c[7]))


@pytest.mark.parametrize("n", [64, 129])
@pytest.mark.parametrize("case", CASES, **IDS)
def test_vjp_and_train_step(nmg, oracle, case, n):
    import torch
    lobes, sel = case[6], case[7]
    f, rng, x, draw, params, blocks = make(nmg, torch, case, n)
    try:
        net = oracle.make_net(**nmg.oracle_net_spec(f.cfg))
        xd = torch.from_numpy(x).cuda()
        raw, grad = f.vjp(xd, torch.from_numpy(draw).cuda())
        raw64 = oracle.network_forward(net, params, x)
        got = raw.cpu().numpy()
        assert np.abs(got - raw64).max() < 1e-4 * max(1.0, np.abs(raw64).max())
        close(grad.cpu().numpy(), oracle.network_backward(net, params, x, draw), blocks, 1e-3)
        rec = np.zeros((n, f.info.record_floats), np.float32)
        rec[:, 0] = rng.uniform(0.0, np.pi, n)
        rec[:, 1] = rng.uniform(0.0, 2 * np.pi, n)
        rec[:, 2:6] = rng.uniform(0.05, 1.0, (n, 4))
        if sel:
            rec[:, 6] = rng.uniform(0.05, 1.0, n)
        f.train_step(xd, torch.from_numpy(rec).cuda())
        d64 = oracle.mixture_loss_grad(got, lobes, rec, 128.0, selection=bool(sel), fp64=True)[0]
        close(f.get_gradients().cpu().numpy(), oracle.network_backward(net, params, x, d64), blocks, 2e-3)
        assert f.step == 1
    finally:
        f.close()


@pytest.mark.parametrize("case", CASES, **IDS)
def test_several_tiles_per_block(nmg, case):
    import torch
    part = 152 * 2 * 64
    n = 2 * part + 65
    f, _, x, draw, _, blocks = make(nmg, torch, case, n)
    try:
        xd, dd = torch.from_numpy(x).cuda(), torch.from_numpy(draw).cuda()
        raw, grad = f.vjp(xd, dd)
        want = torch.zeros(f.n_params, device="cuda", dtype=torch.float64)
        for q in range(0, n, part):
            r, g = f.vjp(xd[q:q + part].contiguous(), dd[q:q + part].contiguous())
            assert torch.equal(r, raw[q:q + part])
            want += g
        close(grad.cpu().numpy(), want.cpu().numpy(), blocks, 1e-4)
    finally:
        f.close()
