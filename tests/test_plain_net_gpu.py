"""The plain FP32 network kernels (forward, backward, weight gradient) against
the FP64 oracle where they can go wrong: every feature width of the grid, the
smallest and largest networks, tiles of 64 rows with 1, 63, 64, 65 and 129 rows,
outputs and gradients that are not 16-byte aligned.

Tolerances, those of test_field_gpu: raw outputs 1e-4 max(1, |y|); parameter
gradient 1e-3 of the largest |g| of its block (each weight matrix, the grid)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HASH = dict(grid_hash=1, grid_log2_hashmap=9, grid_base_resolution=4, grid_per_level_scale=1.5)
CASES = [
    # feats, levels, mode, sh, bins, hidden, lobes, selection, rows
    (1, 16, 1, 4, 4, 3, 8, 1, 65),
    (2, 16, 1, 4, 4, 3, 16, 1, 129),
    (2, 3, 0, 3, 5, 1, 7, 0, 1),
    (4, 8, 0, 2, 4, 3, 8, 0, 63),
    (4, 24, 1, 2, 8, 7, 16, 0, 64),
    (8, 5, 0, 1, 16, 2, 8, 1, 130),
]


def unaligned(torch, n, fill=0.0):
    """n floats at 4 bytes past a 16-byte boundary."""
    return torch.full((n + 1,), fill, device="cuda")[1:]


@pytest.mark.parametrize("aligned", [True, False], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "F%dL%dh%dK%d-%d" % (c[0], c[1], c[5], c[6], c[8]))
def test_forward_and_vjp(nmg, oracle, case, aligned):
    import ctypes as C

    import torch
    feats, levels, mode, sh, bins, hidden, lobes, sel, n = case
    cfg = nmg.config(nmg.PRESET_HASHGRID, path=nmg.PATH_FP32, grid_features=feats, grid_levels=levels, input_mode=mode,
                     sh_degree=sh, oneblob_bins=bins, hidden_layers=hidden, n_lobes=lobes, selection=sel, **HASH)
    f = nmg.GuidingField(cfg, max_queries=n, max_batch=n)
    try:
        net = oracle.make_net(**nmg.oracle_net_spec(cfg))
        rng = np.random.default_rng(11)
        x = rng.random((n, f.info.n_input)).astype(np.float32)
        draw = rng.standard_normal((n, f.info.n_output_padded)).astype(np.float32)
        p = f.get_params(0)
        p[int(f.info.n_mlp_params):] = torch.from_numpy(
            rng.uniform(-0.3, 0.3, int(f.info.n_grid_params)).astype(np.float32)).cuda()
        f.set_params(p)
        params = p.cpu().numpy()
        xd, dd = torch.from_numpy(x).cuda(), torch.from_numpy(draw).cuda()
        if aligned:
            raw = torch.empty(n * f.info.n_output_padded, device="cuda")
            grad = torch.zeros(f.n_params, device="cuda")
        else:
            raw, grad = unaligned(torch, n * f.info.n_output_padded), unaligned(torch, f.n_params)
        P = lambda t: C.c_void_p(t.data_ptr())
        raw.fill_(7.0)
        nmg.check(f.L.nmg_infer_raw(f.h, P(xd), n, 1, P(raw), None))
        raw64 = oracle.network_forward(net, params, x)
        got = raw.view(n, -1).cpu().numpy()
        assert np.abs(got - raw64).max() < 1e-4 * max(1.0, np.abs(raw64).max())
        raw.fill_(7.0)
        nmg.check(f.L.nmg_network_vjp(f.h, P(xd), P(dd), n, P(raw), P(grad), None))
        torch.cuda.synchronize()
        assert np.array_equal(raw.view(n, -1).cpu().numpy(), got)
        g, g64 = grad.cpu().numpy(), oracle.network_backward(net, params, x, draw)
        offs, w_in = [0], net.n_enc_padded
        for _ in range(net.n_hidden):
            offs.append(offs[-1] + net.width * w_in)
            w_in = net.width
        offs += [offs[-1] + net.n_out_padded * net.width, net.n_params]
        for a, b in zip(offs[:-1], offs[1:]):
            assert np.abs(g[a:b] - g64[a:b]).max() <= 1e-3 * np.abs(g64[a:b]).max(), (a, b)
    finally:
        f.close()
