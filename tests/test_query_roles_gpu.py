"""The warp-specialised query kernels and the cell records where they can go
wrong: one row, a partial tile, one tile more than the SMs, several tiles per
SM and a remainder; positions outside the box, whose cells have no record, and
grids whose dense levels get 8-corner records, 4-corner records or none.

Against the one-pipeline-per-warpgroup kernel (tiling 4): the raw outputs are
the same bits (same operands, same MMAs), and the mixture the same FP32
operations up to FMA contraction, as in test_fused_gpu (lobes 0.9999, direction
and pdf 1e-5). Raw outputs against the FP64 oracle on the kernels' own 16-bit
parameters: test_fused_gpu's 1% (FP16) and 4% (BF16) of the largest output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NETS = [(1, 1, 8), (1, 2, 16), (0, 1, 8)]  # preset, path, lobes


def perturbed(nmg, torch, cfg, n):
    f = nmg.GuidingField(cfg, max_queries=n, max_batch=0)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    p = f.get_params(0)
    n_mlp = int(f.info.n_mlp_params)
    p[n_mlp:] = 0.4 * torch.rand(p.numel() - n_mlp, generator=g, device="cuda") - 0.2
    f.set_params(p)
    return f


@pytest.mark.parametrize("n", [1, 127, 129, 152 * 128 + 1, 4 * 152 * 128 + 77])
@pytest.mark.parametrize("net", NETS, ids=["hash", "hash-K16", "reference"])
def test_default_tiling_matches_one_pipeline(nmg, synth, net, n):
    import torch
    preset, path, lobes = net
    f = perturbed(nmg, torch, nmg.config(preset, path=path, n_lobes=lobes), n)
    try:
        q = synth.wavefront(n, seed=21)
        a = [torch.from_numpy(q[k]).cuda() for k in ("pos", "wo", "normal", "rough", "u4")]
        wi = torch.from_numpy(synth.uniform_sphere(np.random.default_rng(3), (n,)).astype(np.float32)).cuda()

        def outputs():
            return {"dir": torch.full((n + 1, 3), 7.0, device="cuda"), "pdf": torch.full((n + 1,), -1.0, device="cuda"),
                    "lobe": torch.full((n + 1,), -5, dtype=torch.int32, device="cuda"),
                    "selection": torch.full((n + 1,), -2.0, device="cuda") if f.cfg.selection else None}
        got = f.query(*a, outputs=outputs())
        raw = f.query(*a, want_raw=True)["raw"]
        p = f.pdf(*a[:4], wi)
        f.set_query_tiling(4)
        want = f.query(*a, outputs=outputs())
        assert torch.equal(raw, f.query(*a, want_raw=True)["raw"])
        pw = f.pdf(*a[:4], wi)
        f.check_errors()
        same = got["lobe"][:n] == want["lobe"][:n]
        assert float(same.float().mean()) >= 0.9999
        assert float((got["dir"][:n] - want["dir"][:n])[same].abs().max()) <= 1e-5
        assert float(((got["pdf"][:n] - want["pdf"][:n]).abs() / want["pdf"][:n])[same].max()) <= 1e-5
        assert float(((p - pw).abs() / pw).max()) <= 1e-5
        if f.cfg.selection:
            assert torch.equal(got["selection"], want["selection"])
        assert bool((got["dir"][n] == 7).all()) and float(got["pdf"][n]) == -1 and int(got["lobe"][n]) == -5
    finally:
        f.close()


GRIDS = [
    (1, dict()),
    (1, dict(grid_log2_hashmap=10, grid_base_resolution=5)),                               # one dense level
    (1, dict(grid_base_resolution=20, grid_per_level_scale=1.2)),                          # the records' limit
    (1, dict(grid_hash=0, grid_base_resolution=4, grid_per_level_scale=1.3)),              # all dense
    (0, dict()),
    (0, dict(grid_base_resolution=16, grid_per_level_scale=1.1)),
]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "-".join([str(g[0])] + ["%s%s" % (k[5:9], v) for k, v in g[1].items()]))
@pytest.mark.parametrize("path", [1, 2], ids=["bf16", "fp16"])
def test_cell_records_and_positions_outside(nmg, oracle, grid, path):
    import torch
    preset, over = grid
    n = 3001
    cfg = nmg.config(preset, path=path, **over)
    f = perturbed(nmg, torch, cfg, n)
    try:
        net = oracle.make_net(**nmg.oracle_net_spec(cfg))
        rng = np.random.default_rng(8)
        x = rng.random((n, f.info.n_input)).astype(np.float32)
        x[::3, :3] = rng.uniform(-0.3, 1.3, (len(x[::3]), 3))       # some outside the box, on either side
        x[1::7, :3] = rng.integers(0, 2, (len(x[1::7]), 3))         # corners of the box
        raw = f.infer_raw(torch.from_numpy(x).cuda(), which=1).cpu().numpy()
        f.check_errors()
        raw64 = oracle.network_forward(net, f.operand_params(1).cpu().numpy(), x)
        err = np.abs(raw - raw64)
        assert err.max() <= (1e-2 if path == 2 else 4e-2) * np.abs(raw64).max()
    finally:
        f.close()
