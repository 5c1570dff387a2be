"""Tiling 12 of the 8-lobe networks over the depths: up to four hidden layers the
three-role kernel, from five on the two-role one, but for launches of at most
four tiles per SM and for raw outputs alone: at five layers, and at six of the
hash grid with more than 32 tiles per SM.

Against the one-pipeline-per-warpgroup kernel (tiling 4), the bounds of
test_query_roles_gpu: raw outputs the same bits, lobes 0.9999, direction and pdf
1e-5 (the same FP32 mixture up to FMA contraction)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHARED = 4 * 152 * 128  # rows of the largest launch whose tiles are shared


@pytest.mark.parametrize("n", [129, SHARED, SHARED + 1])
@pytest.mark.parametrize("preset,hidden", [(1, 1), (1, 4), (1, 5), (1, 6), (1, 7), (0, 5), (0, 7)])
def test_deep_networks(nmg, synth, preset, hidden, n):
    import torch
    f = nmg.GuidingField(nmg.config(preset, path=1, hidden_layers=hidden), max_queries=n, max_batch=0)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(9)
        p = f.get_params(0)
        n_mlp = int(f.info.n_mlp_params)
        p[n_mlp:] = 0.4 * torch.rand(p.numel() - n_mlp, generator=g, device="cuda") - 0.2
        f.set_params(p)
        q = synth.wavefront(n, seed=15)
        a = [torch.from_numpy(q[k]).cuda() for k in ("pos", "wo", "normal", "rough", "u4")]
        x = f.featurize(*a[:4])
        wi = torch.from_numpy(synth.uniform_sphere(np.random.default_rng(16), (n,)).astype(np.float32)).cuda()

        def call(tiling):
            f.set_query_tiling(tiling)
            o = f.query(*a, want_raw=True)
            return o, f.query(*a), f.pdf(*a[:4], wi), f.infer_raw(x)
        got, got2, p12, r12 = call(12)
        want, _, p4, r4 = call(4)
        f.check_errors()
        assert torch.equal(got["raw"], want["raw"]) and torch.equal(r12, r4)
        for k in ("dir", "pdf", "lobe"):
            assert torch.equal(got[k], got2[k])
        same = got["lobe"] == want["lobe"]
        assert float(same.float().mean()) >= 0.9999
        assert float((got["dir"] - want["dir"])[same].abs().max()) <= 1e-5
        assert float(((got["pdf"] - want["pdf"]).abs() / want["pdf"])[same].max()) <= 1e-5
        assert float(((p12 - p4).abs() / p4).max()) <= 1e-5
    finally:
        f.close()


@pytest.mark.parametrize("n", [32 * 152 * 128, 32 * 152 * 128 + 1])
def test_raw_outputs_at_six_layers(nmg, n):
    import torch
    f = nmg.GuidingField(nmg.config(1, path=1, hidden_layers=6), max_queries=n, max_batch=0)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(10)
        x = torch.rand(n, int(f.info.n_input), generator=g, device="cuda")
        f.set_query_tiling(12)
        got = f.infer_raw(x)
        f.set_query_tiling(4)
        assert torch.equal(got, f.infer_raw(x))
        f.check_errors()
    finally:
        f.close()
