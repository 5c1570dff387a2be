"""Normals of zeros (no surface) beside concentrations from 1e-3 down through the
squares that FP32 holds as subnormals or not at all (softplus of raw outputs from
-8 to -110): the product with the cosine lobe leaves each lobe's mean as it is and
uniform (the product's concentration is below 1e-3), with a weight factor that all
lobes share, so the pdf is 1 / (4 pi) to a few roundings, in every kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNIFORM = 1 / (4 * np.pi)


@pytest.mark.parametrize("K", [4, 7, 8, 16])
def test_mixture_kernels(nmg, K):
    import torch
    n = 4096
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    raw = torch.randn(n, (4 * K + 3) // 4 * 4, generator=g, device="cuda")
    raw[:, 1:4 * K:4] = -8 - 102 * torch.rand(n, K, generator=g, device="cuda")
    wi = torch.randn(n, 3, generator=g, device="cuda")
    wi = wi / wi.norm(dim=1, keepdim=True)
    zero = torch.zeros(n, 3, device="cuda")
    p = nmg.mixture_pdf(raw, wi, K, zero, kappa_softplus=True)
    d, q, _ = nmg.mixture_sample(raw, torch.rand(n, 4, generator=g, device="cuda"), K, zero, kappa_softplus=True)
    assert bool(torch.isfinite(d).all())
    assert float((p / UNIFORM - 1).abs().max()) <= 1e-5
    assert float((q / UNIFORM - 1).abs().max()) <= 1e-5


NETS = [((0, 1, 8), (0, 4, 7, 8, 9, 12)), ((1, 1, 8), (0, 4, 7, 8, 9, 12)), ((1, 2, 16), (0, 4, 7, 8)), ((1, 0, 16), (0,))]


@pytest.mark.parametrize("preset,path,lobes,tiling", [net + (t,) for net, tilings in NETS for t in tilings])
def test_queries(nmg, preset, path, lobes, tiling):
    import torch
    n = 20000
    f = nmg.GuidingField(nmg.config(preset, path=path, n_lobes=lobes, kappa_softplus=1), max_queries=n, max_batch=0)
    try:
        if tiling:
            f.set_query_tiling(tiling)
        g = torch.Generator(device="cuda")
        g.manual_seed(4)
        p = f.get_params(0)
        n_mlp, out = int(f.info.n_mlp_params), int(f.info.n_output_padded)
        p[n_mlp:] = 0.4 * torch.rand(p.numel() - n_mlp, generator=g, device="cuda") - 0.2
        a = [torch.rand(n, 3, generator=g, device="cuda"), torch.randn(n, 3, generator=g, device="cuda"),
             torch.zeros(n, 3, device="cuda"), torch.rand(n, generator=g, device="cuda"),
             torch.rand(n, 4, generator=g, device="cuda")]
        wi = torch.randn(n, 3, generator=g, device="cuda")
        wi = wi / wi.norm(dim=1, keepdim=True)
        last = p[n_mlp - out * 64:n_mlp].view(out, 64)   # hidden activations are >= 0: a raw output as negative
        last[1:4 * lobes:4] = -torch.rand(lobes, 64, generator=g, device="cuda")
        f.set_params(p)
        kappa = f.query(*a, want_raw=True)["raw"][:, 1:4 * lobes:4]
        last[1:4 * lobes:4] *= -60.0 / float(kappa.mean())
        f.set_params(p)
        o = f.query(*a, want_raw=True)
        kappa = o["raw"][:, 1:4 * lobes:4]
        low = kappa.max(dim=1).values < -8               # every product below 1e-3
        assert float(low.float().mean()) > 0.5 and bool(((kappa > -53) & (kappa < -43)).any())
        pdf = f.pdf(*a[:4], wi)
        f.check_errors()
        for v in (o["pdf"], pdf):
            assert float((v[low] / UNIFORM - 1).abs().max()) <= 1e-5
        assert bool(torch.isfinite(o["dir"][low]).all())
    finally:
        f.close()
