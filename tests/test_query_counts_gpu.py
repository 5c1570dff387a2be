"""Queries and pdfs whose device count is far below the array's length, so that
most CTAs have no tile: the default kernels of every network at counts of none,
one, a tile's edge, and one tile fewer and more than the SMs. Calls follow one
another without a wait, a full one after each, so that a CTA that left work in
flight would write into its successor's shared memory.

Rows below the count hold the bits of the full call (a row's arithmetic does not
depend on the others), rows from the count on keep what they held."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152
N = (4 * SMS + 3) * 128 + 77
COUNTS = [0, 1, 127, 128, 129, (SMS - 1) * 128, SMS * 128 + 1, N]
NETS = [(0, 1, 8), (0, 2, 8), (1, 1, 8), (1, 2, 16)]  # preset, path, lobes


@pytest.mark.parametrize("net", NETS, ids=["reference-bf16", "reference-fp16", "hash", "hash-K16"])
def test_counts_below_capacity(nmg, synth, net):
    import torch
    preset, path, lobes = net
    f = nmg.GuidingField(nmg.config(preset, path=path, n_lobes=lobes), max_queries=N, max_batch=0)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(7)
        p = f.get_params(0)
        n_mlp = int(f.info.n_mlp_params)
        p[n_mlp:] = 0.4 * torch.rand(p.numel() - n_mlp, generator=g, device="cuda") - 0.2
        f.set_params(p)
        q = synth.wavefront(N, seed=5)
        a = [torch.from_numpy(q[k]).cuda() for k in ("pos", "wo", "normal", "rough", "u4")]
        wi = torch.from_numpy(synth.uniform_sphere(np.random.default_rng(6), (N,)).astype(np.float32)).cuda()

        def outputs():
            o = {"dir": torch.full((N, 3), 7.0, device="cuda"), "pdf": torch.full((N,), -1.0, device="cuda"),
                 "lobe": torch.full((N,), -5, dtype=torch.int32, device="cuda")}
            if f.cfg.selection:
                o["selection"] = torch.full((N,), -2.0, device="cuda")
            return o
        want, want_pdf = f.query(*a, outputs=outputs()), f.pdf(*a[:4], wi)
        counts = [torch.tensor([c], dtype=torch.int32, device="cuda") for c in COUNTS]
        got, full = [], []
        for c in counts:
            got.append(f.query(*a, count=c, outputs=outputs()))
            full.append(f.pdf(*a[:4], wi))
            f.pdf(*a[:4], wi, count=c)
            full.append(f.query(*a, outputs=outputs())["dir"])
        f.check_errors()
        for c, o in zip(COUNTS, got):
            fresh = outputs()
            for k in o:
                assert torch.equal(o[k][:c], want[k][:c]), (c, k)
                assert torch.equal(o[k][c:], fresh[k][c:]), (c, k)
        assert all(torch.equal(p, want_pdf) for p in full[0::2])
        assert all(torch.equal(d, want["dir"]) for d in full[1::2])
    finally:
        f.close()
