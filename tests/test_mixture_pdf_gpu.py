"""The pdf with the cosine lobe and of the odd lobe count (one thread per query)
at one query, partial blocks and one more than a wave of resident blocks, with
lobes that are nearly uniform, that are concentrated at the direction asked for,
and that cancel the cosine lobe (their product is uniform).

Against the FP64 oracle with the bounds of test_mixture_gpu: relative 1e-4 +
4e-7 kappa where the density is above 1e-20, absolute 1e-20 below."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def logit(t):
    return np.log(t / (1 - t))


@pytest.mark.parametrize("n", [1, 127, 129, 152 * 8 * 128 + 1])
@pytest.mark.parametrize("K,cosine", [(7, False), (4, True), (7, True), (8, True), (16, True)])
def test_pdf_one_thread_per_query(nmg, oracle, synth, K, cosine, n):
    import torch
    raw, _, _ = synth.mixture_batch(n, K, seed=33)
    rng = np.random.default_rng(34)
    wi = synth.uniform_sphere(rng, (n,)).astype(np.float32)
    normal = synth.uniform_sphere(rng, (n,)).astype(np.float32) * rng.uniform(0.1, 10, (n, 1)).astype(np.float32)

    def aim(rows, lobe, d):
        th, ph = np.arccos(np.clip(d[:, 2], -1, 1)), np.arctan2(d[:, 1], d[:, 0]) % (2 * np.pi)
        raw[rows, 4 * lobe + 2] = logit(np.clip(th / np.pi, 1e-6, 1 - 1e-6))
        raw[rows, 4 * lobe + 3] = logit(np.clip(ph / (2 * np.pi), 1e-6, 1 - 1e-6))
    raw[0::4, 1] = -9.5                               # kappa 7.5e-5
    aim(slice(1, None, 4), 1, wi[1::4].astype(np.float64))  # a mean at wi
    u = normal / np.linalg.norm(normal, axis=1, keepdims=True)
    raw[2::4, 4 * (K - 1) + 1] = np.log(2.18853)      # kappa and mean of the cosine lobe's opposite
    aim(slice(2, None, 4), K - 1, -u[2::4].astype(np.float64))
    c = normal if cosine else None
    p = nmg.mixture_pdf(torch.from_numpy(raw).cuda(), torch.from_numpy(wi).cuda(), K,
                        None if c is None else torch.from_numpy(c).cuda()).cpu().numpy()
    p64 = oracle.mixture_pdf(raw, K, wi, c, fp64=True)
    kap = np.exp(np.clip(raw[:, 1:4 * K:4].astype(np.float64), -10, 15)).max(axis=1) + (2.2 if cosine else 0)
    err, live = np.abs(p - p64), p64 > 1e-20
    assert np.all(err[live] <= (1e-4 + 4e-7 * kap[live]) * p64[live])
    assert np.all(err[~live] <= 1e-20)
