"""The one-thread-per-query pdf at concentrations whose normaliser times lambda
leaves FP32's range (softplus of a raw output above 1e30), which it leaves to the
form that keeps the lobes, and just below.

Without the cosine lobe, odd K: against FP64 at directions away from
the extreme lobe's mean, whose density is 0 there while its lambda counts, with
test_mixture_gpu's bound for the other lobes (kappa of at most 7.4: 1e-4). With
it: the product's squared length overflows, and the lobe falls back to a uniform
one that outweighs the others: 1 / (4 pi) to a few roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KAPPA = [1e20, 0.9e30, 1.1e30, 6e32, 1e35, 3e38]


def rows(K, lam, n):
    rng = np.random.default_rng(41)
    raw = rng.standard_normal((n, (4 * K + 3) // 4 * 4)).astype(np.float32)
    at = np.arange(n) % K
    i = np.arange(n)
    raw[i, 4 * at] = lam
    raw[i, 4 * at + 1] = np.float32(KAPPA)[i % len(KAPPA)]
    raw[i, 4 * at + 2] = raw[i, 4 * at + 3] = 0.0  # mean (-1, 0, 0)
    wi = rng.standard_normal((n, 3)).astype(np.float32)
    wi[:, 0] = np.abs(wi[:, 0])
    return raw, wi / np.linalg.norm(wi, axis=1, keepdims=True)


@pytest.mark.parametrize("lam", [-10.0, 0.0, 15.0])
def test_odd_lobes(nmg, lam):
    import torch
    K = 7
    raw, wi = rows(K, lam, 600)
    p = nmg.mixture_pdf(torch.from_numpy(raw).cuda(), torch.from_numpy(wi).cuda(), K, kappa_softplus=True).cpu().numpy()
    r = raw[:, :4 * K].astype(np.float64).reshape(-1, K, 4)
    lm, kp = np.exp(np.clip(r[..., 0], -10, 15)), np.logaddexp(0, r[..., 1])
    th, ph = np.pi / (1 + np.exp(-r[..., 2])), 2 * np.pi / (1 + np.exp(-r[..., 3]))
    mu = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], -1)
    c = np.minimum(0.0, np.einsum("nki,ni->nk", mu, wi.astype(np.float64)) - 1)
    vmf = np.where(kp > 1e10, 0.0, kp / (2 * np.pi * -np.expm1(-2 * np.minimum(kp, 700))) * np.exp(np.maximum(kp * c, -700)))
    want = (lm * vmf).sum(1) / lm.sum(1)
    assert np.isfinite(p).all()
    assert np.abs(p / want - 1).max() <= 1e-4


@pytest.mark.parametrize("K", [4, 7, 8, 16])
def test_cosine(nmg, K):
    import torch
    raw, wi = rows(K, -10.0, 600)
    n = torch.tensor([[0.0, 0.6, 0.8]]).repeat(600, 1).cuda()
    p = nmg.mixture_pdf(torch.from_numpy(raw).cuda(), torch.from_numpy(wi).cuda(), K, n,
                        kappa_softplus=True).cpu().numpy()
    assert np.abs(p * (4 * np.pi) - 1).max() <= 1e-5
