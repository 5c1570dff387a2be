"""The mixture kernels' exponential and reciprocal (the approximate PTX
instructions with subnormals flushed) over the ranges they are used on, against
FP64: lambda and kappa = e^x for x in the clamp's [-10, 15], the logistic of the
selection logit, and beyond the ranges where they saturate.

Bounds. PTX states 2^-22 relative for ex2.approx.ftz and 1 ulp (2^-23) for
rcp.approx.ftz. e^x = 2^(x log2 e): the product's rounding and the constant's add
|x| log2(e) (2^-24 + 2^-26) ln 2 = |x| 7.5e-8, so 1.4e-6 at x = 15 and 1.0e-6 at
x = -10.
 * A weight lambda_0 = e^x against three of 1, all uniform but lobe 0, whose
   density at the direction is below e^-1000: pdf = 3 / (3 + e^x) / 4 pi, relative
   error at most that of e^x and a few roundings: 2e-6.
 * A lobe's normaliser, kappa / (2 pi (1 - e^-2kappa)) at its mean: the error of
   kappa, of 1 - e^-x (x >= 0.5: at most e^-0.5 / (1 - e^-0.5) = 1.6 times that of
   the exponential, 3e-7) and a few roundings: 3e-6.
 * The logistic: the exponential's error times e / (1 + e), at most
   |x| 7.5e-8 + 2.4e-7, the sum's and the reciprocal's roundings, 2^-22; 0 from
   x = -89 down, where 1 + e^-x leaves the reciprocal subnormal, 1 from x = 18 up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_weights(nmg):
    import torch
    K, x = 4, np.linspace(-12, 17, 20001).astype(np.float32)  # beyond the clamp on either side
    raw = np.zeros((len(x), 16), np.float32)
    raw[:, 0] = x
    raw[:, 1::4] = -np.inf                     # the clamp's e^-10
    raw[:, 1] = 15.0                           # lobe 0: e^15, its mean at theta = pi / 2, phi = pi
    wi = np.tile(np.float32([1, 0, 0]), (len(x), 1))
    p = nmg.mixture_pdf(torch.from_numpy(raw).cuda(), torch.from_numpy(wi).cuda(), K).cpu().numpy().astype(np.float64)
    k = np.exp(-10.0)
    side = k / (2 * np.pi * -np.expm1(-2 * k)) * np.exp(-2 * k)  # the others at the direction opposite to their mean
    want = 3 * side / (3 + np.exp(np.clip(x.astype(np.float64), -10, 15)))
    assert np.abs(p / want - 1).max() <= 2e-6


@pytest.mark.parametrize("softplus", [False, True])
def test_normaliser(nmg, softplus):
    import torch
    K, x = 4, np.linspace(-10, 15, 20001).astype(np.float32)
    raw = np.zeros((len(x), 16), np.float32)
    raw[:, 1::4] = x[:, None]
    wi = np.tile(np.float32([-1, 0, 0]), (len(x), 1))  # every mean: theta = pi / 2, phi = pi
    p = nmg.mixture_pdf(torch.from_numpy(raw).cuda(), torch.from_numpy(wi).cuda(), K,
                        kappa_softplus=softplus).cpu().numpy().astype(np.float64)
    x64 = x.astype(np.float64)
    k = np.logaddexp(0, x64) if softplus else np.exp(x64)
    k = np.maximum(k, 1e-30)
    want = k / (2 * np.pi * -np.expm1(-2 * k))
    err = np.abs(p / want - 1)
    assert err[k >= 1e-5].max() <= 3e-6, x[err.argmax()]


def test_logistic(nmg):
    import torch
    n = 20000
    f = nmg.GuidingField(nmg.config(1, path=1), max_queries=n)
    try:
        g = torch.Generator(device="cuda")
        g.manual_seed(2)
        p = f.get_params(0)
        n_mlp, width, out = int(f.info.n_mlp_params), 64, int(f.info.n_output_padded)
        p[n_mlp:] = 0.4 * torch.rand(p.numel() - n_mlp, generator=g, device="cuda") - 0.2
        row = n_mlp - out * width + 32 * width           # the selection logit's weights
        w = 120.0 * (torch.rand(width, generator=g, device="cuda") - 0.5)
        a = [torch.rand(n, 3, generator=g, device="cuda") for _ in range(3)]
        r, u4 = torch.rand(n, generator=g, device="cuda"), torch.rand(n, 4, generator=g, device="cuda")
        xs, ss = [], []
        for sign in (1, -1):                             # the network has no biases: the logits change sign
            p[row:row + width] = sign * w
            f.set_params(p)
            o = f.query(a[0], a[1] - 0.5, a[2] - 0.5, r, u4, want_raw=True)
            xs.append(o["raw"][:, 32].cpu().numpy().astype(np.float64))
            ss.append(o["selection"].cpu().numpy().astype(np.float64))
        x, s = np.concatenate(xs), np.concatenate(ss)
        assert x.min() < -20 and x.max() > 20            # the range that is tested
        want = 1 / (1 + np.exp(-x))
        live = x > -85
        assert np.all(np.abs(s - want)[live] <= want[live] * (np.abs(x[live]) * 7.5e-8 + 2.4e-7 + 2.4e-7 + 1.2e-7))
        assert np.all(s[x < -89] == 0) and np.all(s[x > 18] == 1)
    finally:
        f.close()
