"""The work that is timed: the guiding step's public calls over the sizes and options a renderer uses.

Kinds of case, each one call of the Python binding (and through it of the C ABI):
  mix_sample, mix_pdf, mix_loss   the mixture kernels on raw network outputs
  query, pdf                      the network-backed query and MIS pdf of one bounce's shading points
  train_step                      one optimiser step on a batch of training records
  train_frame                     one frame's training on its per-pixel radiance records
"""
import importlib
import math

import numpy as np
import torch

nmg = importlib.import_module("neural-mixture-guiding_gb300")

EPS = 1e-5
INV_4PI = 1.0 / (4.0 * math.pi)
COSINE_KAPPA = 2.18853
PATHS = {"fp32": 0, "bf16": 1, "fp16": 2}
PRESETS = {"reference": 0, "hashgrid": 1}


def _field_case(name, kind, preset, path, n, lobes=8):
    return {"name": name, "kind": kind, "preset": preset, "path": path, "lobes": lobes, "n": n}


def listed():
    return [
        # every query of a 2M-point batch sampled from raw outputs the caller's own network produced
        {"name": "mix_sample_2m", "kind": "mix_sample", "lobes": 8, "n": 2097152, "cosine": False, "softplus": False},
        # MIS pdf with the cosine lobe for the odd lobe count, a ragged mid-sized queue
        {"name": "mix_pdf_k7_cosine", "kind": "mix_pdf", "lobes": 7, "n": 300001, "cosine": True, "softplus": False},
        # the loss of a small batch with learned selection: the smallest call, launch-bound
        {"name": "mix_loss_4k", "kind": "mix_loss", "lobes": 8, "n": 4096, "selection": True, "softplus": False},
        # the first bounce of a 1920x1080 frame, hash-grid network
        _field_case("query_1080p", "query", "hashgrid", "bf16", 2073600),
        # a late bounce, when few paths are left
        _field_case("query_late", "query", "hashgrid", "bf16", 4999),
        # a middle bounce with the 16-lobe network on FP16 operands
        _field_case("query_k16_fp16", "query", "hashgrid", "fp16", 900000, 16),
        # MIS pdf of a middle bounce's BSDF-sampled directions, the reference's own network
        _field_case("pdf_reference", "pdf", "reference", "bf16", 550001),
        # the training batch of the benchmark
        _field_case("train_262k", "train_step", "hashgrid", "bf16", 262144),
        # the smallest batch that a frame's training takes by default
        _field_case("train_65k_fp16", "train_step", "hashgrid", "fp16", 65536),
        # one frame's training from its radiance records: every third pixel of 1920x1080, two path vertices each
        {"name": "train_frame", "kind": "train_frame", "preset": "hashgrid", "path": "bf16", "lobes": 8,
         "res_x": 1920, "res_y": 1080, "stride": 3, "depths": 2},
        # the plain FP32 path, which a configuration takes by default: a bounce's queries, and a batch
        _field_case("query_fp32", "query", "reference", "fp32", 524288),
        _field_case("train_fp32", "train_step", "hashgrid", "fp32", 65536),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mix_sample", "mix_pdf", "mix_loss", "query", "query", "pdf", "train_step", "train_step",
                       "train_frame"])
    if kind.startswith("mix_"):
        c = {"kind": kind, "lobes": rng.choice([4, 7, 8, 8, 16]), "n": _log_size(rng, 1000, 2000000),
             "softplus": rng.random() < 0.25}
        if kind == "mix_loss":
            c["selection"] = rng.random() < 0.5
        else:
            c["cosine"] = rng.random() < 0.5
        return c
    if kind == "train_frame":
        # every vertex is kept and the batch takes all of them: the records are a whole number of 128
        stride = rng.choice([2, 3, 4])
        res_x, res_y = 128 * stride * rng.randint(1, 4), stride * rng.randint(64, 270)
        return {"kind": kind, "preset": "hashgrid", "path": rng.choice(["bf16", "bf16", "fp16"]), "lobes": 8,
                "res_x": res_x, "res_y": res_y, "stride": stride, "depths": rng.randint(1, 3)}
    preset, lobes = rng.choice([("hashgrid", 8), ("hashgrid", 8), ("hashgrid", 16), ("reference", 8)])
    path = rng.choice(["bf16", "bf16", "fp16", "fp16", "fp32"])
    if kind == "train_step":
        n = _log_size(rng, 16384, 65536 if path == "fp32" else 524288)
    else:
        n = _log_size(rng, 1000, 300000 if path == "fp32" else 2000000)
    return {"kind": kind, "preset": preset, "path": path, "lobes": lobes, "n": n}


# ------------------------------------------------------------------ inputs
class _Rng:
    """Seeded draws on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) & 0x7FFFFFFF)

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda")

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def sphere(self, *shape):
        v = self.normal(*shape, 3)
        return v / v.norm(dim=-1, keepdim=True)


def _angles(v):
    th = torch.acos(v[..., 2].clamp(-1, 1))
    ph = torch.atan2(v[..., 1], v[..., 0])
    return th, torch.where(ph < 0, ph + 2 * math.pi, ph)


def _logit(p):
    p = p.clamp(1e-6, 1 - 1e-6)
    return torch.log(p / (1 - p))


def _round16(x):
    return (x + 15) // 16 * 16


def _surface_points(r, n):
    """70% of the positions on 64 planes, 30% anywhere in the unit box."""
    p = r.uniform(n, 3)
    pn = r.sphere(64)
    off = (pn * r.uniform(64, 3)).sum(-1)
    k = torch.randint(0, 64, (n,), generator=r.g, device="cuda")
    d = (p * pn[k]).sum(-1) - off[k]
    on = torch.clamp(p - d[:, None] * pn[k], 0, 1)
    return torch.where(r.uniform(n, 1) < 0.7, on, p).contiguous()


def _mixture_inputs(c, seed):
    r, n, K = _Rng(seed), c["n"], c["lobes"]
    sel = bool(c.get("selection"))
    stride = _round16(4 * K + (1 if sel else 0))
    raw = torch.zeros(n, stride, device="cuda")
    lam = r.normal(n, K)
    kap = 10.0 ** (4 * r.uniform(n, K) - 1)  # concentrations over [0.1, 1000]
    th, ph = _angles(r.sphere(n, K))
    raw[:, :4 * K] = torch.stack([lam, torch.log(kap), _logit(th / math.pi), _logit(ph / (2 * math.pi))], -1).view(n, 4 * K)
    if sel:
        raw[:, 4 * K] = r.normal(n)
    s = {"case": c, "raw": raw}
    if c["kind"] == "mix_sample":
        s["u4"] = r.uniform(n, 4)
    elif c["kind"] == "mix_pdf":
        s["wi"] = r.sphere(n).contiguous()
    else:
        wth, wph = _angles(r.sphere(n))
        wpdf = INV_4PI * (0.5 + r.uniform(n))
        L = wpdf * torch.exp(1.5 * r.normal(n))
        cols = [wth, wph, 0.8 * L, L, 1.2 * L, wpdf] + ([torch.full_like(L, INV_4PI)] if sel else [])
        s["records"] = torch.stack(cols, -1).contiguous()
    s["normal"] = r.sphere(n).contiguous() if c.get("cosine") else None
    return s


def _config(c):
    # training at the learning rate 1e-3 and with Adam's usual epsilon
    return nmg.config(PRESETS[c["preset"]], path=PATHS[c["path"]], n_lobes=c["lobes"], learning_rate=1e-3, epsilon=1e-8)


def _params(info, cfg, seed):
    """Weights as in the middle of a render: Xavier-sized matrices and O(0.1) grid entries."""
    r = _Rng(seed + 1)
    n, n_mlp = int(info.n_params), int(info.n_mlp_params)
    p = 0.1 * (2 * r.uniform(n) - 1)
    off = 0
    for i, o in _layer_sizes(info, cfg):
        p[off:off + i * o] = (2 * r.uniform(i * o) - 1) * math.sqrt(6 / (i + o))
        off += i * o
    assert off == n_mlp
    return p


def _layer_sizes(info, cfg):
    w = cfg.width
    return [(info.n_encoded_padded, w)] + [(w, w)] * (cfg.hidden_layers - 1) + [(w, info.n_output_padded)]


def _shading(r, n):
    return {"pos": _surface_points(r, n), "wo": r.sphere(n).contiguous(), "normal": r.sphere(n).contiguous(),
            "rough": r.uniform(n)}


def _radiance(r, n, wi):
    """Radiance that arrives from wi: a lobe around one of 64 lights over a constant, with noise."""
    light = r.sphere(64)[torch.randint(0, 64, (n,), generator=r.g, device="cuda")]
    return (0.05 + torch.exp(20 * ((wi * light).sum(-1) - 1))) * torch.exp(0.5 * r.normal(n))


def _training_rows(r, n, mode, sel):
    """(x, records): network input rows and their guided outputs."""
    pos, wo, nrm, rough = _surface_points(r, n), r.sphere(n), r.sphere(n), r.uniform(n)
    infl = math.sqrt(3) * 0.005
    cols = [0.5 + (pos - 0.5) / (1 + 2 * infl), (wo + 1) * 0.5]
    if mode == 0:
        th, ph = _angles(nrm)
        cols.append(torch.stack([th / math.pi, ph / (2 * math.pi)], -1))
    else:
        cols.append((nrm + 1) * 0.5)
    cols.append((1 - torch.exp(-rough))[:, None])
    wi = r.sphere(n)
    L = _radiance(r, n, wi)
    th, ph = _angles(wi)
    rec = [th, ph, 0.8 * L, L, 1.2 * L, INV_4PI * (0.5 + r.uniform(n))] + ([torch.full_like(L, INV_4PI)] if sel else [])
    return torch.cat(cols, 1).contiguous(), torch.stack(rec, -1).contiguous()


def _frame_records(c, seed):
    """Per-pixel radiance records of a frame, one dict of arrays per path vertex."""
    r, n = _Rng(seed), c["res_x"] * c["res_y"]
    depths = []
    for _ in range(c["depths"]):
        wi = r.sphere(n)
        L = _radiance(r, n, wi)
        thp = 0.2 + 0.8 * r.uniform(n, 3)
        depths.append({
            "L": (thp * L[:, None] * torch.tensor([0.8, 1.0, 1.2], device="cuda")).contiguous(), "thp": thp.contiguous(),
            "pos": _surface_points(r, n), "dir": torch.stack(_angles(wi), -1).contiguous(),
            "wi_pdf": INV_4PI * (0.5 + r.uniform(n)), "bsdf_pdf": INV_4PI * (0.5 + r.uniform(n)),
            "mis_weight": 0.5 + 0.5 * r.uniform(n), "delta": torch.zeros(n, device="cuda", dtype=torch.uint8),
            "bsdf_val": (0.2 + r.uniform(n, 3)).contiguous(), "wo": torch.stack(_angles(r.sphere(n)), -1).contiguous(),
            "normal": torch.stack(_angles(r.sphere(n)), -1).contiguous(), "roughness": r.uniform(n)})
    return depths, torch.full((n,), c["depths"], device="cuda", dtype=torch.int32)


def _frame_size(c):
    train_res = (c["res_x"] // c["stride"], c["res_y"] // c["stride"])
    return train_res, train_res[0] * train_res[1] * c["depths"]


def prepare(case, seed):
    c = dict(case)
    if c["kind"].startswith("mix_"):
        return _mixture_inputs(c, seed)
    cfg = _config(c)
    train = c["kind"].startswith("train")
    n = _frame_size(c)[1] if c["kind"] == "train_frame" else c["n"]
    f = nmg.GuidingField(cfg, max_queries=0 if train else n, max_batch=n if train else 0)
    f.set_params(_params(f.info, cfg, seed))
    s = {"case": c, "field": f}
    r = _Rng(seed)
    if c["kind"] == "train_frame":
        s["records"], s["cur_depth"] = _frame_records(c, seed)
    elif train:
        s["x"], s["records"] = _training_rows(r, n, cfg.input_mode, cfg.selection)
    else:
        s.update(_shading(r, n))
        if c["kind"] == "query":
            s["u4"] = r.uniform(n, 4)
        else:
            s["wi"] = r.sphere(n).contiguous()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    c = s["case"]
    if c["kind"] == "mix_sample":
        d, p, lobe = nmg.mixture_sample(s["raw"], s["u4"], c["lobes"], s["normal"], c["softplus"])
        return {"dir": d, "pdf": p, "lobe": lobe}
    if c["kind"] == "mix_pdf":
        return {"pdf": nmg.mixture_pdf(s["raw"], s["wi"], c["lobes"], s["normal"], c["softplus"])}
    if c["kind"] == "mix_loss":
        g, loss, total = nmg.mixture_loss_grad(s["raw"], s["records"], c["lobes"], selection=c["selection"],
                                               kappa_softplus=c["softplus"])
        return {"grad": g, "loss": loss, "loss_sum": total}
    f = s["field"]
    if c["kind"] == "query":
        return f.query(s["pos"], s["wo"], s["normal"], s["rough"], s["u4"])
    if c["kind"] == "pdf":
        return {"pdf": f.pdf(s["pos"], s["wo"], s["normal"], s["rough"], s["wi"])}
    if c["kind"] == "train_step":
        stats = f.train_step(s["x"], s["records"])
    else:
        train_res, n = _frame_size(c)
        _, _, stats = f.train_frame(s["records"], s["cur_depth"], (0, 0), (c["stride"],) * 2, train_res,
                                    (c["res_x"], c["res_y"]), n, n, 1, 128)
    return {"grad": f.get_gradients(), "stats": stats.float()}


# ------------------------------------------------------------------ least work
def work(case):
    """Each input read once and each output written once; the arithmetic of the network and the mixture."""
    c = dict(case)
    K = c["lobes"]
    mix = 120 * K  # operations of one mixture evaluation, about
    if c["kind"].startswith("mix_"):
        n = c["n"]
        row = 16 * K + (12 if c.get("cosine") else 0)
        if c["kind"] == "mix_sample":
            return {"bytes": n * (row + 16 + 20), "flops": n * mix}
        if c["kind"] == "mix_pdf":
            return {"bytes": n * (row + 12 + 4), "flops": n * mix}
        sel = 1 if c["selection"] else 0
        return {"bytes": n * (2 * (row + 4 * sel) + 24 + 4 * sel + 4), "flops": 2 * n * mix}
    cfg = _config(c)
    info = nmg.config_info(cfg)
    macs = sum(i * o for i, o in _layer_sizes(info, cfg))
    grid = int(info.n_encoded) * 16
    small = c["path"] != "fp32"
    if c["kind"] in ("query", "pdf"):
        n = c["n"]
        out = 40 + 16 + 20 + (4 if cfg.selection else 0) if c["kind"] == "query" else 40 + 12 + 4
        return {"bytes": n * out + (2 if small else 4) * int(info.n_params), "flops": n * (2 * macs + grid + mix)}
    if c["kind"] == "train_frame":
        n = _frame_size(c)[1]
        rows = 93
    else:
        n = c["n"]
        rows = 4 * (int(info.n_input) + int(info.record_floats))
    # weights, moments, step counters, average and gradient read; all of them and the 16-bit copies written
    return {"bytes": n * rows + int(info.n_params) * (24 + 24 + (4 if small else 0)), "flops": n * (6 * macs + 2 * grid + 2 * mix)}


# ------------------------------------------------------------------ the same in 64 bits
def _vmf_norm(k):
    return torch.where(k < EPS, torch.full_like(k, INV_4PI), k / (2 * math.pi * -torch.expm1(-2 * k.clamp_min(EPS))))


def _activate(raw, K, softplus):
    r = raw[:, :4 * K].double().view(-1, K, 4)
    lam = torch.exp(r[..., 0].clamp(-10, 15))
    kap = torch.nn.functional.softplus(r[..., 1]) if softplus else torch.exp(r[..., 1].clamp(-10, 15))
    st, sp = torch.sigmoid(r[..., 2]), torch.sigmoid(r[..., 3])
    return lam, kap, math.pi * st, 2 * math.pi * sp, st, sp


def _unit(th, ph):
    return torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)], -1)


def _times_cosine(lam, kap, mu, normal):
    mb = (normal / normal.norm(dim=-1, keepdim=True))[:, None, :]
    nm = kap[..., None] * mu + COSINE_KAPPA * mb
    nk = nm.norm(dim=-1)
    some = nk >= 1e-3
    nm = torch.where(some[..., None], nm / nk[..., None].clamp_min(1e-30), mu)
    nk = torch.where(some, nk, torch.zeros_like(nk))
    e = torch.exp(kap * ((nm * mu).sum(-1) - 1) + COSINE_KAPPA * ((nm * mb).sum(-1) - 1))

    def norm(k):
        return torch.where(k < 1e-3, torch.full_like(k, INV_4PI), k / (2 * math.pi * -torch.expm1(-2 * k.clamp_min(1e-3))))

    nb = COSINE_KAPPA / (2 * math.pi * -math.expm1(-2 * COSINE_KAPPA))
    return norm(kap) * nb / norm(nk) * e * lam, nk, nm


def _frame_of(mu, loc):
    a = mu.abs()
    xm = (a[:, 0] < a[:, 1]) & (a[:, 0] < a[:, 2])
    ym = ~xm & (a[:, 1] < a[:, 2])
    axis = torch.stack([xm, ym, ~(xm | ym)], -1).double()
    t = torch.nn.functional.normalize(torch.cross(mu, axis, dim=-1), dim=-1)
    b = torch.nn.functional.normalize(torch.cross(mu, t, dim=-1), dim=-1)
    return t * loc[:, :1] + b * loc[:, 1:2] + mu * loc[:, 2:3]


def _mixture(raw, K, softplus, normal, u4=None, wi=None):
    """(dir, pdf, lobe) of the mixture: sampled with u4, or the pdf at wi."""
    lam, kap, th, ph, _, _ = _activate(raw, K, softplus)
    mu = _unit(th, ph)
    if normal is not None:
        lam, kap, mu = _times_cosine(lam, kap, mu, normal.double())
    total = lam.sum(1, keepdim=True)
    w = lam / (total.clamp_min(EPS) if normal is not None else total)
    lobe = None
    if wi is None:
        u = u4.double()
        over = u[:, 1:2] >= torch.cumsum(w, 1)
        lobe = over.sum(1)
        lobe = torch.where(lobe >= K, torch.zeros_like(lobe), lobe)
        at = torch.arange(len(lobe), device=lobe.device)
        k, m = kap[at, lobe], mu[at, lobe]
        flat = k < EPS
        ct = torch.where(flat, 1 - 2 * u[:, 2], 1 + torch.log1p(u[:, 2] * torch.expm1(-2 * k)) / k.clamp_min(EPS))
        st = torch.sqrt((1 - ct * ct).clamp_min(0))
        az = 2 * math.pi * u[:, 3]
        wi = _frame_of(m, torch.stack([torch.cos(az) * st, torch.sin(az) * st, ct], -1))
    c = (wi.double()[:, None, :] * mu).sum(-1)
    pdf = (w * _vmf_norm(kap) * torch.exp(kap * torch.clamp(c - 1, max=0))).sum(1)
    return wi, pdf, lobe


def _kl_gradient(raw, rec, K, softplus, sel, scale):
    """(dL/draw, loss): the loss's gradient as the reference defines it, its polynomial below kappa 1 included."""
    lam, kap, th, ph, st, sp = _activate(raw, K, softplus)
    dkap = torch.sigmoid(raw[:, 1:4 * K:4].double()) if softplus else kap
    mu = _unit(th, ph)
    rec = rec.double()
    wi = _unit(rec[:, 0], rec[:, 1])[:, None, :]
    c = (wi * mu).sum(-1)
    vmf = _vmf_norm(kap) * torch.exp(torch.where(kap < EPS, 0 * kap, kap) * torch.clamp(c - 1, max=0))
    total = lam.sum(1, keepdim=True)
    q = (lam * vmf).sum(1, keepdim=True) / total
    L = rec[:, 2:5].mean(1, keepdim=True)
    s = torch.sigmoid(raw[:, 4 * K:4 * K + 1].double()) if sel else 1.0
    if sel:
        wp = s * (q + EPS) + (1 - s) * rec[:, 6:7]
        pre, loss = -L / wp / wp * scale, -L / wp * torch.log(wp)
    else:
        wp = rec[:, 5:6] + EPS
        pre, loss = -L / wp / (q + EPS) * scale, -L / wp * torch.log(q + EPS)
    wv = lam / total * vmf
    k = kap.clamp_min(1e-4)
    ik = torch.where(kap < 1, 0.000926 - 0.344883 * kap + 0.030147 * kap * kap, 1 / k - 1 / torch.tanh(k))
    dt = (wi * torch.stack([torch.cos(th) * torch.cos(ph), torch.cos(th) * torch.sin(ph), -torch.sin(th)], -1)).sum(-1)
    dp = (wi * torch.stack([-torch.sin(th) * torch.sin(ph), torch.sin(th) * torch.cos(ph), 0 * th], -1)).sum(-1)
    g = torch.stack([pre * (vmf - q) / total * s * lam, pre * wv * (c + ik) * s * dkap,
                     pre * wv * kap * dt * s * math.pi * st * (1 - st),
                     pre * wv * kap * dp * s * 2 * math.pi * sp * (1 - sp)], -1).view(len(raw), 4 * K)
    out = torch.zeros(raw.shape, dtype=torch.float64, device=raw.device)
    if sel:
        out[:, 4 * K:4 * K + 1] = 0.01 * pre * (q - rec[:, 6:7]) * s * (1 - s)
    else:
        g = torch.where(torch.isfinite(g), g.clamp(max=150.0), torch.zeros_like(g))
    out[:, :4 * K] = g
    return out, loss[:, 0]


def _sh(degree, v):
    x, y, z = v.unbind(-1)
    o = [torch.full_like(x, 0.28209479177387814), -0.48860251190291987 * y, 0.48860251190291987 * z,
         -0.48860251190291987 * x]
    if degree > 2:
        x2, y2, z2 = x * x, y * y, z * z
        o += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.94617469575755997 * z2 - 0.31539156525251999,
              -1.0925484305920792 * x * z, 0.54627421529603959 * (x2 - y2), 0.59004358992664352 * y * (-3 * x2 + y2),
              2.8906114426405538 * x * y * z, 0.45704579946446572 * y * (1 - 5 * z2),
              0.3731763325901154 * z * (5 * z2 - 3), 0.45704579946446572 * x * (1 - 5 * z2),
              1.4453057213202769 * z * (x2 - y2), 0.59004358992664352 * x * (-x2 + 3 * y2)]
    return torch.stack(o[:degree * degree], -1)


def _oneblob(x, bins):
    def cdf(t):
        u = t * bins
        return ((15.0 / 16.0) * u * (1 - (2.0 / 3.0) * u ** 2 + 0.2 * u ** 4) + 0.5).clamp(0, 1).where(u.abs() < 1, (u > 0).to(u.dtype))

    e = torch.arange(bins + 1, device=x.device, dtype=torch.float64) / bins
    at = e[None, :] - x[:, None]
    return torch.diff(cdf(at) + cdf(at - 1) + cdf(at + 1), dim=1)


def _grid_levels(cfg):
    """(scale, resolution, first entry, entries) of each level."""
    step, off, out = np.log2(np.float32(cfg.grid_per_level_scale)), 0, []
    for lv in range(cfg.grid_levels):
        scale = np.float32(2.0 ** float(np.float32(lv) * np.float32(step))) * np.float32(cfg.grid_base_resolution) - np.float32(1)
        res = int(math.ceil(scale)) + 1
        n = (res ** 3 + 7) // 8 * 8
        if cfg.grid_hash:
            n = min(n, 1 << cfg.grid_log2_hashmap)
        out.append((float(scale), res, off, n))
        off += n
    return out


def _encode(cfg, x, table):
    """Encoded rows of network input rows x; table [entries, features]."""
    feats = []
    for scale, res, off, T in _grid_levels(cfg):
        p = x[:, :3] * scale + 0.5
        g = torch.floor(p)
        f = p - g
        f = f * f * (3 - 2 * f) if cfg.grid_smoothstep else f
        g = g.long()
        acc = 0
        for k in range(8):
            b = [(k >> d) & 1 for d in range(3)]
            e = [g[:, d] + b[d] for d in range(3)]
            if cfg.grid_hash and res ** 3 > T:
                i = (e[0] ^ (e[1] * 2654435761 & 0xFFFFFFFF) ^ (e[2] * 805459861 & 0xFFFFFFFF)) & (T - 1)
            else:
                i = (e[0] + e[1] * res + e[2] * res * res) % T
            w = 1
            for d in range(3):
                w = w * (f[:, d] if b[d] else 1 - f[:, d])
            acc = acc + w[:, None] * table[off + i]
        feats.append(acc)
    out = feats + [_sh(cfg.sh_degree, x[:, 3:6] * 2 - 1)]
    if cfg.input_mode == 0:
        out += [_oneblob(x[:, d], cfg.oneblob_bins) for d in (6, 7, 8)]
    else:
        out += [_sh(cfg.sh_degree, x[:, 6:9] * 2 - 1), _oneblob(x[:, 9], cfg.oneblob_bins)]
    h = torch.cat(out, 1)
    return torch.nn.functional.pad(h, (0, _round16(h.shape[1]) - h.shape[1]), value=1.0)


def _network(cfg, info, x, params):
    n_mlp = int(info.n_mlp_params)
    h = _encode(cfg, x, params[n_mlp:].view(-1, cfg.grid_features))
    off = 0
    sizes = _layer_sizes(info, cfg)
    for l, (i, o) in enumerate(sizes):
        h = h @ params[off:off + i * o].view(o, i).T
        off += i * o
        if l < len(sizes) - 1:
            h = torch.relu(h)
    return h


def _input_rows(cfg, pos, wo, normal, rough):
    infl = math.sqrt(3) * 0.005
    wo = wo / wo.norm(dim=-1, keepdim=True)
    n = normal / normal.norm(dim=-1, keepdim=True)
    cols = [0.5 + (pos - 0.5) / (1 + 2 * infl), (wo + 1) * 0.5]
    if cfg.input_mode == 0:
        th, ph = _angles(n)
        cols.append(torch.stack([th / math.pi, ph / (2 * math.pi)], -1))
    else:
        cols.append((n + 1) * 0.5)
    cols.append((1 - torch.exp(-rough))[:, None])
    return torch.cat(cols, 1)


def _frame_rows(cfg, c, depths):
    """(x, records) of a frame's training pixels: every stride-th pixel's vertices."""
    at = (torch.arange(c["res_y"] // c["stride"], device="cuda")[:, None] * c["stride"] * c["res_x"] +
          torch.arange(c["res_x"] // c["stride"], device="cuda")[None, :] * c["stride"]).reshape(-1)
    xs, recs = [], []
    for d in depths:
        v = {k: t[at].double() for k, t in d.items()}
        L = v["L"] / v["thp"] * v["mis_weight"][:, None] * v["bsdf_val"]
        xs.append(_input_rows(cfg, v["pos"], _unit(v["wo"][:, 0], v["wo"][:, 1]), _unit(v["normal"][:, 0], v["normal"][:, 1]), v["roughness"]))
        recs.append(torch.cat([v["dir"], L, v["wi_pdf"][:, None], v["bsdf_pdf"][:, None]], 1))
    return torch.cat(xs), torch.cat(recs)


def exact(case, seed):
    c = dict(case)
    K = c["lobes"]
    if c["kind"].startswith("mix_"):
        s = _mixture_inputs(c, seed)
        if c["kind"] == "mix_loss":
            g, loss = _kl_gradient(s["raw"], s["records"], K, c["softplus"], c["selection"], 128.0 / c["n"])
            return {"grad": g, "loss": loss, "loss_sum": loss.sum().view(1)}
        d, p, _ = _mixture(s["raw"], K, c["softplus"], s["normal"], s.get("u4"), s.get("wi"))
        return {"dir": d, "pdf": p, "lobe": None} if c["kind"] == "mix_sample" else {"pdf": p}
    cfg = _config(c)
    info = nmg.config_info(cfg)
    params = _params(info, cfg, seed).double()
    r, step = _Rng(seed), 1 << 16
    if c["kind"] in ("query", "pdf"):
        n = c["n"]
        s = _shading(r, n)
        u4 = r.uniform(n, 4) if c["kind"] == "query" else None
        wi = None if c["kind"] == "query" else r.sphere(n)
        out = []
        for i in range(0, n, step):
            at = slice(i, i + step)
            pos, wo, nrm, rough = (s[k][at].double() for k in ("pos", "wo", "normal", "rough"))
            raw = _network(cfg, info, _input_rows(cfg, pos, wo, nrm, rough), params)
            facing = torch.where((nrm * wo).sum(-1, keepdim=True) > 0, nrm, -nrm) if cfg.cosine_aware else None
            d, p, _ = _mixture(raw, K, False, facing, None if u4 is None else u4[at], None if wi is None else wi[at])
            out.append((d, p, torch.sigmoid(raw[:, 4 * K]) if cfg.selection else None))
        if c["kind"] == "pdf":
            return {"pdf": torch.cat([p for _, p, _ in out])}
        full = {"dir": torch.cat([d for d, _, _ in out]), "pdf": torch.cat([p for _, p, _ in out]), "lobe": None}
        if cfg.selection:
            full["selection"] = torch.cat([q for _, _, q in out])
        return full
    if c["kind"] == "train_frame":
        x, rec = _frame_rows(cfg, c, _frame_records(c, seed)[0])
    else:
        x, rec = (t.double() for t in _training_rows(r, c["n"], cfg.input_mode, cfg.selection))
    n, total = len(x), 0.0
    params.requires_grad_(True)
    for i in range(0, n, step):
        raw = _network(cfg, info, x[i:i + step], params)
        g, loss = _kl_gradient(raw.detach(), rec[i:i + step], K, False, bool(cfg.selection), 128.0 / n)
        raw.backward(g)
        total += loss.sum()
    return {"grad": params.grad, "stats": torch.stack([total / n, params.grad.norm() / 128.0])}
