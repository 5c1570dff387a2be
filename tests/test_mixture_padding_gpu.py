"""The gradient's padding columns: zeros from the binding, for every lobe count,
with and without selection, in rows with no padding, with four and with many
columns of it; untouched by the C function that says so."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("selection", [False, True])
@pytest.mark.parametrize("K", [4, 7, 8, 16])
def test_gradient_padding(nmg, synth, K, selection):
    import torch
    nout = 4 * K + int(selection)
    for n in (1, 129, 5000):
        for stride in sorted({(nout + 3) // 4 * 4, (nout + 3) // 4 * 4 + 4, 80}):
            rows, _, rec = synth.mixture_batch(n, K, seed=3)
            raw = torch.full((n, stride), 9.0, device="cuda")
            raw[:, :4 * K] = torch.from_numpy(rows[:, :4 * K]).cuda()
            r = torch.zeros(n, 7 if selection else 6, device="cuda")
            r[:, :6] = torch.from_numpy(rec[:, :6]).cuda()
            if selection:
                raw[:, 4 * K] = 0.3
                r[:, 6] = 0.08
            torch.full((n, stride), 5.0, device="cuda")  # what the allocation may hold
            g, loss, _ = nmg.mixture_loss_grad(raw, r, K, selection=selection)
            assert bool((g[:, nout:] == 0).all())
            want = torch.full_like(raw, 5.0)
            ws = torch.empty(nmg.lib().nmg_mixture_loss_workspace_bytes(n), device="cuda", dtype=torch.uint8)
            tot = torch.empty(1, device="cuda", dtype=torch.float64)
            p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
            o = nmg.mixture_opts(K, stride, selection=selection)
            nmg.check(nmg.lib().nmg_mixture_loss_grad(C.byref(o), p(raw), p(r), r.shape[1], n, 128.0, p(want), None, p(tot),
                                                      p(ws), ws.numel(), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            assert torch.equal(g[:, :nout], want[:, :nout])
            assert bool((want[:, nout:] == 5).all())
