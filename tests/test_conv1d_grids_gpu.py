"""Causal conv1d backward on the grids between which it chooses its form, with documents that break inside groups of steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# blocks of 128 steps: 2 per sequence of 130
@pytest.mark.parametrize("B", [1, 32, 33, 148, 149, 222, 223])
@pytest.mark.parametrize("W", [2, 3, 4])
@pytest.mark.parametrize("dtype,packed", [(torch.float32, True), (torch.float32, False), (torch.bfloat16, True)])
def test_conv_backward_grids(B, W, dtype, packed):
    from archscale_b200.ops.conv1d import causal_conv1d
    L, C, dev = 130, 16, "cuda"
    x = torch.randn(B, L, C, device=dev).to(dtype).requires_grad_(True)
    w, bias = torch.randn(C, W, device=dev).requires_grad_(True), torch.randn(C, device=dev).requires_grad_(True)
    g = torch.randn(B, L, C, device=dev).to(dtype)
    sid = (torch.rand(B, L, device=dev) < 0.2).cumsum(1).to(torch.int32) if packed else None
    got = torch.autograd.grad(causal_conv1d(x, w, bias, sid, "silu", channel_last=True), (x, w, bias), g)
    xd, wd, bd = refs = [t.detach().double().requires_grad_(True) for t in (x, w, bias)]
    pre = bd.view(1, 1, C)
    for j in range(W):
        s = W - 1 - j
        tap = torch.nn.functional.pad(xd, (0, 0, s, 0))[:, :L]
        if packed:
            tap = tap * (torch.nn.functional.pad(sid, (s, 0), value=-1)[:, :L] == sid).unsqueeze(-1)
        pre = pre + wd[:, j] * tap
    ref = torch.autograd.grad(torch.nn.functional.silu(pre), refs, g.double())
    # bf16: one rounding (2^-9) of dx; fp32: the fast exponential and sums over at most B·L = 29 K terms
    for a, r in zip(got, ref):
        assert float((a.double() - r).norm()) <= (4e-3 if a.dtype == torch.bfloat16 else 1e-5) * float(r.norm())
