"""Gated RMSNorm with 1, 2, 4 and 8 warps per (row, group) and the loop for wider groups, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,groups,g,nbg,gated", [
    (1, 1, 8, True, True), (37, 6, 512, True, True), (9, 2, 520, False, True), (301, 1, 1024, False, True), (5, 3, 1032, True, True),
    (64, 1, 2048, False, False), (7, 1, 2056, True, True), (2300, 1, 3968, False, True), (3, 1, 4096, True, False), (4, 1, 4104, False, True),
])
def test_gated_norm(rows, groups, g, nbg, gated, dtype):
    from archscale_b200.ops.norm import gated_rms_norm
    torch.manual_seed(8)
    n = groups * g
    mk = lambda: torch.randn(rows, n, device="cuda").to(dtype).requires_grad_(True)
    x, z = mk(), (mk() if gated else None)
    w = (1 + 0.2 * torch.randn(n, device="cuda")).requires_grad_(True)
    y = gated_rms_norm(x, w, z, 1e-5, g, nbg)
    gy = torch.randn(rows, n, device="cuda").to(dtype)
    ins = [t for t in (x, w, z) if t is not None]
    got = torch.autograd.grad(y, ins, gy)
    refs = [t.detach().double().requires_grad_(True) for t in ins]
    xd, wd = refs[:2]
    s = torch.nn.functional.silu(refs[2]) if gated else torch.ones_like(xd)
    xin = (xd if nbg else xd * s).view(rows, groups, g)
    nrm = (xin * torch.rsqrt(xin.pow(2).mean(-1, keepdim=True) + 1e-5)).view(rows, n) * wd
    yd = nrm * s if nbg else nrm
    ref = torch.autograd.grad(yd, refs, gy.double())
    # bf16 results are rounded once (2^-9); fp32: sums over up to 4104 columns or 2300 rows and the fast exponential
    for a, r in zip((y, *got), (yd, *ref)):
        tol = 4e-3 if a.dtype == torch.bfloat16 else 2e-6
        assert float((a.double() - r).norm()) <= tol * float(r.norm())
