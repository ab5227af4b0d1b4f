"""One-group SSD scan: whole op on its kernels against the recurrence in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Bb,L,H,P,N,dtype,packed,with_D", [
    (2, 200, 4, 64, 16, torch.bfloat16, True, True),
    (1, 64, 2, 128, 32, torch.float32, False, True),
    (3, 65, 16, 64, 16, torch.bfloat16, False, False),
    (1, 130, 5, 64, 128, torch.float32, True, True),
])
def test_ssd_one_group(Bb, L, H, P, N, dtype, packed, with_D):
    from archscale_b200.ops import ssd
    torch.manual_seed(6)
    dev = "cuda"
    x = torch.randn(Bb, L, H, P, device=dev).to(dtype).requires_grad_(True)
    dt = (torch.rand(Bb, L, H, device=dev) * 0.5).requires_grad_(True)
    A = (-torch.rand(H, device=dev) - 0.1).requires_grad_(True)
    B, C = (torch.randn(Bb, L, 1, N, device=dev).to(dtype).requires_grad_(True) for _ in range(2))
    D = torch.randn(H, device=dev).requires_grad_(True) if with_D else None
    seq_idx = None
    if packed:
        seq_idx = torch.zeros(Bb, L, dtype=torch.int32, device=dev)
        for i, cut in enumerate((40, 41, 64, 129)):
            seq_idx[:, cut:] = i + 1
    assert ssd._chunk_scan_ok(x, B, 64)
    y = ssd.ssd_scan(x, dt, A, B, C, D, seq_idx)
    assert y.dtype == dtype
    g = torch.randn(y.shape, device=dev).to(dtype)
    ins = [t for t in (x, dt, A, B, C, D) if t is not None]
    grads = torch.autograd.grad(y, ins, g)
    refs = [t.detach().double().requires_grad_(True) for t in ins]
    xr, dtr, Ar, Br, Cr = refs[:5]
    Dr = refs[5] if with_D else None
    # the recurrence in fp64 (the oracle of the module works in fp32)
    S = xr.new_zeros(Bb, H, P, N)
    ys = []
    for s in range(L):
        if seq_idx is not None and s > 0:
            S = S * (seq_idx[:, s] == seq_idx[:, s - 1]).view(Bb, 1, 1, 1)
        S = S * torch.exp(dtr[:, s] * Ar).view(Bb, H, 1, 1) + torch.einsum("bh,bhp,bn->bhpn", dtr[:, s], xr[:, s], Br[:, s, 0])
        ys.append(torch.einsum("bhpn,bn->bhp", S, Cr[:, s, 0]) + (0 if Dr is None else xr[:, s] * Dr.view(1, H, 1)))
    yr = torch.stack(ys, 1)
    gr = torch.autograd.grad(yr, refs, g.double())
    # the batched products may run with 10-bit mantissas (TF32: 2^-11 per operand); bf16 results carry 2^-9 each
    for a, r in zip((y, *grads), (yr, *gr)):
        assert float((a.double() - r).norm()) <= 6e-3 * float(r.norm()) + 1e-6
