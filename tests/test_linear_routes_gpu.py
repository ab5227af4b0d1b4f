"""Fused linear routes on the GPU: what they must not lose of the layers they stand for."""
import pytest
import torch
import torch.nn.functional as F

from archscale_b200.config import Config
from archscale_b200.models.gpt import LLaMAMLP
from archscale_b200.models.layers import Linear
from archscale_b200.ops import backend, gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("neighbours", [False, True])
@pytest.mark.parametrize("T", [8, 41, 64, 65, 72])
def test_hooks_of_the_projections_act_at_every_token_count(T, neighbours):
    torch.manual_seed(0)
    layers = [Linear(256, n, bias=False, device="cuda", dtype=torch.bfloat16) for n in (256, 64, 64)]
    if neighbours:
        flat = torch.cat([l.weight.detach() for l in layers])
        for l, w in zip(layers, flat.split([256, 64, 64])):
            l.weight = torch.nn.Parameter(w)
    x = torch.randn(1, T, 256, device="cuda").bfloat16()
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            plain = list(gemm.linear_multi(x, layers))
            h = layers[0].register_forward_hook(lambda m, a, y: y + 1)
            layers[2].forward = lambda x: x.new_zeros(*x.shape[:-1], 64)
            y = gemm.linear_multi(x, layers, keep_fused=True)
            assert not torch.is_tensor(y)
            tol = dict(rtol=2.0 ** -7, atol=2.0 ** -7)        # the fused product may sum in another order: one rounding to bf16 each
            torch.testing.assert_close(y[0], plain[0] + 1, **tol)
            torch.testing.assert_close(y[1], plain[1], **tol)
            assert not y[2].any()
            h.remove()
            del layers[2].forward


@pytest.mark.parametrize("T", [41, 64, 65, 72])
def test_a_hook_on_the_up_projection_acts_at_every_token_count(T):
    cfg = Config.from_name("transformer_gqa4_d8", intermediate_size=704)
    mlp = LLaMAMLP(cfg).cuda().bfloat16()
    mlp.reset_parameters()
    mlp.w1.register_forward_hook(lambda m, a, y: torch.zeros_like(y))
    with torch.no_grad():
        y, _ = mlp(torch.randn(1, T, cfg.n_embd, device="cuda").bfloat16(), 0)
    assert not y.any()


@pytest.mark.parametrize("T", [65, 257, 1001, 4099])
def test_odd_token_counts_without_gradients_run_the_library(T):
    torch.manual_seed(0)
    x, w = torch.randn(T, 256, device="cuda").bfloat16(), (torch.randn(264, 256, device="cuda") / 16).bfloat16()
    n0 = backend.launches()
    with torch.no_grad():
        y = gemm.linear(x, w)
    assert backend.launches() == n0 and torch.equal(y, F.linear(x, w))
    gemm.linear(x, w.requires_grad_())                       # with gradients: the own GEMM, whose backward pays
    assert backend.launches() == n0 + 1
    with torch.no_grad():
        gemm.linear(x[:T // 8 * 8], w)
        assert backend.launches() == n0 + 2
