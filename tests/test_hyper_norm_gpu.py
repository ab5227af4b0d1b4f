"""Norm of an updated embedding or head under the hyperball rule: error of the sum, its order, and the optimizer's two routes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("u_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [4, 1020, 4096, 4100, 1024 * 4096, 1024 * 4096 + 4, 200064 * 2560])
def test_sum_of_squares_after_update(n, u_dtype):
    """One segment: the sum repeats bit for bit and is a tree's, not a chain's.  A square passes through at most 17 fp32 additions
    inside its block of 4096 elements (independent roundings, of which sums of many blocks keep next to nothing), the blocks are added
    in double, and the result is rounded twice: a few times 2^-24.  A chain of one addition per block shows 3.6e-6 at the largest
    size."""
    from archscale_b200.ops import backend
    ext = backend.require_extension()
    g = torch.Generator(device="cuda").manual_seed(12)
    x0, u = torch.randn(n, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g).to(u_dtype)
    bounds, kidx = torch.tensor([0, n], device="cuda"), torch.tensor([1], dtype=torch.int32, device="cuda")
    coef = torch.tensor([9.0, 0.03, 9.0], device="cuda")
    runs = []
    for _ in range(3):
        x, acc = x0.clone(), torch.tensor([0.0, 2.0, 0.0], device="cuda")
        ext.seg_update_(1, x, u, bounds, kidx, coef, acc)
        runs.append((x, acc))
    x, acc = runs[0]
    assert all(torch.equal(a, acc) and torch.equal(b, x) for b, a in runs[1:])
    sq, step = 2.0, 1 << 26
    for a in range(0, n, step):
        xd = x[a:a + step].double()
        want = x0[a:a + step].double() - coef[1].double() * u[a:a + step].double()
        assert float((xd - want).abs().max()) <= 2 ** -23 * float(want.abs().max())
        sq += float(xd.square().sum())
    assert float(acc[0]) == 0.0 and float(acc[2]) == 0.0
    assert abs(float(acc[1]) - sq) <= 4 * 2 ** -24 * sq


def test_optimizer_routes_agree(monkeypatch):
    """The same step with the embeddings' update on the segment kernels and in the foreach form."""
    from archscale_b200 import Config
    from archscale_b200.models.gpt import GPT, Block
    from archscale_b200.ops import fused_linear_cross_entropy
    from archscale_b200.optim.sharded import ShardedOptimizer
    from archscale_b200.parallel.fsdp import FSDPEngine
    dev = torch.device("cuda", 0)
    cfg = Config.from_name("transformer_gqa4_d16", n_layer=2, ar=None, n_embd=512, n_head=4, n_query_groups=2, head_dim=128,
                           intermediate_size=1408, block_size=512, qk_norm=True, mup=True, depth_scale=True, use_muon=True,
                           use_muonh=True, head_init_std=0.02)

    def run(seg):
        torch.manual_seed(0)
        with torch.device(dev):
            model = GPT(cfg)
        model.reset_parameters()
        eng = FSDPEngine(model, unit_classes=(Block,), param_dtype=torch.bfloat16, device=dev)
        opt = ShardedOptimizer(eng, lr=1e-2, algorithm="muonh")
        taken = []
        own = opt._hyper_seg_ok
        monkeypatch.setattr(opt, "_hyper_seg_ok", lambda x, u: taken.append(own(x, u)) or (seg and taken[-1]))
        data = torch.randint(0, cfg.vocab_size, (2, 513), device=dev, generator=torch.Generator(device=dev).manual_seed(3))
        out = model(data[:, :-1], use_flce_loss=True)
        eng.backward(fused_linear_cross_entropy(out.logits, out.weight, data[:, 1:]))
        before = [g.master.clone() for g in eng.groups()]
        opt.step()
        assert any(taken)                                             # embeddings and head qualify
        return before, [g.master.clone() for g in eng.groups()]

    (b0, w0), (_, w1) = run(True), run(False)
    for b, a, r in zip(b0, w0, w1):
        # of the step itself: fp32 products and sums in another order, and gradients that agree to their atomics' order
        assert float((a - r).norm()) <= 1e-4 * float((r - b).norm()) + 1e-7 * float(r.norm())
