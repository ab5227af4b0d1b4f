"""The workloads whose speed matters to a user of this framework, as cases that a timing tool can run.

A case is a plain dict.  Its ``kind`` says which public entry point a pass goes through:

* ``step``    one optimizer step of pre-training: ``Trainer.forward_backward`` of one micro-batch + ``Trainer.optimizer_step``
              (gradient clip, Newton-Schulz / MuonH, AdamW); returns the loss and the updated fp32 weights
* ``score``   long-window scoring without gradients (perplexity evaluation): hidden states and the fused linear
              cross-entropy loss
* ``logits``  the forward pass behind one token of ``ModelWrapper.generate`` (the prefix is re-run for every token) and
              behind log-likelihood requests: full logits of a short ragged prefix

Sizes are those of the launch scripts, the registry and the headline benchmark: depth-8..16 models of every mixer family,
a depth-8 cut of the Phi-4-mini-flash shape, contexts up to 32768, up to 65536 tokens per pass.
"""
import functools
import math
import os
import tempfile

import numpy as np
import torch

from archscale_b200.config import Config
from archscale_b200.eval.common import ModelWrapper
from archscale_b200.models.gpt import GPT
from archscale_b200.ops.cross_entropy import FusedLinearCrossEntropyLoss
from archscale_b200.train.pretrain import setup
from archscale_b200.utils.speed_monitor import matmul_parameter_count

EOS = 2

# What a run of each family passes to setup(): registry name, train name (its switches), registry depth if it is fixed
FAMILIES = {
    "dense": dict(model="transformer_gqa4", name="scaling_mup_muonh_qknorm"),
    "moe": dict(model="transformer_gqa4_h2_moe", name="scaling_mup_muonh_qknorm"),
    "sambay": dict(model="sambay", name="scaling_mup_muonh"),
    "gdny": dict(model="gdny", name="scaling_mup_muonh"),
    "mambay2": dict(model="mambay2", name="scaling_mup_muonh"),
    # differential attention, LayerNorm, vocabulary 200064, tied embeddings, packed documents; `depth` cuts the layer count
    "phi4": dict(model="phi4miniflash", name="scaling_mup_muonh_tie_rbase_varlen", fixed_depth=32),
}


def listed():
    return [
        # one token of greedy generation / one log-likelihood request: latency of a small forward pass, odd length
        dict(name="logits_dense_d8_t41", kind="logits", family="dense", depth=8, batch=1, ctx=41, low="bf16"),
        # a proxy run on a small batch (hyper-parameter sweeps at small depth): launches and host work count
        dict(name="step_dense_d8_1x1000", kind="step", family="dense", depth=8, batch=1, ctx=1000, low="bf16"),
        # the headline dense configuration, a whole optimizer step
        dict(name="step_dense_d16_8x4096", kind="step", family="dense", depth=16, batch=8, ctx=4096, low="bf16"),
        # the same model with MXFP8 linear layers (--fp8)
        dict(name="step_dense_d16_fp8_4x4096", kind="step", family="dense", depth=16, batch=4, ctx=4096, low="fp8"),
        # long-context training: attention is the larger part
        dict(name="step_dense_d8_1x32768", kind="step", family="dense", depth=8, batch=1, ctx=32768, low="bf16"),
        # the headline MoE configuration, a whole optimizer step
        dict(name="step_moe_d8_16x4096", kind="step", family="moe", depth=8, batch=16, ctx=4096, low="bf16"),
        # hybrid with Mamba-1: training step, and perplexity over a long window
        dict(name="step_sambay_d16_4x4096", kind="step", family="sambay", depth=16, batch=4, ctx=4096, low="bf16"),
        dict(name="score_sambay_d16_1x32768", kind="score", family="sambay", depth=16, batch=1, ctx=32768, low="bf16"),
        # packed variable-length documents in one 8 K row, Phi-4-mini-flash layers
        dict(name="step_phi4_l8_1x8192", kind="step", family="phi4", depth=8, batch=1, ctx=8192, low="bf16"),
        # hybrid with Gated DeltaNet, sequences that are no multiple of a chunk or tile
        dict(name="step_gdny_d16_3x2731", kind="step", family="gdny", depth=16, batch=3, ctx=2731, low="bf16"),
        # hybrid with Mamba-2
        dict(name="step_mambay2_d16_4x4096", kind="step", family="mambay2", depth=16, batch=4, ctx=4096, low="bf16"),
    ]


def draw(rng):
    """Another run of the same ranges: family, depth, kind of pass, odd or even context and batch."""
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    family = rng.choice(["dense", "dense", "dense", "moe", "sambay", "sambay", "gdny", "mambay2", "phi4"])
    # passes that return activations are drawn where a correct implementation reproduces them to a few bf16 roundings
    # (not where routing, a recurrence over many layers or nearly empty softmax rows amplify them)
    kind = rng.choice(["step", "step", "score", "logits"]) if family in ("dense", "sambay") else "step"
    if kind != "step":
        depth = 8 if family == "dense" else rng.choice([8, 16])
    else:
        depth = {"moe": 8, "phi4": 8, "gdny": 16, "mambay2": 16}.get(family) or rng.choice([8, 12, 16])
    low = "fp8" if (family == "dense" and kind == "step" and rng.random() < 0.35) else "bf16"
    if kind == "logits":
        return dict(kind=kind, family=family, depth=depth, batch=rng.choice([1, 2, 4]), ctx=log(17, 1200), low=low)
    if family == "phi4":
        return dict(kind=kind, family=family, depth=depth, batch=1, ctx=log(700, 12288), low=low)
    most = 65536 if family == "moe" or depth == 8 else 32768 if depth == 12 else 24576 if family == "dense" else 16384
    tokens = log(900, most)
    ctx = min(log(200, 32768), tokens)
    if family == "dense" and rng.random() < 0.5:
        ctx = ctx // 8 * 8
    return dict(kind=kind, family=family, depth=depth, batch=max(tokens // ctx, 1), ctx=ctx, low=low)


# ------------------------------------------------------------------------------------------------ what a program has in hand
def _overrides(case):
    d = case["depth"]
    if case["family"] == "dense":
        return {"intermediate_size": d * 128 * 11 // 4}
    if case["family"] == "moe":
        return {"n_head": d, "n_query_groups": 2, "n_routed_experts": 64, "router_top_k": 8, "moe_intermediate_size": 256,
                "shared_intermediate_size": 2048}
    if case["family"] == "phi4":
        return {"n_layer": d, "ar": None, "n_embd": 2560, "n_head": 40, "n_query_groups": 20, "intermediate_size": 10240}
    return {}


def _tokens(case, seed, vocab, extra):
    g = torch.Generator(device="cuda").manual_seed(1_000_003 * seed + 17)
    T = case["ctx"] + extra
    x = torch.randint(3, vocab, (case["batch"], T), generator=g, device="cuda")
    if case["family"] == "phi4":
        # documents of lognormal length (mean 1500, sigma 1), clipped to [64, 8192], packed back to back
        r, pos = np.random.default_rng(seed), 0
        while True:
            pos += int(np.clip(r.lognormal(math.log(1500) - 0.5, 1.0), 64, 8192))
            if pos > T:
                break
            x[:, pos - 1] = EOS
    return x


def _eval_config(case):
    fam = FAMILIES[case["family"]]
    name = fam["model"] + ("_s8_k8" if case["family"] == "moe" else "") + "_d%d" % fam.get("fixed_depth", case["depth"])
    ov = dict(_overrides(case), mup=True, depth_scale=True, block_size=max(case["ctx"], 8), eos_token_id=EOS, head_init_std=0.02,
              qk_norm="qknorm" in fam["name"], use_muon=True, use_muonh=True)
    if case["family"] == "moe":
        ov.update(share_expert=True, sqrt_gate=True, global_aux=True, aux_gamma=0.01)
    if case["family"] == "phi4":
        ov.update(tied_embed=True, rope_base=640_000, use_cu_seqlen=True)
    return Config.from_name(name, **ov)


def prepare(case, seed):
    fam = FAMILIES[case["family"]]
    if case["kind"] in ("logits", "score"):
        # as eval.common.load_model leaves it: bf16 weights on the device, eval mode (random instead of trained values)
        cfg = _eval_config(case)
        torch.manual_seed(seed)
        with torch.device("cuda"):
            model = GPT(cfg)
        model.reset_parameters()
        torch.nn.init.normal_(model.transformer.wte.weight, std=0.02)
        model.to(torch.bfloat16).eval()
        model.compute_dtype = torch.bfloat16
        ids = _tokens(case, seed, cfg.vocab_size, 0)
        return dict(kind=case["kind"], model=ModelWrapper(model), ids=ids, loss=FusedLinearCrossEntropyLoss())
    os.environ.setdefault("LIGHTNING_ARTIFACTS_DIR", os.path.join(tempfile.gettempdir(), "archscale_b200_perf"))
    kw = dict(train_data_dir="synthetic", train_model=fam["model"], train_name=fam["name"], depth=fam.get("fixed_depth", case["depth"]),
              micro_bsz=case["batch"], ctx_len=case["ctx"], total_bsz=case["batch"] * case["ctx"], max_tokens=1e10, use_flce=True,
              config_overrides=_overrides(case), fp8=case["low"] == "fp8", return_trainer=True, quiet=True)
    if case["family"] == "moe":
        kw.update(sparsity=8, top_k=8, share_expert=True, sqrt_gate=True, global_aux=True, aux_gamma=0.01)
    trainer = setup(**kw)
    trainer.model.train()
    return dict(kind=case["kind"], trainer=trainer, batch=_tokens(case, seed, trainer.config.vocab_size, 1),
                lr=trainer.plan.learning_rate)


def run(state):
    if state["kind"] == "logits":
        with torch.no_grad():
            return state["model"](state["ids"]).logits
    if state["kind"] == "score":
        with torch.no_grad():
            ids = state["ids"]
            out = state["model"](ids, use_flce_loss=True)
            hidden = out.logits
            loss = state["loss"](hidden[:, :-1].reshape(-1, hidden.shape[-1]), out.weight, ids[:, 1:].reshape(-1))
            return {"hidden": hidden, "loss": loss}
    trainer = state["trainer"]
    loss, _ = trainer.forward_backward(state["batch"])
    trainer.optimizer_step(state["lr"])
    return {"loss": loss, "weights": [g.master for g in trainer.engine.groups()]}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
@functools.lru_cache(maxsize=None)
def _counts(family, depth):
    """(parameters, parameters a token multiplies with, of these the head's, Newton-Schulz FLOPs of one step)."""
    case = dict(family=family, depth=depth, ctx=128)
    cfg = _eval_config(case)
    with torch.device("meta"):
        model = GPT(cfg)
    ns = 0.0
    for name, p in model.named_parameters():
        if p.dim() >= 2 and "weight" in name and not any(k in name for k in ("conv1d", "wte", "lm_head", "norm", "ln")):
            m, n = sorted(p.shape[-2:])
            # per iteration: a symmetric Gram product, a symmetric square, the product with X
            ns += 5.0 * (p.numel() // (m * n)) * (1.0 * m * m * n + 1.0 * m ** 3 + 2.0 * m * m * n)
    total = sum(p.numel() for p in model.parameters())
    body = matmul_parameter_count(model, cfg)
    return total, body, cfg.padded_vocab_size * cfg.n_embd, ns, cfg


def work(case):
    total, body, head, ns, cfg = _counts(case["family"], case["depth"])
    n_tok, T = case["batch"] * case["ctx"], case["ctx"]
    pairs = 0.0                                    # visible (query, key) pairs per head and sequence, over the attention layers
    full = T * (T + 1) / 2.0
    if case["family"] == "phi4":
        full = n_tok * 0.5 * min(T, 3000.0)        # length-weighted mean document
    w = cfg.local_window
    win = full if w is None or w < 0 else min(full, float(T) * min(w, T))
    L = cfg.n_layer
    if case["family"] in ("dense", "moe"):
        pairs = L * full
    else:
        # first half: mixers (and windowed attention every other layer); second half: full / cross attention every other layer
        windowed = L // 4 if case["family"] in ("sambay", "phi4") else 0
        pairs = windowed * win + (L // 4) * full
    attn = case["batch"] * pairs * 4.0 * cfg.n_head * cfg.head_size
    fwd = 2.0 * (body + head) * n_tok + attn
    act = 2.0 * n_tok * cfg.n_embd
    if case["kind"] == "logits":
        return {"flops": fwd, "bytes": 2.0 * (total if case["family"] != "moe" else body + 2 * head) + 4.0 * n_tok * cfg.padded_vocab_size}
    if case["kind"] == "score":
        return {"flops": fwd, "bytes": 2.0 * total + 2 * act}
    flops = 3.0 * fwd + 0.5 * attn                 # the backward of attention recomputes the scores
    # weights read in forward and backward, gradients written, layer inputs kept and read again
    nbytes = 4.0 * total + 4.0 * total + 4.0 * L * act
    if case["kind"] == "step":
        flops += ns
        nbytes += 4.0 * total + 16.0 * total + 2.0 * total      # gradient read, master and momentum read and written, bf16 copy
    return {"flops": flops, "bytes": nbytes}


def tolerance(case):
    """Four times what kernels that are correct in other ways showed (split / single-kernel attention backward, one- and
    two-CTA GEMM tiles, library GEMMs and PyTorch forms of the element-wise ops): updated weights differ by 1e-4 (1e-3 where
    a router can flip), the loss by 2e-4; hidden states and logits by 0.008 (dense) to 0.018 (hybrid, 16 layers)."""
    if case["kind"] == "step":
        return {"rel": 4e-3, "max": 0.04} if case["family"] == "moe" else {"rel": 1e-3, "max": 0.02}
    return {"rel": 0.03, "max": 0.4}
