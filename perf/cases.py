"""The work that programs built on this framework have it do, as cases that can be timed and compared.

Kinds of cases (``case["kind"]``):

* ``gpt_train``  one training step of the FSDP GPT: forward, backward, fused Adam (``build_fsdp_gpt``, ``FusedAdam``)
* ``gpt_eval``   logits of the plain bf16 GPT without gradients (scoring, evaluation)
* ``llama_train``  one training step of the RMSNorm / RoPE / SwiGLU model on the model-parallel layers, one rank
* ``moe``        forward and backward of a top-2 mixture-of-experts layer with stacked experts
* ``attention``  forward and backward of causal attention on the packed QKV projection
* ``clip_adam``  global gradient norm, clipping, and the optimizer step over a model's list of parameters

Sizes are those of the flagship configuration, of the language-model, mixture-of-experts and tensor-parallel benchmarks,
of the tests, and odd ones in between.
"""

import math

import torch
import torch.distributed as dist

DEVICE = "cuda"


def _group():
    """The single-process group that a one-GPU program sets up before it wraps a model."""
    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    from fairscale_b200.nn import model_parallel

    if not model_parallel.model_parallel_is_initialized():
        model_parallel.initialize_model_parallel(1)


def listed():
    return [
        # a debugging-size model: what a step costs in launches and host work
        dict(name="gpt_train_tiny", kind="gpt_train", layers=2, d=128, heads=2, ffn=512, vocab=512, batch=2, seq=128, checkpoint=True),
        # a small model on sequences cut to an odd length, activations kept
        dict(name="gpt_train_ragged", kind="gpt_train", layers=6, d=768, heads=12, ffn=3072, vocab=10000, batch=5, seq=715, checkpoint=False),
        # the dense half of the mixture-of-experts benchmark: ordinary training, heads of 64
        dict(name="gpt_train_medium", kind="gpt_train", layers=12, d=1024, heads=16, ffn=4096, vocab=32000, batch=8, seq=1024, checkpoint=True),
        # the flagship benchmark's model and batch
        dict(name="gpt_train_1p3b", kind="gpt_train", layers=24, d=2048, heads=16, ffn=8192, vocab=50304, batch=8, seq=2048, checkpoint=True),
        # scoring one short prompt: a small number of rows through every matrix
        dict(name="gpt_eval_prompt", kind="gpt_eval", layers=12, d=1024, heads=16, ffn=4096, vocab=32000, batch=1, seq=77),
        # evaluating long documents whose length is no multiple of anything
        dict(name="gpt_eval_documents", kind="gpt_eval", layers=24, d=2048, heads=16, ffn=8192, vocab=50304, batch=3, seq=1990),
        # the tensor-parallel benchmark's layer sizes on one rank
        dict(name="llama_train", kind="llama_train", layers=4, d=4096, heads=32, ffn=11008, vocab=32000, batch=2, seq=2048),
        # the mixture-of-experts benchmark's layer and batch
        dict(name="moe_8_experts", kind="moe", experts=8, d=1024, ffn=4096, batch=8, seq=1024),
        # a small mixture with few tokens for each expert
        dict(name="moe_small", kind="moe", experts=4, d=512, ffn=2048, batch=4, seq=205),
        # long sequences with heads of 64
        dict(name="attention_long", kind="attention", batch=2, seq=8192, heads=16, head_dim=64),
        # heads of 128, odd length
        dict(name="attention_ragged", kind="attention", batch=4, seq=1543, heads=16, head_dim=128),
        # mixed-precision optimizer step over the matrices, biases and norms of a medium model
        dict(name="clip_adam", kind="clip_adam", layers=12, d=1024, ffn=4096, vocab=32000, dtype="bfloat16"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _of(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(_log(rng, lo, hi) / step)) * step))


def _seq(rng, lo, hi):
    """A sequence length: as often padded to a multiple of 128 as not padded at all."""
    return _of(rng, max(lo, 128), hi, 128) if rng.random() < 0.5 else _of(rng, lo, hi)


def draw(rng):
    kind = rng.choice(["gpt_train", "gpt_train", "gpt_train", "gpt_eval", "gpt_eval", "llama_train", "moe", "moe", "attention", "attention", "clip_adam"])
    head_dim = rng.choice([64, 128])
    if kind in ("gpt_train", "gpt_eval"):
        heads = _of(rng, 1, 2048 // head_dim)
        d = heads * head_dim
        layers = _of(rng, 1, 24)
        seq = _seq(rng, 16, 2048)
        tokens = _of(rng, seq, 16384)
        return dict(kind=kind, layers=layers, d=d, heads=heads, ffn=4 * d, vocab=_of(rng, 512, 50304, 64), batch=max(1, tokens // seq), seq=seq,
                    **({"checkpoint": rng.random() < 0.5} if kind == "gpt_train" else {}))
    if kind == "llama_train":
        heads = _of(rng, 2, 4096 // head_dim)
        d = heads * head_dim
        seq = _seq(rng, 32, 4096)
        return dict(kind=kind, layers=_of(rng, 1, 4), d=d, heads=heads, ffn=_of(rng, 2 * d, 3 * d, 8), vocab=_of(rng, 512, 32000, 64),
                    batch=max(1, _of(rng, seq, 8192) // seq), seq=seq)
    if kind == "moe":
        experts = rng.choice([2, 4, 8, 16])
        d = _of(rng, 256, 2048, 64)
        return dict(kind=kind, experts=experts, d=d, ffn=rng.choice([2, 4]) * d, batch=experts, seq=_of(rng, 16, 16384 // experts))
    if kind == "attention":
        seq = _seq(rng, 64, 8192)
        heads = _of(rng, 2, 32)
        batch = max(1, _of(rng, seq, 32768) // seq)
        return dict(kind=kind, batch=batch, seq=seq, heads=heads, head_dim=head_dim)
    d = _of(rng, 256, 2048, 8)
    return dict(kind=kind, layers=_of(rng, 1, 24), d=d, ffn=4 * d, vocab=_of(rng, 512, 50304), dtype=rng.choice(["float32", "bfloat16", "float16"]))


def _gpt_config(case):
    from fairscale_b200.models.gpt import GPTConfig

    return GPTConfig(case["vocab"], case["d"], case["heads"], case["layers"], case["ffn"], case["seq"])


def _tokens(case, gen):
    t = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), generator=gen, device=DEVICE)
    return t[:, :-1].contiguous(), t[:, 1:].contiguous()


def _randn(shape, gen, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=gen, device=DEVICE) * std).to(dtype)


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("gpt_train", "llama_train", "moe"):
        _group()
    if kind == "gpt_train":
        from fairscale_b200.models.gpt import build_fsdp_gpt
        from fairscale_b200.optim import FusedAdam

        with torch.device(DEVICE):
            model = build_fsdp_gpt(_gpt_config(case), torch.device(DEVICE, torch.cuda.current_device()), checkpoint_blocks=case["checkpoint"])
        state["opt"] = FusedAdam(model.parameters(), lr=1e-4, betas=(0.9, 0.95), eps=1e-8)
        model.attach_optimizer(state["opt"])
        state["model"], state["batch"] = model, _tokens(case, gen)
    elif kind == "gpt_eval":
        from fairscale_b200.models.gpt import GPT

        with torch.device(DEVICE):
            state["model"] = GPT(_gpt_config(case)).to(torch.bfloat16).eval()
        state["batch"] = _tokens(case, gen)
    elif kind == "llama_train":
        from fairscale_b200.models.tp_llama import TPLlama, TPLlamaConfig
        from fairscale_b200.optim import FusedAdam

        cfg = TPLlamaConfig(case["vocab"], case["d"], case["heads"], case["layers"], case["ffn"], case["seq"])
        with torch.device(DEVICE):
            model = TPLlama(cfg).to(DEVICE).to(torch.bfloat16)
        state["opt"] = FusedAdam(model.parameters(), lr=1e-4)
        state["model"], state["batch"] = model, _tokens(case, gen)
    elif kind == "moe":
        from fairscale_b200.nn.moe import GroupedExperts, MOELayer, Top2Gate

        with torch.device(DEVICE):
            gate = Top2Gate(case["d"], case["experts"])
            torch.nn.init.normal_(gate.wg.weight, 0.0, 0.02)
            state["model"] = MOELayer(gate, GroupedExperts(case["experts"], case["d"], case["ffn"])).to(torch.bfloat16)
        shape = (case["batch"], case["seq"], case["d"])
        state["x"] = _randn(shape, gen).requires_grad_()  # the output of a LayerNorm
        state["dy"] = _randn(shape, gen, 1e-3)
    elif kind == "attention":
        B, S, HD = case["batch"], case["seq"], case["heads"] * case["head_dim"]
        state["heads"] = case["heads"]
        state["x"] = _randn((B, S, 3 * HD), gen).requires_grad_()
        state["dy"] = _randn((B, S, HD), gen, 1e-2)
    elif kind == "clip_adam":
        from fairscale_b200.optim import FusedAdam

        dtype = getattr(torch, case["dtype"])
        params = []
        for shape in _model_shapes(case):
            p = torch.nn.Parameter(_randn(shape, gen, 0.02, dtype))
            p.grad = _randn(shape, gen, 1e-2, dtype)
            params.append(p)
        state["params"] = params
        state["opt"] = FusedAdam(params, lr=1e-4, weight_decay=0.01)
        state["max_norm"] = torch.ones((), device=DEVICE)
    return state


def _model_shapes(case):
    d, f = case["d"], case["ffn"]
    block = [(d,), (d,), (3 * d, d), (3 * d,), (d, d), (d,), (d,), (d,), (f, d), (f,), (d, f), (d,)]
    return [(case["vocab"], d)] + case["layers"] * block + [(d,), (d,), (case["vocab"], d)]


def run(state):
    kind = state["kind"]
    if kind in ("gpt_train", "llama_train"):
        model, opt = state["model"], state["opt"]
        loss = model(*state["batch"])
        loss.backward()
        opt.step()
        opt.zero_grad(set_to_none=True)
        return {"loss": loss.detach(), "weights": [p.detach() for p in model.parameters()]}
    if kind == "gpt_eval":
        with torch.no_grad():
            return state["model"](state["batch"][0])
    if kind == "moe":
        model, x = state["model"], state["x"]
        y = model(x)
        torch.autograd.backward([y, model.l_aux], [state["dy"], torch.full_like(model.l_aux, 0.01)])
        grads = [x.grad] + [p.grad for p in model.parameters()]
        x.grad = None
        model.zero_grad(set_to_none=True)
        return {"y": y.detach(), "l_aux": model.l_aux.detach(), "grads": grads}
    if kind == "attention":
        from fairscale_b200.ops.attention import causal_attention

        x = state["x"]
        y = causal_attention(x, state["heads"])
        y.backward(state["dy"])
        dx, x.grad = x.grad, None
        return {"y": y.detach(), "dx": dx}
    from fairscale_b200.ops import multi_tensor

    grads = [p.grad for p in state["params"]]
    norm = multi_tensor.l2_norm(grads)
    multi_tensor.scale_(grads, (state["max_norm"] / (norm + 1e-6)).clamp(max=1.0))
    state["opt"].step()
    # the largest kinds of parameter, whole: table, first block, head
    return {"norm": norm, "grads": grads[:13] + grads[-1:], "params": [p.detach() for p in state["params"][:13] + state["params"][-1:]]}


def _attention_work(batch, seq, heads, head_dim):
    """Causal: half of the score matrix; two products forward and five backward (the scores once again)."""
    one = 2.0 * batch * heads * head_dim * seq * (seq + 1) / 2
    return 2 * one, 5 * one


def work(case):
    kind = case["kind"]
    if kind == "clip_adam":
        n = sum(math.prod(s) for s in _model_shapes(case))
        size = {"float32": 4, "bfloat16": 2, "float16": 2}[case["dtype"]]
        # gradient read for the norm, read and written by the clipping; master weight and two fp32 moments read and
        # written; the low-precision weight written where it is not the master itself
        return {"bytes": n * (3 * size + 24 + (size if size == 2 else 0)), "flops": 20.0 * n}
    if kind == "attention":
        fwd, bwd = _attention_work(case["batch"], case["seq"], case["heads"], case["head_dim"])
        rows = case["batch"] * case["seq"] * case["heads"] * case["head_dim"]
        return {"bytes": 2.0 * rows * (3 + 1 + 1 + 3), "flops": fwd + bwd}
    T = case["batch"] * case["seq"]
    d = case["d"]
    if kind == "moe":
        weights = case["experts"] * 2 * d * case["ffn"]
        # every token visits two experts; forward and twice that backward
        return {"bytes": 2.0 * (2 * weights + 4 * T * d), "flops": 6.0 * 2 * T * 2 * d * case["ffn"]}
    head_dim = d // case["heads"]
    fwd, bwd = _attention_work(case["batch"], case["seq"], case["heads"], head_dim)
    L, V = case["layers"], case["vocab"]
    if kind == "gpt_eval":
        matrices = L * (4 * d * d + 2 * d * case["ffn"]) + V * d
        return {"bytes": 2.0 * (matrices + T * d + T * V), "flops": 2.0 * T * matrices + L * fwd}
    if kind == "gpt_train":
        block = L * (4 * d * d + 2 * d * case["ffn"])
        again = 1 if case["checkpoint"] else 0  # activation checkpointing is asked for: blocks run forward twice
        params = block + 2 * V * d
        # bf16 weights read and gradients written; fp32 master and moments read and written, bf16 weight written
        return {"bytes": params * (2.0 + 2 + 2 + 24 + 2), "flops": (6.0 + 2 * again) * T * block + 6.0 * T * V * d + L * ((1 + again) * fwd + bwd)}
    matrices = L * (4 * d * d + 3 * d * case["ffn"]) + V * d
    return {"bytes": (matrices + V * d) * (2.0 + 2 + 2 + 24 + 2), "flops": 6.0 * T * matrices + L * (fwd + bwd)}


def tolerance(case):
    """About four times what the path shows against the same computation in fp32 on the same bf16 weights."""
    kind = case["kind"]
    if kind in ("gpt_train", "llama_train"):
        # Weights after a step of 1e-4 on matrices of 0.02: a weight whose gradient is lost in the bf16 noise (1 to 1.5 %
        # of the gradient) steps the other way, 2e-4.  Measured 3e-4 (2 layers) to 6e-4 (24 layers), largest 0.01.
        return {"rel": 2.5e-3, "max": 0.06}
    if kind == "gpt_eval":
        return {"rel": 0.025, "max": 0.3}  # measured 0.009 to 0.012, largest 0.07
    if kind == "moe":
        return {"rel": 0.012, "max": 0.1}  # measured 0.004, largest 0.022
    if kind == "attention":
        return {"rel": 0.01, "max": 0.5}  # measured 0.0024, largest 0.145
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 1e-3, "max": 0.02}  # a last bit of a 16-bit weight or gradient
