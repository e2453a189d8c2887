"""The work whose speed counts: training steps, scoring and text generation of the model families this framework ships
configurations for, called the way a user's program calls them.

A training case is one ``gpt_neox_b200.training.train_step``: every micro-batch of the step forward and backward, gradient
clipping, the Adam update of the fp32 masters and the learning-rate schedule.  A scoring case is one forward of a batch of
token sequences to logits.  A generation case is one ``gpt_neox_b200.text_generation.stream_tokens`` call run to its last
token: the prompt pass and every decoding step.  Models have random weights of the configuration's architecture; token ids
are uniform over the vocabulary.
"""
from __future__ import annotations

import math

import torch

from gpt_neox_b200.config import NeoXArgs
from gpt_neox_b200.initialize import initialize_megatron
from gpt_neox_b200.text_generation import forward_model, stream_tokens
from gpt_neox_b200.training import setup_model_and_optimizer, train_step
from gpt_neox_b200.utils import Timers


def _case(name, kind, arch, **over):
    """``kind``: train | score | generate.  ``arch``: neox (parallel residual, LayerNorm, GeLU, partial rotary),
    gpt (the same with the sequential residual and full rotary), llama (RMSNorm, SwiGLU, no biases, full rotary,
    optionally grouped queries and a sliding window), mamba, rwkv."""
    c = {"name": name, "kind": kind, "arch": arch, "dtype": "bfloat16", "layers": 2, "hidden": 512, "heads": 8,
         "kv_heads": 0, "window": 0, "ffn": 0, "vocab": 50304, "seq": 2048, "batch": 1, "accum": 1, "recompute": False,
         "prompt": 0, "shortest": 0, "new": 0, "graph": False, "temperature": 0.0}
    c.update(over)
    return c


def listed():
    return [
        # Short fine-tuning samples on the smallest model with a supported head size (configs/pythia/70M.yml, fp16 with
        # loss scaling): the step is a few hundred small launches.
        _case("train_70m_short", "train", "neox", dtype="fp16", layers=6, seq=512),
        # Pre-training of the smallest GPT (configs/bf16_125M.yml: micro-batch 4 of 2048 tokens, activations recomputed).
        _case("train_125m", "train", "gpt", layers=12, hidden=768, heads=12, batch=4, recompute=True),
        # A mid-size model in fp16 (configs/pythia/410M.yml) on batches of a length no tile divides.
        _case("train_410m_ragged", "train", "neox", dtype="fp16", layers=24, hidden=1024, heads=16, seq=1927, batch=3),
        # The headline model (configs/20B.yml: hidden 6144, 64 heads of 96, micro-batch 4, activations recomputed), as
        # many layers as let several copies with their optimizer state fit one GPU; two accumulation steps.
        _case("train_20b_layers", "train", "neox", layers=2, hidden=6144, heads=64, vocab=50432, batch=4, accum=2,
              recompute=True),
        # Long sequences with grouped-query, windowed attention (configs/mistral/7B.yml: 32 / 8 heads, window 4096, 8192
        # tokens), two of its layers.
        _case("train_mistral_layers", "train", "llama", layers=2, hidden=4096, heads=32, kv_heads=8, window=4096,
              ffn=14336, vocab=32000, seq=8192, recompute=True),
        # Selective state-space model (configs/mamba/mamba-130M.yml) in bf16.
        _case("train_mamba_130m", "train", "mamba", layers=24, hidden=768, heads=12, batch=4),
        # RWKV-6 (configs/rwkv/170M.yml: micro-batch 4 of 512 tokens) in bf16.
        _case("train_rwkv_170m", "train", "rwkv", layers=12, hidden=768, heads=12, seq=512, batch=4),
        # Evaluation: log-likelihoods of a few harness requests of odd length (configs/pythia/1-4B.yml, head size 128).
        _case("score_1b4", "score", "neox", layers=24, hidden=2048, heads=16, seq=777, batch=3),
        # One interactive request: a short prompt, greedy, as generate.py runs by default (configs/pythia/410M.yml).
        _case("generate_410m_one", "generate", "neox", dtype="fp16", layers=24, hidden=1024, heads=16, prompt=37,
              shortest=37, new=48),
        # A batch of prompts of different lengths, sampled (configs/text_generation.yml: temperature 1).
        _case("generate_1b4_batch", "generate", "neox", layers=24, hidden=2048, heads=16, batch=8, prompt=96, shortest=64,
              new=48, temperature=1.0),
        # The same model behind the CUDA-graph decoder (``cuda_graph_decode``), longer prompts.
        _case("generate_1b4_graph", "generate", "neox", layers=24, hidden=2048, heads=16, batch=4, prompt=520,
              shortest=500, new=64, graph=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    limit = max(work(c)["flops"] for c in listed())
    while True:
        arch = rng.choice(["neox", "neox", "gpt", "llama", "mamba", "rwkv"])
        kind = rng.choice(["train", "train", "score", "generate"]) if arch in ("neox", "gpt", "llama") else "train"
        c = _case("", kind, arch)
        del c["name"]
        head = rng.choice([64, 128]) if arch == "llama" else rng.choice([64, 96, 128])
        if arch in ("mamba", "rwkv"):
            c["hidden"] = 128 * rng.randint(2, 16)
            c["heads"] = c["hidden"] // 64
        else:
            c["heads"] = 4 * _log_uniform(rng, 1, 16)
            c["hidden"] = head * c["heads"]
            c["dtype"] = rng.choice(["bfloat16", "bfloat16", "fp16"])
        c["layers"] = _log_uniform(rng, 2, 24)
        c["vocab"] = rng.choice([32000, 50304, 50432])
        if arch == "llama":
            c["kv_heads"] = rng.choice([0, c["heads"] // 4])
            c["window"] = rng.choice([0, 0, _log_uniform(rng, 128, 4096)])
            c["ffn"] = 256 * max(1, round(c["hidden"] * 8 / 3 / 256))
        if kind == "generate":
            c["batch"] = _log_uniform(rng, 1, 16)
            c["prompt"] = _log_uniform(rng, 8, 768)
            c["new"] = rng.randint(8, 64)
            c["shortest"] = max(1, c["prompt"] - rng.randint(0, c["new"] // 2)) if c["batch"] > 1 else c["prompt"]
            c["graph"] = rng.random() < 0.4 and c["window"] == 0
            c["temperature"] = rng.choice([0.0, 1.0])
            if c["layers"] * c["new"] > 1600:
                continue
        else:
            c["seq"] = _log_uniform(rng, 128, 2048 if arch in ("mamba", "rwkv") else 8192)
            c["batch"] = _log_uniform(rng, 1, 8)
            c["accum"] = rng.choice([1, 1, 2]) if kind == "train" else 1
            c["recompute"] = kind == "train" and rng.random() < 0.5
        tokens = c["batch"] * c["seq"]
        if _params(c) <= 1.4e9 and work(c)["flops"] <= limit and (kind == "generate" or tokens <= 16384):
            return c


def _mlp(c):
    return 3 * c["hidden"] * c["ffn"] if c["arch"] == "llama" else 8 * c["hidden"] ** 2


def _layer_params(c):
    h = c["hidden"]
    if c["arch"] == "mamba":
        inner, rank = 2 * h, math.ceil(h / 16)
        return 2 * h * inner + inner * (rank + 32) + rank * inner + inner * h + inner * 16
    if c["arch"] == "rwkv":
        return 5 * h * h + (2 * int(3.5 * h) + h) * h + 320 * h + 128 * h
    kv = (c["kv_heads"] or c["heads"]) * (h // c["heads"])
    return 2 * h * h + 2 * h * kv + _mlp(c)


def _params(c):
    return c["layers"] * _layer_params(c) + (1 if c["arch"] == "mamba" else 2) * c["vocab"] * c["hidden"]


def _pairs(c, seq):
    """Query-key pairs one causal (windowed) sequence attends to."""
    w = c["window"]
    if w and w + 1 < seq:
        return (w + 1) * (w + 2) // 2 + (seq - w - 1) * (w + 1)
    return seq * (seq + 1) // 2


def _mixer_flops(c, seq):
    """Forward operations of one layer's sequence mixing over one sequence, projections apart."""
    h = c["hidden"]
    if c["arch"] == "mamba":
        return seq * 2 * h * (16 * 6 + 16)
    if c["arch"] == "rwkv":
        return seq * h * 64 * 5
    return 4 * h * _pairs(c, seq)


def work(case):
    c = case
    n_head = c["vocab"] * c["hidden"]
    n_layers = c["layers"] * _layer_params(c)
    if c["kind"] == "generate":
        # prompt pass over the shortest prompt, then one step per token; every step reads all weights, and the cache of
        # keys and values as far as it is filled, and writes one row of it and the logits of the batch
        kv = 2 * (c["kv_heads"] or c["heads"]) * (c["hidden"] // c["heads"]) * c["layers"] * 2 * c["batch"]
        steps, first = c["new"], c["shortest"]
        filled = sum(first + i for i in range(steps))
        flops = 2.0 * (n_layers * c["batch"] * (first + steps - 1) + n_head * c["batch"] * steps)
        flops += c["layers"] * c["batch"] * 4 * c["hidden"] * (_pairs(c, first) + filled)
        return {"bytes": 2.0 * (n_layers + n_head) * steps + kv * (filled + first + steps) + 4.0 * c["vocab"] * steps,
                "flops": flops}
    tokens = c["batch"] * c["seq"] * c["accum"]
    flops = 2.0 * tokens * (n_layers + n_head) + c["layers"] * c["batch"] * c["accum"] * float(_mixer_flops(c, c["seq"]))
    if c["kind"] == "score":
        return {"bytes": 2.0 * (n_layers + n_head) + 2.0 * tokens * c["vocab"] + 2.0 * tokens * c["hidden"], "flops": flops}
    # backward costs twice the forward; the optimizer reads and writes master, both moments, and writes the 16-bit weights
    return {"bytes": 26.0 * _params(c) + 8.0 * tokens, "flops": 3.0 * flops}


def tolerance(case):
    # Between this code's kernels and alternatives of the same precision (library GEMMs with a separate GeLU, the other
    # generation of attention kernels) the listed cases differ by 0.0144 (moments, logits) in bf16 and 0.0021 in fp16, single
    # elements by 0.36 and 0.039: 16-bit activations rounded in another order and carried through all layers.  Four times
    # that, as far as a bound still means something.  The tokens of a generation stay the same.
    if case["dtype"] == "fp16":
        return {"rel": 0.0085, "max": 0.16, "differ": 0.0}
    return {"rel": 0.03, "max": 0.95, "differ": 0.0}


def _config(c, seed):
    train = c["kind"] == "train"
    length = c["seq"] if c["kind"] != "generate" else 2048
    d = {
        "num_layers": c["layers"], "hidden_size": c["hidden"], "num_attention_heads": c["heads"], "seq_length": length,
        "max_position_embeddings": max(length, 2048), "pos_emb": "rotary", "rotary_pct": 0.25, "no_weight_tying": True,
        "gpt_j_residual": c["arch"] == "neox", "output_layer_parallelism": "column", "norm": "layernorm",
        "attention_config": [[["flash"], "all"]], "scaled_upper_triang_masked_softmax_fusion": True,
        "bias_gelu_fusion": True, "init_method": "small_init", "output_layer_init_method": "wang_init",
        "optimizer": {"type": "Adam", "params": {"lr": 3.0e-4, "betas": [0.9, 0.95], "eps": 1.0e-8}}, "min_lr": 3.0e-5,
        "zero_optimization": {"stage": 1}, "train_micro_batch_size_per_gpu": c["batch"],
        "gradient_accumulation_steps": c["accum"], "checkpoint_activations": c["recompute"], "checkpoint_num_layers": 1,
        "gradient_clipping": 1.0, "weight_decay": 0.1, "hidden_dropout": 0.0, "attention_dropout": 0.0,
        "train_iters": 143000, "lr_decay_iters": 143000, "lr_decay_style": "cosine", "warmup": 0.01,
        "data_path": "synthetic", "tokenizer_type": "CharLevelTokenizer", "make_vocab_size_divisible_by": 128,
        "log_interval": 10 ** 9, "eval_interval": 10 ** 9, "eval_iters": 1, "checkpoint_factor": 10 ** 9,
        "num_workers": 0, "seed": 1 + seed % (2 ** 31 - 2), "global_num_gpus": 1, "distributed_backend": "nccl",
    }
    if c["dtype"] == "fp16":
        d["fp16"] = {"fp16": True, "enabled": True, "loss_scale": 0, "loss_scale_window": 1000, "initial_scale_power": 12,
                     "hysteresis": 2, "min_loss_scale": 1}
    else:
        d["precision"] = "bfloat16"
    if c["arch"] in ("gpt", "llama"):
        d["rotary_pct"] = 1.0
    if c["arch"] == "llama":
        d.update(norm="rmsnorm", rms_norm_epsilon=1.0e-5, activation="swiglu", intermediate_size=3 * c["ffn"],
                 mlp_multiple_of=256, use_bias_in_mlp=False, use_bias_in_attn_linear=False, use_bias_in_norms=False,
                 bias_gelu_fusion=False)
        if c["kv_heads"]:
            d["num_kv_heads"] = c["kv_heads"]
        if c["window"]:
            d["sliding_window_width"] = c["window"]
    if c["arch"] in ("mamba", "rwkv"):
        d.update(norm="rmsnorm", rms_norm_epsilon=1.0e-5, pos_emb="none", attention_config=[[[c["arch"]], "all"]],
                 bias_gelu_fusion=False)
    if c["arch"] == "mamba":
        d.update(mamba_selective_scan_fusion=True, mamba_causal_conv_fusion=True, mamba_inner_func_fusion=False,
                 mamba_selective_fp32_params=True, mamba_use_bias_in_conv=True, mamba_use_bias_in_linears=False,
                 no_weight_tying=False)
    if c["arch"] == "rwkv":
        d.update(activation="silu")
    if not train:
        d.update(optimizer=None, no_load_optim=True)
    if c["kind"] == "generate":
        d.update(return_logits=True, cuda_graph_decode=c["graph"])
    return d


def _continue_last_token(model):
    """Embeddings and projection under which a model continues with the token it has just read, by a wide margin and on top
    of what its layers add: a generation is then the same token for token under another rounding, as with a trained model
    that is sure of its answer, and the logits still carry every layer's contribution."""
    layers = list(model.module.sequential)
    emb, out = layers[0].word_embeddings.weight, layers[-1].final_linear.weight
    with torch.no_grad():
        emb.mul_(0.5 / emb.float().std())
        out.copy_(emb * (0.08 * math.sqrt(1024.0 / emb.shape[1])))


class _State(dict):
    """What a program holds for one model.  The optimizer's gradient hooks tie parameters and buckets together in a ring
    that outlives them: a program that builds one model after another takes the hooks off when it is done with one."""

    def __del__(self):
        if self.get("optimizer") is not None:
            for hook in self["optimizer"]._hooks:
                hook.remove()


def prepare(case, seed):
    c = case
    args = NeoXArgs.from_dict(_config(c, seed))
    args.configure_distributed_args()
    args.build_tokenizer()
    args.padded_vocab_size = c["vocab"]
    initialize_megatron(args)
    model, optimizer, scheduler, _ = setup_model_and_optimizer(args, use_cache=c["kind"] == "generate")
    g = torch.Generator().manual_seed(seed)
    state = _State(case=c, args=args, model=model)
    if c["kind"] == "train":
        model.train()
        batches = [torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=g).cuda() for _ in range(c["accum"])]

        def stream():
            while True:
                for b in batches:
                    yield {"text": b}

        state.update(optimizer=optimizer, scheduler=scheduler, data=stream(), timers=Timers())
    elif c["kind"] == "score":
        model.eval()
        model.module.inference_mode(use_cache=False)
        tokens = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g).cuda()
        state.update(tokens=tokens, positions=torch.arange(c["seq"], device="cuda").expand(c["batch"], -1))
    else:
        model.eval()
        model.module.inference_mode(use_cache=True)
        _continue_last_token(model)
        lengths = [c["prompt"], c["shortest"]][: c["batch"]]
        while len(lengths) < c["batch"]:
            lengths.append(int(torch.randint(c["shortest"], c["prompt"] + 1, (1,), generator=g)))
        state["prompts"] = [torch.randint(300, c["vocab"], (n,), generator=g).tolist() for n in lengths]
    return state


def run(state):
    c, args, model = state["case"], state["args"], state["model"]
    if c["kind"] == "train":
        metrics, _ = train_step(args, state["timers"], state["data"], model, state["optimizer"], state["scheduler"])
        opt = state["optimizer"]
        moments = [opt.optimizer.state[b.master] for b in opt.buckets]
        return {"loss": metrics["lm_loss"], "weights": [b.flat_param for b in opt.buckets],
                "masters": [b.master for b in opt.buckets], "exp_avg": [m["exp_avg"] for m in moments],
                "exp_avg_sq": [m["exp_avg_sq"] for m in moments]}
    if c["kind"] == "score":
        with torch.no_grad():
            return forward_model(model, (state["tokens"], state["positions"], None))
    last = None
    for last in stream_tokens(args, model, state["prompts"], maximum_tokens=c["new"], temperature=c["temperature"]):
        pass
    tokens, _, ends, logits, _ = last
    return {"tokens": tokens, "ends": ends, "logits": logits}
