"""Timed cases: the work a training job has this package do on one GPU, through the package's public entry points.

``listed()`` are the named cases, ``draw(rng)`` gives another one of the same ranges, ``prepare`` makes what a program
holds before the call, ``run`` is one pass, ``work`` the bytes and operations the pass cannot do without, and
``tolerance`` how far two correct implementations of it may be apart.

Kinds of case
  step      one minibatch through the sharded decoder engine: gradients of all microbatches in the accumulators
  layer     one decoder layer, forward and backward (weights held in bf16)
  attention packed causal attention on a fused qkv activation, forward and backward
  loss      LM head + weighted cross-entropy, forward and backward
  logprobs  LM head per-token log-probabilities with a temperature, forward and backward
  score     log-probabilities of given tokens by the whole decoder, forward only (evaluation, reference policy)
  adamw     optimizer update of a flat fp32 shard and its bf16 copy
  unit      gather one sharded unit, scatter-accumulate its gradient, synchronise

Sequence lengths belong to the case (``lengths`` seeds them), values belong to the seed given to ``prepare``.
"""
import math
import random

import numpy as np
import torch

import odc_b200 as odc
from odc_b200 import ops
from odc_b200.data import LengthSpec
from odc_b200.data.synthetic import pack_microbatch, sample_until_budget
from odc_b200.models import DecoderLayer, DecoderLM, get_config
from odc_b200.parallel import FusedDecoderLM

# the package's presets, and the small decoder its smoke test trains
SMOKE = dict(hidden_size=512, intermediate_size=1536, num_heads=8, num_kv_heads=2, vocab_size=4096)
MODELS = {
    "smoke": lambda: get_config("tiny", **SMOKE),
    "llama3.2-1b": lambda: get_config("llama3.2-1b"),
    "llama3-8b": lambda: get_config("llama3-8b"),
    "qwen2.5-1.5b": lambda: get_config("qwen2.5-1.5b"),
    "qwen2.5-14b": lambda: get_config("qwen2.5-14b"),
}
# how long the packed sequences are: the benchmark's three workloads, the smoke test's, and one single sequence
MIXES = {
    "headline": LengthSpec("lognormal", lo=16, median=512.0, sigma=1.0, cap=8192),
    "wide": LengthSpec("lognormal", lo=16, median=1024.0, sigma=1.2, cap=16384),
    "longtail": LengthSpec("longtail", short=(256, 2048), long=(8192, 32768), long_frac=0.25),
    "short": LengthSpec("uniform", lo=64, hi=512),
    "one": None,
}


def listed():
    return [
        # the smallest training step (smoke and parity runs): launches and host work are all of it
        dict(name="step smoke", kind="step", model="smoke", layers=2, mix="short", budget=2048, microbatches=2, lengths=1),
        # the headline step, cut to four of its layers: embedding, layers, LM head, gradient accumulation over microbatches
        dict(name="step 1b", kind="step", model="llama3.2-1b", layers=4, mix="headline", budget=16384, microbatches=2, lengths=2),
        # what the headline step spends most of its time in
        dict(name="layer 1b 16k", kind="layer", model="llama3.2-1b", mix="headline", budget=16384, lengths=3),
        # a layer of the hybrid-sharded configuration: head dimension 128, 32k-token packs
        dict(name="layer 8b 32k", kind="layer", model="llama3-8b", mix="wide", budget=32768, lengths=4),
        # the last, short pack of a minibatch, with qkv bias: few rows, weights and launches dominate
        dict(name="layer 1.5b 1k", kind="layer", model="qwen2.5-1.5b", mix="headline", budget=1024, lengths=5),
        # one long rollout of the long-tail configuration
        dict(name="attention 14b 32k", kind="attention", model="qwen2.5-14b", mix="one", budget=32768, lengths=0),
        # the loss of one headline microbatch
        dict(name="loss 1b 16k", kind="loss", model="llama3.2-1b", mix="headline", budget=16384, lengths=6),
        # the policy-gradient form of the head, a medium pack, temperature below one
        dict(name="logprobs 1.5b 6k", kind="logprobs", model="qwen2.5-1.5b", mix="headline", budget=6000, lengths=7, temperature=0.8),
        # scoring a pack of rollouts with the whole 1B decoder
        dict(name="score 1b 16k", kind="score", model="llama3.2-1b", layers=16, mix="headline", budget=16384, lengths=8),
        # one rank's eighth of the 1B parameters
        dict(name="adamw 154m", kind="adamw", numel=154476800, grad="fp32"),
        # all norm weights of the 1B decoder: latency of the primitives
        dict(name="unit 68k", kind="unit", numel=67584, shard="bf16", grad="fp32"),
        # one 1B decoder layer
        dict(name="unit 61m", kind="unit", numel=60821504, shard="bf16", grad="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "layer", "layer", "attention", "loss", "logprobs", "score", "adamw", "unit", "unit"])
    c = dict(kind=kind, lengths=rng.randrange(1 << 20))
    packs = ["headline", "headline", "wide", "short", "longtail", "one"]
    if kind == "step":
        c.update(model=rng.choice(["smoke", "llama3.2-1b"]), layers=rng.randint(1, 4), mix=rng.choice(packs), microbatches=rng.randint(1, 2))
        c.update(budget=_log(rng, 256, 12288 if c["model"] != "smoke" else 8192))
    elif kind == "layer":
        c.update(model=rng.choice(["llama3.2-1b", "llama3-8b", "qwen2.5-1.5b", "qwen2.5-14b"]), mix=rng.choice(packs))
        c.update(budget=_log(rng, 256, 32768 if c["model"] != "qwen2.5-14b" else 16384))
    elif kind == "attention":
        c.update(model=rng.choice(["llama3.2-1b", "llama3-8b", "qwen2.5-1.5b", "qwen2.5-14b"]), mix=rng.choice(packs),
                 budget=_log(rng, 512, 32768))
    elif kind == "loss":
        c.update(model=rng.choice(["llama3.2-1b", "llama3-8b", "qwen2.5-1.5b"]), mix=rng.choice(packs), budget=_log(rng, 256, 16384))
    elif kind == "logprobs":
        c.update(model=rng.choice(["llama3.2-1b", "qwen2.5-1.5b"]), mix=rng.choice(packs), budget=_log(rng, 256, 16384),
                 temperature=rng.choice([1.0, 0.8, 0.6]))
    elif kind == "score":
        c.update(model=rng.choice(["smoke", "llama3.2-1b"]), layers=rng.randint(2, 16), mix=rng.choice(packs), budget=_log(rng, 256, 16384))
    elif kind == "adamw":
        c.update(numel=_log(rng, 2000000, 154476800), grad=rng.choice(["fp32", "fp32", "bf16"]))
        del c["lengths"]
    else:
        # shards are padded to whole 16-byte pieces by every engine
        c.update(numel=max(8, _log(rng, 8192, 67108864) // 8 * 8), shard=rng.choice(["bf16", "bf16", "fp32"]), grad=rng.choice(["fp32", "bf16"]))
        del c["lengths"]
    return c


# ---------------------------------------------------------------------------------------------------------------------
def _config(case):
    cfg = MODELS[case["model"]]()
    if "layers" in case:
        cfg.num_layers = case["layers"]
    return cfg


def _lengths(case, pack=0):
    if case["mix"] == "one":
        return [case["budget"]]
    return sample_until_budget(MIXES[case["mix"]], case["budget"], np.random.default_rng([case["lengths"], pack]))


def _randn(gen, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(mean, std, generator=gen)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _pack(case, seed, vocab, pack=0, packs=1):
    """One packed microbatch on the GPU, as the trainers hold it after the copy from the host."""
    lens = _lengths(case, pack)
    rng = np.random.default_rng([seed, pack])
    mb = pack_microbatch([torch.from_numpy(rng.integers(0, vocab, size=n)) for n in lens], len(lens) * packs)
    return {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in mb.items()}


class _Session:
    """The one symmetric heap of the process and what lives on it: an engine, or the two primitive services.

    A training job has one model and many minibatches, so states of one case share it; it is rebuilt for another one.
    """

    current = None

    def __init__(self, key, cfg=None):
        odc.init_nvshmem(torch.device("cuda", 0))
        self.key, self.engine, self.free = key, None, {}
        if cfg is not None:
            self.engine = FusedDecoderLM(cfg, device=torch.device("cuda", 0), seed=0)
        else:
            self.gather = odc.GatherService()
            self.reduction = odc.ReductionService(accumulation_dtype=torch.float32)
            self.units = 0

    @classmethod
    def get(cls, key, cfg=None):
        if cls.current is None or cls.current.key != key:
            old, cls.current = cls.current, None
            if old is not None:
                torch.cuda.synchronize()
                if old.engine is not None:
                    old.engine.stop()
                else:
                    old.reduction.stop()
                    odc.finalize_distributed()
                old.engine = None
                torch.cuda.empty_cache()
            cls.current = cls(key, cfg)
        return cls.current


class _Unit:
    """Symmetric buffers of one sharded unit; they go back to the session's pool with the state that used them."""

    def __init__(self, session, numel, dtype):
        self.pool = session.free.setdefault((numel, dtype), [])
        if self.pool:
            self.key, self.shard, self.acc = self.pool.pop()
        else:
            session.units += 1
            self.key = f"unit{session.units}"
            self.shard = odc.SymmBufferRegistry.get_instance().allocate_symm_buffer(self.key, (numel,), dtype)
            self.acc = session.reduction.register(self.key, numel, torch.float32)

    def __del__(self):
        self.pool.append((self.key, self.shard, self.acc))


DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    s = {"kind": kind}
    if kind == "adamw":
        n = case["numel"]
        s["p"] = _randn(gen, n, std=0.02, dtype=torch.float32)
        s["m"] = _randn(gen, n, std=1e-4, dtype=torch.float32)
        s["v"] = _randn(gen, n, std=1e-4, dtype=torch.float32).square_()
        s["g"] = _randn(gen, n, std=1e-4, dtype=DTYPES[case["grad"]])
        s["low"] = s["p"].to(torch.bfloat16)
        return s
    if kind == "unit":
        n, dtype = case["numel"], DTYPES[case["shard"]]
        s["session"] = _Session.get("primitives")
        s["unit"] = _Unit(s["session"], n, dtype)
        s["unit"].shard.normal_(0.0, 0.02, generator=gen)
        s["unit"].acc.zero_()
        s["full"] = torch.empty(n, dtype=torch.bfloat16, device="cuda")
        s["grad"] = _randn(gen, n, std=1e-3, dtype=DTYPES[case["grad"]])
        return s
    cfg = _config(case)
    if kind == "step":
        key = ("engine",) + tuple((k, case[k]) for k in ("model", "layers"))
        s["engine"] = _Session.get(key, cfg).engine
        s["packs"] = [_pack(case, seed, cfg.vocab_size, i, case["microbatches"]) for i in range(case["microbatches"])]
        return s
    mb = _pack(case, seed, cfg.vocab_size)
    T, H = mb["num_tokens"], cfg.hidden_size
    s["mb"] = mb
    if kind == "score":
        with torch.device("cuda"):
            model = DecoderLM(cfg)
        model.reset_parameters(seed=seed)
        s["model"] = model.bfloat16()
    elif kind == "layer":
        with torch.device("cuda"):
            layer = DecoderLayer(cfg).bfloat16()
        with torch.no_grad():
            for name, p in layer.named_parameters():
                if p.dim() == 2:
                    p.normal_(0.0, cfg.init_std, generator=gen)
                else:
                    p.normal_(1.0 if "norm" in name else 0.0, 0.1, generator=gen)
        s["layer"], s["params"] = layer, list(layer.parameters())
        s["x"] = _randn(gen, T, H).requires_grad_()
        s["dy"] = _randn(gen, T, H, std=1e-2)
    elif kind == "attention":
        s["cfg"] = cfg
        s["qkv"] = _randn(gen, T, cfg.qkv_dim).requires_grad_()
        s["do"] = _randn(gen, T, cfg.num_heads, cfg.head_dim, std=1e-2)
    else:
        s["h"] = _randn(gen, T, H).requires_grad_()
        s["w"] = _randn(gen, cfg.vocab_size, H, std=cfg.init_std).requires_grad_()
        if kind == "logprobs":
            s["temperature"] = case["temperature"]
            s["dlogp"] = _randn(gen, T, std=1e-3, dtype=torch.float32)
    return s


def run(s):
    kind = s["kind"]
    if kind == "adamw":
        ops.fused_adamw_(s["p"], s["g"], s["m"], s["v"], s["low"], 1e-4, 0.9, 0.999, 1e-8, 0.01, 10, 1.0)
        return [s["p"], s["m"], s["v"], s["low"]]
    if kind == "unit":
        session, unit = s["session"], s["unit"]
        session.gather.gather_into_tensor(s["full"], unit.shard)
        session.reduction.scatter_accumulate(unit.key, s["grad"])
        session.reduction.sync()
        return [s["full"], unit.acc]
    if kind == "step":
        engine, total = s["engine"], None
        engine.start_minibatch()
        for mb in s["packs"]:
            loss = engine(mb["input_ids"], mb["position_ids"], mb["cu_seqlens"], mb["max_seqlen"], labels=mb["labels"],
                          loss_scale=mb["loss_scale"])
            loss.backward()
            total = loss.detach() if total is None else total + loss.detach()
        engine.finish_minibatch()
        return [total] + [group.flat()[1] for group in engine.optimizer_groups()]
    mb = s["mb"]
    where = (mb["position_ids"], mb["cu_seqlens"], mb["max_seqlen"])
    if kind == "score":
        with torch.no_grad():
            return s["model"](mb["input_ids"], *where, labels=mb["labels"], return_logprobs=True)
    if kind == "layer":
        y = s["layer"](s["x"], *where)
        return [y.detach(), *torch.autograd.grad(y, [s["x"], *s["params"]], s["dy"])]
    if kind == "attention":
        c = s["cfg"]
        o = ops.varlen_attention_qkv(s["qkv"], c.num_heads, c.num_kv_heads, c.head_dim, *where[1:])
        return [o.detach(), *torch.autograd.grad(o, [s["qkv"]], s["do"])]
    if kind == "loss":
        loss = ops.linear_cross_entropy(s["h"], s["w"], mb["labels"], mb["loss_scale"])
        return [loss.detach(), *torch.autograd.grad(loss, [s["h"], s["w"]])]
    logp = ops.linear_token_logprobs(s["h"], s["w"], mb["labels"], s["temperature"])
    return [logp.detach(), *torch.autograd.grad(logp, [s["h"], s["w"]], s["dlogp"])]


# ---------------------------------------------------------------------------------------------------------------------
def _layer_params(cfg):
    h, f = cfg.hidden_size, cfg.intermediate_size
    return cfg.qkv_dim * h + h * cfg.num_heads * cfg.head_dim + 3 * h * f


def _attention_flops(cfg, lens):
    """Forward: two products over the visible half of every score matrix."""
    return 4.0 * cfg.num_heads * cfg.head_dim * sum(n * (n + 1) / 2 for n in lens)


def work(case):
    kind = case["kind"]
    if kind == "adamw":
        n, g = case["numel"], 4 if case["grad"] == "fp32" else 2
        return {"bytes": n * (12 + g + 12 + 2), "flops": 15.0 * n}
    if kind == "unit":
        n = case["numel"]
        size = {"fp32": 4, "bf16": 2}
        return {"bytes": n * (size[case["shard"]] + 2 + size[case["grad"]] + 8), "flops": float(n)}
    cfg = _config(case)
    H, V = cfg.hidden_size, cfg.vocab_size
    if kind == "step":
        flops = 0.0
        for i in range(case["microbatches"]):
            lens = _lengths(case, i)
            flops += 6.0 * sum(lens) * (cfg.num_layers * _layer_params(cfg) + V * H) + 3.5 * cfg.num_layers * _attention_flops(cfg, lens)
        return {"bytes": 6 * (cfg.num_layers * _layer_params(cfg) + V * H * (1 if cfg.tie_embeddings else 2)), "flops": flops}
    lens = _lengths(case)
    T = sum(lens)
    if kind == "score":
        return {"bytes": 2 * (cfg.num_layers * _layer_params(cfg) + V * H) + 20 * T,
                "flops": 2.0 * T * (cfg.num_layers * _layer_params(cfg) + V * H) + cfg.num_layers * _attention_flops(cfg, lens)}
    if kind == "layer":
        return {"bytes": 4 * _layer_params(cfg) + 8 * T * H, "flops": 6.0 * T * _layer_params(cfg) + 3.5 * _attention_flops(cfg, lens)}
    if kind == "attention":
        return {"bytes": 2 * T * (2 * cfg.qkv_dim + 2 * cfg.num_heads * cfg.head_dim), "flops": 3.5 * _attention_flops(cfg, lens)}
    return {"bytes": 4 * V * H + 4 * T * H, "flops": 6.0 * T * H * V}


def tolerance(case):
    kind = case["kind"]
    if kind == "unit":
        return "exact"  # bytes moved, and one fp32 addition per element
    if kind == "adamw":
        return {"rel": 5e-5, "max": 8e-3}  # fp32 state; the bf16 copy may round the other way
    # chains of bf16 activations and their gradients; this package's kernels against cuBLAS and flash-attn on the same inputs
    # differ by 1.2e-2 (max 0.7, a rarely hit row of the embedding gradient) and 0.8e-2 (max 0.07)
    if kind == "step":
        return {"rel": 2e-2, "max": 0.99}
    if kind == "layer":
        return {"rel": 1.5e-2, "max": 0.3}
    return {"rel": 1e-2, "max": 0.4}
