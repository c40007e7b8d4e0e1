"""Workloads on which the speed of this package is measured.

Two groups.  The first runs whole programs through the classes a user's script calls: one decoded token on a carried
cache, scoring of a batch of sequences, one optimizer step of a language model and of the view-synthesis model, the
rendering of held-out views.  They use the named 124M configurations and the view-synthesis configuration of the
quick start.  The second group calls the stages that dominate a training step of the named 760M model at that model's own
sizes (attention of one chunk, read and write of the routed fast-weight pool, forward and backward), through the
functions the models call; attention also at the view-synthesis model's sizes.

Sizes between the listed ones, odd lengths among them, come from :func:`draw`.
"""
from __future__ import annotations

import math

import torch

from uttt_b200 import ops
from uttt_b200.config import named_config
from uttt_b200.models import build_model
from uttt_b200.models import fast_weights as fw
from uttt_b200.models.generation import GenerationCache
from uttt_b200.nvs.data import SyntheticScenes
from uttt_b200.nvs.model import LVSMModel
from uttt_b200.nvs.trainer import NVSTrainer, load_config
from uttt_b200.train.data import SyntheticZipfTokens
from uttt_b200.train.engine import EngineConfig, TrainEngine

DEVICE = "cuda"
NVS_CONFIG = "configs/nvs/ownership/obj/uttt_moe_e64a1.yaml"


# ------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one token of interactive generation early in a document: everything is latency and launches
        dict(name="decode_b1", kind="decode", model="124M-uttt-moe", batch=1, context=700),
        # a small serving batch past the first chunk: carried window history, a pool that has been written once
        dict(name="decode_b8", kind="decode", model="124M-uttt-moe", batch=8, context=3000),
        # scoring a batch of documents of a ragged length (harness log-likelihoods): logits of every position
        dict(name="score_moe", kind="score", model="124M-uttt-moe", batch=2, seq=3001),
        # one optimizer step as the benchmark runs it (captured forward and backward), routed and dense fast weights
        dict(name="train_moe", kind="train", model="124M-uttt-moe", batch=1, seq=8192),
        dict(name="train_dense", kind="train", model="124M-uttt-dense", batch=1, seq=4096),
        # view synthesis: evaluation renders of one scene, and an optimizer step on a small per-GPU batch
        dict(name="render", kind="render", scenes=1, views=5, size=256),
        dict(name="train_views", kind="train_views", scenes=4, views=7, size=256),
        # one layer's attention over one chunk of the 760M model, forward and backward: 2048 queries on a window of
        # 2048 carried keys
        dict(name="attention_chunk", kind="attention", batch=4, queries=2048, history=2048, heads=16, head_dim=96,
             window=2048, causal=True, backward=True),
        # full attention inside the views of a view-synthesis batch, as in evaluation
        dict(name="attention_view", kind="attention", batch=12, queries=1024, history=0, heads=12, head_dim=64,
             window=0, causal=False, backward=False),
        # one layer's read of the routed pool over one chunk of the 760M model, forward and backward
        dict(name="pool_read", kind="pool_read", model="760M-uttt-moe", batch=2, tokens=2048),
        # one layer's write of that pool: inner gradient, momentum, orthogonalisation, master step, and its backward
        dict(name="pool_write", kind="pool_write", model="760M-uttt-moe", batch=2, tokens=2048),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "score", "train", "render", "train_views", "attention", "attention", "pool_read",
                       "pool_write"])
    if kind == "decode":
        return dict(kind=kind, model="124M-uttt-moe", batch=_log_uniform(rng, 1, 16),
                    context=_log_uniform(rng, 1, 4000))
    if kind == "score":
        return dict(kind=kind, model=rng.choice(["124M-uttt-moe", "124M-uttt-dense"]), batch=rng.randint(1, 3),
                    seq=_log_uniform(rng, 200, 4000))
    if kind == "train":
        model = rng.choice(["124M-uttt-moe", "124M-uttt-dense"])
        return dict(kind=kind, model=model, batch=1, seq=rng.randint(1500, 8192 if model == "124M-uttt-moe" else 4096))
    if kind in ("render", "train_views"):
        return dict(kind=kind, scenes=rng.randint(1, 4), views=rng.randint(2, 7),
                    size=rng.choice([128, 192, 256]))
    if kind == "attention":
        causal = rng.random() < 0.7
        window = rng.choice([256, 512, 1024, 2048]) if causal else 0
        return dict(kind=kind, batch=rng.randint(1, 4), queries=_log_uniform(rng, 100, 2048),
                    history=rng.randint(0, window) if causal else 0, heads=rng.choice([12, 16]),
                    head_dim=rng.choice([64, 96, 128]), window=window, causal=causal, backward=rng.random() < 0.6)
    return dict(kind=kind, model=rng.choice(["760M-uttt-moe", "124M-uttt-moe"]), batch=rng.randint(1, 2),
                tokens=rng.randint(200, 2048))


# ------------------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _normal(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=gen, device=DEVICE) * std).to(dtype)


def _language_model(name, seed, **overrides):
    torch.manual_seed(seed)
    config = named_config(name, **overrides)
    with torch.device(DEVICE):
        return config, build_model(config)


def _tokens(config, batch, seq, seed):
    return next(SyntheticZipfTokens(config.vocab_size, seq, batch, seed=seed))["input_ids"].to(DEVICE)


def _prepare_decode(c, seed):
    config, lm = _language_model(c["model"], seed)
    lm = lm.to(torch.bfloat16).eval()
    ids = _tokens(config, c["batch"], c["context"] + 1, seed)
    with torch.no_grad():
        cache = lm(input_ids=ids[:, :-1], use_cache=True, logits_to_keep=1).past_key_values
    return dict(lm=lm, cache=cache, token=ids[:, -1:].contiguous())


def _prepare_score(c, seed):
    config, lm = _language_model(c["model"], seed)
    return dict(lm=lm.to(torch.bfloat16).eval(), ids=_tokens(config, c["batch"], c["seq"], seed))


def _prepare_train(c, seed):
    config, lm = _language_model(c["model"], seed)
    engine = TrainEngine(config, EngineConfig(micro_batch_size=c["batch"], lr=1e-3, eps=1e-15, warmup_steps=1,
                                              seed=seed, cuda_graph=True), torch.device(DEVICE, torch.cuda.current_device()),
                         model=lm)
    ids = _tokens(config, c["batch"], c["seq"], seed)
    batch = {"input_ids": ids, "labels": ids}
    for _ in range(3):                    # a job under way: the engine captures its graph in the third step
        engine.train_step(batch)
    return dict(engine=engine, batch=batch)


def _nvs_config(c, seed):
    config = load_config(NVS_CONFIG)
    config["model"]["image_size"] = c["size"]
    config["training"].update(batch_size_per_gpu=c["scenes"], total_batch_size=c["scenes"], num_views=c["views"],
                              out_dir="/tmp/uttt_perf_cases", checkpoint_every=10 ** 9, print_every=10 ** 9, warmup=0,
                              seed=seed, cuda_graph=True)
    scenes = next(SyntheticScenes(c["scenes"], c["views"], c["size"], seed=seed))
    return config, {k: v.to(DEVICE) for k, v in scenes.items()}


def _prepare_render(c, seed):
    config, scenes = _nvs_config(c, seed)
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        model = LVSMModel(config)
    return dict(model=model.to(torch.bfloat16).eval(), scenes=scenes)


def _prepare_train_views(c, seed):
    config, scenes = _nvs_config(c, seed)
    with torch.device(DEVICE):
        trainer = NVSTrainer(config, torch.device(DEVICE, torch.cuda.current_device()))
    for _ in range(3):                    # a job under way, as above
        trainer.train_pass(scenes)
    return dict(trainer=trainer, scenes=scenes)


def _prepare_attention(c, seed):
    gen = _generator(seed)
    keys = c["queries"] + c["history"]
    shape = (c["heads"], c["head_dim"])
    q = _normal(gen, c["batch"], c["queries"], *shape)
    k, v = _normal(gen, c["batch"], keys, *shape), _normal(gen, c["batch"], keys, *shape)
    state = dict(q=q, k=k, v=v, window=c["window"] or None, causal=c["causal"], backward=c["backward"])
    if c["backward"]:
        state["dout"] = _normal(gen, c["batch"], c["queries"], *shape)
        for t in (q, k, v):
            t.requires_grad_()
    return state


def _unit_rows(gen, *shape):
    return torch.nn.functional.normalize(torch.randn(*shape, generator=gen, device=DEVICE), dim=-1).to(torch.bfloat16)


def _pool(gen, config, batch):
    """Experts at their initial scale, one bank per sequence: fp32 masters and the bf16 copies the kernels read."""
    e, i, d = config.memory_num_experts, config.fw_inter_dim, config.fw_head_dim
    m02 = _normal(gen, batch, e, 2 * i, d, std=d ** -0.5, dtype=torch.float32)
    m1 = _normal(gen, batch, e, d, i, std=i ** -0.5, dtype=torch.float32)
    router = _normal(gen, e, d, std=d ** -0.5)
    return m02, m1, router


def _prepare_pool_read(c, seed):
    gen, config = _generator(seed), named_config(c["model"])
    m02, m1, router = _pool(gen, config, c["batch"])
    rows = _unit_rows(gen, c["batch"], c["tokens"] * config.fw_heads, config.fw_head_dim)
    leaves = [t.requires_grad_() for t in (rows, router, m02.to(torch.bfloat16), m1.to(torch.bfloat16))]
    return dict(config=config, leaves=leaves, dout=_normal(gen, *rows.shape))


def _write_rows(gen, config, batch, n):
    d = config.fw_head_dim
    keys = _unit_rows(gen, batch, n, d)
    values = torch.nn.functional.silu(_normal(gen, batch, n, d))
    rates = torch.nn.functional.softplus(_normal(gen, batch, n, 3, std=0.5, dtype=torch.float32) - 6.9)
    return keys, values, rates


def _prepare_pool_write(c, seed):
    gen, config = _generator(seed), named_config(c["model"])
    m02, m1, router = _pool(gen, config, c["batch"])
    w02, w1 = m02.to(torch.bfloat16), m1.to(torch.bfloat16)
    n = c["tokens"] * config.fw_heads
    with torch.no_grad():                 # the momentum the previous chunk left behind
        keys, values, rates = _write_rows(gen, config, c["batch"], n)
        z02, z1 = fw.pool_raw_grad(keys, values, rates, w02, w1, fw.route_rows(keys, router, None, config))
    decay = torch.rand(c["batch"], 1, 1, 1, generator=gen, device=DEVICE)
    leaves = [t.detach().requires_grad_() for t in (*_write_rows(gen, config, c["batch"], n), router, w02, w1, m02, m1,
                                                    z02, z1, decay)]
    cotangents = [_normal(gen, *t.shape, std=1e-3, dtype=t.dtype) for t in (w02, w1, m02, m1, z02, z1)]
    return dict(config=config, leaves=leaves, cotangents=cotangents)


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


# ------------------------------------------------------------------------------------------------------- one pass
def _run_decode(s):
    c = s["cache"]                        # the call extends the cache it is given: continue from a fork of the prefix
    fork = GenerationCache(list(c.states), list(c.hist), list(c.chunk_kv), [list(f) for f in c.feats], c.chunk_start,
                           c.chunk_fill, c.seen_tokens)
    with torch.no_grad():
        out = s["lm"](input_ids=s["token"], past_key_values=fork, use_cache=True, logits_to_keep=1)
    return [out.logits] + [t for kv in out.past_key_values.chunk_kv for t in kv]


def _run_score(s):
    with torch.no_grad():
        return s["lm"](input_ids=s["ids"]).logits


def _run_train(s):
    loss = s["engine"].train_step(s["batch"])
    return [loss] + [u.master for u in s["engine"].trainer.units]


def _run_render(s):
    with torch.no_grad():
        return s["model"](s["scenes"])["rendering"]


def _run_train_views(s):
    stats = s["trainer"].train_pass(s["scenes"])
    return [stats["loss"]] + [u.master for u in s["trainer"].trainer.units]


def _run_attention(s):
    if not s["backward"]:
        with torch.no_grad():
            return ops.swa_attention(s["q"], s["k"], s["v"], s["window"], causal=s["causal"])
    out = ops.swa_attention(s["q"], s["k"], s["v"], s["window"], causal=s["causal"])
    return [out.detach(), *torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])]


def _run_pool_read(s):
    rows, router, w02, w1 = s["leaves"]
    y = fw.pool_read(rows, w02, w1, fw.route_rows(rows, router, None, s["config"]))
    return [y.detach(), *torch.autograd.grad(y, s["leaves"], s["dout"])]


def _run_pool_write(s):
    keys, values, rates, router, w02, w1, m02, m1, z02, z1, decay = s["leaves"]
    routing = fw.route_rows(keys, router, None, s["config"])
    g02, g1 = fw.pool_raw_grad(keys, values, rates, w02, w1, routing)
    new = fw.apply_pool_update(g02, g1, fw.PoolState(w02, w1, m02, m1, z02, z1), decay, 1.0, True).tensors()
    return [*[t.detach() for t in new], *torch.autograd.grad(new, s["leaves"][:-1], s["cotangents"])]


def run(state):
    return globals()["_run_" + state["kind"]](state)


# ------------------------------------------------------------------------------------------------------- work
def _lm_work(config, tokens, keys):
    """(weight elements, forward flops) of a language model over ``tokens`` tokens that see ``keys`` keys on average.
    A dense fast-weight model routes every row to the one operator of its head."""
    d, layers = config.hidden_size, config.num_hidden_layers
    inter, heads, hd = config.fw_inter_dim, config.fw_heads, config.fw_head_dim
    routed = config.model_type != "uttt_dense"
    k, e = (config.memory_num_active_experts, config.memory_num_experts) if routed else (1, heads)
    block = 5 * d * d + 3 * d * config.mlp_intermediate_size
    head = config.vocab_size * d
    weights = layers * block + 2 * head + 3 * e * inter * hd
    read = 6 * k * heads * inter * hd
    flops = tokens * (2 * (layers * block + head) + layers * (read + 4 * keys * d))
    return weights, flops, tokens * layers * 2 * read, e


def _orthogonalise_flops(inter, d, matrices):
    return matrices * 5 * (4 * inter * d * d + 2 * d ** 3)


def _mean_keys(queries, history, window, causal):
    """Average number of visible keys per query."""
    if not causal:
        return float(queries + history)
    return sum(min(history + i + 1, window) for i in range(queries)) / queries


def _nvs_work(c):
    """(weight elements, forward flops, bytes of one side's images): every view but the last is an
    input, every view but the first a target, each in a slot of its own."""
    model = load_config(NVS_CONFIG)["model"]
    p = model["block_config"]["params"]
    dim, layers, hd, k = model["dim"], model["layers"], p["fw_head_dim"], p["num_active_experts"]
    slot = (c["size"] // model["patch_size"]) ** 2
    inputs = c["scenes"] * (c["views"] - 1) * slot
    expert = 3 * int(hd * p["fw_inter_multi"]) * (dim // hd)      # per element of a head vector
    passed = (4 + 2 + 3 * p["inter_multi"]) * dim * dim           # attention, memory and MLP weights of every token
    write = 2 * dim * dim + 2 * k * expert * hd                   # key and value projections, inner gradient
    flops = 2 * layers * (2 * inputs * (passed + k * expert * hd + 2 * slot * dim) + inputs * write)
    weights = layers * (passed + 2 * dim * dim) + p["num_experts"] * 3 * hd * int(hd * p["fw_inter_multi"])
    return weights, flops, c["scenes"] * (c["views"] - 1) * 3 * c["size"] ** 2 * 4


def work(case):
    c, kind = case, case["kind"]
    if kind in ("decode", "score", "train"):
        config = named_config(c["model"])
        kv = config.num_hidden_layers * 2 * config.hidden_size * 2          # bytes of keys and values per token
        if kind == "decode":
            seen = min(c["context"], config.window_size)
            weights, flops, _, _ = _lm_work(config, c["batch"], seen)
            rows = min(c["batch"] * config.fw_heads * config.memory_num_active_experts,
                       c["batch"] * config.memory_num_experts)
            expert = 3 * config.fw_inter_dim * config.fw_head_dim
            dense = weights - config.vocab_size * config.hidden_size - config.memory_num_experts * expert
            return {"bytes": 2 * (dense + config.num_hidden_layers * rows * expert) + c["batch"] * seen * kv
                    + c["batch"] * config.vocab_size * 2, "flops": flops}
        tokens = c["batch"] * c["seq"]
        keys = _mean_keys(c["seq"], 0, config.window_size, True)
        weights, flops, write, e = _lm_work(config, tokens, keys)
        writes = (c["seq"] - 1) // config.chunk_size
        bank = 3 * c["batch"] * e * config.fw_inter_dim * config.fw_head_dim
        if writes:
            flops += write * writes * config.chunk_size // c["seq"]
            flops += writes * _orthogonalise_flops(config.fw_inter_dim, config.fw_head_dim, 3 * c["batch"] * e)
        if kind == "score":
            return {"bytes": 2 * weights + tokens * config.vocab_size * 2 + writes * bank * 14, "flops": flops}
        # every weight is read and its gradient written in bf16; master and two moments are read and written in fp32
        return {"bytes": weights * (2 + 2 + 2 + 24) + 3 * writes * bank * 14, "flops": 3 * flops}
    if kind in ("render", "train_views"):
        weights, flops, images = _nvs_work(c)
        if kind == "render":
            return {"bytes": 2 * weights + 2 * images, "flops": flops}
        return {"bytes": weights * (2 + 2 + 2 + 24) + 2 * images, "flops": 3 * flops}
    if kind == "attention":
        keys = _mean_keys(c["queries"], c["history"], c["window"], c["causal"])
        width = c["batch"] * c["heads"] * c["head_dim"]
        q, kv = 2 * width * c["queries"], 2 * width * (c["queries"] + c["history"])
        products = 2 * width * c["queries"] * keys
        if not c["backward"]:
            return {"bytes": 2 * q + 2 * kv, "flops": 2 * products}
        return {"bytes": 4 * q + 4 * kv, "flops": 7 * products}
    config = named_config(c["model"])
    rows = c["batch"] * c["tokens"] * config.fw_heads
    d, inter, e, k = (config.fw_head_dim, config.fw_inter_dim, config.memory_num_experts,
                      config.memory_num_active_experts)
    bank = 3 * c["batch"] * e * inter * d
    product = 2 * rows * k * inter * d
    if kind == "pool_read":
        return {"bytes": 4 * rows * d * 2 + 2 * bank * 2, "flops": 9 * product + 4 * rows * d * e}
    # bf16 copy read, master and momentum read and written, their cotangents read and gradients written
    return {"bytes": 4 * rows * d * 2 + bank * (2 + 2 + 8 + 8 + 2 + 8 + 2 + 8),
            "flops": 18 * product + 3 * _orthogonalise_flops(inter, d, 3 * c["batch"] * e) + 4 * rows * d * e}


# ------------------------------------------------------------------------------------------------------- tolerance
def tolerance(case):
    """bf16 throughout.  Measured: the whole programs with bf16-sized noise (2^-9 relative) on their embedding weights
    are apart by 1.5e-2 (one token), 1.3e-2 (scoring), 7e-3 (weights after a step), 3e-3 (renderings) and 1e-3
    (view-synthesis weights); a routed model sends a row whose last chosen and first refused expert are level with
    that noise to the other one.  The write differs by 9e-3 from itself run twice (its matrix norms are summed in any
    order, and the orthogonalisation passes rounding of small singular directions on).  Attention and read: 2e-3, the
    rounding of bf16 results and of the probabilities between the two products."""
    return {"decode": {"rel": 0.03, "max": 0.6}, "score": {"rel": 0.03, "max": 0.6},
            "train": {"rel": 0.028, "max": 0.95}, "render": {"rel": 0.011, "max": 0.1},
            "train_views": {"rel": 0.004, "max": 0.25}, "attention": {"rel": 0.01, "max": 0.3},
            "pool_read": {"rel": 0.01, "max": 0.9}, "pool_write": {"rel": 0.03, "max": 0.4}}[case["kind"]]
