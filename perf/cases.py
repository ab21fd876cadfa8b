"""The work whose speed this repository answers for, as a user's program calls it.

Four kinds of call, each through its public entry point:

* ``ns``    - ``HiMuon.newton_schulz(G)``: orthogonalises a batch of gradient tiles or matrices.
* ``opt``   - ``optimizer.step()`` of HiMuon, Muon or AdamW on the weights of a few decoder layers and an embedding.
* ``train`` - ``Trainer.train_step(host_batches)``: host copies of the tokens, forward, backward, optimizer step.
* ``eval``  - ``model(ids).logits`` under ``no_grad``.

Shapes are those of ``himuon_b200.models.MODEL_CONFIGS``, the tests and the benchmark.  A model is cut in depth and its
vocabulary is cut in the same proportion, so that the head keeps its share of the work.
"""

from __future__ import annotations

import argparse
import math

import torch

from himuon_b200.models import CausalLM, DecoderConfig
from himuon_b200.optim import get_optimizer
from himuon_b200.optimizers import AdamW, HiMuon, Muon
from himuon_b200.parallel.fsdp import ShardedEngine
from himuon_b200.trainer import Trainer

WHOLE = 10 ** 9          # a tile that covers every matrix: full-matrix Newton-Schulz (the reconfigure schedule's first phase)


# ------------------------------------------------------------------------------------------------ cases
def _ns(name, batch, rows, cols, dtype="bf16"):
    return {"name": name, "kind": "ns", "batch": batch, "rows": rows, "cols": cols, "dtype": dtype}


def _opt(name, optimizer, layers, hidden, inter, heads, kv_heads, head_dim, vocab, tile, dtype="bf16", banks=False):
    return {"name": name, "kind": "opt", "optimizer": optimizer, "layers": layers, "hidden": hidden, "inter": inter,
            "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim, "vocab": vocab, "tile": tile, "dtype": dtype,
            "banks": banks}


def _model(name, kind, family, layers, hidden, inter, heads, kv_heads, head_dim, vocab, tie, batch, seq, **more):
    return {"name": name, "kind": kind, "family": family, "layers": layers, "hidden": hidden, "inter": inter,
            "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim, "vocab": vocab, "tie": tie, "batch": batch,
            "seq": seq, **more}


def listed():
    return [
        # One small layer's tiles: the smallest call of the kernel microbenchmark (32 tiles of 128 x 128).
        _ns("ns small", 32, 128, 128),
        # A few fp32 gradients of odd shape, as a user's own modules have them.
        _ns("ns odd fp32", 6, 333, 500, "fp32"),
        # The default tile size at a mid-size model's batch.
        _ns("ns tile 512", 128, 512, 512),
        # The optimizer microbenchmark's model: square linear layers, tile 512 (here seven per layer of a 1024-wide model).
        _opt("opt small", "himuon", 1, 1024, 1024, 8, 8, 128, 0, 512),
        # fp32 parameters of the 220M-parameter model, tile 256: matrices that are no whole number of tiles.
        _opt("opt 220m fp32", "himuon", 4, 640, 1728, 10, 10, 64, 42752, 256, "fp32"),
        # The headline configuration's optimizer step: Qwen3-4B banks, tile 512, AdamW on the embedding.
        _opt("opt 4b banks", "himuon", 6, 2560, 9728, 32, 8, 128, 25320, 512, banks=True),
        # Full-matrix Muon on a 0.6B-parameter model's layers.
        _opt("opt muon", "muon", 4, 1024, 3072, 16, 8, 128, 21704, WHOLE),
        # The smallest training step: the smoke test's model, AdamW (the command line's default), eager.
        _model("train tiny", "train", "qwen3", 2, 512, 1536, 4, 2, 128, 4096, True, 2, 256,
               optimizer="adamw", tile=0, accumulate=1, graph=False, banks=False, checkpoint=False),
        # The tile-shape experiment's 220M-parameter Llama at its batch: heads of 64, HiMuon.
        _model("train 220m", "train", "llama", 6, 640, 1728, 10, 10, 64, 64128, False, 8, 512,
               optimizer="himuon", tile=256, accumulate=1, graph=False, banks=False, checkpoint=False),
        # Qwen3-0.6B as train_ddp.py runs it: activation checkpointing on, 2048 tokens a sequence.
        _model("train 0.6b", "train", "qwen3", 4, 1024, 3072, 16, 8, 128, 21704, True, 4, 2048,
               optimizer="himuon", tile=512, accumulate=1, graph=False, banks=False, checkpoint=True),
        # The headline training step: Qwen3-4B banks, two sequences of 1024, micro-batches replayed from CUDA graphs.
        _model("train 4b", "train", "qwen3", 4, 2560, 9728, 32, 8, 128, 16880, True, 2, 1024,
               optimizer="himuon", tile=512, accumulate=2, graph=True, banks=True, checkpoint=False),
        # Scoring text of odd length with Qwen3-1.7B: logits of five sequences of 777 tokens.
        _model("eval odd", "eval", "qwen3", 4, 2048, 6144, 16, 8, 128, 21704, True, 5, 777),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, v, step):
    """`v` as it comes half of the time, else the nearest multiple of `step`."""
    return v if rng.random() < 0.5 else max(step, round(v / step) * step)


# (hidden, intermediate, heads, kv heads, head_dim, family, tied) of the architectures the repository knows
_ARCH = [(512, 1536, 4, 2, 128, "qwen3", True), (640, 1728, 10, 10, 64, "llama", False),
         (1024, 3072, 16, 8, 128, "qwen3", True), (2048, 6144, 16, 8, 128, "qwen3", True),
         (2048, 8192, 32, 8, 64, "llama", True), (2560, 9728, 32, 8, 128, "qwen3", True),
         (3072, 8192, 24, 8, 128, "llama", True)]


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= most:
            return c


def _cost(c):
    w = work(c)
    return w["bytes"] / 6e12 + w["flops"] / 1e15


def _draw(rng):
    kind = rng.choice(["ns", "ns", "opt", "opt", "train", "train", "eval"])
    if kind == "ns":
        rows, cols = _ragged(rng, _log_int(rng, 16, 1024), 64), _ragged(rng, _log_int(rng, 64, 1024), 64)
        batch = max(1, _log_int(rng, 2 ** 17, 2 ** 25) // (rows * cols))
        c = _ns("", batch, rows, cols, rng.choice(["bf16", "bf16", "fp32"]))
    elif kind == "opt":
        hidden, inter, heads, kv, hd, _, _ = rng.choice(_ARCH)
        optimizer = rng.choice(["himuon", "himuon", "himuon", "muon", "adamw"])
        layers = rng.choice([1, 2] if optimizer == "adamw" else [1, 2, 3, 4])
        tile = rng.choice([128, 256, 512, 1024, WHOLE]) if optimizer == "himuon" else WHOLE
        c = _opt("", optimizer, layers, hidden, inter, heads, kv, hd, 8 * _log_int(rng, 512, 4096), tile,
                 rng.choice(["bf16", "bf16", "bf16", "fp32"]), optimizer == "himuon" and rng.random() < 0.5)
    else:
        hidden, inter, heads, kv, hd, family, tie = rng.choice(_ARCH)
        layers = rng.choice([1, 2, 3])
        seq = _ragged(rng, _log_int(rng, 64, 2048), 128)
        batch = max(1, _log_int(rng, 256, 4096) // seq)
        c = _model("", kind, family, layers, hidden, inter, heads, kv, hd, 8 * _log_int(rng, 512, 2048), tie, batch, seq)
        if kind == "train":
            c.update(optimizer=rng.choice(["himuon", "adamw"]), tile=rng.choice([128, 256, 512]),
                     accumulate=rng.choice([1, 2]), graph=rng.random() < 0.4, banks=rng.random() < 0.4,
                     checkpoint=rng.random() < 0.3)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ state
def _dtype(c):
    return torch.float32 if c.get("dtype") == "fp32" else torch.bfloat16


def _gradient(shape, gen, dtype):
    """Noise around a low-rank part, which is how a weight gradient looks: most of its norm in few directions."""
    *lead, m, n = shape
    noise = torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
    left = torch.randn(*lead, m, 8, generator=gen, device="cuda", dtype=dtype)
    right = torch.randn(*lead, 8, n, generator=gen, device="cuda", dtype=dtype)
    return torch.add(noise, left @ right, alpha=0.5).mul_(1e-3)


def _matrix_shapes(c):
    """(rows, columns) of one layer's projections: q, k, v, o, gate, up, down."""
    h, i, q, kv = c["hidden"], c["inter"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    return [(q, h), (kv, h), (kv, h), (h, q), (i, h), (i, h), (h, i)]


def _bank_shapes(c):
    q, k, _, o, g, _, d = _matrix_shapes(c)
    n = c["layers"]
    return [(n, *q), (2 * n, *k), (n, *o), (2 * n, *g), (n, *d)]


def _optimizer(c, model):
    return get_optimizer(c["optimizer"], model, argparse.Namespace(
        lr=1e-3 if c["optimizer"] == "adamw" else 1e-2, weight_decay=0.1, tile_size=c["tile"] or None, cuda_graph=True))


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    c = case
    if c["kind"] == "ns":
        return {"case": c, "grad": _gradient((c["batch"], c["rows"], c["cols"]), gen, _dtype(c))}
    if c["kind"] == "opt":
        dtype = _dtype(c)
        shapes = _bank_shapes(c) if c["banks"] else [s for _ in range(c["layers"]) for s in _matrix_shapes(c)]
        mats = [torch.nn.Parameter(torch.randn(s, generator=gen, device="cuda", dtype=dtype).mul_(0.02)) for s in shapes]
        rest = [torch.nn.Parameter(torch.ones(c["hidden"], device="cuda", dtype=dtype))]
        if c["vocab"]:
            rest.append(torch.nn.Parameter(torch.randn(c["vocab"], c["hidden"], generator=gen, device="cuda", dtype=dtype).mul_(0.02)))
        for p in mats:
            p.grad = _gradient(p.shape, gen, dtype)
        for p in rest:
            p.grad = torch.randn(p.shape, generator=gen, device="cuda", dtype=dtype).mul_(1e-3)
        if c["optimizer"] == "adamw":
            opt = AdamW([{"params": mats + rest[1:], "weight_decay": 0.1}, {"params": rest[:1], "weight_decay": 0.0}], lr=1e-3)
        else:
            groups = [{"params": mats, "use_muon": True}, {"params": rest[:1], "use_muon": False, "lr": 1e-3, "weight_decay": 0.0},
                      {"params": rest[1:], "use_muon": False, "lr": 1e-3}]
            groups = [g for g in groups if g["params"]]
            opt = HiMuon(groups, lr=1e-2, tile_size=c["tile"]) if c["optimizer"] == "himuon" else Muon(groups, lr=1e-2)
        return {"case": c, "optimizer": opt, "params": mats + rest}
    torch.manual_seed(seed)
    qwen = c["family"] == "qwen3"
    cfg = DecoderConfig(model_type=c["family"], vocab_size=c["vocab"], hidden_size=c["hidden"], intermediate_size=c["inter"],
                        num_hidden_layers=c["layers"], num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"],
                        head_dim=c["head_dim"], rms_norm_eps=1e-6 if qwen else 1e-5, rope_theta=1e6 if qwen else 5e5,
                        tie_word_embeddings=c["tie"], max_position_embeddings=8192)
    with torch.device("cuda"):
        model = CausalLM(cfg).to(torch.bfloat16)
    if c["kind"] == "eval":
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=gen, device="cuda")
        return {"case": c, "model": model.eval(), "ids": ids}
    if c["checkpoint"]:
        model.gradient_checkpointing_enable()
    engine = ShardedEngine(model) if c["banks"] else None
    opt = _optimizer(c, model)
    if engine is not None:
        engine.attach_optimizer(opt)
    trainer = Trainer(model.train(), opt, engine=engine, grad_acc=c["accumulate"], graph_microbatch=c["graph"])
    if engine is not None:
        trainer.zero_set_to_none = False
    host = torch.Generator().manual_seed(seed)
    batches = []
    for _ in range(c["accumulate"]):
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=host).pin_memory()
        batches.append({"input_ids": ids, "labels": ids})
    return {"case": c, "trainer": trainer, "batches": batches, "params": [p for p in model.parameters() if p.requires_grad]}


# ------------------------------------------------------------------------------------------------ one pass
def _optimizer_state(opt, params):
    out = []
    for p in params:
        st = opt.state.get(p, {})
        out.append({k: v for k, v in st.items() if torch.is_tensor(v) and v.dim() > 0})
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "ns":
        return HiMuon.newton_schulz(state["grad"])
    if kind == "opt":
        opt, params = state["optimizer"], state["params"]
        opt.step()
        return {"params": [p.detach() for p in params], "state": _optimizer_state(opt, params)}
    if kind == "eval":
        with torch.no_grad():
            return state["model"](state["ids"]).logits
    loss = state["trainer"].train_step(state["batches"])
    return {"loss": loss, "params": [p.detach() for p in state["params"]]}


# ------------------------------------------------------------------------------------------------ what a pass costs at least
def _ns_flops(rows, cols, tile=WHOLE):
    """Five iterations on every tile: half of X X^T and of A A (both are symmetric), all of B X."""
    total = 0
    for r in range(0, rows, tile):
        for q in range(0, cols, tile):
            h, w = min(tile, rows - r), min(tile, cols - q)
            m, n = min(h, w), max(h, w)
            total += 5 * (m * m * n + m ** 3 + 2 * m * m * n)
    return total


def _step_cost(c, n_other, esz):
    """Optimizer step: gradient, parameter and state read once, parameter and state written once."""
    mats = [s for _ in range(c["layers"]) for s in _matrix_shapes(c)]
    n_mat = sum(a * b for a, b in mats)
    if c["optimizer"] == "adamw":
        return {"bytes": 7 * esz * (n_mat + n_other), "flops": 0}
    tile = WHOLE if c["optimizer"] == "muon" else c["tile"]
    return {"bytes": esz * (5 * n_mat + 7 * n_other), "flops": sum(_ns_flops(a, b, tile) for a, b in mats)}


def work(case):
    c = case
    if c["kind"] == "ns":
        n = c["batch"] * c["rows"] * c["cols"]
        return {"bytes": 2 * n * (4 if c["dtype"] == "fp32" else 2), "flops": c["batch"] * _ns_flops(c["rows"], c["cols"])}
    if c["kind"] == "opt":
        return _step_cost(c, c["vocab"] * c["hidden"] + c["hidden"], 4 if c["dtype"] == "fp32" else 2)
    n_mat = c["layers"] * sum(a * b for a, b in _matrix_shapes(c))
    table = c["vocab"] * c["hidden"]
    tables = table * (1 if c["tie"] else 2)
    tokens = c["batch"] * c["seq"]
    attn = 2 * c["layers"] * tokens * c["seq"] * c["heads"] * c["head_dim"]      # causal half of Q K^T and P V, forward
    if c["kind"] == "eval":
        return {"bytes": 2 * (n_mat + tables + tokens * c["vocab"]) + 8 * tokens, "flops": 2 * tokens * (n_mat + table) + attn}
    acc = c["accumulate"]
    step = _step_cost(c, tables + c["layers"] * 4 * c["hidden"], 2)
    return {"bytes": step["bytes"] + 16 * acc * tokens, "flops": step["flops"] + acc * (6 * tokens * (n_mat + table) + 3.5 * attn)}


def tolerance(case):
    """About four times what was measured between this path and another correct one (2-norm of the difference over the
    2-norm of the result, largest difference over the result's root mean square), at most 0.03.

    ns: five bf16 iterations against the same rounding points with PyTorch's order of sums: 0.004-0.010, largest 0.21;
    against 64 bits: 0.011-0.021.  opt: three steps against the PyTorch path: 0.0016-0.0027, largest 0.07 (AdamW alone
    is element-wise: the rounding of its storage type).  train: two runs of the same code differ by up to 0.0095, largest
    0.13, because embedding and norm gradients are summed by atomics.  eval: logits against fp32: 0.016, largest 0.09."""
    if case["kind"] == "opt":
        if case["optimizer"] == "adamw":
            return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "fp32" else {"rel": 4e-3, "max": 0.03}
        return {"rel": 0.01, "max": 0.3}
    return {"rel": 0.03, "max": 0.5}
