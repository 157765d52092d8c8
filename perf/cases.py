"""Work that programs have this framework do, as measurable cases.

Six kinds, one per public surface:

    linear    PackedLinear.forward: one block linear called by itself (any host that swaps single layers)
    shards    torch.ops.shapequant.linear over PackedShards: the stacked projections of a serving layer
    dense     PackedLinear.dense / DeviceMatrix.dequant: the weights decoded for a consumer that wants a plain matrix
    step      one captured decode step of DecodeEngine for B sequences, caches filled to each one's position
    prefill   DecodeEngine.prefill of a prompt that arrives as host token ids
    snap      codebook.snap + pack_bits: a weight matrix encoded into the format

Shapes are those of the two benchmark models (hidden 3584 / intermediate 18944; hidden 5120 / intermediate 27648 with
two summed books and 16 column orders), of the test suite (4864 x 896) and ragged ones between.  Weights are random in
the storage format: uniform 12-bit tags (a fitted book is used evenly), N(0, 1) fp16 codewords, row scales that give
outputs of unit variance; activations are N(0, 1)."""

from __future__ import annotations

import math

import torch

from quantexperiments_b200 import codebook as cb
from quantexperiments_b200.engine import Cfg, random_engine
from quantexperiments_b200.linear import PackedLinear
from quantexperiments_b200.packed import seeded_perms
from quantexperiments_b200.vllm_ext import core

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
# block shapes of the two benchmark models, as engine configurations
CFGS = {"7b": dict(hidden=3584, n_heads=28, n_kv=4, inter=18944), "32b": dict(hidden=5120, n_heads=40, n_kv=8, inter=27648)}
VOCAB = 152064
K, D, BITS = 4096, 8, 12


def _linear(name, tokens, R, C, dtype="bf16", books=1, orders=1, bias=False):
    return dict(name=name, kind="linear", tokens=tokens, R=R, C=C, dtype=dtype, books=books, orders=orders, bias=bias)


def listed():
    return [
        # the smallest product of a decode step (key / value projection), one token: launch and host cost decide
        _linear("linear_kv_1tok", 1, 512, 3584),
        # the widest product of a decode step, one token
        _linear("linear_gate_1tok", 1, 18944, 3584),
        # gate projection of the larger model: two summed books, rows in 16 column orders, one token
        _linear("linear_gate32b_1tok", 1, 27648, 5120, books=2, orders=16),
        # a few sequences decoded together, the long reduction
        _linear("linear_down_5tok", 5, 3584, 18944),
        # gate|up of a serving layer with a dozen sequences in flight
        dict(name="shards_gateup_12tok", kind="shards", stack="gate_up", model="7b", tokens=12, dtype="bf16", books=1, orders=1),
        # an odd batch on a small model's projection, fp16 and with a bias
        _linear("linear_small_37tok", 37, 4864, 896, dtype="fp16", bias=True),
        # a long prompt through the widest product
        _linear("linear_gate_2048tok", 2048, 18944, 3584),
        # weights decoded to 16 bits for a consumer of plain matrices
        dict(name="dense_down", kind="dense", R=3584, C=18944, dtype="fp16", books=1, orders=1),
        # interactive generation: one sequence, a long context, the whole model
        dict(name="step_b1", kind="step", model="7b", layers=28, batch=1, context=2048, books=1, orders=1, head="16"),
        # batched generation: sequences of different lengths
        dict(name="step_b32", kind="step", model="7b", layers=28, batch=32, context=1024, books=1, orders=1, head="16"),
        # a prompt of ordinary length
        dict(name="prefill_700", kind="prefill", model="7b", layers=28, tokens=700, books=1, orders=1),
        # a matrix encoded: nearest codewords and packing
        dict(name="snap_gate", kind="snap", R=18944, C=3584, weighted=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "shards", "shards", "dense", "step", "step", "prefill", "snap"])
    books = rng.choice([1, 1, 1, 2])
    orders = rng.choice([1, 1, 1, 4, 16])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "linear":
        # one token is by far the commonest call; the rest of the range is even over the logarithm
        tokens = 1 if rng.random() < 0.3 else _log(rng, 2, 2048)
        return dict(kind=kind, tokens=tokens, R=_log(rng, 64, 18944), C=8 * _log(rng, 32, 2368), dtype=dtype, books=books, orders=orders,
                    bias=rng.random() < 0.3)
    if kind == "shards":
        tokens = 1 if rng.random() < 0.2 else _log(rng, 2, 1024)
        return dict(kind=kind, stack=rng.choice(["qkv", "gate_up"]), model=rng.choice(["7b", "7b", "32b"]), tokens=tokens, dtype=dtype,
                    books=books, orders=orders)
    if kind == "dense":
        return dict(kind=kind, R=_log(rng, 256, 18944), C=8 * _log(rng, 64, 2368), dtype=rng.choice(["fp16", "bf16", "fp32"]), books=books,
                    orders=orders)
    if kind == "step":
        return dict(kind=kind, model=rng.choice(["7b", "7b", "32b"]), layers=rng.randint(2, 8), batch=_log(rng, 1, 32), context=_log(rng, 16, 2048),
                    books=books, orders=orders, head=rng.choice(["16", "16", "q8"]))
    if kind == "prefill":
        return dict(kind=kind, model=rng.choice(["7b", "7b", "32b"]), layers=rng.randint(2, 4), tokens=_log(rng, 16, 1024), books=books, orders=orders)
    return dict(kind="snap", R=_log(rng, 256, 18944), C=_log(rng, 500, 3584), weighted=rng.random() < 0.3)


# ------------------------------------------------------------------------------------------------ inputs
def _packed_linear(R, C, books, orders, g, bias_dtype=None):
    """One matrix in the file layout, on the GPU, as a PackedLinear."""
    W = (C // D * BITS + 31) // 32
    words = [torch.randint(-2**31, 2**31 - 1, (R, W), dtype=torch.int32, device="cuda", generator=g) for _ in range(books)]
    table = [torch.randn(K, D, device="cuda", generator=g).half() for _ in range(books)]
    scale = ((torch.rand(R, device="cuda", generator=g) * 0.5 + 0.75) / math.sqrt(C * books)).half()
    bias = None if bias_dtype is None else torch.randn(R, device="cuda", generator=g).to(bias_dtype)
    mask, perms = None, torch.arange(C, device="cuda")[None]
    if orders > 1:
        mask = torch.randint(0, orders, (R,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
        perms = seeded_perms(C, orders, torch.Generator().manual_seed(g.initial_seed() + R)).to("cuda")
    more = dict(words2=words[1], table2=table[1]) if books == 2 else {}
    return PackedLinear(words[0], table[0], scale, None, mask, perms, K, D, bias=bias, **more)


def _pieces(case):
    c = CFGS[case["model"]]
    if case["stack"] == "qkv":
        return c["hidden"], [c["n_heads"] * 128, c["n_kv"] * 128, c["n_kv"] * 128]
    return c["hidden"], [c["inter"], c["inter"]]


def _positions(case, seed):
    """Sequences of a batch stand at different positions, up to the context."""
    g = torch.Generator().manual_seed(seed)
    pos = (case["context"] * (0.25 + 0.75 * torch.rand(case["batch"], generator=g))).to(torch.int32)
    pos[0] = case["context"]
    return pos


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(kind=kind)
    if kind in ("linear", "dense"):
        dt = DTYPES[case["dtype"]]
        s["lin"] = _packed_linear(case["R"], case["C"], case["books"], case["orders"], g, dt if case.get("bias") else None)
        if kind == "dense":
            s["dtype"] = dt
        else:
            s["x"] = torch.randn(case["tokens"], case["C"], device="cuda", generator=g).to(dt)
    elif kind == "shards":
        C, Rs = _pieces(case)
        s["shards"] = core.PackedShards([_packed_linear(R, C, case["books"], case["orders"], g) for R in Rs])
        # serving registers each layer once for the life of the process; the slot is reused so that states can be dropped
        s["handle"] = _Handle(s["shards"])
        s["x"] = torch.randn(case["tokens"], C, device="cuda", generator=g).to(DTYPES[case["dtype"]])
    elif kind in ("step", "prefill"):
        length = case["context"] + 1 if kind == "step" else case["tokens"]
        cfg = Cfg(**CFGS[case["model"]], vocab=VOCAB, layers=case["layers"], max_len=length)
        eng = random_engine(cfg, seed=seed, B=case.get("batch", 1), books=case["books"], M=case["orders"], head=case.get("head", "16"))
        s["eng"] = eng
        if kind == "step":
            eng.capture()
            eng.kc.normal_(generator=g)
            eng.vc.normal_(generator=g)
            s["tok"] = torch.randint(0, VOCAB, (case["batch"],), device="cuda", generator=g)
            s["pos"] = _positions(case, seed).to("cuda")
        else:
            s["ids"] = torch.randint(0, VOCAB, (case["tokens"],), generator=torch.Generator().manual_seed(seed))
    else:
        s["w"] = 0.02 * torch.randn(case["R"], case["C"], device="cuda", generator=g)
        s["book"] = torch.randn(K, D, device="cuda", generator=g).half()
        s["weight"] = torch.rand(case["C"], device="cuda", generator=g) + 0.5 if case["weighted"] else None
    if kind in ("linear", "shards", "prefill"):
        run(s)                  # the kernel layouts are built on a layer's first use; a server does that before it takes requests
    return s


class _Handle:
    """A registered layer whose registry slot becomes free with the state that holds it."""

    _free: list = []

    def __init__(self, shards):
        self.slot = _Handle._free.pop() if _Handle._free else core.register(None)
        core._REGISTRY[self.slot] = shards

    def __del__(self):
        core._REGISTRY[self.slot] = None
        _Handle._free.append(self.slot)


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"](state["x"])
    if kind == "shards":
        return torch.ops.shapequant.linear(state["x"], state["handle"].slot)
    if kind == "dense":
        lin = state["lin"]
        return lin.dense() if state["dtype"] == torch.float32 else lin.dm.dequant(dtype=state["dtype"])
    if kind == "step":
        eng = state["eng"]
        eng.tok.copy_(state["tok"])
        eng.pos.copy_(state["pos"])
        eng.graph.replay()
        # the greedy token follows from the logits, where near-ties make it the less telling of the two
        return dict(logits=eng.logits, pos=eng.pos, keys=eng.kc, values=eng.vc)
    if kind == "prefill":
        eng = state["eng"]
        logits = eng.prefill(state["ids"])
        return dict(logits=logits, pos=eng.pos, keys=eng.kc, values=eng.vc)
    r = cb.snap(state["w"], state["book"], col_weight=state["weight"])
    return dict(idx=r["idx"], row_scale=r["row_scale"], err=r.err, mse=r.stats["normalized_chunk_mse"], words=cb.pack_bits(r["idx"], BITS))


# ------------------------------------------------------------------------------------------------ what a pass needs
def _matrix(R, C, books, orders):
    """Stored bytes of one matrix: tags, books, row scales, the rows' order numbers and the orders."""
    W = (C // D * BITS + 31) // 32
    return books * (R * W * 4 + K * D * 2) + 2 * R + ((R + 4 * orders * C) if orders > 1 else 0)


def _product(tokens, R, C, books, orders):
    return _matrix(R, C, books, orders) + 2 * tokens * (R + C), 2 * tokens * R * C


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _product(case["tokens"], case["R"], case["C"], case["books"], case["orders"])
        return dict(bytes=b + (2 * case["R"] if case["bias"] else 0), flops=f)
    if kind == "shards":
        C, Rs = _pieces(case)
        t = case["tokens"]
        b = sum(_matrix(R, C, case["books"], case["orders"]) + 2 * t * R for R in Rs) + 2 * t * C
        return dict(bytes=b, flops=sum(2 * t * R * C for R in Rs))
    if kind == "dense":
        size = 4 if case["dtype"] == "fp32" else 2
        return dict(bytes=_matrix(case["R"], case["C"], case["books"], case["orders"]) + size * case["R"] * case["C"], flops=case["R"] * case["C"] * case["books"])
    if kind == "snap":
        R, C = case["R"], case["C"]
        n = R * -(-C // D)
        # fp32 weights in; tags as int64, errors, packed tags and row scales out; a multiply-add per value of every codeword
        return dict(bytes=4 * R * C + n * (8 + 4) + R * 4 * ((n // R * BITS + 31) // 32) + 2 * R + K * D * 2, flops=2 * n * D * K * (2 if case["weighted"] else 1))
    c = CFGS[case["model"]]
    H, I, Q, KV, L = c["hidden"], c["inter"], c["n_heads"] * 128, c["n_kv"] * 128, case["layers"]
    mats = [(Q, H), (KV, H), (KV, H), (H, Q), (I, H), (I, H), (H, I)]
    weights = sum(_matrix(R, C, case["books"], case["orders"]) for R, C in mats) * L
    macs = sum(R * C for R, C in mats) * L
    head = VOCAB * H * 2 if case.get("head", "16") == "16" else VOCAB * H * 34 // 32
    if kind == "step":
        B = case["batch"]
        seen = case["context"] if B == 1 else B * case["context"] * 5 // 8      # positions are spread over 1/4 .. 1 of the context
        return dict(bytes=weights + head + seen * 2 * KV * 2 * L + B * VOCAB * 4, flops=2 * B * (macs + VOCAB * H) + seen * 4 * Q * L)
    T = case["tokens"]
    return dict(bytes=weights + head + T * (H * 2 + 2 * KV * 2 * L) + VOCAB * 4, flops=2 * T * macs + 2 * VOCAB * H + T * T // 2 * 4 * Q * L)


def tolerance(case):
    kind = case["kind"]
    if kind == "dense":
        return "exact"                                      # the decode is bit-defined
    if kind == "snap":
        return dict(rel=1e-4, differ=1e-3)                  # fp32 distances; two codewords can all but tie
    if kind in ("step", "prefill"):
        return dict(rel=2e-2, max=0.5)                      # activations are rounded to bf16 between operators, layer after layer
    # fp32 accumulation, one rounding to the output type (two roundings with a bias)
    return dict(rel=1e-2 if case["dtype"] == "bf16" else 2e-3, max=0.1)
