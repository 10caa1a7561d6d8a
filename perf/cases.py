"""What a program built on this library spends its time on, as cases that can be timed: single projections, a dense
decoder layer from one row to a prompt chunk, a routed mixture-of-experts layer, one rank's share of a tensor-parallel
block, the vocabulary ends of a decode step, and the load path.

Weights are MLX affine words with uniform codes, scales |N(0, 0.01)| + 1e-4 and biases -2^(bits-1) * scale + N(0, 0.002);
activations are N(0, 1).  Everything is drawn on the GPU from the seed."""

from __future__ import annotations

import torch

from tensorfold_b200.cuda import experts, moe, tp
from tensorfold_b200.cuda.kernels import affine, qmm
from tensorfold_b200.families.qwen3_5.cuda import glue, qmm_fast
from tensorfold_b200.families.qwen3_5.cuda.weights import QLinear

DEV = "cuda"
GS = 64                   # group of the 4-bit layers; single projections vary it
EPS = 1e-6
WINDOW = 16               # rows of a decode or verify window that run as sets of projections
EXACT_ROWS = 256          # rows of batched verify windows; longer inputs are prompt chunks
ROUTED_DECODE_ROWS = 128  # routed layers take the prompt form past this


def listed() -> list[dict]:
    return [
        # one 4096 x 4096 projection for a four-row window: the smallest call, all latency
        {"name": "linear 4096 4b m4", "kind": "linear", "n": 4096, "k": 4096, "bits": 4, "gs": 64, "rows": 4},
        # a wide projection of a mixed-width checkpoint, whose sensitive layers stay at 8 bits, in a verify window
        {"name": "linear 14336 8b m16", "kind": "linear", "n": 14336, "k": 4096, "bits": 8, "gs": 64, "rows": 16},
        # a dense layer (hidden 5120): plain decoding of one stream
        {"name": "layer m1", "kind": "layer", "hidden": 5120, "inner": 17408, "q": 6144, "kv": 1024, "rows": 1},
        # the same layer verifying a window of drafts
        {"name": "layer m16", "kind": "layer", "hidden": 5120, "inner": 17408, "q": 6144, "kv": 1024, "rows": 16},
        # four streams' twelve-row windows in one batch, with the bits each stream gets alone
        {"name": "layer m48", "kind": "layer", "hidden": 5120, "inner": 17408, "q": 6144, "kv": 1024, "rows": 48},
        # the ragged last chunk of a prompt
        {"name": "layer m391", "kind": "layer", "hidden": 5120, "inner": 17408, "q": 6144, "kv": 1024, "rows": 391},
        # a whole prompt chunk
        {"name": "layer m2048", "kind": "layer", "hidden": 5120, "inner": 17408, "q": 6144, "kv": 1024, "rows": 2048},
        # a routed layer (128 experts, top 6, a wider shared expert) in a verify window
        {"name": "moe m16", "kind": "moe", "hidden": 2688, "experts": 128, "width": 1856, "top_k": 6, "shared": 3712, "rows": 16},
        # the same routed layer on a prompt chunk
        {"name": "moe m2048", "kind": "moe", "hidden": 2688, "experts": 128, "width": 1856, "top_k": 6, "shared": 3712,
         "rows": 2048},
        # what one of eight ranks computes of a tensor-parallel routed block on a prompt chunk, between the reductions
        {"name": "rank of 8 m2048", "kind": "rank", "hidden": 6144, "experts": 160, "width": 1536, "top_k": 8, "o": 8192,
         "world": 8, "rows": 2048},
        # the two ends of a decode step: a token's embedding row, and the logits over the whole vocabulary
        {"name": "vocabulary m1", "kind": "vocabulary", "vocab": 248320, "hidden": 5120, "rows": 1},
        # the load path: a stored projection to the library's layout and back (a sharding loader undoes the layout)
        {"name": "repack 17408 4b", "kind": "repack", "n": 17408, "k": 5120, "bits": 4, "gs": 64},
    ]


def _log(rng, lo: int, hi: int, step: int = 1) -> int:
    """An integer of [lo, hi], spread evenly over its logarithm, a multiple of ``step``."""

    v = lo * (hi / lo) ** rng.random()
    return max(lo, min(hi, round(v / step) * step))


def _rows(rng) -> int:
    """Rows of a layer call: windows, batches of windows and prompt chunks alike."""

    return rng.choice([rng.randint(1, WINDOW), _log(rng, WINDOW + 1, EXACT_ROWS), _log(rng, EXACT_ROWS + 1, 2048)])


def draw(rng) -> dict:
    kind = rng.choice(["linear", "linear", "layer", "layer", "layer", "moe", "moe", "rank", "vocabulary", "repack"])
    if kind == "linear":
        return {"kind": kind, "n": _log(rng, 256, 17408, rng.choice([1, 16, 128])), "k": _log(rng, 512, 16384, 128),
                "bits": rng.choice(affine.BITS), "gs": rng.choice(affine.GROUPS), "rows": _log(rng, 1, 64)}
    if kind == "layer":
        hidden = _log(rng, 1024, 5120, 64)
        return {"kind": kind, "hidden": hidden, "inner": min(17408, round(hidden * rng.uniform(2.5, 3.5) / 64) * 64),
                "q": _log(rng, 1024, 6144, 64), "kv": rng.choice([256, 512, 1024]), "rows": _rows(rng)}
    if kind == "moe":
        return {"kind": kind, "hidden": _log(rng, 1024, 2688, 64), "experts": rng.choice([32, 64, 96, 128]),
                "width": _log(rng, 512, 1856, 64), "top_k": rng.randint(2, 6), "shared": _log(rng, 512, 3712, 64),
                "rows": _rows(rng)}
    if kind == "rank":
        world = rng.choice([4, 8])
        return {"kind": kind, "hidden": _log(rng, 2048, 6144, 64), "experts": 160, "width": _log(rng, 512, 1536, 64),
                "top_k": 8, "o": world * _log(rng, 256, 1024, 64), "world": world, "rows": _rows(rng)}
    if kind == "vocabulary":
        return {"kind": kind, "vocab": _log(rng, 32000, 248320, rng.choice([1, 64])), "hidden": _log(rng, 1024, 5120, 64),
                "rows": rng.randint(1, WINDOW)}
    return {"kind": kind, "n": _log(rng, 256, 17408, rng.choice([1, 16, 128])), "k": _log(rng, 512, 16384, 128),
            "bits": rng.choice(affine.BITS), "gs": rng.choice(affine.GROUPS)}


# ---------------------------------------------------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------------------------------------------------

class _Make:
    def __init__(self, seed: int) -> None:
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape: int, std: float = 1.0) -> torch.Tensor:
        return (torch.randn(shape, generator=self.g, device=DEV) * std).to(torch.bfloat16)

    def words(self, *shape: int, bits: int = 4, gs: int = GS):
        """Stored words [..., n, k * bits / 32], scales and biases [..., n, k / gs] of shape (..., n, k)."""

        *lead, n, k = shape
        words = torch.randint(-(1 << 31), 1 << 31, (*lead, n, k * bits // 32), generator=self.g, device=DEV, dtype=torch.int32)
        scales = (torch.randn((*lead, n, k // gs), generator=self.g, device=DEV) * 0.01).abs() + 1e-4
        biases = torch.randn((*lead, n, k // gs), generator=self.g, device=DEV) * 0.002 - (1 << (bits - 1)) * scales
        return words, scales.to(torch.bfloat16), biases.to(torch.bfloat16)

    def packed(self, n: int, k: int, bits: int = 4, gs: int = GS) -> qmm.Q4:
        return qmm.pack(*self.words(n, k, bits=bits, gs=gs), gs, bits=bits)


def _linear(c, make):
    return {"x": make.normal(c["rows"], c["k"]), "q": make.packed(c["n"], c["k"], c["bits"], c["gs"])}


def _layer(c, make):
    h, i, nq, nkv, m = c["hidden"], c["inner"], c["q"], c["kv"], c["rows"]
    shapes = {"q": (nq, h), "k": (nkv, h), "v": (nkv, h), "o": (h, nq), "gate": (i, h), "up": (i, h), "down": (h, i)}
    s = {name: make.packed(*shape) for name, shape in shapes.items()}
    s["splits"] = [qmm.set_splits([shapes[name] for name in names], GS) for names in (("q", "k", "v"), ("gate", "up"))]
    s.update(x=make.normal(m, h), r=make.normal(m, h, std=0.5), attn=make.normal(m, nq),
             norms=[1 + make.normal(h, std=0.1) for _ in range(2)])
    return s


def _experts(c, make, count):
    d, w = c["hidden"], c["width"]
    return experts.make([make.words(count, w, d), make.words(count, w, d)], make.words(count, d, w), GS)


def _moe(c, make):
    d = c["hidden"]
    shared = moe.SharedExpert(qmm.pack_pair(make.words(c["shared"], d), make.words(c["shared"], d), GS),
                              make.packed(d, c["shared"]))
    router = make.normal(c["experts"] + 1, d, std=d ** -0.5)
    return {"x": make.normal(c["rows"], d),
            "layer": moe.Routed(router, _experts(c, make, c["experts"]), c["top_k"], shared)}


def _rank(c, make):
    d, m, rank, local = c["hidden"], c["rows"], 1, c["experts"] // c["world"]
    share = tp.ExpertParallelMoE(make.normal(c["experts"], d, std=d ** -0.5), _experts(c, make, local), c["top_k"],
                                 rank * local, c["experts"])
    o = tp.RowParallelLinear.shard(QLinear(*make.words(d, c["o"]), gs=GS), rank, c["world"])
    return {"attn": make.normal(m, c["o"] // c["world"]), "h": make.normal(m, d), "o": o, "moe": share,
            "buffers": share.buffers(m, DEV, prefill=m > ROUTED_DECODE_ROWS)}


def _vocabulary(c, make):
    v, h = c["vocab"], c["hidden"]
    return {"ids": torch.randint(0, v, (c["rows"],), generator=make.g, device=DEV), "norm": 1 + make.normal(h, std=0.1),
            "table": QLinear(*make.words(v, h), gs=GS), "head": qmm_fast.tile(QLinear(*make.words(v, h), gs=GS))}


def _repack(c, make):
    return {"stored": make.words(c["n"], c["k"], bits=c["bits"], gs=c["gs"])}


_PREPARE = {"linear": _linear, "layer": _layer, "moe": _moe, "rank": _rank, "vocabulary": _vocabulary, "repack": _repack}


def prepare(case: dict, seed: int) -> dict:
    return {**_PREPARE[case["kind"]](case, _Make(seed)), "case": case}


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------

def _run_layer(s) -> dict:
    """The layer around its attention: norm, q/k/v, output projection of the attention's rows, norm, MLP."""

    m = s["case"]["rows"]
    h, y, xs = glue.add_rmsnorm(s["x"], s["r"], s["norms"][0], EPS, GS)
    if m > EXACT_ROWS:
        q, k, v = (qmm.prefill_matmul(y, s[name]) for name in "qkv")
        o = qmm.prefill_matmul(s["attn"], s["o"])
    elif m > WINDOW:
        q, k, v = (qmm.matmul(y, s[name], xs, sk=sk) for name, sk in zip("qkv", s["splits"][0]))
        o = qmm.matmul(s["attn"], s["o"])
    else:
        q, k, v = qmm.matmul_set(y, [s["q"], s["k"], s["v"]], xs, sks=s["splits"][0], pdl=True)
        o = qmm.matmul(s["attn"], s["o"], pdl=True)
    h, y, xs = glue.add_rmsnorm(h, o, s["norms"][1], EPS, GS)
    if m > EXACT_ROWS:
        gate, up = (qmm.prefill_matmul(y, s[name]) for name in ("gate", "up"))
        act, _ = glue.swiglu(gate, up, GS)
        d = qmm.prefill_matmul(act, s["down"])
    elif m > WINDOW:
        gate, up = (qmm.matmul(y, s[name], xs, sk=sk) for name, sk in zip(("gate", "up"), s["splits"][1]))
        act, xs = glue.swiglu(gate, up, GS)
        d = qmm.matmul(act, s["down"], xs)
    else:
        gate, up = qmm.matmul_set(y, [s["gate"], s["up"]], xs, sks=s["splits"][1], pdl=True)
        act, xs = glue.swiglu(gate, up, GS)
        d = qmm.matmul(act, s["down"], xs, pdl=True)
    return {"q": q, "k": k, "v": v, "h": h, "d": d}


def run(state: dict):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "linear":
        return qmm.matmul(s["x"], s["q"])
    if kind == "layer":
        return _run_layer(s)
    if kind == "moe":
        return moe.run(s["x"], s["layer"], prefill=c["rows"] > ROUTED_DECODE_ROWS)
    if kind == "rank":
        o = qmm.prefill_matmul(s["attn"], s["o"].q) if c["rows"] > EXACT_ROWS else s["o"].partial(s["attn"])
        return {"o": o, "moe": s["moe"].partial(s["h"], s["buffers"])}
    if kind == "vocabulary":
        rows = affine.embed(s["ids"], s["table"])
        _, y, xs = glue.add_rmsnorm(rows, None, s["norm"], EPS, GS)
        return {"rows": rows, "logits": qmm_fast.matmul(y, s["head"], xs)}
    return qmm.unpack(qmm.pack(*s["stored"], c["gs"], bits=c["bits"]))


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how close two correct results are
# ---------------------------------------------------------------------------------------------------------------------

def _weight(n: int, k: int, bits: int = 4, gs: int = GS) -> float:
    return n * k * bits / 8 + 4 * n * k / gs


def work(case: dict) -> dict:
    c, m = case, case.get("rows", 0)
    kind = c["kind"]
    if kind == "linear":
        n, k = c["n"], c["k"]
        return {"bytes": _weight(n, k, c["bits"], c["gs"]) + 2 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "layer":
        h, i, nq, nkv = c["hidden"], c["inner"], c["q"], c["kv"]
        weights = (nq + 2 * nkv, h), (h, nq), (2 * i, h), (h, i)
        rows = 2 * h + nq + (nq + 2 * nkv + 2 * h)           # x, r and the attention's rows in; q, k, v, h and d out
        return {"bytes": sum(_weight(*w) for w in weights) + 2 * m * rows, "flops": sum(2 * m * n * k for n, k in weights)}
    if kind == "moe":
        d, w, e, t, sw = c["hidden"], c["width"], c["experts"], c["top_k"], c["shared"]
        touched = e * (1 - (1 - t / e) ** m)                 # experts that see a row, in expectation
        weights = touched * 3 * _weight(w, d) + 3 * _weight(sw, d) + 2 * (e + 1) * d
        return {"bytes": weights + 4 * m * d, "flops": 2 * m * d * (3 * w * t + 3 * sw + e + 1)}
    if kind == "rank":
        d, w, e, t, k = c["hidden"], c["width"], c["experts"], c["top_k"], c["o"] // c["world"]
        local, pairs = e // c["world"], m * t / c["world"]
        weights = local * (1 - (1 - t / e) ** m) * 3 * _weight(w, d) + _weight(d, k) + 2 * e * d
        return {"bytes": weights + 2 * m * (k + d) + (2 if m > EXACT_ROWS else 4) * m * d + 2 * m * d,
                "flops": 2 * pairs * 3 * w * d + 2 * m * d * (k + e)}
    if kind == "vocabulary":
        v, h = c["vocab"], c["hidden"]
        return {"bytes": _weight(v, h) + m * (_weight(1, h) + 2 * h) + 2 * m * v, "flops": 2 * m * v * h}
    return {"bytes": 2 * _weight(c["n"], c["k"], c["bits"], c["gs"]), "flops": 0}


def tolerance(case: dict):
    """bf16 results of fp32 sums: two correct orders of summation round a few values to neighbouring bf16 numbers, and a
    layer's later projections see those."""

    return "exact" if case["kind"] == "repack" else {"rel": 4e-3} if case["kind"] in ("linear", "vocabulary") else {"rel": 1e-2}
