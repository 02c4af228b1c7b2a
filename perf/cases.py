"""The attention and projection work that users of this framework have it do, as cases that can be timed and compared.

A case is one operator of ``nano_omni_b200.ops`` at one shape.  ``prepare`` makes what a generation program holds before
a denoising step (activations, weights, the planned operator, its scratch arena); ``run`` is one ``Op.run`` of it.
The shapes are those of the benchmark (24 heads), of the 7168-wide transformer (56 heads in slices of 14, hidden size
5376, rank-64 adapters) and generic odd ones, from a single small image to a long video.
"""

import math

import torch

from nano_omni_b200 import ops
from nano_omni_b200.core import TensorDesc

DIM = 128
HIDDEN = 5376  # columns of the transformer's residual stream
WIDE = 7168  # 56 heads x 128
SLICE_ROWS = 4096  # queries of one slice where K and V are quantised once and kept


def listed():
    return [
        # the routing-free correctness shape of the benchmark: a small image, one launch
        {"name": "dense_bf16_small", "kind": "dense_bf16", "tokens": 4096, "heads": 4, "total_heads": 4, "rotate": False},
        # one head slice of a short clip, straight from the projections (norm and rotary embedding inside), odd length
        {"name": "dense_bf16_slice_rope", "kind": "dense_bf16", "tokens": 9461, "heads": 14, "total_heads": 56, "rotate": True},
        # the headline benchmark: a video of 32256 tokens with 512 text tokens
        {"name": "dense_bf16_headline", "kind": "dense_bf16", "tokens": 32768, "heads": 24, "total_heads": 24, "rotate": False},
        # the smallest quantised call: text and a thumbnail; seven short launches
        {"name": "dense_int8_fp8_tiny", "kind": "dense_int8_fp8", "tokens": 1021, "heads": 14, "total_heads": 14, "rotate": True},
        # a video attended in query slices against K and V quantised once, as when activations are offloaded
        {"name": "int8_fp8_query_slices", "kind": "slices", "tokens": 30389, "heads": 24, "total_heads": 24, "rotate": True},
        # a medium video at the lowest precision
        {"name": "dense_nvfp4_medium", "kind": "dense_nvfp4", "tokens": 20011, "heads": 24, "total_heads": 24, "rotate": False},
        # threshold routing over 64-token blocks, a head slice of a short clip
        {"name": "sol_bf16_threshold", "kind": "sol_bf16", "tokens": 7310, "heads": 14, "total_heads": 56, "rotate": True, "block": 64},
        # the benchmark's long video: 128-token blocks, the top quarter of the key blocks
        {"name": "sol_bf16_long", "kind": "sol_bf16", "tokens": 131072, "heads": 24, "total_heads": 24, "rotate": False, "block": 128},
        # a head slice of a full-length generation with quantised block-sparse attention
        {"name": "sol_int8_fp8_slice", "kind": "sol_int8_fp8", "tokens": 60778, "heads": 14, "total_heads": 56, "rotate": False},
        # the same at nvfp4 and the headline's length
        {"name": "sol_nvfp4_medium", "kind": "sol_nvfp4", "tokens": 32768, "heads": 24, "total_heads": 24, "rotate": False},
        # the output-side projection of a clip: int8 weights, rotated activations, one adapter, residual
        {"name": "linear_int8_adapter", "kind": "linear_int8", "tokens": 15104, "n": HIDDEN, "k": WIDE, "adapters": 1, "residual": True},
        # a projection of the text tokens alone
        {"name": "linear_bf16_text", "kind": "linear_bf16", "tokens": 512, "n": WIDE, "k": HIDDEN, "adapters": 0, "residual": False},
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(
        ["dense_bf16", "dense_int8_fp8", "slices", "dense_nvfp4", "sol_bf16", "sol_int8_fp8", "sol_nvfp4", "linear_int8", "linear_bf16"]
    )
    if kind.startswith("linear"):
        n, k = rng.choice([(HIDDEN, WIDE), (WIDE, HIDDEN), (WIDE, WIDE), (HIDDEN, HIDDEN)])
        return {
            "kind": kind, "tokens": _log_between(rng, 256, 60778), "n": n, "k": k,
            "adapters": rng.choice([0, 1]), "residual": rng.random() < 0.5,
        }  # fmt: skip
    heads = rng.choice([4, 6, 8, 14, 24])
    block = rng.choice([64, 128]) if kind == "sol_bf16" else 64
    shortest = 6000 if kind == "slices" else 640
    longest = 60778 if not kind.startswith("sol") else 131072 if block == 128 else 65536
    # dense work grows with tokens^2: many heads only at the lengths that keep a call below the long sol case
    while True:
        tokens = _log_between(rng, shortest, longest)
        if kind.startswith("sol") or tokens * tokens * heads <= 3.2e10:
            break
    case = {
        "kind": kind, "tokens": tokens, "heads": heads,
        "total_heads": heads if kind in ("dense_int8_fp8", "slices") else heads * rng.choice([1, 4]),
        "rotate": rng.random() < 0.5,
    }  # fmt: skip
    if kind == "sol_bf16":
        case["block"] = block
    return case


# ---------------------------------------------------------------------------------------------------- inputs
def _normal(generator, *shape, std=1.0):
    return torch.randn(*shape, generator=generator, device="cuda", dtype=torch.float32) * std


def _qkv(case, generator):
    """Q, K, V [tokens, heads * 128] bf16.  Unit-variance noise on patterns shared by neighbouring tokens (what routing
    by block means finds), one outlier channel of K per head, and a per-channel offset of V."""
    t, h = case["tokens"], case["heads"]
    near, far = -(-t // 64), -(-t // 512)
    q = _normal(generator, t, h, DIM)
    q += _normal(generator, far, h, DIM, std=0.3).repeat_interleave(512, 0)[:t]
    k = _normal(generator, t, h, DIM)
    k += _normal(generator, near, h, DIM, std=0.3).repeat_interleave(64, 0)[:t]
    channel = torch.randint(0, DIM, (h,), generator=generator, device="cuda")
    k[:, torch.arange(h, device="cuda"), channel] *= 8.0
    v = _normal(generator, t, h, DIM) + _normal(generator, 1, h, DIM, std=0.25)
    return tuple(x.bfloat16().view(t, h * DIM) for x in (q, k, v))


def _rotation(case, generator, rows=None):
    """Norm weights near one and rotary planes of growing frequency; ``rows`` takes a part of the planes."""
    t = case["tokens"]
    weights = [(1.0 + _normal(generator, DIM, std=0.1)).bfloat16() for _ in range(2)]
    angle = torch.arange(t, device="cuda", dtype=torch.float32)[:, None] * torch.logspace(0, -4, 48, device="cuda")
    return weights, angle.cos().contiguous(), angle.sin().contiguous()


def _arena(num_bytes):
    buffer = torch.empty(num_bytes + 256, dtype=torch.uint8, device="cuda")
    return buffer[(-buffer.data_ptr()) % 256 :]


def prepare(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    kind, t, desc = case["kind"], case["tokens"], TensorDesc.from_torch
    if kind.startswith("linear"):
        return _prepare_linear(case, generator)
    h, total = case["heads"], case["total_heads"]
    q, k, v = _qkv(case, generator)
    rotation = None
    if case["rotate"]:
        (query_norm, key_norm), cosines, sines = _rotation(case, generator)
        rotation = ops.Rotation(desc(query_norm), desc(key_norm), desc(cosines), desc(sines))
    if kind == "slices":
        padded = -(-t // 64) * 64
        kept = (
            torch.empty(h, padded, DIM, dtype=torch.int8, device="cuda"),
            torch.empty(h, padded // 64, device="cuda"),
            torch.empty(h, DIM, padded, dtype=torch.float8_e4m3fn, device="cuda"),
            torch.empty(h, DIM, device="cuda"),
        )
        out = torch.empty(t, h * DIM, dtype=torch.bfloat16, device="cuda")
        steps = [ops.PrepareKeyValue(desc(k), desc(v), rotation=rotation).to(*(desc(x) for x in kept))]
        for start in range(0, t, SLICE_ROWS):
            rows = slice(start, min(t, start + SLICE_ROWS))
            part = rotation and ops.Rotation(rotation.query_norm, rotation.key_norm, desc(cosines[rows]), desc(sines[rows]))
            step = ops.QuerySlice(desc(q[rows]), *(desc(x) for x in kept), total_tokens=t, rotation=part)
            steps.append(step.to(desc(out[rows])))
        scratch = _arena(max(step.prepare()[1] for step in steps))
        return {"steps": steps, "scratch": scratch, "out": out}
    # a slice of heads is written beside the others into the full-width tensor
    options = {"rotation": rotation}
    if kind != "dense_int8_fp8":
        options |= {"total_heads": total, "head_offset": (total - h) // 2}
    if kind.startswith("sol"):
        options["protected_tokens"] = min(512, t // 4)
    if kind == "sol_bf16":
        options |= {"block": case["block"], "topk_fraction": 0.25 if case["block"] == 128 else 0.0}
    attention, precision = kind.split("_", 1)
    op = ops.ATTENTION_OPS[(attention, precision)](desc(q), desc(k), desc(v), **options)
    out = torch.zeros(*op.output_specs[0][1], dtype=torch.bfloat16, device="cuda")
    op.to(desc(out))
    return {"steps": [op], "scratch": _arena(op.prepare()[1]), "out": out}


def _prepare_linear(case, generator):
    t, n, k, desc = case["tokens"], case["n"], case["k"], TensorDesc.from_torch
    x = _normal(generator, t, k)
    x[:, torch.randint(0, k, (k // 128,), generator=generator, device="cuda")] *= 8.0  # outlier channels
    x = x.bfloat16()
    options = {}
    if case["kind"] == "linear_int8":
        weight = torch.randint(-127, 128, (n, k), generator=generator, device="cuda", dtype=torch.int8)
        options["weight_scale"] = desc((0.5 + torch.rand(n, 1, generator=generator, device="cuda")) / (73 * math.sqrt(k)))
        options["rotation_group"] = 256
    else:
        weight = _normal(generator, n, k, std=1 / math.sqrt(k)).bfloat16()
        options["bias"] = desc(_normal(generator, n, std=0.1).bfloat16())
    if case["residual"]:
        options["residual"] = desc(_normal(generator, t, n).bfloat16())
    options["loras"] = tuple(
        (desc(_normal(generator, 64, k, std=1 / math.sqrt(k)).bfloat16()), desc(_normal(generator, n, 64, std=0.02).bfloat16()), 0.8)
        for _ in range(case["adapters"])
    )
    out = torch.empty(t, n, dtype=torch.bfloat16, device="cuda")
    op = ops.Linear(desc(x), desc(weight), **options).to(desc(out))
    return {"steps": [op], "scratch": _arena(op.prepare()[1]), "out": out}


# ---------------------------------------------------------------------------------------------------- one pass
def run(state):
    for step in state["steps"]:
        step.run(state["scratch"])
    return state["out"]


# ---------------------------------------------------------------------------------------------------- figures
def work(case):
    """Inputs read once and outputs written once; two operations per multiply-add that the result needs."""
    kind, t = case["kind"], case["tokens"]
    if kind.startswith("linear"):
        n, k, ranks = case["n"], case["k"], 64 * case["adapters"]
        weight = n * k * (1 if kind == "linear_int8" else 2)
        traffic = 2 * t * k + weight + 2 * ranks * (n + k) + 2 * t * n * (2 if case["residual"] else 1)
        return {"bytes": traffic, "flops": 2 * t * n * k + 2 * t * ranks * (n + k)}
    h = case["heads"]
    traffic = 4 * t * h * DIM * 2 + (t * 48 * 4 * 2 if case["rotate"] else 0)
    share, routing = 1.0, 0
    if kind.startswith("sol"):
        block = case.get("block", 64)
        blocks = -(-t // block)
        # the top quarter, or the blocks more than one standard deviation above the mean; and the protected ones
        share = min(1.0, (0.25 if block == 128 else 0.16) + min(512, t // 4) / t)
        # block scores, and the pooled blocks that stand in for the unselected ones
        routing = 2 * h * blocks * blocks * DIM + 4 * h * t * blocks * DIM
    return {"bytes": traffic, "flops": 4 * h * t * t * DIM * share + routing}


def tolerance(case):
    """bf16 results; where probabilities are rounded to e4m3 (3 bits) or e2m1 (1 bit) the grid they are rounded on may
    differ between correct implementations, and shows in the part of the output that the values' noise makes up."""
    kind = case["kind"]
    if kind in ("dense_int8_fp8", "slices", "sol_int8_fp8"):
        return {"rel": 0.02}
    if kind in ("dense_nvfp4", "sol_nvfp4"):
        return {"rel": 0.03}
    return {"rel": 0.01}
