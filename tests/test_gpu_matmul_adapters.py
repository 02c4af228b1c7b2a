"""GEMMs with low-rank adapters multiplied inside, against float64 (sm_100a)."""

import itertools

import pytest
import torch

from nano_omni_b200 import ops
from nano_omni_b200.core import DType, TensorDesc
from nano_omni_b200.kernels.matmul import MatmulBf16Arguments, MatmulBf16Kernel, MatmulInt8Arguments, MatmulInt8Kernel
from oracle import reference_math as rm

pytestmark = pytest.mark.gpu

# one row; ragged tiles; K of one chunk and of fewer chunks than the int8 form waits for; several tiles per pair of CTAs
# (74 pairs), so that both accumulators are used more than once
SHAPES = [(1, 64, 64), (130, 264, 512), (257, 520, 192), (300, 96, 1280), (2600, 4096, 128), (5200, 4104, 1408)]


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("ranks", [(64,), (128, 64)])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_adapters_join_the_sum(m, n, k, ranks, int8):
    g = torch.Generator(device="cuda").manual_seed(m + n + k + len(ranks))

    def normal(*shape, std=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()

    if int8:
        x, w = (torch.randint(-127, 128, s, generator=g, device="cuda", dtype=torch.int8) for s in ((m, k), (n, k)))
        ws = 0.5 + torch.rand(n, 1, generator=g, device="cuda")
        xs = (0.5 + torch.rand(m, generator=g, device="cuda")) / (5329 * k**0.5)
    else:
        x, w = normal(m, k), normal(n, k, std=k**-0.5)
    pairs = [(normal(m, r), normal(n, r, std=0.1)) for r in ranks]
    main = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    if int8:
        main, size = (v * ws.double().T * xs.double()[:, None] for v in (main, size))
    for a, b in pairs:
        main, size = main + a.double() @ b.double().T, size + a.double().abs() @ b.double().abs().T
    desc = TensorDesc.from_torch
    for use_bias, use_residual, use_silu in itertools.product((False, True), (False, True), (False, True)):
        bias, residual = normal(n) if use_bias else None, normal(m, n) if use_residual else None
        multiply = normal(m, n) if use_silu else None
        out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        optional = [None if t is None else desc(t) for t in (bias, residual, multiply)]
        adapters = tuple((desc(a), desc(b)) for a, b in pairs)
        if int8:
            MatmulInt8Kernel(
                MatmulInt8Arguments(desc(x), desc(w), *optional, desc(out), desc(ws), desc(xs), use_silu, adapters)
            ).submit()
        else:
            MatmulBf16Kernel(MatmulBf16Arguments(desc(x), desc(w), *optional, desc(out), 1.0, use_silu, adapters)).submit()
        want, bound = main, size
        for extra in (bias, residual):
            if extra is not None:
                want, bound = want + extra.double(), bound + extra.double().abs()
        if use_silu:  # its slope is at most 1.1; __expf and __fdividef are good to 2^-20
            want, bound = torch.nn.functional.silu(want) * multiply.double(), 1.1 * bound * multiply.double().abs()
        # one rounding to bf16 (8 significant bits: at most 2^-8 of the value), fp32 sums whose terms add up to `bound`
        error = (out.double() - want).abs()
        assert (error <= 2**-8 * 1.01 * want.abs() + 4e-6 * bound + 1e-30).all(), (error - 2**-8 * want.abs()).max()


def test_ranks_are_checked():
    desc = TensorDesc.empty
    x, w, out = desc(DType.BF16, (8, 64)), desc(DType.BF16, (16, 64)), desc(DType.BF16, (8, 16))
    for rank in (32, 96):
        pair = (desc(DType.BF16, (8, rank)), desc(DType.BF16, (16, rank)))
        with pytest.raises(AssertionError):
            MatmulBf16Kernel(MatmulBf16Arguments(x, w, None, None, None, out, 1.0, False, (pair,)))


class Siblings(ops.Op):
    """Projections of one input, each with (weight, weight scale or None, output, pairs)."""

    def __init__(self, x, projections, residual):
        desc = TensorDesc.from_torch
        super().__init__(desc(x), outputs=())
        self.residual = desc(residual)
        self.projections = [
            (desc(w), 1.0 if ws is None else desc(ws), desc(out), tuple((desc(a), desc(b), s) for a, b, s in loras))
            for w, ws, out, loras in projections
        ]

    def kernels(self, scratch):
        sequence = ops.KernelSequence(scratch)
        prepared = sequence.prepare(self.inputs[0])
        for i, (weight, scale, out, loras) in enumerate(self.projections):
            sequence.linear(f"p{i}", prepared, weight, out, weight_scale=scale, residual=self.residual, loras=loras)
        return sequence.calls


# ranks and strengths of each sibling's pairs, in order, the last two of whole chunks of 64 inside; whether siblings have their
# down-projections in common; GEMMs that are expected: compressions, updates outside and the projections themselves
ADAPTERS = {
    "one": ([[(64, 0.75)]], 1 + 1),
    "two strengths": ([[(64, 0.75), (128, -1.5)]], 2 + 1),
    "three, the last two inside": ([[(64, 2.0), (128, -0.75), (64, 0.5)]], 3 + 1 + 1),
    "one outside beside one inside": ([[(64, -0.75), (32, 1.5)]], 2 + 1 + 1),
    "siblings of one strength": ([[(64, 0.75)], [(64, 0.75)]], 1 + 2),
    "siblings of two strengths": ([[(64, 0.75)], [(64, -1.5)]], 1 + 1 + 2),
}


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("name", ADAPTERS)
def test_projections_with_adapters_against_float64(name, int8):
    m, n, k = 300, 264, 1024
    siblings, gemms = ADAPTERS[name]
    g = torch.Generator(device="cuda").manual_seed(len(name))

    def normal(*shape, std=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()

    x, residual = normal(m, k), normal(m, n)
    down = {rank: normal(rank, k, std=k**-0.5) for rank in (32, 64, 128)}
    projections = []
    for pairs in siblings:
        first = {rank: True for rank in down}
        loras = []
        for rank, strength in pairs:  # a second pair of a rank has a down-projection of its own
            a = down[rank] if first[rank] else normal(rank, k, std=k**-0.5)
            first[rank] = False
            loras.append((a, normal(n, rank, std=rank**-0.5), strength))
        if int8:
            w = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
            ws = (0.5 + torch.rand(n, 1, generator=g, device="cuda")) / (73 * k**0.5)
        else:
            w, ws = normal(n, k, std=k**-0.5), None
        projections.append((w, ws, torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda"), loras))
    op = Siblings(x, projections, residual).to()
    calls, need = op.prepare()
    assert sum(c.name.startswith("matmul") for c in calls) == gemms, [c.name for c in calls]
    op.run(torch.empty(max(need, 256), dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    if int8:
        quantised, scales = rm.int8_rowwise(x.cpu())
        quantised, scales = quantised.cuda().double(), scales.cuda().double()[:, None]
    for w, ws, out, loras in projections:
        if int8:
            main, size = (
                (a @ b.T) * scales * ws.double().T for a, b in ((quantised, w.double()), (quantised.abs(), w.double().abs()))
            )
        else:
            main, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        want, size = main + residual.double(), size + residual.double().abs()
        bound = torch.zeros_like(want)
        for a, b, strength in loras:
            compressed = strength * (x.double() @ a.double().T)
            want, size = want + compressed @ b.double().T, size + compressed.abs() @ b.double().abs().T
            # each compressed activation is rounded to bf16 once (at most 2^-8 of it), and an update outside the GEMM
            # rounds the residual and what was added to it so far
            bound += 2**-8 * compressed.abs() @ b.double().abs().T
        outside = max(0, gemms - len(siblings) - len({(a.data_ptr()) for *_, ls in projections for a, _, _ in ls}))
        bound += 2**-8 * (1.01 * want.abs() + outside * size) + 1e-5 * size
        error = (out.double() - want).abs()
        assert (error <= bound).all(), (name, float((error - bound).max()))
        # typical errors lie far below that bound of the worst case: a strength dropped or taken twice does not
        assert error.norm() < 0.006 * want.norm(), float(error.norm() / want.norm())
