"""GEMMs with low-rank adapters multiplied inside, against float64 (sm_100a)."""

import itertools

import pytest
import torch

from nano_omni_b200.core import DType, TensorDesc
from nano_omni_b200.kernels.matmul import MatmulBf16Arguments, MatmulBf16Kernel, MatmulInt8Arguments, MatmulInt8Kernel

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
