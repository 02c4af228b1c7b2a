"""Branches of the statistics and row-wise quantisers that depend on the size, bit for bit at their edges."""

import pytest
import torch

from oracle import reference_math as rm
from tests.gpu_util import desc, randn_bf16, run
from tests.test_gpu_norm_rope import rowwise
from tests.test_gpu_quantize import _mean

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [7, 64, 513, 2047, 2048, 2049])  # one CTA per 64 columns up to 2048 tokens
def test_value_scale_short_and_long(T):
    from nano_omni_b200.kernels.quantize import Int8Fp8ValueScaleArguments, Int8Fp8ValueScaleKernel

    h = 3
    src = randn_bf16(300 + T, T, h * 128, outlier=True)
    scale = torch.full((h, 128), float("nan"), device="cuda")
    run(Int8Fp8ValueScaleKernel(Int8Fp8ValueScaleArguments(desc(src), desc(scale), h)))
    assert torch.equal(scale.cpu(), rm.int8_fp8_value_scale(src.cpu(), h))


@pytest.mark.parametrize("T", [31, 32, 33, 96, 127, 128, 159, 160, 161])  # batches of 32 tokens in chunks of 128
def test_mean_batches(T):
    src = randn_bf16(400 + T, T, 256, outlier=True)
    assert torch.equal(_mean(src, T, False).cpu(), rm.token_group_mean(src.cpu(), T, False))


@pytest.mark.parametrize("groups", [1, 8, 9, 15, 16, 17, 28])  # a round rotates 16 groups, two per half-warp
def test_rowwise_rounds(groups):
    src = randn_bf16(500 + groups, 5, groups * 256, outlier=True).cpu()
    src[1] = 0.0
    src[2] *= 1e-30  # the scale's lower bound
    got_q, got_s = rowwise(src, 256)
    want_q, want_s = rm.int8_rowwise(src, 256)
    assert torch.equal(got_s, want_s) and torch.equal(got_q, want_q)


def test_rowwise_non_finite_columns():
    """An infinite column makes the scale infinite: finite columns give 0, infinite ones and NaNs -127."""
    src = randn_bf16(600, 1, 264).cpu()
    src[0, 5], src[0, 6], src[0, 260] = float("inf"), float("-inf"), float("nan")
    got_q, got_s = rowwise(src, 0)
    want = torch.zeros(1, 264, dtype=torch.int8)
    want[0, [5, 6, 260]] = -127
    assert got_s.isinf().all() and torch.equal(got_q, want)
