"""Attention launched directly behind the kernel that writes one of its operands, nothing between and nothing waited for.

The kernels are programmatic dependents: their CTAs may be on the SMs while the quantiser before them still stores.  The
same calls with a synchronisation before the attention give the expected bits."""

import pytest
import torch

from nano_omni_b200 import _lib
from nano_omni_b200.core import DType
from nano_omni_b200.kernels.dense_int8_fp8 import DenseInt8Fp8AttentionArguments, DenseInt8Fp8AttentionKernel
from nano_omni_b200.kernels.quantize import (
    Int8Fp8QuantizeQKArguments,
    Int8Fp8QuantizeQKKernel,
    Int8Fp8QuantizeValueArguments,
    Int8Fp8QuantizeValueKernel,
    Int8Fp8ValueScaleArguments,
    Int8Fp8ValueScaleKernel,
)
from tests.gpu_util import desc, randn_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", ["key", "query", "value"])
def test_attention_behind_the_quantiser_of_its_operand(last):
    h, Tq, Tk = 8, 1000, 20011
    q, v = randn_bf16(71, Tq, h * 128), randn_bf16(72, Tk, h * 128)
    base = randn_bf16(73, Tk, h * 128)
    mean = torch.zeros(1, h * 128, device="cuda")
    q8 = torch.empty(h, -(-Tq // 32) * 32, 128, dtype=torch.int8, device="cuda")
    qs = torch.empty(h, -(-Tq // 32), device="cuda")
    k8 = torch.empty(h, -(-Tk // 64) * 64, 128, dtype=torch.int8, device="cuda")
    ks = torch.empty(h, -(-Tk // 64), device="cuda")
    v8 = torch.empty(h, 128, -(-Tk // 64) * 64, dtype=torch.uint8, device="cuda")
    vs = torch.empty(h, 128, device="cuda")

    def attend(k, out, wait):
        for tensor in (qs, ks, vs):  # what an early read would see
            tensor.fill_(float("nan"))
        quantise = {
            "value": [
                Int8Fp8ValueScaleKernel(Int8Fp8ValueScaleArguments(desc(v), desc(vs), h)),
                Int8Fp8QuantizeValueKernel(Int8Fp8QuantizeValueArguments(desc(v), desc(vs), desc(v8, DType.FP8_E4M3), h)),
            ],
            "query": [Int8Fp8QuantizeQKKernel(Int8Fp8QuantizeQKArguments(desc(q), desc(mean), desc(q8), desc(qs), h, 32, False))],
            "key": [Int8Fp8QuantizeQKKernel(Int8Fp8QuantizeQKArguments(desc(k), desc(mean), desc(k8), desc(ks), h, 64, False))],
        }
        attention = DenseInt8Fp8AttentionKernel(
            DenseInt8Fp8AttentionArguments(
                desc(q8), desc(k8), desc(v8, DType.FP8_E4M3), desc(qs), desc(ks), desc(vs), desc(out), Tk, h, Tq
            )
        )
        order = [name for name in quantise if name != last] + [last]
        torch.cuda.synchronize()
        for kernel in [kernel for name in order for kernel in quantise[name]]:
            kernel.submit()
        if wait:
            torch.cuda.synchronize()
        attention.submit()
        assert _lib.read_status() == 0

    for i in range(8):
        k = base * (0.5 + i)  # other scales in the same tensor every time
        want, got = (torch.empty(Tq, h * 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        attend(k, want, True)
        attend(k, got, False)
        assert torch.isfinite(want).all() and torch.equal(got.view(torch.int16), want.view(torch.int16))
