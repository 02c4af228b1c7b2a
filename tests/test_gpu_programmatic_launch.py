"""Attention launched directly behind the kernel that writes one of its operands, nothing between and nothing waited for.

The kernels are programmatic dependents: their CTAs may be on the SMs while the quantiser before them still stores.  The
same calls with a synchronisation before the attention give the expected bits."""

import pytest
import torch

from nano_omni_b200 import _lib
from nano_omni_b200.core import DType
from nano_omni_b200.kernels.dense_int8_fp8 import DenseInt8Fp8AttentionArguments, DenseInt8Fp8AttentionKernel
from nano_omni_b200.kernels.dense_nvfp4 import DenseNvfp4Arguments, DenseNvfp4Kernel
from nano_omni_b200.kernels.quantize import (
    Int8Fp8QuantizeQKArguments,
    Int8Fp8QuantizeQKKernel,
    Int8Fp8QuantizeValueArguments,
    Int8Fp8QuantizeValueKernel,
    Int8Fp8ValueScaleArguments,
    Int8Fp8ValueScaleKernel,
    Nvfp4PrepareArguments,
    Nvfp4PrepareKernel,
)
from nano_omni_b200.kernels.sol import (
    SolNvfp4SelectArguments,
    SolNvfp4SelectKernel,
    SolPoolArguments,
    SolPoolKernel,
    SolStatsArguments,
    SolStatsKernel,
)
from nano_omni_b200.kernels.sol_exact import (
    SolInt8Fp8AttentionArguments,
    SolInt8Fp8AttentionKernel,
    SolNvfp4Arguments,
    SolNvfp4Kernel,
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


def run_behind(kernels, outputs, wait):
    """The kernels in order, all but the last one's launch behind a synchronisation if ``wait``; copies of the outputs."""
    for kernel in kernels[:-1]:
        kernel.submit()
    if wait:
        torch.cuda.synchronize()
    kernels[-1].submit()
    assert _lib.read_status() == 0
    return [x.clone() for x in outputs]


def nvfp4_operands(h, T):
    """(sources, tensors, kernels by name) of Q, K and V through the nvfp4 quantiser."""
    P = -(-T // 128) * 128
    sources, tensors, kernels = {}, {}, {}
    for i, name in enumerate(("query", "key", "value")):
        rows, columns = (128, P) if name == "value" else (P, 128)
        sources[name] = randn_bf16(81 + i, T, h * 128)
        tensors[name] = (
            torch.empty(h, rows, columns // 2, dtype=torch.uint8, device="cuda"),
            torch.empty(h, rows, columns // 16, dtype=torch.uint8, device="cuda"),
        )
        packed, scales = tensors[name]
        kernels[name] = Nvfp4PrepareKernel(
            Nvfp4PrepareArguments(desc(sources[name]), None, desc(packed), desc(scales, DType.FP8_UE4M3), h, name == "value")
        )
    return sources, tensors, kernels


def nvfp4_descriptors(tensors):
    order = ("query", "key", "value")
    return [desc(tensors[n][0]) for n in order] + [desc(tensors[n][1], DType.FP8_UE4M3) for n in order]


@pytest.mark.parametrize("T", [900, 9000])
@pytest.mark.parametrize("last", ["key", "query", "value"])
def test_nvfp4_attention_behind_the_quantiser_of_its_operand(last, T):
    h = 8
    sources, tensors, kernels = nvfp4_operands(h, T)
    base = {name: x.clone() for name, x in sources.items()}
    out = torch.empty(T, h, 128, dtype=torch.bfloat16, device="cuda")
    attention = DenseNvfp4Kernel(DenseNvfp4Arguments(*nvfp4_descriptors(tensors), desc(out), T, T, 0))
    chain = [kernel for name, kernel in kernels.items() if name != last] + [kernels[last], attention]
    for i in range(6):
        results = []
        for wait in (True, False):
            for name, x in sources.items():
                x.copy_(base[name] * (0.5 + i))
            for _, scales in tensors.values():
                scales.fill_(0x7F)  # NaN: what an early read would see
            out.fill_(float("nan"))
            torch.cuda.synchronize()
            results.append(run_behind(chain, [out], wait)[0])
        assert torch.isfinite(results[0]).all() and torch.equal(*(r.view(torch.int16) for r in results))


@pytest.mark.parametrize("T", [900, 9000])
@pytest.mark.parametrize("last", ["mask", "key", "value"])
@pytest.mark.parametrize("precision", ["int8_fp8", "nvfp4"])
def test_sol_attention_behind_the_selector_and_the_quantisers(precision, last, T):
    h, nb = 8, -(-T // 64)
    mask = torch.empty(nb, h, nb, dtype=torch.uint8, device="cuda")
    if precision == "nvfp4":
        sources, tensors, kernels = nvfp4_operands(h, T)
        scales = [s for _, s in tensors.values()]
        descriptors = nvfp4_descriptors(tensors)
    else:
        sources = {name: randn_bf16(91 + i, T, h * 128) for i, name in enumerate(("query", "key", "value"))}
        mean = torch.zeros(1, h * 128, device="cuda")
        k_rows = nb * 64
        q8 = torch.empty(h, -(-T // 32) * 32, 128, dtype=torch.int8, device="cuda")
        k8 = torch.empty(h, k_rows, 128, dtype=torch.int8, device="cuda")
        v8 = torch.empty(h, 128, k_rows, dtype=torch.uint8, device="cuda")
        qs, ks, vs = (torch.empty(h, n, device="cuda") for n in (-(-T // 32), nb, 128))
        scales = [qs, ks, vs]
        q, k, v = (desc(sources[name]) for name in ("query", "key", "value"))
        v_scale = Int8Fp8ValueScaleKernel(Int8Fp8ValueScaleArguments(v, desc(vs), h))
        kernels = {
            "query": Int8Fp8QuantizeQKKernel(Int8Fp8QuantizeQKArguments(q, desc(mean), desc(q8), desc(qs), h, 32, False)),
            "key": Int8Fp8QuantizeQKKernel(Int8Fp8QuantizeQKArguments(k, desc(mean), desc(k8), desc(ks), h, 64, False)),
            "value": Int8Fp8QuantizeValueKernel(Int8Fp8QuantizeValueArguments(v, desc(vs), desc(v8, DType.FP8_E4M3), h)),
        }
        descriptors = [desc(q8), desc(k8), desc(v8, DType.FP8_E4M3), desc(qs), desc(ks), desc(vs)]
    base = {name: x.clone() for name, x in sources.items()}
    # the selector reads Q and pooled K, which are there before the chain begins
    pooled = torch.empty(2, h, nb, 128, dtype=torch.bfloat16, device="cuda")
    stats = torch.empty(h, 2, 128, device="cuda")
    heads = {name: x.view(T, h, 128) for name, x in sources.items()}
    pool = SolPoolKernel(SolPoolArguments(desc(heads["key"]), desc(heads["value"]), desc(pooled)))
    statistics = SolStatsKernel(SolStatsArguments(desc(pooled), desc(stats)))
    kernels["mask"] = SolNvfp4SelectKernel(
        SolNvfp4SelectArguments(desc(heads["query"]), desc(pooled[0]), desc(stats), desc(mask), 1.0, 1)
    )
    out = torch.empty(T, h, 128, dtype=torch.bfloat16, device="cuda")
    state = torch.empty(T, h, 2, device="cuda")
    if precision == "nvfp4":
        attention = SolNvfp4Kernel(SolNvfp4Arguments(*descriptors, desc(mask), desc(out), desc(state), T, T, 0, 1.0, 1))
    else:
        attention = SolInt8Fp8AttentionKernel(
            SolInt8Fp8AttentionArguments(*descriptors, desc(mask), desc(out), desc(state), T, 0, 1.0, 1)
        )
    chain = [kernel for name, kernel in kernels.items() if name != last] + [kernels[last], attention]
    if precision == "int8_fp8":
        chain.insert(0, v_scale)
    for i in range(6):
        results = []
        for wait in (True, False):
            for name, x in sources.items():
                # other scales, and other blocks chosen, in the same tensors every time
                x.copy_(base[name].roll(64 * i, 0) * (0.5 + i))
            for tensor in scales:
                tensor.fill_(0x7F if tensor.dtype == torch.uint8 else float("nan"))
            pool.submit()
            statistics.submit()
            mask.fill_(1)
            torch.cuda.synchronize()
            results.append(run_behind(chain, [out, state], wait))
        (want, want_state), (got, got_state) = results
        assert torch.isfinite(want).all() and not mask.all()
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)) and torch.equal(got_state, want_state)
