"""Which calls a projection with low-rank adapters becomes, and what the C entries with adapters refuse before a launch."""

import ctypes

import pytest

from nano_omni_b200 import _lib, ops
from nano_omni_b200.core import DType, ScratchLayout, TensorDesc

TOKENS, K = 300, 1024
WEIGHT = (0x11000000, 0)  # where the projection's own weight lies


def tensor(index, dtype, *shape):
    return TensorDesc.from_pointer(0x10000000 + index * 0x1000000, dtype, shape)


def project(prepared, name, n, loras):
    sequence, first = prepared.sequence, len(prepared.sequence.calls)
    weight, out = tensor(1, DType.BF16, n, K), tensor(2, DType.BF16, TOKENS, n)
    sequence.linear(name, prepared, weight, out, loras=loras)
    return sequence.calls[first:]


def pair(index, rank, n, strength):
    return tensor(10 + index, DType.BF16, rank, K), tensor(40 + index, DType.BF16, n, rank), strength


def start():
    return ops.KernelSequence(ScratchLayout()).prepare(tensor(0, DType.BF16, TOKENS, K))


def compressions(calls, prepared):
    return [c for c in calls if c.arguments.input == prepared.input and c.arguments.weight.info != WEIGHT]


def test_siblings_of_one_strength_share_the_compression_inside():
    prepared = start()
    first, second = (project(prepared, name, 256, (pair(0, 64, 256, 0.5),)) for name in "ab")
    assert [len(first), len(second)] == [2, 1]
    assert first[1].arguments.adapters[0][0] == second[0].arguments.adapters[0][0] == first[0].arguments.output
    assert first[0].arguments.output_scale == 0.5


def test_siblings_of_two_strengths_share_it_where_reading_the_input_again_costs_more():
    prepared = start()
    first, second = (project(prepared, name, 256, (pair(0, 64, 256, s),)) for name, s in (("a", 0.5), ("b", -2.0)))
    assert len(compressions(first, prepared)) == 1 and not compressions(second, prepared)
    update, main = second
    assert update.arguments.input == first[0].arguments.output and update.arguments.output_scale == -4.0
    assert main.arguments.residual == update.arguments.output and not main.arguments.adapters
    # and with a wide output both are inside
    prepared = start()
    first, second = (project(prepared, name, 512, (pair(0, 64, 512, s),)) for name, s in (("a", 0.5), ("b", -2.0)))
    assert len(compressions(second, prepared)) == 1 and second[0].arguments.output_scale == -2.0
    assert second[1].arguments.adapters and second[1].arguments.residual is None


def test_the_last_two_pairs_of_whole_chunks_are_inside():
    prepared = start()
    loras = tuple(pair(i, rank, 1024, 0.5 + i) for i, rank in enumerate((64, 32, 128, 64)))
    calls = project(prepared, "a", 1024, loras)
    main = calls[-1].arguments
    assert [a.shape[1] for a, _ in main.adapters] == [128, 64] and [b for _, b in main.adapters] == [loras[2][1], loras[3][1]]
    down = compressions(calls, prepared)
    assert [c.arguments.output_scale for c in down] == [1.0, 1.0, 2.5, 3.5]
    updates = [c for c in calls[:-1] if c not in down]
    assert [c.arguments.output_scale for c in updates] == [0.5, 1.5]
    assert updates[1].arguments.residual == updates[0].arguments.output and main.residual == updates[1].arguments.output


@pytest.mark.parametrize("strength", [0.0, 1e-30, 1e30])
def test_a_strength_out_of_the_ordinary_scales_the_fp32_sum(strength):
    prepared = start()
    project(prepared, "a", 256, (pair(0, 64, 256, 0.5),))
    compression, update, main = project(prepared, "b", 256, (pair(0, 64, 256, strength),))
    assert compression.arguments.output_scale == 1.0 and update.arguments.output_scale == strength
    assert not main.arguments.adapters


@pytest.mark.parametrize("strength", [float("nan"), float("inf")])
def test_a_strength_that_is_no_number_is_refused(strength):
    with pytest.raises(ValueError):
        project(start(), "a", 256, (pair(0, 64, 256, strength),))


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize(
    "ranks,missing", [((0, 0), None), ((96, 0), None), ((64, 32), None), ((-64, 0), None), ((64, 64), 1), ((64, 0), 0)]
)
def test_the_c_entries_refuse_ranks_and_absent_tensors(int8, ranks, missing):
    """The checks come ahead of every use of the pointers, which are only marks here."""
    mark, null, i = ctypes.c_void_p(0x1000), ctypes.c_void_p(0), ctypes.c_int
    adapters = []
    for index, rank in enumerate(ranks):
        adapters += mark if rank else null, null if missing == index else (mark if rank else null), i(rank)
    scales = [mark, mark] if int8 else []
    function = _lib.symbol("nob200_matmul_int8_adapters" if int8 else "nob200_matmul_bf16_adapters")
    code = function(i(8), mark, mark, null, null, null, mark, *scales, i(16), i(64), i(0), *adapters, ctypes.c_void_p(0))
    assert code != 0 and ("rank" in _lib.last_error() or "NULL" in _lib.last_error())
