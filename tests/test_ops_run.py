"""``Op.run`` on CPU: the C calls it makes are those of its kernels' ``submit``, also after a change of scratch or options.

Stand-ins for the library's symbols note every call, so nothing is launched and no GPU is needed.
"""

import ctypes

import pytest
import torch

from nano_omni_b200 import _lib, ops
from nano_omni_b200.core import DType, Kernel, TensorDesc
from nano_omni_b200.kernels.dense_bf16 import UnitPlan
from tests.test_ops_plan import EXPECTED, make


@pytest.fixture
def calls(monkeypatch):
    made = []

    def symbol(name):
        def call(*arguments):
            made.append((name, tuple(getattr(a, "value", a) for a in arguments)))
            return 0

        call.__name__ = name
        return call

    monkeypatch.setattr(_lib, "symbol", symbol)
    return made


def arena(num_bytes):
    buffer = torch.empty(num_bytes + 256, dtype=torch.uint8)
    return buffer[(-buffer.data_ptr()) % 256 :]


def submitted(op, scratch, stream, calls):
    del calls[:]
    for kernel in op.bind(scratch.data_ptr()):
        kernel.submit(stream)
    expected = list(calls)
    del calls[:]
    return expected


def linear(tokens=300, n=256, k=512, **options):
    pointer = iter(range(0x10000000, 0x60000000, 0x8000000))
    x = TensorDesc.from_pointer(next(pointer), DType.BF16, (tokens, k))
    weight = TensorDesc.from_pointer(next(pointer), DType.BF16, (n, k))
    return ops.Linear(x, weight, **options).to(TensorDesc.from_pointer(next(pointer), DType.BF16, (tokens, n)))


@pytest.mark.parametrize("kind,precision", list(EXPECTED))
def test_run_makes_the_calls_of_submit(calls, kind, precision):
    """Two addresses in turn, then more of them than plans are kept, on streams of their own."""
    op = make(kind, precision)
    need = op.prepare()[1]
    arenas = [arena(need) for _ in range(6)]
    for round, index in enumerate((0, 0, 1, 0, 1, 2, 3, 4, 5, 0, 5)):
        stream = 0x100 + round
        expected = submitted(op, arenas[index], stream, calls)
        op.run(arenas[index], stream)
        assert calls == expected
        assert len(op._plans) <= ops._KEPT_PLANS


def test_scratch_is_checked_on_every_run(calls):
    op = make("sol", "bf16")
    scratch = arena(op.prepare()[1])
    op.run(scratch, 1)
    with pytest.raises(AssertionError):
        op.run(scratch[:256], 1)  # the same address
    with pytest.raises(AssertionError):
        op.run(scratch[1:], 1)


CHANGES = {
    "tau": lambda: (make("sol", "bf16"), lambda op: setattr(op, "tau", 0.25)),
    "topk_fraction": lambda: (make("sol", "bf16"), lambda op: setattr(op, "topk_fraction", 0.5)),
    "head_offset": lambda: (make("dense", "nvfp4"), lambda op: setattr(op, "head_offset", 0)),
    "global_scales": lambda: (make("dense", "nvfp4"), lambda op: setattr(op, "global_scales", (1.0, 2.0, 3.0))),
    "hadamard": lambda: (make("dense", "int8_fp8"), lambda op: setattr(op, "hadamard", True)),
    "inputs": lambda: (make("dense", "bf16"), lambda op: setattr(op, "inputs", (op.inputs[1], op.inputs[0], op.inputs[2]))),
    "kv_splits": lambda: (make("dense", "bf16"), lambda op: setattr(op, "kv_splits", 2)),
    "options": lambda: (linear(), lambda op: op.options.update(use_silu=True)),
    "options replaced": lambda: (linear(), lambda op: setattr(op, "options", {"use_silu": True})),
    "loras": lambda: (linear(loras=[]), lambda op: op.options["loras"].append(adapter())),
    "strength": lambda: (linear(loras=[list(adapter())]), lambda op: op.options["loras"][0].__setitem__(2, 0.25)),
}


def adapter():
    down = TensorDesc.from_pointer(0x70000000, DType.BF16, (64, 512))
    return down, TensorDesc.from_pointer(0x71000000, DType.BF16, (256, 64)), 0.5


@pytest.mark.parametrize("what", list(CHANGES))
def test_an_option_changed_after_a_run_counts(calls, what):
    op, change = CHANGES[what]()
    scratch = arena(1 << 24)
    before = submitted(op, scratch, 1, calls)
    op.run(scratch, 1)
    assert calls == before
    change(op)
    after = submitted(op, scratch, 1, calls)
    op.run(scratch, 1)
    assert calls == after != before


def test_key_split_count_divides_every_unit(calls):
    op = make("dense", "bf16")
    op.kv_splits = 3
    assert op.kv_splits == 3 and op.prepare()[0][-1].config.kv_splits == 3 and op.units == UnitPlan(256, 3, 0)


def test_submit_of_a_kernel_class_is_called(calls, monkeypatch):
    """Classes (or tools) that put their own ``submit`` around a launch see the launches of operators too."""
    op = make("sol", "bf16")
    scratch = arena(op.prepare()[1])
    expected = submitted(op, scratch, 0, calls)
    op.run(scratch, 0)
    assert calls == expected
    seen = []
    plain = Kernel.submit
    monkeypatch.setattr(Kernel, "submit", lambda self, stream=None: (seen.append((self.name, stream)), plain(self, stream))[1])
    del calls[:]
    op.run(scratch, 0)
    assert calls == expected and seen == [(name, 0) for name in EXPECTED[("sol", "bf16")]]

    class Counted(ops.SolPoolKernel):
        def submit(self, stream=None):
            seen.append("counted")
            super().submit(stream)

    monkeypatch.undo()
    monkeypatch.setattr(ops, "SolPoolKernel", Counted)
    monkeypatch.setattr(_lib, "symbol", lambda name: lambda *arguments: 0)
    op = make("sol", "bf16")
    del seen[:]
    for _ in range(2):
        op.run(scratch, 7)
    assert seen == ["counted"] * 2


def test_bind_of_an_operator_class_is_used(calls):
    class Twice(ops.DenseBf16Attention):
        def bind(self, scratch_base):
            return 2 * super().bind(scratch_base)

    plain = make("dense", "bf16")
    op = Twice(*plain.inputs, total_heads=plain.total_heads, head_offset=plain.head_offset).to(*plain.outputs)
    scratch = arena(op.prepare()[1])
    expected = submitted(plain, scratch, 3, calls)
    op.run(scratch, 3)
    assert calls == 2 * expected


def test_a_failing_call_is_an_error(calls, monkeypatch):
    op = make("dense", "bf16")
    scratch = arena(op.prepare()[1])

    def failing(*arguments):
        return -1

    monkeypatch.setattr(_lib, "symbol", lambda name: failing)
    monkeypatch.setattr(_lib, "last_error", lambda: "why")
    with pytest.raises(RuntimeError, match="why"):
        op.run(scratch, ctypes.c_void_p(1).value)
