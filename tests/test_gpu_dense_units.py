"""The dense attention kernels by units: 128- and 256-row units, keys of the last units divided into fp32 shares.

Every plan computes the same attention; what differs is the grid the probabilities are rounded on, because a share
tracks the running maximum of its own keys.  A normalised weight is off by at most half a step of that rounding in each
of the two results (bf16 2^-9, e4m3 2^-4, the ue4m3 block scale of nvfp4 2^-4, relative; the row sums are unrounded).
The values are independent N(0, 1), so the errors of a row's weights add by their squares, as the row itself does: over
the rows of a query tile the results differ by at most sqrt(2) * step of their norm, and 2^-8 for the output in bf16.
(A lost share of five changes a tile by 0.5 of its norm, heads or rows in the wrong place by 1.4.)
"""

import pytest
import torch

from nano_omni_b200 import _lib, ops
from nano_omni_b200.kernels.dense_bf16 import UnitPlan, plan_units
from tests.gpu_util import desc, randn_bf16

pytestmark = pytest.mark.gpu

STEP = {"bf16": 2.0**-9, "int8_fp8": 2.0**-4, "nvfp4": 2.0**-4}


def attend(monkeypatch, precision, plan, q, k, v, T, h):
    monkeypatch.setattr(ops, "plan_units", lambda *a, **kw: plan)
    out = torch.full((T, h, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    if precision == "int8_fp8":
        op = ops.DenseInt8Fp8Attention(desc(q), desc(k), desc(v)).to(desc(out.view(T, h * 128)))
    else:
        op = ops.ATTENTION_OPS[("dense", precision)](desc(q), desc(k), desc(v), total_heads=h).to(desc(out))
    scratch = torch.full((op.prepare()[1] + 256,), 0xA5, dtype=torch.uint8, device="cuda")
    op.run(scratch[(-scratch.data_ptr()) % 256 :])
    assert _lib.read_status() == 0
    return out.float()


@pytest.mark.parametrize("precision", ["bf16", "int8_fp8", "nvfp4"])
@pytest.mark.parametrize(
    "T,plan",
    [
        (1, UnitPlan(128, 1, 0)),
        (129, UnitPlan(128, 1, 0)),  # last unit one row
        (257, UnitPlan(256, 2, 1)),  # three key tiles over two shares, divided unit of one row
        (640, UnitPlan(256, 5, 4)),  # one key tile per share, units of two heads divided
        (1000, UnitPlan(128, 3, 0)),  # every unit divided
        (1000, UnitPlan(256, 2, 12)),  # tail = every unit, named
        (2100, UnitPlan(128, 4, 7)),
    ],
)
def test_unit_plans_agree_with_whole_units(monkeypatch, precision, T, plan):
    h = 3
    q, k, v = (randn_bf16(4000 + T + i, T, h * 128) for i in range(3))
    whole = attend(monkeypatch, precision, UnitPlan(256, 1, 0), q, k, v, T, h)
    got = attend(monkeypatch, precision, plan, q, k, v, T, h)
    assert torch.isfinite(got).all()
    for tile_got, tile_whole in zip(got.split(128), whole.split(128)):
        off = (tile_got - tile_whole).norm(dim=(0, 2)) / tile_whole.norm(dim=(0, 2))  # per head
        assert off.max().item() <= 2**0.5 * STEP[precision] + 2.0**-8


@pytest.mark.parametrize("precision", ["bf16", "int8_fp8", "nvfp4"])
@pytest.mark.parametrize(
    "T,plan",
    [
        (257, UnitPlan(256, 2, 1)),
        (640, UnitPlan(256, 5, 4)),
        (1000, UnitPlan(128, 3, 0)),
        (2100, UnitPlan(128, 4, 7)),
        (2100, UnitPlan(256, 16, 5)),
    ],
)
def test_every_share_counts_by_its_keys(monkeypatch, precision, T, plan):
    """Equal weights, and values that name their key tile (the channel) and head (the height): a channel of the output is
    its tile's part of the keys.  Values survive the quantisers exactly but for nvfp4's block scale (2^-4)."""
    h = 3
    q = torch.zeros(T, h * 128, dtype=torch.bfloat16, device="cuda")
    k = randn_bf16(4700, T, h * 128)
    tile = torch.arange(T, device="cuda") // 128
    named = torch.nn.functional.one_hot(tile, 128).float()
    height = torch.arange(1, h + 1, device="cuda", dtype=torch.float32)[:, None]
    v = (named[:, None] * height).bfloat16().view(T, h * 128)
    got = attend(monkeypatch, precision, plan, q, k, v, T, h)
    want = (named.mean(0) * height).expand(T, h, 128)
    assert ((got - want).abs() <= (2.0**-8 + (2.0**-4 if precision == "nvfp4" else 0.0)) * want + 1e-6).all()


def test_plans_fill_the_last_wave():
    assert plan_units(32768, 24) == UnitPlan(256, 1, 0)  # 20.8 waves
    assert plan_units(9461, 14) == UnitPlan(256, 2, 74)  # 3.5 waves: the last 74 units on all SMs
    assert plan_units(1021, 14).query_rows == 128  # 56 units of 256 rows leave most SMs idle
    assert plan_units(512, 37, 4096).kv_splits == 2


def test_int8_key_scales_past_the_kept_ones():
    """More than 8192 64-key scales (524288 keys) are read from global memory: a softmax over keys of which only those
    past that point carry values.  Expected: their share of the softmax mass, in fp32 from the same integers."""
    from tests.test_gpu_attention_int8 import attend as run_int8

    kept, extra, h = 524288, 640, 1
    Tk = kept + extra
    g = torch.Generator(device="cuda").manual_seed(5)
    q8 = torch.randint(-127, 128, (h, 32, 128), generator=g, device="cuda", dtype=torch.int8)
    k8 = torch.randint(-127, 128, (h, Tk, 128), generator=g, device="cuda", dtype=torch.int8)
    ks = torch.full((h, Tk // 64), 2.0**-12, device="cuda")
    ks[:, kept // 64 :] = 2.0**-6 * (1 + torch.arange(extra // 64, device="cuda") / 16)
    qs = torch.full((h, 1), 2.0**-4, device="cuda")
    v8 = torch.zeros(h, 128, Tk, device="cuda")
    v8[:, :, kept:] = 1.0
    vs = torch.ones(h, 128, device="cuda")
    got = run_int8((q8, k8, v8.to(torch.float8_e4m3fn), qs, ks, vs), 32, Tk, h).float()
    logits = (q8[0].float() @ k8[0].float().T) * qs[0, 0] * ks[0].repeat_interleave(64) / 128**0.5
    want = torch.softmax(logits.double(), dim=1)[:, kept:].sum(1)
    # probabilities rounded to e4m3 in the numerator only: 2^-4 relative
    assert ((got.reshape(32, 128) - want[:, None]).abs() <= (2.0**-4 + 2.0**-8) * want[:, None] + 1e-4).all()


@pytest.mark.parametrize("plan", [UnitPlan(256, 1, 0), UnitPlan(256, 2, 0), UnitPlan(256, 2, 1), UnitPlan(128, 4, 0)])
@pytest.mark.parametrize("first", [False, True])
def test_keys_of_no_weight_fill_a_share(monkeypatch, plan, first):
    """Keys whose scores are minus infinity (here: overflow) weigh nothing, also where they are all that a share has."""
    T, h = 512, 2
    q, k, v = (randn_bf16(4900 + i, T, h * 128).float() for i in range(3))
    none = slice(0, 256) if first else slice(256, 512)
    live = slice(256, 512) if first else slice(0, 256)
    big = 2.0**64
    k = k / big
    k[none] = -big / 4
    q, k = (q.abs() * big).bfloat16(), k.bfloat16()
    got = attend(monkeypatch, "bf16", plan, q, k, v.bfloat16(), T, h)
    qs, ks, vs = (x.double().view(T, h, 128) for x in (q, k, v.bfloat16()))
    weights = torch.softmax(torch.einsum("qhd,khd->hqk", qs, ks[live]) / 128**0.5, -1)
    want = torch.einsum("hqk,khd->qhd", weights, vs[live])
    # probabilities and output rounded to bf16
    assert ((got - want).abs() <= 2 * 2.0**-9 * vs.abs().max() + 2.0**-8 * want.abs()).all()
