"""Lists of 64-key blocks in the nvfp4 sol exact stage: lists of neighbouring query blocks that agree, differ, end at
different places or hold block 0 alone (which always attends), odd counts, a partial last block, CTAs with one and with two
query tiles (sm_100a)."""

import pytest
import torch

from oracle import reference_math as rm
from oracle import sol_math as sm
from tests.gpu_util import randn_bf16
from tests.test_gpu_attention_nvfp4 import prepare
from tests.test_gpu_sol_exact import check_state_and_numerator, numerator_error, nvfp4_exact

pytestmark = pytest.mark.gpu


def pattern(name, nb, h):
    g = torch.Generator().manual_seed(nb * h)
    chosen = torch.rand(nb, h, nb, generator=g) < 0.4
    qb, kb = torch.arange(nb)[:, None, None], torch.arange(nb)[None, None, :]
    if name == "same":  # both query blocks of a tile have one list
        chosen = chosen[qb.flatten() // 2 * 2]
    elif name == "disjoint":
        chosen = ((qb ^ kb) & 1 == 0).expand(nb, h, nb)
    elif name == "one side":  # the second query block of every tile attends to block 0 alone, the third tile to nothing else
        chosen = chosen & (qb % 2 == 0) & (qb // 2 != 2)
    elif name == "counts":  # 1 to 5 blocks, another count for each query block
        chosen = ((kb + qb) % nb < 1 + qb % 5).expand(nb, h, nb)
    elif name == "last":  # the partial last block, alone or beside one other
        chosen = ((kb == nb - 1) | ((kb == qb) & (qb % 3 == 0))).expand(nb, h, nb)
    elif name == "all":
        chosen = torch.ones(nb, h, nb, dtype=torch.bool)
    return chosen.to(torch.uint8).contiguous()


# (tokens, heads): 8, 7 and 3 query tiles of 128 rows, so that the last CTA of a head has two, one and one; 16, 14 and 5 blocks
@pytest.mark.parametrize("T,h", [(1000, 2), (850, 1), (300, 3)])
@pytest.mark.parametrize("name", ["random", "same", "disjoint", "one side", "counts", "last", "all"])
def test_nvfp4(name, T, h):
    flat = [randn_bf16(50 + i, T, h, 128).reshape(T, h * 128).contiguous() for i in range(3)]
    ops = [prepare(x, h, i == 2) for i, x in enumerate(flat)]
    selected = pattern(name, -(-T // 64), h)
    exact, state = nvfp4_exact(ops, selected.cuda(), T, h)
    dq, dk = (rm.nvfp4_dequantize(a.cpu(), s.cpu())[:, :T] for a, s in ops[:2])
    dv = rm.nvfp4_dequantize(ops[2][0].cpu(), ops[2][1].cpu()).transpose(1, 2)[:, :T]
    truth, want_state = sm.sol_exact_generic(dq, dk, dv, selected, always_first_block=True)
    rounded, _ = sm.sol_exact_generic(
        dq, dk, dv, selected, always_first_block=True, round_probability=sm.round_nvfp4_groups, probability_scale=2688.0
    )
    # against unrounded probabilities: no further from them than 1.5x what the reference's rounding is
    theirs = numerator_error(rounded, truth, want_state, 0.0).max()
    check_state_and_numerator(exact, state, truth, want_state, rtol=0.03, atol=float(1.5 * theirs + 1e-3))


@pytest.mark.parametrize("T,width", [(128, 1), (128, 4), (240, 4), (500, 1), (1000, 4)])
@pytest.mark.parametrize("name", ["all", "random", "counts"])
def test_nvfp4_probabilities_are_rounded_block_by_block(name, T, width):
    """The maximum that P is rounded against is raised with every listed block, as the oracle does it.  What is left between
    the two is the store to bf16 (.0017 of the norm: errors spread evenly up to 2^-9 of the value's power of two) and the few
    codes that fp32 rounding moves across a boundary of the grid.  One raise per two blocks instead, which makes the
    error against unrounded probabilities larger, puts .004 to .017 between them on lists of two to sixteen blocks."""
    h = 2
    flat = [randn_bf16(80 + i, T, h, 128).reshape(T, h * 128).contiguous() for i in range(3)]
    flat[0] = flat[0] * width  # wider scores: fewer keys hold a row's probability mass
    ops = [prepare(x, h, i == 2) for i, x in enumerate(flat)]
    selected = pattern(name, -(-T // 64), h)
    exact, state = nvfp4_exact(ops, selected.cuda(), T, h)
    dq, dk = (rm.nvfp4_dequantize(a.cpu(), s.cpu())[:, :T] for a, s in ops[:2])
    dv = rm.nvfp4_dequantize(ops[2][0].cpu(), ops[2][1].cpu()).transpose(1, 2)[:, :T]
    rounded, _ = sm.sol_exact_generic(
        dq, dk, dv, selected, always_first_block=True, round_probability=sm.round_nvfp4_groups, probability_scale=2688.0
    )
    distance = float((exact.cpu().double() - rounded.double()).norm() / rounded.double().norm())
    assert distance < 0.0025, distance
