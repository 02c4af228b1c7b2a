"""Steps of two 64-key blocks in the nvfp4 sol exact stage: lists of neighbouring query blocks that agree, differ, end
at different places or are empty, odd counts, a partial last block, CTAs with one and with two query tiles (sm_100a)."""

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
    elif name == "one side":  # the second query block of every tile attends to nothing, the third tile to nothing at all
        chosen = chosen & (qb % 2 == 0) & (qb // 2 != 2)
    elif name == "counts":  # 1 to 5 blocks, another count for each query block
        chosen = ((kb + qb) % nb < 1 + qb % 5).expand(nb, h, nb)
    elif name == "last":  # the partial last block, alone or beside one other
        chosen = ((kb == nb - 1) | ((kb == qb) & (qb % 3 == 0))).expand(nb, h, nb)
    elif name == "all":
        chosen = torch.ones(nb, h, nb, dtype=torch.bool)
    return chosen.to(torch.uint8).contiguous()


# (tokens, heads): an odd number of query tiles, so that the last CTA of a head has one; odd and even block counts
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
    # the maximum is raised per step of two blocks, the reference's per block: two legitimate grids of e2m1
    theirs = numerator_error(rounded, truth, want_state, 0.0).max()
    check_state_and_numerator(exact, state, truth, want_state, rtol=0.03, atol=float(1.5 * theirs + 1e-3))
