"""The finalize and the fused sol kernel on pairs of 64-key blocks, at their edges.

Both against the fp32 oracle from the same inputs: probabilities and outputs are rounded to bf16, 2^-9 relative each, of
terms that partly cancel; the tolerances are those of the tests of the whole stages."""

import pytest
import torch

from oracle import sol_math as sm
from tests.gpu_util import randn_bf16
from tests.test_gpu_sol_attention import sol_attend
from tests.test_gpu_sol_exact import finalize, routed_case
from tests.test_gpu_sol_route import gpu_stats

pytestmark = pytest.mark.gpu


# one row, tiles full and of one row, several tiles of pseudo-keys
@pytest.mark.parametrize("T", [1, 128, 129, 255, 256, 257, 385, 16449])
def test_finalize_tiles(T):
    h = 2
    q, _, _, _, pooled3, selected = routed_case(T, h, 900 + T)
    exact = randn_bf16(901 + T, T, h, 128)
    g = torch.Generator().manual_seed(T)
    state = torch.stack((torch.randn(T, h, generator=g) * 8, 1 + 30 * torch.rand(T, h, generator=g)), -1).cuda()
    want = sm.sol_finalize(q.cpu(), pooled3.cpu(), selected.cpu(), exact.cpu(), state.cpu())
    for in_place in (False, True):
        out = finalize(q, pooled3, selected, exact, state, in_place=in_place)
        torch.testing.assert_close(out.cpu().float(), want, rtol=0.02, atol=0.01)


@pytest.mark.parametrize("T", [1, 129, 191, 193, 449, 705])  # odd lists, a last block of one key
def test_fused_pairs_of_blocks(T):
    h = 2
    q, k, v, _, pooled3, _ = routed_case(T, h, 950 + T)
    pooled = torch.stack((pooled3[0], pooled3[2])).contiguous()
    stats = gpu_stats(pooled)
    out, mask = sol_attend(q, k, v, pooled, stats, 1.0, 1)
    want = sm.sol_attention(q.cpu(), k.cpu(), v.cpu(), pooled.cpu(), mask.cpu(), 64)
    torch.testing.assert_close(out.cpu().float(), want, rtol=0.02, atol=0.01)
