"""The router's tiles at their edges: masks bit for bit against the CPU oracle."""

import pytest
import torch

from oracle import sol_math as sm
from tests.gpu_util import randn_bf16
from tests.test_gpu_sol_route import gpu_pool, gpu_select, gpu_stats, structured_keys

pytestmark = pytest.mark.gpu


# heads 3: four query blocks per warp; heads 60 x 5 CTAs: eight.  Blocks 127-129: the edge of a tile of key blocks.
@pytest.mark.parametrize("T,h", [(127 * 64, 3), (128 * 64 - 5, 3), (129 * 64 - 63, 3), (131 * 64, 60), (156 * 64 - 1, 60)])
@pytest.mark.parametrize("topk", [0.0, 0.3])
def test_select_tile_edges(T, h, topk):
    q = randn_bf16(60 + T, T, h, 128)
    k = structured_keys(61 + T, T, h)
    pooled = gpu_pool(k, k, None, 64)
    stats = gpu_stats(pooled)
    assert torch.equal(stats.cpu(), sm.sol_stats(pooled.cpu()))
    mask = gpu_select(q, pooled[0].contiguous(), stats, 0.5, 2, topk=topk)
    if topk:
        want = sm.route_topk(q.cpu(), pooled[0].cpu(), topk, 2, 64)
    else:
        want = sm.sol_select(q.cpu(), pooled[0].cpu(), stats.cpu(), 0.5, 2, 64)
    assert torch.equal(mask.cpu(), want)


def test_stats_over_several_chunks_of_blocks():
    pooled = randn_bf16(70, 2, 3, 1025, 128)
    assert torch.equal(gpu_stats(pooled).cpu(), sm.sol_stats(pooled.cpu()))


@pytest.mark.parametrize("nb", [5, 255, 257, 513, 1025])  # each count of scores per lane, and one past its range
@pytest.mark.parametrize("fraction", [0.001, 0.25, 1.0])
def test_topk_ties_take_the_lowest_blocks(nb, fraction):
    """Scores of a few distinct values, zeros of both signs among them: the cut falls inside a group of equals."""
    T, h = nb * 64, 2
    q = torch.zeros(T, h, 128, dtype=torch.bfloat16, device="cuda")
    q[:, :, 0] = 1.0
    pooled = torch.zeros(h, nb, 128, dtype=torch.bfloat16, device="cuda")
    g = torch.Generator().manual_seed(nb)
    pooled[:, :, 0] = torch.tensor([-2.0, -0.0, 0.0, 1.0])[torch.randint(0, 4, (h, nb), generator=g)].bfloat16().cuda()
    mask = gpu_select(q, pooled, torch.zeros(h, 2, 128, device="cuda"), 1.0, 1, topk=fraction)
    keep = min(nb - 1, max(1, -int(-fraction * nb // 1)))
    value = (pooled[:, :, 0].float() + 0.0).cpu()
    for head in range(h):
        order = sorted(range(1, nb), key=lambda b: (-float(value[head, b]), b))[:keep]
        want = torch.zeros(nb, dtype=torch.uint8)
        want[[0, *order]] = 1
        assert torch.equal(mask[:, head].cpu(), want.expand(nb, nb))


def test_select_of_tensors_off_the_16_byte_boundary():
    T, h = 1000, 2

    def shifted(x):
        flat = torch.empty(x.numel() + 1, dtype=x.dtype, device="cuda")[1:]
        return flat.copy_(x.flatten()).view(x.shape)

    q, k = randn_bf16(80, T, h, 128), structured_keys(81, T, h)
    pooled = gpu_pool(k, k, None, 64)
    stats = gpu_stats(shifted(pooled))
    assert torch.equal(stats.cpu(), sm.sol_stats(pooled.cpu()))
    mask = gpu_select(shifted(q), shifted(pooled[0]), stats, 1.0, 1)
    assert torch.equal(mask.cpu(), sm.sol_select(q.cpu(), pooled[0].cpu(), stats.cpu(), 1.0, 1, 64))
