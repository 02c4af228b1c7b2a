"""The paired-CTA GEMM at every tile width its rule chooses, bit for bit against the oracle: ragged row and column edges,
a follower CTA without rows, residual tiles through the staging ring over several tiles per CTA, residual in place."""

import pytest
import torch

from oracle import reference_math as rm
from tests.gpu_util import desc, run
from tests.test_gpu_matmul_int8 import case, gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "M,N,K",
    # on 148 SMs: tiles of 64, 96, 128, 160, 192, 224 and 256 columns
    [(100, 1064, 128), (385, 2552, 400), (1000, 2072, 128), (300, 5368, 128), (1300, 2080, 256), (515, 7160, 144), (2000, 2080, 512),
     (5000, 2568, 64)],
)  # fmt: skip
@pytest.mark.parametrize("residual", [False, True])
def test_tile_widths(M, N, K, residual):
    x, w, ws, xs, b, r, m = case(M, N, K, 9500 + M, True, residual, False)
    got = gemm(x, w, ws, xs, b, r, m, False)
    want = rm.matmul_int8(x, w, ws, xs, b, r, m, False)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_output_over_its_own_residual():
    from nano_omni_b200.kernels.matmul import MatmulInt8Arguments, MatmulInt8Kernel

    x, w, ws, xs, b, r, _ = case(3000, 2560, 64, 9600, False, True, False)
    out = r.cuda()
    run(MatmulInt8Kernel(MatmulInt8Arguments(
        desc(x.cuda()), desc(w.cuda()), None, desc(out), None, desc(out), desc(ws.cuda()), desc(xs.cuda()), False)))  # fmt: skip
    want = rm.matmul_int8(x, w, ws, xs, None, r, None, False)
    assert torch.equal(out.cpu().view(torch.int16), want.view(torch.int16))
