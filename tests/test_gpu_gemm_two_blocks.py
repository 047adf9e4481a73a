"""Products that take tiles of 256 x 256 (two blocks of 128 rows on one B tile), at the edges of
the rows and columns: a last tile whose second block is partial, one whose second block lies
past the operand, outputs stored by TMA and by lanes. The kernel that ran is looked up by
its name, so that a rule that turns elsewhere does not leave these untested unseen. Each
product is exact in FP32 (integers below 2^24)."""
import re

import pytest

from test_gpu_gemm_tma import _gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,pad", [
    (2248, 4000, 4096, 0),   # 2248 = 8·256 + 200: the last tile's second block has 72 rows
    (2248, 3999, 4096, 8),   # and outputs by lanes, the last column tile of 159
    (2088, 4000, 4096, 0),   # 2088 = 8·256 + 40: the last tile's second block is past the end
    (2088, 3871, 4104, 0),   # the same by lanes, a last k tile of 8
    (2304, 4096, 4096, 0)])  # whole tiles
def test_edges_of_two_block_tiles(M, N, K, pad):
    import torch
    from torch.profiler import ProfilerActivity, profile
    g = torch.Generator().manual_seed(M + N)
    A = torch.randint(-3, 4, (M, K + pad), generator=g).to(torch.bfloat16).cuda()[:, :K]
    B = torch.randint(-3, 4, (N, K + pad), generator=g).to(torch.bfloat16).cuda()[:, :K]
    C = torch.full((M + 1, N), -7.0, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        _gemm(A, B, C[:M])
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if "k_gemm" in e.name]
    # (none where another profiler holds the device)
    assert all(re.search(r"k_gemm_tma<256, false, false, 2>", n) for n in names), names
    assert torch.equal(C[:M].double(), A.double() @ B.double().T)
    assert torch.all(C[M] == -7.0)
