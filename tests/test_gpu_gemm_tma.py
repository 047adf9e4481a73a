"""The TMA form of the tensor-core product at the edges of its shapes: rows, columns and k
around its tiles, every N tile, K slices (one of them empty), more work items than SMs,
leading dimensions past the row and an output whose rows are not 16-byte aligned. Each
product is exact in FP32 (integers small enough), so the result is exact; the form whose
operands only plain loads can read gives the same bits on operands that are not."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gemm(A, B, C):
    import sitk_b200 as sb
    import torch
    L = sb._lib.load()
    vp, ci = ctypes.c_void_p, ctypes.c_int
    L.mi_gemm_bf16_tn.argtypes = [vp, ci, ci, ci, vp, ci, vp, ci, vp, ci]
    L.mi_gemm_bf16_tn.restype = ci
    ctx = sb.default_context()
    torch.cuda.synchronize()
    sb._lib.check(L.mi_gemm_bf16_tn(ctx.handle, A.shape[0], B.shape[0], A.shape[1], A.data_ptr(), A.stride(0),
                                    B.data_ptr(), B.stride(0), C.data_ptr(), C.stride(0)), ctx.handle)
    return C


@pytest.mark.parametrize("M,N,K,pad,cpad", [
    (1, 1, 8, 0, 0), (127, 15, 64, 0, 0), (128, 16, 72, 8, 0), (129, 17, 56, 0, 1), (200, 33, 200, 0, 3),
    (64, 65, 128, 8, 0), (256, 128, 640, 0, 0), (130, 129, 64, 0, 0), (300, 257, 8, 0, 2), (384, 511, 136, 16, 0),
    (16, 56, 20000, 0, 0), (128, 1728, 520, 0, 0), (40, 24, 1000, 0, 0), (2560, 2304, 128, 0, 0), (20000, 16, 56, 0, 0)])
def test_products_are_exact(M, N, K, pad, cpad):
    import torch
    g = torch.Generator().manual_seed(M + N + K)
    # |sum| ≤ 9·20000 < 2^24: every partial sum is an integer FP32 holds
    A = torch.randint(-3, 4, (M, K + pad), generator=g).to(torch.bfloat16).cuda()[:, :K]
    B = torch.randint(-3, 4, (N, K + pad), generator=g).to(torch.bfloat16).cuda()[:, :K]
    C = torch.full((M, N + cpad), -7.0, device="cuda")
    _gemm(A, B, C[:, :N])
    assert torch.equal(C[:, :N].double(), A.double() @ B.double().T)
    assert torch.all(C[:, N:] == -7.0)


@pytest.mark.parametrize("M,N,K", [(129, 300, 264), (70, 40, 2000), (512, 128, 1728)])
def test_both_forms_give_the_same_bits(M, N, K):
    import torch
    g = torch.Generator().manual_seed(5)
    A = torch.randn((M, K), generator=g).to(torch.bfloat16).cuda()
    B = torch.randn((N, K), generator=g).to(torch.bfloat16).cuda()
    A1 = torch.zeros((M, K + 1), dtype=torch.bfloat16, device="cuda")  # an odd row pitch: plain loads
    A1[:, :K] = A
    C, C1 = torch.empty((M, N), device="cuda"), torch.empty((M, N), device="cuda")
    assert np.array_equal(_gemm(A, B, C).cpu().numpy(), _gemm(A1[:, :K], B, C1).cpu().numpy())


@pytest.mark.parametrize("M,N,pitch,first", [
    (33, 20, 24, 0), (161, 36, 48, 4), (31, 44, 64, 8), (129, 148, 152, 4), (97, 260, 264, 0),  # blocks stored by TMA
    (33, 20, 25, 0), (161, 36, 48, 1), (31, 43, 48, 0)])                                        # by lanes
def test_output_blocks_end_where_the_product_does(M, N, pitch, first):
    import torch
    g = torch.Generator().manual_seed(M * N)
    A = torch.randint(-3, 4, (M, 72), generator=g).to(torch.bfloat16).cuda()
    B = torch.randint(-3, 4, (N, 72), generator=g).to(torch.bfloat16).cuda()
    C = torch.full((M + 2, pitch), -7.0, device="cuda")
    want = C.clone()
    want[1:M + 1, first:first + N] = (A.double() @ B.double().T).float()  # integers below 2^24: exact
    _gemm(A, B, C[1:M + 1, first:first + N])
    assert torch.equal(C, want)


@pytest.mark.parametrize("M,N,K,pad", [
    (1300, 4100, 1032, 0),   # the last pair of row blocks: one full, one of 20 rows; a last column tile of 4
    (2432, 3999, 1024, 8),   # a last pair without its second block; outputs by lanes
    (4096, 2304, 2056, 0)])
def test_two_row_blocks_a_tile(M, N, K, pad):
    import torch
    g = torch.Generator().manual_seed(M + N)
    A = torch.randint(-3, 4, (M, K + pad), generator=g).to(torch.bfloat16).cuda()[:, :K]
    B = torch.randint(-3, 4, (N, K + pad), generator=g).to(torch.bfloat16).cuda()[:, :K]
    C = torch.full((M, N), -7.0, device="cuda")
    _gemm(A, B, C)
    assert torch.equal(C.double(), A.double() @ B.double().T)  # integers below 2^24: exact
