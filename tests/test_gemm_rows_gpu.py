"""The tensor-core GEMM at every alignment of its rows: FP32 outputs whose rows are whole
16-byte chunks but not whole 32-byte ones, and operands staged by the threads in chunks of
16, 8, 4 and 2 bytes (row pitch and base offset), with partial chunks at the ends.

Bound: K products of bf16 values are exact in float32; K float32 additions in any order err
by at most K 2^-24 of the sum of magnitudes, and the tensor core may truncate instead of
rounding, so K 2^-23 (|A| |B|) elementwise.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t, skip=0):
    return ctypes.c_void_p(t.data_ptr() + skip * t.element_size())


@pytest.mark.parametrize("M,N,K", [(130, 60, 72), (64, 500, 500), (200, 20, 61), (128, 12, 130), (33, 132, 16)])
@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad,skip", [(0, 0), (4, 0), (2, 0), (1, 0), (0, 4), (0, 2), (0, 1), (4, 1)])
def test_rows_of_every_alignment(pkg, M, N, K, tA, tB, pad, skip):
    rng = np.random.default_rng(M + 3 * N + 5 * K + 2 * tA + tB)

    def operand(rows, cols):
        ld = cols + (-cols % 8) + pad
        v = torch.as_tensor(rng.normal(size=(rows, cols)).astype(np.float32)).to(torch.bfloat16)
        flat = torch.full((rows * ld + 8,), float("nan"), dtype=torch.bfloat16)
        torch.as_strided(flat, (rows, cols), (ld, 1), skip).copy_(v)
        return flat.cuda(), ld, v.double().numpy()

    A, lda, a = operand(*((K, M) if tA else (M, K)))
    B, ldb, b = operand(*((N, K) if tB else (K, N)))
    a, b = (a.T if tA else a), (b.T if tB else b)
    bias = torch.as_tensor(rng.normal(size=N).astype(np.float32)).cuda()
    lib = pkg._lib.lib()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ref = a @ b + bias.double().cpu().numpy()
    tol = K * 2.0 ** -23 * (np.abs(a) @ np.abs(b)) + 2.0 ** -22 * (np.abs(ref) + 4)
    for ldc in (N, N + 4, N + 1):
        C = torch.zeros((M, ldc), dtype=torch.float32, device="cuda")
        pkg._lib.check(lib.rgs_gemm_bf16(M, N, K, _p(A, skip), lda, tA, _p(B, skip), ldb, tB, 1.0, _p(bias), 0, None,
                                         None, _p(C), None, ldc, s))
        torch.cuda.synchronize()
        assert np.all(np.abs(C[:, :N].double().cpu().numpy() - ref) <= tol), ldc
        assert not bool(C[:, N:].any())
    flag = ctypes.c_int32(-1)
    pkg._lib.check(lib.rgs_tensor_core_status(ctypes.byref(flag)))
    assert flag.value == 0
