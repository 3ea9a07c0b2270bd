"""The tensor-core GEMM where K is long (split over a cluster) and where operands are
MN-major (loaded by TMA without a transpose), and the bias-gradient column sums.

Bound: K products of bf16 values are exact in float32; K float32 additions in any order
err by at most K 2^-24 of the sum of magnitudes, and the tensor core may truncate instead
of rounding, so K 2^-23 (|A| |B|) elementwise.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("M,N,K", [(128, 128, 1024), (512, 512, 4096), (56, 512, 4096), (512, 56, 1030),
                                   (40, 24, 1023), (264, 136, 1088), (72, 8, 2049), (130, 70, 1500), (128, 128, 64)])
@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_long_k_and_mn_major(pkg, M, N, K, tA, tB):
    rng = np.random.default_rng(M * 7 + N * 3 + K + 2 * tA + tB)
    bf = lambda a: torch.as_tensor(a.astype(np.float32)).cuda().to(torch.bfloat16)  # noqa: E731
    A, B = bf(rng.normal(size=(K, M) if tA else (M, K))), bf(rng.normal(size=(N, K) if tB else (K, N)))
    bias = torch.as_tensor(rng.normal(size=N).astype(np.float32)).cuda()
    mask = torch.as_tensor((rng.random((M, N)) < 0.7).astype(np.uint8)).cuda()
    gate = bf(rng.normal(size=(M, N)))
    lib = pkg._lib.lib()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    a, b = A.double().cpu().numpy(), B.double().cpu().numpy()
    a, b = (a.T if tA else a), (b.T if tB else b)
    keep = mask.cpu().numpy() * (gate.double().cpu().numpy() > 0)
    ref = (0.5 * (a @ b) + bias.double().cpu().numpy()) * keep
    tol = K * 2.0 ** -23 * (np.abs(a) @ np.abs(b)) + 2.0 ** -22 * (np.abs(ref) + 4)
    for tma in (1, 0):
        pkg._lib.check(lib.rgs_gemm_set_tma(tma))
        try:
            C = torch.empty((M, N), dtype=torch.float32, device="cuda")
            Cb = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
            for out, outb in ((C, None), (None, Cb)):
                pkg._lib.check(lib.rgs_gemm_bf16(M, N, K, _p(A), A.shape[1], tA, _p(B), B.shape[1], tB, 0.5, _p(bias),
                                                 0, _p(mask), _p(gate), _p(out), _p(outb), N, s))
            torch.cuda.synchronize()
        finally:
            pkg._lib.check(lib.rgs_gemm_set_tma(1))
        assert np.all(np.abs(C.cpu().numpy() - ref) <= tol), tma
        assert torch.equal(C.to(torch.bfloat16), Cb), tma
    flag = ctypes.c_int32(-1)
    pkg._lib.check(lib.rgs_tensor_core_status(ctypes.byref(flag)))
    assert flag.value == 0


@pytest.mark.parametrize("n,hidden,rows", [(10, 64, 1), (56, 512, 4096), (51, 500, 1100), (17, 72, 33)])
def test_bias_gradients(pkg, n, hidden, rows):
    """Bias gradients are the column sums of the bf16 deltas the backward pass leaves in its
    buffers: rows 2^-24 of the sum of magnitudes."""
    net = pkg.MadeProposal(n, hidden=hidden, seed=1)
    rng = np.random.default_rng(n)
    x = torch.as_tensor(rng.integers(0, 2, (rows, n)).astype(np.float32)).cuda()
    _, g = net.gradients(x, torch.as_tensor(rng.random((rows, n)).astype(np.float32)).cuda())
    buf = net._buffers(rows)
    for got, delta in ((g[1], buf["dh1"]), (g[3], buf["dh2"]), (g[5], buf["dz"])):
        d = delta.double()
        tol = rows * 2.0 ** -24 * d.abs().sum(0) + 1e-30
        assert bool(((got.double() - d.sum(0)).abs() <= tol).all())
