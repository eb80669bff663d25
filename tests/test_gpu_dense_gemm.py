"""The table-free FP64 GEMM kernel (tk_gemm_f64_noalloc, and tk_gemm_f64 where the
digits do not pay): tile edges, the cluster's shares of K, strides, no K at all."""
import ctypes as C

import pytest

from tk_gb300 import _abi
from tk_gb300.heff import context

pytestmark = pytest.mark.gpu

# M, N, K: single elements, tile edges, K around the 64 that a share needs at least,
# K that leaves the last CTAs of a cluster with little or nothing, outputs past one wave
SHAPES = [(1, 1, 1), (1, 1, 1025), (16, 16, 127), (16, 16, 128), (17, 15, 129), (33, 16, 513), (15, 49, 1041), (100, 100, 2000),
          (16, 2049, 65), (640, 33, 515), (200, 201, 999), (5, 7, 0)]


@pytest.mark.parametrize("entry", ["tk_gemm_f64_noalloc", "tk_gemm_f64"])
@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_dense_gemm_against_fp64(lib_built, entry, M, N, K, ta, tb):
    import torch

    g = torch.Generator().manual_seed(M * 7 + N * 3 + K)
    pad = 3  # rows longer than their matrix, and an output with gaps that must stay as they are
    A = torch.randn(K if ta else M, (M if ta else K) + pad, dtype=torch.float64, generator=g)
    B = torch.randn(N if tb else K, (K if tb else N) + pad, dtype=torch.float64, generator=g)
    Cm = torch.randn(M, N + pad, dtype=torch.float64, generator=g)
    dA, dB, dC = A.cuda(), B.cuda(), Cm.cuda()
    one = torch.zeros(1, dtype=torch.float64, device="cuda")  # a valid address where a matrix is empty
    a = _abi.tk_mat((dA if dA.numel() else one).data_ptr(), M, K, 1 if ta else A.shape[1], A.shape[1] if ta else 1, 0)
    b = _abi.tk_mat((dB if dB.numel() else one).data_ptr(), K, N, 1 if tb else B.shape[1], B.shape[1] if tb else 1, 0)
    c = _abi.tk_mat_mut(dC.data_ptr(), M, N, N + pad, 1)
    alpha, beta = -0.5, 2.0
    torch.cuda.synchronize()
    _abi.check(getattr(_abi.load(), entry)(context(0), alpha, C.byref(a), C.byref(b), beta, C.byref(c), None))
    torch.cuda.synchronize()
    got = dC.cpu()
    a64 = (A[:, :M].T if ta else A[:, :K]).contiguous()
    b64 = (B[:, :K].T if tb else B[:, :N]).contiguous()
    want = alpha * (a64 @ b64) + beta * Cm[:, :N]
    # both sides: K rounded sums of rounded products, then three more roundings
    bound = 2 * (K + 3) * 2.0**-53 * (0.5 * (a64.abs() @ b64.abs()) + 2.0 * Cm[:, :N].abs())
    assert bool(((got[:, :N] - want).abs() <= bound).all())
    assert torch.equal(got[:, N:], Cm[:, N:])
