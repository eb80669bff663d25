"""Which dense products tk_gemm_f64 computes on digits (csrc/linalg.cu, csrc/digit_gemm.cu): those whose
every output keeps the componentwise bound of an FP64 chain.  The others give the FP64 kernel's bits, those
of tk_gemm_f64_noalloc, which never uses digits."""
import ctypes as C

import numpy as np
import pytest

from tk_gb300 import _abi
from tk_gb300.heff import context

pytestmark = pytest.mark.gpu


def _run(A, B, entry):
    import torch

    (M, K), N = A.shape, B.shape[1]
    dA, dB = torch.from_numpy(np.ascontiguousarray(A)).cuda(), torch.from_numpy(np.ascontiguousarray(B)).cuda()
    dC = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    a, b = _abi.tk_mat(dA.data_ptr(), M, K, K, 1, 0), _abi.tk_mat(dB.data_ptr(), K, N, N, 1, 0)
    c = _abi.tk_mat_mut(dC.data_ptr(), M, N, N, 1)
    torch.cuda.synchronize()
    _abi.check(getattr(_abi.load(), entry)(context(0), 1.0, C.byref(a), C.byref(b), 0.0, C.byref(c), None))
    torch.cuda.synchronize()
    return dC.cpu().numpy()


def _excess(A, B, got):
    """The largest error over the bound K 2^-52 |A| |B|, on 16 rows in extended precision."""
    rows = np.linspace(0, A.shape[0] - 1, 16).astype(int)
    want = np.stack([(A[r].astype(np.longdouble)[:, None] * B.astype(np.longdouble)).sum(0) for r in rows])
    bound = A.shape[1] * 2.0 ** -52 * (np.abs(A[rows]) @ np.abs(B))
    return float((np.abs(got[rows] - want) / bound).max())


def _weak_coupling(c):
    """64 x 64 diagonal blocks and couplings of c: no row is far from flat by its norm."""
    rng = np.random.default_rng(1)
    blocks = np.kron(np.eye(8), np.ones((64, 64)))
    return tuple(rng.uniform(-1.0, 1.0, (512, 512)) * np.where(blocks > 0, 1.0, c) for _ in range(2))


def _scaled(K):
    """X D and D^-1 Y with D over twelve decades."""
    rng = np.random.default_rng(2)
    d = np.logspace(0, -12, K)
    return rng.standard_normal((384, K)) * d, rng.standard_normal((K, 640)) / d[:, None]


def _spikes(K):
    """One element of a row just below a power of two, the rest 1e-9: they meet in few outputs."""
    rng = np.random.default_rng(3)
    A, B = 1e-9 * rng.standard_normal((512, K)), 1e-9 * rng.standard_normal((K, 640))
    A[np.arange(512), np.arange(512) % K] = 1.999
    B[(7 * np.arange(640) + 3) % K, np.arange(640)] = 1.999
    return A, B


def _halves(K):
    """A's large half of k is B's small one."""
    rng = np.random.default_rng(4)
    s = np.where(np.arange(K) < K // 2, 1.0, 1e-10)
    return rng.standard_normal((1024, K)) * s, rng.standard_normal((K, 1024)) * s[::-1][:, None]


UNEVEN = [("weak coupling 1e-10", _weak_coupling, 1e-10), ("weak coupling 1e-6", _weak_coupling, 1e-6), ("scaled", _scaled, 256),
          ("spikes", _spikes, 340), ("halves", _halves, 17), ("halves", _halves, 20), ("halves", _halves, 128)]


@pytest.mark.parametrize("what,make,arg", UNEVEN)
def test_uneven_operands_take_the_fp64_kernel(lib_built, what, make, arg):
    A, B = make(arg)
    got = _run(A, B, "tk_gemm_f64")
    assert _excess(A, B, got) <= 1.0
    assert np.array_equal(got, _run(A, B, "tk_gemm_f64_noalloc"))


@pytest.mark.parametrize("M,N,K", [(512, 512, 512), (300, 700, 1000), (600, 1000, 64), (1030, 1025, 19), (2050, 1090, 65), (2048, 2048, 17)])
@pytest.mark.parametrize("kind", ["normal", "uniform", "integers"])
def test_even_operands_stay_on_digits(lib_built, M, N, K, kind):
    """Also with rows and columns of zeros, whose products are exact on any grid."""
    rng = np.random.default_rng(M + N + K)
    draw = {"normal": rng.standard_normal, "uniform": rng.random,
            "integers": lambda s: rng.integers(-2 ** 25, 2 ** 25, s) * (rng.random(s) < 0.02)}[kind]
    A, B = np.asarray(draw((M, K)), dtype=float), np.asarray(draw((K, N)), dtype=float)
    A[5] = 0.0
    B[:, 7] = 0.0
    got = _run(A, B, "tk_gemm_f64")
    if kind == "integers":  # sparse, but exact
        assert np.array_equal(got, A @ B) and np.abs(got).max() < 2.0 ** 53
        return
    assert _excess(np.delete(A, 5, 0), np.delete(B, 7, 1), np.delete(np.delete(got, 5, 0), 7, 1)) <= 1.0
    assert (got[5] == 0.0).all() and (got[:, 7] == 0.0).all()
    assert not np.array_equal(got, _run(A, B, "tk_gemm_f64_noalloc"))
    assert np.array_equal(got, _run(A, B, "tk_gemm_f64"))  # the same path and bits every time
