"""FP64 products on the fp16 tensor cores (csrc/digit_gemm.cu): dense products at the edges of
tiles, K chunks and panels against exact integer sums and extended precision, and the operands
that go to the FP64 kernel instead."""
import ctypes as C

import numpy as np
import pytest

from tk_gb300 import _abi
from tk_gb300.heff import context

pytestmark = pytest.mark.gpu


def _gemm(A, B, ta=False, tb=False, alpha=1.0, beta=0.0, C0=None, pad=0):
    """alpha op(A) op(B) + beta C0 through tk_gemm_f64; operands given as op(A), op(B); `pad` widens every row."""
    import torch

    (M, K), N = A.shape, B.shape[1]

    def put(X, t):
        X = X.T if t else X
        buf = np.zeros((X.shape[0], X.shape[1] + pad))
        buf[:, :X.shape[1]] = X
        return torch.from_numpy(buf).cuda(), buf.shape[1]

    dA, la = put(A, ta)
    dB, lb = put(B, tb)
    dC = torch.full((M, N + pad), float("nan"), dtype=torch.float64, device="cuda")
    if C0 is not None:
        dC[:, :N] = torch.from_numpy(C0).cuda()
    a = _abi.tk_mat(dA.data_ptr(), M, K, 1 if ta else la, la if ta else 1, 0)
    b = _abi.tk_mat(dB.data_ptr(), K, N, 1 if tb else lb, lb if tb else 1, 0)
    c = _abi.tk_mat_mut(dC.data_ptr(), M, N, N + pad, 1)
    _abi.check(_abi.load().tk_gemm_f64(context(0), alpha, C.byref(a), C.byref(b), beta, C.byref(c), None))
    if pad:
        assert bool(torch.isnan(dC[:, N:]).all())
    return dC[:, :N].cpu().numpy()


# 1 and 63..65 past tiles of 128 x 64 and chunks of 64; one SM's share of tiles and several
SHAPES = [(512, 512, 512), (513, 321, 385), (383, 577, 449), (129, 1025, 1023), (2050, 1090, 65),
          (1999, 2048, 17), (1280, 1216, 48), (257, 257, 4160)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_is_correctly_rounded_on_integers(lib_built, M, N, K):
    """Rows of 26-bit integers on scales of their own: sums exact in int64; the result's error is the
    final rounding and half a unit of 2^-58 of row maximum times column maximum per 64 k."""
    rng = np.random.default_rng(M + 7 * N + K)
    a, b = rng.integers(-2 ** 25, 2 ** 25, (M, K)), rng.integers(-2 ** 25, 2 ** 25, (K, N))
    ea, eb = rng.integers(-40, 40, M), rng.integers(-40, 40, N)
    got = _gemm(np.ldexp(a.astype(float), ea[:, None]), np.ldexp(b.astype(float), eb[None, :]), ta=K % 2 == 1, tb=N % 2 == 1,
                pad=3 if M % 2 else 0)
    exact = np.zeros((M, N), dtype=np.int64)
    for k0 in range(0, K, 256):
        exact += a[:, k0:k0 + 256] @ b[k0:k0 + 256]
    back = np.ldexp(np.ldexp(got, -ea[:, None]), -eb[None, :])  # exact
    hi = back.astype(np.int64)
    err = np.abs((hi - exact).astype(float) + (back - hi))
    bound = np.abs(exact) * 2.0 ** -53 + np.ceil(K / 64) * 2.0 ** (50 - 57)
    assert (err <= bound).all()


def test_gemm_too_small_for_digits_stays_an_fp64_chain(lib_built):
    """Few tiles over a long K: the FP64 kernel runs, its error that of a chain of K multiply-adds."""
    rng = np.random.default_rng(640 + 7 * 33 + 2049)
    A, B = rng.standard_normal((640, 2049)), rng.standard_normal((2049, 33))
    assert (np.abs(_gemm(A, B) - A @ B) <= 2 * 2049 * 2.0 ** -53 * (np.abs(A) @ np.abs(B))).all()


@pytest.mark.parametrize("M,N,K", [(512, 512, 512), (300, 700, 1000), (600, 600, 4096)])
def test_gemm_error_below_an_fma_chain(lib_built, M, N, K):
    """N(0, 1) operands against extended precision: the 2-norm error is the final rounding's (2^-53 / sqrt(3) of the
    result at most) and the grid's, 2^-59 sqrt(K) of row maximum times column maximum."""
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    C0 = rng.standard_normal((M, N))
    got = _gemm(A, B)
    rows = rng.choice(M, 4, replace=False)
    want = np.stack([(A[r].astype(np.longdouble)[:, None] * B.astype(np.longdouble)).sum(0) for r in rows])
    err = np.linalg.norm((got[rows] - want).astype(float))
    grid = 2.0 ** -59 * np.sqrt(K) * np.linalg.norm(np.abs(A[rows]).max(1)[:, None] * np.abs(B).max(0)[None, :])
    assert err <= 2.0 ** -53 / np.sqrt(3.0) * np.linalg.norm(want.astype(float)) + 4.0 * grid
    # alpha and beta act on the rounded product, as in the FP64 kernel
    full = _gemm(A, B, alpha=-0.5, beta=2.0, C0=C0)
    assert np.array_equal(full, 2.0 * C0 + -0.5 * got)


def test_gemm_all_digits_at_their_largest(lib_built):
    """Constant operands whose digits all have one sign and full size: every level sum at its bound."""
    x = float(2 ** 53 - 1) * 2.0 ** -53
    y = (255 * 2 ** 45 + 127 * sum(256 ** j for j in range(5)) * 2 ** 5) * 2.0 ** -53
    for K in (512, 1024):
        for u, v in ((x, x), (x, -y), (y, y)):
            got = _gemm(np.full((384, K), u), np.full((K, 640), v))
            want = float(np.longdouble(u) * np.longdouble(v) * K)
            assert (got == got[0, 0]).all()
            assert abs(got[0, 0] - want) <= 2.0 ** -52 * abs(want)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_gemm_nonfinite_operands(lib_built, bad):
    """Infinities and NaNs come out where the FP64 kernel puts them."""
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((512, 512)), rng.standard_normal((512, 576))
    A[17, 3] = bad
    B[100, 401] = bad
    C0 = rng.standard_normal((512, 576))
    with np.errstate(invalid="ignore"):
        want = A @ B
        got = _gemm(A, B)
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
        fin = np.isfinite(want)
        assert np.abs(got[fin] - want[fin]).max() < 1e-11
        kept = _gemm(A, B, beta=1.0, C0=C0)  # C is read once
        assert np.abs(kept[fin] - (want + C0)[fin]).max() < 1e-11


def test_gemm_rows_far_from_flat(lib_built):
    """Entries over sixty binary orders inside a row: as exact as an FP64 sum, element by element."""
    rng = np.random.default_rng(4)
    A = rng.standard_normal((512, 512)) * np.exp2(rng.uniform(-60, 0, (512, 512)))
    B = rng.standard_normal((512, 512)) * np.exp2(rng.uniform(-60, 0, (512, 512)))
    got = _gemm(A, B)
    err = np.abs(got - A @ B)
    assert (err <= 512 * 2.0 ** -52 * (np.abs(A) @ np.abs(B))).all()


def test_gemm_tiny_and_huge_values(lib_built):
    """Results that are subnormal, overflow or come from subnormal operands are rounded like FP64's."""
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((512, 512)), rng.standard_normal((512, 512))
    base = _gemm(A, B)
    assert np.array_equal(_gemm(A * 2.0 ** 600, B * 2.0 ** -580), base * 2.0 ** 20)
    tiny = _gemm(A * 2.0 ** -520, B * 2.0 ** -530)  # results around 2^-1045
    assert np.abs(tiny * 2.0 ** 500 - base * 2.0 ** -550).max() <= 2.0 ** -574
    with np.errstate(over="ignore"):
        assert np.array_equal(_gemm(A * 2.0 ** 600, B * 2.0 ** 422), base * 2.0 ** 1022)
