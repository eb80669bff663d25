"""Device memory of tk_gemm_f64 (csrc/linalg.cu): what stays with the context is bounded and given back
when memory runs out, and a product without memory for its digits takes the FP64 kernel."""
import numpy as np
import pytest

from helpers import small_problem
from test_gpu_digit_gate import _run
from tk_gb300 import TkError, _abi
from tk_gb300.heff import context

pytestmark = pytest.mark.gpu
MiB = 1 << 20


def _used():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _refuse(n):
    _abi.load().tk_debug_fail_device_alloc(n)


def _refused_plan():
    """A plan whose first allocation finds no memory: the contexts' idle buffers are released."""
    try:
        _refuse(1)
        with pytest.raises(TkError):
            small_problem("hubbard", 48).plan()
    finally:
        _refuse(0)


def test_kept_memory_is_bounded_and_given_back(lib_built):
    rng = np.random.default_rng(1)
    context(0)
    A, B = rng.standard_normal((300, 300)), rng.standard_normal((300, 300))
    _run(A, B, "tk_gemm_f64")  # module and pool are there
    _refused_plan()  # (what earlier tests left with the context goes)
    before = _used()
    big = rng.standard_normal((5000, 5000))  # 708 MB of digits
    _run(big, big, "tk_gemm_f64")
    assert _used() - before <= 576 * MiB  # 512 and what the driver adds to a mapping
    mid = big[:2048, :2048].copy()  # 117 MB
    _run(mid, mid, "tk_gemm_f64")
    kept = _used()
    assert kept - before >= 100 * MiB  # (else there is nothing to give back)
    _refused_plan()
    assert _used() <= kept - 100 * MiB
    assert np.isfinite(_run(mid, mid, "tk_gemm_f64")).all()


def test_product_without_memory_for_digits_runs_in_fp64(lib_built):
    rng = np.random.default_rng(2)
    A, B = rng.standard_normal((512, 300)), rng.standard_normal((300, 640))
    want = _run(A, B, "tk_gemm_f64_noalloc")
    assert not np.array_equal(_run(A, B, "tk_gemm_f64"), want)  # on digits
    _refused_plan()
    try:
        _refuse(1)
        got = _run(A, B, "tk_gemm_f64")
    finally:
        _refuse(0)
    assert np.array_equal(got, want)
