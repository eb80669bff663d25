"""Operands of the FP64 matvec on digits (csrc/stack_f64.cu, csrc/digit_gemm.cu): what lies behind
them in memory."""
import numpy as np
import pytest

from test_gpu_digit_matvec import _apply, _apply_complex, _complex_plan, _problem
from tk_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0x7B, 0x7E, 0xFB])  # fp16 61,280, NaN, -61,280
def stale(request, lib_built):
    """Arms and disarms the filling of a plan's allocations."""
    fill = _abi.load().tk_debug_fail_device_alloc
    yield lambda on: fill(-request.param if on else 0)
    fill(0)


# column tiles of few columns, beside rows of other stacks and of later chunks
@pytest.mark.parametrize("name,D", [("hubbard", 700), ("heisenberg", 401), ("cylinder", 257)])
def test_result_does_not_depend_on_unwritten_memory(stale, name, D):
    p = _problem(name, D, lambda e, side: e)
    plan = p.plan()
    x = np.random.default_rng(D).standard_normal(plan.block_dim)
    want = _apply(plan, x)
    stale(True)
    assert np.array_equal(_apply(p.plan(), x), want)


@pytest.mark.parametrize("name,D", [("hubbard", 700), ("heisenberg", 401), ("cylinder", 257)])
def test_complex_result_does_not_depend_on_unwritten_memory(stale, name, D):
    p = _problem(name, D, lambda e, side: e)
    plan = _complex_plan(p, np.random.default_rng(D), False)
    x = np.random.default_rng(1).standard_normal(plan.block_dim) * (1.0 + 0.3j)
    want = _apply_complex(plan, x, _abi.SCHED_STACKED)
    stale(True)
    got = _apply_complex(_complex_plan(p, np.random.default_rng(D), False), x, _abi.SCHED_STACKED)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
