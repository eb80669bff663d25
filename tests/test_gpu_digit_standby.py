"""The FP64 kernels behind the matvec on digits (csrc/stack_f64.cu): a plan without memory for the digits,
and the time of a vector that digits cannot hold."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_digit_matvec import _apply, _apply_complex, _complex_plan, _problem
from tk_gb300 import Environment, TkError, _abi

pytestmark = pytest.mark.gpu


def _plan_without_its_last_allocation(make):
    """The plan made while the last allocation of its creation, the digits', finds no memory."""
    lib = _abi.load()
    try:
        n = 0
        while True:  # allocations of a creation: the countdown that none reaches
            n += 1
            lib.tk_debug_fail_device_alloc(n)
            try:
                plan = make()
            except TkError as e:
                assert e.status == 3  # TK_ERR_OOM
                continue
            return plan, n
    finally:
        lib.tk_debug_fail_device_alloc(0)


@pytest.mark.parametrize("name,D", [("hubbard", 700), ("cylinder", 257)])
@pytest.mark.parametrize("cplx", [False, True])
def test_plan_without_memory_for_digits_runs_in_fp64(lib_built, name, D, cplx):
    p = _problem(name, D, lambda e, side: e)
    make = (lambda: _complex_plan(p, np.random.default_rng(3), False)) if cplx else p.plan
    assert make().launches() == 6
    plan, _ = _plan_without_its_last_allocation(make)
    assert plan.launches() == 3
    x = np.random.default_rng(2).standard_normal(plan.block_dim)
    if cplx:
        got, want = (np.concatenate(_apply_complex(plan, x * (1 + 0.5j), s)) for s in (_abi.SCHED_STACKED, _abi.SCHED_GROUPED))
    else:
        got, want = (_apply(plan, x, s) for s in (_abi.SCHED_STACKED, _abi.SCHED_GROUPED))
    assert rel_err(got, want) < 1e-14
    assert make().launches() == 6  # nothing is left armed


def test_profile_counts_the_bytes_of_digits(lib_built):
    """Against the same plan without digits: fourteen bytes an operand element for eight."""
    import torch

    p = _problem("cylinder", 257, lambda e, side: e)
    plan = p.plan()
    fp64, _ = _plan_without_its_last_allocation(p.plan)
    x = torch.from_numpy(np.random.default_rng(2).standard_normal(plan.block_dim)).cuda()
    y = torch.empty_like(x)
    (_, fl, by), (_, fl64, by64) = plan.profile(x, y, reps=1), fp64.profile(x, y, reps=1)
    vec = 8.0 * plan.block_dim
    assert list(fl) == list(fl64)
    assert by[2] - vec == 14.0 / 8.0 * (by64[2] - vec)
    assert by[0] > by64[0] + 28.0 * plan.block_dim / 2 and by[1] > by64[1]


def _time(plan, x):
    import torch

    xd = torch.from_numpy(x).cuda()
    yd = torch.empty_like(xd)
    best = float("inf")
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        plan.apply(xd, yd, stream=torch.cuda.current_stream().cuda_stream)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_nonfinite_vector_costs_about_an_fp64_matvec(lib_built):
    """Against a plan that keeps the FP64 kernels (its environment holds an infinity): the same work on
    the same pipe, which the whole GPU has to share in."""
    p = _problem("cylinder", 1000, lambda e, side: e)
    plan = p.plan()
    assert plan.launches() == 6
    e = p.env_r.data.copy()
    e[tuple(np.argwhere(e != 0.0)[7])] = np.inf
    q = type(p)(p.kind, p.env_l, Environment(e, p.env_r.bra_idx, p.env_r.mpo_idx, p.env_r.ket_idx), p.w_i, p.w_j, p.flux, p.name)
    fp64 = q.plan()
    assert fp64.launches() == 3
    x = np.random.default_rng(1).standard_normal(plan.block_dim)
    bad = x.copy()
    bad[plan.block_dim // 2] = np.nan
    assert _time(plan, bad) < 2.0 * _time(fp64, x)
