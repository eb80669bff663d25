"""The FP64 matvec on digits (csrc/stack_f64.cu, csrc/digit_gemm.cu): exact on integers, as exact
as the grouped FP64 schedule on environments whose channels differ by many orders, and back on
the FP64 kernels for infinities and NaNs."""
import numpy as np
import pytest

from helpers import models, rel_err, small_problem
from tk_gb300 import Environment, _abi

pytestmark = pytest.mark.gpu

# one or several K chunks and column tiles, one tile to many, ragged sectors
CASES = [("heisenberg", 401), ("heisenberg", 1024), ("hubbard", 700), ("cylinder", 257), ("cylinder", 500)]


def _problem(name, D, change):
    if name == "hubbard":
        md, bl, br = models.hubbard(), models.gaussian_bond_u1u1(D, 6, 2.0, 2.0, 5), models.gaussian_bond_u1u1(D, 8, 2.0, 2.0, 5)
        p = models.two_site_problem(md, bl, br, 3, "hubbard")
    else:
        p = small_problem(name, D, 3)
    return models.TwoSiteProblem(p.kind, change(p.env_l, 0), change(p.env_r, 1), p.w_i, p.w_j, p.flux, p.name)


def _apply(plan, x, schedule=None):
    import torch

    if schedule is not None:
        plan.set_schedule(schedule)
    xd = torch.from_numpy(x).cuda()
    yd = torch.full_like(xd, float("nan"))
    plan.apply(xd, yd)
    torch.cuda.synchronize()
    return yd.cpu().numpy()


@pytest.mark.parametrize("name,D", CASES)
def test_digit_matvec_exact_on_integers(lib_built, name, D):
    """Integer environments and vectors: both schedules' sums are exact, so the results are equal."""
    def ints(e, side):
        return Environment(np.rint(4.0 * e.data), e.bra_idx, e.mpo_idx, e.ket_idx)

    plan = _problem(name, D, ints).plan()
    assert plan.launches() == 6  # digits of psi and T2, two products, the combine, the stand-by
    rng = np.random.default_rng(D)
    for hi in (3, 1000):
        x = rng.integers(-hi, hi + 1, plan.block_dim).astype(float)
        y = _apply(plan, x, _abi.SCHED_STACKED)
        assert np.array_equal(y, _apply(plan, x, _abi.SCHED_GROUPED))
        assert np.abs(y).max() < 2.0 ** 53


@pytest.mark.parametrize("name,D", CASES)
def test_digit_matvec_channels_of_many_orders(lib_built, name, D):
    """Channels scaled by 2^-20 .. 2^20 (an energy beside identities), sectors of psi by 2^-30 .. 1: the
    difference from the grouped schedule stays that of two FP64 chains, a few 2^-53 sqrt(K)."""
    rng = np.random.default_rng(D + 1)

    def scaled(e, side):
        s = np.exp2(rng.integers(-20, 21, e.data.shape[1]).astype(float))
        return Environment(e.data * s[None, :, None], e.bra_idx, e.mpo_idx, e.ket_idx)

    p = _problem(name, D, scaled)
    plan = p.plan()
    keys, offs = plan.blocks()
    x = rng.standard_normal(plan.block_dim)
    for a, b in zip(offs, list(offs[1:]) + [plan.block_dim]):
        x[a:b] *= np.exp2(-30.0 * rng.random())
    assert rel_err(_apply(plan, x, _abi.SCHED_STACKED), _apply(plan, x, _abi.SCHED_GROUPED)) < 64 * 2.0 ** -53


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_digit_matvec_nonfinite(lib_built, bad):
    p = _problem("cylinder", 257, lambda e, side: e)
    plan = p.plan()
    x = np.random.default_rng(1).standard_normal(plan.block_dim)
    good = _apply(plan, x)
    xb = x.copy()
    xb[plan.block_dim // 3] = bad
    got, want = _apply(plan, xb, _abi.SCHED_STACKED), _apply(plan, xb, _abi.SCHED_GROUPED)
    assert not np.isfinite(want).all()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    fin = np.isfinite(want)
    assert rel_err(got[fin], want[fin]) < 1e-14
    assert np.array_equal(_apply(plan, x, _abi.SCHED_STACKED), good)  # the next matvec is on digits again
    # an environment with one: the plan keeps the FP64 kernels
    e = p.env_r.data.copy()
    i = np.argwhere(e != 0.0)[7]
    e[tuple(i)] = bad
    q = models.TwoSiteProblem(p.kind, p.env_l, Environment(e, p.env_r.bra_idx, p.env_r.mpo_idx, p.env_r.ket_idx), p.w_i,
                              p.w_j, p.flux, p.name)
    plan = q.plan()
    assert plan.launches() == 3
    got, want = _apply(plan, x, _abi.SCHED_STACKED), _apply(plan, x, _abi.SCHED_GROUPED)
    # (the grouped kernel's rows also meet channels that W leaves empty: 0 * inf, the stacked one's do not)
    assert not np.isfinite(got).all()
    both = np.isfinite(got) & np.isfinite(want)
    assert rel_err(got[both], want[both]) < 1e-14


def test_digit_matvec_two_plans_on_two_streams(lib_built):
    import torch

    plans = [_problem(n, d, lambda e, side: e).plan() for n, d in (("cylinder", 257), ("hubbard", 700))]
    xs = [torch.from_numpy(np.random.default_rng(i).standard_normal(p.block_dim)).cuda() for i, p in enumerate(plans)]
    alone = [torch.empty_like(x) for x in xs]
    for p, x, y in zip(plans, xs, alone):
        p.apply(x, y)
    torch.cuda.synchronize()
    ys = [torch.empty_like(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in plans]
    for _ in range(10):
        for p, x, y, s in zip(plans, xs, ys, streams):
            p.apply(x, y, stream=s.cuda_stream)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(alone, ys))


def _complex_plan(p, rng, integers):
    """A plan over complex environments (not Hermitian: the matvec does not need it)."""
    from tk_gb300 import Heff2Plan, sweep

    def dev(e):
        im = rng.standard_normal(e.data.shape) * (e.data != 0.0)
        z = e.data + 1j * im
        if integers:
            z = np.rint(4.0 * z.real) + 1j * np.rint(4.0 * z.imag)
        return sweep.DeviceEnv.from_dense(p.kind, z, e.bra_idx, e.mpo_idx, e.ket_idx)

    return Heff2Plan.from_device_envs_complex(dev(p.env_l), dev(p.env_r), p.w_i, p.w_j, p.flux)


def _apply_complex(plan, x, schedule):
    import torch

    plan.set_schedule(schedule)
    xr, xi = torch.from_numpy(x.real.copy()).cuda(), torch.from_numpy(x.imag.copy()).cuda()
    yr, yi = torch.full_like(xr, float("nan")), torch.full_like(xr, float("nan"))
    plan.apply_complex(xr, xi, yr, yi)
    torch.cuda.synchronize()
    return yr.cpu().numpy(), yi.cpu().numpy()


# K of a part below 32 (its two parts drained together), below 64, of several chunks
@pytest.mark.parametrize("name,D", [("heisenberg", 130), ("heisenberg", 401), ("hubbard", 400), ("cylinder", 257)])
def test_digit_matvec_complex(lib_built, name, D):
    p = _problem(name, D, lambda e, side: e)
    rng = np.random.default_rng(D)
    plan = _complex_plan(p, rng, True)
    assert plan.launches() == 6
    x = rng.integers(-9, 10, plan.block_dim) + 1j * rng.integers(-9, 10, plan.block_dim)
    for got, want in zip(_apply_complex(plan, x, _abi.SCHED_STACKED), _apply_complex(plan, x, _abi.SCHED_GROUPED)):
        assert np.array_equal(got, want)  # every sum is exact
    plan = _complex_plan(p, rng, False)
    x = rng.standard_normal(plan.block_dim) + 1j * rng.standard_normal(plan.block_dim)
    got, want = _apply_complex(plan, x, _abi.SCHED_STACKED), _apply_complex(plan, x, _abi.SCHED_GROUPED)
    assert rel_err(got[0] + 1j * got[1], want[0] + 1j * want[1]) < 64 * 2.0 ** -53
    x[plan.block_dim // 2] = complex(np.inf, 1.0)
    got, want = _apply_complex(plan, x, _abi.SCHED_STACKED), _apply_complex(plan, x, _abi.SCHED_GROUPED)
    for g, w in zip(got, want):
        assert np.array_equal(np.isfinite(g), np.isfinite(w)) and not np.isfinite(w).all()
        assert rel_err(g[np.isfinite(w)], w[np.isfinite(w)]) < 1e-13
