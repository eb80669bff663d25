"""Operands of the FP64 matvec on digits (csrc/stack_f64.cu, csrc/digit_gemm.cu): what lies behind
them in memory, and columns of R that are zero or subnormal."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_digit_matvec import _apply, _apply_complex, _complex_plan, _problem
from tk_gb300 import Environment, _abi

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


def _right_sector(key, nc):
    """Charges of leg 3 of a packed block key (8 bits of two's complement a component)."""
    q = [(int(key) >> (8 * (3 * nc + c))) & 255 for c in range(nc)]
    return tuple(v - 256 if v > 127 else v for v in q)


# ket states of R that no operator connects, and states connected by subnormal elements alone, with large
# amplitudes in psi: they add nothing, or nothing that counts, to the result
@pytest.mark.parametrize("scale,boost", [(0.0, 2.0 ** 30), (2.0 ** -1060, 2.0 ** 900)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("name,D", [("heisenberg", 401), ("hubbard", 700), ("cylinder", 257)])
def test_vanishing_columns_of_r_cost_the_others_no_digits(lib_built, name, D, cplx, scale, boost):
    def change(e, side):
        if side == 0:
            return e
        d = e.data.copy()
        d[:, :, ::5] *= scale
        return Environment(d, e.bra_idx, e.mpo_idx, e.ket_idx)

    p = _problem(name, D, change)
    rng = np.random.default_rng(D)
    plan = _complex_plan(p, rng, False) if cplx else p.plan()
    if cplx:  # (imaginary parts are drawn where the real part is not zero: scaled here as well)
        from tk_gb300 import Heff2Plan, sweep

        def dev(e, side):
            im = rng.standard_normal(e.data.shape) * (e.data != 0.0)
            if side:
                im[:, :, ::5] *= scale
            return sweep.DeviceEnv.from_dense(p.kind, e.data + 1j * im, e.bra_idx, e.mpo_idx, e.ket_idx)

        plan = Heff2Plan.from_device_envs_complex(dev(p.env_l, 0), dev(p.env_r, 1), p.w_i, p.w_j, p.flux)
    assert plan.launches() == 6
    ket = p.env_r.ket_idx
    nc = len(ket.sectors[0][0])
    first, at = {}, 0
    for q, n in ket.sectors:
        first[tuple(q)] = (at, n)
        at += n
    x = rng.standard_normal(plan.block_dim) + (1j * rng.standard_normal(plan.block_dim) if cplx else 0.0)
    keys, offs = plan.blocks()
    for key, a, b in zip(keys, offs, list(offs[1:]) + [plan.block_dim]):
        o, n = first[_right_sector(key, nc)]
        cols = (o + np.arange(n)) % 5 == 0
        x[a:b].reshape(-1, n)[:, cols] *= boost
    if cplx:
        got, want = ([np.concatenate(_apply_complex(plan, x, s))] for s in (_abi.SCHED_STACKED, _abi.SCHED_GROUPED))
    else:
        got, want = ([_apply(plan, x, s)] for s in (_abi.SCHED_STACKED, _abi.SCHED_GROUPED))
    assert np.isfinite(want[0]).all() and np.linalg.norm(want[0]) < 2.0 ** 40
    assert rel_err(got[0], want[0]) < 64 * 2.0 ** -53


def _left_sector(key, nc):
    q = [(int(key) >> (8 * (2 * nc + c))) & 255 for c in range(nc)]
    return tuple(v - 256 if v > 127 else v for v in q)


# the same for L's ket states; and ket states on scales of their own (2^-20 .. 2^20, taken back in psi),
# which a stack's rows must not see
@pytest.mark.parametrize("kind", ["zero", "subnormal", "scales"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("name,D", [("heisenberg", 401), ("hubbard", 700), ("cylinder", 257), ("cylinder", 500)])
def test_uneven_columns_of_l_cost_no_digits(lib_built, name, D, cplx, kind):
    from tk_gb300 import Heff2Plan, sweep

    p = _problem(name, D, lambda e, side: e)
    rng = np.random.default_rng(D)
    n = p.env_l.data.shape[2]
    if kind == "scales":
        left = np.exp2(rng.integers(-20, 21, n).astype(float))
        back = 1.0 / left
    else:
        left, back = np.ones(n), np.ones(n)
        left[::5], back[::5] = (0.0, 2.0 ** 30) if kind == "zero" else (2.0 ** -1060, 2.0 ** 900)
    if cplx:
        def dev(e, s):
            z = e.data + 1j * rng.standard_normal(e.data.shape) * (e.data != 0.0)
            re, im = z.real * s, z.imag * s
            return sweep.DeviceEnv.from_dense(p.kind, re + 1j * im, e.bra_idx, e.mpo_idx, e.ket_idx)

        plan = Heff2Plan.from_device_envs_complex(dev(p.env_l, left), dev(p.env_r, np.ones(p.env_r.data.shape[2])), p.w_i, p.w_j, p.flux)
    else:
        e = p.env_l
        plan = type(p)(p.kind, Environment(e.data * left, e.bra_idx, e.mpo_idx, e.ket_idx), p.env_r, p.w_i, p.w_j, p.flux, p.name).plan()
    assert plan.launches() == 6
    first, at = {}, 0
    for q, m in p.env_l.ket_idx.sectors:
        first[tuple(q)] = (at, m)
        at += m
    nr = dict((tuple(q), m) for q, m in p.env_r.ket_idx.sectors)
    nc = len(p.env_l.ket_idx.sectors[0][0])
    x = rng.standard_normal(plan.block_dim) + (1j * rng.standard_normal(plan.block_dim) if cplx else 0.0)
    keys, offs = plan.blocks()
    for key, a, b in zip(keys, offs, list(offs[1:]) + [plan.block_dim]):
        o, m = first[_left_sector(key, nc)]
        x[a:b].reshape(-1, m, nr[_right_sector(key, nc)])[:] *= back[o:o + m, None]
    run = (lambda s: np.concatenate(_apply_complex(plan, x, s))) if cplx else (lambda s: _apply(plan, x, s))
    got, want = run(_abi.SCHED_STACKED), run(_abi.SCHED_GROUPED)
    assert np.isfinite(want).all() and np.linalg.norm(want) < 2.0 ** 40
    assert rel_err(got, want) < 64 * 2.0 ** -53


# a converged state in mixed canonical form: identity channels in both environments, amplitudes that fall
# from 1 to 1e-8 along both bonds inside every sector
@pytest.mark.parametrize("name,D", [("heisenberg", 401), ("hubbard", 700), ("cylinder", 257)])
def test_rows_of_a_graded_state_beside_identity_channels(lib_built, name, D):
    """Digits hold rows and columns to 2^-58 of their largest element, so the promise is by norm, as for the
    eigensolvers: the result to a few 2^-53, and each of its rows to the bound of an FP64 chain (2 K 2^-53)
    on the row's largest sum of magnitudes, K the terms of an output."""
    def change(e, side):
        d = e.data.copy()
        w = 0 if side == 0 else d.shape[1] - 1
        d[:, w, :] = np.eye(d.shape[0])
        return Environment(d, e.bra_idx, e.mpo_idx, e.ket_idx)

    p = _problem(name, D, change)
    plan = p.plan()
    assert plan.launches() == 6
    fall = [{tuple(q): np.logspace(0, -8, n) for q, n in e.ket_idx.sectors} for e in (p.env_l, p.env_r)]
    nc = len(p.env_l.ket_idx.sectors[0][0])
    x = np.random.default_rng(D).standard_normal(plan.block_dim)
    keys, offs = plan.blocks()
    blocks = [(a, b, _left_sector(k, nc), _right_sector(k, nc)) for k, a, b in zip(keys, offs, list(offs[1:]) + [plan.block_dim])]
    for a, b, ql, qr in blocks:
        x[a:b].reshape(-1, len(fall[0][ql]), len(fall[1][qr]))[:] *= fall[0][ql][:, None] * fall[1][qr]
    got, want = _apply(plan, x, _abi.SCHED_STACKED), _apply(plan, x, _abi.SCHED_GROUPED)
    assert rel_err(got, want) < 64 * 2.0 ** -53

    def absolute(t):
        out = type(t).__new__(type(t))
        out.__dict__.update(t.__dict__)
        out.blocks = {k: np.abs(v) for k, v in t.blocks.items()}
        return out

    q = type(p)(p.kind, *(Environment(np.abs(e.data), e.bra_idx, e.mpo_idx, e.ket_idx) for e in (p.env_l, p.env_r)),
                absolute(p.w_i), absolute(p.w_j), p.flux, p.name)
    mags = _apply(q.plan(), np.abs(x), _abi.SCHED_GROUPED)
    K = p.env_l.data.shape[1] * (p.env_l.data.shape[2] + p.env_r.data.shape[2])
    for a, b, ql, qr in blocks:
        n = len(fall[1][qr])
        err, row = np.abs(got - want)[a:b].reshape(-1, n).max(1), mags[a:b].reshape(-1, n).max(1)
        assert (err <= 2 * K * 2.0 ** -53 * row).all()


def _structured(e, rng):
    """An environment with some of: channels, bra and ket states on scales of 2^-20 .. 2^20, nine elements in
    ten left out, groups of states with couplings of 1e-10, an identity channel; and the ket scales."""
    d = e.data.copy()
    nb, nw, nk = d.shape
    ket = np.ones(nk)
    pick = rng.random(6)
    if pick[0] < 0.4:
        d *= np.exp2(rng.integers(-20, 21, nw).astype(float))[None, :, None]
    if pick[1] < 0.4:
        d *= np.exp2(rng.integers(-20, 21, nb).astype(float))[:, None, None]
    if pick[2] < 0.6:
        ket = np.exp2(rng.integers(-20, 21, nk).astype(float))
        d *= ket
    if pick[3] < 0.3:
        d *= rng.random(d.shape) < 0.1
    if pick[4] < 0.3:
        g = rng.integers(0, 3, nb)
        d *= np.where(g[:, None, None] == g[None, None, :], 1.0, 1e-10)
    if pick[5] < 0.4:
        d[:, rng.integers(2) * (nw - 1), :] = np.eye(nb)
    return Environment(d, e.bra_idx, e.mpo_idx, e.ket_idx), ket


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("seed", range(24))
def test_norm_error_of_structured_environments(lib_built, seed, cplx):
    """The difference from FP64 chains, in the 2-norm, against what they promise themselves: 2 K 2^-53 of
    the sums of magnitudes, K the terms of an output."""
    from tk_gb300 import Heff2Plan, sweep

    rng = np.random.default_rng(seed)
    p = _problem(*[("heisenberg", 401), ("cylinder", 257), ("hubbard", 700)][seed % 3], lambda e, side: e)
    (el, kl), (er, kr) = _structured(p.env_l, rng), _structured(p.env_r, rng)

    def absolute(t):
        out = type(t).__new__(type(t))
        out.__dict__.update(t.__dict__)
        out.blocks = {k: np.abs(v) for k, v in t.blocks.items()}
        return out

    def turned(e):
        return sweep.DeviceEnv.from_dense(p.kind, e.data * np.exp(2j * np.pi * rng.random(e.data.shape)), e.bra_idx, e.mpo_idx, e.ket_idx)

    q = type(p)(p.kind, el, er, p.w_i, p.w_j, p.flux, p.name)
    plan = Heff2Plan.from_device_envs_complex(turned(el), turned(er), p.w_i, p.w_j, p.flux) if cplx else q.plan()
    nc = len(el.ket_idx.sectors[0][0])
    first, at = {}, 0
    legs = []
    for e, scale in ((el, kl), (er, kr)):
        n = len(scale)
        # taken back, left alone, falling, on scales of its own
        f = [1.0 / scale, np.ones(n), None, np.exp2(rng.integers(-20, 21, n).astype(float))][rng.integers(4)]
        if f is None:
            f = np.concatenate([np.logspace(0, -8, m) for _, m in e.ket_idx.sectors])
        first, at = {}, 0
        for c, m in e.ket_idx.sectors:
            first[tuple(c)] = f[at:at + m]
            at += m
        legs.append(first)
    x = rng.standard_normal(plan.block_dim)
    keys, offs = plan.blocks()
    for key, a, b in zip(keys, offs, list(offs[1:]) + [plan.block_dim]):
        fl, fr = legs[0][_left_sector(key, nc)], legs[1][_right_sector(key, nc)]
        x[a:b].reshape(-1, len(fl), len(fr))[:] *= fl[:, None] * fr
    z = x * np.exp(2j * np.pi * rng.random(len(x))) if cplx else x
    run = (lambda s: np.concatenate(_apply_complex(plan, z, s))) if cplx else (lambda s: _apply(plan, z, s))
    got, want = run(_abi.SCHED_STACKED), run(_abi.SCHED_GROUPED)
    mags = type(p)(p.kind, *(Environment(np.abs(e.data), e.bra_idx, e.mpo_idx, e.ket_idx) for e in (el, er)),
                   absolute(p.w_i), absolute(p.w_j), p.flux, p.name)
    size = np.linalg.norm(_apply(mags.plan(), np.abs(x), _abi.SCHED_GROUPED))
    K = el.data.shape[1] * (max(m for _, m in el.ket_idx.sectors) + max(m for _, m in er.ket_idx.sectors))
    assert np.linalg.norm(got - want) <= 2 * K * 2.0 ** -53 * size
