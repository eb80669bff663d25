"""Environments with sectors that no operator reaches (csrc/stack_f64.cu): the matvec's rows there are zeros,
whatever kernels the plan runs."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_digit_matvec import _apply, _apply_complex, _complex_plan, _problem
from tk_gb300 import Environment, _abi

pytestmark = pytest.mark.gpu


def _without(e, sectors, axis):
    d = e.data.copy()
    at = 0
    for i, (_, n) in enumerate(e.bra_idx.sectors):
        if i in sectors:
            d[(slice(None),) * axis + (slice(at, at + n),)] = 0.0
        at += n
    return Environment(d, e.bra_idx, e.mpo_idx, e.ket_idx)


# plans on FP64 kernels and on digits
@pytest.mark.parametrize("name,D", [("heisenberg", 40), ("heisenberg", 401), ("hubbard", 700), ("cylinder", 257)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("side,axis", [(1, 0), (1, 2), (0, 0), (0, 2)])
@pytest.mark.parametrize("which", ["first", "middle", "last", "all but one"])
def test_sectors_without_blocks(lib_built, name, D, cplx, side, axis, which):
    def change(e, s):
        n = len(e.bra_idx.sectors)
        gone = {"first": [0], "middle": [n // 2, n // 2 + 1], "last": [n - 1], "all but one": [i for i in range(n) if i != n // 2]}
        return _without(e, gone[which], axis) if s == side else e

    p = _problem(name, D, change)
    rng = np.random.default_rng(D)
    plan = _complex_plan(p, rng, False) if cplx else p.plan()
    x = rng.standard_normal(plan.block_dim) + (1j * rng.standard_normal(plan.block_dim) if cplx else 0.0)
    run = (lambda s: np.concatenate(_apply_complex(plan, x, s))) if cplx else (lambda s: _apply(plan, x, s))
    got, want = run(_abi.SCHED_STACKED), run(_abi.SCHED_GROUPED)  # (written over NaNs)
    assert np.isfinite(got).all() and np.array_equal(got == 0.0, want == 0.0)
    assert rel_err(got, want) < 64 * 2.0 ** -53
