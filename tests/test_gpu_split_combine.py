"""The split path's combine in pairs of columns (csrc/tc_gemm.cu, form 0, 64 or 128 threads a job)
against the form that takes one element at a time: the same sums in the same order, so the same bits."""
import numpy as np
import pytest

from helpers import small_problem
from tk_gb300 import PREC_BF16X3

pytestmark = pytest.mark.gpu


# few jobs and small ones, jobs of one pass and of several, rows longer than the block, odd sectors
# (jobs that begin or end inside a pair), from one K chunk to many
@pytest.mark.parametrize("name,D", [("heisenberg", 16), ("heisenberg", 401), ("hubbard", 37), ("hubbard", 700),
                                    ("cylinder", 64), ("cylinder", 107), ("cylinder", 701)])
def test_pairs_match_single_elements(lib_built, name, D):
    import torch

    plan = small_problem(name, D).plan(precision=PREC_BF16X3)
    x = torch.from_numpy(np.random.default_rng(D).standard_normal(plan.block_dim)).cuda()
    ys = []
    for form in (0, 1):
        plan.set_tc_options(3, 0, form, 0, 0)
        y = torch.full_like(x, float("nan"))
        plan.apply(x, y)
        torch.cuda.synchronize()
        ys.append(y.cpu().numpy())
    assert np.isfinite(ys[0]).all()
    assert np.array_equal(ys[0], ys[1])
