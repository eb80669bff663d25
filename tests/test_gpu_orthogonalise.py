"""The solvers' one-launch orthogonalisation (csrc/eigensolver.cu): Krylov dimensions at the edges of
its eight-vector groups, vectors from less than one CTA to several elements a thread."""
import numpy as np
import pytest

from helpers import models, small_problem

pytestmark = pytest.mark.gpu


def _plan(name, D):
    if name == "wide":
        return models.workload("heisenberg_d1024", scale=D / 1024.0).plan()
    return small_problem(name, D).plan()


def _basis(plan, x, k):
    """k Lanczos vectors of the plan's matvec, orthogonalised twice in torch; (basis, tridiagonal matrix)."""
    import torch

    q = [x / x.norm()]
    T = np.zeros((k, k))
    for j in range(k):
        w = torch.empty_like(x)
        plan.apply(q[j], w)
        T[j, j] = float(q[j] @ w)
        Q = torch.stack(q)
        for _ in range(2):
            w = w - Q.T @ (Q @ w)
        if j + 1 < k:
            T[j, j + 1] = T[j + 1, j] = float(w.norm())
            q.append(w / w.norm())
    return torch.stack(q), T


@pytest.mark.parametrize("name,D", [("heisenberg", 24), ("hubbard", 64), ("wide", 512)])
@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 16, 17, 33])
def test_lanczos_steps(lib_built, name, D, k):
    """The Ritz value of k steps: the projected matrix's entries agree to a few roundings of |H|, and so its
    lowest eigenvalue (Weyl)."""
    import torch

    plan = _plan(name, D)
    x = torch.from_numpy(np.random.default_rng(k).standard_normal(plan.block_dim)).cuda()
    _, T = _basis(plan, x, k)
    e = np.linalg.eigvalsh(T)
    r = plan.lanczos(krylov_dim=k, tol=0.0, x0=x)
    assert abs(r.eigenvalue - e[0]) <= 1e-12 * max(abs(e[0]), abs(e[-1]))
    assert abs(float(r.eigenvector.norm()) - 1.0) < 1e-13


@pytest.mark.parametrize("k", [1, 8, 9, 17])
def test_expm_steps(lib_built, k):
    """exp(-i dt H) v on k Krylov vectors against the same space in torch."""
    import torch

    plan = _plan("hubbard", 64)
    rng = np.random.default_rng(k)
    x = torch.from_numpy(rng.standard_normal(plan.block_dim)).cuda()
    Q, T = _basis(plan, x, k)
    w, z = np.linalg.eigh(T)
    c = z @ (np.exp(-0.01j * w) * z[0]) * float(x.norm())
    re, im, used, _ = plan.expm(-0.01j, x, krylov_dim=k, tol=1e-14)
    assert used == k
    want = torch.from_numpy(c.real).cuda() @ Q, torch.from_numpy(c.imag).cuda() @ Q
    for got, ref in zip((re, im), want):
        assert float((got - ref).norm()) <= 1e-11 * float(x.norm())


def test_davidson_from_an_eigenvector(lib_built):
    """A start vector that is already converged; then one whose first corrections nearly vanish."""
    import torch

    plan = _plan("heisenberg", 24)
    r = plan.davidson(max_subspace=30, max_iter=400, tol=1e-10)
    again = plan.davidson(max_subspace=30, max_iter=5, tol=1e-9, x0=r.eigenvector)
    assert again.converged and again.matvec_count == 1 and abs(again.eigenvalue - r.eigenvalue) < 1e-11 * abs(r.eigenvalue)
    tight = plan.davidson(max_subspace=30, max_iter=3, tol=0.0, x0=r.eigenvector)
    assert abs(tight.eigenvalue - r.eigenvalue) < 1e-11 * abs(r.eigenvalue)
    assert bool(torch.isfinite(tight.eigenvector).all())


def test_solvers_on_two_threads(lib_built):
    """Two plans solved at once from two threads on two streams: the results of solving them in turn."""
    import threading

    import torch

    plans = [_plan("hubbard", 64), _plan("wide", 512)]
    alone = [p.davidson(max_subspace=20, max_iter=12, tol=1e-14) for p in plans]
    got = [[], []]

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(4):
                got[i].append(plans[i].davidson(max_subspace=20, max_iter=12, tol=1e-14, stream=s.cuda_stream))
                s.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for ref, runs in zip(alone, got):
        assert len(runs) == 4
        for r in runs:
            assert r.eigenvalue == ref.eigenvalue and torch.equal(r.eigenvector, ref.eigenvector)
