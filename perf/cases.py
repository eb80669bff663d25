"""Timed cases: the work a DMRG / TDVP program has this library do, through its public entry points.

Every case is a dict with a "kind":
  apply      y = H_eff x on device vectors (Heff2Plan.apply), the inner step of every eigensolver
  host       the same on page-locked host vectors (Heff2Plan.apply_host_flat), the closure a host program calls
  lanczos    LanczosSolver's k-step run; davidson: a bounded Davidson run (the sweep's default solver)
  expm       exp(-i dt H) v on a complex plan, one local TDVP update
  grow       one environment growth (sweep.grow_left / grow_right) between two sweep steps
  gemm       LinAlgBackend::gemm on device matrices (tk_gemm_f64)
  block_gemm SparseLinAlgBackend::block_gemm on host tensors

Models, MPO bonds and sector shapes are those of tk_gb300.models (spin-1/2 Heisenberg, Fermi-Hubbard, J1 cylinder).
Environments are Hermitian (L_pi(w) = L_w^H) with N(0, 1) / sqrt(largest sector) entries, so that H_eff stays O(1)
at every bond dimension.  Two-site vectors are normalised; "graded" ones fall off along both bonds as a state in mixed
canonical form does (Schmidt values from 1 down to 1e-6 inside every sector)."""
import ctypes as C
import math
import os
import sys
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensorkraft-design_gb300"))
from tk_gb300 import PREC_BF16X3, PREC_FP64, Heff2Plan, _abi, context, contract, models, sweep  # noqa: E402
from tk_gb300.symmetry import U1U1, BlockSparseTensor, QIndex  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # first sweeps of a run and every chain edge: tiny sectors, launch latency
        {"name": "apply_fp64_heisenberg_d64", "kind": "apply", "model": "heisenberg", "d": 64, "precision": "fp64", "graded": False},
        # the benchmark's two-site bond: many small U(1)xU(1) sectors
        {"name": "apply_fp64_hubbard_d2048", "kind": "apply", "model": "hubbard", "d": 2048, "precision": "fp64", "graded": False},
        # wide bond of a two-dimensional system: a few large sectors, the state graded as in a converged sweep
        {"name": "apply_fp64_cylinder_d2048", "kind": "apply", "model": "cylinder", "d": 2048, "precision": "fp64", "graded": True},
        # split precision: the operator inside Jacobi-Davidson corrections
        {"name": "apply_split_hubbard_d2048", "kind": "apply", "model": "hubbard", "d": 2048, "precision": "split", "graded": False},
        {"name": "apply_split_cylinder_d2048", "kind": "apply", "model": "cylinder", "d": 2048, "precision": "split", "graded": True},
        # a host program's closure: vectors in page-locked host memory, both transfers in the call
        {"name": "host_split_hubbard_d2048", "kind": "host", "model": "hubbard", "d": 2048, "precision": "split", "graded": False},
        # one Lanczos run of 20 steps (a DMRG step of a small spin chain)
        {"name": "lanczos_fp64_heisenberg_d1024", "kind": "lanczos", "model": "heisenberg", "d": 1024, "steps": 20, "graded": True},
        # a Davidson run as a sweep step makes it, stopped after a fixed number of iterations
        {"name": "davidson_fp64_hubbard_d512", "kind": "davidson", "model": "hubbard", "d": 512, "steps": 16, "graded": True},
        # one real-time update of two-site TDVP: Krylov 16, dt = 0.05
        {"name": "expm_complex_hubbard_d512", "kind": "expm", "model": "hubbard", "d": 512, "steps": 16, "graded": True},
        # the environment update after a sweep step
        {"name": "grow_left_hubbard_d2048", "kind": "grow", "model": "hubbard", "d": 2048, "left": True},
        # dense backend product
        {"name": "gemm_2048", "kind": "gemm", "m": 2048, "n": 2048, "k": 2048, "ta": False, "tb": False, "alpha": 1.0, "beta": 0.0},
        # block-sparse backend product on host tensors: 15 U(1) sectors, D = 1024
        {"name": "block_gemm_u1_d1024", "kind": "block_gemm", "sectors": 15, "d": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


MODELS = {"heisenberg": (16, 1024), "hubbard": (32, 2048), "cylinder": (64, 2048)}


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "apply", "host", "lanczos", "davidson", "expm", "grow", "gemm", "gemm", "block_gemm"])
    if kind == "gemm":
        return {"kind": kind, "m": _log(rng, 16, 2048), "n": _log(rng, 16, 2048), "k": _log(rng, 16, 2048),
                "ta": rng.random() < 0.5, "tb": rng.random() < 0.5, "alpha": rng.choice([1.0, -0.5]), "beta": rng.choice([0.0, 1.0, 2.0])}
    if kind == "block_gemm":
        return {"kind": kind, "sectors": rng.choice([3, 5, 7, 9, 11, 15]), "d": _log(rng, 32, 1024)}
    if kind == "grow":
        return {"kind": kind, "model": "hubbard", "d": _log(rng, 32, 2048), "left": rng.random() < 0.5}
    if kind == "expm":
        return {"kind": kind, "model": "hubbard", "d": _log(rng, 32, 512), "steps": rng.randint(6, 16), "graded": rng.random() < 0.5}
    model = rng.choice(sorted(MODELS))
    lo, hi = MODELS[model]
    if kind in ("lanczos", "davidson"):
        return {"kind": kind, "model": model, "d": _log(rng, lo, min(hi, 640)), "steps": rng.randint(8, 20 if kind == "lanczos" else 16),
                "graded": rng.random() < 0.5}
    prec = "split" if kind == "host" else rng.choice(["fp64", "fp64", "split"])
    return {"kind": kind, "model": model, "d": _log(rng, lo, hi), "precision": prec, "graded": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------- inputs


@lru_cache(maxsize=None)
def _model(name):
    return {"heisenberg": models.heisenberg, "hubbard": models.hubbard, "cylinder": lambda: models.cylinder_j1(4)}[name]()


@lru_cache(maxsize=None)
def _bonds(name, d):
    """The two bonds of a case: the sector shapes of the library's own workloads at dimension d."""
    if name == "heisenberg":
        b = models.gaussian_bond_u1(d, 15, 3.0)
        return b, b
    if name == "hubbard":
        return models.gaussian_bond_u1u1(d, 30), models.gaussian_bond_u1u1(d, 32)
    b = models.heavy_tailed_bond_u1(d, 41, np.random.default_rng(1241))
    return b, b


def _pack(kind, qns):
    """Packed sector key: leg l from bit l * width, 8 bits of two's complement per charge component, component 0 lowest."""
    nc = 2 if kind == U1U1 else 1
    key = 0
    for leg, q in enumerate(qns):
        for c in range(nc):
            key |= (int(q[c]) & 255) << (8 * (leg * nc + c))
    return key


def _offsets(ix):
    out, o = [], 0
    for q, dim in ix.sectors:
        out.append((tuple(q), o, dim))
        o += dim
    return out


def _blocks(kind, legs, signs):
    """[(sector entry of each leg)] with sum sign * charge == 0, ascending by packed key."""
    nc = 2 if kind == U1U1 else 1
    last = {q: (q, o, n) for q, o, n in _offsets(legs[-1])}
    found = []

    def rec(i, cur, tot):
        if i == len(legs) - 1:
            q = tuple(-signs[-1] * t for t in tot)
            if q in last:
                ent = cur + [last[q]]
                found.append((_pack(kind, [e[0] for e in ent]), ent))
            return
        for e in _offsets(legs[i]):
            rec(i + 1, cur + [e], tuple(t + signs[i] * c for t, c in zip(tot, e[0])))

    rec(0, [], (0,) * nc)
    found.sort(key=lambda f: f[0])
    return found


def _flat_index(found, legs):
    """Dense row-major index of every element of the block layout."""
    dims = [ix.total_dim for ix in legs]
    strides = np.cumprod([1] + dims[:0:-1])[::-1]
    parts = []
    for _, ent in found:
        idx = np.zeros((1,), dtype=np.int64)
        for (q, o, n), st in zip(ent, strides):
            idx = (idx[:, None] + (o + np.arange(n, dtype=np.int64))[None, :] * int(st)).reshape(-1)
        parts.append(idx)
    return np.concatenate(parts) if parts else np.zeros(0, dtype=np.int64)


@lru_cache(maxsize=None)
def _psi_blocks(name, d):
    md, (bl, br) = _model(name), _bonds(name, d)
    return _blocks(md.kind, [md.phys, md.phys, bl, br], [1, 1, 1, -1])


@lru_cache(maxsize=4)
def _psi_index(name, d):
    md, (bl, br) = _model(name), _bonds(name, d)
    return torch.from_numpy(_flat_index(_psi_blocks(name, d), [md.phys, md.phys, bl, br])).to(DEV)


@lru_cache(maxsize=4)
def _env_index(name, d, side):
    md, b = _model(name), _bonds(name, d)[side]
    legs = [b, md.bond, b]
    return torch.from_numpy(_flat_index(_blocks(md.kind, legs, [1, -1, -1]), legs)).to(DEV)


def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _env_dense(name, d, side, seed, cplx=False):
    """Hermitian random environment as a dense (bra, w, ket) tensor, zero outside the allowed blocks."""
    md, b = _model(name), _bonds(name, d)[side]
    D, nw = b.total_dim, md.bond.total_dim
    g = _gen(seed, 11 + side)
    idx = _env_index(name, d, side)
    flat = torch.zeros(D * nw * D, dtype=torch.complex128 if cplx else torch.float64, device=DEV)
    v = torch.randn(idx.numel(), generator=g, device=DEV, dtype=torch.float64)
    flat[idx] = torch.complex(v, torch.randn(idx.numel(), generator=g, device=DEV, dtype=torch.float64)) if cplx else v
    e = flat.view(D, nw, D)
    pi = torch.from_numpy(md.pi).to(DEV)
    return (e + e.conj().transpose(0, 2)[:, pi, :]) * (0.5 / math.sqrt(int(b.dims().max())))


def _fall(ix):
    """Schmidt-like weights of a bond's states: from 1 down to 1e-6 inside each sector."""
    return torch.cat([torch.logspace(0, -6, n, dtype=torch.float64) if n > 1 else torch.ones(1, dtype=torch.float64) for _, n in ix.sectors]).to(DEV)


def _psi(case, seed, salt=5):
    """Normalised two-site vector in the block layout."""
    md, (bl, br) = _model(case["model"]), _bonds(case["model"], case["d"])
    idx = _psi_index(case["model"], case["d"])
    x = torch.randn(idx.numel(), generator=_gen(seed, salt), device=DEV, dtype=torch.float64)
    if case["graded"]:
        D = br.total_dim
        x *= _fall(bl)[(idx // D) % bl.total_dim] * _fall(br)[idx % D]
    return x / x.norm()


def _device_env(name, d, side, seed, cplx=False):
    md, b = _model(name), _bonds(name, d)[side]
    e = _env_dense(name, d, side, seed, cplx).reshape(-1)[_env_index(name, d, side)]
    if cplx:
        return sweep.DeviceEnv(md.kind, b, md.bond, b, e.real.contiguous(), e.imag.contiguous())
    return sweep.DeviceEnv(md.kind, b, md.bond, b, e)


def _plan(case, seed, precision=PREC_FP64):
    md = _model(case["model"])
    flux = (0,) * (2 if md.kind == U1U1 else 1)
    el, er = (_device_env(case["model"], case["d"], s, seed) for s in (0, 1))
    return Heff2Plan.from_device_envs(el, er, md.bulk, md.bulk, flux, precision=precision)


def _site_blocks(case):
    """Legs and blocks of the MPS site tensor (s, a_L, a_R) between an environment's bond and the next one (one more, or
    to the left one fewer, spin-up particle)."""
    md, b = _model(case["model"]), _bonds(case["model"], case["d"])[0]
    step = 1 if case["left"] else -1
    nb = QIndex(md.kind, [(tuple(c + step for c in q), n) for q, n in b.sectors])
    legs = [md.phys, b, nb] if case["left"] else [md.phys, nb, b]
    return legs, _blocks(md.kind, legs, [1, 1, -1])


def _site(case, seed):
    legs, found = _site_blocks(case)
    sizes = [math.prod(e[2] for e in ent) for _, ent in found]
    offs = np.zeros(len(sizes), dtype=np.int64)
    offs[1:] = np.cumsum(sizes)[:-1]
    data = torch.randn(max(1, sum(sizes)), generator=_gen(seed, 21), device=DEV, dtype=torch.float64) / math.sqrt(case["d"])
    return sweep.SiteTensor(_model(case["model"]).kind, legs, np.array([k for k, _ in found], dtype=np.uint64), offs, data)


def _bst_pair(case, seed):
    b = models.gaussian_bond_u1(case["d"], case["sectors"], 3.0)
    rng = np.random.default_rng(int(seed))
    out = []
    for _ in range(2):
        t = BlockSparseTensor([b, b], (0,), [0, 1])
        for q, n in b.sectors:
            t.set_block([q, q], rng.standard_normal((n, n)))
        out.append(t)
    return out


def _mats(case, seed):
    m, n, k = case["m"], case["n"], case["k"]
    g = _gen(seed, 31)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    return (r(k, m) if case["ta"] else r(m, k)), (r(n, k) if case["tb"] else r(k, n)), r(m, n)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("apply", "host"):
        plan = _plan(case, seed, PREC_FP64 if case["precision"] == "fp64" else PREC_BF16X3)
        x = _psi(case, seed)
        if kind == "host":
            x = x.cpu().pin_memory()
            y = torch.empty_like(x).pin_memory()
            return {"kind": kind, "plan": plan, "x": x, "y": y, "xn": x.numpy(), "yn": y.numpy()}
        return {"kind": kind, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind in ("lanczos", "davidson"):
        return {"kind": kind, "plan": _plan(case, seed), "x": _psi(case, seed), "steps": case["steps"]}
    if kind == "expm":
        md = _model(case["model"])
        el, er = (_device_env(case["model"], case["d"], s, seed, True) for s in (0, 1))
        plan = Heff2Plan.from_device_envs_complex(el, er, md.bulk, md.bulk, (0, 0))
        return {"kind": kind, "plan": plan, "re": _psi(case, seed), "im": _psi(case, seed, 6), "steps": case["steps"]}
    if kind == "grow":
        return {"kind": kind, "left": case["left"], "env": _device_env(case["model"], case["d"], 0, seed), "site": _site(case, seed),
                "w": _model(case["model"]).bulk}
    if kind == "gemm":
        a, b, c = _mats(case, seed)
        m, n, k = case["m"], case["n"], case["k"]
        ma = _abi.tk_mat(a.data_ptr(), m, k, 1 if case["ta"] else k, m if case["ta"] else 1, 0)
        mb = _abi.tk_mat(b.data_ptr(), k, n, 1 if case["tb"] else n, k if case["tb"] else 1, 0)
        return {"kind": kind, "a": a, "b": b, "c": c, "ma": ma, "mb": mb, "m": m, "n": n, "alpha": case["alpha"], "beta": case["beta"],
                "lib": _abi.load(), "ctx": context(0)}
    a, b = _bst_pair(case, seed)
    return {"kind": kind, "a": a, "b": b}


def run(state):
    kind = state["kind"]
    if kind == "apply":
        state["plan"].apply(state["x"], state["y"])
        return state["y"]
    if kind == "host":
        state["plan"].apply_host_flat(state["xn"], state["yn"])
        return state["y"]
    if kind == "lanczos":
        r = state["plan"].lanczos(krylov_dim=state["steps"], max_restarts=0, tol=1e-14, x0=state["x"])
        return {"energy": r.eigenvalue, "vector": r.eigenvector}
    if kind == "davidson":
        r = state["plan"].davidson(max_subspace=60, max_iter=state["steps"], tol=1e-14, x0=state["x"])
        return {"energy": r.eigenvalue, "vector": r.eigenvector}
    if kind == "expm":
        re, im, _, _ = state["plan"].expm(-0.05j, state["re"], state["im"], krylov_dim=state["steps"], tol=1e-14)
        return {"re": re, "im": im}
    if kind == "grow":
        return (sweep.grow_left if state["left"] else sweep.grow_right)(state["env"], state["site"], state["w"]).data
    if kind == "gemm":
        out = state["c"].clone() if state["beta"] else torch.empty_like(state["c"])
        mc = _abi.tk_mat_mut(out.data_ptr(), state["m"], state["n"], state["n"], 1)
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _abi.check(state["lib"].tk_gemm_f64(state["ctx"], state["alpha"], C.byref(state["ma"]), C.byref(state["mb"]), state["beta"],
                                            C.byref(mc), s))
        return out
    t = contract.block_gemm(state["a"], state["b"])
    return [t.blocks[k] for k in sorted(t.blocks)]


# ---------------------------------------------------------------------------------------------- what a pass cannot do without


@lru_cache(maxsize=None)
def _wij(name):
    """Fused two-site operator: (d*d in, d*d out, w_L, w_R)."""
    w = torch.from_numpy(_model(name).bulk.to_dense())
    d, nw = w.shape[0], w.shape[2]
    return torch.einsum("abwm,cdmv->acbdwv", w, w).reshape(d * d, d * d, nw, nw)


def _matvec_work(name, d):
    """Multiply-adds of one factored matvec over the sectors (L psi once per sector pair and channel, then R) and the
    elements of L, R and psi."""
    md, (bl, br) = _model(name), _bonds(name, d)
    nc = 2 if md.kind == U1U1 else 1
    add = lambda *q: tuple(sum(c[i] for c in q) for i in range(nc))  # noqa: E731
    neg = lambda q: tuple(-c for c in q)  # noqa: E731
    da, db = ({tuple(q): n for q, n in ix.sectors} for ix in (bl, br))
    wq = [tuple(q) for q in md.bond.state_charges()]
    ps = [add(u, v) for u in md.phys.state_charges() for v in md.phys.state_charges()]
    W = (_wij(name) != 0).numpy()
    flops = 0.0
    for p, qp in enumerate(ps):
        used = W[p].any(axis=(0, 2))
        for qa, na in da.items():
            nb = db.get(add(qp, qa), 0)
            flops += 2.0 * na * nb * sum(da.get(add(qa, w), 0) for w, u in zip(wq, used) if u)
    for p, qp in enumerate(ps):
        for qa, na in da.items():
            qb2 = add(qp, qa)
            if qb2 not in db:
                continue
            for v, w in enumerate(wq):
                nb = db.get(add(qb2, neg(w)), 0)
                if nb and W[:, p, :, v].any():
                    flops += 2.0 * na * nb * db[qb2]
    env = sum(n * x.get(add(q, w), 0) for x in (da, db) for q, n in x.items() for w in wq)
    return flops, env, sum(math.prod(e[2] for e in ent) for _, ent in _psi_blocks(name, d))


def work(case):
    kind = case["kind"]
    if kind in ("apply", "host"):
        f, env, psi = _matvec_work(case["model"], case["d"])
        return {"bytes": 8.0 * (env + 2 * psi), "flops": f}
    if kind in ("lanczos", "davidson", "expm"):
        f, env, psi = _matvec_work(case["model"], case["d"])
        s, c = case["steps"], 4.0 if kind == "expm" else 1.0
        # s matvecs and the orthogonalisation of s basis vectors
        return {"bytes": (2.0 if kind == "expm" else 1.0) * 8.0 * (s * (env + 2 * psi) + s * s * psi), "flops": c * s * (f + 4.0 * s * psi)}
    if kind == "grow":
        md = _model(case["model"])
        legs, found = _site_blocks(case)
        bond, new = (legs[1], legs[2]) if case["left"] else (legs[2], legs[1])
        dims = {tuple(q): n for q, n in bond.sectors}
        dims2 = {tuple(q): n for q, n in new.sectors}
        wq = [tuple(q) for q in md.bond.state_charges()]
        add = lambda a, b: tuple(x + y for x, y in zip(a, b))  # noqa: E731
        env = sum(n * dims.get(add(q, w), 0) for q, n in dims.items() for w in wq)
        out = sum(n * dims2.get(add(q, w), 0) for q, n in dims2.items() for w in wq)
        site = sum(math.prod(e[2] for e in ent) for _, ent in found)
        i, j = (1, 2) if case["left"] else (2, 1)
        f = 0.0
        for _, ent in found:
            q, n, q2, n2 = ent[i][0], ent[i][2], ent[j][0], ent[j][2]
            f += sum(2.0 * n * n2 * dims.get(add(q, w), 0) + 2.0 * n * n2 * dims2.get(add(q2, w), 0) for w in wq)
        return {"bytes": 8.0 * (env + out + site), "flops": f}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8.0 * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2.0 * m * n * k}
    dims = models.gaussian_bond_u1(case["d"], case["sectors"], 3.0).dims()
    return {"bytes": 24.0 * float((dims.astype(float) ** 2).sum()), "flops": 2.0 * float((dims.astype(float) ** 3).sum())}


# ---------------------------------------------------------------------------------------------- the same in plain 64-bit torch


def _dense_heff(case, seed, cplx=False):
    """H_eff on dense (p, a, b) tensors: L, then W_i W_j, then R."""
    el, er = (_env_dense(case["model"], case["d"], s, seed, cplx) for s in (0, 1))
    w = _wij(case["model"]).to(DEV)
    if cplx:
        w = w.to(torch.complex128)
    D, nw, _ = el.shape
    E, P = er.shape[0], w.shape[0]
    L2, R2 = el.reshape(D * nw, D), er.reshape(E, nw * E)  # R2[b', (w, b)]

    def apply(x):
        y = torch.zeros(P, D, E, dtype=x.dtype, device=DEV)
        t = [(L2 @ x[p]).view(D, nw, E) for p in range(P)]
        for q in range(P):
            t2 = torch.zeros(D, nw, E, dtype=x.dtype, device=DEV)
            for p, u, v in torch.nonzero(w[:, q]).tolist():
                t2[:, v] += w[p, q, u, v] * t[p][:, u]
            y[q] = t2.view(D, nw * E) @ R2.T
        return y

    idx = _psi_index(case["model"], case["d"])

    def flat(v):
        d = torch.zeros(P * D * E, dtype=v.dtype, device=DEV)
        d[idx] = v
        return apply(d.view(P, D, E)).reshape(-1)[idx]

    return flat


def _krylov(h, v, steps):
    """Orthonormal Krylov basis (twice orthogonalised) and the projected matrix."""
    basis = [v / v.norm()]
    t = torch.zeros(steps, steps, dtype=v.dtype, device=DEV)
    for k in range(steps):
        w = h(basis[k])
        q = torch.stack(basis)
        c = q.conj() @ w
        t[: k + 1, k] = c
        for _ in range(2):
            w = w - q.T @ (q.conj() @ w)
        b = w.norm()
        if k + 1 < steps:
            if float(b) < 1e-13:
                return torch.stack(basis), t[: k + 1, : k + 1]
            t[k + 1, k] = b
            basis.append(w / b)
    return torch.stack(basis), t


def exact(case, seed):
    kind = case["kind"]
    if kind in ("apply", "host"):
        y = _dense_heff(case, seed)(_psi(case, seed))
        return y.cpu() if kind == "host" else y
    if kind == "lanczos":
        q, t = _krylov(_dense_heff(case, seed), _psi(case, seed), case["steps"])
        e, _ = torch.linalg.eigh(t)  # the lower triangle is read
        return {"energy": float(e[0]), "vector": None}  # the vector's sign is the solver's choice
    if kind == "davidson":
        return None  # its iterates are the algorithm's own
    if kind == "expm":
        h = _dense_heff(case, seed, True)
        v = torch.complex(_psi(case, seed), _psi(case, seed, 6))
        q, t = _krylov(h, v, case["steps"])
        e, z = torch.linalg.eigh(t)  # the lower triangle is read
        c = z @ (torch.exp(-0.05j * e) * z[0].conj()) * v.norm()
        y = q.T @ c
        return {"re": y.real.contiguous(), "im": y.imag.contiguous()}
    if kind == "grow":
        md = _model(case["model"])
        legs, found = _site_blocks(case)
        e = _env_dense(case["model"], case["d"], 0, seed)
        s = _site(case, seed)
        a = torch.zeros(math.prod(ix.total_dim for ix in legs), dtype=torch.float64, device=DEV)
        a[torch.from_numpy(_flat_index(found, legs)).to(DEV)] = s.data
        a = a.view(*[ix.total_dim for ix in legs])
        w = torch.from_numpy(md.bulk.to_dense()).to(DEV)  # (s_in, s_out, w_L, w_R)
        if not case["left"]:
            a, w = a.transpose(1, 2).contiguous(), w.transpose(2, 3).contiguous()  # mirror image
        d, D, F = a.shape
        nw = e.shape[1]
        out = torch.zeros(F, nw, F, dtype=torch.float64, device=DEV)
        t = [(e.reshape(D * nw, D) @ a[i]).view(D, nw, F) for i in range(d)]
        for o in range(d):
            t2 = torch.zeros(D, nw, F, dtype=torch.float64, device=DEV)
            for i, u, v in torch.nonzero(w[:, o]).tolist():
                t2[:, v] += w[i, o, u, v] * t[i][:, u]
            out += (a[o].T @ t2.reshape(D, nw * F)).view(F, nw, F)
        new = legs[2] if case["left"] else legs[1]
        nl = [new, md.bond, new]
        return out.reshape(-1)[torch.from_numpy(_flat_index(_blocks(md.kind, nl, [1, -1, -1]), nl)).to(DEV)]
    if kind == "gemm":
        a, b, c = _mats(case, seed)
        y = case["alpha"] * ((a.T if case["ta"] else a) @ (b.T if case["tb"] else b))
        return y + case["beta"] * c if case["beta"] else y
    a, b = _bst_pair(case, seed)
    return [a.blocks[k] @ b.blocks[k] for k in sorted(a.blocks)]
