"""The workloads that the performance of this library is judged by.

Each case is one call sequence that a program built on the library makes through
the Python mirror of the C ABI (modal-cmb_gb300/modal_gb300.py).  Sizes are those
of the benchmark configurations (cfg1 .. cfg4 of CONFIGS) and of the tests, and
generic ones between them.  Inputs are synthetic and follow from the seed alone:
the shifted Legendre (or B-spline) basis under a C_l whose shape and noise level
vary with the seed, power-law and Gaussian-bump shapes, smooth transfer functions.

  listed()            the fixed cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs, and the context a program keeps
  run(state)          one pass through the public entry points
  work(case)          bytes and operations a pass cannot do without
  exact(case, seed)   the outputs in plain 64-bit numpy / torch
"""
import importlib.util
import math
import os

import numpy as np
import torch

_ROOT = os.getcwd()


def _load():
    path = os.path.join(_ROOT, "modal-cmb_gb300", "modal_gb300.py")
    spec = importlib.util.spec_from_file_location("modal_gb300", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


mg = _load()

LMIN = 2
FLOOR = 1e-4       # PCA floor of the orthogonalisation (the reference's floor-free rule is ill-posed in alpha)
DELTAPHI = 1.5e-8  # primordial amplitude of the transfer Gamma


def listed():
    return [
        # The smallest whole program: a fresh process's first and only pass over the
        # CPU-runnable configuration (cfg1) in the plain FP64 form, context creation
        # included: Gamma, orthogonalisation, four shapes, alpha.
        {"name": "run_l500_p10", "kind": "run", "lmax": 500, "P": 10, "S": 4},
        # The stand-alone quadrature primitives (asy() and the gl_Pl loop of the
        # reference) at the basis-optimisation size (cfg4).
        {"name": "quadrature_n1501", "kind": "quadrature", "n": 1501, "lmax": 1000},
        # Gamma of a new basis in the plain FP64 form at the headline size (cfg2).
        {"name": "gamma_fp64_l2000_p30", "kind": "gamma", "prec": 0, "lmax": 2000, "P": 30},
        # Gamma of a new basis on the tensor cores: a ragged mid size and the headline size.
        {"name": "gamma_split_l1201_p17", "kind": "gamma", "prec": 1, "lmax": 1201, "P": 17},
        {"name": "gamma_split_l2000_p30", "kind": "gamma", "prec": 1, "lmax": 2000, "P": 30},
        # Orthogonalisation (PCA branch) of a Gamma read back from its file, and alpha
        # of 16 shapes: a mid size and the headline size.
        {"name": "ortho_l1000_p16", "kind": "ortho", "lmax": 1000, "P": 16, "S": 16},
        {"name": "ortho_l2000_p30", "kind": "ortho", "lmax": 2000, "P": 30, "S": 16},
        # Projection of 16 separable shapes in the single-precision form (cfg2).
        {"name": "project_l2000_p30_s16", "kind": "project", "lmax": 2000, "P": 30, "sep": 16, "bump": 0, "terms": 2,
         "batch": False},
        # The 256-shape batch, half separable and half bumps, through the captured graph (cfg3).
        {"name": "batch_l2000_p30_s256", "kind": "project", "lmax": 2000, "P": 30, "sep": 128, "bump": 128, "terms": 4,
         "batch": True},
        # Projection in the plain FP64 form (the default precision of modal_project).
        {"name": "project64_l1000_p20_s4", "kind": "project64", "lmax": 1000, "P": 20, "sep": 4, "bump": 0, "terms": 2},
        # One step of the differentiable basis optimisation (cfg4): new B-spline
        # coefficients, FP64 Gamma, Cholesky, residual of 32 shapes and its gradient.
        {"name": "adjoint_l1000_p12_s32", "kind": "adjoint", "lmax": 1000, "P": 12, "S": 32},
        # Late x primordial transfer Gamma, the reference's gamma_mpi driver.
        {"name": "transfer_l600_p16", "kind": "transfer", "lmax": 600, "P": 16, "Pp": 8, "xsize": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "quadrature", "gamma", "gamma", "ortho", "project", "project", "project64", "adjoint",
                       "transfer"])
    if kind == "run":
        return {"kind": kind, "lmax": _log_int(rng, 50, 700), "P": rng.randint(3, 12), "S": rng.randint(1, 8)}
    if kind == "quadrature":
        lmax = _log_int(rng, 50, 2000)
        return {"kind": kind, "n": 3 * lmax // 2 + 1, "lmax": lmax}
    if kind == "gamma":
        return {"kind": kind, "prec": rng.randint(0, 1), "lmax": _log_int(rng, 60, 2000), "P": rng.randint(4, 30)}
    if kind == "ortho":
        return {"kind": kind, "lmax": _log_int(rng, 300, 1500), "P": rng.randint(8, 24), "S": rng.randint(1, 40)}
    if kind == "project":
        batch = rng.random() < 0.5
        most = 24 if batch else 8
        return {"kind": kind, "lmax": _log_int(rng, 100, 1800), "P": rng.randint(6, 40), "sep": rng.randint(1, most),
                "bump": rng.randint(0, most), "terms": rng.randint(1, 4), "batch": batch}
    if kind == "project64":
        return {"kind": kind, "lmax": _log_int(rng, 60, 1000), "P": rng.randint(4, 24), "sep": rng.randint(1, 4),
                "bump": rng.randint(0, 2), "terms": rng.randint(1, 3)}
    if kind == "adjoint":
        return {"kind": kind, "lmax": _log_int(rng, 200, 1000), "P": rng.randint(5, 12), "S": rng.randint(2, 32)}
    return {"kind": kind, "lmax": _log_int(rng, 60, 600), "P": rng.randint(5, 16), "Pp": rng.randint(3, 8),
            "xsize": rng.randint(12, 40)}


# ------------------------------------------------------------------- inputs

def _spectrum(lmax, seed):
    """C_l + N_l: the synthetic spectrum with a seeded smooth modulation and noise level."""
    rng = np.random.default_rng(1000003 * seed + 17)
    cl = mg.synthetic_cl(lmax)
    l = np.arange(lmax + 1.0)
    tilt, amp, freq = rng.uniform(-0.1, 0.1), rng.uniform(0.0, 0.2), rng.uniform(2.0, 6.0)
    return cl * (1.0 + l / lmax) ** tilt * (1.0 + amp * np.sin(freq * l / lmax + rng.uniform(0.0, 6.0)))


def _basis(lmax, P, seed):
    cl = _spectrum(lmax, seed)
    return mg.weighted_q(mg.legendre_q(LMIN, lmax, P), cl, LMIN), cl


def _shapes(case, seed):
    out = mg.separable_shapes(case["lmax"], case["sep"], seed + 1, 1, case["terms"])
    return out + (mg.bump_shapes(case["bump"], seed + 2) if case["bump"] else [])


def _adjoint_inputs(case, seed):
    lmax, P = case["lmax"], case["P"]
    cl = _spectrum(lmax, seed)
    Bw = mg.weighted_q(mg.bspline_matrix(LMIN, lmax, 64), cl, LMIN)
    C = np.random.default_rng(seed).standard_normal((P, 64))
    return Bw @ C.T, mg.mode_triples(P), cl, mg.separable_shapes(lmax, case["S"], seed + 3, 1, 2)


def _transfer_inputs(case, seed):
    lmax, Pp = case["lmax"], case["Pp"]
    xvec, qt = mg.transfer_workload(lmax, Pp, case["xsize"])
    rng = np.random.default_rng(seed)
    ph = rng.uniform(0.0, 0.5, Pp)
    l = np.arange(lmax + 1.0)
    return xvec, qt * (1.0 + 0.3 * np.sin(ph[None, :, None] + 4.0 * l[None, None, :] / lmax)), mg.mode_triples(Pp)


def _ortho_beta(case, seed, N):
    """Projections with the decay of real ones: a seeded vector per shape."""
    rng = np.random.default_rng(seed + 5)
    return rng.standard_normal((case["S"], N)) * np.exp(-np.arange(N) / (0.2 * N))


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    if kind == "quadrature":
        # the seed moves the upper end of the table: its nodes are those of the rule
        rng = np.random.default_rng(seed)
        st["scale"] = 1.0 - 1e-3 * rng.random()
        return st
    if kind == "adjoint":
        q, tri, cl, shapes = _adjoint_inputs(case, seed)
        c = mg.Context(0)
        c.set_basis(LMIN, case["lmax"], q)
        c.set_modes(tri)
        c.set_spectrum(cl)
        st.update(ctx=c, q=q, shapes=shapes)
        return st
    q, cl = _basis(case["lmax"], case["P"], seed)
    tri = mg.mode_triples(case["P"])
    N = len(tri)
    st.update(q=q, cl=cl, tri=tri)
    if kind == "run":
        st["shapes"] = mg.separable_shapes(case["lmax"], case["S"], seed + 1, 1, 2)
        return st
    c = mg.Context(0)
    c.set_basis(LMIN, case["lmax"], q)
    c.set_modes(tri)
    st["ctx"] = c
    if kind == "gamma":
        st["out"] = _pinned(N, N)
    elif kind == "ortho":
        g = _gamma_exact(q, case["lmax"], tri)
        st["gamma"] = _pinned(N, N)
        torch.from_numpy(st["gamma"]).copy_(g)
        st["beta"] = _ortho_beta(case, seed, N)
        c.set_pca_floor(FLOOR)
    elif kind in ("project", "project64"):
        c.set_spectrum(cl)
        st["shapes"] = _shapes(case, seed)
    else:
        xvec, qt, prim = _transfer_inputs(case, seed)
        c.set_spectrum(cl)
        c.set_transfer(xvec, qt, prim)
        c.init_glint()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "quadrature":
        x, w = mg.gl_nodes(case["n"])
        return {"nodes": x, "weights": w, "table": mg.legendre_table(x * st["scale"], case["lmax"])}
    if kind == "run":
        with mg.Context(0) as c:
            c.set_basis(LMIN, case["lmax"], st["q"])
            c.set_modes(st["tri"])
            c.set_spectrum(st["cl"])
            c.set_pca_floor(FLOOR)
            g = c.gamma(mg.PREC_FP64)
            _, _, _, rank = c.orthogonalise(pca_flag=0, download=False)
            beta = c.project(st["shapes"], mg.PREC_FP64)
            alpha, _ = c.alpha(case["S"])
        return {"gamma": g, "rank": rank, "beta": beta, "alpha": alpha}
    c = st["ctx"]
    if kind == "gamma":
        c.set_basis(LMIN, case["lmax"], st["q"])
        c.init_glint()
        return {"gamma": c.gamma(case["prec"], out=st["out"])}
    if kind == "ortho":
        # modesR rides on the eigenvectors' signs; alpha = lambda^T lambda beta does not
        _, _, _, rank = c.orthogonalise(st["gamma"], pca_flag=0, download=False)
        alpha, _ = c.alpha(case["S"], st["beta"])
        return {"rank": rank, "alpha": alpha}
    if kind == "project":
        # the split form computes in single precision: its beta carries FP32 accuracy
        # in a double array, and is kept as what it is
        call = c.project_batch if case["batch"] else c.project
        return {"beta": call(st["shapes"], mg.PREC_SPLIT).astype(np.float32)}
    if kind == "project64":
        return {"beta": c.project(st["shapes"], mg.PREC_FP64)}
    if kind == "adjoint":
        c.set_basis(LMIN, case["lmax"], st["q"])
        c.init_glint()
        c.gamma(mg.PREC_FP64, download=False)
        c.orthogonalise(download=False)
        J, dq = c.adjoint_residual(st["shapes"])
        return {"J": J, "dq": dq}
    return {"gamma_t": c.gamma_transfer(DELTAPHI)}


# --------------------------------------------------------------------- work

def _points(lmax):
    """Tetrapyd points 2 <= i <= j <= k <= lmax, k <= i + j, i + j + k even."""
    i = np.arange(LMIN, lmax + 1)[:, None]
    j = np.arange(LMIN, lmax + 1)[None, :]
    n = (np.minimum(i + j, lmax) - (j + (i & 1))) // 2 + 1
    return int(np.where((j >= i) & (n > 0), n, 0).sum())


def work(case):
    kind = case["kind"]
    lmax = case["lmax"]
    if kind == "quadrature":
        n = case["n"]
        # one recurrence of n steps (4 operations) per root and 4 operations per table entry
        return {"bytes": 8.0 * n * (lmax + 3), "flops": 2.0 * n * n + 4.0 * n * (lmax + 1)}
    P = case["P"]
    L, N, K = lmax - LMIN + 1, P * (P + 1) * (P + 2) // 6, 3 * lmax // 2 + 1
    U = P * (P + 1) // 2
    lift = 2.0 * K * U * (U + 1) * (U + 2) / 6 + 2.0 * K * U * L  # every distinct product of three M entries once
    if kind == "gamma":
        return {"bytes": 8.0 * (L * P + N * N), "flops": lift}
    pts = _points(lmax) if kind in ("run", "project", "project64") else 0
    if kind == "run":
        S = case["S"]
        return {"bytes": 8.0 * (L * P + N * N + S * 5 * L + 2 * S * N), "flops": lift + 4 / 3 * N ** 3 + 2.0 * P * pts * S}
    if kind == "ortho":
        S = case["S"]
        return {"bytes": 8.0 * (N * N + 2 * S * N), "flops": 4 / 3 * N ** 3 + 4.0 * N * N * S}
    if kind in ("project", "project64"):
        S, T = case["sep"] + case["bump"], (1 + case["terms"]) / 2
        return {"bytes": 8.0 * (L * P + case["sep"] * T * 3 * L + S * N), "flops": 2.0 * P * pts * S}
    if kind == "adjoint":
        S, E = case["S"], 3 * case["S"] * 1.5
        # Gamma and its adjoint (three products of the same size), the shapes' legs both ways
        return {"bytes": 8.0 * (2 * L * P + E * L), "flops": 4.0 * lift + 8.0 * K * L * E * P + 18.0 * 1.5 * S * N * K * 3}
    Pp, X = case["Pp"], case["xsize"]
    V = P * Pp
    return {"bytes": 8.0 * (X * Pp * L + L * P + N * Pp * (Pp + 1) * (Pp + 2) / 6),
            "flops": 2.0 * X * K * (V * L + V * (V + 1) * (V + 2) / 6)}


# -------------------------------------------------------------------- exact
# Plain float64 numpy / torch restatements of the formulas in include/modal_gb300.h.

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_PERMS = ((0, 1, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0), (1, 0, 2), (0, 2, 1))


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_DEV)


def _gauss(n):
    """Gauss-Legendre nodes (ascending) and weights by Newton in theta, P_n from the
    differences P_l - P_{l-1} (accurate next to x = 1)."""
    half = n // 2
    k = np.arange(1, half + 1 + (n & 1), dtype=np.float64)
    th = np.pi * (4 * k - 1) / (4 * n + 2)
    th = np.arccos((1 - (n - 1) / (8.0 * n ** 3)) * np.cos(th))
    if n & 1:
        th[-1] = np.pi / 2
    for it in range(5):
        y = 2 * np.sin(0.5 * th) ** 2
        p, d = np.ones_like(th), np.zeros_like(th)
        for l in range(n):
            d = (l * d - (2 * l + 1) * y * p) / (l + 1)
            p = p + d
        q = -d + y * p
        if it < 4:
            step = p * np.sin(th) / (n * q)
            if n & 1:
                step[-1] = 0.0
            th = th + step
    w = 2 * np.sin(th) ** 2 / (float(n) * n * q * q)
    x = np.cos(th)
    if n & 1:
        x[-1] = 0.0
        return np.concatenate([-x, x[:-1][::-1]]), np.concatenate([w, w[:-1][::-1]])
    return np.concatenate([-x, x[::-1]]), np.concatenate([w, w[::-1]])


def _pl(x, lmax):
    """[lmax+1][n] (2l+1)^{2/3} P_l(x)."""
    x = _t(x)
    out = torch.empty((lmax + 1, x.numel()), dtype=torch.float64, device=_DEV)
    out[0] = 1.0
    if lmax >= 1:
        out[1] = x
    for l in range(1, lmax):
        out[l + 1] = ((2 * l + 1) * x * out[l] - l * out[l - 1]) / (l + 1)
    l = torch.arange(lmax + 1, dtype=torch.float64, device=_DEV)
    return out * ((2 * l + 1) ** (2.0 / 3.0))[:, None]


def _gamma_exact(q, lmax, tri):
    """Gamma [N][N]: the triple products of pair sums, gathered over the six orderings."""
    P = q.shape[1]
    x, w = _gauss(3 * lmax // 2 + 1)
    pl = _pl(x, lmax)[LMIN:]
    a, b = np.triu_indices(P)
    U = len(a)
    qt = _t(q)
    X = torch.cat([(qt[:, _t(a[i:i + 64])] * qt[:, _t(b[i:i + 64])]).T @ pl for i in range(0, U, 64)])
    Xw = X * (_t(w) / (48 * math.pi))
    # T[u][v][t] for v <= t, rows v in turn
    T = torch.empty((U, U, U), dtype=torch.float64, device=_DEV)
    for v in range(U):
        T[:, v, v:] = X @ (Xw[v] * X[v:]).T
        T[:, v:, v] = T[:, v, v:]
    pid = np.zeros((P, P), dtype=np.int64)
    pid[a, b] = pid[b, a] = np.arange(U)
    pid, t3, N = _t(pid), _t(np.asarray(tri, dtype=np.int64)), len(tri)
    G = torch.zeros((N, N), dtype=torch.float64, device=_DEV)
    for m0 in range(0, N, 512):
        m = t3[m0:m0 + 512]
        for s in _PERMS:
            i, j, k = (pid[m[:, r, None], t3[None, :, s[r]]] for r in range(3))
            G[m0:m0 + 512] += T[i, j, k]
    return (G + G.T) / 2


def _alpha_exact(G, beta):
    d = torch.sqrt(torch.diagonal(G))
    e, V = torch.linalg.eigh(G / torch.outer(d, d))
    keep = e > FLOOR * e[-1]
    V = V[:, keep]
    return int(keep.sum()), ((((_t(beta) / d) @ V) / e[keep]) @ V.T) / d


def _beta_exact(case, q, cl, shapes):
    """beta [S][N] over the tetrapyd, slab by slab, the two parities of j apart."""
    lmax, P = case["lmax"], case["P"]
    pts = lmax ** 3 / 6
    if pts * len(shapes) > 3e10:
        return None  # about 20 s
    l = np.arange(lmax + 1.0)
    v = np.zeros(lmax + 1)
    v[2:] = (2 * l[2:] + 1) ** (-1 / 3) * (2 * l[2:] + 1) ** (1 / 6) / np.sqrt(cl[2:])
    v, lt = _t(v), torch.arange(lmax + 1, dtype=torch.float64, device=_DEV)
    qf = torch.zeros((lmax + 1, P), dtype=torch.float64, device=_DEV)
    qf[LMIN:] = _t(q)
    tabs = [_t(s["tab"]) if s["kind"] == mg.SHAPE_SEPARABLE else None for s in shapes]
    B = torch.zeros((len(shapes), P, P, P), dtype=torch.float64, device=_DEV)
    for i in range(LMIN, lmax + 1):
        F = torch.zeros((len(shapes), P, P), dtype=torch.float64, device=_DEV)
        for par in (0, 1):
            j0 = i + ((i + par) & 1)
            k0 = j0 + (i & 1)  # k has the parity of i + j
            if j0 > lmax or k0 > lmax:
                continue
            js, ks = slice(j0, lmax + 1, 2), slice(k0, lmax + 1, 2)
            J, K = lt[js][:, None], lt[ks][None, :]
            a1, a2, a3, L = J + K - i, K + i - J, i + J - K, i + J + K
            ok = (K >= J) & (a3 >= 0)
            a3 = torch.where(ok, a3, torch.ones_like(a3))
            h = (0.5 / math.pi ** 2 * (2.0 * i + 1) * (2 * J + 1) * (2 * K + 1) / (L + 1) * (L + 1 / 3) /
                 ((a1 + 1 / 3) * (a2 + 1 / 3) * (a3 + 1 / 3)) *
                 torch.sqrt((a1 + 1 / 6) * (a2 + 1 / 6) * (a3 + 1 / 6) / (L + 1 / 6)))
            same = (J == i).to(torch.float64) + (K == J).to(torch.float64) + (K == i).to(torch.float64)
            perm = torch.where(same == 0, 6.0, torch.where(same == 1, 3.0, 1.0))
            W = torch.where(ok, perm * h * v[i] * v[js][:, None] * v[ks][None, :], torch.zeros_like(h))
            for s, sh in enumerate(shapes):
                if tabs[s] is not None:
                    f, g, hh = tabs[s][:, 0], tabs[s][:, 1], tabs[s][:, 2]
                    left = torch.cat([f[:, i, None] * g[:, js] + g[:, i, None] * f[:, js],
                                      f[:, i, None] * hh[:, js] + hh[:, i, None] * f[:, js],
                                      g[:, i, None] * hh[:, js] + hh[:, i, None] * g[:, js]])
                    val = left.T @ torch.cat([hh[:, ks], g[:, ks], f[:, ks]]) / 6.0
                else:
                    c, sg = sh["c"], float(sh["sigma"])
                    r2 = (i / L - float(c[0])) ** 2 + (J / L - float(c[1])) ** 2 + (K / L - float(c[2])) ** 2
                    val = torch.exp(-r2 / (2 * sg * sg))
                F[s] += qf[js].T @ ((W * val) @ qf[ks])
        B += qf[i][None, :, None, None] * F[:, None]
    t3 = _t(np.asarray(mg.mode_triples(P), dtype=np.int64))
    out = 0.0
    for s in _PERMS:
        out = out + B[:, t3[:, s[0]], t3[:, s[1]], t3[:, s[2]]]
    return out / 6.0


def _perm_sum(A, w, ri, ci):
    """sum_k w_k perm3(A[k][ri[i][a]][ci[j][b]]) -> [len(ri)][len(ci)]."""
    def part(a, ww):
        acc = 0.0
        for s in _PERMS:
            acc = acc + (a[:, ri[:, 0, None], ci[None, :, s[0]]] * a[:, ri[:, 1, None], ci[None, :, s[1]]] *
                         a[:, ri[:, 2, None], ci[None, :, s[2]]])
        return torch.einsum("k,kmn->mn", ww, acc)

    out = 0.0
    for k in range(0, A.shape[0], 64):
        if A.requires_grad:
            out = out + torch.utils.checkpoint.checkpoint(part, A[k:k + 64], w[k:k + 64], use_reentrant=False)
        else:
            out = out + part(A[k:k + 64], w[k:k + 64])
    return out


def _adjoint_exact(case, seed):
    import torch.utils.checkpoint  # noqa: F401
    q, tri, cl, shapes = _adjoint_inputs(case, seed)
    lmax = case["lmax"]
    x, w = _gauss(3 * lmax // 2 + 1)
    pl, wk = _pl(x, lmax)[LMIN:], _t(w) / (48 * math.pi)
    l = np.arange(LMIN, lmax + 1.0)
    wl = (2 * l + 1) ** (1 / 6) / np.sqrt(cl[LMIN:lmax + 1])
    qt = _t(q).requires_grad_(True)
    t3 = _t(np.asarray(tri, dtype=np.int64))
    M = torch.einsum("lk,lp,lq->kpq", pl, qt, qt)
    G = _perm_sum(M, wk, t3, t3)
    betas, n2 = [], []
    for sh in shapes:
        T = sh["tab"].shape[0]
        legs = _t((wl * sh["tab"][:, :, LMIN:lmax + 1]).reshape(3 * T, -1))
        ri = torch.arange(3 * T, device=_DEV).reshape(T, 3)
        betas.append(_perm_sum(torch.einsum("lk,el,lq->keq", pl, legs, qt), wk, ri, t3).sum(0))
        n2.append(_perm_sum(torch.einsum("lk,el,fl->kef", pl, legs, legs), wk, ri, ri).sum())
    beta, n2 = torch.stack(betas), torch.stack(n2)
    J = torch.mean((n2 - (beta * torch.linalg.solve(G, beta.T).T).sum(1)) / n2)
    J.backward()
    return {"J": float(J.detach()), "dq": qt.grad.cpu().numpy()}


def _spline_weights(x):
    """c_x with sum_x c_x y_x the integral of the cubic spline through (x, y) whose end
    conditions are the third differences of the first and last four points."""
    n = len(x)
    h = np.diff(x)
    A, R = np.zeros((n, n)), np.zeros((n, n))
    D = np.zeros((n - 1, n))
    for i in range(n - 1):
        D[i, i], D[i, i + 1] = -1 / h[i], 1 / h[i]
    for i in range(1, n - 1):
        A[i, i - 1], A[i, i], A[i, i + 1] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
        R[i] = D[i] - D[i - 1]
    A[0, 0], A[0, 1] = -h[0], h[0]
    R[0] = ((D[2] - D[1]) / (x[3] - x[1]) - (D[1] - D[0]) / (x[2] - x[0])) * h[0] ** 2 / (x[3] - x[0])
    A[-1, -1], A[-1, -2] = -h[-1], h[-1]
    R[-1] = -((D[-1] - D[-2]) / (x[-1] - x[-3]) - (D[-2] - D[-3]) / (x[-2] - x[-4])) * h[-1] ** 2 / (x[-1] - x[-4])
    S = np.linalg.solve(A, R)  # second derivative / 6 at the nodes
    c = np.zeros(n)
    for i in range(n - 1):
        c[i] += h[i] / 2
        c[i + 1] += h[i] / 2
        c -= h[i] ** 3 / 4 * (S[i] + S[i + 1])
    return c


def _transfer_exact(case, seed):
    lmax, P, Pp = case["lmax"], case["P"], case["Pp"]
    q, cl = _basis(lmax, P, seed)
    xvec, qt, prim = _transfer_inputs(case, seed)
    x, w = _gauss(3 * lmax // 2 + 1)
    l = np.arange(LMIN, lmax + 1.0)
    pl = _pl(x, lmax)[LMIN:] * _t(((2 * l + 1) ** (1 / 6) / np.sqrt(cl[LMIN:lmax + 1])))[:, None]
    qd, tr, pr = _t(q), _t(np.asarray(mg.mode_triples(P), dtype=np.int64)), _t(np.asarray(prim, dtype=np.int64))
    c = _spline_weights(xvec)
    out = torch.zeros((len(tr), len(pr)), dtype=torch.float64, device=_DEV)
    for ix in range(len(xvec)):
        M = torch.einsum("lk,lq,pl->kqp", pl, qd, _t(qt[ix][:, LMIN:]))
        y = _perm_sum(M, _t(w), tr, pr) * xvec[ix] ** 2
        if ix < 10:
            y = torch.where(y.abs() > 1e-18, torch.zeros_like(y), y)
        out += c[ix] * y
    return out.cpu().numpy() * (DELTAPHI ** 2 / (8 * math.pi))


def exact(case, seed):
    kind = case["kind"]
    if kind == "quadrature":
        st = prepare(case, seed)
        x, w = _gauss(case["n"])
        return {"nodes": x, "weights": w, "table": _pl(x * st["scale"], case["lmax"]).T.cpu().numpy()}
    if kind == "adjoint":
        return _adjoint_exact(case, seed)
    if kind == "transfer":
        return {"gamma_t": _transfer_exact(case, seed)}
    q, cl = _basis(case["lmax"], case["P"], seed)
    if kind in ("project", "project64"):
        b = _beta_exact(case, q, cl, _shapes(case, seed))
        return None if b is None else {"beta": b.cpu().numpy()}
    G = _gamma_exact(q, case["lmax"], mg.mode_triples(case["P"]))
    if kind == "gamma":
        return {"gamma": G.cpu().numpy()}
    if kind == "ortho":
        rank, a = _alpha_exact(G, _ortho_beta(case, seed, G.shape[0]))
        return {"rank": rank, "alpha": a.cpu().numpy()}
    beta = _beta_exact(case, q, cl, mg.separable_shapes(case["lmax"], case["S"], seed + 1, 1, 2))
    rank, a = _alpha_exact(G, beta.cpu().numpy())
    return {"gamma": G.cpu().numpy(), "rank": rank, "beta": beta.cpu().numpy(), "alpha": a.cpu().numpy()}
