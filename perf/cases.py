"""Performance cases: what a user of the library has it do, through its Python entry points.

A case is a dict of plain values.  ``call`` names the entry point:

  apply       ``apply``: one H-apply on a column-major CUDA block
  recurrence  ``clenshaw_recurrence``: the mapping callback of one filter step
  filter      ``chebyshev_filter``: a whole Chebyshev filter of order K
  kpm         ``kpm_moments``: density-of-states moments
  extrema     ``lanczos_extrema``: the spectrum's edges
  solve       ``polfed``: one complete solve
  batch       ``polfed_batch``: disorder realisations in flight together

``model`` is "xxz" (random-field XXZ chain), "j1j2" (J1-J2 chain), "csr" (the
XXZ chain handed over as a sparse matrix) or "qsun" (Quantum Sun, a grain of
``G`` spins and ``L`` outer spins).  Chains live in the sector with L // 2
spins up.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The repository's package; its folder name carries a dot, so it is imported by path."""
    if "polfed_b200" not in sys.modules:
        folder = os.path.join(ROOT, "polfed.jl_b200")
        spec = importlib.util.spec_from_file_location("polfed_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["polfed_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["polfed_b200"]


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest call: one matrix-vector product inside a user's own loop (the L = 14 chain of the FP64
        # configuration), where launch latency is all there is
        {"name": "apply_xxz14_s1", "call": "apply", "model": "xxz", "L": 14, "G": 0, "W": 5.0, "s": 1, "dtype": "fp64"},
        # the mapping callback a user's own Clenshaw loop makes per step, on the Quantum Sun of the benchmark
        {"name": "recurrence_qsun13_s8", "call": "recurrence", "model": "qsun", "L": 13, "G": 3, "W": 0.5, "s": 8,
         "dtype": "fp64"},
        # a filter application of one disorder realisation (L = 16 of the disorder batch)
        {"name": "filter_xxz16_s8", "call": "filter", "model": "xxz", "L": 16, "G": 0, "W": 3.0, "s": 8,
         "dtype": "fp64", "K": 300},
        # a filter application of the benchmark's solve
        {"name": "filter_qsun13_s8", "call": "filter", "model": "qsun", "L": 13, "G": 3, "W": 0.5, "s": 8,
         "dtype": "fp64", "K": 430},
        # the large end: the J1-J2 L = 24 chain's single-precision bulk at block size 16, a short filter
        {"name": "filter_j1j2_24_s16_fp32", "call": "filter", "model": "j1j2", "L": 24, "G": 0, "W": 1.0, "s": 16,
         "dtype": "fp32", "K": 40},
        # a user's own sparse matrix, odd dimension (L = 15, 7 up: 6435) and a small block
        {"name": "filter_csr15_s4", "call": "filter", "model": "csr", "L": 15, "G": 0, "W": 5.0, "s": 4,
         "dtype": "fp64", "K": 200},
        # the density of states a benchmark solve takes: 300 random probes, 250 moments
        {"name": "kpm_qsun13_r300", "call": "kpm", "model": "qsun", "L": 13, "G": 3, "W": 0.5, "dtype": "fp64",
         "N": 250, "R": 300, "given": False},
        # single-precision moments with the caller's +-1 probes (64 probes, 512 moments) on a larger chain
        {"name": "kpm_j1j2_20_r64_fp32", "call": "kpm", "model": "j1j2", "L": 20, "G": 0, "W": 1.0, "dtype": "fp32",
         "N": 512, "R": 64, "given": True},
        # the spectrum's edges of a disorder realisation (L = 18)
        {"name": "extrema_xxz18", "call": "extrema", "model": "xxz", "L": 18, "G": 0, "W": 3.0},
        # the plain configuration: scalar Lanczos, 20 pairs in the middle of the L = 14 chain
        {"name": "solve_xxz14_s1", "call": "solve", "model": "xxz", "L": 14, "G": 0, "W": 5.0, "s": 1, "nev": 20,
         "target": 0.5},
        # the benchmark's solve: 200 pairs of the 65536-dimensional Quantum Sun, block size 8
        {"name": "solve_qsun13_s8", "call": "solve", "model": "qsun", "L": 13, "G": 3, "W": 0.5, "s": 8, "nev": 200,
         "target": 0.5},
        # a disorder average: eight realisations in flight together
        {"name": "batch_xxz16_s8", "call": "batch", "model": "xxz", "L": 16, "G": 0, "W": 3.0, "s": 8, "nev": 50,
         "target": 0.5, "n": 8},
    ]


def draw(rng):
    """One more case: models, sizes, block widths and precisions between the listed ones."""
    call = rng.choice(["apply", "recurrence", "filter", "filter", "filter", "kpm", "kpm", "extrema", "solve", "batch"])
    model = rng.choice(["xxz", "j1j2", "csr", "qsun", "qsun"])
    whole = call in ("solve", "batch")
    if whole and model in ("csr", "j1j2"):
        model = "xxz"
    case = {"call": call, "model": model, "G": 0, "W": round(rng.uniform(0.5, 5.0), 2)}
    if model == "qsun":
        case["G"] = rng.choice([2, 3, 3])
        case["W"] = round(rng.uniform(0.3, 0.5), 2)
        case["L"] = rng.randint(9, 12) if whole else rng.randint(8, 15)
    elif model == "csr":
        case["L"] = rng.randint(12, 17)
    else:
        case["L"] = rng.randint(13, 16) if whole else rng.randint(12, 21)
    work = _dim(case) * _row_terms(case)
    if call != "extrema" and not whole:
        case["dtype"] = rng.choice(["fp64", "fp64", "fp32"])
    if call in ("apply", "recurrence", "filter"):
        case["s"] = rng.choice([1, 2, 3, 4, 5, 8, 8, 12, 16, 24])
    if call == "filter":
        top = min(600, int(2.0e10 / (work * case["s"])))
        case["K"] = max(3, round(math.exp(rng.uniform(math.log(20), math.log(max(21, top))))))
    elif call == "kpm":
        case["R"] = max(2, min(rng.randint(10, 300), int(1.0e10 / (work * 64))))
        case["N"] = max(20, min(rng.randint(50, 512), int(4.0e10 / (work * case["R"]))))
        case["given"] = rng.random() < 0.5
    elif whole:
        case["W"] = round(rng.uniform(2.5, 5.0), 2) if model == "xxz" else case["W"]
        case["s"] = rng.choice([1, 4, 8]) if call == "solve" else rng.choice([4, 8])
        case["nev"] = rng.randint(20, 50)
        case["target"] = round(rng.uniform(0.3, 0.55), 3)
        if call == "batch":
            case["n"] = rng.randint(2, 6)
    return case


def _dim(case):
    return 1 << (case["L"] + case["G"]) if case["model"] == "qsun" else math.comb(case["L"], case["L"] // 2)


def _row_terms(case):
    """Average non-zeros of a row of H."""
    L = case["L"]
    if case["model"] == "qsun":
        return L + (1 << case["G"])
    bonds = 2 * L if case["model"] == "j1j2" else L
    up = L // 2
    return 1 + bonds * 2.0 * up * (L - up) / (L * (L - 1))


def work(case):
    """Each input read once and each output written once; every multiply-add the recurrence needs."""
    D, terms = _dim(case), _row_terms(case)
    call = case["call"]
    w = 4 if case.get("dtype") == "fp32" else 8
    if call == "apply":
        return {"bytes": 2 * D * case["s"] * w, "flops": 2 * D * case["s"] * terms}
    if call == "recurrence":
        return {"bytes": 4 * D * case["s"] * w, "flops": 2 * D * case["s"] * (terms + 3)}
    if call == "filter":
        return {"bytes": 2 * D * case["s"] * w, "flops": 2 * D * case["s"] * (terms + 3) * case["K"]}
    if call == "kpm":
        steps = case["N"] // 2
        return {"bytes": (D * case["R"] * w if case["given"] else 0) + 8 * case["N"],
                "flops": 2 * D * case["R"] * (terms + 4) * steps}
    if call == "extrema":
        return {"bytes": 8 * D, "flops": 2 * 2 * D * 100 * (terms + 2 * 100)}
    # a solve: about (20.4 s + 1.7 nev) Krylov vectors, each one filter of an order set by the density of states
    m = 20.427 * case["s"] + 1.696 * case["nev"]
    K = max(20.0, 2.0 * D / case["nev"])
    n = case.get("n", 1)
    return {"bytes": n * 8 * D * case["s"], "flops": n * (2 * D * m * (terms + 3) * K + 4 * D * m * m)}


# ------------------------------------------------------------------ inputs

def _model(case, seed):
    """The realisation's parameters, from the seed alone."""
    rng = np.random.default_rng([int(seed), 11])
    L, W = case["L"], case["W"]
    if case["model"] == "qsun":
        dg = 1 << case["G"]
        goe = rng.standard_normal((dg, dg))
        return {"fields": 1.0 - W + 2 * W * rng.random(L), "nbr": rng.integers(0, case["G"], size=L),
                "coup": 0.75 ** np.maximum(0.0, np.arange(L) + 0.4 * rng.random(L) - 0.2),
                "grain": (goe + goe.T) / math.sqrt(2 * (dg + 1))}
    bonds = [(i, (i + 1) % L) for i in range(L)]
    J = [1.0] * L
    if case["model"] == "j1j2":
        bonds += [(i, (i + 2) % L) for i in range(L)]
        J += [0.5] * L
    return {"fields": W * (2 * rng.random(L) - 1), "bonds": bonds, "J": J}


def _operator(case, m):
    pkg = _package()
    L = case["L"]
    if case["model"] == "qsun":
        return pkg.QSunOperator(L, case["G"], 1.0, m["coup"], m["nbr"], m["fields"], m["grain"])
    if case["model"] == "xxz":
        return pkg.xxz_hamiltonian(L, L // 2, 1.0, 1.0, 0.0, fields=m["fields"])
    if case["model"] == "j1j2":
        return pkg.j1j2_hamiltonian(L, L // 2, 1.0, 0.5, 1.0, 1.0, 0.0, fields=m["fields"])
    diag, idx, on, J = _chain_tables(case, m)
    D = len(diag)
    rows = torch.arange(D, device=diag.device)
    r = [rows] + [rows[o] for o in on]
    c = [rows] + [i[o] for i, o in zip(idx, on)]
    v = [diag] + [torch.full((int(o.sum()),), j / 2, dtype=torch.float64, device=diag.device) for o, j in zip(on, J)]
    r, c, v = torch.cat(r), torch.cat(c), torch.cat(v)
    order = torch.argsort(r * D + c)
    indptr = torch.searchsorted(r[order].contiguous(), torch.arange(D + 1, device=diag.device))
    return pkg.SparseOperator((indptr.cpu().numpy(), c[order].cpu().numpy(), v[order].cpu().numpy()))


def _scale(case, m):
    """(a, b): a bound of H's spectrum, as the caller of a filter has it."""
    h = float(np.abs(m["fields"]).sum()) / 2
    if case["model"] == "qsun":
        return h + float(np.abs(m["coup"]).sum()) / 4 + float(np.linalg.norm(m["grain"], 2)), 0.0
    return h + 0.75 * float(np.sum(m["J"])), 0.0


def _coefficients(case):
    """The Dirac-delta expansion around 0.3: c_0 = 1, c_n = 2 cos(n acos 0.3), scaled to a unit peak."""
    n = np.arange(case["K"] + 1)
    c = (2.0 - (n == 0)) * np.cos(n * math.acos(0.3))
    return c / (1.0 + 2.0 * np.sum(np.cos(n[1:] * math.acos(0.3)) ** 2))


def _block(D, s, case, seed, salt):
    """A column-major block of unit columns."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 16 + salt)
    t = torch.randn((s, D), generator=g, device="cuda", dtype=torch.float64)
    t = t / t.norm(dim=1, keepdim=True)
    return t.to(torch.float32 if case["dtype"] == "fp32" else torch.float64).t()


def _probes(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 16 + 9)
    D = _dim(case)
    t = (torch.randint(0, 2, (case["R"], D), generator=g, device="cuda") * 2 - 1).to(
        torch.float32 if case["dtype"] == "fp32" else torch.float64)
    return (t / math.sqrt(D)).t()


def _start(case, seed):
    """A host start vector or block, as a solve takes it."""
    rng = np.random.default_rng([int(seed), 23])
    s = case.get("s", 1)
    return rng.random(_dim(case)) if s == 1 else np.asfortranarray(rng.random((_dim(case), s)))


def prepare(case, seed):
    call, D = case["call"], _dim(case)
    if call == "batch":
        ops, x0s = [], []
        for i in range(case["n"]):
            ops.append(_operator(case, _model(case, seed * 64 + i)))
            x0s.append(_start(case, seed * 64 + i))
        assert all(op.dim == D for op in ops)
        return {"case": case, "ops": ops, "x0s": x0s, "seed": int(seed)}
    m = _model(case, seed)
    op = _operator(case, m)
    assert op.dim == D
    a, b = _scale(case, m)
    st = {"case": case, "op": op, "a": a, "b": b, "seed": int(seed)}
    if call in ("apply", "recurrence", "filter"):
        st["X"] = _block(D, case["s"], case, seed, 1)
        st["Y"] = torch.empty_like(st["X"])
    if call == "recurrence":
        st["b2"], st["b3"] = _block(D, case["s"], case, seed, 2), _block(D, case["s"], case, seed, 3)
    if call == "filter":
        st["coeffs"] = _coefficients(case)
    if call == "kpm" and case["given"]:
        st["probes"] = _probes(case, seed)
    if call in ("extrema", "solve"):
        st["x0"] = _start(case, seed)
    return st


# ------------------------------------------------------------------ one pass

def run(st):
    pkg, case = _package(), st["case"]
    call = case["call"]
    if call == "apply":
        return pkg.apply(st["op"], st["Y"], st["X"], st["a"], st["b"])
    if call == "recurrence":
        return pkg.clenshaw_recurrence(st["op"], st["Y"], st["b2"], st["b3"], 0.7, st["X"], st["a"], st["b"])
    if call == "filter":
        return pkg.chebyshev_filter(st["op"], st["Y"], st["X"], st["coeffs"], st["a"], st["b"])
    if call == "kpm":
        return pkg.kpm_moments(st["op"], case["N"], case["R"], st["a"], st["b"], probes=st.get("probes"),
                               seed=st["seed"], dtype=case["dtype"])
    if call == "extrema":
        return pkg.lanczos_extrema(st["op"], st["x0"])
    # Solves for level statistics: eigenvalues only.  At the default Lanczos tolerance of 1e-14 and Krylov budget the
    # last pairs hang on rounding; these settings return every pair asked for.
    opts = dict(fact=pkg.FactorizationConfig(tol=1e-11, eigentol=1e-9, overestimate_iters=3.0),
                dos=pkg.DoSConfig(seed=st["seed"]), vecs=False)
    if call == "solve":
        vals, _ = pkg.polfed(st["op"], st["x0"], case["nev"], ("rescaled", case["target"]), **opts)
        return vals
    out = pkg.polfed_batch(st["ops"], st["x0s"], case["nev"], ("rescaled", case["target"]), workers=8, **opts)
    return [vals for vals, _ in out]


# ------------------------------------------------------------------ the same in plain torch

def _chain_tables(case, m):
    """(diagonal, partner index of every bond, where the bond flips, couplings) of a chain sector."""
    L, up = case["L"], case["L"] // 2
    st = torch.arange(1 << L, device="cuda", dtype=torch.int32)
    ones = torch.zeros_like(st)
    for i in range(L):
        ones += (st >> i) & 1
    st = st[ones == up].to(torch.int64)
    diag = torch.zeros(len(st), dtype=torch.float64, device="cuda")
    for i in range(L):
        diag += float(m["fields"][i]) * (((st >> i) & 1).double() - 0.5)
    idx, on = [], []
    for (i, j), J in zip(m["bonds"], m["J"]):
        differ = ((st >> i) ^ (st >> j)) & 1 == 1
        diag += torch.where(differ, -0.25 * J, 0.25 * J)
        to = torch.where(differ, st ^ ((1 << i) | (1 << j)), st)
        idx.append(torch.searchsorted(st, to))
        on.append(differ)
    return diag, idx, on, m["J"]


def _exact_apply(case, m):
    """X -> H X on D x s float64 blocks."""
    if case["model"] != "qsun":
        diag, idx, on, J = _chain_tables(case, m)

        def chain(X):
            Y = diag[:, None] * X
            for i, o, j in zip(idx, on, J):
                Y.add_(X[i] * (o * (j / 2))[:, None])
            return Y
        return chain
    L, G = case["L"], case["G"]
    st = torch.arange(1 << (L + G), device="cuda", dtype=torch.int64)
    diag = torch.zeros(len(st), dtype=torch.float64, device="cuda")
    for j in range(L):
        diag += float(m["fields"][j]) * (((st >> (G + j)) & 1).double() - 0.5)
    grain = torch.from_numpy(m["grain"]).cuda()
    masks = [(1 << (G + j)) | (1 << int(m["nbr"][j])) for j in range(L)]

    def sun(X):
        Y = diag[:, None] * X
        for mask, c in zip(masks, m["coup"]):
            Y.add_(X[st ^ mask], alpha=float(c) / 4)
        Y += torch.einsum("gh,ohs->ogs", grain, X.view(-1, 1 << G, X.shape[1])).reshape(X.shape)
        return Y
    return sun


def _edges(H, x0):
    """The extremal eigenvalues by Lanczos with full reorthogonalisation."""
    D = len(x0)
    steps = min(D, 320)
    V = torch.zeros((steps, D), dtype=torch.float64, device="cuda")
    T = torch.zeros((steps, steps), dtype=torch.float64)
    v = torch.from_numpy(x0).cuda()
    V[0] = v / v.norm()
    for k in range(steps):
        r = H(V[k][:, None])[:, 0]
        T[k, k] = r @ V[k]
        for _ in range(2):
            r = r - V[:k + 1].t() @ (V[:k + 1] @ r)
        beta = float(r.norm())
        if k + 1 == steps or beta < 1e-10:
            T = T[:k + 1, :k + 1]
            break
        T[k, k + 1] = T[k + 1, k] = beta
        V[k + 1] = r / beta
    ev = torch.linalg.eigvalsh(T)
    return float(ev[0]), float(ev[-1])


def exact(case, seed):
    call = case["call"]
    if call == "batch" or (call == "solve" and _dim(case) > 4000) or (call == "kpm" and not case["given"]):
        return None
    m = _model(case, seed)
    H = _exact_apply(case, m)
    a, b = _scale(case, m)
    if call in ("apply", "recurrence", "filter"):
        X = _block(_dim(case), case["s"], case, seed, 1).double().contiguous()
        if call == "apply":
            return (H(X) - b * X) / a
        if call == "recurrence":
            b2, b3 = (_block(_dim(case), case["s"], case, seed, k).double().contiguous() for k in (2, 3))
            return 0.7 * X + 2 * (H(b2) - b * b2) / a - b3
        c = _coefficients(case)
        b1, b2 = torch.zeros_like(X), torch.zeros_like(X)
        for k in range(case["K"], 0, -1):
            b1, b2 = float(c[k]) * X + 2 * (H(b1) - b * b1) / a - b2, b1
        return float(c[0]) * X + (H(b1) - b * b1) / a - b2
    if call == "kpm":
        p = _probes(case, seed).double().contiguous()
        mu = np.zeros(case["N"])
        t0, t1 = p, (H(p) - b * p) / a
        for n in range(case["N"]):
            mu[n] = float((p * t0).sum())
            t0, t1 = t1, 2 * (H(t1) - b * t1) / a - t0
        return mu * (_dim(case) / case["R"])
    if call == "extrema":
        return _edges(H, _start(case, seed))
    # a small solve: the nev eigenvalues nearest the target, from the dense matrix
    ev = torch.linalg.eigvalsh(H(torch.eye(_dim(case), dtype=torch.float64, device="cuda")))
    at = (ev[0] + ev[-1]) / 2 + case["target"] * (ev[-1] - ev[0]) / 2
    near = torch.argsort((ev - at).abs())[:case["nev"]]
    return torch.sort(ev[near])[0].cpu().numpy()
