"""Filters and moments that run whole on chip against the step kernels.

Operators small enough for a thread-block cluster to hold a column run a
filter as one launch (and the moments as another).  Its rows are summed in the
step kernels' order with the same rounded operations, so a filter must equal
the step-by-step filter (a pinned step variant) bit for bit, at every split of
the rows over CTAs.  Moments add each probe's dots in another order: two sums
of D products of the same vectors differ by at most 2 D eps times the sum of
the absolute products, here 2 * 2^16 * 2.2e-16 = 3e-11 of |v|^2.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _block(torch, D, s, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((s, D), generator=g, device="cuda", dtype=torch.float64).to(dtype).t()


def _qsun(pkg, L_loc, L_grain, seed):
    f, n, c, g = pkg.qsun_parameters(L_loc, L_grain, 0.75, rng=np.random.default_rng(seed))
    return pkg.QSunOperator(L_loc, L_grain, 0.9, c, n, f, g)


def _chain(pkg, L, Lup, seed, distance=1, uniform=True, boundary="periodic"):
    rng = np.random.default_rng(seed)
    bonds = pkg.chain_bonds(L, 1, boundary) + (pkg.chain_bonds(L, 2, boundary) if distance == 2 else [])
    J = np.ones(len(bonds)) if uniform else rng.random(len(bonds)) + 0.5
    return pkg.SpinChainOperator(L, Lup, bonds, J, rng.random(len(bonds)), 2 * rng.random(L) - 1)


def _csr(pkg, D, longest, seed):
    """Rows of 0 .. longest entries in arbitrary order (one row full, one empty)."""
    rng = np.random.default_rng(seed)
    n = rng.integers(0, longest + 1, size=D)
    n[0], n[-1] = longest, 0
    ptr = np.concatenate([[0], np.cumsum(n)])
    return pkg.SparseOperator((ptr, rng.integers(0, D, size=ptr[-1]), rng.standard_normal(ptr[-1])))


# (operator, columns): every grain size, one CTA to sixteen per column, ragged last CTAs and warps, the largest and
# smallest dimensions that fit, rows as long as the lists take and one entry longer (which run step by step)
CASES = {
    "qsun_4_1": (lambda p: _qsun(p, 4, 1, 1), 3),
    "qsun_5_1": (lambda p: _qsun(p, 5, 1, 2), 2),
    "qsun_12_1": (lambda p: _qsun(p, 12, 1, 3), 8),
    "qsun_9_2": (lambda p: _qsun(p, 9, 2, 4), 5),
    "qsun_8_3": (lambda p: _qsun(p, 8, 3, 5), 1),
    "qsun_11_3": (lambda p: _qsun(p, 11, 3, 6), 8),
    "qsun_13_3": (lambda p: _qsun(p, 13, 3, 7), 1),
    "qsun_14_3": (lambda p: _qsun(p, 14, 3, 8), 3),
    "qsun_9_4": (lambda p: _qsun(p, 9, 4, 9), 4),
    "qsun_12_4": (lambda p: _qsun(p, 12, 4, 10), 2),
    "chain_3_1": (lambda p: _chain(p, 3, 1, 11), 1),
    "chain_13_4": (lambda p: _chain(p, 13, 4, 12, uniform=False), 5),
    "chain_14_7": (lambda p: _chain(p, 14, 7, 13), 1),
    "chain_15_7_open": (lambda p: _chain(p, 15, 7, 14, boundary="open"), 3),
    "chain_16_8_j1j2": (lambda p: _chain(p, 16, 8, 15, distance=2), 8),
    "chain_18_9": (lambda p: _chain(p, 18, 9, 16), 2),
    "chain_full_10": (lambda p: _chain(p, 10, -1, 17, uniform=False), 7),
    "chain_none": (lambda p: p.SpinChainOperator(8, 4, [], [], [], np.linspace(-1, 1, 8)), 2),
    "csr_1": (lambda p: _csr(p, 1, 1, 18), 1),
    "csr_33": (lambda p: _csr(p, 33, 9, 19), 2),
    "csr_2047": (lambda p: _csr(p, 2047, 8, 20), 4),
    "csr_9001": (lambda p: _csr(p, 9001, 17, 21), 3),
    "csr_64": (lambda p: _csr(p, 700, 64, 22), 2),
    "csr_65": (lambda p: _csr(p, 700, 65, 23), 2),
}


@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
@pytest.mark.parametrize("name", list(CASES))
def test_filter_equals_the_step_kernels(pkg, cuda, name, dtype):
    torch = cuda
    make, s = CASES[name]
    op, ref = make(pkg), make(pkg)
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    pkg.set_step_width(ref, s, 1, dtype)   # a pinned variant: step by step
    X = _block(torch, op.dim, s, tdt, 5)
    for K in (0, 1, 2, 3, 30):
        c = np.cos(np.arange(K + 1) * 1.1) / (K + 1)
        got, want = torch.full_like(X, math.nan), torch.empty_like(X)
        pkg.chebyshev_filter(op, got, X, c, 9.0, 0.3)
        pkg.chebyshev_filter(ref, want, X, c, 9.0, 0.3)
        assert torch.equal(got, want), (K, float((got - want).abs().max()))


@pytest.mark.parametrize("L_loc,L_grain,s,K", [(13, 3, 8, 203), (13, 3, 17, 120), (14, 3, 8, 64), (13, 2, 16, 301), (12, 4, 9, 150)])
@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
def test_filter_of_more_columns_than_clusters(pkg, cuda, L_loc, L_grain, s, K, dtype):
    """Large Quantum Sun columns run in several launches, each column resting in
    some of them; orders that the launches do not divide."""
    torch = cuda
    op, ref = _qsun(pkg, L_loc, L_grain, 40), _qsun(pkg, L_loc, L_grain, 40)
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    pkg.set_step_width(ref, s, 1, dtype)
    X = _block(torch, op.dim, s, tdt, 6)
    c = np.cos(np.arange(K + 1) * 0.8) / (K + 1)
    got, want = torch.full_like(X, math.nan), torch.empty_like(X)
    pkg.chebyshev_filter(op, got, X, c, 9.0, 0.3)
    pkg.chebyshev_filter(ref, want, X, c, 9.0, 0.3)
    assert torch.equal(got, want), float((got - want).abs().max())


@pytest.mark.parametrize("L,s,K", [(16, 8, 200), (16, 15, 131), (16, 9, 0), (12, 3, 64), (14, 40, 90), (17, 3, 50)])
@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
def test_chain_filter_with_a_row_per_thread(pkg, cuda, L, s, K, dtype):
    """Lists in registers, in one launch and in rotating ones."""
    torch = cuda
    op, ref = _chain(pkg, L, L // 2, 41, uniform=False), _chain(pkg, L, L // 2, 41, uniform=False)
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    pkg.set_step_width(ref, s, 1, dtype)
    X = _block(torch, op.dim, s, tdt, 6)
    c = np.cos(np.arange(K + 1) * 0.8) / (K + 1)
    got, want = torch.full_like(X, math.nan), torch.empty_like(X)
    pkg.chebyshev_filter(op, got, X, c, 11.0, 0.3)
    pkg.chebyshev_filter(ref, want, X, c, 11.0, 0.3)
    assert torch.equal(got, want), float((got - want).abs().max())


@pytest.mark.parametrize("kind", ["chain", "qsun"])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_filter_output_over_its_input(pkg, cuda, kind, shift):
    """Y over X: the same block, one starting a column later, one two rows later."""
    torch = cuda
    op = _chain(pkg, 12, 6, 41, uniform=False) if kind == "chain" else _qsun(pkg, 8, 3, 5)
    D, s, K = op.dim, 12, 40
    X = _block(torch, D, s, torch.float64, 9)
    c = np.cos(np.arange(K + 1) * 0.8) / (K + 1)
    want = torch.empty_like(X)
    pkg.chebyshev_filter(op, want, X, c, 11.0, 0.3)
    at = (0, D, 2)[shift]
    base = torch.zeros((s + 1) * D, dtype=torch.float64, device=X.device)
    Xv = base[: s * D].view(s, D).t()
    Yv = base[at : at + s * D].view(s, D).t()
    Xv.copy_(X)
    pkg.chebyshev_filter(op, Yv, Xv, c, 11.0, 0.3)
    assert torch.equal(Yv, want)


def test_filter_takes_strided_blocks(pkg, cuda):
    """Column-major blocks with padded columns, in place."""
    torch = cuda
    op = _chain(pkg, 14, 7, 30)
    D = op.dim
    c = np.cos(np.arange(12) * 0.7)
    big = torch.randn((4, D + 13), device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(1))
    X = big.t()[:D]
    want = torch.empty((4, D), device="cuda", dtype=torch.float64).t()
    pkg.chebyshev_filter(op, want, X.t().contiguous().t(), c, 9.0, 0.0)
    pad = big[:, D:].clone()
    pkg.chebyshev_filter(op, X, X, c, 9.0, 0.0)
    assert torch.equal(X, want) and torch.equal(big[:, D:], pad)


@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
@pytest.mark.parametrize("name", ["qsun_5_1", "qsun_9_2", "qsun_13_3", "qsun_9_4", "chain_3_1", "chain_13_4",
                                  "chain_16_8_j1j2", "chain_full_10", "csr_33", "csr_9001"])
def test_moments_match_the_recurrence(pkg, orc, cuda, name, dtype):
    """Moments of given probes against the doubled recurrence built from
    single applies (the step kernels) with FP64 dots; drawn probes twice the
    same."""
    torch = cuda
    op = CASES[name][0](pkg)
    D, R, N = op.dim, 5, 12
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    a, b = 12.0, 0.2
    P = _block(torch, D, R, tdt, 9) / math.sqrt(D)
    P = P.t().contiguous().t()
    got = pkg.kpm_moments(op, N, R, a, b, probes=P)
    v0 = P
    v1 = pkg.apply(op, torch.empty_like(P), P, a, b)
    dot = lambda x, y: float((x.double() * y.double()).sum())
    want = [dot(v0, v0), dot(v1, v0)]
    m0, m1 = want
    prev, cur = v0, v1
    zero = torch.zeros_like(P)
    for _ in range(N // 2):
        want.append(2 * dot(cur, cur) - m0)
        nxt = pkg.clenshaw_recurrence(op, torch.empty_like(P), cur, prev, 0.0, zero, a, b)
        want.append(2 * dot(nxt, cur) - m1)
        prev, cur = cur, nxt
    want = np.array(want[:N]) * D / R
    assert np.max(np.abs(got - want)) <= 4 * 3e-11 * m0 * D / R
    r1 = pkg.kpm_moments(op, N, R, a, b, seed=3, dtype=dtype)
    r2 = pkg.kpm_moments(op, N, R, a, b, seed=3, dtype=dtype)
    assert np.array_equal(r1, r2) and abs(r1[0] / D - 1) < (1e-12 if dtype == "fp64" else 1e-6)
