"""Listed chain steps (a chain's flips ranked once per call) against the steps
that rank their own: a filter must equal the filter of a pinned step variant
bit for bit, moments the recurrence built from single steps to the rounding of
their dots, extremal probes the dense spectrum."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(pkg, L, Lup, seed, distance=1, boundary="periodic"):
    rng = np.random.default_rng(seed)
    bonds = pkg.chain_bonds(L, 1, boundary) + (pkg.chain_bonds(L, 2, boundary) if distance == 2 else [])
    return pkg.SpinChainOperator(L, Lup, bonds, rng.random(len(bonds)) + 0.5, rng.random(len(bonds)), 2 * rng.random(L) - 1)


# dimensions no cluster holds a column of, rows of every number of flips modulo the list's chunks, 32 and more bonds
OPS = {
    "L19": lambda p: _chain(p, 19, 9, 1),
    "L19_open": lambda p: _chain(p, 19, 9, 2, boundary="open"),
    "L19_j1j2": lambda p: _chain(p, 19, 9, 3, distance=2),
    "L17_full": lambda p: _chain(p, 17, -1, 4),
    "L30_4_j1j2": lambda p: _chain(p, 30, 5, 5, distance=2),
}


@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
@pytest.mark.parametrize("name", list(OPS))
def test_filter_equals_the_ranking_steps(pkg, cuda, name, dtype):
    torch = cuda
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    op, ref = OPS[name](pkg), OPS[name](pkg)
    for s in (1, 2, 3, 4, 6, 8, 16):
        pkg.set_step_width(ref, s, 1, dtype)
        g = torch.Generator(device="cuda").manual_seed(s)
        X = torch.randn((s, op.dim), generator=g, device="cuda", dtype=torch.float64).to(tdt).t()
        got, want = torch.full_like(X, math.nan), torch.empty_like(X)
        for K in (8, 11):
            c = np.cos(np.arange(K + 1) * 0.9) / (K + 1)
            pkg.chebyshev_filter(op, got, X, c, 11.0, -0.2)
            pkg.chebyshev_filter(ref, want, X, c, 11.0, -0.2)
            assert torch.equal(got, want), (s, K)


@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
def test_moments_match_single_steps(pkg, cuda, dtype):
    """Sums of D products added in another order: 2 D eps = 4e-11 of |v|^2."""
    torch = cuda
    op = OPS["L19_j1j2"](pkg)
    D, R, N, a, b = op.dim, 7, 20, 25.0, 0.3
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(3)
    P = (torch.randn((R, D), generator=g, device="cuda", dtype=torch.float64) / math.sqrt(D)).to(tdt).t()
    got = pkg.kpm_moments(op, N, R, a, b, probes=P)
    dot = lambda x, y: float((x.double() * y.double()).sum())
    prev, cur = P, pkg.apply(op, torch.empty_like(P), P, a, b)
    m0, m1 = dot(prev, prev), dot(cur, prev)
    want, zero = [m0, m1], torch.zeros_like(P)
    for _ in range(N // 2):
        want.append(2 * dot(cur, cur) - m0)
        nxt = pkg.clenshaw_recurrence(op, torch.empty_like(P), cur, prev, 0.0, zero, a, b)
        want.append(2 * dot(nxt, cur) - m1)
        prev, cur = cur, nxt
    assert np.max(np.abs(got - np.array(want[:N]) * D / R)) <= 4 * 4e-11 * m0 * D / R


def test_extrema_match_the_dense_spectrum(pkg, orc, cuda):
    """Probes of a chain with 20 listed bonds a row at most and of one with 60."""
    for L, Lup, distance in ((10, 5, 2), (30, 2, 2)):
        op = _chain(pkg, L, Lup, 7, distance=distance)
        H = orc.spin_chain_matrix(L, Lup, op.bonds, op.couplings, op.anisotropies, op.fields)
        ev = np.linalg.eigvalsh(H.toarray())
        lo, hi = pkg.lanczos_extrema(op, np.random.default_rng(1).random(op.dim))
        assert abs(lo - ev[0]) < 1e-9 and abs(hi - ev[-1]) < 1e-9
