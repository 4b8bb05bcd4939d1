"""Which kernels a call runs, and how much device memory it takes.

The kernels are read from the profiler's list of launches, the memory from the
high-water mark of the device's stream-ordered pool, which holds every
workspace of the library's calls."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kernels(torch, call):
    """Names of the kernels that call() launches."""
    from torch.profiler import ProfilerActivity, profile
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    names = {e.name for e in prof.events()}
    if not any("(" in n for n in names):
        pytest.skip("the profiler records no kernels here (another tool holds the device's activity records)")
    assert any("pf::" in n for n in names), names
    return names


def ran(names, kernel):
    return any(n.split("<")[0].split("(")[0].split("::")[-1] == kernel for n in names)


class PoolHigh:
    """Bytes the device's default pool held at most inside the block, above what it held before."""
    USED_CURRENT, USED_HIGH = 7, 8   # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH

    def __enter__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0
        zero = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, self.USED_HIGH, ctypes.byref(zero)) == 0
        self.before = self._get(self.USED_CURRENT)
        return self

    def _get(self, attr):
        v = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, ctypes.byref(v)) == 0
        return v.value

    def __exit__(self, *a):
        self.bytes = self._get(self.USED_HIGH) - self.before


def _block(torch, D, s, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((s, D), generator=g, device="cuda", dtype=torch.float64).to(dtype).t()


def _qsun(pkg, L_loc, L_grain, seed):
    f, n, c, g = pkg.qsun_parameters(L_loc, L_grain, 0.75, rng=np.random.default_rng(seed))
    return pkg.QSunOperator(L_loc, L_grain, 0.9, c, n, f, g)


def _chain(pkg, L, Lup, seed, distance=1):
    rng = np.random.default_rng(seed)
    bonds = pkg.chain_bonds(L, 1) + (pkg.chain_bonds(L, 2) if distance == 2 else [])
    return pkg.SpinChainOperator(L, Lup, bonds, rng.random(len(bonds)) + 0.5, rng.random(len(bonds)), 2 * rng.random(L) - 1)


# ------------------------------------------------------------ moments on chip

def _signs(seed, D, cols):
    """The +-1 probes of a seed: the low bit of two chained splitmix64 finalisers of (row, column)."""
    def mix(z):
        with np.errstate(over="ignore"):
            z = z + np.uint64(0x9E3779B97F4A7C15)
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            return z ^ (z >> np.uint64(31))
    key = (np.arange(cols, dtype=np.uint64)[:, None] << np.uint64(32)) ^ np.arange(D, dtype=np.uint64)[None, :]
    return np.where(mix(np.uint64(seed) ^ mix(key)) & np.uint64(1), 1.0, -1.0)


@pytest.mark.parametrize("R", [1, 64, 301])
@pytest.mark.parametrize("kind", ["qsun", "chain"])
def test_moments_of_many_probes(pkg, cuda, kind, R):
    """Drawn probes against the same probes given, and against the average of
    two halves: the columns that one launch takes do not show.  Sums of D
    products in the same order differ at most in the probes' normalisation, a
    few eps of each moment's bound |v|^2 = 1 (times 2 for the doubling)."""
    torch = cuda
    op = _qsun(pkg, 13, 3, 7) if kind == "qsun" else _chain(pkg, 14, 7, 5)
    D, N, seed = op.dim, 9, 77
    P = torch.from_numpy(_signs(seed, D, R)).cuda().t() / math.sqrt(D)
    drawn = pkg.kpm_moments(op, N, R, 12.0, 0.2, probe_kind="rademacher", seed=seed) / D
    given = pkg.kpm_moments(op, N, R, 12.0, 0.2, probes=P.t().contiguous().t()) / D
    assert np.max(np.abs(drawn - given)) < 1e-13
    if R > 1:
        h = R // 2
        part = [pkg.kpm_moments(op, N, n, 12.0, 0.2, probes=P[:, a:a + n].t().contiguous().t()) / D
                for a, n in ((0, h), (h, R - h))]
        assert np.max(np.abs(drawn - (h * part[0] + (R - h) * part[1]) / R)) < 1e-13


def test_moments_on_chip_hold_a_bounded_workspace(pkg, cuda):
    """512 MB, however many probes there are."""
    op = _qsun(pkg, 13, 3, 7)
    for R in (64, 2000):
        with PoolHigh() as high:
            pkg.kpm_moments(op, 3, R, 12.0, 0.2, seed=3)
        assert high.bytes <= (513 << 20), (R, high.bytes)


def test_solve_stays_within_the_footprint_a_pool_charges(pkg, cuda):
    """A request of few pairs and many probes, whose moments hold the most."""
    op = _qsun(pkg, 13, 3, 7)
    x0 = np.random.default_rng(1).standard_normal((op.dim, 1))
    kw = dict(mapping=pkg.MappingConfig(Emin=-12.0, Emax=12.0), transform=pkg.TransformConfig(order=12),
              dos=pkg.DoSConfig(N=60, R=1200, seed=3))
    with PoolHigh() as high:
        pkg.polfed(op, x0, 1, ("rescaled", 0.1), vecs=False, **kw)
    assert high.bytes <= pkg.SolverPool.footprint(op, 1, ("rescaled", 0.1), 1, **kw), high.bytes


# ------------------------------------------------------------ a solve's flip list

_NEAR_FULL = """
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, {root!r})
import __graft_entry__ as ge
pkg = ge.load_package()
rng = np.random.default_rng(1)
L = 24
bonds = pkg.chain_bonds(L, 1)
op = pkg.SpinChainOperator(L, L // 2, bonds, [1.0] * L, [1.0] * L, 2 * rng.random(L) - 1)
x0 = rng.standard_normal((op.dim, 1))
solve = lambda: pkg.polfed(op, x0, 1, ("rescaled", 0.1), vecs=False, mapping=pkg.MappingConfig(Emin=-30.0, Emax=30.0),
                           transform=pkg.TransformConfig(order=9), dos=pkg.DoSConfig(N=4, R=1, seed=3))
cu, pool, v = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(), ctypes.c_uint64(0)
solve()
torch.cuda.synchronize()
assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
assert cu.cuMemPoolGetAttribute(pool, 8, ctypes.byref(v)) == 0      # the solve's high-water mark, with the list
assert cu.cuMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0
listed = op.dim * (L // 4 + 1) * 16
free = torch.cuda.mem_get_info()[0]
keep = torch.empty(int(free - (v.value - listed // 2)), dtype=torch.uint8, device="cuda")
solve()
print("solved", v.value, listed)
"""


def test_solve_without_room_for_a_flip_list(pkg, cuda):
    """A solve whose flip list (303 MB) would leave too little for its basis runs
    without one.  In a process of its own, which leaves the solve half a list
    less than it took with the list."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _NEAR_FULL.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("solved"), r.stdout + r.stderr


# ------------------------------------------------------------ pinned variants

@pytest.mark.parametrize("kind", ["qsun", "chain"])
def test_pinned_variant_governs_every_later_step(pkg, cuda, kind):
    """Applies, recurrences, final sums, filters and extremal probes of a width
    run the step kernel that the caller pinned for it; results are the same bits."""
    torch = cuda
    mk = (lambda: _qsun(pkg, 8, 3, 2)) if kind == "qsun" else (lambda: _chain(pkg, 12, 6, 3))
    op, ref, s = mk(), mk(), 4
    pkg.set_step_width(op, s, 2)
    pkg.set_step_width(op, 1, 1)
    q, p, x, y, z = (_block(torch, op.dim, s, torch.float64, k) for k in range(5))
    v0 = np.random.default_rng(1).standard_normal(op.dim)
    calls = {"apply": lambda o, out: pkg.apply(o, out, q, 3.0, 0.2),
             "recurrence": lambda o, out: pkg.clenshaw_recurrence(o, out, q, p, 0.7, x, 3.0, 0.2),
             "finalsum": lambda o, out: pkg.clenshaw_finalsum(o, q, p, 0.7, out, x, 3.0, 0.2),
             "filter": lambda o, out: pkg.chebyshev_filter(o, out, q, np.cos(np.arange(20)), 9.0, 0.1)}
    for name, call in calls.items():
        names = kernels(torch, lambda: call(op, y))
        assert ran(names, "k_step"), (name, names)
        for other in ("k_step_cm", "k_res_qsun", "k_res_list", "k_res_pinned", "k_step_chain_list"):
            assert not ran(names, other), (name, other)
        call(ref, z)
        assert torch.equal(y, z), name
    names = kernels(torch, lambda: pkg.lanczos_extrema(op, v0))
    assert ran(names, "k_step") and not ran(names, "k_step_chain_list"), names
    assert pkg.lanczos_extrema(op, v0) == pkg.lanczos_extrema(ref, v0)


def test_autotune_releases_a_pinned_variant(pkg, cuda):
    """A pin holds until the caller has the variant chosen by timing again."""
    torch = cuda
    op, s = _chain(pkg, 12, 6, 3), 4
    X = _block(torch, op.dim, s, torch.float64, 1)
    Y = torch.empty_like(X)
    call = lambda: pkg.chebyshev_filter(op, Y, X, np.cos(np.arange(20)), 9.0, 0.1)
    pkg.set_step_width(op, s, 2)
    assert ran(kernels(torch, call), "k_step")
    pkg.autotune(op, s)
    names = kernels(torch, call)
    assert ran(names, "k_res_pinned") and not ran(names, "k_step"), names


# ------------------------------------------------------------ sparse matrices on chip

def _band(pkg, D, k, width, seed):
    rng = np.random.default_rng(seed)
    idx = (np.repeat(np.arange(D), k) + rng.integers(-width, width + 1, size=D * k)) % D
    return pkg.SparseOperator((np.arange(D + 1) * k, idx, rng.standard_normal(D * k)))


@pytest.mark.parametrize("D,k,width,s,R", [(12000, 8, 40, 4, 64), (400, 7, 200, 8, 64), (6435, 30, 3217, 8, 64),
                                           (50000, 15, 25000, 2, 64)])
def test_sparse_matrices_run_on_chip_where_their_columns_are_near(pkg, cuda, D, k, width, s, R):
    """Rows whose entries lie in the same CTA, or a matrix that fits a few, run on
    chip; rows with 30 and 15 entries anywhere do not: a remote read for each
    made them up to six times slower than the step kernels."""
    torch = cuda
    op = _band(pkg, D, k, width, 3)
    X = _block(torch, D, s, torch.float64, 1)
    Y = torch.empty_like(X)
    c = np.cos(np.arange(40))
    near = 2 * width < D // 16 or D <= 1000
    for names in (kernels(torch, lambda: pkg.chebyshev_filter(op, Y, X, c, 30.0, 0.1)),
                  kernels(torch, lambda: pkg.kpm_moments(op, 40, R, 30.0, 0.1, seed=1))):
        assert ran(names, "k_res_list") == near and ran(names, "k_step") != near, names


# ------------------------------------------------------------ one step on column-major blocks

def test_steps_are_staged_where_that_is_faster(pkg, cuda):
    """Column-major steps on either side of the rule's lines: a wide apply of a
    4-site grain (2.3 times slower column-major), a matrix with 15 entries a row
    anywhere, the same sizes with a narrow block, a smaller grain or near columns."""
    torch = cuda
    rng = np.random.default_rng(5)
    far = pkg.SparseOperator((np.arange(50001) * 15, rng.integers(0, 50000, size=50000 * 15), rng.standard_normal(50000 * 15)))
    idx = (np.repeat(np.arange(50000), 8) + rng.integers(-300, 301, size=400000)) % 50000
    near = pkg.SparseOperator((np.arange(50001) * 8, np.sort(idx.reshape(-1, 8), axis=1).ravel(), rng.standard_normal(400000)))
    cases = [(_qsun(pkg, 14, 4, 1), 16, torch.float32, False), (_qsun(pkg, 14, 4, 1), 4, torch.float32, True),
             (_qsun(pkg, 15, 3, 1), 8, torch.float64, True), (far, 12, torch.float64, False), (far, 2, torch.float64, True),
             (near, 8, torch.float64, True), (_chain(pkg, 16, 8, 1), 8, torch.float64, True),
             (_chain(pkg, 20, 10, 1), 8, torch.float64, False)]
    for op, s, dtype, direct in cases:
        X = _block(torch, op.dim, s, dtype, 1)
        Y = torch.empty_like(X)
        names = kernels(torch, lambda: pkg.apply(op, Y, X, 3.0, 0.1))
        assert ran(names, "k_step_cm") == direct and ran(names, "k_step") != direct, (op.dim, s, names)


# ------------------------------------------------------------ every on-chip filter form, by name

def _xxz_csr(pkg, L, k):
    """The matrix of an XXZ chain's sector, rows cut to at most k entries (in storage order)."""
    st = np.array([s for s in range(1 << L) if bin(s).count("1") == L // 2])
    rows, cols = [np.arange(len(st))], [np.arange(len(st))]
    for a in range(L):
        m = (1 << a) | (1 << (a + 1) % L)
        on = np.nonzero((st & m) * (st & m ^ m))[0]
        rows.append(on)
        cols.append(np.searchsorted(st, st[on] ^ m))
    r, c = np.concatenate(rows), np.concatenate(cols)
    o = np.lexsort((c, r))
    r, c = r[o], c[o]
    keep = np.arange(len(r)) - np.searchsorted(r, r) < k
    r, c = r[keep], c[keep]
    return pkg.SparseOperator((np.searchsorted(r, np.arange(len(st) + 1)), c, np.random.default_rng(L).standard_normal(len(c))))


# (operator, columns, dtype, the kernel's name with its first template arguments): the forms' widths, a column count
# that the width does not divide, one CTA and several, rows of more entries or more rows a CTA than a thread's registers take
FORMS = {
    "pinned_1": (lambda p: _chain(p, 14, 7, 1), 1, "fp64", "k_res_pinned<double, 1,"),
    "pinned_2": (lambda p: _chain(p, 15, 7, 1), 41, "fp64", "k_res_pinned<double, 2,"),
    "pinned_rotating": (lambda p: _chain(p, 16, 8, 1), 7, "fp64", "k_res_pinned<double, 1,"),
    "pinned_fp32_2": (lambda p: _chain(p, 14, 7, 1), 41, "fp32", "k_res_pinned<float, 2,"),
    "pinned_fp32_4": (lambda p: _chain(p, 15, 7, 1), 41, "fp32", "k_res_pinned<float, 4,"),
    "list_28_bonds": (lambda p: _chain(p, 14, 7, 2, 2), 1, "fp64", "k_res_list<double, 1, false, false>"),
    "list_28_bonds_wide": (lambda p: _chain(p, 14, 7, 2, 2), 21, "fp64", "k_res_list<double, "),
    "list_28_bonds_fp32": (lambda p: _chain(p, 14, 7, 2, 2), 43, "fp32", "k_res_list<float, "),
    "csr_1": (lambda p: _xxz_csr(p, 14, 64), 3, "fp64", "k_res_list<double, 1, true, false>"),
    "csr_2": (lambda p: _xxz_csr(p, 13, 9), 41, "fp64", "k_res_list<double, 2, true, false>"),
    "csr_fp32_4": (lambda p: _xxz_csr(p, 14, 64), 43, "fp32", "k_res_list<float, 4, true, false>"),
    "csr_one_cta": (lambda p: _xxz_csr(p, 10, 64), 7, "fp64", "k_res_list<double, 1, true, false>"),
    "qsun_one_cta": (lambda p: _qsun(p, 8, 3, 1), 5, "fp64", "k_res_qsun<double, 3, false>"),
    "qsun_rotating": (lambda p: _qsun(p, 13, 3, 1), 9, "fp64", "k_res_qsun<double, 3, false>"),
    "qsun_grain_4": (lambda p: _qsun(p, 12, 4, 1), 8, "fp64", "k_res_qsun<double, 4, false>"),
    "qsun_fp32": (lambda p: _qsun(p, 13, 2, 1), 9, "fp32", "k_res_qsun<float, 2, false>"),
}


@pytest.mark.parametrize("name", list(FORMS))
def test_filter_on_chip_equals_the_steps(pkg, cuda, name):
    """The form runs, and gives the pinned step kernels' bits."""
    torch = cuda
    make, s, dtype, kernel = FORMS[name]
    op, ref = make(pkg), make(pkg)
    pkg.set_step_width(ref, s, 1, dtype)
    X = _block(torch, op.dim, s, torch.float64 if dtype == "fp64" else torch.float32, 4)
    Y, Z = torch.full_like(X, math.nan), torch.empty_like(X)
    for K in (41, 3):
        c = np.cos(np.arange(K + 1) * 0.6) / (K + 1)
        names = kernels(torch, lambda: pkg.chebyshev_filter(op, Y, X, c, 21.0, -0.3))
        assert any(kernel in n for n in names), names
        assert ran(kernels(torch, lambda: pkg.chebyshev_filter(ref, Z, X, c, 21.0, -0.3)), "k_step")
        assert torch.equal(Y, Z), (K, float((Y - Z).abs().max()))


# ------------------------------------------------------------ moments by steps

@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["qsun_small", "qsun_large", "csr"])
def test_moments_by_steps(pkg, cuda, kind, dtype):
    """The fused-dots step of operators no cluster holds (or too small for one):
    against the recurrence built from single steps (2 D eps of |v|^2, D <= 2^18:
    1.2e-10), and the same bits with and without the steps' launch overlap."""
    torch = cuda
    rng = np.random.default_rng(2)
    op = {"qsun_small": lambda: _qsun(pkg, 4, 1, 1), "qsun_large": lambda: _qsun(pkg, 16, 2, 1),
          "csr": lambda: pkg.SparseOperator((np.arange(901) * 70, rng.integers(0, 900, size=63000), rng.standard_normal(63000) / 8))}[kind]()
    D, R, N, a, b = op.dim, 11, 14, 30.0, 0.1
    P = _block(torch, D, R, torch.float64 if dtype == "fp64" else torch.float32, 3) / math.sqrt(D)
    P = P.t().contiguous().t()
    call = lambda: pkg.kpm_moments(op, N, R, a, b, probes=P)
    if not (kind == "qsun_large" and dtype == "fp32"):
        names = kernels(torch, call)
        assert ran(names, "k_step") and not ran(names, "k_res_qsun") and not ran(names, "k_res_list"), names
    got = call()
    try:
        pkg.set_launch_overlap(False)
        assert np.array_equal(got, call())
    finally:
        pkg.set_launch_overlap(True)
    dot = lambda x, y: float((x.double() * y.double()).sum())
    prev, cur = P, pkg.apply(op, torch.empty_like(P), P, a, b)
    m0, m1 = dot(prev, prev), dot(cur, prev)
    want, zero = [m0, m1], torch.zeros_like(P)
    for _ in range(N // 2):
        want.append(2 * dot(cur, cur) - m0)
        nxt = pkg.clenshaw_recurrence(op, torch.empty_like(P), cur, prev, 0.0, zero, a, b)
        want.append(2 * dot(nxt, cur) - m1)
        prev, cur = cur, nxt
    assert np.max(np.abs(got - np.array(want[:N]) * D / R)) <= 4 * 1.2e-10 * m0 * D / R


# ------------------------------------------------------------ the start block

def _start(kind, D, s, rng):
    x = rng.standard_normal((D, s))
    if kind == "near":            # the last column 1e-5 from the first: inside what CholQR2 takes
        x[:, -1] = x[:, 0] + 1e-5 * x[:, -1]
    elif kind == "dependent":     # beyond it: the Householder form decides
        x[:, -1] = x[:, 0] + 1e-9 * x[:, -1]
    elif kind == "scaled":
        x *= 10.0 ** rng.integers(-6, 7, size=s)
    elif kind == "tiny":
        x *= 1e-20
    elif kind == "orthonormal":
        x = np.linalg.qr(x)[0]
    return x


@pytest.mark.parametrize("s", [1, 5])
@pytest.mark.parametrize("kind", ["plain", "near", "dependent", "scaled", "tiny", "orthonormal"])
def test_start_block_spans_what_it_is_given(pkg, cuda, kind, s):
    """Eigenvalues from a start block, host or device, are those from numpy's
    orthonormal factor of it: the block's span is kept, whichever form
    orthonormalises it."""
    torch = cuda
    op = _chain(pkg, 10, 5, 3)
    x = _start(kind, op.dim, s, np.random.default_rng(6))
    q = np.linalg.qr(x)[0]
    kw = dict(fact=pkg.FactorizationConfig(tol=1e-13, eigentol=1e-10), dos=pkg.DoSConfig(seed=1), vecs=False)
    want = np.asarray(pkg.polfed(op, q if s > 1 else q[:, 0], 6, ("rescaled", 0.4), **kw)[0])
    for start in (x, torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t()):
        got = np.asarray(pkg.polfed(op, start if s > 1 else start[:, 0], 6, ("rescaled", 0.4), **kw)[0])
        assert len(got) == len(want) >= 6 and np.max(np.abs(got - want)) < 1e-9


def test_start_block_refusals(pkg, cuda):
    """Entries that are not finite and a zero vector are refused, a zero column is replaced."""
    from polfed_b200 import _lib
    op = _chain(pkg, 10, 5, 3)
    rng = np.random.default_rng(7)
    kw = dict(dos=pkg.DoSConfig(seed=1), vecs=False)
    for s in (1, 4):
        for bad in (math.nan, math.inf):
            x = rng.standard_normal((op.dim, s))
            x[17, -1] = bad
            with pytest.raises((_lib.PolfedArgumentError, ValueError)):
                pkg.polfed(op, x if s > 1 else x[:, 0], 4, ("rescaled", 0.4), **kw)
    with pytest.raises((_lib.PolfedArgumentError, ValueError)):
        pkg.polfed(op, np.zeros(op.dim), 4, ("rescaled", 0.4), **kw)
    x = rng.standard_normal((op.dim, 3))
    x[:, 1] = 0.0
    pkg.polfed(op, x, 4, ("rescaled", 0.4), **kw)
