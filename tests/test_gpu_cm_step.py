"""Steps straight on column-major blocks (apply, recurrence, final sum) against
a one-column call per column, which runs the step kernels on the column itself:
the same bits, for every operator kind, padded leading dimensions, outputs in
place of an input, and blocks on either side of the staging rule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ops(pkg):
    rng = np.random.default_rng(3)
    f, n, c, g = pkg.qsun_parameters(7, 3, 0.75, rng=rng)
    f2, n2, c2, g2 = pkg.qsun_parameters(14, 2, 0.75, rng=rng)
    b = pkg.chain_bonds(13, 1) + pkg.chain_bonds(13, 2)
    chain = lambda L, Lup, bonds: pkg.SpinChainOperator(L, Lup, bonds, rng.random(len(bonds)), rng.random(len(bonds)), rng.random(L))
    k = rng.integers(0, 9, size=501)
    ptr = np.concatenate([[0], np.cumsum(k)])
    return {"qsun_7_3": pkg.QSunOperator(7, 3, 0.9, c, n, f, g), "qsun_14_2": pkg.QSunOperator(14, 2, 0.9, c2, n2, f2, g2),
            "chain_13": chain(13, 6, b), "chain_full": chain(9, -1, pkg.chain_bonds(9, 1)), "chain_19": chain(19, 9, pkg.chain_bonds(19, 1)),
            "csr": pkg.SparseOperator((ptr, rng.integers(0, 501, size=ptr[-1]), rng.standard_normal(ptr[-1])))}


@pytest.fixture(scope="module")
def ops(pkg, cuda):
    return _ops(pkg)


def _padded(torch, D, s, pad, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((s, D + pad), generator=g, device="cuda", dtype=torch.float64).to(dtype).t()[:D]


@pytest.mark.parametrize("name", ["qsun_7_3", "qsun_14_2", "chain_13", "chain_full", "chain_19", "csr"])
@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
def test_blocks_equal_their_columns(pkg, cuda, ops, name, dtype):
    torch, op = cuda, ops[name]
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    for s in (2, 3, 4, 5, 9, 16):
        for pad in (0, 3):
            q, p, x, out = (_padded(torch, op.dim, s, pad, tdt, k) for k in range(4))
            pkg.apply(op, out, q, 3.0, 0.2)
            for c in range(s):
                y = torch.empty_like(q[:, c])
                pkg.apply(op, y, q[:, c].clone(), 3.0, 0.2)
                assert torch.equal(out[:, c], y), (s, pad, c)
            for call in ("recurrence", "finalsum"):
                cols = []
                for c in range(s):
                    y = torch.empty_like(q[:, c])
                    a = [t[:, c].clone() for t in (q, p, x)]
                    if call == "recurrence":
                        pkg.clenshaw_recurrence(op, y, a[0], a[1], 0.7, a[2], 3.0, 0.2)
                    else:
                        pkg.clenshaw_finalsum(op, a[0], a[1], 0.7, y, a[2], 3.0, 0.2)
                    cols.append(y)
                want = torch.stack(cols).t()
                for target in ("fresh", "p", "x", "q"):
                    b = {"q": q, "p": p, "x": x}
                    b = {k: _padded(torch, op.dim, s, pad, tdt, 9).copy_(v) for k, v in b.items()}
                    o = _padded(torch, op.dim, s, pad, tdt, 8) if target == "fresh" else b[target]
                    if call == "recurrence":
                        pkg.clenshaw_recurrence(op, o, b["q"], b["p"], 0.7, b["x"], 3.0, 0.2)
                    else:
                        pkg.clenshaw_finalsum(op, b["q"], b["p"], 0.7, o, b["x"], 3.0, 0.2)
                    assert torch.equal(o, want), (s, pad, call, target)


def test_apply_in_place(pkg, cuda, ops):
    torch, op = cuda, ops["qsun_7_3"]
    X = _padded(torch, op.dim, 4, 0, torch.float64, 1)
    want = torch.empty_like(X)
    pkg.apply(op, want, X, 2.0, 0.1)
    pkg.apply(op, X, X, 2.0, 0.1)
    assert torch.equal(X, want)


@pytest.mark.parametrize("kind,s", [("chain", 65535), ("chain", 70000), ("qsun", 262140), ("qsun", 300001)])
def test_more_columns_than_a_launch_has_column_blocks(pkg, cuda, kind, s):
    """Very wide blocks of a handful of states: a chain with one state, 65536
    and more columns of one thread each; a Quantum Sun with four, 262144 and more
    of four columns a thread.  Against two calls of half the columns."""
    torch = cuda
    rng = np.random.default_rng(8)
    if kind == "chain":
        op = pkg.SpinChainOperator(5, 0, pkg.chain_bonds(5, 1), rng.random(5), rng.random(5), rng.random(5))
    else:
        f, n, c, g = pkg.qsun_parameters(1, 1, 0.75, rng=rng)
        op = pkg.QSunOperator(1, 1, 0.9, c, n, f, g)
    q, p, x = (_padded(torch, op.dim, s, 0, torch.float64, k) for k in range(3))
    for call in ("apply", "recurrence"):
        def run(c0, c1):
            out = torch.empty_like(q[:, c0:c1].t().contiguous().t())
            a = [t[:, c0:c1] for t in (q, p, x)]
            if call == "apply":
                return pkg.apply(op, out, a[0], 3.0, 0.2)
            return pkg.clenshaw_recurrence(op, out, a[0], a[1], 0.7, a[2], 3.0, 0.2)
        h = s // 2
        assert torch.equal(run(0, s), torch.cat([run(0, h), run(h, s)], dim=1))
