"""The eigenvector of a projected tridiagonal matrix by inverse iteration
(pf_spectral.cpp), compiled on its own: every vector it accepts has a residual
of a few roundings of the matrix's norm, and what it cannot give that well it
refuses, so that the caller takes the dense solver."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "polfed.jl_b200", "csrc")
EPS = 2.0 ** -52

MAIN = r"""
#include <cstdio>
#include "pf_spectral.h"
int main() {
    int n;
    while (std::scanf("%d", &n) == 1) {
        std::vector<double> d(n), e(n > 1 ? n - 1 : 0), z;
        double lam;
        for (double &v : d) if (std::scanf("%lf", &v) != 1) return 1;
        for (double &v : e) if (std::scanf("%lf", &v) != 1) return 1;
        if (std::scanf("%lf", &lam) != 1) return 1;
        const bool ok = pf::tridiag_vector(d, e, lam, z);
        std::printf("%d", ok ? 1 : 0);
        for (double v : z) std::printf(" %.17g", v);
        std::printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def tridiag_vector(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("tridiag")
    src, exe = tmp / "main.cpp", tmp / "main"
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", CSRC, "-I", "/usr/local/cuda/include", str(src),
                           os.path.join(CSRC, "pf_spectral.cpp"), "-o", str(exe)])

    def run(d, e, lam):
        row = lambda v: " ".join("%.17g" % x for x in v)
        out = subprocess.run([str(exe)], input=f"{len(d)} {row(d)} {row(e)} {lam:.17g}\n", capture_output=True, text=True,
                             check=True).stdout.split()
        return out[0] == "1", np.array([float(x) for x in out[1:]])
    return run


def _matrices():
    rng = np.random.default_rng(3)
    out = {"one": (np.array([2.5]), np.array([])), "two": (np.array([1.0, -1.0]), np.array([0.5]))}
    for k in (7, 40, 130, 400):   # projected spectra of random sparse operators are of this kind
        out[f"random{k}"] = (rng.standard_normal(k), 0.5 + rng.random(k - 1))
    out["wilkinson"] = (np.abs(np.arange(-20, 21)).astype(float), np.ones(40))   # pairs of nearly equal eigenvalues
    out["decoupled"] = (np.arange(12.0), np.r_[np.ones(5), 0.0, np.ones(5)])
    out["graded"] = (10.0 ** -np.arange(20.0), 10.0 ** -(np.arange(19.0) + 0.5))
    return out


@pytest.mark.parametrize("name", list(_matrices()))
def test_residual_is_of_rounding_size(tridiag_vector, name):
    """The bound the code states, 64 eps of the norm, for extremal eigenvalues to
    rounding; one eigenvalue wrong in its 12th digit of the norm is refused or
    still met."""
    d, e = _matrices()[name]
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    nrm = np.abs(T).sum(axis=1).max()
    ev = np.linalg.eigvalsh(T)
    for lam in (ev[0], ev[-1]):
        ok, z = tridiag_vector(d, e, lam)
        assert ok and abs(np.linalg.norm(z) - 1) < 1e-14
        assert np.linalg.norm(T @ z - lam * z) <= 70 * EPS * nrm
        off = lam + 1e-12 * nrm
        ok, z = tridiag_vector(d, e, off)
        assert not ok or np.linalg.norm(T @ z - off * z) <= 70 * EPS * nrm
