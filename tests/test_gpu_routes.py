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
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    names = {e.name for e in prof.events()}
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
