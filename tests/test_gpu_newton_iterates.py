"""The iterates of the batch Newton solve, bit for bit: against recorded ones
(iteration counts, statuses and a checksum of the solutions, of the solver that
ran each solve to its end in one loop) up to three components, against
cl_eq_solve_noalloc, which runs the in-step loops, at one to five, and a batch
whose warm misses fill the queue kernel's list (more than 8192) against the
same systems in batches short enough for one solve per warp.  The inputs are
exact multiples of powers of two, the same on every machine."""
import ctypes
import zlib

import numpy as np
import pytest

from test_gpu_newton_batch import TABLEAUX

pytestmark = pytest.mark.gpu

N = 20000
# (tableau, start): sum of iterations, the same weighted by row % 97, statuses, CRC-32 of the solutions
RECORDED = {
    ("one", "cold"): (93084, 4464840, [20000, 0, 0], 0x875a26ea),
    ("one", "given"): (165217, 7930102, [9111, 10889, 0], 0xd97507c3),
    ("carbonate", "cold"): (238778, 11452825, [20000, 0, 0], 0x36ba78f5),
    ("carbonate", "given"): (320415, 15331740, [3175, 16825, 0], 0x945aa8fb),
    ("three", "cold"): (2029756, 97316230, [10654, 0, 9346], 0x8dd08a56),
    ("three", "given"): (2117135, 101485749, [58, 10635, 9307], 0xc205f1e7),
    ("cube", "cold"): (84773, 4065992, [20000, 0, 0], 0x809645f5),
    ("cube", "given"): (189230, 9078462, [2861, 17139, 0], 0x2423a35b),
    ("half", "cold"): (60014, 2878438, [20000, 0, 0], 0xd58df293),
    ("half", "given"): (161750, 7762768, [5508, 14492, 0], 0x28da6dda),
}


def _problem(pkg, wl, name):
    if name in TABLEAUX:
        S, logk = np.array(TABLEAUX[name][0], float), np.array(TABLEAUX[name][1], float)
        cs = list(range(S.shape[1]))
    else:
        S, logk, cs = wl.tableau({"four": 4, "five": 5}[name], 9, seed=4)
    nc = S.shape[1]
    sys_ = pkg.EqSystem()
    pkg.set_eq_system(sys_, S, logk, cs, max_iter=200, tol=1e-10, warm_iter=6)
    k = np.arange(N * nc, dtype=np.uint64).reshape(N, nc)
    T = ((k * np.uint64(2654435761) % np.uint64(1 << 20)) + np.uint64(1)).astype(float) * 2.0 ** -30
    x0 = -((k * np.uint64(40503) % np.uint64(512)) + np.uint64(64)).astype(float) / 64
    return sys_, T, wl.cold_species(S, T, cs), x0


@pytest.mark.parametrize("start", ["cold", "given"])
@pytest.mark.parametrize("name", ["one", "carbonate", "three", "cube", "half", "four", "five"])
def test_iterates(gpu_lib, pkg, wl, name, start):
    import torch
    sys_, T, cold, x0 = _problem(pkg, wl, name)
    mode = pkg.EQ_START_COLD if start == "cold" else pkg.EQ_START_GIVEN
    eq = pkg.EqSolver(sys_)
    x, it, st = eq.solve(T, cold, x0=x0, start=mode)
    if start == "given":
        assert np.count_nonzero(st > 0) > 8192          # the cold phase took its systems from the list
    # the same systems one solve per warp
    parts = [eq.solve(T[a:a + 8192], cold[a:a + 8192], x0=x0[a:a + 8192], start=mode) for a in range(0, N, 8192)]
    for got, want in zip((np.concatenate(p) for p in zip(*parts)), (x, it, st)):
        np.testing.assert_array_equal(got, want)
    # and in the loops of the step, one thread each
    vp = ctypes.c_void_p
    gpu_lib.cl_eq_solve_noalloc.restype = ctypes.c_int
    gpu_lib.cl_eq_solve_noalloc.argtypes = [vp] * 6 + [ctypes.c_int64, ctypes.c_int32, vp]
    d = [torch.tensor(a, device="cuda") for a in (T, cold, x0, np.zeros(N, np.int32), np.zeros(N, np.uint8))]
    torch.cuda.synchronize()
    assert gpu_lib.cl_eq_solve_noalloc(ctypes.byref(sys_), *[a.data_ptr() for a in d], N, mode, None) == 0
    torch.cuda.synchronize()
    for got, want in zip(d[2:], (x, it, st)):
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    if (name, start) in RECORDED:
        weighted = int((it.astype(np.int64) * (np.arange(N) % 97)).sum())
        assert (int(it.sum()), weighted, np.bincount(st, minlength=3).tolist(), zlib.crc32(x.tobytes())) == \
            RECORDED[name, start]
