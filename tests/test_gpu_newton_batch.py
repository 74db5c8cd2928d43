"""The batch Newton solve's two kernels (one solve per thread from a queue,
above 8192 systems; one solve per warp, up to 8192): the same systems take the
same iterates on either, bit for bit, over tableaux of one to five components
with unit, negative, large and fractional coefficients and inactive species;
and converged solutions agree with the FP64 oracle to 1e-8 in log10 (both stop
at a 1e-10 relative mass-balance residual)."""
import numpy as np
import pytest

from oracle import oracle as o

pytestmark = pytest.mark.gpu

# name -> (stoichiometry, logK); the components come first
TABLEAUX = {
    "one": ([[1], [2]], [0, 3.0]),
    "carbonate": ([[1, 0], [0, 1], [1, -1], [1, 1], [0, 0]], [0, 0, -10.33, 6.35, 0]),
    "three": ([[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 0]], [0, 0, 0, 10.33, 3.2]),
    "cube": ([[1, 0], [0, 1], [3, 1], [1, -1]], [0, 0, 5.0, -4.0]),
    "half": ([[1, 0], [0, 1], [0.5, 1.5], [1, 1]], [0, 0, 1.0, 2.0]),
}


def _system(pkg, wl, name):
    if name == "five":
        S, logk, cs = wl.tableau(5, 9, seed=4)
    else:
        S, logk = np.array(TABLEAUX[name][0], float), np.array(TABLEAUX[name][1], float)
        cs = list(range(S.shape[1]))
    sys_ = pkg.EqSystem()
    pkg.set_eq_system(sys_, S, logk, cs, max_iter=200, tol=1e-10, warm_iter=6)
    return sys_, S, logk


def _totals(wl, name, S, logk, n):
    if name == "five":
        return wl.speciation_batch(S, logk, n, seed=21)[0]
    rng = np.random.default_rng(22)
    T = np.empty((0, S.shape[1]))
    while len(T) < n:
        x = rng.uniform(-6, -2, (2 * n, S.shape[1]))
        t = (10.0 ** np.clip(logk + x @ S.T, -30, 1)) @ S
        T = np.concatenate([T, t[(t > 0).all(1)]])
    return T[:n]


@pytest.mark.parametrize("name", ["one", "carbonate", "three", "cube", "half", "five"])
@pytest.mark.parametrize("start", ["cold", "given"])
def test_queue_and_warp_kernels_take_the_same_iterates(gpu_lib, pkg, wl, name, start):
    sys_, S, logk = _system(pkg, wl, name)
    n = 8193
    T = _totals(wl, name, S, logk, n)
    cold = wl.cold_species(S, T)
    # a given start some decades off: part of the solves fall back to the cold start
    x0 = np.log10(T) + np.random.default_rng(3).uniform(-3, 1, T.shape)
    mode = pkg.EQ_START_COLD if start == "cold" else pkg.EQ_START_GIVEN
    eq = pkg.EqSolver(sys_)
    run = lambda a, b: eq.solve(T[a:b], cold[a:b], x0=x0[a:b], start=mode)
    x, it, st = run(0, n)
    for a, b in ((0, 8192), (8192, 8193), (100, 131)):
        for got, want in zip(run(a, b), (x[a:b], it[a:b], st[a:b])):
            np.testing.assert_array_equal(got, want)
    xo, _, sto = o.eq_batch(sys_, T[:500], cold[:500], start=0)
    # (totals formed from clamped species have no root: neither converges there)
    assert np.mean((st[:500] < 2) == (sto < 2)) > 0.99
    both = (st[:500] < 2) & (sto < 2)
    assert both.mean() > 0.5
    np.testing.assert_allclose(x[:500][both], xo[both], atol=1e-8)


def test_iteration_limits(gpu_lib, pkg, wl):
    """max_iter ends a solve where it stands; without warm iterations the given start is not used."""
    sys_, S, logk = _system(pkg, wl, "five")
    n = 8200
    T = _totals(wl, "five", S, logk, n)
    cold = wl.cold_species(S, T)
    full = pkg.EqSolver(sys_).solve(T, cold)
    sys_.max_iter = 9
    x, it, st = pkg.EqSolver(sys_).solve(T, cold)
    assert it.max() == 9
    done = full[1] <= 9
    np.testing.assert_array_equal(st[done], full[2][done])
    np.testing.assert_array_equal(x[done], full[0][done])
    assert (st[full[1] > 9] == 2).all()
    sys_.max_iter, sys_.warm_iter = 200, 0
    x, it, st = pkg.EqSolver(sys_).solve(T, cold, x0=np.zeros_like(T), start=pkg.EQ_START_GIVEN)
    np.testing.assert_array_equal(x, full[0])
    np.testing.assert_array_equal(it, full[1])
    np.testing.assert_array_equal(st, np.where(full[2] == 0, 1, full[2]))


def test_solve_after_a_refused_allocation(gpu_lib, pkg, wl):
    """A batch whose lists do not fit is refused before anything runs on it,
    gives its memory back and leaves the solver able to solve: a batch of the
    size it had solved before (large enough for the queue kernel, which writes
    the lists) comes out as before.  The first size fails on the first list,
    the second (two lists of 0.6 of the free memory each) on the second."""
    import torch
    sys_, S, logk = _system(pkg, wl, "five")
    T = _totals(wl, "five", S, logk, 9000)
    cold = wl.cold_species(S, T)
    x0 = np.log10(T) - 1.0
    d = [torch.tensor(a, dtype=torch.float64, device="cuda") for a in (T, cold, x0)]
    for part in (1, 2):
        eq = pkg.EqSolver(sys_)
        want = [eq.solve(T, cold, x0=x0, start=s) for s in (pkg.EQ_START_COLD, pkg.EQ_START_GIVEN)]
        free = torch.cuda.mem_get_info()[0]
        n = 1 << 40 if part == 1 else int(0.6 * free) // 8
        with pytest.raises(pkg.CLError, match=r"\(%d\)" % pkg.ERR_NOMEM):
            eq.solve_device(*[a.data_ptr() for a in d], 0, 0, n, pkg.EQ_START_COLD)
        assert torch.cuda.mem_get_info()[0] >= free
        for s, w in zip((pkg.EQ_START_COLD, pkg.EQ_START_GIVEN), want):
            for got, ref in zip(eq.solve(T, cold, x0=x0, start=s), w):
                np.testing.assert_array_equal(got, ref)
        eq.close()
