"""Training calls at their edges: pairs that are not numbers, memory after a
large call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(pkg, wl, n):
    import torch
    S, logk, cs = wl.tableau(5, 9, seed=4)
    sys_ = pkg.EqSystem()
    pkg.set_eq_system(sys_, S, logk, cs)
    T, xs, _, _ = wl.speciation_batch(S, logk, n, seed=21)
    return pkg.EqSolver(sys_), T, xs, lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("where", ["total", "solution"])
def test_a_pair_that_is_not_a_number_shows_in_the_loss(gpu_lib, pkg, wl, where):
    """The normalisation takes such a pair as it is, so the loss says so; the
    same call without it trains."""
    n = 4096
    eq, T, xs, dev = _solver(pkg, wl, n)
    dT, dX = dev(T), dev(xs)
    assert np.isfinite(eq.train_device(dT.data_ptr(), dX.data_ptr(), n, epochs=1, batch=1024))
    eq.close()
    eq, T, xs, dev = _solver(pkg, wl, n)
    (T if where == "total" else xs)[5, 0] = np.nan
    dT, dX = dev(T), dev(xs)
    assert np.isnan(eq.train_device(dT.data_ptr(), dX.data_ptr(), n, epochs=1, batch=1024))
    eq.close()


def test_a_large_call_gives_its_memory_back(gpu_lib, pkg, wl):
    """80 MiB of standardised pairs: free memory after the call is what it was,
    and a short call before it keeps its own."""
    import torch
    eq, T, xs, dev = _solver(pkg, wl, 1 << 14)
    dT, dX = dev(np.tile(T, (128, 1))), dev(np.tile(xs, (128, 1)))
    run = lambda n: eq.train_device(dT.data_ptr(), dX.data_ptr(), n, epochs=1, batch=8192)
    run(1 << 14)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        assert np.isfinite(run(1 << 21))
        assert torch.cuda.mem_get_info()[0] >= free
    assert np.isfinite(run(1 << 14))
    eq.close()
