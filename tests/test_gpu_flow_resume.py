"""Flow solves that start where earlier steps ended: the AA storage alternates
between two layouts, so a solve has to leave the context at the layout of the
steps run so far, whatever number of them came before it.  The same number of
steps in one call gives the same populations and velocity, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(pkg, wl):
    mask = wl.sphere_pack(22, 16, 16, 0.55, 2.0, 4.0, seed=7)
    lat = pkg.Lattice(pkg.make_config(*mask.shape, tau_ns=0.8, rho_in=1.001, rho_out=1.0))
    lat.upload_mask(mask)
    lat.flow_init()
    return lat


def _state(pkg, lat):
    lat.couple_velocity()
    return [lat.flow_populations()] + [lat.field(pkg.FIELD_VELOCITY, k) for k in range(3)]


# runs of flow_steps (s) and unconverged flow_solve (v) calls
@pytest.mark.parametrize("runs", [[("s", 1), ("v", 4)], [("v", 1), ("v", 2)], [("s", 33), ("v", 70), ("v", 1), ("s", 3)],
                                  [("s", 1), ("v", 0)], [("s", 2), ("v", 3), ("s", 1)]])
def test_solve_after_other_steps(gpu_lib, pkg, wl, runs):
    lat = _lattice(pkg, wl)
    for kind, n in runs:
        if kind == "s":
            lat.flow_steps(n)
        else:
            assert lat.flow_solve(n, 0.0)[0] == n
    got = _state(pkg, lat)
    lat.close()
    lat = _lattice(pkg, wl)
    lat.flow_steps(sum(n for _, n in runs))
    want = _state(pkg, lat)
    lat.close()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("before", [0, 1, 2])
def test_solves_that_converge(gpu_lib, pkg, wl, before):
    """Two converging solves in a row (the second has its window of 500 steps
    to fill first), then more steps: the converging step's index counts the
    solve's own steps."""
    lat = _lattice(pkg, wl)
    lat.flow_steps(before)
    total = before
    for _ in range(2):
        it, status = lat.flow_solve(20000, 1e-5)
        assert status == pkg.OK
        total += it + 1
    lat.flow_steps(3)
    got = _state(pkg, lat)
    lat.close()
    lat = _lattice(pkg, wl)
    lat.flow_steps(total + 3)
    want = _state(pkg, lat)
    lat.close()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
