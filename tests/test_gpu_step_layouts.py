"""The layouts and launch choices of the transport and flow steps at the sizes
where they can go wrong: solutes in chunks of four, two and one, the surrogate
step in one launch and in three, and the flow energy summed once a run.

Tolerances: solute transport against the FP64 oracle, relative L2 <= 1e-5
(FP32 populations, as in the transport tests); the compiled surrogate step
against the run-time-table launches, relative L2 <= 1e-12 (the same arithmetic);
an FP64 sum over n sites in another order, n * 2^-52 relative; populations
given and read back, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as o

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("steps", [1, 4])
@pytest.mark.parametrize("n_mob", [1, 2, 3, 4, 5, 6, 7, 8])
def test_solute_chunks(gpu_lib, pkg, wl, n_mob, steps):
    mask = wl.sphere_pack(13, 9, 11, 0.6, 1.5, 2.5, seed=3)
    nx, ny, nz = mask.shape
    sol = [{"tau": 0.6 + 0.05 * s, "c0": 0.1 * s, "left": "D", "left_value": 1.0 - 0.1 * s, "right": "N"}
           for s in range(n_mob)]
    cfg = pkg.make_config(nx, ny, nz, tau_ns=0.8, rho_in=1.001, rho_out=1.0, solutes=sol)
    lat = pkg.Lattice(cfg)
    lat.upload_mask(mask)
    lat.flow_init()
    lat.flow_steps(40)
    lat.couple_velocity()
    u = np.stack([lat.field(pkg.FIELD_VELOCITY, k).reshape(-1) for k in range(3)])
    lat.ade_init()
    lat.step(steps)
    ref = o.Transport(cfg, mask, u=u)
    ref.step(steps)
    for s in range(n_mob):
        assert rel_l2(lat.field(pkg.FIELD_CONC, s).reshape(-1), ref.density(s)) < 1e-5, s
    # each solute's populations come back as they were given, at either parity
    pops = [lat.solute_populations(s).copy() for s in range(n_mob)]
    for s in range(n_mob):
        lat.set_solute_populations(s, pops[n_mob - 1 - s])
    for s in range(n_mob):
        np.testing.assert_array_equal(lat.solute_populations(s), pops[n_mob - 1 - s])
    lat.close()


# a lattice of a few hundred live sites (one launch, lists per block) and one
# above two waves of that launch's blocks (three launches); neither a multiple
# of a block
@pytest.mark.parametrize("shape", [(13, 9, 11), (68, 61, 63)])
@pytest.mark.parametrize("frac", [(0.0, 0.0), (0.02, 0.0), (0.0, 0.3), (0.2, 0.2), (1.0, 1.0)])
def test_surrogate_launches_match_table(gpu_lib, pkg, wl, shape, frac):
    mask = wl.sphere_pack(*shape, 0.85, 1.5, 2.5, seed=8)
    nx, ny, nz = mask.shape
    cfg = wl.surrogate_config(pkg, nx, ny, nz)
    nets = wl.surrogate_nets(pkg)
    rng = np.random.default_rng(9)
    bio = []
    for m in range(2):
        pick = (mask == wl.MAT_PORE) & (rng.random(mask.shape) < frac[m])
        pick[0] = pick[-1] = False
        b = np.where(pick, rng.uniform(0.005, 0.05, mask.shape), 0.0)
        b[pick & (rng.random(mask.shape) < 0.1)] = 1e-12      # at the threshold itself: no network
        bio.append(b)
    out = []
    for compiled in (1, 0):
        lat = pkg.Lattice(cfg)
        lat.upload_mask(mask)
        lat.flow_init()
        lat.flow_steps(20)
        lat.couple_velocity()
        lat.set_option(pkg.OPT_COMPILED_CHEM, compiled)
        for slot in range(2):
            lat.set_surrogate(slot, nets[slot])
        lat.ade_init()
        for m in range(2):
            lat.set_field(pkg.FIELD_BIOMASS, m, bio[m])
        lat.step(3)
        for m in range(2):                                    # the lists follow the biomass
            lat.set_field(pkg.FIELD_BIOMASS, m, bio[1 - m])
        lat.step(2)
        assert lat.get_option(pkg.OPT_COMPILED_CHEM) == (pkg.CHEM_SURROGATE2 if compiled else 0)
        out.append([lat.field(pkg.FIELD_CONC, s).reshape(-1) for s in range(cfg.n_solutes)]
                   + [lat.field(pkg.FIELD_BIOMASS, m).reshape(-1) for m in range(2)])
        lat.close()
    for a, b in zip(*out):
        assert rel_l2(a, b) <= 1e-12


@pytest.mark.parametrize("steps", [1, 2, 7, 33, 64])
def test_flow_energy_after_a_run(gpu_lib, pkg, wl, steps):
    mask = wl.sphere_pack(22, 16, 16, 0.55, 2.0, 4.0, seed=7)
    cfg = pkg.make_config(*mask.shape, tau_ns=0.8, rho_in=1.001, rho_out=1.0)
    energy = []
    for run in (True, False):
        lat = pkg.Lattice(cfg)
        lat.upload_mask(mask)
        lat.flow_init()
        if run:
            lat.flow_steps(steps)
        else:
            for _ in range(steps):
                lat.flow_steps(1)
        energy.append(lat.flow_energy())
        lat.close()
    assert energy[0] > 0
    assert energy[0] == pytest.approx(energy[1], rel=mask.size * 2.0 ** -52)
