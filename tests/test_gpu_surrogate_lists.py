"""The compiled surrogate step's voxel lists against the run-time-table
launches (the same arithmetic: relative L2 <= 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300))


def _lattice(pkg, wl, mask, bio, compiled, variant=0):
    cfg = wl.surrogate_config(pkg, *mask.shape)
    lat = pkg.Lattice(cfg)
    lat.upload_mask(mask)
    lat.flow_init()
    lat.flow_steps(20)
    lat.couple_velocity()
    lat.set_option(pkg.OPT_COMPILED_CHEM, compiled)
    lat.set_option(pkg.OPT_FAST_VARIANT, variant)
    for slot, net in enumerate(wl.surrogate_nets(pkg)):
        lat.set_surrogate(slot, net)
    lat.ade_init()
    for m in range(2):
        lat.set_field(pkg.FIELD_BIOMASS, m, bio[m])
    return lat


def _state(pkg, lat):
    return [lat.field(pkg.FIELD_CONC, s).reshape(-1) for s in range(6)] + \
        [lat.field(pkg.FIELD_BIOMASS, m).reshape(-1) for m in range(2)]


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
def test_block_lists_at_the_edges_of_a_warp(gpu_lib, pkg, wl, variant):
    """Planes of 128 sites, so that a plane is one block of the launch (two of
    the shapes with 64 threads): every pair of list lengths around the 32 voxels
    that a warp takes, none and a full block among them."""
    lengths = (0, 1, 31, 32, 33, 64, 65, 97, 128)
    mask = np.full((2 + len(lengths) ** 2, 8, 16), wl.MAT_PORE, np.uint8)
    rng = np.random.default_rng(4)
    bio = [np.zeros(mask.shape) for _ in range(2)]
    for j, a in enumerate(lengths):
        for i, b in enumerate(lengths):
            for m, n in enumerate((a, b)):
                plane = bio[m][1 + j * len(lengths) + i].reshape(-1)
                plane[rng.permutation(128)[:n]] = rng.uniform(0.005, 0.05, n)
    out = []
    for compiled in (1, 0):
        lat = _lattice(pkg, wl, mask, bio, compiled, variant if compiled else 0)
        lat.step(2)
        out.append(_state(pkg, lat))
        lat.close()
    for a, b in zip(*out):
        assert rel_l2(a, b) <= 1e-12


def _large(wl, frac, shape=(90, 70, 66)):
    """A lattice large enough for the voxel lists, and biomass on a fraction of its pores."""
    mask = wl.sphere_pack(*shape, 0.85, 1.5, 2.5, seed=8)
    rng = np.random.default_rng(9)
    bio = []
    for m in range(2):
        pick = (mask == wl.MAT_PORE) & (rng.random(mask.shape) < frac[m])
        pick[0] = pick[-1] = False
        bio.append(np.where(pick, rng.uniform(0.005, 0.05, mask.shape), 0.0))
    return mask, bio


def test_the_lists_take_no_memory_in_a_step(gpu_lib, pkg, wl):
    """The lists lie in the context's scratch, so the step needs no memory of
    its own and cannot be refused any: the compiled step and the run-time
    table's hold the same after it."""
    mask, bio = _large(wl, (0.1, 0.1))
    held = []
    for compiled in (1, 0):
        lat = _lattice(pkg, wl, mask, bio, compiled)
        n0 = lat.launch_count()
        lat.step(1)
        held.append(lat.device_bytes())
        if compiled:
            assert lat.launch_count() - n0 == 4          # list, chain, streaming, boundary
        lat.close()
    assert held[0] == held[1]


@pytest.mark.parametrize("frac", [(0.0, 0.0), (0.02, 0.0), (0.0, 0.3), (0.2, 0.2), (1.0, 1.0)])
def test_launches_by_size_and_share(gpu_lib, pkg, wl, frac):
    """Above the lattice size that lists its voxels: four launches a step while
    the lists are short of most sites, two (the one launch and the boundary)
    from the step after the first list that was not, and the list again at
    every 32nd step and after the biomass was set.  Small lattices:
    two launches.  The same fields as the run-time table's launches."""
    dense = frac == (1.0, 1.0)
    small, bio_s = _large(wl, frac, (20, 16, 12))
    lat = _lattice(pkg, wl, small, bio_s, 1)
    n0 = lat.launch_count()
    lat.step(3)
    assert lat.launch_count() - n0 == 6
    lat.close()
    mask, bio = _large(wl, frac)
    _, other = _large(wl, (0.1, 0.1))
    out = []
    for compiled in (1, 0):
        lat = _lattice(pkg, wl, mask, bio, compiled)
        counts = []

        def step(n):
            n0 = lat.launch_count()
            lat.step(n)
            counts.append(lat.launch_count() - n0)

        step(3)                                          # one wait after the first list
        for _ in range(2):
            step(1)
        for m in range(2):
            lat.set_field(pkg.FIELD_BIOMASS, m, other[m])
        step(1)
        for m in range(2):
            lat.set_field(pkg.FIELD_BIOMASS, m, bio[m])
        step(1)
        step(25)                                         # steps 7 to 31
        step(2)                                          # step 32 lists
        if compiled:
            assert counts == ([4 + 2 + 2, 2, 2, 4, 4, 50, 6] if dense else [12, 4, 4, 4, 4, 100, 8])
        out.append(_state(pkg, lat))
        lat.close()
    for a, b in zip(*out):
        assert rel_l2(a, b) <= 1e-12


def test_the_listed_chemistry_has_no_phases(gpu_lib, pkg, wl):
    """The lists hold the voxels with biomass alone, because a phase needs an
    immobile mineral: a phase on one of the chemistry's solutes is refused."""
    cfg = wl.surrogate_config(pkg, 12, 8, 8)
    cfg.dissol_enabled, cfg.reopen_fraction = 1, 0.5
    pkg.add_phase(cfg, 0, 1.0)
    with pytest.raises(pkg.CLError, match="immobile"):
        pkg.Lattice(cfg)
