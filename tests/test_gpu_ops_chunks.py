"""The per-operator entry points over every number of mobile solutes, so over
solutes in chunks of four, two and one: collide, kinetics and stream taken
apart against the FP64 oracle (relative L2 <= 1e-4, as the other reaction
tests) at both parities of the storage, and without reactions against cl_step,
which collides and streams with the same arithmetic (bit for bit)."""
import numpy as np
import pytest

from oracle import oracle as o

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300))


def _config(pkg, shape, n_mob, kinetics):
    sol = [{"tau": 0.6 + 0.05 * s, "c0": 0.02 + 0.01 * s, "left": "D", "left_value": 0.5 - 0.05 * s, "right": "N"}
           for s in range(n_mob)]
    cfg = pkg.make_config(*shape, tau_ns=0.8, rho_in=1.001, rho_out=1.0, solutes=sol, microbes=1, dt=1.0)
    if kinetics:
        cfg.enable_kinetics = 1
        # every other solute takes part: the rest of a chunk keeps its populations
        pkg.add_rxn(cfg, microbe=0, k=2e-2, monod=[(0, 5e-2)],
                    nu={s: -1.0 / (s + 1) for s in range(0, n_mob, 2)}, yield_=0.4)
    return cfg


def _lattice(pkg, wl, cfg, mask, bio):
    lat = pkg.Lattice(cfg)
    lat.upload_mask(mask)
    lat.flow_init()
    lat.flow_steps(40)
    lat.couple_velocity()
    lat.ade_init()
    lat.set_field(pkg.FIELD_BIOMASS, 0, bio)
    return lat


@pytest.mark.parametrize("n_mob", [1, 2, 3, 4, 5, 6, 7, 8])
def test_operators_by_number_of_solutes(gpu_lib, pkg, wl, n_mob):
    mask = wl.sphere_pack(13, 9, 11, 0.6, 1.5, 2.5, seed=3)
    bio = wl.seed_biomass(mask, 4, frac=0.5)
    cfg = _config(pkg, mask.shape, n_mob, True)
    lat = _lattice(pkg, wl, cfg, mask, bio)
    ref = o.Transport(cfg, mask, u=np.stack([lat.field(pkg.FIELD_VELOCITY, k).reshape(-1) for k in range(3)]))
    ref.set_biomass(0, bio)
    for _ in range(3):
        lat.op_collide()
        lat.op_reactions(pkg.OP_ALL)
        lat.op_stream()
        ref.step(1)
        for s in range(n_mob):
            assert rel_l2(lat.field(pkg.FIELD_CONC, s).reshape(-1), ref.density(s)) <= 1e-4, s
    lat.close()
    cfg = _config(pkg, mask.shape, n_mob, False)
    a, b = _lattice(pkg, wl, cfg, mask, bio), _lattice(pkg, wl, cfg, mask, bio)
    for _ in range(3):
        a.step(1)
        b.op_collide()
        b.op_stream()
        for s in range(n_mob):
            np.testing.assert_array_equal(a.solute_populations(s), b.solute_populations(s))
    a.close()
    b.close()
