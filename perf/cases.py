"""Performance cases: the work a user of the library has it do, through its public entry points.

The lattice cases advance a context by a stretch of steps, as a run does
between two saves, and read the fields back as the driver's field output
does: FP64 from the library, written as single precision where the state is
single precision (concentrations, velocities), FP64 where it is FP64 (mineral
inventory, biomass).  The batch cases call the speciation and network entry
points on device arrays.

`exact` is an independent FP64 restatement in torch of what each pass
computes: dense two-buffer lattice Boltzmann, the rate laws, the equilibrium
by bisection in one unknown.
"""
import ctypes
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "complb3d-lattice-boltzmann-fba-surrogate-cobrapy-glpk_b200")
F64 = torch.float64
SOLID, WALL, PORE, BIOFILM = 0, 1, 2, 3
THRD = 1e-12


def _pkg():
    if "complab_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("complab_b200", os.path.join(PKG_DIR, "__init__.py"),
                                                      submodule_search_locations=[PKG_DIR])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["complab_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["complab_b200"]


def _wl():
    _pkg()
    return importlib.import_module("complab_b200.workloads")


def listed():
    return [
        # the reference's example suite: a 24 x 24 x 6 channel (plus the two boundary planes) with the
        # carbonate system, run as the driver runs it: flow, then one call per transport step
        {"name": "example_channel", "kind": "carbonate", "nx": 26, "ny": 24, "nz": 6, "porosity": 0.85, "rmin": 2.0,
         "rmax": 3.0, "flow": 300, "steps": 200, "per_call": 1, "warm": False},
        # flow to a developed field, then one solute's breakthrough, at 64^3
        {"name": "flow_transport_64", "kind": "solute", "nx": 66, "ny": 64, "nz": 64, "porosity": 0.40, "rmin": 4.0,
         "rmax": 8.0, "flow": 500, "steps": 250},
        # the flow solve alone on a large pore space (permeability)
        {"name": "flow_256", "kind": "flow", "nx": 258, "ny": 256, "nz": 256, "porosity": 0.35, "rmin": 5.0,
         "rmax": 10.0, "flow": 300},
        # biotic kinetics with the biofilm automaton's block after every step
        {"name": "biotic_ca_128", "kind": "biotic", "nx": 128, "ny": 128, "nz": 128, "porosity": 0.35, "rmin": 5.0,
         "rmax": 10.0, "steps": 100},
        # a user's own chemistry (the run-time rate table and tableau): carbonate speciation in every pore voxel
        {"name": "carbonate_table", "kind": "carbonate", "nx": 128, "ny": 96, "nz": 96, "porosity": 0.40, "rmin": 4.0,
         "rmax": 8.0, "flow": 50, "steps": 50, "per_call": 50, "warm": True},
        # two organisms' surrogate networks in the step
        {"name": "surrogate_256", "kind": "surrogate", "nx": 256, "ny": 256, "nz": 256, "porosity": 0.40, "rmin": 4.0,
         "rmax": 8.0, "steps": 100},
        # one interval of the coupled loop (transport, node conversions, flow re-solve) on a medium domain ...
        {"name": "coupled_medium", "kind": "coupled", "nx": 256, "ny": 128, "nz": 128, "porosity": 0.35, "rmin": 5.0,
         "rmax": 10.0, "steps": 200, "flow": 500},
        # ... and on the benchmark's domain
        {"name": "coupled_large", "kind": "coupled", "nx": 512, "ny": 256, "nz": 256, "porosity": 0.35, "rmin": 5.0,
         "rmax": 10.0, "steps": 200, "flow": 500},
        # speciation of a pore field, from the cold start and from a trained network's start
        {"name": "speciation_cold", "kind": "speciation", "n": 1 << 20, "start": "cold"},
        {"name": "speciation_learned", "kind": "speciation", "n": 1 << 20, "start": "learned"},
        # batched surrogate inference on the tensor cores
        {"name": "surrogate_batch", "kind": "network", "n": 1 << 21, "mode": "tcgen05"},
        # training of the warm-start network on Newton's pairs (forward and backward)
        {"name": "train_network", "kind": "train", "n": 1 << 18, "batch": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["carbonate", "solute", "flow", "biotic", "surrogate", "coupled", "speciation", "network", "train"])
    if kind == "speciation":
        return {"kind": kind, "n": _log(rng, 500, 1 << 20), "start": rng.choice(["cold", "learned"])}
    if kind == "network":
        return {"kind": kind, "n": _log(rng, 1000, 1 << 21), "mode": rng.choice(["tcgen05", "tensor", "fp32"])}
    if kind == "train":
        return {"kind": kind, "n": _log(rng, 1 << 15, 1 << 18), "batch": rng.choice([1024, 2048, 4096])}
    top = {"carbonate": 1.2e6, "solute": 2e6, "flow": 1.6e7, "biotic": 2e6, "surrogate": 8e6, "coupled": 8e6}[kind]
    low = {"carbonate": 4e3, "solute": 4e3, "flow": 4e3, "biotic": 3e4, "surrogate": 3e4, "coupled": 3e4}[kind]
    sites = math.exp(rng.uniform(math.log(low), math.log(top)))
    # a box somewhat longer along the flow, odd extents among them
    ny = max(7, int(round((sites / rng.uniform(1.0, 2.5)) ** (1.0 / 3.0))) + rng.randint(-1, 1))
    nz = max(6, ny + rng.randint(-ny // 5, ny // 5))
    nx = max(10, int(sites / (ny * nz)))
    big = min(ny, nz) >= 40
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "porosity": round(rng.uniform(0.35, 0.6) if big else rng.uniform(0.6, 0.85), 3),
         "rmin": 4.0 if big else 2.0, "rmax": rng.choice([8.0, 10.0]) if big else 3.0}
    if kind in ("carbonate", "solute", "flow", "coupled"):
        c["flow"] = rng.randint(30, 100) if kind == "carbonate" else rng.randint(60, 300)
    if kind == "flow":
        return c
    c["steps"] = rng.randint(20, 120)
    if kind == "carbonate":
        c["per_call"] = rng.choice([1, c["steps"]])
        c["warm"] = rng.choice([False, True])
    return c


# ---------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


D3Q19 = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1), (0, -1, -1),
         (0, -1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1)]


def _shift(a, dx, dy, dz, fill):
    """a at the site (x - dx, y - dy, z - dz): y and z periodic, `fill` beyond the x ends."""
    b = torch.roll(a, (dy, dz), (-2, -1)) if dy or dz else a
    if dx == 0:
        return b
    out = torch.full_like(b, fill)
    if dx > 0:
        out[..., 1:, :, :] = b[..., :-1, :, :]
    else:
        out[..., :-1, :, :] = b[..., 1:, :, :]
    return out


def _pack(case, seed):
    """Overlapping spheres placed until the porosity is reached (uint8 material numbers, on the device): pore 2,
    solid 0, a solid next to a pore along a D3Q19 link bounce-back 1; the x end planes copy their neighbours."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev, nxi = _device(), nx - 2
    g = torch.Generator(device="cpu").manual_seed(int(seed) * 7919 + 17)
    vol, r0, r1 = nxi * ny * nz, case["rmin"], case["rmax"]
    rmean3 = (r1 ** 4 - r0 ** 4) / (4.0 * (r1 - r0))
    count = int(-math.log(case["porosity"]) * vol / (4.18879 * rmean3) * 1.5) + 40
    ctr = torch.rand((count, 3), generator=g, dtype=F64) * torch.tensor([nxi, ny, nz], dtype=F64)
    rad = (r0 + (r1 - r0) * torch.rand(count, generator=g, dtype=F64)).to(dev)
    ctr = ctr.to(dev)
    half = int(math.ceil(r1)) + 1
    o = torch.arange(-half, half + 1, device=dev)
    off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3)
    first = torch.full((vol,), count, dtype=torch.int32, device=dev)
    chunk = max(1, 16_000_000 // off.shape[0])
    for s in range(0, count, chunk):
        c = ctr[s:s + chunk]
        vox = torch.floor(c).long()[:, None, :] + off[None]
        d2 = ((vox + 0.5 - c[:, None, :]) ** 2).sum(-1)
        ok = (d2 <= (rad[s:s + chunk, None] ** 2)) & (vox[..., 0] >= 0) & (vox[..., 0] < nxi)
        idx = (vox[..., 0] * ny + vox[..., 1] % ny) * nz + vox[..., 2] % nz
        who = torch.arange(s, s + c.shape[0], device=dev, dtype=torch.int32)[:, None].expand_as(idx)
        first.scatter_reduce_(0, idx[ok], who[ok], "amin")
    cum = torch.cumsum(torch.bincount(first.long(), minlength=count + 1)[:count], 0)
    last = int((cum < (1.0 - case["porosity"]) * vol).sum())
    solid = (first <= last).reshape(nxi, ny, nz)
    pore = torch.ones((nx, ny, nz), dtype=torch.bool, device=dev)
    pore[1:-1] = ~solid
    if case.get("kind") == "carbonate":       # a channel: walls along y
        pore[:, 0] = False
        pore[:, -1] = False
    pore[0], pore[-1] = pore[1], pore[-2]
    near = torch.zeros_like(pore)
    for dx, dy, dz in D3Q19[1:]:
        near |= _shift(pore, dx, dy, dz, False)
    return torch.where(pore, PORE, torch.where(near, WALL, SOLID)).to(torch.uint8)


def _wall_adjacent(mat):
    """Pore voxels of the interior planes with a wall across a face."""
    wall = (mat == SOLID) | (mat == WALL)
    near = torch.zeros_like(wall)
    for dx, dy, dz in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)):
        near |= _shift(wall, dx, dy, dz, False)
    cand = (mat == PORE) & near
    cand[0] = cand[-1] = False
    return cand


def _seeded(mat, seed, frac, lo, hi):
    """U[lo, hi) on a fraction of the wall-adjacent pore voxels (FP64, on the device)."""
    g = torch.Generator(device=mat.device).manual_seed(int(seed) * 104729 + 5)
    pick = _wall_adjacent(mat) & (torch.rand(mat.shape, generator=g, device=mat.device) < frac)
    v = lo + (hi - lo) * torch.rand(mat.shape, generator=g, device=mat.device, dtype=F64)
    return torch.where(pick, v, torch.zeros((), dtype=F64, device=mat.device))


def _material(case, seed):
    if case["kind"] != "biotic":
        return _pack(case, seed)
    # a duct whose pore space is one cluster, as the biofilm automaton's age field needs it
    m = _wl().walled_pack(case["nx"], case["ny"], case["nz"], case["porosity"], case["rmin"], case["rmax"], int(seed) % (1 << 31))
    return torch.from_numpy(m).to(_device())


def _config(case, seed):
    """The context's configuration; tau, rates and boundary values from the seed where they are not part of the case."""
    pkg, wl, kind = _pkg(), _wl(), case["kind"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(int(seed) + 11)
    if kind in ("flow", "solute"):
        sol = [{"tau": 0.7, "c0": float(rng.uniform(0.0, 0.2)), "left": "D", "left_value": 1.0, "right": "N"}]
        return pkg.make_config(nx, ny, nz, tau_ns=0.8, rho_in=1.001, rho_out=1.0, solutes=sol if kind == "solute" else [])
    if kind == "biotic":
        return wl.biotic_config(pkg, nx, ny, nz, seed=int(seed) % 1000)
    if kind == "surrogate":
        return wl.surrogate_config(pkg, nx, ny, nz, seed=int(seed) % 1000)
    if kind == "coupled":
        return wl.coupled_config(pkg, nx, ny, nz, seed=int(seed) % 1000, dissolution=True)
    # carbonate system: components HCO3- and H+, species CO3-- and H2CO3; acid enters on the left
    h = float(10.0 ** rng.uniform(-6.5, -5.5))
    sol = [{"tau": 0.8, "c0": 1e-3, "left": "D", "left_value": 2e-3, "right": "N"},
           {"tau": 0.8, "c0": 1e-7, "left": "D", "left_value": h, "right": "N"},
           {"tau": 0.8, "c0": 0.0, "left": "N", "right": "N"}, {"tau": 0.8, "c0": 0.0, "left": "N", "right": "N"}]
    cfg = pkg.make_config(nx, ny, nz, tau_ns=0.8, rho_in=1.0005, rho_out=1.0, solutes=sol)
    cfg.use_equilibrium = 1
    pkg.set_eq_system(cfg.eq, [[1, 0], [0, 1], [1, -1], [1, 1]], [0.0, 0.0, -10.33, 6.35], [0, 1], max_iter=200,
                      tol=1e-10, warm_iter=8)
    cfg.eq_warm_previous = 1 if case["warm"] else 0
    return cfg


def _nets(seed):
    return _wl().surrogate_nets(_pkg(), seed=int(seed) % 1000)


def _biomass(case, mat, seed):
    if case["kind"] == "biotic":
        return [_seeded(mat, seed, 0.02, 10.0, 50.0)]
    if case["kind"] == "coupled":
        return [_seeded(mat, seed, 0.02, 10.0, 50.0)]
    if case["kind"] == "surrogate":
        return [_seeded(mat, seed + 1000 * m, 0.3, 0.005, 0.05) for m in range(2)]
    return []


START_FLOW = {"biotic": 60, "surrogate": 30, "coupled": 60}    # flow steps that give the transport its first velocity


class _Output:
    """Host buffers of one context's field output: pinned FP64 staging, one tensor per saved field."""

    def __init__(self, shape, fields, mask):
        n = shape[0] * shape[1] * shape[2]
        self.fields = fields
        self.stage = torch.empty(n, dtype=F64, pin_memory=torch.cuda.is_available())
        self.out = {name: torch.zeros(shape, dtype=dt) for name, _, _, dt in fields}
        if mask:
            self.out["mask"] = torch.zeros(shape, dtype=torch.uint8)

    def read(self, lat):
        for name, field, index, dtype in self.fields:
            st = lat.lib.cl_get_field(lat.h, field, index, self.stage.data_ptr())
            if st < 0:
                raise RuntimeError("cl_get_field: %d" % st)
            self.out[name].view(-1).copy_(self.stage)
        if "mask" in self.out:
            lat.lib.cl_download_mask(lat.h, self.out["mask"].data_ptr())
        return self.out


def _lattice(case, seed):
    pkg, kind = _pkg(), case["kind"]
    cfg, mat = _config(case, seed), _material(case, seed)
    lat = pkg.Lattice(cfg)
    lat.upload_mask(mat.cpu().numpy())
    lat.flow_init()
    if kind in START_FLOW:
        lat.flow_steps(START_FLOW[kind])
        lat.couple_velocity()
    f32, fields = torch.float32, []
    if kind != "flow":
        if kind == "surrogate":
            for o, net in enumerate(_nets(seed)):
                lat.set_surrogate(o, net)
        lat.ade_init()
        for m, b in enumerate(_biomass(case, mat, seed)):
            lat.set_field(pkg.FIELD_BIOMASS, m, b.cpu().numpy())
            fields.append(("biomass%d" % m, pkg.FIELD_BIOMASS, m, F64))
        if kind == "coupled":
            lat.set_field(pkg.FIELD_CONC, 8, _seeded(mat, seed + 77, 0.5, 0.0, 1.0).cpu().numpy())
        if kind == "biotic":
            lat.ca_update_mask()
        for s in range(cfg.n_solutes):
            fields.append(("c%d" % s, pkg.FIELD_CONC, s, F64 if cfg.immobile[s] else f32))
    if "flow" in case:
        fields += [("u%d" % k, pkg.FIELD_VELOCITY, k, f32) for k in range(3)]
    if kind == "flow":
        fields.append(("rho", pkg.FIELD_FLOW_RHO, 0, f32))
    return {"lat": lat, "case": case, "out": _Output((case["nx"], case["ny"], case["nz"]), fields, kind in ("biotic", "coupled"))}


def _tableau():
    return _wl().tableau(5, 9, seed=4)


def _speciation(n, seed):
    """Well-posed totals of the 5-component tableau: free components drawn first, totals formed from them; (T, x)."""
    S, logk, _ = _tableau()
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed) * 31 + 3)
    S, logk = torch.tensor(S, device=dev), torch.tensor(logk, device=dev)
    got, Ts, xs = 0, [], []
    while got < n:
        m = 1 << 22
        x = -7.0 + 6.0 * torch.rand((m, 5), generator=g, device=dev, dtype=F64)
        x[:, 4] = -9.0 + 4.0 * torch.rand(m, generator=g, device=dev, dtype=F64)
        lc = logk + x @ S.T
        T = (10.0 ** lc.clamp(-30, 1)) @ S
        ok = (lc <= 0.5).all(1) & (lc >= -30).all(1) & (T > 0).all(1) & ((T[:, :4] >= 1e-6) & (T[:, :4] <= 1e-1)).all(1)
        Ts.append(T[ok]), xs.append(x[ok])
        got += int(ok.sum())
    return torch.cat(Ts)[:n].contiguous(), torch.cat(xs)[:n].contiguous()


_stream_ = []


def _side_stream():
    """The stream the batch solver and the arrays around it run on."""
    if not _stream_:
        _stream_.append(torch.cuda.Stream())
    return _stream_[0]


def _solver():
    pkg = _pkg()
    S, logk, cs = _tableau()
    sys_ = pkg.EqSystem()
    pkg.set_eq_system(sys_, S, logk, cs, max_iter=200, tol=1e-10, warm_iter=6)
    return pkg.EqSolver(sys_, stream=_side_stream().cuda_stream)


def _network_inputs(case, seed):
    """Donor, acceptor and biomass over the networks' box, a tenth of them beyond it."""
    g = torch.Generator(device=_device()).manual_seed(int(seed) + 9)
    u = torch.rand((case["n"], 3), generator=g, device=_device()) * 1.1
    return u * torch.tensor([2e-3, 1e-3, 60.0], device=u.device)


def prepare(case, seed):
    pkg, kind = _pkg(), case["kind"]
    if kind == "speciation":
        n = case["n"]
        T, _ = _speciation(n, seed)
        s = {"eq": _solver(), "n": n, "T": T, "learned": case["start"] == "learned", "x": torch.zeros_like(T), "status": torch.zeros(n, dtype=torch.uint8, device=T.device),
             "cold": torch.full((n, 14), 1e-30, dtype=F64, device=T.device)}
        s["cold"][:, :5] = T
        if s["learned"]:
            Tt, xt = _speciation(1 << 17, seed + 500)
            torch.cuda.synchronize()
            s["eq"].train_device(Tt.data_ptr(), xt.data_ptr(), Tt.shape[0], epochs=20, batch=2048, lr=3e-3, seed=7)
        torch.cuda.synchronize()
        return s
    if kind == "train":
        T, x = _speciation(case["n"], seed)
        eq = _solver()
        torch.cuda.synchronize()
        return {"eq": eq, "T": T, "x": x, "batch": case["batch"], "start": eq.params()}
    if kind == "network":
        x = _network_inputs(case, seed)
        return {"net": _nets(seed)[0], "x": x, "y": torch.zeros((case["n"], 4), device=x.device), "n": case["n"],
                "mode": {"tcgen05": pkg.SRG_TCGEN05, "tensor": pkg.SRG_TENSOR, "fp32": pkg.SRG_FP32}[case["mode"]]}
    return _lattice(case, seed)


def run(state):
    pkg = _pkg()
    if "lat" not in state:
        if "net" in state:
            pkg.surrogate_batch_device(state["net"], state["x"].data_ptr(), state["y"].data_ptr(), state["n"], state["mode"],
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            return state["y"]
        eq, T, x = state["eq"], state["T"], state["x"]
        if "batch" in state:
            eq.set_params(state["start"])
            loss = eq.train_device(T.data_ptr(), x.data_ptr(), T.shape[0], epochs=1, batch=state["batch"], lr=3e-3, seed=3)
            return {"loss": np.float32(loss), "params": eq.params()}
        eq.solve_device(T.data_ptr(), state["cold"].data_ptr(), x.data_ptr(), None, state["status"].data_ptr(), state["n"],
                        pkg.EQ_START_LEARNED if state["learned"] else pkg.EQ_START_COLD)
        with torch.cuda.stream(_side_stream()):      # what did not converge is not applied
            applied = x * (state["status"] < 2).unsqueeze(1)
        return {"x": applied, "status": state["status"]}
    lat, case = state["lat"], state["case"]
    kind = case["kind"]
    if kind in ("flow", "solute", "carbonate"):
        lat.flow_steps(case["flow"])
        lat.couple_velocity()
    if kind == "biotic":
        for _ in range(case["steps"]):
            lat.step(1)
            lat.ca_redistribute()
    elif kind == "carbonate":
        for _ in range(case["steps"] // case["per_call"]):
            lat.step(case["per_call"])
    elif kind != "flow":
        lat.step(case["steps"])
    if kind == "coupled":
        lat.precip_convert()
        lat.dissol_convert()
        lat.update_dynamics()
        lat.flow_steps(case["flow"])
        lat.couple_velocity()
    return state["out"].read(lat)


def work(case):
    kind = case["kind"]
    if kind == "speciation":
        # totals in, logs and status out; one evaluation and one 5 x 5 solve of the 14 species per Newton step
        steps = 12 if case["start"] == "cold" else 3
        net = 0 if case["start"] == "cold" else 2 * (5 * 64 + 64 * 64 + 64 * 5)
        return {"bytes": case["n"] * (5 * 8 * 2 + 1 + (14 * 8 if case["start"] == "cold" else 0)), "flops": case["n"] * (steps * 900 + net)}
    if kind == "network":
        return {"bytes": case["n"] * (3 + 4) * 4, "flops": case["n"] * 2 * (3 * 20 + 20 * 20 + 20 * 4)}
    if kind == "train":
        return {"bytes": case["n"] * 10 * 8, "flops": case["n"] * 6 * (5 * 64 + 64 * 64 + 64 * 5)}
    sites = case["nx"] * case["ny"] * case["nz"]
    pore = sites * case["porosity"]
    flow, steps = case.get("flow", 0), case.get("steps", 0)
    solutes, extra, flops = {"flow": (0, 0, 0), "solute": (1, 12, 60), "carbonate": (4, 12, 1200), "biotic": (4, 20, 300),
                             "surrogate": (6, 28, 500), "coupled": (8, 28, 2500)}[kind]
    fields = {"flow": 4, "solute": 4, "carbonate": 7, "biotic": 5, "surrogate": 8, "coupled": 13}[kind]
    return {"bytes": pore * (flow * 152 + steps * (solutes * 56 + extra)) + sites * 8 * fields,
            "flops": pore * (flow * 400 + steps * (solutes * 60 + flops))}


# ---------------------------------------------------------------- FP64 restatement
W19 = [1 / 3 if d == (0, 0, 0) else 1 / 18 if abs(d[0]) + abs(d[1]) + abs(d[2]) == 1 else 1 / 36 for d in D3Q19]
D3Q7 = [(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
W7 = [0.25] + [0.125] * 6
OPP19 = [0] + [i + 9 for i in range(1, 10)] + [i - 9 for i in range(10, 19)]
OPP7 = [0, 4, 5, 6, 1, 2, 3]


def _stream(f, dirs, opp, out):
    """Push streaming of f[..., i, x, y, z] into out; a population leaving through an x end stays in its own site's
    opposite direction."""
    for i, (dx, dy, dz) in enumerate(dirs):
        src = f[..., i, :, :, :]
        src = torch.roll(src, (dy, dz), (-2, -1)) if dy or dz else src
        dst = out[..., i, :, :, :]
        if dx == 0:
            dst.copy_(src)
        elif dx > 0:
            dst[..., 1:, :, :] = src[..., :-1, :, :]
            dst[..., 0, :, :] = f[..., opp[i], 0, :, :]
        else:
            dst[..., :-1, :, :] = src[..., 1:, :, :]
            dst[..., -1, :, :] = f[..., opp[i], -1, :, :]


def _feq19(i, rb, j, jj):
    d = D3Q19[i]
    cj = sum(d[k] * j[k] for k in range(3) if d[k]) if i else torch.zeros_like(rb)
    return W19[i] * (rb + 3.0 * cj + 4.5 * cj * cj - 1.5 * jj)


def _pressure_face(f, rb, side):
    """Regularised density boundary of one x plane, f[19, y, z]: (rebuilt populations, j_x)."""
    s0 = sum(f[i] for i in range(19) if D3Q19[i][0] == 0)
    sn = sum(f[i] for i in range(19) if D3Q19[i][0] == side)
    jx = rb - s0 - 2 * sn if side < 0 else s0 + 2 * sn - rb
    z = torch.zeros_like(jx)
    j, rbt, jj = (jx, z, z), torch.full_like(jx, rb), jx * jx
    pi = [[z for _ in range(3)] for _ in range(3)]
    for i in range(19):
        if D3Q19[i][0] == -side:
            continue
        fn = (1.0 if D3Q19[i][0] == 0 else 2.0) * (f[i] - _feq19(i, rbt, j, jj))
        for a in range(3):
            for b in range(3):
                if D3Q19[i][a] and D3Q19[i][b]:
                    pi[a][b] = pi[a][b] + D3Q19[i][a] * D3Q19[i][b] * fn
    out = torch.empty_like(f)
    for i in range(19):
        q = sum((D3Q19[i][a] * D3Q19[i][b] - (1 / 3 if a == b else 0.0)) * pi[a][b] for a in range(3) for b in range(3))
        out[i] = _feq19(i, rbt, j, jj) + W19[i] * 4.5 * q
    return out, jx


class _Flow:
    def __init__(self, cfg, mat):
        self.pore, self.wall = (mat == PORE) | (mat == BIOFILM), mat == WALL
        self.om = 1.0 / cfg.tau_ns
        self.rb = (cfg.rho_in - 1.0, cfg.rho_out - 1.0)
        nx = mat.shape[0]
        rb = cfg.rho_in + (cfg.rho_out - cfg.rho_in) * torch.arange(nx, device=mat.device, dtype=F64) / (nx - 1) - 1.0
        self.f = torch.stack([self.pore * (w * rb)[:, None, None] for w in W19])
        self.tmp = torch.empty_like(self.f)

    def _faces(self, f):
        for x, side in ((0, -1), (-1, 1)):
            new, _ = _pressure_face(f[:, x], self.rb[0 if side < 0 else 1], side)
            f[:, x] = torch.where(self.pore[x], new, f[:, x])

    def _moments(self, f):
        rb = f.sum(0)
        return rb, [sum(D3Q19[i][k] * f[i] for i in range(19) if D3Q19[i][k]) for k in range(3)]

    def step(self, n):
        f, om = self.f, self.om
        for _ in range(n):
            self._faces(f)
            rb, j = self._moments(f)
            rb[0], rb[-1] = self.rb
            for k in (1, 2):
                j[k][0] = j[k][-1] = 0.0
            jj = j[0] * j[0] + j[1] * j[1] + j[2] * j[2]
            for i in range(10):
                o = OPP19[i]
                a, b = f[i], f[o]
                na = torch.where(self.pore, a * (1 - om) + om * _feq19(i, rb, j, jj), torch.where(self.wall, b, a))
                if o != i:
                    nb = torch.where(self.pore, b * (1 - om) + om * _feq19(o, rb, j, jj), torch.where(self.wall, a, b))
                    f[o] = nb
                f[i] = na
            _stream(f, D3Q19, OPP19, self.tmp)
            f, self.tmp = self.tmp, f
            self.f = f

    def macro(self):
        f = self.f.clone()
        self._faces(f)
        rb, j = self._moments(f)
        rb0 = self.f.sum(0)
        for x, v in ((0, self.rb[0]), (-1, self.rb[1])):
            rb[x] = torch.where(self.pore[x], torch.full_like(rb[x], v), rb0[x])
            for k in (1, 2):
                j[k][x] = 0.0
        return 1.0 + rb, torch.stack([torch.where(self.pore, v, torch.zeros_like(v)) for v in j])


class _Transport:
    def __init__(self, cfg, mat, u):
        self.cfg = cfg
        self.mob = [s for s in range(cfg.n_solutes) if not cfg.immobile[s]]
        dev = mat.device
        self.fluid, self.wall = (mat == PORE) | (mat == BIOFILM), mat == WALL
        col = lambda v: torch.tensor([v[s] for s in self.mob], device=dev, dtype=F64)
        self.om = col(cfg.omega_pore).view(-1, 1, 1, 1)
        c0 = col(cfg.c0)
        self.u = u
        self.g = torch.empty((len(self.mob), 7) + tuple(mat.shape), device=dev, dtype=F64)
        for i in range(7):
            self.g[:, i] = (W7[i] * c0).view(-1, 1, 1, 1)
        self.tmp = torch.empty_like(self.g)
        self.neu = [[t[s] == 1 for s in self.mob] for t in (cfg.left_type, cfg.right_type)]
        val = (col(cfg.left_value), col(cfg.right_value))
        self.face = [torch.where(torch.tensor(self.neu[k], device=dev), c0, val[k]).view(-1, 1, 1).expand(-1, *mat.shape[1:]).clone()
                     for k in range(2)]
        inner = self.fluid.clone()
        inner[0] = inner[-1] = False
        self.inner = inner.reshape(-1).nonzero().squeeze(1)
        self.imm, self.bio = {}, []

    def _adjacent(self):
        for k, x in ((0, 1), (1, -2)):
            r = self.g[:, :, x].sum(1)
            sel = torch.tensor(self.neu[k], device=r.device).view(-1, 1, 1)
            self.face[k] = torch.where(sel, r, self.face[k])

    def step(self, n, react=None):
        for _ in range(n):
            g = self.g
            for k, x, unk in ((0, 0, 4), (1, -1, 1)):
                known = g[:, :, x].sum(1) - g[:, unk, x]
                g[:, unk, x] = torch.where(self.fluid[x], self.face[k] - known, g[:, unk, x])
            rho = g.sum(1)
            add = react(self, rho) if react else None
            for i in (0, 1, 2, 3):
                o = OPP7[i]
                a, b = g[:, i], g[:, o]
                cu = sum(D3Q7[i][k] * self.u[k] for k in range(3)) if i else 0.0
                na = torch.where(self.fluid, a - self.om * (a - W7[i] * rho * (1.0 + 4.0 * cu)), torch.where(self.wall, b, a))
                if o != i:
                    nb = torch.where(self.fluid, b - self.om * (b - W7[o] * rho * (1.0 - 4.0 * cu)), torch.where(self.wall, a, b))
                    g[:, o] = nb
                g[:, i] = na
            if add is not None:
                flat = g.reshape(g.shape[0], 7, -1)
                for i in range(7):
                    flat[:, i, self.inner] += W7[i] * add
            _stream(g, D3Q7, OPP7, self.tmp)
            self.g, self.tmp = self.tmp, g
            self._adjacent()

    def conc(self, m):
        r = self.g[m].sum(0)
        for k, x in ((0, 0), (1, -1)):
            r[x] = torch.where(self.fluid[x], self.face[k][m], r[x])
        return r


def _above(d):
    return torch.where(d.abs() > THRD, d, torch.zeros_like(d))


def _kinetics(cfg, C, B):
    """dC (list) and dB of the biotic reactions of microbe 0 and its decay."""
    zero = torch.zeros_like(B)
    B = torch.where(B < THRD, zero, B)
    Cf = [torch.where(c < THRD, torch.zeros_like(c), c) for c in C]
    R, BR = [zero.clone() for _ in C], zero.clone()
    for k in range(cfg.n_rxn):
        r = cfg.rxn[k]
        if r.microbe < 0:
            continue
        rate = r.k * B
        for j in range(r.n_monod):
            c = Cf[r.monod_s[j]]
            rate = rate * (c / (r.monod_ks[j] + c))
        for s in range(len(C)):
            if r.nu[s]:
                R[s] = R[s] + r.nu[s] * rate
        BR = BR + r.yield_ * rate
    BR = BR - cfg.decay[0] * B
    return [_above(v * cfg.dt) for v in R], _above(BR * cfg.dt)


def _limited(c, eq):
    """The increment run_equilibrium_biotic applies: towards eq, at most a tenth of the concentration per step."""
    conc = c.clamp(min=1e-30)
    d = eq.clamp(1e-30, 10.0) - conc
    mx = (0.1 * conc).clamp(min=1e-9)
    d = torch.minimum(torch.maximum(d, -mx), mx)
    d = torch.where(conc + d < 1e-20, 1e-20 - conc, d)
    return _above(d)


def _root(lo, hi, fn, n=70):
    """Root of an increasing function by bisection of log10 in [lo, hi]."""
    lo, hi = lo.clone(), hi.clone()
    for _ in range(n):
        mid = 0.5 * (lo + hi)
        up = fn(10.0 ** mid) > 0
        hi = torch.where(up, mid, hi)
        lo = torch.where(up, lo, mid)
    return 10.0 ** (0.5 * (lo + hi))


def _react_carbonate(t, rho):
    C = [rho[s].reshape(-1)[t.inner] for s in range(4)]
    k2, k3 = 10.0 ** -10.33, 10.0 ** 6.35
    q = [c.clamp(1e-30, 10.0) for c in C]
    TA, TH = (q[0] + q[2] + q[3]).clamp(min=1e-30), (q[1] - q[2] + q[3]).clamp(min=1e-30)
    free = lambda h: TA / (1.0 + k2 / h + k3 * h)
    one = torch.ones_like(TA)
    h = _root(-16.0 * one, 1.0 * one, lambda h: h + free(h) * (k3 * h - k2 / h) - TH)
    a = free(h)
    return torch.stack([_limited(c, e) for c, e in zip(C, (a, h, k2 * a / h, k3 * a * h))])


def _react_biotic(t, rho):
    C = [rho[s].reshape(-1)[t.inner] for s in range(4)]
    b = t.bio[0].reshape(-1)
    d, db = _kinetics(t.cfg, C, b[t.inner])
    b[t.inner] += db
    return torch.stack(d)


def _react_coupled(t, rho):
    cfg = t.cfg
    C = [rho[s].reshape(-1)[t.inner] for s in range(8)]
    total = [torch.zeros_like(c) for c in C]
    b, mineral = t.bio[0].reshape(-1), t.imm[8].reshape(-1)
    d, db = _kinetics(cfg, C + [mineral[t.inner]], b[t.inner])
    b[t.inner] += db
    for s in range(8):
        C[s], total[s] = C[s] + d[s], total[s] + d[s]
    r = cfg.rxn[2]
    prod = C[4].clamp(min=0.0) * C[6].clamp(min=0.0)
    rate = torch.where(t.surface, r.k * (prod / r.ksp - 1.0).clamp(min=0.0), torch.zeros_like(prod))
    for s in (4, 6):
        v = _above(r.nu[s] * rate * cfg.dt)
        C[s], total[s] = C[s] + v, total[s] + v
    mineral[t.inner] += _above(r.nu[8] * rate * cfg.dt)
    # CO3-- (6), Ca++ (4), H+ (5), HCO3- (3) = k1 CO3 H, CaCO3(aq) (7) = k2 CO3 Ca
    k1, k2 = 10.0 ** 10.33, 10.0 ** 3.2
    q = [c.clamp(1e-30, 10.0) for c in C]
    TC, TCa, TH = q[6] + q[3] + q[7], q[4] + q[7], q[5] + q[3]
    ca, h = (lambda c: TCa / (1.0 + k2 * c)), (lambda c: TH / (1.0 + k1 * c))
    c3 = _root(torch.log10(TC) - 8.0, torch.log10(TC), lambda c: c * (1.0 + k1 * h(c) + k2 * ca(c)) - TC)
    # the root polished by Newton in the concentration itself
    for _ in range(2):
        f = c3 * (1.0 + k1 * h(c3) + k2 * ca(c3)) - TC
        c3 = c3 - f / (1.0 + k1 * h(c3) / (1.0 + k1 * c3) + k2 * ca(c3) / (1.0 + k2 * c3))
    eq = {6: c3, 4: ca(c3), 5: h(c3), 3: k1 * c3 * h(c3), 7: k2 * c3 * ca(c3)}
    for s in range(8):
        total[s] = total[s] + _limited(C[s], eq.get(s, C[s].clamp(1e-30, 10.0)))
    return torch.stack(total)


def _forward(net, x):
    """The network in FP64: clamp, mapminmax, tanh hidden layers, linear output, reverse mapminmax."""
    L, w = net.n_layers, list(net.widths)
    dev = x.device
    vec = lambda v, k: torch.tensor([v[i] for i in range(k)], device=dev, dtype=F64)
    p, off = torch.tensor(list(net.params), device=dev, dtype=F64), 0
    a = torch.minimum(torch.maximum(x, vec(net.x_lo, w[0])), vec(net.x_hi, w[0]))
    a = (a - vec(net.x_offset, w[0])) * vec(net.x_gain, w[0]) + net.x_ymin
    for layer in range(L):
        wi, wo = w[layer], w[layer + 1]
        a = a @ p[off:off + wi * wo].view(wo, wi).T + p[off + wi * wo:off + wi * wo + wo]
        off += wi * wo + wo
        if layer < L - 1:
            a = torch.tanh(a)
    return (a - net.y_ymin) / vec(net.y_gain, w[L]) + vec(net.y_offset, w[L])


def _react_surrogate(t, rho):
    cfg = t.cfg
    C = torch.stack([rho[s].reshape(-1)[t.inner] for s in range(6)])
    conc = torch.where(C > THRD, C, torch.zeros_like(C))
    draw_ = torch.zeros_like(C)
    for o in range(2):
        org, b = cfg.srg[o], t.bio[o].reshape(-1)
        here = t.inner[b[t.inner] > THRD]
        at = (b[t.inner] > THRD).nonzero().squeeze(1)
        bb = b[here]
        denom = bb * org.mw * cfg.dt
        fout = []
        for s in range(6):
            av = conc[s][at]
            mm = av / (org.kc[s] + av)
            cap = (av * 3.6e6 / denom).clamp(max=1e4)
            v = org.vmax[s] * mm if org.vmax[s] > THRD else cap * mm
            fout.append(torch.where((cap > 0) & (v > cap), cap, v))
        y = _forward(t.nets[o], torch.stack([conc[3 * o][at], conc[3 * o + 1][at], bb], 1))
        mu = torch.where(y[:, 0] < 1e-8, torch.zeros_like(bb), y[:, 0])
        for q in range(3):
            fout[3 * o + q] = y[:, 1 + q]
        db = torch.where(mu < THRD, -org.kd * bb * cfg.dt, mu * bb * cfg.dt / 3600.0)
        b[here] += _above(torch.maximum(db, -bb))
        for s in range(6):
            draw_[s, at] += -fout[s] * bb * org.mw * cfg.dt / 3.6e6
    return _above(torch.minimum(torch.maximum(_above(draw_), -conc), torch.zeros_like(conc)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None                    # BF16 arithmetic through many updates has no such value
    if kind == "speciation":
        return {"x": _speciation(case["n"], seed)[1].cpu(), "status": None}
    if kind == "network":
        return _forward(_nets(seed)[0], _network_inputs(case, seed).double()).cpu()
    sites = case["nx"] * case["ny"] * case["nz"]
    if sites * (case.get("flow", 0) * 19 * (kind != "coupled") + START_FLOW.get(kind, 0) * 19 + case.get("steps", 0) * 70) > 1.3e11:
        return None                    # more than some 20 seconds of dense FP64
    cfg, mat = _config(case, seed), _material(case, seed)
    flow = _Flow(cfg, mat)
    flow.step(START_FLOW[kind] if kind in START_FLOW else case["flow"])
    rho, u = flow.macro()
    del flow
    if kind == "flow":
        return {"rho": rho.cpu(), "u0": u[0].cpu(), "u1": u[1].cpu(), "u2": u[2].cpu()}
    t = _Transport(cfg, mat, u)
    t.bio = _biomass(case, mat, seed)
    if kind == "coupled":
        t.imm[8] = _seeded(mat, seed + 77, 0.5, 0.0, 1.0)
        t.surface = _wall_adjacent(mat).reshape(-1)[t.inner]
    if kind == "surrogate":
        t.nets = _nets(seed)
    t.step(case["steps"], {"solute": None, "carbonate": _react_carbonate, "biotic": _react_biotic, "coupled": _react_coupled,
                           "surrogate": _react_surrogate}[kind])
    out = {"c%d" % s: t.conc(m).cpu() for m, s in enumerate(t.mob)}
    out.update({"biomass%d" % m: b.cpu() for m, b in enumerate(t.bio)})
    if kind in ("biotic", "coupled"):
        out["mask"] = None
    if kind == "coupled":
        out.update({"c8": t.imm[8].cpu(), "u0": None, "u1": None, "u2": None})    # the velocity follows the conversions
    if kind in ("solute", "carbonate"):
        out.update({"u%d" % k: u[k].cpu() for k in range(3)})
    return out
