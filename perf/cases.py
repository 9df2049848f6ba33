"""Timed workloads of the short-range force-and-integrate path.

Five families, each through the entry points a program calls:

* ``md``: ``Simulation.run`` for a number of timesteps, then the state read back on
  the device (``azp_md_get_state``), which is what a coupled analysis or a logger does
  between runs. Systems: ``fluid`` (PerturbedLennardJones, LangevinFlow), ``melt``
  (WCA beads and Quartic bonds, LangevinFlow in a ParabolicFlow), ``colloid``
  (two-type Colloid mixture, BrownianFlow) and ``dpd`` (DPDGeneralWeight,
  ConstantVolume). Each pass goes on from the state the last one left.
* ``step``: the drop-in drivers as a host code calls them: one ``azp_nlist_build``, then
  a few timesteps of ``azp_langevin_step1``, ``azp_pair_forces`` (plus
  ``azp_bond_forces`` for the melt) and ``azp_langevin_step2``.
* ``dpd``: one ``azp_dpd_forces`` call over a list the program keeps.
* ``batch``: ``ReplicaBatch.run`` over uneven ExpandedYukawa replicas, arrays read back.
* ``grad``: ``autodiff.pair_forces`` and its backward pass.

Every input is generated here from the seed: jittered lattices (fluids and the
colloids' solvent), chains threaded along a lattice (melt), uniform random beads
(DPD), with Maxwell-Boltzmann velocities.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

F64 = torch.float64
DT = 0.005
CHAIN = 100
QUARTIC = dict(k=1434.3, r_0=1.5, b_1=-0.7589, b_2=0.0, U_0=67.2234, sigma=1.0, epsilon=1.0, delta=0.0)
WCA_RCUT = 2.0 ** (1.0 / 6.0)
# two particle types: the second a little larger, the cross term between
FLUID_SIGMA = ((1.0, 1.05), (1.05, 1.1))
DPD_PARAMS = {(0, 0): (25.0, 4.5, 0.5), (0, 1): (30.0, 4.5, 1.0), (1, 1): (25.0, 4.5, 2.0)}
COLLOID = {(0, 0): (144.0, 0.0, 0.0, 3.0), (0, 1): (100.0, 0.0, 2.5, 6.0), (1, 1): (40.0, 2.5, 2.5, 10.0)}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest fluid of the benchmark suite in the default precision: launches and latency count
        dict(name="md_fluid_4k_fp64", family="md", system="fluid", n=4096, precision="fp64", types=1, mode="none", steps=50),
        # the same fluid with FP32 forces, the production precision
        dict(name="md_fluid_4k_fp32", family="md", system="fluid", n=4096, precision="fp32", types=1, mode="none", steps=50),
        # an ordinary two-type fluid in the default precision
        dict(name="md_fluid_55k_fp64", family="md", system="fluid", n=54872, precision="fp64", types=2, mode="shift", steps=10),
        # the headline melt: 10,486 chains of 100 beads, FP32 forces
        dict(name="md_melt_1m_fp32", family="md", system="melt", n=1048600, precision="fp32", types=1, mode="none", steps=20),
        # a melt of ordinary size in the default precision
        dict(name="md_melt_131k_fp64", family="md", system="melt", n=131300, precision="fp64", types=1, mode="none", steps=20),
        # colloids and solvent, disparate cutoffs, Brownian dynamics
        dict(name="md_colloid_66k_fp32", family="md", system="colloid", n=65537, precision="fp32", types=2, mode="shift", steps=10),
        # a DPD fluid thermostatted by its pair force
        dict(name="md_dpd_250k_fp32", family="md", system="dpd", n=250007, precision="fp32", types=2, mode="none", steps=20),
        # many small systems advanced together
        dict(name="batch_yukawa_48", family="batch", n=48, layout=4, precision="fp32", steps=20),
        # a host code that drives the path call by call in double precision
        dict(name="step_fluid_104k_fp64", family="step", system="fluid", n=103823, precision="fp64", types=2, mode="shift", steps=5),
        # the same for the large melt with FP32 forces
        dict(name="step_melt_1m_fp32", family="step", system="melt", n=1048600, precision="fp32", types=1, mode="none", steps=5),
        # DPD forces of one timestep in double precision
        dict(name="dpd_forces_262k_fp64", family="dpd", n=262144, precision="fp64", types=2),
        # forces and their gradients for parameter learning
        dict(name="grad_fluid_66k", family="grad", n=65536, mode="shift"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["md", "md", "md", "step", "step", "dpd", "batch", "grad"])
    precision = rng.choice(["fp64", "fp32"])
    if family == "batch":
        return dict(family="batch", n=rng.randint(8, 48 if precision == "fp32" else 16), layout=rng.randrange(1000),
                    precision=precision, steps=rng.randint(10, 20))
    if family == "dpd":
        return dict(family="dpd", n=_log_int(rng, 4000, 400000), precision=precision, types=rng.randint(1, 2))
    if family == "grad":
        return dict(family="grad", n=_log_int(rng, 2000, 65536), mode=rng.choice(["none", "shift", "xplor"]))
    system = rng.choice(["fluid", "melt", "colloid", "dpd"] if family == "md" else ["fluid", "melt"])
    types, mode, steps = 1, "none", rng.randint(10, 20) if family == "md" else rng.randint(3, 5)
    if system == "fluid":
        n = _log_int(rng, 1000, 110000)
        types, mode = rng.randint(1, 2), rng.choice(["none", "shift", "xplor"])
    elif system == "melt":
        n = CHAIN * _log_int(rng, 20, 10486 if precision == "fp32" else 1500)
    elif system == "colloid":
        n, types, mode, steps = _log_int(rng, 8000, 66000), 2, "shift", rng.randint(5, 10)
    else:
        n, types = _log_int(rng, 4000, 250000 if precision == "fp32" else 60000), 2
    return dict(family=family, system=system, n=n, precision=precision, types=types, mode=mode, steps=steps)


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _wrap(x, L):
    img = torch.floor(x / L + 0.5)
    x = x - img * L
    for lo, s in ((-0.5 * L, 1.0), (0.5 * L, -1.0)):
        out = (x < lo) if s > 0 else (x >= lo)
        x = torch.where(out, x + s * L, x)
        img = torch.where(out, img - s, img)
    return x, img.to(torch.int32)


def _lattice(m, L, gen, jitter):
    g = (torch.arange(m, dtype=F64, device="cuda") + 0.5) * (L / m) - 0.5 * L
    x = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), dim=-1).reshape(-1, 3)
    return x + (2.0 * torch.rand(x.shape, generator=gen, dtype=F64, device="cuda") - 1.0) * jitter


def _velocities(n, gen):
    v = torch.randn((n, 3), generator=gen, dtype=F64, device="cuda")
    return v - v.mean(dim=0)


def _fluid(n, types, gen, density=0.8, jitter=0.05):
    m = math.ceil(round(n ** (1.0 / 3.0), 9))
    L = (n / density) ** (1.0 / 3.0)
    sites = torch.randperm(m ** 3, generator=gen, device="cuda")[:n]
    x, img = _wrap(_lattice(m, L, gen, jitter)[sites], L)
    typ = torch.randint(0, types, (n,), generator=gen, device="cuda")
    return dict(L=L, x=x, img=img, typ=typ, v=_velocities(n, gen), types=types)


def _melt(n, gen, density=0.85):
    # chains follow a boustrophedon path through the lattice, so that every bond is one lattice spacing;
    # which stretch of the path a chain takes is random
    m = math.ceil(round(n ** (1.0 / 3.0), 9))
    L = (n / density) ** (1.0 / 3.0)
    s = torch.arange(n, device="cuda")
    z, r = s // (m * m), s % (m * m)
    y, q = r // m, r % m
    y = torch.where(z % 2 == 1, m - 1 - y, y)
    q = torch.where((s // m) % 2 == 1, m - 1 - q, q)
    x = (torch.stack([q, y, z], dim=1).to(F64) + 0.5) * (L / m) - 0.5 * L
    x = x.reshape(-1, CHAIN, 3)[torch.randperm(n // CHAIN, generator=gen, device="cuda")].reshape(n, 3)
    x = x + (2.0 * torch.rand(x.shape, generator=gen, dtype=F64, device="cuda") - 1.0) * 0.05
    x, img = _wrap(x, L)
    i = torch.arange(n, device="cuda").reshape(-1, CHAIN)
    bonds = torch.stack([i[:, :-1].reshape(-1), i[:, 1:].reshape(-1)], dim=1)
    return dict(L=L, x=x, img=img, typ=torch.zeros(n, dtype=torch.int64, device="cuda"), v=_velocities(n, gen), types=1,
                bonds=bonds)


def _colloid(n, gen):
    # 4 % colloids of diameter 5 at a volume fraction of 0.3, on a jittered lattice with surface gaps of at
    # least 0.4; solvent on a jittered grid outside their shells
    nc = max(1, round(0.04 * n))
    L = ((math.pi / 6.0) * (nc * 125.0 + (n - nc)) / 0.3) ** (1.0 / 3.0)
    m = math.ceil(round(nc ** (1.0 / 3.0), 9))
    jit = 0.5 * (L / m - 5.0 - 0.4)
    if jit < 0.0:
        raise ValueError("colloid lattice too tight")
    slot = torch.full((m ** 3,), -1, dtype=torch.int64, device="cuda")
    slot[torch.randperm(m ** 3, generator=gen, device="cuda")[:nc]] = torch.arange(nc, device="cuda")
    sites = _lattice(m, L, gen, jit)
    col = torch.empty((nc, 3), dtype=F64, device="cuda")
    col[slot[slot >= 0]] = sites[slot >= 0]
    k = int(L // 1.1)
    pts = _lattice(k, L, gen, 0.04 * L / k)
    home = ((pts / L + 0.5) * m).floor().to(torch.int64) % m
    keep = torch.ones(len(pts), dtype=torch.bool, device="cuda")
    for o in np.ndindex(3, 3, 3):
        c = (home + torch.tensor(o, device="cuda") - 1) % m
        s = slot[(c[:, 0] * m + c[:, 1]) * m + c[:, 2]]
        d = pts - col[s.clamp(min=0)]
        d = d - L * torch.round(d / L)
        keep &= (s < 0) | ((d * d).sum(dim=1) >= 3.5 ** 2)
    pts = pts[keep]
    pts = pts[torch.randperm(len(pts), generator=gen, device="cuda")[: n - nc]]
    x, img = _wrap(torch.cat([pts, col]), L)
    typ = (torch.arange(len(x), device="cuda") >= len(pts)).to(torch.int64)
    return dict(L=L, x=x, img=img, typ=typ, v=_velocities(len(x), gen), types=2,
                diameter=torch.where(typ == 1, 5.0, 1.0).to(F64))


def _dpd(n, types, gen):
    L = (n / 3.0) ** (1.0 / 3.0)
    x = (torch.rand((n, 3), generator=gen, dtype=F64, device="cuda") - 0.5) * L
    typ = torch.randint(0, types, (n,), generator=gen, device="cuda")
    return dict(L=L, x=x, img=torch.zeros((n, 3), dtype=torch.int32, device="cuda"), typ=typ, v=_velocities(n, gen),
                types=types)


def _system(case, seed):
    gen = _gen(seed)
    system = "dpd" if case["family"] == "dpd" else "fluid" if case["family"] == "grad" else case["system"]
    if system == "fluid":
        return _fluid(case["n"], case.get("types", 1), gen)
    if system == "melt":
        return _melt(case["n"], gen)
    if system == "colloid":
        return _colloid(case["n"], gen)
    return _dpd(case["n"], case["types"], gen)


def _replicas(case, seed):
    # particle numbers log-uniform in [500, 20000], as uneven as the batched benchmark's; the sizes and
    # potentials belong to the case, the configurations to the seed
    rng = np.random.Generator(np.random.PCG64(case["layout"]))
    gen = _gen(seed)
    reps = []
    for _ in range(case["n"]):
        n = int(round(math.exp(rng.uniform(math.log(500), math.log(20000)))))
        rho = rng.uniform(0.3, 0.8)
        closest = 0.9 * (n / rho) ** (1.0 / 3.0) / math.ceil(n ** (1.0 / 3.0))
        while True:
            kappa, delta = rng.uniform(0.5, 3.0), rng.uniform(0.0, 1.0)
            r_cut = delta + 5.0 / kappa
            if (n / rho) ** (1.0 / 3.0) >= 2.0 * (r_cut + 0.4) and delta <= closest - 0.25:
                break
        s = _fluid(n, 1, gen, density=rho, jitter=0.05 * (n / rho) ** (1.0 / 3.0) / math.ceil(n ** (1.0 / 3.0)))
        s.update(kappa=kappa, delta=delta, r_cut=r_cut)
        reps.append(s)
    return reps


def _np(t):
    return t.cpu().numpy()


def _snapshot(s):
    import azplugins_gb300 as az

    snap = az.Snapshot(len(s["x"]))
    p = snap.particles
    p.types = ["A", "B"][: s["types"]]
    p.position, p.velocity, p.image = _np(s["x"]), _np(s["v"]), _np(s["img"])
    p.typeid = _np(s["typ"]).astype(np.int32)
    p.acceleration = np.zeros((len(s["x"]), 3))
    if "diameter" in s:
        p.diameter = _np(s["diameter"])
    snap.configuration.box = [s["L"]] * 3 + [0.0, 0.0, 0.0]
    if "bonds" in s:
        snap.resize_bonds(len(s["bonds"]))
        snap.bonds.types = ["A-A"]
        snap.bonds.group = _np(s["bonds"])
    return snap


def _pair(case):
    """The case's pair potential object."""
    import azplugins_gb300 as az

    system = "dpd" if case["family"] == "dpd" else "fluid" if case["family"] == "grad" else case["system"]
    names = ["A", "B"]
    if system == "dpd":
        pot = az.pair.DPDGeneralWeight(nlist=az.nlist.Cell(buffer=0.3), kT=1.0, default_r_cut=1.0)
        for (a, b), (A, gamma, s) in DPD_PARAMS.items():
            pot.params[(names[a], names[b])] = dict(A=A, gamma=gamma, s=s)
    elif system == "colloid":
        pot = az.pair.Colloid(nlist=az.nlist.Cell(buffer=0.4), mode=case["mode"])
        for (a, b), (A, a1, a2, rc) in COLLOID.items():
            pot.params[(names[a], names[b])] = dict(A=A, a_1=a1, a_2=a2, sigma=1.0)
            pot.r_cut[(names[a], names[b])] = rc
    elif system == "melt":
        pot = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=WCA_RCUT)
        pot.params[("A", "A")] = dict(epsilon=1.0, sigma=1.0, attraction_scale_factor=0.0)
    else:
        pot = az.pair.PerturbedLennardJones(nlist=az.nlist.Cell(buffer=0.4), default_r_cut=3.0, default_r_on=2.5,
                                            mode=case["mode"])
        for a in range(2):
            for b in range(a, 2):
                pot.params[(names[a], names[b])] = dict(epsilon=1.0, sigma=FLUID_SIGMA[a][b], attraction_scale_factor=0.5)
    return pot


# ---------------------------------------------------------------- prepare and run
def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    return {"md": _prepare_md, "step": _prepare_step, "dpd": _prepare_dpd, "batch": _prepare_batch,
            "grad": _prepare_grad}[case["family"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_md(case, seed):
    import azplugins_gb300 as az

    s = _system(case, seed)
    N = len(s["x"])
    forces = [_pair(case)]
    if case["system"] == "melt":
        bond = az.bond.Quartic()
        bond.params["A-A"] = QUARTIC
        forces.append(bond)
    dt = DT
    if case["system"] == "colloid":
        dt = 0.001
        method = az.methods.BrownianFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.1, 0.0, 0.0)), alpha=10.0)
    elif case["system"] == "dpd":
        method = az.methods.ConstantVolume("all")
    elif case["system"] == "melt":
        method = az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ParabolicFlow(mean_velocity=2.0 / 3.0,
                                                                                         separation=s["L"]))
    else:
        method = az.methods.LangevinFlow("all", kT=1.0, flow_field=az.flow.ConstantFlow((0.0, 0.0, 0.0)))
    sim = az.Simulation(seed=seed & 0xFFFF, precision=case["precision"])
    sim.create_state_from_snapshot(_snapshot(s))
    sim.operations.integrator = az.md.Integrator(dt=dt, methods=[method], forces=forces)
    sim.run(1)  # the engine with its list and graphs is what a program keeps
    out = dict(pos=torch.empty((N, 4), dtype=F64, device="cuda"), vel=torch.empty((N, 4), dtype=F64, device="cuda"),
               acc=torch.empty((N, 3), dtype=F64, device="cuda"), img=torch.empty((N, 3), dtype=torch.int32, device="cuda"))
    return dict(run=_run_md, sim=sim, steps=case["steps"], out=out)


def _run_md(st):
    from azplugins_gb300 import _lib

    sim, o = st["sim"], st["out"]
    sim.run(st["steps"])
    _lib.check(_lib.load().azp_md_get_state(sim._engine._md, o["pos"].data_ptr(), o["vel"].data_ptr(), o["acc"].data_ptr(),
                                            o["img"].data_ptr(), None, 1, _stream()), "azp_md_get_state")
    return o


def _device_system(s):
    from azplugins_gb300 import _lib

    N = len(s["x"])
    pos = torch.zeros((N, 4), dtype=F64, device="cuda")
    pos[:, :3] = s["x"]
    pos.view(torch.int64)[:, 3] = s["typ"]
    vel = torch.ones((N, 4), dtype=F64, device="cuda")
    vel[:, :3] = s["v"]
    acc = torch.zeros((N, 3), dtype=F64, device="cuda")
    img = s["img"].clone()
    tag = torch.arange(N, dtype=torch.int32, device="cuda")
    sysd = _lib.System()
    sysd.N, sysd.ntypes = N, s["types"]
    sysd.pos, sysd.vel, sysd.accel, sysd.image, sysd.tag = (t.data_ptr() for t in (pos, vel, acc, img, tag))
    for d in range(3):
        sysd.box.L[d] = s["L"]
    return sysd, dict(pos=pos, vel=vel, acc=acc, img=img, tag=tag)


def _force_buffers(N, precision):
    from azplugins_gb300 import _lib

    dt = torch.float32 if precision == "fp32" else F64
    force, vir = torch.zeros((N, 4), dtype=dt, device="cuda"), torch.zeros((6, N), dtype=dt, device="cuda")
    out = _lib.Forces()
    out.force, out.virial, out.virial_pitch = force.data_ptr(), vir.data_ptr(), N
    out.precision = _lib.FP32 if precision == "fp32" else _lib.FP64
    return force, vir, out


def _prepare_step(case, seed):
    from azplugins_gb300 import _compute, _lib
    import azplugins_gb300 as az

    s = _system(case, seed)
    N = len(s["x"])
    pot = _pair(case)
    rec, rc, ro = pot._tables(["A", "B"][: s["types"]])
    sysd, arrays = _device_system(s)
    force, vir, out = _force_buffers(N, case["precision"])
    st = dict(run=_run_step, sysd=sysd, arrays=arrays, force=force, vir=vir, out=out, steps=case["steps"], t=0,
              seed=seed & 0xFFFF, kind=pot.kind, mode=_lib.MODES[case["mode"]],
              tables=[torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (rec, rc, ro)],
              gamma=torch.ones(s["types"], dtype=F64, device="cuda"), bonds=None)
    excl = None
    if case["system"] == "melt":
        # bond table [height][N][2] and exclusions of linear chains
        i = torch.arange(N, device="cuda")
        first, last = i % CHAIN == 0, i % CHAIN == CHAIN - 1
        n = (2 - first.to(torch.int32) - last.to(torch.int32)).to(torch.int32)
        table = torch.zeros((2, N, 2), dtype=torch.int32, device="cuda")
        table[0, :, 0] = torch.where(first, i + 1, i - 1)
        table[1, :, 0] = torch.where(first | last, torch.zeros_like(i), i + 1)
        bond = az.bond.Quartic()
        bond.params["A-A"] = QUARTIC
        st["bonds"] = (n, table, torch.from_numpy(bond._table(["A-A"]).reshape(-1)).cuda(),
                       torch.zeros(1, dtype=torch.int32, device="cuda"))
        start = np.zeros(N + 1, dtype=np.uint32)
        start[1:] = np.cumsum(_np(n))
        both = torch.stack([i - 1, i + 1], dim=1)
        ok = torch.stack([~first, ~last], dim=1)
        excl = (start, np.ascontiguousarray(_np(both[ok])).astype(np.uint32))
    st["nl"] = _compute.NeighborList(N, s["types"], rc, 0.4, excl)
    flow = az.flow.ParabolicFlow(mean_velocity=2.0 / 3.0, separation=s["L"]) if case["system"] == "melt" \
        else az.flow.ConstantFlow((0.0, 0.0, 0.0))
    st["flow"] = flow._record()
    return st


def _run_step(st):
    from azplugins_gb300 import _lib

    L, s, sysd, p = _lib.load(), _stream(), ctypes.byref(st["sysd"]), st["tables"]
    N, out = st["sysd"].N, ctypes.byref(st["out"])
    st["nl"].build(st["sysd"])
    for _ in range(st["steps"]):
        _lib.check(L.azp_langevin_step1(sysd, None, N, DT, s), "azp_langevin_step1")
        _lib.check(L.azp_pair_forces(sysd, st["nl"].handle, st["kind"], p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(),
                                     st["mode"], out, s), "azp_pair_forces")
        if st["bonds"] is not None:
            n, table, params, err = st["bonds"]
            _lib.check(L.azp_bond_forces(sysd, n.data_ptr(), table.data_ptr(), 2, _lib.BOND_KINDS["Quartic"],
                                         params.data_ptr(), 1, out, err.data_ptr(), s), "azp_bond_forces")
        _lib.check(L.azp_langevin_step2(sysd, None, N, st["force"].data_ptr(), st["out"].precision, st["gamma"].data_ptr(),
                                        0, 0.0, st["flow"], DT, 1.0, st["t"], st["seed"], 0, s), "azp_langevin_step2")
        st["t"] += 1
    a = st["arrays"]
    return dict(pos=a["pos"][:, :3], vel=a["vel"], acc=a["acc"], img=a["img"], force=st["force"], virial=st["vir"])


def _prepare_dpd(case, seed):
    from azplugins_gb300 import _compute

    s = _system(case, seed)
    rec, rc, _ = _pair(case)._tables(["A", "B"][: s["types"]])
    sysd, arrays = _device_system(s)
    force, vir, out = _force_buffers(len(s["x"]), case["precision"])
    nl = _compute.NeighborList(len(s["x"]), s["types"], rc, 0.3)
    nl.build(sysd)
    return dict(run=_run_dpd, sysd=sysd, arrays=arrays, force=force, vir=vir, out=out, nl=nl, seed=seed & 0xFFFF,
                tables=[torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (rec, rc)])


def _run_dpd(st):
    from azplugins_gb300 import _lib

    _lib.check(_lib.load().azp_dpd_forces(ctypes.byref(st["sysd"]), st["nl"].handle, st["tables"][0].data_ptr(),
                                          st["tables"][1].data_ptr(), 1.0, DT, 7, st["seed"], ctypes.byref(st["out"]),
                                          _stream()), "azp_dpd_forces")
    return dict(force=st["force"], virial=st["vir"])


def _prepare_batch(case, seed):
    import azplugins_gb300 as az
    from azplugins_gb300.batch import ReplicaBatch

    reps = _replicas(case, seed)
    b = ReplicaBatch([_snapshot(r) for r in reps], az.pair.ExpandedYukawa,
                     [dict(epsilon=1.0, kappa=r["kappa"], delta=r["delta"]) for r in reps], [r["r_cut"] for r in reps],
                     [100 + k for k in range(len(reps))], dt=0.002, precision=case["precision"])
    b.run(1)  # list and graphs, which a program keeps
    return dict(run=_run_batch, batch=b, steps=case["steps"])


def _run_batch(st):
    st["batch"].run(st["steps"])
    pos, vel, acc, img = st["batch"].get_arrays()
    return dict(pos=pos, vel=vel, acc=acc, img=img)


def _prepare_grad(case, seed):
    from azplugins_gb300 import autodiff

    s = _system(case, seed)
    ctx = autodiff.Context(_pair(case), ["A"], _np(s["typ"]), [s["L"]] * 3, 3.0, r_on=2.5)
    gen = _gen(seed + 1)
    x = s["x"].clone().requires_grad_(True)
    vals = torch.tensor([1.0, 1.0, 0.5], dtype=F64, device="cuda", requires_grad=True)
    gF = torch.randn((len(x), 3), generator=gen, dtype=F64, device="cuda")
    gU = torch.randn(len(x), generator=gen, dtype=F64, device="cuda")
    return dict(run=_run_grad, x=x, vals=vals, ctx=ctx, gF=gF, gU=gU)


def _run_grad(st):
    from azplugins_gb300 import autodiff

    F, U = autodiff.pair_forces(st["x"], st["vals"], st["ctx"])
    gx, gv = torch.autograd.grad((F, U), (st["x"], st["vals"]), (st["gF"], st["gU"]))
    return dict(F=F.detach(), U=U.detach(), gx=gx, gv=gv)


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    # pairs inside the cutoff per particle (each pair once) and floating operations per pair
    if case["family"] == "batch":
        n, pairs, ops, steps = 5280.0 * case["n"], 60.0, 45.0, case["steps"]
    else:
        n, steps = float(case["n"]), case.get("steps", 1)
        system = "dpd" if case["family"] == "dpd" else "fluid" if case["family"] == "grad" else case["system"]
        pairs, ops = {"fluid": (45.0, 35.0), "melt": (2.2, 60.0), "colloid": (60.0, 60.0), "dpd": (6.3, 60.0)}[system]
    state = 100.0  # position, velocity, acceleration and image of a particle
    wide = 4.0 if case.get("precision") == "fp32" else 8.0
    if case["family"] == "dpd":
        return dict(bytes=n * (68.0 + 10.0 * wide), flops=n * pairs * ops)
    if case["family"] == "grad":
        return dict(bytes=n * 8.0 * (3 + 4 + 4 + 3), flops=n * pairs * ops * 3.0)
    extra = 10.0 * wide if case["family"] == "step" else 0.0
    return dict(bytes=n * (2.0 * state + extra), flops=n * steps * (pairs * ops + 80.0))


# ---------------------------------------------------------------- 64-bit results
def _near(x, L, r):
    """Pairs i < j or j < i, each once, with |min image| < r; the box is a cube."""
    N, m = len(x), int(L // r)
    if m < 3:
        i, j = torch.triu_indices(N, N, 1, device="cuda")
        d = x[i] - x[j]
        d = d - L * torch.round(d / L)
        k = (d * d).sum(dim=1) < r * r
        return i[k], j[k]
    m = min(m, 200)
    c = ((x / L + 0.5) * m).floor().to(torch.int64) % m
    cell = (c[:, 2] * m + c[:, 1]) * m + c[:, 0]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=m ** 3)
    start = torch.cumsum(count, 0) - count
    ii, jj = [], []
    for o in [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dz, dy, dx) >= (0, 0, 0)]:
        q = (c + torch.tensor(o, device="cuda")) % m
        q = (q[:, 2] * m + q[:, 1]) * m + q[:, 0]
        for a in range(0, N, 200000):
            qa = q[a:a + 200000]
            n = count[qa]
            own = torch.arange(a, a + len(qa), device="cuda")
            i = torch.repeat_interleave(own, n)
            first = torch.repeat_interleave(start[qa] - (torch.cumsum(n, 0) - n), n)
            j = order[first + torch.arange(len(i), device="cuda")]
            if o == (0, 0, 0):
                k = i < j
                i, j = i[k], j[k]
            d = x[i] - x[j]
            d = d - L * torch.round(d / L)
            k = (d * d).sum(dim=1) < r * r
            ii.append(i[k])
            jj.append(j[k])
    return torch.cat(ii), torch.cat(jj)


def _table(rows, ti, tj):
    """rows[(a, b)] (a <= b) as one tensor per column, by the types of each pair."""
    t = torch.zeros((2, 2, len(next(iter(rows.values())))), dtype=F64, device="cuda")
    for (a, b), v in rows.items():
        t[a, b] = t[b, a] = torch.tensor(v, dtype=F64)
    return t[ti, tj].unbind(dim=-1)


def _lj(r2, eps, sig, lam):
    s6 = sig ** 6
    x = 1.0 / r2
    x6 = x * x * x
    f = 4.0 * eps * x * x6 * (12.0 * s6 * s6 * x6 - 6.0 * s6)
    u = 4.0 * eps * x6 * (s6 * s6 * x6 - s6)
    core = r2 < 2.0 ** (1.0 / 3.0) * sig * sig
    return torch.where(core, f, lam * f), torch.where(core, u + eps * (1.0 - lam), lam * u)


def _yukawa(r2, kappa, delta):
    r = torch.sqrt(r2)
    u = torch.exp(-kappa * (r - delta)) / (r - delta)
    return u * (kappa + 1.0 / (r - delta)) / r, u


def _colloid_pair(r2, A, a1, a2):
    """Force / r and energy of the three forms (sigma = 1)."""
    r = torch.sqrt(r2)
    x6 = 1.0 / (r2 * r2 * r2)
    f = A / 36.0 * (12.0 * x6 * x6 - 6.0 * x6) / r2
    u = A / 36.0 * (x6 * x6 - x6)
    one, two = (a1 == 0.0) != (a2 == 0.0), (a1 != 0.0) & (a2 != 0.0)
    a = torch.maximum(a1, a2)
    d = torch.where(one, a * a - r2, torch.ones_like(r2))
    pre = A * a ** 3 / d ** 3
    poly = 2.0 * (a * a + r2) * (5.0 * a ** 4 + 22.0 * a * a * r2 + 5.0 * r2 * r2)
    f1 = 4.0 / 15.0 * pre * (poly / d ** 6 - 5.0) / d
    u1 = 2.0 / 9.0 * pre * (1.0 - (a ** 6 / 3.0 + 3.0 * a ** 4 * r2 + 4.2 * a * a * r2 * r2 + r2 ** 3) / d ** 6)
    f, u = torch.where(one, f1, f), torch.where(one, u1, u)
    # sphere and sphere: the attractive and repulsive parts, the force as the derivative of the energy
    i = two.nonzero().squeeze(1)
    rr = r[i].clone().requires_grad_(True)
    with torch.enable_grad():
        b1, b2, H = a1[i], a2[i], A[i]
        S, D, P = b1 + b2, b1 - b2, b1 * b2
        w1, w2 = rr * rr - S * S, rr * rr - D * D
        att = -H / 6.0 * (2.0 * P / w1 + 2.0 * P / w2 + torch.log(w1 / w2))
        rep = H / 37800.0 / rr * ((rr * rr - 7.0 * rr * S + 6.0 * (b1 * b1 + 7.0 * P + b2 * b2)) / (rr - S) ** 7
                                  + (rr * rr + 7.0 * rr * S + 6.0 * (b1 * b1 + 7.0 * P + b2 * b2)) / (rr + S) ** 7
                                  - (rr * rr + 7.0 * rr * D + 6.0 * (b1 * b1 - 7.0 * P + b2 * b2)) / (rr + D) ** 7
                                  - (rr * rr - 7.0 * rr * D + 6.0 * (b1 * b1 - 7.0 * P + b2 * b2)) / (rr - D) ** 7)
        e = att + rep
        (g,) = torch.autograd.grad(e.sum(), rr) if len(i) else (torch.zeros_like(rr),)
    return f.index_put((i,), -(g / rr).detach()), u.index_put((i,), e.detach())


def _quartic(r2):
    q = QUARTIC
    f, u = _lj(r2, 1.0, 1.0, 0.0)
    core = r2 < 2.0 ** (1.0 / 3.0)
    f, u = torch.where(core, f, 0.0), torch.where(core, u, 0.0)
    r = torch.sqrt(r2)
    y = r - q["r_0"]
    b1, b2 = q["b_1"], q["b_2"]
    g = -q["k"] * y * (4.0 * y * y - 3.0 * (b1 + b2) * y + 2.0 * b1 * b2) / r
    w = q["k"] * (y - b1) * (y - b2) * y * y
    return f + torch.where(y < 0.0, g, 0.0), u + torch.where(y < 0.0, w, 0.0) + q["U_0"]


def _philox(k0, k1, c0, c1, c2):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    M = 0xFFFFFFFF
    c = [c0, c1, c2, torch.zeros_like(c1)]
    for _ in range(10):
        p, q = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((q >> 32) & M) ^ c[1] ^ k0, q & M, ((p >> 32) & M) ^ c[3] ^ k1, p & M]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c


def _open01(hi, lo):
    return ((hi << 21 | lo >> 11).to(F64) + 0.5) * 2.0 ** -53


def _noise(stream, t, seed, tags, c):
    z = torch.zeros_like(tags)
    key = stream << 24 | (seed & 0xFFFF) << 8
    a, b = _philox(key, t, z, tags, z), _philox(key, t, z + 1, tags, z)
    return (2.0 * torch.stack([_open01(a[0], a[1]), _open01(a[2], a[3]), _open01(b[0], b[1])], dim=1) - 1.0) * c


def _forces(s, kind, mode, x, v=None, t=0, seed=0, dt=DT):
    """(F, U, virial [6, N]) of the system's pair force, and of its bonds."""
    N, L, typ = len(x), s["L"], s["typ"]
    F, U = torch.zeros((N, 3), dtype=F64, device="cuda"), torch.zeros(N, dtype=F64, device="cuda")
    W = torch.zeros((6, N), dtype=F64, device="cuda")

    def add(i, j, d, f, fv, u):
        F.index_add_(0, i, d * f[:, None])
        F.index_add_(0, j, -d * f[:, None])
        for e in (i, j):
            U.index_add_(0, e, 0.5 * u)
            for k, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
                W[k].index_add_(0, e, 0.5 * fv * d[:, a] * d[:, b])

    rmax = {"fluid": 3.0, "melt": WCA_RCUT, "colloid": 10.0, "dpd": 1.0, "yukawa": s.get("r_cut")}[kind]
    pi, pj = _near(x, L, rmax)
    for a in range(0, len(pi), 1 << 24):
        i, j = pi[a:a + (1 << 24)], pj[a:a + (1 << 24)]
        if kind == "melt":
            k = ((i - j).abs() != 1) | (i // CHAIN != j // CHAIN)
            i, j = i[k], j[k]
        elif kind == "colloid":
            (rc,) = _table({k: v_[3:] for k, v_ in COLLOID.items()}, typ[i], typ[j])
            d = x[i] - x[j]
            d = d - L * torch.round(d / L)
            k = (d * d).sum(dim=1) < rc * rc
            i, j = i[k], j[k]
        d = x[i] - x[j]
        d = d - L * torch.round(d / L)
        r2 = (d * d).sum(dim=1)
        if kind == "dpd":
            A, gamma, w = _table(DPD_PARAMS, typ[i], typ[j])
            r = torch.sqrt(r2)
            q = (1.0 - r).clamp(min=0.0)
            lo, hi = torch.minimum(i, j), torch.maximum(i, j)
            word = _philox(200 << 24 | (seed & 0xFFFF) << 8, t, torch.zeros_like(lo), lo, hi)
            alpha = 2.0 * _open01(word[0], word[1]) - 1.0
            fc = A * (1.0 / r - 1.0)
            dot = (d * (v[i] - v[j])).sum(dim=1)
            f = fc - gamma * q ** w * dot / r2 + torch.sqrt(6.0 * gamma / dt) * q ** (0.5 * w) * alpha / r
            add(i, j, d, f, fc, A * (1.0 - r) - 0.5 * A * (1.0 - r2))
            continue
        rc = None
        if kind == "fluid":
            (sig,) = _table({(0, 0): (1.0,), (0, 1): (FLUID_SIGMA[0][1],), (1, 1): (FLUID_SIGMA[1][1],)}, typ[i], typ[j])

            def ev(q):
                return _lj(q, 1.0, sig, 0.5)

            rc = torch.full_like(r2, 9.0)
        elif kind == "melt":
            def ev(q):
                return _lj(q, 1.0, 1.0, 0.0)
        elif kind == "yukawa":
            def ev(q):
                return _yukawa(q, s["kappa"], s["delta"])
        else:
            cA, c1, c2, cr = _table(COLLOID, typ[i], typ[j])

            def ev(q):
                return _colloid_pair(q, cA, c1, c2)

            rc = cr * cr
        f, u = ev(r2)
        if mode == "shift":
            u = u - ev(rc)[1]
        elif mode == "xplor":
            ro, c9 = 6.25, 9.0
            g = (c9 - r2) ** 2 * (c9 + 2.0 * r2 - 3.0 * ro) / (c9 - ro) ** 3
            dg = 12.0 * (r2 - ro) * (r2 - c9) / (c9 - ro) ** 3
            sm = r2 >= ro
            f, u = torch.where(sm, g * f - dg * u, f), torch.where(sm, g * u, u)
        add(i, j, d, f, f, u)
    if "bonds" in s:
        i, j = s["bonds"].unbind(dim=1)
        d = x[i] - x[j]
        d = d - L * torch.round(d / L)
        f, u = _quartic((d * d).sum(dim=1))
        add(i, j, d, f, f, u)
    return F, U, W


def _advance(s, kind, mode, steps, seed, dt=DT, brownian=False):
    """The state after `steps` timesteps, and the forces of the last one."""
    L, N = s["L"], len(s["x"])
    x, v, img = s["x"].clone(), s["v"].clone(), s["img"].clone()
    a = torch.zeros_like(v)
    tags = torch.arange(N, device="cuda")
    out = None

    def flow():
        u = torch.zeros_like(x)
        if kind == "melt":
            u[:, 0] = 1.0 - (x[:, 1] / (0.5 * L)) ** 2
        elif kind == "colloid":
            u[:, 0] = 0.1
        return u

    for t in range(steps):
        if brownian:
            gamma = 10.0 * s["diameter"][:, None]
            F = _forces(s, kind, mode, x)[0]
            R = _noise(201, t, seed, tags, 1.0) * torch.sqrt(6.0 * gamma / dt)
            x, w = _wrap(x + (flow() + (F + R) / gamma) * dt, L)
            img += w
            continue
        x, w = _wrap(x + (v + 0.5 * dt * a) * dt, L)
        img += w
        v = v + 0.5 * dt * a
        if kind == "dpd":
            out = _forces(s, kind, mode, x, v, t + 1, seed, dt)
            a = out[0]
        else:
            out = _forces(s, kind, mode, x)
            a = out[0] + _noise(202, t, seed, tags, math.sqrt(6.0 / dt)) - (v - flow())
        v = v + 0.5 * dt * a
    return x, v, a, img, out


def _with(x, last):
    return torch.cat([x, torch.as_tensor(last, dtype=F64, device="cuda").expand(len(x)).reshape(-1, 1)], dim=1)


def exact(case, seed):
    if case["family"] == "batch":
        rows = []
        for k, r in enumerate(_replicas(case, seed)):
            x, v, a, img, _ = _advance(r, "yukawa", "none", case["steps"] + 1, 100 + k, dt=0.002)
            rows.append((_with(x, 0.0), _with(v, 1.0), a, img))
        return {k: _np(torch.cat(c)) for k, c in zip(("pos", "vel", "acc", "img"), zip(*rows))}
    s = _system(case, seed)
    if case["family"] == "md":
        system = case["system"]
        x, v, a, img, _ = _advance(s, system, case["mode"], case["steps"] + 1, seed & 0xFFFF,
                                   dt=0.001 if system == "colloid" else DT, brownian=system == "colloid")
        return dict(pos=_with(x, s["typ"].to(F64)), vel=_with(v, 1.0), acc=a, img=img)
    if case["family"] == "step":
        x, v, a, img, (F, U, W) = _advance(s, case["system"], case["mode"], case["steps"], seed & 0xFFFF)
        return dict(pos=x, vel=_with(v, 1.0), acc=a, img=img, force=torch.cat([F, U[:, None]], dim=1), virial=W)
    if case["family"] == "dpd":
        F, U, W = _forces(s, "dpd", "none", s["x"], s["v"], 7, seed & 0xFFFF)
        return dict(force=torch.cat([F, U[:, None]], dim=1), virial=W)
    return _exact_grad(case, seed, s)


def _exact_grad(case, seed, s):
    gen = _gen(seed + 1)
    N, L, mode = len(s["x"]), s["L"], case["mode"]
    gF = torch.randn((N, 3), generator=gen, dtype=F64, device="cuda")
    gU = torch.randn(N, generator=gen, dtype=F64, device="cuda")
    F, U, _ = _forces(s, "fluid", mode, s["x"])
    i, j = _near(s["x"], L, 3.0)
    gx, gv = torch.zeros((N, 3), dtype=F64, device="cuda"), torch.zeros(3, dtype=F64, device="cuda")
    for a in range(0, len(i), 1 << 22):
        p, q = i[a:a + (1 << 22)], j[a:a + (1 << 22)]
        d = s["x"][p] - s["x"][q]
        d = (d - L * torch.round(d / L)).requires_grad_(True)
        val = torch.tensor([1.0, 1.0, 0.5], dtype=F64, device="cuda", requires_grad=True)
        r2 = (d * d).sum(dim=1)
        f, u = _lj(r2, val[0], val[1], val[2])
        if mode == "shift":
            u = u - _lj(torch.full_like(r2, 9.0), val[0], val[1], val[2])[1]
        elif mode == "xplor":
            g = (9.0 - r2) ** 2 * (9.0 + 2.0 * r2 - 18.75) / 2.75 ** 3
            dg = 12.0 * (r2 - 6.25) * (r2 - 9.0) / 2.75 ** 3
            sm = r2 >= 6.25
            f, u = torch.where(sm, g * f - dg * u, f), torch.where(sm, g * u, u)
        loss = ((gF[p] - gF[q]) * d * f[:, None]).sum() + (0.5 * (gU[p] + gU[q]) * u).sum()
        gd, gval = torch.autograd.grad(loss, (d, val))
        gx.index_add_(0, p, gd)
        gx.index_add_(0, q, -gd)
        gv += gval
    return dict(F=F, U=U, gx=gx, gv=gv)
