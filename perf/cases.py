"""The work that users of this package have it do, as cases that can be timed.

Kinds of case (each through the package's public entry points):

  rect      rectangle stiffness (``assemble.assemble_rect_dev``): whole fault
            systems, and the single blocks that ``hmatrix.build_rect`` asks for
  tri       triangle stiffness of a whole mesh (``assemble.assemble_tri_dev``)
  pairs     triangle entries from index lists (``assemble.assemble_tri_pairs_dev``),
            the near-field batches of ``hmatrix.build_tri``
  main      the reference's entry point ``simulate.main`` on host arrays: context,
            operator, run and recorded history
  run       one context advanced by some steps, its state in pinned host memory
            before and after (``Simulation.set_state_all`` / ``get_state_all``)
  ensemble  many networks of uneven size with friction draws in one launch
  hmat      one context on an H-matrix of a curved triangle mesh
  adjoint   gradients of a final-slip loss with respect to a, b and Dc

Sizes are those of the benchmark's workloads and of the tests: the 800-patch
single fault, the 30-fault network of ~12,800 patches, ensemble members of
900-5,900 patches, the 4,005 patches (5 of them loading) of the default bulk
input, the 1,100-triangle mesh, the 49-patch test system.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quake-dfn_gb300"))

from qdfn import adjoint, assemble, ensemble, geometry, hmatrix, simulate, synth  # noqa: E402

G, NU = 32e9, 0.25
FIELDS = simulate.Simulation.STATE_FIELDS
LEAF, ETA, ACA_TOL = 64, 2.0, 1e-6


def listed():
    return [
        # one near-field block of an H-matrix build: latency of a single small launch
        dict(name="rect_block_64", kind="rect", geometry="network", sources=61, receivers=64, layout="col"),
        # a vertical fault (cos dip = 0) of the single-fault size beside a dipping one
        dict(name="rect_faults_800", kind="rect", geometry="faults", sources=800, receivers=800, layout="row"),
        # the largest ensemble member's network
        dict(name="rect_network_5850", kind="rect", geometry="network", sources=5850, receivers=5850, layout="col"),
        # the reference's triangle mesh size
        dict(name="tri_mesh_1100", kind="tri", triangles=1100, layout="col"),
        # a batch of near-field blocks of a triangle H-matrix build
        dict(name="tri_pairs_256x64x64", kind="pairs", triangles=6000, blocks=256, side=64),
        # a reference user's first run: FP64, host matrices in, history out
        dict(name="main_fault_800", kind="main", patches=800, steps=200, record=10, precision="fp64"),
        # the smallest systems: barriers and latency
        dict(name="run_49_fp64", kind="run", patches=49, draws=1, precision="fp64", steps=32, phase="creep",
             loading=0),
        # the default input's size with loading faults and a running rupture (high-velocity solver)
        dict(name="run_4005_rupture_fp64", kind="run", patches=4005, draws=1, precision="fp64", steps=20,
             phase="rupture", loading=5),
        # the 30-fault network with four friction draws, mixed precision
        dict(name="run_12813x4_fp32", kind="run", patches=12813, draws=4, precision="fp32", steps=20, phase="creep",
             loading=0),
        # a batched ensemble, advanced by the 15 steps between two divisions of the SMs
        dict(name="ensemble_40x4_fp32", kind="ensemble", members=40, draws=4, smallest=907, largest=2900,
             precision="fp32", steps=15),
        # curved faults as a triangle mesh with an H-matrix
        dict(name="hmat_6000_fp32", kind="hmat", faults=3, cells_u=40, cells_v=25, draws=1, precision="fp32",
             steps=24),
        # gradients: forward, replay and reverse sweep
        dict(name="adjoint_3001_fp32", kind="adjoint", patches=3001, draws=1, precision="fp32", steps=36),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rect", "rect", "tri", "pairs", "main", "run", "run", "run", "ensemble", "hmat", "adjoint"])
    if kind == "rect":
        geo = rng.choice(["network", "network", "faults"])
        top = 5850 if geo == "network" else 800
        return dict(kind=kind, geometry=geo, sources=_log_int(rng, 16, top), receivers=_log_int(rng, 16, top),
                    layout=rng.choice(["col", "row"]))
    if kind == "tri":
        return dict(kind=kind, triangles=_log_int(rng, 48, 1100), layout=rng.choice(["col", "row"]))
    if kind == "pairs":
        return dict(kind=kind, triangles=6000, blocks=_log_int(rng, 4, 256), side=rng.randint(24, 64))
    if kind == "main":
        return dict(kind=kind, patches=_log_int(rng, 60, 800), steps=rng.randint(40, 200), record=rng.randint(1, 20),
                    precision=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "run":
        precision = rng.choice(["fp64", "fp32", "fp32", "bf16x2"])
        n = _log_int(rng, 18, 5800 if precision == "fp64" else 12813)
        load = rng.choice([0, 0, 5]) if n > 60 else 0
        return dict(kind=kind, patches=n, draws=rng.randint(1, 4), precision=precision, steps=rng.randint(8, 20),
                    phase=rng.choice(["creep", "creep", "rupture"]), loading=load)
    if kind == "ensemble":
        return dict(kind=kind, members=_log_int(rng, 3, 40), draws=rng.randint(1, 4), smallest=_log_int(rng, 60, 907),
                    largest=_log_int(rng, 1000, 2900), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    steps=rng.randint(4, 15))
    if kind == "hmat":
        return dict(kind=kind, faults=rng.randint(1, 3), cells_u=rng.randint(12, 40), cells_v=rng.randint(8, 25),
                    draws=rng.randint(1, 2), precision=rng.choice(["fp32", "fp64"]), steps=rng.randint(8, 24))
    return dict(kind=kind, patches=_log_int(rng, 100, 3001), draws=rng.randint(1, 2),
                precision=rng.choice(["fp32", "fp64"]), steps=rng.randint(9, 36))


# --------------------------------------------------------------- inputs
_KEPT = {}   # geometries that do not depend on the seed (made once per process)


def _network(n):
    """n patches of 100 m of a random fault network."""
    faults = max(1, n // 330)
    while True:
        key = ("network", faults)
        if key not in _KEPT:
            _KEPT[key] = synth.fault_network(seed=7, n_faults=faults)
        if _KEPT[key]["N"] >= n:
            return _KEPT[key]["records"][:n].copy()
        faults += 1 + faults // 8


def _fault(n):
    if "fault" not in _KEPT:
        _KEPT["fault"] = synth.single_fault()["records"]
    return _KEPT["fault"][:n].copy()


def _mesh(faults, cells_u, cells_v):
    key = ("mesh", faults, cells_u, cells_v)
    if key not in _KEPT:
        _KEPT[key] = synth.curved_fault_network(seed=5, n_faults=faults, length=80.0 * cells_u, width=80.0 * cells_v,
                                                edge=80.0)
    return _KEPT[key]


def _mesh_of(n):
    """A mesh of at least n triangles (one curved fault per 2,000)."""
    faults = max(1, -(-n // 2000))
    v = max(4, int(math.sqrt(n / faults / 2 / 1.6)) + 1)
    return _mesh(faults, -(-n // (2 * v * faults)), v)


def _cuda(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _rect_inputs(case, seed):
    rng = np.random.default_rng([seed, 1])
    if case["geometry"] == "faults":
        rec = np.vstack([_fault(400), synth.grid_fault(6000.0, 0.0, 5500.0, 10000.0, 10000.0, 60.0, 60.0, 0.0, 500.0)])
    else:
        rec = _network(5850)
    rec[:, 2] += rng.uniform(0.0, 300.0)          # deeper by up to 300 m
    rec[:, 7] = rng.uniform(-180.0, 180.0)        # another rake
    first = len(rec) - case["sources"]            # another fault's patches where there are enough
    start = int(rng.integers(min(case["receivers"] + 400, first), first + 1))
    return rec[start:start + case["sources"]], rec[:case["receivers"]]


def _tri_inputs(seg, seed):
    """Vertices, rake and unit vectors of a mesh, shifted in depth and with a rake of its own."""
    rng = np.random.default_rng([seed, 2])
    seg = seg.copy()
    seg[:, [2, 5, 8]] -= rng.uniform(0.0, 300.0)
    seg[:, 9] = rng.uniform(-180.0, 180.0)
    P1, P2, P3, un, _, _, us = geometry.rot_verts_unit_vectors_abi(seg, seg[:, 9])
    return P1, P2, P3, seg[:, 9], (P1 + P2 + P3) / 3, un, us


def _pair_inputs(case, seed):
    seg = _mesh(3, 40, 25)["seg"][:case["triangles"]]
    tri = _tri_inputs(seg, seed)
    rng = np.random.default_rng([seed, 3])
    k, m = case["side"], seg.shape[0]
    r0 = rng.integers(0, m - k, case["blocks"])
    s0 = np.clip(r0 + rng.integers(-2 * k, 2 * k, case["blocks"]), 0, m - k)
    r = np.repeat(r0[:, None] + np.arange(k), k, axis=1).ravel()
    s = np.tile(s0[:, None] + np.arange(k), (1, k)).ravel()
    return tri, r, s


def _friction(n, draws, rng, sigma0, Dc_log):
    """Per-patch friction of `draws` instances around steady creep: slip rates
    and states spread around 1e-9 m/s, friction consistent with both."""
    m = n * draws
    a = rng.uniform(0.008, 0.012, m)
    b = a + rng.uniform(-0.004, 0.004, m)
    Dc = 10.0 ** rng.uniform(*Dc_log, m)
    V = 1e-9 * np.exp(0.3 * rng.standard_normal(m))
    th = Dc / 1e-9 * np.exp(0.2 * rng.standard_normal(m))
    return dict(a=a, b=b, Dc=Dc, V_i=V, theta_i=th, sigma0=np.tile(sigma0, draws))


def _initial_friction(p):
    p["f_i"] = 0.6 + p["a"] * np.log(p["V_i"] / 1e-6) + p["b"] * np.log(p["theta_i"] * 1e-6 / p["Dc"])


def _problem(case, seed, n, draws, sigma0, mass, kself, phase="creep", loading=0, told=0):
    rng = np.random.default_rng([seed, 4])
    p = _friction(n, draws, rng, sigma0, (-2, -1) if phase == "rupture" else (-4, -2))
    if phase == "rupture":   # a nucleation zone starts at 0.03 m/s, as in the default input
        hot = (np.arange(n * draws) % n) < max(1, n // 20)
        p["V_i"][hot] = 0.03 * np.exp(0.3 * rng.standard_normal(int(hot.sum())))
    p["V_const"] = np.zeros(n * draws)
    if loading:
        last = (np.arange(n * draws) % n) >= n - loading
        p["V_const"][last] = p["V_i"][last] = 1e-9
    _initial_friction(p)
    p.update(N=n, Nload=loading, G=G, rho=G / synth.CS ** 2, sigma_min=1e6, switch_v=1e-2, dt_cut=5.0, max_dt=1e7,
             alpha_evo=0.0, evolution_dr=1, interp_at_told=told, mass=np.tile(mass, draws),
             rupture_dt=geometry.rupture_dt(mass, kself, 3.0))
    return p


def _rect_operator(rec, layout="col"):
    """(Ks, Kn) on the device, entry (receiver r, source s) at [s, r]."""
    d = _cuda(rec)
    Ks = torch.empty((len(rec), len(rec)), dtype=torch.float64, device="cuda")
    Kn = torch.empty_like(Ks)
    assemble.assemble_rect_dev(d, d, G, NU, Ks, Kn, layout=layout)
    return Ks, Kn


def _patches(case):
    """Records of a `run` / `adjoint` / ensemble system, its loading faults last."""
    n, load = case["patches"], case.get("loading", 0)
    rec = _network(n - load)
    if load:   # wide patches below the network
        deep = np.array([[4000.0 * (k - load / 2), 3000.0 * k, 20000.0, 20000.0, 10000.0, 20.0 * k, 80.0, 0.0]
                         for k in range(load)])
        rec = np.vstack([rec, deep])
    return rec


def _system(case, seed, rec, told=0, phase="creep", loading=0):
    """Context with its operator set, and the problem."""
    Ks, Kn = _rect_operator(rec)
    kdiag = torch.diagonal(Ks).cpu().numpy()
    p = _problem(case, seed, len(rec), case["draws"], _sigma0(rec), _mass(rec), kdiag, phase, loading, told)
    sim = simulate.Simulation(p, n_inst=case["draws"])
    sim.set_dense_device(Ks, Kn, case["precision"])
    return sim, p


def _sigma0(rec):
    return 18e6 * rec[:, 2] / 1000.0


def _mass(rec):
    return geometry.fault_mass(rec[:, 3], rec[:, 4], G / synth.CS ** 2)


def _start(p, phase):
    """The state a run starts from: the problem's initial values, and a time
    step of 10 s for slow creep (the controller lets it grow by 1.2 a step)."""
    n = p["V_i"].shape[0]
    return dict(V=p["V_i"], D=np.zeros(n), theta=p["theta_i"], friction=p["f_i"], accel=np.zeros(n),
                sigma_old=p["sigma0"]), (10.0 if phase == "creep" else 1.0)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def _state_io(p, draws, phase):
    st, dt = _start(p, phase)
    given = {k: _pinned(v) for k, v in st.items()}
    back = {k: torch.empty_like(v).pin_memory() for k, v in given.items()}
    f = lambda v, t: torch.full((draws,), v, dtype=t).pin_memory()  # noqa: E731
    scal = [f(0.0, torch.float64), f(dt, torch.float64), f(0, torch.int64)]
    return dict(given=given, back=back, scal=scal, out=[torch.empty_like(s).pin_memory() for s in scal])


def _mesh_system(case, seed):
    """Context of an H-matrix on a curved mesh (its blocks are kept: a program
    builds them once per mesh), its problem and the mesh in the tree's order."""
    net = _mesh(case["faults"], case["cells_u"], case["cells_v"])
    key = ("hmat", case["faults"], case["cells_u"], case["cells_v"])
    if key not in _KEPT:
        seg = net["seg"]
        P1, P2, P3, un, _, _, us = geometry.rot_verts_unit_vectors_abi(seg, seg[:, 9])
        cen = (P1 + P2 + P3) / 3
        H, perm = hmatrix.build_tri(P1, P2, P3, seg[:, 9], cen, un, us, G, NU, leaf=LEAF, eta=ETA, tol=ACA_TOL)
        kdiag = np.zeros(net["N"])
        for b, (s0, s1, r0, r1) in enumerate(H.ranges):
            if s0 == r0 and s1 == r1 and H.dense_s[b] is not None:
                kdiag[r0:r1 + 1] = np.diag(H.dense_s[b])
        _KEPT[key] = H, kdiag, [x[perm] for x in (P1, P2, P3, seg[:, 9], cen, un, us)], perm
    H, kdiag, tri, perm = _KEPT[key]
    p = _problem(case, seed, net["N"], case["draws"], net["sigma0"][perm], net["mass"][perm], kdiag, told=1)
    sim = simulate.Simulation(p, n_inst=case["draws"])
    hmatrix.set_hmatrix(sim, H, case["precision"])
    return sim, p, tri, H


def _member_sizes(case):
    n = case["members"]
    f = [(k + 0.5) / n for k in range(n)]
    return [int(round(case["smallest"] * (case["largest"] / case["smallest"]) ** (x ** 1.5))) for x in f]


def _member(case, seed, k, n):
    rec = _network(n)
    rec[:, 2] += 40.0 * (k % 8)
    return rec, dict(patches=n, draws=case["draws"]), seed + 7919 * (k + 1)


def _main_args(case, seed):
    rng = np.random.default_rng([seed, 5])
    rec = _fault(case["patches"])
    rec[:, 2] += rng.uniform(0.0, 300.0)
    n = len(rec)
    s = synth.single_fault()
    Ks, Kn = (K.cpu().numpy() for K in _rect_operator(rec, layout="row"))
    V = 1e-9 * np.exp(0.3 * rng.standard_normal(n))
    p = dict(a=s["a"][:n], b=s["b"][:n], Dc=s["Dc"][:n], V_i=V,
             theta_i=1e-3 / 1e-9 * np.exp(0.2 * rng.standard_normal(n)), sigma0=s["sigma0"][:n],
             V_const=np.zeros(n), mass=_mass(rec), N=n, Nload=0, G=G, rho=s["rho"], sigma_min=1e6, switch_v=1e-2,
             dt_cut=5.0, max_dt=1e7, alpha_evo=0.0, evolution_dr=1, interp_at_told=0)
    _initial_friction(p)
    p["rupture_dt"] = geometry.rupture_dt(p["mass"], np.diag(Ks), 3.0)
    return rec, p, Ks, Kn, synth.external_ramp(n, s["stressing_rate"], 1e11)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rect":
        src, recv = (_cuda(r) for r in _rect_inputs(case, seed))
        shape = (len(src), len(recv)) if case["layout"] == "col" else (len(recv), len(src))
        K = [torch.empty(shape, dtype=torch.float64, device="cuda") for _ in range(2)]
        return dict(case=case, src=src, recv=recv, K=K)
    if kind == "tri":
        tri = [_cuda(x) for x in _tri_inputs(_mesh_of(case["triangles"])["seg"][:case["triangles"]], seed)]
        n = case["triangles"]
        return dict(case=case, tri=tri, K=[torch.empty((n, n), dtype=torch.float64, device="cuda") for _ in range(2)])
    if kind == "pairs":
        tri, r, s = _pair_inputs(case, seed)
        return dict(case=case, tri=[_cuda(x) for x in tri], r=torch.tensor(r, device="cuda"),
                    s=torch.tensor(s, device="cuda"))
    if kind == "main":
        rec, p, Ks, Kn, ext = _main_args(case, seed)
        args = [Ks, Kn, 0, G, p["N"], 0, p["mass"], p["a"], p["b"], p["Dc"], p["theta_i"], p["V_i"], p["f_i"],
                p["sigma0"], p["V_const"], case["steps"], case["record"], p["switch_v"], p["dt_cut"], p["rupture_dt"],
                p["max_dt"], None, p["rho"], rec[:, :3], rec[:, 3], rec[:, 4], rec[:, 5], rec[:, 6], rec[:, 7], 0,
                p["sigma_min"], 0.0, 1]
        return dict(case=case, args=args, ext=ext)
    if kind == "run":
        sim, p = _system(case, seed, _patches(case), phase=case["phase"], loading=case["loading"])
        return dict(case=case, sim=sim, **_state_io(p, case["draws"], case["phase"]))
    if kind == "hmat":
        sim, p, _, _ = _mesh_system(case, seed)
        return dict(case=case, sim=sim, **_state_io(p, case["draws"], "creep"))
    if kind == "adjoint":
        sim, p = _system(case, seed, _patches(case))
        st, dt = _start(p, "creep")
        rng = np.random.default_rng([seed, 6])
        n = case["patches"]
        states = [dict({k: v[r * n:(r + 1) * n] for k, v in st.items()}, T=0.0, dt=dt, step=0)
                  for r in range(case["draws"])]
        return dict(case=case, sim=sim, states=states, loss=rng.standard_normal((case["draws"], n)))
    members = []
    for k, n in enumerate(_member_sizes(case)):
        rec, c, s = _member(case, seed, k, n)
        Ks, Kn = _rect_operator(rec)
        p = _problem(c, s, n, c["draws"], _sigma0(rec), _mass(rec), torch.diagonal(Ks).cpu().numpy())
        members.append(dict(problem=p, n_inst=c["draws"], Ks=Ks, Kn=Kn))
    ens = ensemble.Ensemble(members, precision=case["precision"])
    given = torch.empty(ens.state_words(), dtype=torch.float64).pin_memory()
    states = []
    for m in members:
        st, dt = _start(m["problem"], "creep")
        n = m["problem"]["N"]
        states.append([dict({k: v[r * n:(r + 1) * n] for k, v in st.items()}, T=0.0, dt=dt, step=0)
                       for r in range(case["draws"])])
    ens.pack_states(states, given)
    back = torch.empty_like(given).pin_memory()
    views, at = {k: [] for k in (*FIELDS, "T", "dt", "step")}, 0
    for m in members:
        w = m["problem"]["N"] * case["draws"]
        for k in FIELDS:
            views[k].append(back[at:at + w])
            at += w
        for k in ("T", "dt", "step"):
            v = back[at:at + case["draws"]]
            views[k].append(v.view(torch.int64) if k == "step" else v)
            at += case["draws"]
    return dict(case=case, ens=ens, given=given, back=back, views=views)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rect":
        assemble.assemble_rect_dev(state["src"], state["recv"], G, NU, *state["K"], layout=case["layout"])
        return state["K"]
    if kind == "tri":
        assemble.assemble_tri_dev(*state["tri"], G, NU, *state["K"], layout=case["layout"])
        return state["K"]
    if kind == "pairs":
        return list(assemble.assemble_tri_pairs_dev(state["r"], state["s"], *state["tri"], G, NU))
    if kind == "main":
        return simulate.main(*state["args"], external_stress=state["ext"], precision=case["precision"])
    if kind in ("run", "hmat"):
        sim = state["sim"]
        sim.set_state_all(state["given"], *state["scal"])
        sim.run_async(case["steps"])
        sim.get_state_all(state["back"], *state["out"], wait=True)
        T, dt, step = state["out"]
        return dict(state["back"], T=T, dt=dt, step=step)
    if kind == "adjoint":
        sim = state["sim"]
        for r, st in enumerate(state["states"]):
            sim.set_state(r, st)
        return adjoint.gradient(sim, case["steps"], dL_dD_final=state["loss"])
    ens = state["ens"]
    ens.set_state_all(state["given"])
    ens.run_async(case["steps"])
    ens.get_state_all(state["back"])
    return {k: torch.cat(v) for k, v in state["views"].items()}


# --------------------------------------------------------------- least work
# FP64 operations that one entry cannot do without: the eight corner terms of
# a rectangle, the nine angular dislocations of a triangle
RECT_FLOPS, TRI_FLOPS = 1500.0, 6000.0
SOLVE_FLOPS = 120.0           # one patch's friction solve: two Newton iterations with a logarithm and an exponential
ELEMENT = {"fp64": 8, "fp32": 4, "bf16x2": 4}


def _run_work(n, draws, precision, steps, entries=None):
    stored = 2.0 * n * n if entries is None else float(entries)
    state = 14.0 * 8 * n * draws
    return dict(bytes=steps * (stored * ELEMENT[precision] + state), flops=steps * (2 * stored * draws +
                                                                                    SOLVE_FLOPS * n * draws))


def work(case):
    kind = case["kind"]
    if kind == "rect":
        n = float(case["sources"]) * case["receivers"]
        return dict(bytes=16 * n + 64.0 * (case["sources"] + case["receivers"]), flops=RECT_FLOPS * n)
    if kind == "tri":
        n = float(case["triangles"]) ** 2
        return dict(bytes=16 * n + 152.0 * case["triangles"], flops=TRI_FLOPS * n)
    if kind == "pairs":
        n = float(case["blocks"]) * case["side"] ** 2
        return dict(bytes=32 * n, flops=TRI_FLOPS * n)
    if kind == "main":
        w = _run_work(case["patches"], 1, case["precision"], case["steps"])
        w["bytes"] += 16.0 * case["patches"] ** 2 + 32.0 * case["patches"] * (case["steps"] // case["record"])
        return w
    if kind == "run":
        return _run_work(case["patches"], case["draws"], case["precision"], case["steps"])
    if kind == "hmat":
        # stored entries of a leaf-64 tree at ACA tolerance 1e-6 grow like n log n
        n = 2.0 * case["faults"] * case["cells_u"] * case["cells_v"]
        return _run_work(n, case["draws"], case["precision"], case["steps"], entries=n * 280 * math.log2(n))
    if kind == "adjoint":   # forward and replay, and the reverse step's transposed products
        w = _run_work(case["patches"], case["draws"], case["precision"], case["steps"])
        return {k: 3 * v for k, v in w.items()}
    w = [_run_work(n, case["draws"], case["precision"], case["steps"]) for n in _member_sizes(case)]
    return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}


# --------------------------------------------------------------- values in 64 bits
def _sincosd(deg):
    """(sin, cos) of degrees, exact at multiples of 90."""
    q = torch.round(deg / 90)
    r = (deg - 90 * q) * (math.pi / 180)
    s, c = torch.sin(r), torch.cos(r)
    q = torch.remainder(q, 4)
    sn = torch.where(q == 0, s, torch.where(q == 1, c, torch.where(q == 2, -s, -c)))
    cs = torch.where(q == 0, c, torch.where(q == 1, -s, torch.where(q == 2, -c, s)))
    return sn, cs


def _okada(X, Y, Z, depth, dip, AL, AW, U1, U2, alpha):
    """Displacement gradients (UXX, UYX, UZX, UXY, ..., UZZ) of a rectangular
    strike (U1) and dip (U2) dislocation in a half-space (Okada 1992, DC3D)."""
    A1, A2, A3, A4, A5 = (1 - alpha) / 2, alpha / 2, (1 - alpha) / alpha, 1 - alpha, alpha
    SD, CD = torch.sin(dip * (math.pi / 180)), torch.cos(dip * (math.pi / 180))
    flat = CD.abs() < 1e-6
    CD = torch.where(flat, torch.zeros_like(CD), CD)
    SD = torch.where(flat, torch.sign(SD), SD)
    SDSD, CDCD, SDCD = SD * SD, CD * CD, SD * CD
    out = [torch.zeros_like(X) for _ in range(9)]
    for image in (False, True):
        d = depth - Z if image else depth + Z
        p, Q = Y * CD + d * SD, Y * SD - d * CD
        for K in (0, 1):
            for J in (0, 1):
                XI, ET = (X - AL if J else X + AL), (p - AW if K else p + AW)
                small = lambda t: torch.where(t.abs() < 1e-6, torch.zeros_like(t), t)  # noqa: E731
                x, e, q = small(XI), small(ET), small(Q)
                XI2, ET2, Q2 = x * x, e * e, q * q
                R2 = XI2 + ET2 + Q2
                R = torch.sqrt(R2)
                R3, R5 = R * R2, R * R2 * R2
                Yt, D = e * CD + q * SD, e * SD - q * CD
                z = torch.zeros_like(R)
                on = (x < 0) & (q == 0) & (e == 0)
                X11 = torch.where(on, z, 1 / (R * (R + x)))
                X32 = torch.where(on, z, (2 * R + x) * X11 * X11 / R)
                on = (e < 0) & (q == 0) & (x == 0)
                Y11 = torch.where(on, z, 1 / (R * (R + e)))
                Y32 = torch.where(on, z, (2 * R + e) * Y11 * Y11 / R)
                EY, EZ = SD / R - Yt * Q / R3, CD / R + D * Q / R3
                FY, FZ = D / R3 + XI2 * Y32 * SD, Yt / R3 + XI2 * Y32 * CD
                GY, GZ = 2 * X11 * SD - Yt * Q * X32, 2 * X11 * CD + D * Q * X32
                XY, QY = XI * Y11, Q * Y11
                s1 = [-A1 * QY - A2 * XI2 * Q * Y32, -A2 * XI * Q / R3, A1 * XY + A2 * XI * Q2 * Y32,
                      A1 * XY * SD + A2 * XI * FY + D / 2 * X11, A2 * EY, A1 * (CD / R + QY * SD) - A2 * Q * FY,
                      A1 * XY * CD + A2 * XI * FZ + Yt / 2 * X11, A2 * EZ, -A1 * (SD / R - QY * CD) - A2 * Q * FZ]
                s2 = [-A2 * XI * Q / R3, -QY / 2 - A2 * ET * Q / R3, A1 / R + A2 * Q2 / R3, A2 * EY,
                      A1 * D * X11 + XY / 2 * SD + A2 * ET * GY, A1 * Yt * X11 - A2 * Q * GY, A2 * EZ,
                      A1 * Yt * X11 + XY / 2 * CD + A2 * ET * GZ, -A1 * D * X11 - A2 * Q * GZ]
                a = [U1 * m + U2 * n for m, n in zip(s1, s2)]
                if not image:
                    du = []
                    for i in (0, 3, 6):
                        row = [-a[i], -a[i + 1] * CD + a[i + 2] * SD, -a[i + 1] * SD - a[i + 2] * CD]
                        du += row if i < 6 else [-t for t in row]
                else:
                    RD = R + D
                    D11 = 1 / (R * RD)
                    J2, J5 = XI * Yt / RD * D11, -(D + Yt * Yt / RD) * D11
                    C1 = torch.where(flat, torch.ones_like(CD), CD)
                    K1 = torch.where(flat, XI * Q / RD * D11, XI * (D11 - Y11 * SD) / C1)
                    K3 = torch.where(flat, SD / RD * (XI2 * D11 - 1), (Q * Y11 - Yt * D11) / C1)
                    J3 = torch.where(flat, -XI / RD ** 2 * (Q2 * D11 - 0.5), (K1 - J2 * SD) / C1)
                    J6 = torch.where(flat, -Yt / RD ** 2 * (XI2 * D11 - 0.5), (K3 - J5 * SD) / C1)
                    K2, K4 = 1 / R + K3 * SD, XY * CD - K1 * SD
                    J1, J4 = J5 * CD - J6 * SD, -XY - J2 * CD + J3 * SD
                    s1 = [XI2 * Q * Y32 - A3 * J1 * SD, XI * Q / R3 - A3 * J2 * SD, -XI * Q2 * Y32 - A3 * J3 * SD,
                          -XI * FY - D * X11 + A3 * (XY + J4) * SD, -EY + A3 * (1 / R + J5) * SD,
                          Q * FY - A3 * (QY - J6) * SD, -XI * FZ - Yt * X11 + A3 * K1 * SD, -EZ + A3 * Yt * D11 * SD,
                          Q * FZ + A3 * K2 * SD]
                    s2 = [XI * Q / R3 + A3 * J4 * SDCD, ET * Q / R3 + QY + A3 * J5 * SDCD, -Q2 / R3 + A3 * J6 * SDCD,
                          -EY + A3 * J1 * SDCD, -ET * GY - XY * SD + A3 * J2 * SDCD, Q * GY + A3 * J3 * SDCD,
                          -EZ - A3 * K3 * SDCD, -ET * GZ - XY * CD - A3 * XI * D11 * SDCD, Q * GZ - A3 * K4 * SDCD]
                    b = [U1 * m + U2 * n for m, n in zip(s1, s2)]
                    C = D + Z
                    X53 = (8 * R2 + 9 * R * XI + 3 * XI2) * X11 ** 3 / R2
                    Y53 = (8 * R2 + 9 * R * ET + 3 * ET2) * Y11 ** 3 / R2
                    H = Q * CD - Z
                    Z32, Z53 = SD / R3 - H * Y32, 3 * SD / R5 - H * Y53
                    Y0, Z0 = Y11 - XI2 * Y32, Z32 - XI2 * Z53
                    PY, PZ = CD / R3 + Q * Y32 * SD, SD / R3 - Q * Y32 * CD
                    QQ = Z * Y32 + Z32 + Z0
                    QQY, QQZ = 3 * C * D / R5 - QQ * SD, 3 * C * Yt / R5 - QQ * CD + Q * Y32
                    QR, CDR, YY0 = 3 * Q / R5, (C + D) / R3, Yt / R3 - Y0 * CD
                    s1 = [A4 * XY * CD - A5 * XI * Q * Z32, A4 * (CD / R + 2 * QY * SD) - A5 * C * Q / R3,
                          A4 * QY * CD - A5 * (C * ET / R3 - Z * Y11 + XI2 * Z32), A4 * Y0 * CD - A5 * Q * Z0,
                          -A4 * XI * (CD / R3 + 2 * Q * Y32 * SD) + A5 * C * XI * QR,
                          -A4 * XI * Q * Y32 * CD + A5 * XI * (3 * C * ET / R5 - QQ),
                          -A4 * XI * PY * CD - A5 * XI * QQY,
                          A4 * 2 * (D / R3 - Y0 * SD) * SD - Yt / R3 * CD - A5 * (CDR * SD - ET / R3 - C * Yt * QR),
                          -A4 * Q / R3 + YY0 * SD + A5 * (CDR * CD + C * D * QR - (Y0 * CD + Q * Z0) * SD),
                          A4 * XI * PZ * CD - A5 * XI * QQZ,
                          A4 * 2 * (Yt / R3 - Y0 * CD) * SD + D / R3 * CD - A5 * (CDR * CD + C * D * QR),
                          YY0 * CD - A5 * (CDR * SD - C * Yt * QR - Y0 * SDSD + Q * Z0 * CD)]
                    s2 = [A4 * CD / R - QY * SD - A5 * C * Q / R3, A4 * Yt * X11 - A5 * C * ET * Q * X32,
                          -D * X11 - XY * SD - A5 * C * (X11 - Q2 * X32),
                          -A4 * XI / R3 * CD + A5 * C * XI * QR + XI * Q * Y32 * SD,
                          -A4 * Yt / R3 + A5 * C * ET * QR, D / R3 - Y0 * SD + A5 * C / R3 * (1 - 3 * Q2 / R2),
                          -A4 * ET / R3 + Y0 * SDSD - A5 * (CDR * SD - C * Yt * QR),
                          A4 * (X11 - Yt * Yt * X32) - A5 * C * ((D + 2 * Q * CD) * X32 - Yt * ET * Q * X53),
                          XI * PY * SD + Yt * D * X32 + A5 * C * ((Yt + 2 * Q * SD) * X32 - Yt * Q2 * X53),
                          -Q / R3 + Y0 * SDCD - A5 * (CDR * CD + C * D * QR),
                          A4 * Yt * D * X32 - A5 * C * ((Yt - 2 * Q * SD) * X32 + D * ET * Q * X53),
                          -XI * PZ * SD + X11 - D * D * X32 - A5 * C * ((D - 2 * Q * CD) * X32 - D * Q2 * X53)]
                    c = [U1 * m + U2 * n for m, n in zip(s1, s2)]
                    du = []
                    for i in (0, 3, 6):
                        u = [a[i + k] + b[i + k] for k in range(3)]
                        w = [Z * c[3 + i + k] for k in range(3)]
                        du += [u[0] + w[0], (u[1] + w[1]) * CD - (u[2] + w[2]) * SD,
                               (u[1] - w[1]) * SD + (u[2] - w[2]) * CD]
                    du[6] = du[6] + c[0]
                    du[7] = du[7] + c[1] * CD - c[2] * SD
                    du[8] = du[8] - c[1] * SD - c[2] * CD
                sign = 1.0 if J == K else -1.0
                out = [o + sign / (2 * math.pi) * t for o, t in zip(out, du)]
    return out


def _rect64(src, recv, chunk=1 << 21):
    """(Ks, Kn)[receiver, source] of rectangular patches."""
    lam = 2 * G * NU / (1 - 2 * NU)
    alpha = (lam + G) / (lam + 2 * G)
    src, recv = _cuda(src), _cuda(recv)
    rows = max(1, chunk // len(src))
    Ks = torch.empty((len(recv), len(src)), dtype=torch.float64, device="cuda")
    Kn = torch.empty_like(Ks)
    for k in range(0, len(recv), rows):
        r = recv[k:k + rows].repeat_interleave(len(src), 0)
        s = src.repeat(r.shape[0] // len(src), 1)
        ss, cs = _sincosd(-s[:, 5])
        dx, dy = r[:, 0] - s[:, 0], r[:, 1] - s[:, 1]
        u2, u1 = _sincosd(s[:, 7])
        U = _okada(dx * cs - dy * ss, dx * ss + dy * cs, -r[:, 2], s[:, 2], s[:, 6], s[:, 3] / 2, s[:, 4] / 2, u1, u2,
                   alpha)
        tr = lam * (U[0] + U[4] + U[8])
        S = [tr + 2 * G * U[0], tr + 2 * G * U[4], tr + 2 * G * U[8], G * (U[3] + U[1]), G * (U[6] + U[2]),
             G * (U[7] + U[5])]
        sr, cr = _sincosd(-(r[:, 5] - s[:, 5]))
        sd, cd = _sincosd(-r[:, 6])
        z = torch.zeros_like(cr)
        rows3 = [[cr, -sr, z], [cd * sr, cd * cr, -sd], [sd * sr, sd * cr, cd]]
        M = [[S[0], S[3], S[4]], [S[3], S[1], S[5]], [S[4], S[5], S[2]]]
        t = [sum(M[i][j] * rows3[2][j] for j in range(3)) for i in range(3)]
        t = [sum(rows3[m][i] * t[i] for i in range(3)) for m in range(3)]
        sk, ck = _sincosd(r[:, 7])
        Ks[k:k + rows] = (ck * t[0] + sk * t[1]).view(-1, len(src))
        Kn[k:k + rows] = (-t[2]).view(-1, len(src))
    return Ks, Kn


def sq(x):
    return x * x


def cube(x):
    return x * x * x


def p5(x):
    return x * x * x * x * x


def _ang_dis_strain(x, y, z, alpha, bx, by, bz, nu):
    """Strains of an angular dislocation in a full space (Nikkhoo & Walter 2015)."""
    sinA = torch.sin(alpha)
    cosA = torch.cos(alpha)
    eta = y * cosA - z * sinA
    zeta = y * sinA + z * cosA
    x2 = sq(x)
    y2 = sq(y)
    z2 = sq(z)
    r2 = x2 + y2 + z2
    r = torch.sqrt(r2)
    r3 = r * r2
    rz = r * (r - z)
    r2z2 = r2 * sq(r - z)
    r3z = r3 * (r - z)
    W = zeta - r
    W2 = sq(W)
    Wr = W * r
    W2r = W2 * r
    Wr3 = W * r3
    W2r2 = W2 * r2
    C = (r * cosA - z) / Wr
    S = (r * sinA - y) / Wr
    rFi_rx = (eta / r / (r - zeta) - y / r / (r - z)) / 4 / math.pi
    rFi_ry = (x / r / (r - z) - cosA * x / r / (r - zeta)) / 4 / math.pi
    rFi_rz = (sinA * x / r / (r - zeta)) / 4 / math.pi
    e0 = (
        bx * (rFi_rx) + bx / 8 / math.pi / (1 - nu) * (eta / Wr + eta * x2 / W2r2 - eta * x2 / Wr3 + y / rz - x2 * y / r2z2
        - x2 * y / r3z) - by * x / 8 / math.pi / (1 - nu) * (((2 * nu + 1) / Wr + x2 / W2r2 - x2 / Wr3) * cosA + (2 * nu +
        1) / rz - x2 / r2z2 - x2 / r3z) + bz * x * sinA / 8 / math.pi / (1 - nu) * ((2 * nu + 1) / Wr + x2 / W2r2 - x2 /
        Wr3))
    e1 = (
        by * (rFi_ry) + bx / 8 / math.pi / (1 - nu) * ((1 / Wr + sq(S) - y2 / Wr3) * eta + (2 * nu + 1) * y / rz - cube(y)
        / r2z2 - cube(y) / r3z - 2 * nu * cosA * S) - by * x / 8 / math.pi / (1 - nu) * (1 / rz - y2 / r2z2 - y2 / r3z + (1
        / Wr + sq(S) - y2 / Wr3) * cosA) + bz * x * sinA / 8 / math.pi / (1 - nu) * (1 / Wr + sq(S) - y2 / Wr3))
    e2 = (
        bz * (rFi_rz) + bx / 8 / math.pi / (1 - nu) * (eta / W / r + eta * sq(C) - eta * z2 / Wr3 + y * z / r3 + 2 * nu *
        sinA * C) - by * x / 8 / math.pi / (1 - nu) * ((1 / Wr + sq(C) - z2 / Wr3) * cosA + z / r3) + bz * x * sinA / 8 /
        math.pi / (1 - nu) * (1 / Wr + sq(C) - z2 / Wr3))
    e3 = (
        bx * (rFi_ry) / 2 + by * (rFi_rx) / 2 - bx / 8 / math.pi / (1 - nu) * (x * y2 / r2z2 - nu * x / rz + x * y2 / r3z -
        nu * x * cosA / Wr + eta * x * S / Wr + eta * x * y / Wr3) + by / 8 / math.pi / (1 - nu) * (x2 * y / r2z2 - nu * y
        / rz + x2 * y / r3z + nu * cosA * S + x2 * y * cosA / Wr3 + x2 * cosA * S / Wr) - bz * sinA / 8 / math.pi / (1 -
        nu) * (nu * S + x2 * S / Wr + x2 * y / Wr3))
    e4 = (
        bx * (rFi_rz) / 2 + bz * (rFi_rx) / 2 - bx / 8 / math.pi / (1 - nu) * (-x * y / r3 + nu * x * sinA / Wr + eta * x *
        C / Wr + eta * x * z / Wr3) + by / 8 / math.pi / (1 - nu) * (-x2 / r3 + nu / r + nu * cosA * C + x2 * z * cosA /
        Wr3 + x2 * cosA * C / Wr) - bz * sinA / 8 / math.pi / (1 - nu) * (nu * C + x2 * C / Wr + x2 * z / Wr3))
    e5 = (
        by * (rFi_rz) / 2 + bz * (rFi_ry) / 2 + bx / 8 / math.pi / (1 - nu) * (y2 / r3 - nu / r - nu * cosA * C + nu * sinA
        * S + eta * sinA * cosA / W2 - eta * (y * cosA + z * sinA) / W2r + eta * y * z / W2r2 - eta * y * z / Wr3) -
        by * x / 8 / math.pi / (1 - nu) * (y / r3 + sinA * sq(cosA) / W2 - cosA * (y * cosA + z * sinA) / W2r + y * z *
        cosA / W2r2 - y * z * cosA / Wr3) - bz * x * sinA / 8 / math.pi / (1 - nu) * (y * z / Wr3 - sinA * cosA / W2 + (y *
        cosA + z * sinA) / W2r - y * z / W2r2))
    return e0, e1, e2, e3, e4, e5


def _ang_dis_strain_fsc(y1, y2, y3, beta, b1, b2, b3, nu, a):
    """Free-surface correction strains of an angular dislocation (Nikkhoo & Walter 2015)."""
    sinB = torch.sin(beta)
    cosB = torch.cos(beta)
    cotB = 1.0 / torch.tan(beta)
    y3b = y3 + 2 * a
    z1b = y1 * cosB + y3b * sinB
    z3b = -y1 * sinB + y3b * cosB
    rb2 = sq(y1) + sq(y2) + sq(y3b)
    rb = torch.sqrt(rb2)
    W1 = rb * cosB + y3b
    W2 = cosB + a / rb
    W3 = cosB + y3b / rb
    W4 = nu + a / rb
    W5 = 2 * nu + a / rb
    W6 = rb + y3b
    W7 = rb + z3b
    W8 = y3 + a
    W9 = 1 + a / rb / cosB
    N1 = 1 - 2 * nu
    rb3 = cube(rb)
    rb5 = p5(rb)
    rb4 = sq(rb2)
    cot2 = sq(cotB)
    rFib_ry2 = z1b / rb / (rb + z3b) - y1 / rb / (rb + y3b)
    rFib_ry1 = y2 / rb / (rb + y3b) - cosB * y2 / rb / (rb + z3b)
    rFib_ry3 = -sinB * y2 / rb / (rb + z3b)
    K = 0.25
    v0 = (
        b1 * (K * ((-2 + 2 * nu) * N1 * rFib_ry1 * cot2 - N1 * y2 / sq(W6) * ((1 - W5) * cotB - y1 / W6 * W4) / rb *
        y1 + N1 * y2 / W6 * (a / rb3 * y1 * cotB - 1 / W6 * W4 + sq(y1) / sq(W6) * W4 / rb + sq(y1) / W6 * a / rb3) -
        N1 * y2 * cosB * cotB / sq(W7) * W2 * (y1 / rb - sinB) - N1 * y2 * cosB * cotB / W7 * a / rb3 * y1 - 3 * a *
        y2 * W8 * cotB / rb5 * y1 - y2 * W8 / rb3 / W6 * (-N1 * cotB + y1 / W6 * W5 + a * y1 / rb2) * y1 - y2 * W8 /
        rb2 / sq(W6) * (-N1 * cotB + y1 / W6 * W5 + a * y1 / rb2) * y1 + y2 * W8 / rb / W6 * (1 / W6 * W5 - sq(y1) /
        sq(W6) * W5 / rb - sq(y1) / W6 * a / rb3 + a / rb2 - 2 * a * sq(y1) / rb4) - y2 * W8 / rb3 / W7 * (cosB / W7 *
        (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) - a * y3b * cosB * cotB / rb2) *
        y1 - y2 * W8 / rb / sq(W7) * (cosB / W7 * (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1)
        * cosB) - a * y3b * cosB * cotB / rb2) * (y1 / rb - sinB) + y2 * W8 / rb / W7 * (-cosB / sq(W7) * (W1 * (N1 *
        cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) * (y1 / rb - sinB) + cosB / W7 * (1 / rb *
        cosB * y1 * (N1 * cosB - a / rb) * cotB + W1 * a / rb3 * y1 * cotB + (2 - 2 * nu) * (1 / rb * sinB * y1 - 1) *
        cosB) + 2 * a * y3b * cosB * cotB / rb4 * y1)) / math.pi / (1 - nu)) + b2 * (K * (N1 * (((2 - 2 * nu) * cot2 + nu)
        / rb * y1 / W6 - ((2 - 2 * nu) * cot2 + 1) * cosB * (y1 / rb - sinB) / W7) - N1 / sq(W6) * (-N1 * y1 * cotB +
        nu * y3b - a + a * y1 * cotB / rb + sq(y1) / W6 * W4) / rb * y1 + N1 / W6 * (-N1 * cotB + a * cotB / rb - a *
        sq(y1) * cotB / rb3 + 2 * y1 / W6 * W4 - cube(y1) / sq(W6) * W4 / rb - cube(y1) / W6 * a / rb3) + N1 * cotB /
        sq(W7) * (z1b * cosB - a * (rb * sinB - y1) / rb / cosB) * (y1 / rb - sinB) - N1 * cotB / W7 * (sq(cosB) - a *
        (1 / rb * sinB * y1 - 1) / rb / cosB + a * (rb * sinB - y1) / rb3 / cosB * y1) - a * W8 * cotB / rb3 + 3 * a *
        sq(y1) * W8 * cotB / rb5 - W8 / sq(W6) * (2 * nu + 1 / rb * (N1 * y1 * cotB + a) - sq(y1) / rb / W6 * W5 - a *
        sq(y1) / rb3) / rb * y1 + W8 / W6 * (-1 / rb3 * (N1 * y1 * cotB + a) * y1 + 1 / rb * N1 * cotB - 2 * y1 / rb /
        W6 * W5 + cube(y1) / rb3 / W6 * W5 + cube(y1) / rb2 / sq(W6) * W5 + cube(y1) / rb4 / W6 * a - 2 * a / rb3 * y1
        + 3 * a * cube(y1) / rb5) - W8 * cotB / sq(W7) * (-cosB * sinB + a * y1 * y3b / rb3 / cosB + (rb * sinB - y1)
        / rb * ((2 - 2 * nu) * cosB - W1 / W7 * W9)) * (y1 / rb - sinB) + W8 * cotB / W7 * (a * y3b / rb3 / cosB - 3 *
        a * sq(y1) * y3b / rb5 / cosB + (1 / rb * sinB * y1 - 1) / rb * ((2 - 2 * nu) * cosB - W1 / W7 * W9) - (rb *
        sinB - y1) / rb3 * ((2 - 2 * nu) * cosB - W1 / W7 * W9) * y1 + (rb * sinB - y1) / rb * (-1 / rb * cosB * y1 /
        W7 * W9 + W1 / sq(W7) * W9 * (y1 / rb - sinB) + W1 / W7 * a / rb3 / cosB * y1))) / math.pi / (1 - nu)) + b3 * (K *
        (N1 * (-y2 / sq(W6) * (1 + a / rb) / rb * y1 - y2 / W6 * a / rb3 * y1 + y2 * cosB / sq(W7) * W2 * (y1 / rb -
        sinB) + y2 * cosB / W7 * a / rb3 * y1) + y2 * W8 / rb3 * (a / rb2 + 1 / W6) * y1 - y2 * W8 / rb * (-2 * a /
        rb4 * y1 - 1 / sq(W6) / rb * y1) - y2 * W8 * cosB / rb3 / W7 * (W1 / W7 * W2 + a * y3b / rb2) * y1 - y2 * W8 *
        cosB / rb / sq(W7) * (W1 / W7 * W2 + a * y3b / rb2) * (y1 / rb - sinB) + y2 * W8 * cosB / rb / W7 * (1 / rb *
        cosB * y1 / W7 * W2 - W1 / sq(W7) * W2 * (y1 / rb - sinB) - W1 / W7 * a / rb3 * y1 - 2 * a * y3b / rb4 * y1))
        / math.pi / (1 - nu)))
    v1 = (
        b1 * (K * (N1 * (((2 - 2 * nu) * cot2 - nu) / rb * y2 / W6 - ((2 - 2 * nu) * cot2 + 1 - 2 * nu) * cosB / rb *
        y2 / W7) + N1 / sq(W6) * (y1 * cotB * (1 - W5) + nu * y3b - a + sq(y2) / W6 * W4) / rb * y2 - N1 / W6 * (a *
        y1 * cotB / rb3 * y2 + 2 * y2 / W6 * W4 - cube(y2) / sq(W6) * W4 / rb - cube(y2) / W6 * a / rb3) + N1 * z1b *
        cotB / sq(W7) * W2 / rb * y2 + N1 * z1b * cotB / W7 * a / rb3 * y2 + 3 * a * y2 * W8 * cotB / rb5 * y1 - W8 /
        sq(W6) * (-2 * nu + 1 / rb * (N1 * y1 * cotB - a) + sq(y2) / rb / W6 * W5 + a * sq(y2) / rb3) / rb * y2 + W8 /
        W6 * (-1 / rb3 * (N1 * y1 * cotB - a) * y2 + 2 * y2 / rb / W6 * W5 - cube(y2) / rb3 / W6 * W5 - cube(y2) / rb2
        / sq(W6) * W5 - cube(y2) / rb4 / W6 * a + 2 * a / rb3 * y2 - 3 * a * cube(y2) / rb5) - W8 / sq(W7) * (sq(cosB)
        - 1 / rb * (N1 * z1b * cotB + a * cosB) + a * y3b * z1b * cotB / rb3 - 1 / rb / W7 * (sq(y2) * sq(cosB) - a *
        z1b * cotB / rb * W1)) / rb * y2 + W8 / W7 * (1 / rb3 * (N1 * z1b * cotB + a * cosB) * y2 - 3 * a * y3b * z1b
        * cotB / rb5 * y2 + 1 / rb3 / W7 * (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1) * y2 + 1 / rb2 / sq(W7) *
        (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1) * y2 - 1 / rb / W7 * (2 * y2 * sq(cosB) + a * z1b * cotB / rb3
        * W1 * y2 - a * z1b * cotB / rb2 * cosB * y2))) / math.pi / (1 - nu)) + b2 * (K * ((2 - 2 * nu) * N1 * rFib_ry2 *
        cot2 + N1 / W6 * ((W5 - 1) * cotB + y1 / W6 * W4) - N1 * sq(y2) / sq(W6) * ((W5 - 1) * cotB + y1 / W6 * W4) /
        rb + N1 * y2 / W6 * (-a / rb3 * y2 * cotB - y1 / sq(W6) * W4 / rb * y2 - y2 / W6 * a / rb3 * y1) - N1 * cotB /
        W7 * W9 + N1 * sq(y2) * cotB / sq(W7) * W9 / rb + N1 * sq(y2) * cotB / W7 * a / rb3 / cosB - a * W8 * cotB /
        rb3 + 3 * a * sq(y2) * W8 * cotB / rb5 + W8 / rb / W6 * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb * (1 / rb
        + 1 / W6)) - sq(y2) * W8 / rb3 / W6 * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb * (1 / rb + 1 / W6)) -
        sq(y2) * W8 / rb2 / sq(W6) * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb * (1 / rb + 1 / W6)) + y2 * W8 / rb /
        W6 * (2 * nu * y1 / sq(W6) / rb * y2 + a * y1 / rb3 * (1 / rb + 1 / W6) * y2 - a * y1 / rb * (-1 / rb3 * y2 -
        1 / sq(W6) / rb * y2)) + W8 * cotB / rb / W7 * ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) -
        sq(y2) * W8 * cotB / rb3 / W7 * ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) - sq(y2) * W8 *
        cotB / rb2 / sq(W7) * ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) + y2 * W8 * cotB / rb / W7
        * (1 / rb * cosB * y2 / W7 * W9 - W1 / sq(W7) * W9 / rb * y2 - W1 / W7 * a / rb3 / cosB * y2 - 2 * a * y3b /
        rb4 / cosB * y2)) / math.pi / (1 - nu)) + b3 * (K * (N1 * (-sinB / rb * y2 / W7 + y2 / sq(W6) * (1 + a / rb) / rb *
        y1 + y2 / W6 * a / rb3 * y1 - z1b / sq(W7) * W2 / rb * y2 - z1b / W7 * a / rb3 * y2) - y2 * W8 / rb3 * (a /
        rb2 + 1 / W6) * y1 + y1 * W8 / rb * (-2 * a / rb4 * y2 - 1 / sq(W6) / rb * y2) + W8 / sq(W7) * (sinB * (cosB -
        a / rb) + z1b / rb * (1 + a * y3b / rb2) - 1 / rb / W7 * (sq(y2) * cosB * sinB - a * z1b / rb * W1)) / rb * y2
        - W8 / W7 * (sinB * a / rb3 * y2 - z1b / rb3 * (1 + a * y3b / rb2) * y2 - 2 * z1b / rb5 * a * y3b * y2 + 1 /
        rb3 / W7 * (sq(y2) * cosB * sinB - a * z1b / rb * W1) * y2 + 1 / rb2 / sq(W7) * (sq(y2) * cosB * sinB - a *
        z1b / rb * W1) * y2 - 1 / rb / W7 * (2 * y2 * cosB * sinB + a * z1b / rb3 * W1 * y2 - a * z1b / rb2 * cosB *
        y2))) / math.pi / (1 - nu)))
    v2 = (
        b1 * (K * ((2 - 2 * nu) * (N1 * rFib_ry3 * cotB - y2 / sq(W6) * W5 * (y3b / rb + 1) - 0.5 * y2 / W6 * a / rb3
        * 2 * y3b + y2 * cosB / sq(W7) * W2 * W3 + 0.5 * y2 * cosB / W7 * a / rb3 * 2 * y3b) + y2 / rb * (2 * nu / W6
        + a / rb2) - 0.5 * y2 * W8 / rb3 * (2 * nu / W6 + a / rb2) * 2 * y3b + y2 * W8 / rb * (-2 * nu / sq(W6) * (y3b
        / rb + 1) - a / rb4 * 2 * y3b) + y2 * cosB / rb / W7 * (1 - 2 * nu - W1 / W7 * W2 - a * y3b / rb2) - 0.5 * y2
        * W8 * cosB / rb3 / W7 * (1 - 2 * nu - W1 / W7 * W2 - a * y3b / rb2) * 2 * y3b - y2 * W8 * cosB / rb / sq(W7)
        * (1 - 2 * nu - W1 / W7 * W2 - a * y3b / rb2) * W3 + y2 * W8 * cosB / rb / W7 * (-(cosB * y3b / rb + 1) / W7 *
        W2 + W1 / sq(W7) * W2 * W3 + 0.5 * W1 / W7 * a / rb3 * 2 * y3b - a / rb2 + a * y3b / rb4 * 2 * y3b)) / math.pi / (1
        - nu)) + b2 * (K * ((-2 + 2 * nu) * N1 * cotB * ((y3b / rb + 1) / W6 - cosB * W3 / W7) + (2 - 2 * nu) * y1 /
        sq(W6) * W5 * (y3b / rb + 1) + 0.5 * (2 - 2 * nu) * y1 / W6 * a / rb3 * 2 * y3b + (2 - 2 * nu) * sinB / W7 *
        W2 - (2 - 2 * nu) * z1b / sq(W7) * W2 * W3 - 0.5 * (2 - 2 * nu) * z1b / W7 * a / rb3 * 2 * y3b + 1 / rb * (N1
        * cotB - 2 * nu * y1 / W6 - a * y1 / rb2) - 0.5 * W8 / rb3 * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb2) * 2
        * y3b + W8 / rb * (2 * nu * y1 / sq(W6) * (y3b / rb + 1) + a * y1 / rb4 * 2 * y3b) - 1 / W7 * (cosB * sinB +
        W1 * cotB / rb * ((2 - 2 * nu) * cosB - W1 / W7) + a / rb * (sinB - y3b * z1b / rb2 - z1b * W1 / rb / W7)) +
        W8 / sq(W7) * (cosB * sinB + W1 * cotB / rb * ((2 - 2 * nu) * cosB - W1 / W7) + a / rb * (sinB - y3b * z1b /
        rb2 - z1b * W1 / rb / W7)) * W3 - W8 / W7 * ((cosB * y3b / rb + 1) * cotB / rb * ((2 - 2 * nu) * cosB - W1 /
        W7) - 0.5 * W1 * cotB / rb3 * ((2 - 2 * nu) * cosB - W1 / W7) * 2 * y3b + W1 * cotB / rb * (-(cosB * y3b / rb
        + 1) / W7 + W1 / sq(W7) * W3) - 0.5 * a / rb3 * (sinB - y3b * z1b / rb2 - z1b * W1 / rb / W7) * 2 * y3b + a /
        rb * (-z1b / rb2 - y3b * sinB / rb2 + y3b * z1b / rb4 * 2 * y3b - sinB * W1 / rb / W7 - z1b * (cosB * y3b / rb
        + 1) / rb / W7 + 0.5 * z1b * W1 / rb3 / W7 * 2 * y3b + z1b * W1 / rb / sq(W7) * W3))) / math.pi / (1 - nu)) + b3 *
        (K * ((2 - 2 * nu) * rFib_ry3 - (2 - 2 * nu) * y2 * sinB / sq(W7) * W2 * W3 - 0.5 * (2 - 2 * nu) * y2 * sinB /
        W7 * a / rb3 * 2 * y3b + y2 * sinB / rb / W7 * (1 + W1 / W7 * W2 + a * y3b / rb2) - 0.5 * y2 * W8 * sinB / rb3
        / W7 * (1 + W1 / W7 * W2 + a * y3b / rb2) * 2 * y3b - y2 * W8 * sinB / rb / sq(W7) * (1 + W1 / W7 * W2 + a *
        y3b / rb2) * W3 + y2 * W8 * sinB / rb / W7 * ((cosB * y3b / rb + 1) / W7 * W2 - W1 / sq(W7) * W2 * W3 - 0.5 *
        W1 / W7 * a / rb3 * 2 * y3b + a / rb2 - a * y3b / rb4 * 2 * y3b)) / math.pi / (1 - nu)))
    v3 = (
        b1 / 2 * (K * ((-2 + 2 * nu) * N1 * rFib_ry2 * cot2 + N1 / W6 * ((1 - W5) * cotB - y1 / W6 * W4) - N1 * sq(y2)
        / sq(W6) * ((1 - W5) * cotB - y1 / W6 * W4) / rb + N1 * y2 / W6 * (a / rb3 * y2 * cotB + y1 / sq(W6) * W4 / rb
        * y2 + y2 / W6 * a / rb3 * y1) + N1 * cosB * cotB / W7 * W2 - N1 * sq(y2) * cosB * cotB / sq(W7) * W2 / rb -
        N1 * sq(y2) * cosB * cotB / W7 * a / rb3 + a * W8 * cotB / rb3 - 3 * a * sq(y2) * W8 * cotB / rb5 + W8 / rb /
        W6 * (-N1 * cotB + y1 / W6 * W5 + a * y1 / rb2) - sq(y2) * W8 / rb3 / W6 * (-N1 * cotB + y1 / W6 * W5 + a * y1
        / rb2) - sq(y2) * W8 / rb2 / sq(W6) * (-N1 * cotB + y1 / W6 * W5 + a * y1 / rb2) + y2 * W8 / rb / W6 * (-y1 /
        sq(W6) * W5 / rb * y2 - y2 / W6 * a / rb3 * y1 - 2 * a * y1 / rb4 * y2) + W8 / rb / W7 * (cosB / W7 * (W1 *
        (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) - a * y3b * cosB * cotB / rb2) - sq(y2)
        * W8 / rb3 / W7 * (cosB / W7 * (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) - a
        * y3b * cosB * cotB / rb2) - sq(y2) * W8 / rb2 / sq(W7) * (cosB / W7 * (W1 * (N1 * cosB - a / rb) * cotB + (2
        - 2 * nu) * (rb * sinB - y1) * cosB) - a * y3b * cosB * cotB / rb2) + y2 * W8 / rb / W7 * (-cosB / sq(W7) *
        (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) / rb * y2 + cosB / W7 * (1 / rb *
        cosB * y2 * (N1 * cosB - a / rb) * cotB + W1 * a / rb3 * y2 * cotB + (2 - 2 * nu) / rb * sinB * y2 * cosB) + 2
        * a * y3b * cosB * cotB / rb4 * y2)) / math.pi / (1 - nu)) + b2 / 2 * (K * (N1 * (((2 - 2 * nu) * cot2 + nu) / rb *
        y2 / W6 - ((2 - 2 * nu) * cot2 + 1) * cosB / rb * y2 / W7) - N1 / sq(W6) * (-N1 * y1 * cotB + nu * y3b - a + a
        * y1 * cotB / rb + sq(y1) / W6 * W4) / rb * y2 + N1 / W6 * (-a * y1 * cotB / rb3 * y2 - sq(y1) / sq(W6) * W4 /
        rb * y2 - sq(y1) / W6 * a / rb3 * y2) + N1 * cotB / sq(W7) * (z1b * cosB - a * (rb * sinB - y1) / rb / cosB) /
        rb * y2 - N1 * cotB / W7 * (-a / rb2 * sinB * y2 / cosB + a * (rb * sinB - y1) / rb3 / cosB * y2) + 3 * a * y2
        * W8 * cotB / rb5 * y1 - W8 / sq(W6) * (2 * nu + 1 / rb * (N1 * y1 * cotB + a) - sq(y1) / rb / W6 * W5 - a *
        sq(y1) / rb3) / rb * y2 + W8 / W6 * (-1 / rb3 * (N1 * y1 * cotB + a) * y2 + sq(y1) / rb3 / W6 * W5 * y2 +
        sq(y1) / rb2 / sq(W6) * W5 * y2 + sq(y1) / rb4 / W6 * a * y2 + 3 * a * sq(y1) / rb5 * y2) - W8 * cotB / sq(W7)
        * (-cosB * sinB + a * y1 * y3b / rb3 / cosB + (rb * sinB - y1) / rb * ((2 - 2 * nu) * cosB - W1 / W7 * W9)) /
        rb * y2 + W8 * cotB / W7 * (-3 * a * y1 * y3b / rb5 / cosB * y2 + 1 / rb2 * sinB * y2 * ((2 - 2 * nu) * cosB -
        W1 / W7 * W9) - (rb * sinB - y1) / rb3 * ((2 - 2 * nu) * cosB - W1 / W7 * W9) * y2 + (rb * sinB - y1) / rb *
        (-1 / rb * cosB * y2 / W7 * W9 + W1 / sq(W7) * W9 / rb * y2 + W1 / W7 * a / rb3 / cosB * y2))) / math.pi / (1 -
        nu)) + b3 / 2 * (K * (N1 * (1 / W6 * (1 + a / rb) - sq(y2) / sq(W6) * (1 + a / rb) / rb - sq(y2) / W6 * a /
        rb3 - cosB / W7 * W2 + sq(y2) * cosB / sq(W7) * W2 / rb + sq(y2) * cosB / W7 * a / rb3) - W8 / rb * (a / rb2 +
        1 / W6) + sq(y2) * W8 / rb3 * (a / rb2 + 1 / W6) - y2 * W8 / rb * (-2 * a / rb4 * y2 - 1 / sq(W6) / rb * y2) +
        W8 * cosB / rb / W7 * (W1 / W7 * W2 + a * y3b / rb2) - sq(y2) * W8 * cosB / rb3 / W7 * (W1 / W7 * W2 + a * y3b
        / rb2) - sq(y2) * W8 * cosB / rb2 / sq(W7) * (W1 / W7 * W2 + a * y3b / rb2) + y2 * W8 * cosB / rb / W7 * (1 /
        rb * cosB * y2 / W7 * W2 - W1 / sq(W7) * W2 / rb * y2 - W1 / W7 * a / rb3 * y2 - 2 * a * y3b / rb4 * y2)) / math.pi
        / (1 - nu)) + b1 / 2 * (K * (N1 * (((2 - 2 * nu) * cot2 - nu) / rb * y1 / W6 - ((2 - 2 * nu) * cot2 + 1 - 2 *
        nu) * cosB * (y1 / rb - sinB) / W7) + N1 / sq(W6) * (y1 * cotB * (1 - W5) + nu * y3b - a + sq(y2) / W6 * W4) /
        rb * y1 - N1 / W6 * ((1 - W5) * cotB + a * sq(y1) * cotB / rb3 - sq(y2) / sq(W6) * W4 / rb * y1 - sq(y2) / W6
        * a / rb3 * y1) - N1 * cosB * cotB / W7 * W2 + N1 * z1b * cotB / sq(W7) * W2 * (y1 / rb - sinB) + N1 * z1b *
        cotB / W7 * a / rb3 * y1 - a * W8 * cotB / rb3 + 3 * a * sq(y1) * W8 * cotB / rb5 - W8 / sq(W6) * (-2 * nu + 1
        / rb * (N1 * y1 * cotB - a) + sq(y2) / rb / W6 * W5 + a * sq(y2) / rb3) / rb * y1 + W8 / W6 * (-1 / rb3 * (N1
        * y1 * cotB - a) * y1 + 1 / rb * N1 * cotB - sq(y2) / rb3 / W6 * W5 * y1 - sq(y2) / rb2 / sq(W6) * W5 * y1 -
        sq(y2) / rb4 / W6 * a * y1 - 3 * a * sq(y2) / rb5 * y1) - W8 / sq(W7) * (sq(cosB) - 1 / rb * (N1 * z1b * cotB
        + a * cosB) + a * y3b * z1b * cotB / rb3 - 1 / rb / W7 * (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1)) * (y1
        / rb - sinB) + W8 / W7 * (1 / rb3 * (N1 * z1b * cotB + a * cosB) * y1 - 1 / rb * N1 * cosB * cotB + a * y3b *
        cosB * cotB / rb3 - 3 * a * y3b * z1b * cotB / rb5 * y1 + 1 / rb3 / W7 * (sq(y2) * sq(cosB) - a * z1b * cotB /
        rb * W1) * y1 + 1 / rb / sq(W7) * (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1) * (y1 / rb - sinB) - 1 / rb /
        W7 * (-a * cosB * cotB / rb * W1 + a * z1b * cotB / rb3 * W1 * y1 - a * z1b * cotB / rb2 * cosB * y1))) / math.pi /
        (1 - nu)) + b2 / 2 * (K * ((2 - 2 * nu) * N1 * rFib_ry1 * cot2 - N1 * y2 / sq(W6) * ((W5 - 1) * cotB + y1 / W6
        * W4) / rb * y1 + N1 * y2 / W6 * (-a / rb3 * y1 * cotB + 1 / W6 * W4 - sq(y1) / sq(W6) * W4 / rb - sq(y1) / W6
        * a / rb3) + N1 * y2 * cotB / sq(W7) * W9 * (y1 / rb - sinB) + N1 * y2 * cotB / W7 * a / rb3 / cosB * y1 + 3 *
        a * y2 * W8 * cotB / rb5 * y1 - y2 * W8 / rb3 / W6 * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb * (1 / rb + 1
        / W6)) * y1 - y2 * W8 / rb2 / sq(W6) * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb * (1 / rb + 1 / W6)) * y1 +
        y2 * W8 / rb / W6 * (-2 * nu / W6 + 2 * nu * sq(y1) / sq(W6) / rb - a / rb * (1 / rb + 1 / W6) + a * sq(y1) /
        rb3 * (1 / rb + 1 / W6) - a * y1 / rb * (-1 / rb3 * y1 - 1 / sq(W6) / rb * y1)) - y2 * W8 * cotB / rb3 / W7 *
        ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) * y1 - y2 * W8 * cotB / rb / sq(W7) * ((-2 + 2 *
        nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) * (y1 / rb - sinB) + y2 * W8 * cotB / rb / W7 * (1 / rb *
        cosB * y1 / W7 * W9 - W1 / sq(W7) * W9 * (y1 / rb - sinB) - W1 / W7 * a / rb3 / cosB * y1 - 2 * a * y3b / rb4
        / cosB * y1)) / math.pi / (1 - nu)) + b3 / 2 * (K * (N1 * (-sinB * (y1 / rb - sinB) / W7 - 1 / W6 * (1 + a / rb) +
        sq(y1) / sq(W6) * (1 + a / rb) / rb + sq(y1) / W6 * a / rb3 + cosB / W7 * W2 - z1b / sq(W7) * W2 * (y1 / rb -
        sinB) - z1b / W7 * a / rb3 * y1) + W8 / rb * (a / rb2 + 1 / W6) - sq(y1) * W8 / rb3 * (a / rb2 + 1 / W6) + y1
        * W8 / rb * (-2 * a / rb4 * y1 - 1 / sq(W6) / rb * y1) + W8 / sq(W7) * (sinB * (cosB - a / rb) + z1b / rb * (1
        + a * y3b / rb2) - 1 / rb / W7 * (sq(y2) * cosB * sinB - a * z1b / rb * W1)) * (y1 / rb - sinB) - W8 / W7 *
        (sinB * a / rb3 * y1 + cosB / rb * (1 + a * y3b / rb2) - z1b / rb3 * (1 + a * y3b / rb2) * y1 - 2 * z1b / rb5
        * a * y3b * y1 + 1 / rb3 / W7 * (sq(y2) * cosB * sinB - a * z1b / rb * W1) * y1 + 1 / rb / sq(W7) * (sq(y2) *
        cosB * sinB - a * z1b / rb * W1) * (y1 / rb - sinB) - 1 / rb / W7 * (-a * cosB / rb * W1 + a * z1b / rb3 * W1
        * y1 - a * z1b / rb2 * cosB * y1))) / math.pi / (1 - nu)))
    v4 = (
        b1 / 2 * (K * ((-2 + 2 * nu) * N1 * rFib_ry3 * cot2 - N1 * y2 / sq(W6) * ((1 - W5) * cotB - y1 / W6 * W4) *
        (y3b / rb + 1) + N1 * y2 / W6 * (0.5 * a / rb3 * 2 * y3b * cotB + y1 / sq(W6) * W4 * (y3b / rb + 1) + 0.5 * y1
        / W6 * a / rb3 * 2 * y3b) - N1 * y2 * cosB * cotB / sq(W7) * W2 * W3 - 0.5 * N1 * y2 * cosB * cotB / W7 * a /
        rb3 * 2 * y3b + a / rb3 * y2 * cotB - 1.5 * a * y2 * W8 * cotB / rb5 * 2 * y3b + y2 / rb / W6 * (-N1 * cotB +
        y1 / W6 * W5 + a * y1 / rb2) - 0.5 * y2 * W8 / rb3 / W6 * (-N1 * cotB + y1 / W6 * W5 + a * y1 / rb2) * 2 * y3b
        - y2 * W8 / rb / sq(W6) * (-N1 * cotB + y1 / W6 * W5 + a * y1 / rb2) * (y3b / rb + 1) + y2 * W8 / rb / W6 *
        (-y1 / sq(W6) * W5 * (y3b / rb + 1) - 0.5 * y1 / W6 * a / rb3 * 2 * y3b - a * y1 / rb4 * 2 * y3b) + y2 / rb /
        W7 * (cosB / W7 * (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) - a * y3b * cosB
        * cotB / rb2) - 0.5 * y2 * W8 / rb3 / W7 * (cosB / W7 * (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb
        * sinB - y1) * cosB) - a * y3b * cosB * cotB / rb2) * 2 * y3b - y2 * W8 / rb / sq(W7) * (cosB / W7 * (W1 * (N1
        * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) - a * y3b * cosB * cotB / rb2) * W3 + y2 *
        W8 / rb / W7 * (-cosB / sq(W7) * (W1 * (N1 * cosB - a / rb) * cotB + (2 - 2 * nu) * (rb * sinB - y1) * cosB) *
        W3 + cosB / W7 * ((cosB * y3b / rb + 1) * (N1 * cosB - a / rb) * cotB + 0.5 * W1 * a / rb3 * 2 * y3b * cotB +
        0.5 * (2 - 2 * nu) / rb * sinB * 2 * y3b * cosB) - a * cosB * cotB / rb2 + a * y3b * cosB * cotB / rb4 * 2 *
        y3b)) / math.pi / (1 - nu)) + b2 / 2 * (K * (N1 * (((2 - 2 * nu) * cot2 + nu) * (y3b / rb + 1) / W6 - ((2 - 2 * nu)
        * cot2 + 1) * cosB * W3 / W7) - N1 / sq(W6) * (-N1 * y1 * cotB + nu * y3b - a + a * y1 * cotB / rb + sq(y1) /
        W6 * W4) * (y3b / rb + 1) + N1 / W6 * (nu - 0.5 * a * y1 * cotB / rb3 * 2 * y3b - sq(y1) / sq(W6) * W4 * (y3b
        / rb + 1) - 0.5 * sq(y1) / W6 * a / rb3 * 2 * y3b) + N1 * cotB / sq(W7) * (z1b * cosB - a * (rb * sinB - y1) /
        rb / cosB) * W3 - N1 * cotB / W7 * (cosB * sinB - 0.5 * a / rb2 * sinB * 2 * y3b / cosB + 0.5 * a * (rb * sinB
        - y1) / rb3 / cosB * 2 * y3b) - a / rb3 * y1 * cotB + 1.5 * a * y1 * W8 * cotB / rb5 * 2 * y3b + 1 / W6 * (2 *
        nu + 1 / rb * (N1 * y1 * cotB + a) - sq(y1) / rb / W6 * W5 - a * sq(y1) / rb3) - W8 / sq(W6) * (2 * nu + 1 /
        rb * (N1 * y1 * cotB + a) - sq(y1) / rb / W6 * W5 - a * sq(y1) / rb3) * (y3b / rb + 1) + W8 / W6 * (-0.5 / rb3
        * (N1 * y1 * cotB + a) * 2 * y3b + 0.5 * sq(y1) / rb3 / W6 * W5 * 2 * y3b + sq(y1) / rb / sq(W6) * W5 * (y3b /
        rb + 1) + 0.5 * sq(y1) / rb4 / W6 * a * 2 * y3b + 1.5 * a * sq(y1) / rb5 * 2 * y3b) + cotB / W7 * (-cosB *
        sinB + a * y1 * y3b / rb3 / cosB + (rb * sinB - y1) / rb * ((2 - 2 * nu) * cosB - W1 / W7 * W9)) - W8 * cotB /
        sq(W7) * (-cosB * sinB + a * y1 * y3b / rb3 / cosB + (rb * sinB - y1) / rb * ((2 - 2 * nu) * cosB - W1 / W7 *
        W9)) * W3 + W8 * cotB / W7 * (a / rb3 / cosB * y1 - 1.5 * a * y1 * y3b / rb5 / cosB * 2 * y3b + 0.5 / rb2 *
        sinB * 2 * y3b * ((2 - 2 * nu) * cosB - W1 / W7 * W9) - 0.5 * (rb * sinB - y1) / rb3 * ((2 - 2 * nu) * cosB -
        W1 / W7 * W9) * 2 * y3b + (rb * sinB - y1) / rb * (-(cosB * y3b / rb + 1) / W7 * W9 + W1 / sq(W7) * W9 * W3 +
        0.5 * W1 / W7 * a / rb3 / cosB * 2 * y3b))) / math.pi / (1 - nu)) + b3 / 2 * (K * (N1 * (-y2 / sq(W6) * (1 + a /
        rb) * (y3b / rb + 1) - 0.5 * y2 / W6 * a / rb3 * 2 * y3b + y2 * cosB / sq(W7) * W2 * W3 + 0.5 * y2 * cosB / W7
        * a / rb3 * 2 * y3b) - y2 / rb * (a / rb2 + 1 / W6) + 0.5 * y2 * W8 / rb3 * (a / rb2 + 1 / W6) * 2 * y3b - y2
        * W8 / rb * (-a / rb4 * 2 * y3b - 1 / sq(W6) * (y3b / rb + 1)) + y2 * cosB / rb / W7 * (W1 / W7 * W2 + a * y3b
        / rb2) - 0.5 * y2 * W8 * cosB / rb3 / W7 * (W1 / W7 * W2 + a * y3b / rb2) * 2 * y3b - y2 * W8 * cosB / rb /
        sq(W7) * (W1 / W7 * W2 + a * y3b / rb2) * W3 + y2 * W8 * cosB / rb / W7 * ((cosB * y3b / rb + 1) / W7 * W2 -
        W1 / sq(W7) * W2 * W3 - 0.5 * W1 / W7 * a / rb3 * 2 * y3b + a / rb2 - a * y3b / rb4 * 2 * y3b)) / math.pi / (1 -
        nu)) + b1 / 2 * (K * ((2 - 2 * nu) * (N1 * rFib_ry1 * cotB - y1 / sq(W6) * W5 / rb * y2 - y2 / W6 * a / rb3 *
        y1 + y2 * cosB / sq(W7) * W2 * (y1 / rb - sinB) + y2 * cosB / W7 * a / rb3 * y1) - y2 * W8 / rb3 * (2 * nu /
        W6 + a / rb2) * y1 + y2 * W8 / rb * (-2 * nu / sq(W6) / rb * y1 - 2 * a / rb4 * y1) - y2 * W8 * cosB / rb3 /
        W7 * (1 - 2 * nu - W1 / W7 * W2 - a * y3b / rb2) * y1 - y2 * W8 * cosB / rb / sq(W7) * (1 - 2 * nu - W1 / W7 *
        W2 - a * y3b / rb2) * (y1 / rb - sinB) + y2 * W8 * cosB / rb / W7 * (-1 / rb * cosB * y1 / W7 * W2 + W1 /
        sq(W7) * W2 * (y1 / rb - sinB) + W1 / W7 * a / rb3 * y1 + 2 * a * y3b / rb4 * y1)) / math.pi / (1 - nu)) + b2 / 2 *
        (K * ((-2 + 2 * nu) * N1 * cotB * (1 / rb * y1 / W6 - cosB * (y1 / rb - sinB) / W7) - (2 - 2 * nu) / W6 * W5 +
        (2 - 2 * nu) * sq(y1) / sq(W6) * W5 / rb + (2 - 2 * nu) * sq(y1) / W6 * a / rb3 + (2 - 2 * nu) * cosB / W7 *
        W2 - (2 - 2 * nu) * z1b / sq(W7) * W2 * (y1 / rb - sinB) - (2 - 2 * nu) * z1b / W7 * a / rb3 * y1 - W8 / rb3 *
        (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb2) * y1 + W8 / rb * (-2 * nu / W6 + 2 * nu * sq(y1) / sq(W6) / rb -
        a / rb2 + 2 * a * sq(y1) / rb4) + W8 / sq(W7) * (cosB * sinB + W1 * cotB / rb * ((2 - 2 * nu) * cosB - W1 /
        W7) + a / rb * (sinB - y3b * z1b / rb2 - z1b * W1 / rb / W7)) * (y1 / rb - sinB) - W8 / W7 * (1 / rb2 * cosB *
        y1 * cotB * ((2 - 2 * nu) * cosB - W1 / W7) - W1 * cotB / rb3 * ((2 - 2 * nu) * cosB - W1 / W7) * y1 + W1 *
        cotB / rb * (-1 / rb * cosB * y1 / W7 + W1 / sq(W7) * (y1 / rb - sinB)) - a / rb3 * (sinB - y3b * z1b / rb2 -
        z1b * W1 / rb / W7) * y1 + a / rb * (-y3b * cosB / rb2 + 2 * y3b * z1b / rb4 * y1 - cosB * W1 / rb / W7 - z1b
        / rb2 * cosB * y1 / W7 + z1b * W1 / rb3 / W7 * y1 + z1b * W1 / rb / sq(W7) * (y1 / rb - sinB)))) / math.pi / (1 -
        nu)) + b3 / 2 * (K * ((2 - 2 * nu) * rFib_ry1 - (2 - 2 * nu) * y2 * sinB / sq(W7) * W2 * (y1 / rb - sinB) - (2
        - 2 * nu) * y2 * sinB / W7 * a / rb3 * y1 - y2 * W8 * sinB / rb3 / W7 * (1 + W1 / W7 * W2 + a * y3b / rb2) *
        y1 - y2 * W8 * sinB / rb / sq(W7) * (1 + W1 / W7 * W2 + a * y3b / rb2) * (y1 / rb - sinB) + y2 * W8 * sinB /
        rb / W7 * (1 / rb * cosB * y1 / W7 * W2 - W1 / sq(W7) * W2 * (y1 / rb - sinB) - W1 / W7 * a / rb3 * y1 - 2 * a
        * y3b / rb4 * y1)) / math.pi / (1 - nu)))
    v5 = (
        b1 / 2 * (K * (N1 * (((2 - 2 * nu) * cot2 - nu) * (y3b / rb + 1) / W6 - ((2 - 2 * nu) * cot2 + 1 - 2 * nu) *
        cosB * W3 / W7) + N1 / sq(W6) * (y1 * cotB * (1 - W5) + nu * y3b - a + sq(y2) / W6 * W4) * (y3b / rb + 1) - N1
        / W6 * (0.5 * a * y1 * cotB / rb3 * 2 * y3b + nu - sq(y2) / sq(W6) * W4 * (y3b / rb + 1) - 0.5 * sq(y2) / W6 *
        a / rb3 * 2 * y3b) - N1 * sinB * cotB / W7 * W2 + N1 * z1b * cotB / sq(W7) * W2 * W3 + 0.5 * N1 * z1b * cotB /
        W7 * a / rb3 * 2 * y3b - a / rb3 * y1 * cotB + 1.5 * a * y1 * W8 * cotB / rb5 * 2 * y3b + 1 / W6 * (-2 * nu +
        1 / rb * (N1 * y1 * cotB - a) + sq(y2) / rb / W6 * W5 + a * sq(y2) / rb3) - W8 / sq(W6) * (-2 * nu + 1 / rb *
        (N1 * y1 * cotB - a) + sq(y2) / rb / W6 * W5 + a * sq(y2) / rb3) * (y3b / rb + 1) + W8 / W6 * (-0.5 / rb3 *
        (N1 * y1 * cotB - a) * 2 * y3b - 0.5 * sq(y2) / rb3 / W6 * W5 * 2 * y3b - sq(y2) / rb / sq(W6) * W5 * (y3b /
        rb + 1) - 0.5 * sq(y2) / rb4 / W6 * a * 2 * y3b - 1.5 * a * sq(y2) / rb5 * 2 * y3b) + 1 / W7 * (sq(cosB) - 1 /
        rb * (N1 * z1b * cotB + a * cosB) + a * y3b * z1b * cotB / rb3 - 1 / rb / W7 * (sq(y2) * sq(cosB) - a * z1b *
        cotB / rb * W1)) - W8 / sq(W7) * (sq(cosB) - 1 / rb * (N1 * z1b * cotB + a * cosB) + a * y3b * z1b * cotB /
        rb3 - 1 / rb / W7 * (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1)) * W3 + W8 / W7 * (0.5 / rb3 * (N1 * z1b *
        cotB + a * cosB) * 2 * y3b - 1 / rb * N1 * sinB * cotB + a * z1b * cotB / rb3 + a * y3b * sinB * cotB / rb3 -
        1.5 * a * y3b * z1b * cotB / rb5 * 2 * y3b + 0.5 / rb3 / W7 * (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1) *
        2 * y3b + 1 / rb / sq(W7) * (sq(y2) * sq(cosB) - a * z1b * cotB / rb * W1) * W3 - 1 / rb / W7 * (-a * sinB *
        cotB / rb * W1 + 0.5 * a * z1b * cotB / rb3 * W1 * 2 * y3b - a * z1b * cotB / rb * (cosB * y3b / rb + 1)))) /
        math.pi / (1 - nu)) + b2 / 2 * (K * ((2 - 2 * nu) * N1 * rFib_ry3 * cot2 - N1 * y2 / sq(W6) * ((W5 - 1) * cotB + y1
        / W6 * W4) * (y3b / rb + 1) + N1 * y2 / W6 * (-0.5 * a / rb3 * 2 * y3b * cotB - y1 / sq(W6) * W4 * (y3b / rb +
        1) - 0.5 * y1 / W6 * a / rb3 * 2 * y3b) + N1 * y2 * cotB / sq(W7) * W9 * W3 + 0.5 * N1 * y2 * cotB / W7 * a /
        rb3 / cosB * 2 * y3b - a / rb3 * y2 * cotB + 1.5 * a * y2 * W8 * cotB / rb5 * 2 * y3b + y2 / rb / W6 * (N1 *
        cotB - 2 * nu * y1 / W6 - a * y1 / rb * (1 / rb + 1 / W6)) - 0.5 * y2 * W8 / rb3 / W6 * (N1 * cotB - 2 * nu *
        y1 / W6 - a * y1 / rb * (1 / rb + 1 / W6)) * 2 * y3b - y2 * W8 / rb / sq(W6) * (N1 * cotB - 2 * nu * y1 / W6 -
        a * y1 / rb * (1 / rb + 1 / W6)) * (y3b / rb + 1) + y2 * W8 / rb / W6 * (2 * nu * y1 / sq(W6) * (y3b / rb + 1)
        + 0.5 * a * y1 / rb3 * (1 / rb + 1 / W6) * 2 * y3b - a * y1 / rb * (-0.5 / rb3 * 2 * y3b - 1 / sq(W6) * (y3b /
        rb + 1))) + y2 * cotB / rb / W7 * ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) - 0.5 * y2 * W8
        * cotB / rb3 / W7 * ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) * 2 * y3b - y2 * W8 * cotB /
        rb / sq(W7) * ((-2 + 2 * nu) * cosB + W1 / W7 * W9 + a * y3b / rb2 / cosB) * W3 + y2 * W8 * cotB / rb / W7 *
        ((cosB * y3b / rb + 1) / W7 * W9 - W1 / sq(W7) * W9 * W3 - 0.5 * W1 / W7 * a / rb3 / cosB * 2 * y3b + a / rb2
        / cosB - a * y3b / rb4 / cosB * 2 * y3b)) / math.pi / (1 - nu)) + b3 / 2 * (K * (N1 * (-sinB * W3 / W7 + y1 /
        sq(W6) * (1 + a / rb) * (y3b / rb + 1) + 0.5 * y1 / W6 * a / rb3 * 2 * y3b + sinB / W7 * W2 - z1b / sq(W7) *
        W2 * W3 - 0.5 * z1b / W7 * a / rb3 * 2 * y3b) + y1 / rb * (a / rb2 + 1 / W6) - 0.5 * y1 * W8 / rb3 * (a / rb2
        + 1 / W6) * 2 * y3b + y1 * W8 / rb * (-a / rb4 * 2 * y3b - 1 / sq(W6) * (y3b / rb + 1)) - 1 / W7 * (sinB *
        (cosB - a / rb) + z1b / rb * (1 + a * y3b / rb2) - 1 / rb / W7 * (sq(y2) * cosB * sinB - a * z1b / rb * W1)) +
        W8 / sq(W7) * (sinB * (cosB - a / rb) + z1b / rb * (1 + a * y3b / rb2) - 1 / rb / W7 * (sq(y2) * cosB * sinB -
        a * z1b / rb * W1)) * W3 - W8 / W7 * (0.5 * sinB * a / rb3 * 2 * y3b + sinB / rb * (1 + a * y3b / rb2) - 0.5 *
        z1b / rb3 * (1 + a * y3b / rb2) * 2 * y3b + z1b / rb * (a / rb2 - a * y3b / rb4 * 2 * y3b) + 0.5 / rb3 / W7 *
        (sq(y2) * cosB * sinB - a * z1b / rb * W1) * 2 * y3b + 1 / rb / sq(W7) * (sq(y2) * cosB * sinB - a * z1b / rb
        * W1) * W3 - 1 / rb / W7 * (-a * sinB / rb * W1 + 0.5 * a * z1b / rb3 * W1 * 2 * y3b - a * z1b / rb * (cosB *
        y3b / rb + 1)))) / math.pi / (1 - nu)) + b1 / 2 * (K * ((2 - 2 * nu) * (N1 * rFib_ry2 * cotB + 1 / W6 * W5 - sq(y2)
        / sq(W6) * W5 / rb - sq(y2) / W6 * a / rb3 - cosB / W7 * W2 + sq(y2) * cosB / sq(W7) * W2 / rb + sq(y2) * cosB
        / W7 * a / rb3) + W8 / rb * (2 * nu / W6 + a / rb2) - sq(y2) * W8 / rb3 * (2 * nu / W6 + a / rb2) + y2 * W8 /
        rb * (-2 * nu / sq(W6) / rb * y2 - 2 * a / rb4 * y2) + W8 * cosB / rb / W7 * (1 - 2 * nu - W1 / W7 * W2 - a *
        y3b / rb2) - sq(y2) * W8 * cosB / rb3 / W7 * (1 - 2 * nu - W1 / W7 * W2 - a * y3b / rb2) - sq(y2) * W8 * cosB
        / rb2 / sq(W7) * (1 - 2 * nu - W1 / W7 * W2 - a * y3b / rb2) + y2 * W8 * cosB / rb / W7 * (-1 / rb * cosB * y2
        / W7 * W2 + W1 / sq(W7) * W2 / rb * y2 + W1 / W7 * a / rb3 * y2 + 2 * a * y3b / rb4 * y2)) / math.pi / (1 - nu)) +
        b2 / 2 * (K * ((-2 + 2 * nu) * N1 * cotB * (1 / rb * y2 / W6 - cosB / rb * y2 / W7) + (2 - 2 * nu) * y1 /
        sq(W6) * W5 / rb * y2 + (2 - 2 * nu) * y1 / W6 * a / rb3 * y2 - (2 - 2 * nu) * z1b / sq(W7) * W2 / rb * y2 -
        (2 - 2 * nu) * z1b / W7 * a / rb3 * y2 - W8 / rb3 * (N1 * cotB - 2 * nu * y1 / W6 - a * y1 / rb2) * y2 + W8 /
        rb * (2 * nu * y1 / sq(W6) / rb * y2 + 2 * a * y1 / rb4 * y2) + W8 / sq(W7) * (cosB * sinB + W1 * cotB / rb *
        ((2 - 2 * nu) * cosB - W1 / W7) + a / rb * (sinB - y3b * z1b / rb2 - z1b * W1 / rb / W7)) / rb * y2 - W8 / W7
        * (1 / rb2 * cosB * y2 * cotB * ((2 - 2 * nu) * cosB - W1 / W7) - W1 * cotB / rb3 * ((2 - 2 * nu) * cosB - W1
        / W7) * y2 + W1 * cotB / rb * (-cosB / rb * y2 / W7 + W1 / sq(W7) / rb * y2) - a / rb3 * (sinB - y3b * z1b /
        rb2 - z1b * W1 / rb / W7) * y2 + a / rb * (2 * y3b * z1b / rb4 * y2 - z1b / rb2 * cosB * y2 / W7 + z1b * W1 /
        rb3 / W7 * y2 + z1b * W1 / rb2 / sq(W7) * y2))) / math.pi / (1 - nu)) + b3 / 2 * (K * ((2 - 2 * nu) * rFib_ry2 + (2
        - 2 * nu) * sinB / W7 * W2 - (2 - 2 * nu) * sq(y2) * sinB / sq(W7) * W2 / rb - (2 - 2 * nu) * sq(y2) * sinB /
        W7 * a / rb3 + W8 * sinB / rb / W7 * (1 + W1 / W7 * W2 + a * y3b / rb2) - sq(y2) * W8 * sinB / rb3 / W7 * (1 +
        W1 / W7 * W2 + a * y3b / rb2) - sq(y2) * W8 * sinB / rb2 / sq(W7) * (1 + W1 / W7 * W2 + a * y3b / rb2) + y2 *
        W8 * sinB / rb / W7 * (1 / rb * cosB * y2 / W7 * W2 - W1 / sq(W7) * W2 / rb * y2 - W1 / W7 * a / rb3 * y2 - 2
        * a * y3b / rb4 * y2)) / math.pi / (1 - nu)))
    return v0, v1, v2, v3, v4, v5


def _mat(e):
    return [[e[0], e[3], e[4]], [e[3], e[1], e[5]], [e[4], e[5], e[2]]]


def _rotated(e, B):
    """Components of the symmetric tensor e = sum_ij e_ij B_i B_j on the fixed
    axes; B: the three axes it is given on, as rows of components."""
    M = _mat(e)
    at = lambda i, j: sum(B[m][i] * sum(M[m][n] * B[n][j] for n in range(3)) for m in range(3))  # noqa: E731
    return [at(0, 0), at(1, 1), at(2, 2), at(0, 1), at(0, 2), at(1, 2)]


def _dot(a, b):
    return sum(x * y for x, y in zip(a, b))


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _unit(a):
    n = torch.sqrt(_dot(a, a))
    return [x / n for x in a]


def _minus(a, b):
    return [x - y for x, y in zip(a, b)]


def _axes(P):
    n = _unit(_cross(_minus(P[1], P[0]), _minus(P[2], P[0])))
    s = _unit([-n[1], n[0], torch.zeros_like(n[0])])
    return n, s, _cross(n, s)


def _triangle_full_space(x, P, slip, nu):
    """Strains of a triangular dislocation in a full space on the fixed axes."""
    n, s, d = axes = _axes(P)
    local = lambda v: [_dot(v, t) for t in axes]  # noqa: E731
    p = [local(_minus(q, P[1])) for q in P]
    x = local(_minus(x, P[1]))
    e12, e13, e23 = (_unit(_minus(p[j], p[i])) for i, j in ((0, 1), (0, 2), (1, 2)))
    neg = lambda v: [-t for t in v]  # noqa: E731
    A, B, C = torch.acos(_dot(e12, e13)), torch.acos(-_dot(e12, e23)), torch.acos(_dot(e23, e13))
    (x1, y1), (x2, y2), (x3, y3) = ((q[1], q[2]) for q in p)
    den = (y2 - y3) * (x1 - x3) + (x3 - x2) * (y1 - y3)
    a = ((y2 - y3) * (x[1] - x3) + (x3 - x2) * (x[2] - y3)) / den
    b = ((y3 - y1) * (x[1] - x3) + (x1 - x3) * (x[2] - y3)) / den
    c = 1 - a - b
    minus = ((a <= 0) & (b > c) & (c > a)) | ((b <= 0) & (c > a) & (a > b)) | ((c <= 0) & (a > b) & (b > c))
    one, parts = torch.where(minus, -torch.ones_like(a), torch.ones_like(a)), []
    for angle, at, side in ((A, p[0], neg(e13)), (B, p[1], e12), (C, p[2], e23)):
        sv = [one * t for t in side]
        ry, rz = x[1] - at[1], x[2] - at[2]
        e = _ang_dis_strain(x[0], sv[2] * ry - sv[1] * rz, sv[1] * ry + sv[2] * rz, angle - math.pi, slip[0],
                            sv[2] * slip[1] - sv[1] * slip[2], sv[1] * slip[1] + sv[2] * slip[2], nu)
        z, o = torch.zeros_like(a), torch.ones_like(a)
        parts.append(_rotated(e, [[o, z, z], [z, sv[2], -sv[1]], [z, sv[1], sv[2]]]))
    return _rotated([sum(t) for t in zip(*parts)], [n, s, d])


def _side_correction(x, b, PA, PB, nu):
    """Free-surface correction strains of one triangle side on the fixed axes."""
    sv = _minus(PB, PA)
    beta = torch.acos(-sv[2] / torch.sqrt(_dot(sv, sv)))
    z, o = torch.zeros_like(beta), torch.ones_like(beta)
    h1 = _unit([sv[0], sv[1], z])
    axes = [h1, _cross([z, z, -o], h1), [z, z, -o]]
    # coordinates with the axes as columns of the transform (the first two
    # rows of that matrix are symmetric up to the sign of the second axis)
    on = lambda v: [sum(axes[j][i] * v[j] for j in range(3)) for i in range(3)]  # noqa: E731
    yA, yAB, bb = on(_minus(x, PA)), on(sv), on(b)
    yB = _minus(yA, yAB)
    first = beta * yA[0] >= 0
    f = torch.where(first, -o, o)
    ang = torch.where(first, math.pi - beta, beta)
    vA = _ang_dis_strain_fsc(f * yA[0], f * yA[1], yA[2], ang, f * bb[0], f * bb[1], bb[2], nu, -PA[2])
    vB = _ang_dis_strain_fsc(f * yB[0], f * yB[1], yB[2], ang, f * bb[0], f * bb[1], bb[2], nu, -PB[2])
    v = _minus(vB, vA)
    v[4], v[5] = f * v[4], f * v[5]
    return _rotated(v, [list(r) for r in zip(*axes)])


def _tri64(tri, r, s, chunk=1 << 19):
    """(Ks, Kn) of receiver triangles r and source triangles s (index tensors)."""
    lam = 2 * G * NU / (1 - 2 * NU)
    nu = 1 / (1 + lam / G) / 2
    P1, P2, P3, rake, cen, nh, sh = (_cuda(t) for t in tri)
    Ks, Kn = torch.empty(len(r), dtype=torch.float64, device="cuda"), torch.empty(len(r), dtype=torch.float64,
                                                                                  device="cuda")
    for k in range(0, len(r), chunk):
        rr, q = r[k:k + chunk], s[k:k + chunk]
        x = list(cen[rr].T)
        P = [list(p[q].T) for p in (P1, P2, P3)]
        sn, cs = _sincosd(rake[q])
        slip = [torch.zeros_like(sn), -cs, sn]
        E = _triangle_full_space(x, P, slip, nu)
        b = [sum(t[i] * w for t, w in zip(_axes(P), slip)) for i in range(3)]
        for i, j in ((0, 1), (1, 2), (2, 0)):
            E = [u + w for u, w in zip(E, _side_correction(x, b, P[i], P[j], nu))]
        image = [[p[0], p[1], -p[2]] for p in P]
        E = [u + w for u, w in zip(E, _triangle_full_space(x, image, slip, nu))]
        tr = lam * (E[0] + E[1] + E[2])
        M = _mat([2 * G * E[i] + (tr if i < 3 else 0) for i in range(6)])
        n, v = list(nh[rr].T), list(sh[rr].T)
        t = [_dot(row, n) for row in M]
        Ks[k:k + chunk], Kn[k:k + chunk] = _dot(t, v), _dot(t, n)
    return Ks, Kn


class _Unusual(Exception):
    """A step that the plain solution below does not cover (a halved or retried step)."""


def _solve_low(x, V, grad=False):
    """Root of the low-velocity step V = V0 exp((mu(V) - F0 - b ln(V0 theta / Dc)) / a)."""
    for it in range(30):
        den = 1 + x["dt"] * V / x["Dc"]
        th = (x["th"] + x["dt"]) / den
        D = x["D"] + (x["V"] + V) / 2 * x["dt"]
        mu = (x["K"] * (x["tld"] - D) + x["tau0"] - x["eta"] * V + x["dtau"] - x["M"] * (V - x["V"]) / x["dt"]) / x["sig"]
        W = 1e-9 * torch.exp((mu - x["F0"] - x["b"] * torch.log(1e-9 * th / x["Dc"])) / x["a"])
        dmu = -(x["K"] * x["dt"] / 2 + x["eta"] + x["M"] / x["dt"]) / x["sig"]
        slope = 1 - W * (dmu + x["b"] * x["dt"] / x["Dc"] / den) / x["a"]
        if grad:   # one step from the root carries the root's derivatives
            return V - (V - W) / slope.detach()
        new = V - (V - W) / slope
        if not bool(torch.isfinite(new).all()) or not bool((new > 0).all()):
            raise _Unusual
        off = float(((new - V).abs() / new).max())
        V = new
        if off <= 1e-13 or (it >= 8 and off <= 1e-11):
            return V
    raise _Unusual


def _solve_high(x):
    """Root of the high-velocity step by the secant rule with DV = V_old / 100."""
    cO, sO = torch.cos(x["Om"] * x["dt"]), torch.sin(x["Om"] * x["dt"])

    def theta(V):
        c = V / x["Dc"]
        return (x["th"] - 1 / c) * torch.exp(-c * x["dt"]) + 1 / c

    def off(V):
        fr = x["F0"] + x["a"] * torch.log(V / 1e-9) + x["b"] * torch.log(theta(V) * 1e-9 / x["Dc"])
        F = x["tld"] + (x["tau0"] + x["dtau"] - fr * x["sig"] - x["eta"] * V) / x["K"]
        X = (x["D"] - F) * cO + x["V"] / x["Om"] * sO + F
        return V - ((X - x["D"]) / x["dt"] * 2 - x["V"])

    V, h = x["V"] / 1e10, x["V"] / 100
    live = torch.ones_like(V, dtype=torch.bool)
    for it in range(99):
        f = off(V)
        new = torch.where(live, V - f * h / (off(V + h) - f), V)
        if not bool(torch.isfinite(new).all()) or not bool((new > 0).all()):
            raise _Unusual
        live = live & ((new / V - 1).abs() > (1e-13 if it < 40 else 1e-11))
        V = new
        if not bool(live.any()):
            return V, theta(V)
    raise _Unusual


def _number(v):
    return float(v.detach()) if torch.is_tensor(v) else float(v)


def _cycle64(p, E, Kn, kself, steps, dt0, ext=None, want=None, grad=False):
    """One instance's steps in 64 bits: the state's final fields, or (want) the
    recorded history, or (grad) the final slip as a function of a, b and Dc."""
    t = {k: (v if torch.is_tensor(v) else _cuda(v)) for k, v in p.items() if np.ndim(v) or torch.is_tensor(v)}
    n, ns = p["N"], p["N"] - p["Nload"]
    a, b, Dc = t["a"], t["b"], t["Dc"]
    F0 = t["f_i"] - a * torch.log(t["V_i"] / 1e-9) - b * torch.log(t["theta_i"] * 1e-9 / Dc)
    tau0, eta = t["sigma0"] * t["f_i"], math.sqrt(p["G"] * p["rho"]) / 2
    V, D, th, A = t["V_i"], torch.zeros_like(kself), t["theta_i"], torch.zeros_like(kself)
    fr, sig_old, T, dt = t["f_i"], t["sigma0"], 0.0, dt0
    ctl = (a - b < 0).detach()
    ctl = ctl if bool(ctl.any()) else torch.arange(n, device="cuda") < ns
    slip, hist = torch.arange(n, device="cuda") < ns, []
    for step in range(1, steps + 1):
        q = (V / A).abs()[ctl]
        q = q[(q > 0)]
        if float(V.detach()[ctl].max()) > p["switch_v"]:
            ref = p["rupture_dt"]
        else:
            ref = torch.clamp(q.min() / p["dt_cut"], max=p["max_dt"])
        if _number(ref) > p["rupture_dt"] and _number(dt) < _number(ref) / 1.2:
            dt = dt * 1.2
        else:
            dt = ref
        sig = t["sigma0"] + Kn @ D
        if bool((sig < p["sigma_min"]).any()):
            raise _Unusual
        dtau = 0.0 if ext is None else _cuda(ext["shear"][1]) * (T + dt) / float(ext["t"][1])
        x = dict(K=kself, tld=-(E @ D), D=D, V=V, th=th, dt=dt, tau0=tau0, eta=eta, dtau=dtau + torch.zeros_like(D),
                 sig=sig, M=t["mass"], a=a, b=b, Dc=Dc, F0=F0, Om=torch.sqrt(kself / t["mass"]))
        high = (V > p["switch_v"]) & slip
        low = ~high & slip
        new, thn = t["V_const"].clone(), th.clone()
        pick = lambda m: {k: (v[m] if torch.is_tensor(v) and v.ndim else v) for k, v in x.items()}  # noqa: E731
        if bool(low.any()):
            y = pick(low)
            root = _solve_low({k: (v.detach() if torch.is_tensor(v) else v) for k, v in y.items()}, y["V"].detach())
            vl = _solve_low(y, root, grad=True) if grad else root
            new = torch.where(low, torch.zeros_like(new).masked_scatter(low, vl), new)
            thn = torch.where(low, torch.zeros_like(new).masked_scatter(low, (y["th"] + dt) / (1 + dt * vl / y["Dc"])),
                              thn)
        if bool(high.any()):
            y = pick(high)
            vh, tn = _solve_high(y)
            new, thn = new.masked_scatter(high, vh), thn.masked_scatter(high, tn)
            fh = y["F0"] + y["a"] * torch.log(vh / 1e-9) + y["b"] * torch.log(tn * 1e-9 / y["Dc"])
        Dn = D + torch.where(slip, (V + new) / 2 * dt, new * dt)
        An = (new - V) / dt
        mu = (kself * (x["tld"] - Dn) + tau0 - eta * new + x["dtau"] - t["mass"] * An) / sig
        fr = torch.where(low, mu, fr)
        if bool(high.any()):
            fr = fr.masked_scatter(high, fh)
        sig_old = torch.where(slip, sig, torch.full_like(sig, 1e10))
        V, D, th, A = new, Dn, thn, An
        if want and step % want == 0:
            hist.append((T, _number(dt), V, D, th, sig_old))
        T = T + dt
    if grad:
        return D
    if want:
        return dict(zip(("T", "Dt", "V", "D", "theta", "sigma"),
                        [torch.tensor([h[k] for h in hist], dtype=torch.float64) if k < 2 else
                         torch.stack([h[k] for h in hist]) for k in range(6)]))
    return dict(V=V, D=D, theta=th, friction=fr, accel=A, sigma_old=sig_old, T=_number(T), dt=_number(dt))


def _instance(p, r):
    """Instance r of a problem of several friction draws."""
    n = p["N"]
    return {k: (v[r * n:(r + 1) * n] if isinstance(v, np.ndarray) else v) for k, v in p.items()}


def _normalised(Ks):
    d = torch.diagonal(Ks).clone()
    E = Ks / d[:, None]
    E.fill_diagonal_(0.0)
    return E, d.abs()


def _states64(p, draws, Ks, Kn, steps, dt0):
    E, kself = _normalised(Ks)
    each = [_cycle64(_instance(p, r), E, Kn, kself, steps, dt0) for r in range(draws)]
    out = {k: torch.cat([e[k] for e in each]) for k in FIELDS}
    for k in ("T", "dt"):
        out[k] = torch.tensor([e[k] for e in each], dtype=torch.float64)
    return dict(out, step=None)


def exact(case, seed):
    try:
        return _exact(case, seed)
    except _Unusual:
        return None


def _exact(case, seed):
    kind = case["kind"]
    if kind == "rect":
        K = _rect64(*_rect_inputs(case, seed))
        return [k.T.contiguous() if case["layout"] == "col" else k for k in K]
    if kind == "tri":
        n = case["triangles"]
        i = torch.arange(n, device="cuda")
        r, s = i.repeat_interleave(n), i.repeat(n)
        if case["layout"] == "col":
            r, s = s, r
        return [k.view(n, n) for k in _tri64(_tri_inputs(_mesh_of(n)["seg"][:n], seed), r, s)]
    if kind == "pairs":
        tri, r, s = _pair_inputs(case, seed)
        return list(_tri64(tri, torch.tensor(r, device="cuda"), torch.tensor(s, device="cuda")))
    if kind == "main":
        rec, p, _, _, ext = _main_args(case, seed)
        Ks, Kn = _rect64(rec, rec)
        E, kself = _normalised(Ks)
        return _cycle64(p, E, Kn, kself, case["steps"], 1.0, ext, want=case["record"])
    if kind == "hmat":
        _, p, tri, _ = _mesh_system(case, seed)
        n = p["N"]
        i = torch.arange(n, device="cuda")
        Ks, Kn = (k.view(n, n) for k in _tri64(tri, i.repeat_interleave(n), i.repeat(n)))
        return _states64(p, case["draws"], Ks, Kn, case["steps"], 10.0)
    if kind == "run":
        rec = _patches(case)
        Ks, Kn = _rect64(rec, rec)
        p = _problem(case, seed, len(rec), case["draws"], _sigma0(rec), _mass(rec),
                     torch.diagonal(Ks).cpu().numpy(), case["phase"], case["loading"])
        return _states64(p, case["draws"], Ks, Kn, case["steps"], 10.0 if case["phase"] == "creep" else 1.0)
    if kind == "adjoint":
        rec, n = _patches(case), case["patches"]
        Ks, Kn = _rect64(rec, rec)
        E, kself = _normalised(Ks)
        p = _problem(case, seed, n, case["draws"], _sigma0(rec), _mass(rec), torch.diagonal(Ks).cpu().numpy())
        w = np.random.default_rng([seed, 6]).standard_normal((case["draws"], n))
        out = {"a": [], "b": [], "Dc": []}
        for r in range(case["draws"]):
            q = _instance(p, r)
            q.update({k: _cuda(q[k]).requires_grad_() for k in out})
            D = _cycle64(q, E, Kn, kself, case["steps"], 10.0, grad=True)
            (D * _cuda(w[r])).sum().backward()
            for k in out:
                out[k].append(q[k].grad)
        return {k: torch.stack(v) for k, v in out.items()}
    each = []
    for k, n in enumerate(_member_sizes(case)):
        rec, c, s = _member(case, seed, k, n)
        Ks, Kn = _rect64(rec, rec)
        p = _problem(c, s, n, c["draws"], _sigma0(rec), _mass(rec), torch.diagonal(Ks).cpu().numpy())
        each.append(_states64(p, c["draws"], Ks, Kn, case["steps"], 10.0))
    return {k: (None if k == "step" else torch.cat([e[k] for e in each])) for k in (*FIELDS, "T", "dt", "step")}
