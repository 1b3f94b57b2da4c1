"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the public entry points of irbc_b200 (the C ABI of
include/irbc.h).  A pass advances simulations that the program keeps and
takes what such a program takes from them: the whole state into page-locked
arrays, the vertex records, the observables, or a served request's results.
Passes go on from where the pass before ended, as a program's calls do.
"""
import ctypes as C
import math
import os

# many replicas' streams need more than the default 8 hardware queues; read
# by CUDA when the process first uses it (include/irbc.h, batches)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "irbc-code_b200"))
import irbc_b200 as G  # noqa: E402
from irbc_b200 import mesh, workloads  # noqa: E402

TROPH = [os.path.join(ROOT, "tests", "golden", "troph600", "Troph%s600.dat" % c) for c in "VET"]
# largest pass: the benchmark's 780 steps of 5,242,880 particles
MOST = 780 * workloads.LARGE["Ns"]
_meshes = {}


def _mesh(name):
    """(V, E, T): the shipped 600-vertex trophozoite or the 2562-vertex
    discocyte of radius 4"""
    if name not in _meshes:
        _meshes[name] = mesh.discocyte() if name == "discocyte" else mesh.read_reference_files(*TROPH)
    return _meshes[name]


def _box(Lx, Ly, Lz, ns):
    return {"Lx": Lx, "Ly": Ly, "Lz": Lz, "ns": ns}


def listed():
    return [
        # the benchmark: one large simulation, a checkpointed stretch of 780
        # steps (65 collisions, 2 list updates)
        {"name": "large_fp64", "kind": "run", "setting": "sweep", "precision": "fp64", "mesh": "discocyte",
         "knobs": 1000, "steps": 780, **_box(128, 64, 64, 5242880)},
        # the same with the FP32-bulk solvent
        {"name": "large_fp32", "kind": "run", "setting": "sweep", "precision": "fp32", "mesh": "discocyte",
         "knobs": 1000, "steps": 780, **_box(128, 64, 64, 5242880)},
        # the reference's own configuration as shipped (define.h)
        {"name": "reference_fp64", "kind": "run", "setting": "define", "precision": "fp64", "mesh": "trophozoite",
         "knobs": 500, "steps": 500, **_box(60, 40, 40, 960000)},
        # one replica of a sweep, alone
        {"name": "replica_fp32", "kind": "run", "setting": "sweep", "precision": "fp32", "mesh": "trophozoite",
         "knobs": 350, "steps": 480, **_box(64, 32, 32, 675840)},
        # the small box of the long stability runs: launches and latency count
        {"name": "small_fp64", "kind": "run", "setting": "sweep", "precision": "fp64", "mesh": "discocyte",
         "knobs": 1000, "steps": 240, **_box(32, 32, 32, 40000)},
        # a program that takes the vertex record after every step
        {"name": "record_fp64", "kind": "record", "setting": "define", "precision": "fp64", "mesh": "trophozoite",
         "knobs": 500, "steps": 120, **_box(60, 40, 40, 960000)},
        # a parameter sweep: replicas of uneven boxes stepped together
        {"name": "batch_fp32", "kind": "batch", "setting": "sweep", "precision": "fp32", "mesh": "trophozoite",
         "knobs": 350, "steps": 240, "members": 16, **_box(96, 32, 32, 0)},
        # a production run sampled as the precision study samples it
        {"name": "study_fp32", "kind": "study", "setting": "define", "precision": "fp32", "mesh": "trophozoite",
         "knobs": 500, "steps": 160, "samples": 3, **_box(60, 40, 40, 960000)},
        # whole simulations sent to the request server: set-up, steps, observables
        {"name": "served", "kind": "served", "setting": "sweep", "precision": "fp32", "mesh": "both",
         "knobs": 1000, "steps": 960, "members": 6, **_box(96, 36, 36, 0)},
        # the solvent's velocities brought to equilibrium before a run:
        # collisions alone, in each precision
        {"name": "thermalise_fp64", "kind": "thermalise", "setting": "define", "precision": "fp64",
         "mesh": "trophozoite", "knobs": 500, "steps": 40, **_box(60, 40, 40, 960000)},
        {"name": "thermalise_fp32", "kind": "thermalise", "setting": "sweep", "precision": "fp32",
         "mesh": "discocyte", "knobs": 1000, "steps": 24, **_box(128, 64, 64, 5242880)},
        # the standalone binning of particles that another program holds on
        # the device
        {"name": "bin", "kind": "bin", "setting": "define", "precision": "fp64", "mesh": "none", "knobs": 0,
         "steps": 1, **_box(128, 64, 64, 5242880)},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "record", "batch", "study", "served", "thermalise", "bin"])
    c = {"kind": kind, "setting": rng.choice(["define", "sweep"]), "precision": rng.choice(["fp64", "fp32"]),
         "mesh": rng.choice(["trophozoite", "discocyte"])}
    # boxes of whole cells, odd ones among them, 24 to 128 long
    Lx, Ly, Lz = _log_int(rng, 32, 128), _log_int(rng, 24, 64), _log_int(rng, 24, 64)
    # densities from the sparse test boxes to the configured 10 a cell
    ns = int(Lx * Ly * Lz * rng.choice([1.2, 10.0, 10.0])) + rng.randrange(0, 1000)
    c["knobs"] = rng.randrange(100, 600)
    if kind in ("batch", "served"):
        c.update(setting="sweep", precision="fp32", members=rng.randrange(2, 13) if kind == "batch" else
                 rng.randrange(2, 6), steps=rng.randrange(96, 241) if kind == "batch" else rng.randrange(240, 961))
        c["mesh"] = "trophozoite" if kind == "batch" else "both"
        Ly = Lz = rng.randrange(24, 37)
        ns, Lx = 0, rng.randrange(48, 97)
    elif kind == "study":
        c.update(steps=rng.randrange(60, 200), samples=rng.randrange(1, 4))
    elif kind == "record":
        c["steps"] = rng.randrange(40, 200)
    elif kind == "thermalise":
        c["steps"] = rng.randrange(12, 40)
    elif kind == "bin":
        c.update(steps=1, mesh="none", knobs=0, precision="fp64")
    else:
        c["steps"] = min(_log_int(rng, 60, 780), MOST // max(1, ns))
    c.update(_box(Lx, Ly, Lz, ns))
    return c


# ---- preparing ------------------------------------------------------------------
def _params(c, seed, kon=None, koff=None, box=None, mesh_name=None, walls_frac=0.01):
    """irbc_params of a simulation: define.h's own constants, or those of the
    sweeps and the large simulation (130 deg, dtcd 0.025)"""
    Lx, Ly, Lz, ns = box or (c["Lx"], c["Ly"], c["Lz"], c["ns"])
    prec = G.FP64 if c["precision"] == "fp64" else G.FP32
    V, E, _ = _mesh(mesh_name or c["mesh"])
    disc = len(V) != 600
    if c["setting"] == "define":
        over = dict(elap=mesh.scaled_elap(V, E)) if disc else {}
        return G.default_params(Lx=float(Lx), Ly=float(Ly), Lz=float(Lz), Ns=ns, Nt=len(V), seed=seed,
                                precision=prec, **over)
    p = workloads.replica_params(Lx, Ly, Lz, seed, kon or 0.005, koff or 0.015, precision=prec,
                                 walls_frac=walls_frac, mesh_ve=(V, E) if disc else None)
    if ns:
        p.Ns = ns
    return p


def _simulation(c, seed):
    sim = G.Simulation(_params(c, 1 + seed))
    V, E, T = _mesh(c["mesh"])
    sim.init(V, E, T, min(c["knobs"], len(V)))
    return sim


FIELDS = G.State.SOLVENT_D + G.State.SOLVENT_I + G.State.VERT_D + G.State.VERT_I


def _host_states(sims):
    """page-locked arrays for the sims' states, one per field, and a
    G.State over each sim's slice of them"""
    pinned, states = {}, [G.State(0, s.nv, s.nlig, 0, llist=False) for s in sims]
    for k in FIELDS:
        solvent = k in G.State.SOLVENT_D + G.State.SOLVENT_I
        n = [s.params.Ns if solvent else s.nv for s in sims]
        dt = torch.int32 if states[0].a[k].dtype == np.int32 else torch.float64
        pinned[k] = torch.empty(sum(n), dtype=dt, pin_memory=True).numpy()
        at = 0
        for st, m in zip(states, n):
            st.a[k] = pinned[k][at:at + m]
            at += m
    for s, st in zip(sims, states):
        st.ns, st.ncell = s.params.Ns, s.ncell
    return pinned, states


def _replica_boxes(c):
    """uneven boxes (Lx from 32 to the case's, 10 particles a cell), bond
    rates and knob counts: a sweep's table; the seed draws each replica's
    particles"""
    rng = np.random.default_rng([7, c["members"], c["Lx"], c["Ly"]])
    return [(int(rng.integers(32, c["Lx"] + 1)), c["Ly"], c["Lz"], 0, 10 ** rng.uniform(-4, -1),
             10 ** rng.uniform(-3, -1), int(rng.integers(100, 601))) for _ in range(c["members"])]


def _thermal(c, seed):
    """a checkpoint to restart from: solvent uniform in the box with
    Maxwellian velocities on the Couette profile, vertices where set-up
    places them, numbers that the case's precision holds exactly"""
    rng = np.random.default_rng([11, seed])
    n, dt = c["ns"], np.float32 if c["precision"] == "fp32" else np.float64
    a = {k: (rng.random(n) * (L * (1 - 1e-6))).astype(dt).astype(np.float64)
         for k, L in (("sx", c["Lx"]), ("sy", c["Ly"]), ("sz", c["Lz"]))}
    for k in ("svx", "svy", "svz"):
        a[k] = rng.standard_normal(n).astype(dt).astype(np.float64)
    a["svx"] = (a["svx"] + 0.5 * a["sz"] / c["Lz"]).astype(dt).astype(np.float64)
    V = _mesh(c["mesh"])[0]
    centre = np.array([c["Lx"] / 2.0 + 10.0, c["Ly"] / 2.0, -V[:, 2].min() + 0.3])
    P = V + centre
    P[:, 0] %= c["Lx"]
    a["x"], a["y"], a["z"] = (np.ascontiguousarray(P[:, k]) for k in range(3))
    for k in ("vx", "vy", "vz"):
        a[k] = math.sqrt(0.1) * rng.standard_normal(len(V))
    para = np.array([centre[0] % c["Lx"], centre[1], centre[2]])
    return a, para, math.sqrt(0.1) * rng.standard_normal(3)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "bin":
        # particle positions that another program holds in device memory
        g = torch.Generator(device="cuda").manual_seed(seed)
        pos = torch.rand((3, c["ns"]), generator=g, device="cuda", dtype=torch.float64)
        pos *= torch.tensor([[c["Lx"]], [c["Ly"]], [c["Lz"]]], device="cuda", dtype=torch.float64)
        ncell = c["Lx"] * c["Ly"] * (c["Lz"] + 1)
        shift = np.random.default_rng([5, seed]).random(3)
        out = [torch.empty(m, dtype=torch.int32, device="cuda") for m in (c["ns"], ncell + 1, c["ns"])]
        p = G.default_params(Lx=float(c["Lx"]), Ly=float(c["Ly"]), Lz=float(c["Lz"]), Ns=0)
        torch.cuda.synchronize()
        return {"case": c, "p": p, "pos": pos, "shift": [float(r) for r in shift], "out": out}
    if kind == "served":
        # the server and the requests of one submission; alternating meshes
        reqs = []
        for k, (Lx, Ly, Lz, _, kon, koff, nk) in enumerate(_replica_boxes(c)):
            name = ("trophozoite", "discocyte")[k & 1]
            p = _params(c, 1 + 64 * seed + k, kon, koff, (Lx, Ly, Lz, 0), name)
            reqs.append((p, *_mesh(name), nk, c["steps"] - 48 * k))
        return {"case": c, "server": G.Server(nthreads=8, round_steps=96), "reqs": reqs}
    if kind == "batch":
        sims, b = [], G.Batch(nthreads=8)
        V, E, T = _mesh(c["mesh"])
        for k, (Lx, Ly, Lz, _, kon, koff, nk) in enumerate(_replica_boxes(c)):
            s = G.Simulation(_params(c, 1 + 64 * seed + k, kon, koff, (Lx, Ly, Lz, 0)))
            s.init(V, E, T, nk)
            sims.append(s)
            b.add(s)
        pinned, states = _host_states(sims)
        return {"case": c, "batch": b, "sims": sims, "pinned": pinned, "states": states}
    sim = _simulation(c, seed)
    s = {"case": c, "sims": [sim]}
    if kind != "study":
        s["pinned"], s["states"] = _host_states([sim])
    if kind == "record":
        s["rec"] = [G.PinnedArray(sim.record_bytes(), np.uint8) for _ in range(2)]
    if kind == "thermalise":
        a, para, paraV = _thermal(c, seed)
        st = sim.get_state()
        for k, v in a.items():
            st.a[k] = v
        st.s.update(para=para, paraV=paraV, wallspeed=0.5)
        sim.set_state(st)
        s["epoch"] = 0
    return s


# ---- one pass ----------------------------------------------------------------------
def _fetch(s):
    """every sim's state into the page-locked arrays"""
    scal = []
    for sim, st in zip(s["sims"], s["states"]):
        v = st.view()
        sim.call("get_state", C.byref(v))
        st.absorb(v)
        scal.append(np.concatenate([st.s["para"], st.s["paraV"], [st.s["Sarea"], st.s["Volume"]]]))
    out = {k: s["pinned"][k] for k in FIELDS}
    out["scalars"] = np.concatenate(scal)
    return out


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "bin":
        x, y, z = s["pos"]
        cell, start, order = s["out"]
        rc = G.lib().irbc_bin_particles(C.byref(s["p"]), x.data_ptr(), y.data_ptr(), z.data_ptr(), c["ns"],
                                        *s["shift"], cell.data_ptr(), start.data_ptr(), order.data_ptr())
        if rc != 0:
            raise G.IrbcError("irbc_bin_particles failed (%d)" % rc)
        return {"cell": cell, "start": start, "order": order}
    if kind == "served":
        ids = [s["server"].submit(p, V, E, T, nk, n) for p, V, E, T, nk, n in s["reqs"]]
        got = {}
        while len(got) < len(ids):
            for r in s["server"].poll(64, wait=60.0):
                got[r["id"]] = r
        return {"status": np.array([got[i]["status"] for i in ids]), "obs": np.stack([got[i]["obs"] for i in ids])}
    if kind == "batch":
        s["batch"].step(c["steps"])
        return _fetch(s)
    sim = s["sims"][0]
    if kind == "study":
        rows, prof, verts = [], [], []
        for _ in range(c["samples"]):
            sim.step(c["steps"])
            rows.append(sim.observables()[:9])
            prof.append(sim.velocity_profile(c["Lz"]))
            st = sim.get_state(solvent=False, llist=False)
            verts.append(np.stack([st.a[k] for k in ("x", "y", "z", "vx", "vy", "vz")]))
        return {"observables": np.stack(rows), "profile": np.stack(prof), "vertices": np.stack(verts)}
    if kind == "record":
        for k in range(c["steps"]):
            sim.step(1)
            sim.record_async(s["rec"][k & 1])
        out = _fetch(s)
        out["record"] = s["rec"][(c["steps"] - 1) & 1].array.copy()
        return out
    if kind == "thermalise":
        for k in range(c["steps"]):
            sim.call("collide", s["epoch"] + k)
        s["epoch"] += c["steps"]
        return _fetch(s)
    sim.step(c["steps"])
    return _fetch(s)


# ---- what a pass cannot do without ---------------------------------------------------
def work(case):
    """Between two collisions a particle away from the membrane meets
    nothing, so its position and velocity have to be read once and written
    once per collision (dtcd / dtmd steps), however many steps there are;
    the state that is handed over is 56 bytes a particle, 8 more read for a
    served or sampled one."""
    c = case
    if c["kind"] == "bin":
        ncell = c["Lx"] * c["Ly"] * (c["Lz"] + 1)
        return {"bytes": 24 * c["ns"] + 8 * c["ns"] + 4 * (ncell + 1), "flops": 12 * c["ns"]}
    w = 8 if c["precision"] == "fp64" else 4
    ns = c["ns"] or c["members"] * (32 + c["Lx"]) // 2 * c["Ly"] * (c["Lz"] + 1) * 10
    steps = c["steps"] * c.get("samples", 1)
    # a collision: 6 values in and out; a step: 3 products and sums; a
    # collision: sums, relative energies and the rotation, about 50
    coll = steps if c["kind"] == "thermalise" else max(1, steps // (10 if c["setting"] == "define" else 12))
    handed = 0 if c["kind"] in ("study", "served") else 6 * w + 56
    flops = ns * (50 * coll + (0 if c["kind"] == "thermalise" else 6 * steps))
    return {"bytes": ns * (12 * w * coll + handed), "flops": flops}


def tolerance(case):
    """Collisions alone do not amplify rounding: about four times the error
    against exact().  Whole steps do: about four times what the outputs
    moved by when the start's solvent velocities were nudged by one unit in
    the last place of the case's precision (worst output, at 24 to 780
    steps: FP64 1.3e-7 with the trophozoite, 1.2e-4 with the finer
    discocyte; FP32 5e-3 after 240 steps, and beyond about 400 nothing but
    the same bits agrees).  Sampled means move less."""
    c = case
    if c["kind"] == "bin":
        return "exact"
    if c["kind"] == "thermalise":
        return {"rel": 7e-15 if c["precision"] == "fp64" else 2e-6}
    if c["kind"] == "served":
        return {"rel": 1e-4}
    if c["precision"] == "fp32":
        return {"rel": 1e-2 if c["kind"] == "study" else 2e-2, "max": 0.8, "differ": 1e-2}
    return {"rel": 5e-7 if c["mesh"] == "trophozoite" else 5e-4}


# ---- the collision in 64 bits --------------------------------------------------------
def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors of 32-bit words"""
    M = 0xFFFFFFFF
    k0, k1 = seed & M, (seed >> 32) & M

    def mul(m, x):
        # 32 x 32 -> 64 bits, the factor in 16-bit halves so that nothing overflows
        lo, hi = (m & 0xFFFF) * x, (m >> 16) * x
        low = lo + ((hi & 0xFFFF) << 16)
        return ((hi >> 16) + (low >> 32)) & M, low & M
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c0)
        h1, l1 = mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return torch.stack([c0, c1, c2, c3])


def _block(seed, stream, epoch, blk):
    z = torch.zeros_like(blk)
    return _philox(blk & 0xFFFFFFFF, blk >> 32, z + epoch, z + stream, seed)


def _normal(seed, epoch, k):
    o = _block(seed, 3, epoch, k).double() / 4294967296.0
    return torch.sqrt(-2.0 * torch.log(o[0] + 1.0 / 4294967296.0)) * torch.cos(6.283185307179586 * o[1])


def exact(case, seed):
    """The thermalising collisions and the binning in plain 64-bit torch;
    the runs of whole steps are chaotic (two roundings of the same step
    part within a few collisions), and theirs would take minutes."""
    c, dev = case, "cuda"
    f64 = torch.float64
    if c["kind"] == "bin":
        s = prepare(c, seed)
        L, pos = (c["Lx"], c["Ly"]), s["pos"]
        r = s["shift"]
        f = [torch.floor(torch.where(q < 0, q + L[k], q)).long() for k, q in enumerate(pos[k] - r[k] for k in (0, 1))]
        fz = torch.floor(pos[2] - r[2] + 1.0).long()
        ok = (f[0] < c["Lx"]) & (f[1] < c["Ly"]) & (fz >= 0) & (fz <= c["Lz"])
        cell = torch.where(ok, (f[0] * c["Ly"] + f[1]) * (c["Lz"] + 1) + fz, 0)
        n = torch.bincount(cell, minlength=c["Lx"] * c["Ly"] * (c["Lz"] + 1))
        start = torch.cat([torch.zeros(1, dtype=torch.long, device=dev), torch.cumsum(n, 0)])
        return {"cell": cell.int(), "start": start.int(), "order": torch.sort(cell, stable=True)[1].int()}
    if c["kind"] != "thermalise":
        return None
    p = _params(c, 1 + seed)
    a, para, paraV = _thermal(c, seed)
    X = torch.tensor(np.stack([np.concatenate([a["s" + k], a[k], [q]]) for k, q in zip("xyz", para)]), device=dev)
    U = torch.tensor(np.stack([np.concatenate([a["sv" + k], a["v" + k], [q]]) for k, q in zip("xyz", paraV)]),
                     device=dev)
    n, nv = c["ns"], len(a["x"])
    m = torch.ones(n + nv + 1, dtype=f64, device=dev)
    m[n:n + nv], m[-1] = p.pmass, p.PRmass
    nx, ny, nz = c["Lx"], c["Ly"], c["Lz"] + 1
    C_ = nx * ny * nz
    cells = torch.arange(C_, device=dev)
    top, wall = (cells % nz) >= c["Lz"], ((cells % nz) >= c["Lz"]) | ((cells % nz) <= 1)
    zero = torch.zeros(1, dtype=torch.long, device=dev)
    pid = None
    for epoch in range(c["steps"]):
        r = _block(p.seed, 2, epoch, zero)[:3, 0].double() / 4294967296.0
        q = X - r[:, None]
        for k, L in ((0, c["Lx"]), (1, c["Ly"])):
            q[k] = torch.where(q[k] < 0, q[k] + L, q[k])
        q[2] += 1.0
        fx, fy, fz = torch.floor(q).long()
        ok = (fx < nx) & (fy < ny) & (fz >= 0) & (fz < nz)
        cell = torch.where(ok, (fx * ny + fy) * nz + fz, 0)
        pid = cell
        ns = torch.bincount(cell[:n], minlength=C_).double()
        nm = torch.bincount(cell[n:n + nv], minlength=C_).double()
        nc = torch.bincount(cell, minlength=C_).double()
        S = torch.stack([torch.zeros(C_, dtype=f64, device=dev).index_add_(0, cell, m * U[k]) for k in range(3)])
        ncc = ns * p.mass
        # wall ghosts, then the ghosts of the membrane's cells, in cell order
        wf, mf = wall & (ns < p.navg), (nm > 0) & (nc < p.navg)
        ncc = torch.where(wf, torch.full_like(ncc, p.navg * p.mass), ncc) + (ncc * 0).index_add_(0, cell[n:], m[n:])
        for flag, have, first in ((wf, ns, 0), (mf, nc, int(wf.sum()))):
            at = cells[flag]
            g = 3 * (first + torch.arange(len(at), device=dev))
            sd = torch.sqrt((p.navg - have[at]) * p.Theta / p.mass)
            for k in range(3):
                mean = torch.where(top[at], (p.navg - have[at]) * 0.5, 0.0) if k == 0 and first == 0 and flag is wf else 0.0
                S[k, at] += p.mass * (_normal(p.seed, epoch, g + k) * sd + mean)
        ncc = ncc + torch.where(mf, (p.navg - nc) * p.mass, 0.0)
        whole = torch.floor(ncc)
        vcm = torch.where(whole != 0, S / torch.where(whole != 0, whole, 1.0), S)
        D = U - vcm[:, cell]
        e = torch.zeros(C_, dtype=f64, device=dev).index_add_(0, cell, m * (D * D).sum(0))
        th = torch.where((nc > 0) & (e != 0), torch.sqrt(3.0 * (nc - 1.0).clamp(min=0) * p.Theta / e), 1.0)
        k1 = 3 + 2 * cells
        u = [torch.gather(_block(p.seed, 2, epoch, kk >> 2), 0, (kk & 3)[None])[0].double() / 4294967296.0
             for kk in (k1, k1 + 1)]
        w = -1.0 + 2.0 * u[1]
        ax = torch.stack([torch.sqrt(1 - w * w) * torch.cos(2 * p.Pi * u[0]),
                          torch.sqrt(1 - w * w) * torch.sin(2 * p.Pi * u[0]), w])[:, cell]
        par = (D * ax).sum(0) * ax
        nor = D - par
        U = vcm[:, cell] + th[cell] * (p.cosalpha * nor + p.sinalpha * torch.linalg.cross(nor, ax, dim=0) + par)
    out = {k: None for k in FIELDS}
    out["scalars"] = None
    for k in ("sx", "sy", "sz", "x", "y", "z"):
        out[k] = a[k]
    for i, k in enumerate("xyz"):
        out["sv" + k], out["v" + k] = U[i, :n].cpu().numpy(), U[i, n:n + nv].cpu().numpy()
    out["spid"], out["pid"] = pid[:n].int().cpu().numpy(), pid[n:n + nv].int().cpu().numpy()
    return out
