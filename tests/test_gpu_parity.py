"""CUDA library against the CPU oracle on the same seeded inputs.

FP64 tolerance: positions, velocities and forces within 1e-12 normwise
relative error (max|gpu - oracle| / max|oracle| per field); cell indices,
llist entries, bond states, image counters and ligand occupancy exact."""
import numpy as np
import pytest

import oracle as O
import helpers as H

pytestmark = pytest.mark.gpu
RTOL = 1e-12


@pytest.fixture(scope="module")
def base():
    """Oracle after set-up and 25 steps with raised bond rates (so bonds
    exist and two collisions have happened)."""
    op, orc = H.make_oracle(ns=40000, seed=11, onrate=300.0, offrate=50.0)
    orc.step(25)
    return op, orc.get_mesh(), orc.get_state()


def fresh_oracle(op, mesh, st, seed=11):
    o = O.Oracle(op, seed)
    o.set_mesh(mesh)
    o.set_state(st)
    return o


def test_init_matches_oracle():
    op, orc = H.make_oracle(ns=40000, seed=5)
    import irbc_b200 as G
    sim = G.Simulation(H.to_irbc_params(op, 5))
    V, E, T = H.troph()
    sim.init(V, E, T, 500)
    np.testing.assert_array_equal(sim.report(), orc.report())
    a, s = sim.get_mesh_arrays()
    M = orc.get_mesh()
    for k in ("e1", "e2", "es1", "es2", "iedge", "t1", "t2", "t3", "l0", "kappap", "tarea"):
        np.testing.assert_array_equal(a[k], M.a[k], err_msg=k)
    assert s["Sarea0"] == M.s["Sarea0"] and s["Volume0"] == M.s["Volume0"] and s["theta0"] == M.s["theta0"]
    bad = H.compare(sim.get_state(), orc.get_state(), RTOL)
    assert bad == {}


@pytest.mark.parametrize("phase", ["collide", "llist_update", "stream", "total_va", "pfdt", "forces"])
def test_phase_matches_oracle(base, phase):
    op, mesh, st = base
    o = fresh_oracle(op, mesh, st)
    sim = H.gpu_like(op, o, 11, state=st)
    if phase == "collide":
        sim.call("collide", 30)
        o.collide(30)
    else:
        sim.call(phase)
        getattr(o, phase)()
    g, r = sim.get_state(), o.get_state()
    bad = H.compare(g, r, RTOL)
    assert bad == {}, (phase, bad)


def test_stream_crowded_cell_and_long_list(base):
    """Near-membrane streaming off its usual path: 80 particles crowded into
    one listed cell, and a second cell whose list is padded to 1500 entries
    with repeats (longer than the short lists' class); both must follow the reference's sequential triangle walk."""
    op, mesh, st = base
    st2 = st.copy()
    off, lidx = st2.llists()
    llen = st2.a["llen"]
    nz = int(op.Lz / op.a) + 1
    ny = int(op.Ly / op.a)
    listed = np.nonzero(llen > 0)[0]
    assert listed.size >= 2
    c1, c2 = int(listed[listed.size // 3]), int(listed[2 * listed.size // 3])
    rng = np.random.default_rng(3)

    def crowd(c, idx):
        i, j, k = c // (ny * nz), (c // nz) % ny, c % nz
        n = idx.size
        st2.a["sx"][idx] = (i + rng.uniform(0.05, 0.95, n)) * op.a
        st2.a["sy"][idx] = (j + rng.uniform(0.05, 0.95, n)) * op.a
        st2.a["sz"][idx] = (k - 1 + rng.uniform(0.05, 0.95, n)) * op.a

    crowd(c1, np.arange(0, 80))
    crowd(c2, np.arange(80, 100))
    # pad c2's list with repeats of its own entries to 1500
    lists = [lidx[off[c]:off[c + 1]] for c in range(st2.ncell)]
    own = lists[c2]
    lists[c2] = np.resize(own, 1500)
    st2.a["llen"] = np.array([x.size for x in lists], np.int32)
    st2.a["lidx"] = np.concatenate(lists).astype(np.int32)
    o = fresh_oracle(op, mesh, st2)
    sim = H.gpu_like(op, o, 11, state=st2)
    sim.call("stream")
    o.stream()
    bad = H.compare(sim.get_state(), o.get_state(), RTOL)
    assert bad == {}, bad


def test_collide_counts_every_particle_once(base):
    op, mesh, st = base
    o = fresh_oracle(op, mesh, st)
    sim = H.gpu_like(op, o, 11, state=st)
    sim.call("collide", 40)
    g = sim.get_state()
    counts = np.bincount(g.a["spid"], minlength=sim.ncell)
    assert counts.sum() == st.ns
    # momentum of the solvent+membrane changes only by the ghost terms:
    # check the energy stays finite and the ids survive the counting sort
    assert np.isfinite(g.a["svx"]).all()


def test_steps_match_oracle_step_by_step(base):
    """30 steps (three collisions, bonds at raised rates), each started from
    the oracle's state: part 1 and part 2 within 1e-12."""
    op, mesh, st = base
    o = fresh_oracle(op, mesh, st)
    sim = H.gpu_like(op, o, 11, state=st)
    import irbc_b200 as G
    for k in range(30):
        sim.set_state(G.State.from_other(o.get_state()))
        sim.call("step_part1")
        o.step_part1()
        assert H.compare(sim.get_state(), o.get_state(), RTOL) == {}, ("part1", k)
        sim.call("step_part2")
        o.step_part2()
        assert H.compare(sim.get_state(), o.get_state(), RTOL) == {}, ("part2", k)


def test_trajectory_stays_close_to_oracle(base):
    """A continuous 30-step GPU trajectory.  Single steps agree to 1e-12;
    over many coupled steps the ulp differences of libm (cos/sin of the
    collision axes, acos/pow of contact times) grow through the stiff
    membrane springs, so forces are held to 1e-9 here, positions and
    solvent fields to 1e-11, integer state exactly."""
    op, mesh, st = base
    o = fresh_oracle(op, mesh, st)
    sim = H.gpu_like(op, o, 11, state=st)
    sim.step(30)
    o.step(30)
    g, r = sim.get_state(), o.get_state()
    assert H.compare(g, r, 1e-11, skip=("fx", "fy", "fz", "vx", "vy", "vz")) == {}
    assert H.compare(g, r, 1e-9, fields=("fx", "fy", "fz", "vx", "vy", "vz")) == {}


def test_llist_update_step_and_stale_tail():
    """Run through the llist update at step 82 (uplist = 83)."""
    op, orc = H.make_oracle(ns=20000, seed=21)
    orc.step(80)
    st = orc.get_state()
    sim = H.gpu_like(op, orc, 21, state=st)
    for k in range(6):
        sim.call("step_part1"); orc.step_part1()
        sim.call("step_part2"); orc.step_part2()
    assert H.compare(sim.get_state(), orc.get_state(), RTOL) == {}


def test_full_size_config1_init_and_steps():
    """define.h sizes (Ns = 960000): set-up and 12 steps incl. a collision."""
    op, orc = H.make_oracle(ns=960000, seed=3)
    import irbc_b200 as G
    sim = G.Simulation(H.to_irbc_params(op, 3))
    V, E, T = H.troph()
    sim.init(V, E, T, 500)
    assert H.compare(sim.get_state(), orc.get_state(), RTOL) == {}
    sim.step(12)
    orc.step(12)
    assert H.compare(sim.get_state(), orc.get_state(), RTOL) == {}


def _np_cells(op, x, y, z, r):
    """cindex cell of each particle in the shifted grid (Src/solfuncs.cpp:141-144)."""
    def bb(v, L):
        v = v.copy()
        while (v > L).any():
            v[v > L] -= L
        while (v < 0).any():
            v[v < 0] += L
        return v
    nx, ny, nz = int(op.Lx), int(op.Ly), int(op.Lz) + 1
    fx = np.floor(bb(x - r[0], op.Lx)).astype(np.int64)
    fy = np.floor(bb(y - r[1], op.Ly)).astype(np.int64)
    fz = np.floor(z - r[2] + 1.0).astype(np.int64)
    ok = (fx >= 0) & (fx < nx) & (fy >= 0) & (fy < ny) & (fz >= 0) & (fz < nz)
    return np.where(ok, (fx * ny + fy) * nz + fz, 0)


def test_bin_particles_standalone():
    """irbc_bin_particles on device arrays: cells, counting-sort starts and
    the per-cell particle order (ascending index) exactly."""
    import ctypes as C
    import torch
    import irbc_b200 as G
    op = O.default_params(Ns=200000)
    rng = np.random.default_rng(4)
    n = 200000
    pos = np.stack([rng.uniform(0, op.Lx, n), rng.uniform(0, op.Ly, n), rng.uniform(0, op.Lz, n)])
    pos[0, :5] = [0.0, op.Lx, 59.99999999, 1e-300, 30.0]   # edges: x == Lx maps to cell 0
    r = (0.25, 0.5, 0.999)
    dev = [torch.tensor(pos[k], dtype=torch.float64, device="cuda") for k in range(3)]
    p = H.to_irbc_params(op, 1)
    ncell = int(op.Lx) * int(op.Ly) * (int(op.Lz) + 1)
    cell = torch.zeros(n, dtype=torch.int32, device="cuda")
    start = torch.zeros(ncell + 1, dtype=torch.int32, device="cuda")
    order = torch.zeros(n, dtype=torch.int32, device="cuda")
    L = G.lib()
    rc = L.irbc_bin_particles(C.byref(p), dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), n,
                              r[0], r[1], r[2], cell.data_ptr(), start.data_ptr(), order.data_ptr())
    assert rc == 0
    want = _np_cells(op, pos[0], pos[1], pos[2], r)
    np.testing.assert_array_equal(cell.cpu().numpy(), want)
    counts = np.bincount(want, minlength=ncell)
    np.testing.assert_array_equal(start.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
    np.testing.assert_array_equal(order.cpu().numpy(), np.argsort(want, kind="stable"))


def test_pipelined_steps_equal_split_steps():
    """irbc_step runs the membrane chain on a second stream and fuses the
    next half-kick into it; 95 steps (nine collisions, the llist update at
    step 82) must equal part 1 + part 2 run one after the other, bit for bit."""
    op, orc = H.make_oracle(ns=30000, seed=31, onrate=300.0, offrate=50.0)
    st = orc.get_state()
    a = H.gpu_like(op, orc, 31, state=st)
    b = H.gpu_like(op, orc, 31, state=st)
    for n in (7, 3, 40, 45):
        a.step(n)
        for _ in range(n):
            b.call("step_part1")
            b.call("step_part2")
        ga, gb = a.get_state(), b.get_state()
        assert H.compare(ga, gb, 0.0) == {}, n


@pytest.mark.parametrize("precision", [0, 1])
def test_captured_graphs_equal_plain_launches(precision):
    """irbc_step launches 24-step stretches as captured CUDA graphs; 250
    steps (list update at step 83, physical re-sorts between graphs) with
    graphs must equal the same steps launched one kernel at a time, bit for
    bit, in both precisions."""
    op, orc = H.make_oracle(ns=30000, seed=37, onrate=300.0, offrate=50.0)
    st = orc.get_state()
    a = H.gpu_like(op, orc, 37, precision=precision, state=st)
    b = H.gpu_like(op, orc, 37, precision=precision, state=st)
    a.set_graphs(True)
    b.set_graphs(False)
    for n in (5, 60, 185):
        a.step(n)
        b.step(n)
        assert H.compare(a.get_state(), b.get_state(), 0.0) == {}, n


def test_pipelined_single_steps_match_oracle():
    """irbc_step(1) from the oracle's state, 24 times (two collisions)."""
    import irbc_b200 as G
    op, orc = H.make_oracle(ns=30000, seed=32, onrate=300.0, offrate=50.0)
    orc.step(5)
    sim = H.gpu_like(op, orc, 32, state=orc.get_state())
    for k in range(24):
        sim.set_state(G.State.from_other(orc.get_state()))
        sim.step(1)
        orc.step(1)
        assert H.compare(sim.get_state(), orc.get_state(), RTOL) == {}, k
