"""The launches that take several timesteps, or more of the box, at once, at
the sizes where their rules and edges lie.

A stretch of timesteps between two collisions equals the same timesteps one at
a time bit for bit: stretches above the 16 steps that one launch takes, those
in one part and in two, boxes so narrow that every particle lies in a side
wall's band or wraps into its own cell's neighbour, sparse ones, particles fast
enough to cross several cells in a stretch, every form of the membrane, both
precisions."""
import ctypes as C

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


STRETCHES = [  # dtcd, Lx, Ly, particles, speed factor, membrane form
    (0.02, 60.0, 30.0, 30000, 1.0, 1),     # 10 steps: parts of 6 and 4
    (0.014, 60.0, 30.0, 30000, 1.0, 1),    # 7 steps: one part
    (0.05, 60.0, 30.0, 30000, 1.0, 1),     # 25 steps: launches of 16 and 9
    (0.02, 13.0, 13.0, 20000, 1.0, 1),     # the bands of 3 cells meet the membrane
    (0.02, 13.5, 12.25, 12000, 1.0, 1),    # a box of no whole number of cells
    (0.02, 60.0, 30.0, 900, 1.0, 1),       # few particles
    (0.05, 40.0, 20.0, 30000, 25.0, 1),    # up to some cells a stretch
    (0.02, 40.0, 20.0, 20000, 1.0, 2),     # the membrane in one block
    (0.05, 40.0, 20.0, 20000, 1.0, 3),     # ... in a cluster on global memory
]


def _mesh_oracle(V, E, T, nknobs, **over):
    """an oracle with a mesh of its own (elap scaled to it)"""
    import oracle as O
    from irbc_b200 import mesh
    op = O.default_params(Nt=len(V), elap=mesh.scaled_elap(V, E), **over)
    orc = O.Oracle(op, 43)
    orc.init(V, E, T, nknobs)
    return op, orc


def _against_single_steps(op, orc, seed, st, precision, form, counts):
    """stretches of a simulation against one that takes the same steps singly"""
    a = H.gpu_like(op, orc, seed, precision=precision, state=st)
    b = H.gpu_like(op, orc, seed, precision=precision, state=st)
    a.set_membrane_kernels(form)
    b.set_membrane_kernels(form)
    for n in counts:
        a.step(n)
        for _ in range(n):
            b.call("step_part1")
            b.call("step_part2")
        assert H.compare(a.get_state(), b.get_state(), 0.0) == {}, n
    return a.get_state()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", STRETCHES, ids=lambda c: "%g-%gx%g-%d-%g-%d" % c)
def test_stretches_equal_single_steps(case, precision):
    dtcd, Lx, Ly, ns, fast, form = case
    op, orc = H.make_oracle(ns=ns, seed=41, onrate=300.0, offrate=50.0, dtcd=dtcd, Lx=Lx, Ly=Ly)
    st = orc.get_state()
    for k in ("svx", "svy", "svz"):
        st.a[k] = st.a[k] * fast
    # collisions inside and at the ends, the list update
    _against_single_steps(op, orc, 41, st, precision, form, (3, 30, 55))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dtcd", [0.025, 0.05])  # 12 steps in two parts, launches of 16 and 9
def test_stretches_of_the_discocyte(dtcd, precision):
    """The membrane in sixteen blocks, its long lists by 32 lanes."""
    from irbc_b200 import mesh
    V, E, T = mesh.discocyte()
    op, orc = _mesh_oracle(V, E, T, 1000, Ns=30000, onrate=300.0, offrate=50.0, dtcd=dtcd, Lx=40.0, Ly=24.0, Lz=24.0)
    st = _against_single_steps(op, orc, 43, orc.get_state(), precision, 1, (3, 30, 55))
    assert st.a["bondi"].sum() > 0


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("freq,R,room", [(8, 4.0, 64), (15, 2.5, 512)])  # kShortKeep, kLongKeep
def test_lists_that_keep_more_than_there_is_room_for(freq, R, room, precision):
    """Particles whose path in a stretch is longer than three cells reach every
    entry of their list (its centroids lie within two cells of the cell's
    centre), so a list longer than the room is walked whole in each step; single
    steps cull it."""
    V, E, T = H.geodesic(freq, R)
    op, orc = _mesh_oracle(V, E, T, 0, Ns=20000, dtcd=0.05, Lx=40.0, Ly=12.0, Lz=12.0, pmass=1e6)
    st = orc.get_state()
    longest = st.a["llen"].max()
    assert room < longest and (longest <= 128) == (room == 64)
    for k in ("svx", "svy", "svz"):
        st.a[k] = st.a[k] * 120.0
    v = np.sqrt(st.a["svx"] ** 2 + st.a["svy"] ** 2 + st.a["svz"] ** 2)
    cell = (np.floor(st.a["sx"]) * 12 + np.floor(st.a["sy"])) * 13 + np.floor(st.a["sz"]) + 1
    far = (v * 16 * op.dtmd > 3.6) & (st.a["llen"][cell.astype(int)] > room)
    assert far.sum() > 10
    _against_single_steps(op, orc, 43, st, precision, 1, (16, 20))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", ["events", "draws", "parasite"])
def test_more_than_the_tail_of_the_patches_holds(case, precision):
    """More bond events in a step than its list takes (128), more vertices with
    draws (1024) and more in the parasite's reach (768): the patches against the
    cluster on global memory and single steps, in FP64 also against the oracle.
    (Heavy vertices, so that forces of such reaches do not break the mesh.)"""
    from irbc_b200 import mesh
    V, E, T = mesh.discocyte()
    over = dict(events=dict(dthr=0.9, onrate=1e6, offrate=1e4), draws=dict(dthr=2.0, onrate=300.0, offrate=1e4),
                parasite=dict(paraR=6.0, PRmass=1e9))[case]
    op, orc = _mesh_oracle(V, E, T, len(V), Ns=20000, Lx=40.0, Ly=24.0, Lz=24.0, pmass=1e7, **over)
    st = orc.get_state()
    if case == "parasite":
        d2 = sum((st.a[k] - st.s["para"][i]) ** 2 for i, k in enumerate("xyz"))
        assert (d2 < op.paraR ** 2).sum() > 768
    else:
        # each vertex in its own cell, as a collision without a shift leaves it,
        # and its pairs in the first step: the ligands within dthr on that cell's
        # list (cells below z = 2, centres within 1.5)
        f = [np.floor(st.a["x"]), np.floor(st.a["y"]), np.floor(st.a["z"]) + 1]
        st.a["pid"] = ((f[0] * int(op.Ly) + f[1]) * (int(op.Lz) + 1) + f[2]).astype(np.int32)
        orc.set_state(st)
        near = (st.a["z"] < op.dthr) & (st.a["knob"] == 1) & (f[2] <= 2)
        g = np.stack(np.meshgrid(np.arange(0, op.Lx, 0.5), np.arange(0, op.Ly, 0.5), indexing="ij")).reshape(2, -1)
        d = [st.a[k][near][:, None] - g[i][None] for i, k in enumerate("xy")]
        listed = np.logical_and(*[np.abs(f[i][near][:, None] + 0.5 - g[i][None]) < 1.5 for i in (0, 1)])
        d2 = d[0] ** 2 + d[1] ** 2 + st.a["z"][near][:, None] ** 2
        pairs = (listed & (d2 <= op.dthr ** 2)).sum(axis=1)
        assert pairs.max() <= 64
        if case == "events":  # every draw succeeds
            assert (pairs > 0).sum() <= 1024 and pairs.sum() > 128
        else:
            assert (pairs > 0).sum() > 1024
    patches = _against_single_steps(op, orc, 43, st, precision, 1, (3, 22))
    cluster = H.gpu_like(op, orc, 43, precision=precision, state=st)
    cluster.set_membrane_kernels(3)
    cluster.step(25)
    assert H.compare(patches, cluster.get_state(), 0.0) == {}
    if case != "parasite":
        assert patches.a["bondi"].sum() > 0
    if precision == 0:
        s = H.gpu_like(op, orc, 43, precision=0, state=st)
        for k in range(14):
            orc.step(1)
            s.step(1)
            assert H.compare(s.get_state(), orc.get_state()) == {}, k


def test_free_flight_in_a_box_longer_than_a_float_resolves():
    """At x > 2^16 an FP32 particle moves in units of 2^-7: 11 steps of 11.51
    units are rounded to 12 each, more than the 0.99 of a cell that its speed
    gives, so one that starts at the end of the last cell but one leaves the box
    in one stretch and is wrapped as by single steps."""
    import irbc_b200 as G
    V, E, T = H.geodesic(2, 1.0)
    ulp = 2.0 ** -7
    p = G.default_params(Lx=66000.0, Ly=6.0, Lz=6.0, Ns=40, seed=5, precision=G.FP32, dtcd=0.0221, Nt=len(V))
    sims = []
    for _ in range(2):
        s = G.Simulation(p)
        s.init(V, E, T, 0)
        st = s.get_state()
        st.a["sx"] = 65999.0 - ulp * np.arange(1, 41)
        st.a["sy"], st.a["sz"] = np.full(40, 3.5), np.full(40, 3.5)
        st.a["svx"], st.a["svy"], st.a["svz"] = np.full(40, 11.51 * ulp / p.dtmd), np.zeros(40), np.zeros(40)
        s.set_state(st)
        sims.append(s)
    sims[0].step(11)
    for _ in range(11):
        sims[1].call("step_part1")
        sims[1].call("step_part2")
    want = sims[1].get_state()
    assert (want.a["sx"] < 10.0).any()
    assert H.compare(sims[0].get_state(), want, 0.0) == {}


def test_profile_counts_steps_and_launches():
    """A profiled window counts the streamed steps, however many of them a
    launch takes, and the launches of the bulk kernel."""
    op, orc = H.make_oracle(ns=5000, seed=41, Lx=40.0, Ly=20.0, Lz=20.0)
    sim = H.gpu_like(op, orc, 41)
    sim.call("profile_begin")
    sim.step(30)  # three stretches of ten
    sim.call("step_part1")
    sim.call("step_part2")
    out = sim.profile_end()
    assert out["stream_steps"] == 31
    assert out["collides"] == 3
    assert out["bulk_launches"] == 4


# the smallest geodesic mesh that no cluster holds in patches, the largest one
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("freq", [17, 28])
def test_meshes_beyond_the_patches(freq, precision):
    """Meshes above the patches' size run a kernel a phase: stretches, with
    bonds, equal single steps, mode 3 (a cluster on global memory) and replayed
    graphs bit for bit, and in FP64 the oracle step by step within 1e-12."""
    V, E, T = H.geodesic(freq, 0.07 * np.sqrt(10.0 * freq * freq + 2))
    op, orc = _mesh_oracle(V, E, T, 1500, Ns=30000, onrate=300.0, offrate=50.0, Lx=40.0, Ly=24.0, Lz=24.0)
    st = orc.get_state()
    sims = [H.gpu_like(op, orc, 43, precision=precision, state=st) for _ in range(4)]
    sims[1].set_membrane_kernels(3)
    sims[2].set_graphs(True)
    for n in (3, 40):
        for s in sims[:3]:
            s.step(n)
        for _ in range(n):
            sims[3].call("step_part1")
            sims[3].call("step_part2")
        want = sims[3].get_state()
        for k, s in enumerate(sims[:3]):
            assert H.compare(s.get_state(), want, 0.0) == {}, (n, k)
    assert sims[3].get_state().a["bondi"].sum() > 0
    if precision == 1:  # members of a cohort, beside one in patches
        import irbc_b200 as G
        top, torc = H.make_oracle(ns=20000, seed=44, Lx=40.0, Ly=20.0)
        b = G.Batch(nthreads=1)
        members = [H.gpu_like(op, orc, 43, precision=1, state=st) for _ in range(2)]
        members.append(H.gpu_like(top, torc, 44, precision=1))
        alone = H.gpu_like(top, torc, 44, precision=1)
        for s in members:
            b.add(s)
        for n in (3, 40):
            b.step(n)
            alone.step(n)
        for s in members[:2]:
            assert H.compare(s.get_state(), want, 0.0) == {}
        assert H.compare(members[2].get_state(), alone.get_state(), 0.0) == {}
        b.close()
    else:
        s = H.gpu_like(op, orc, 43, precision=0, state=st)
        for k in range(4):
            orc.step(1)
            s.step(1)
            assert H.compare(s.get_state(), orc.get_state()) == {}, k


@pytest.mark.parametrize("precision", [0, 1])
def test_a_mesh_takes_another_ones_place(precision):
    """Meshes set one after the other on one handle, in patches of 8 and 16
    blocks and beyond them: each steps as on a handle of its own."""
    import irbc_b200 as G
    from irbc_b200 import mesh
    box = dict(Ns=8000, Lx=40.0, Ly=20.0, Lz=20.0)
    meshes = [H.troph(), mesh.discocyte(), H.geodesic(17, 3.0), H.geodesic(2, 3.0)]
    sim = None
    for V, E, T in meshes + meshes[:1]:
        op, orc = _mesh_oracle(V, E, T, 12, **box)
        p = H.to_irbc_params(op, 43, precision)
        if sim is None:
            sim = G.Simulation(p)
            p0 = p
        alone = G.Simulation(p0)
        for s in (sim, alone):  # (both with the first mesh's elap)
            s.set_mesh(orc.get_mesh())
            s.set_state(G.State.from_other(orc.get_state()))
            s.step(25)
        assert H.compare(sim.get_state(), alone.get_state(), 0.0) == {}, len(V)
        alone.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("Lz", [20.0, 300.0])  # layers in shared memory (256), beyond
def test_layer_sums(Lz, precision):
    """Temperature, mean velocity and profiles against sums of the state in
    numpy: n additions in any order differ by at most n eps of the terms'
    magnitudes."""
    op, orc = H.make_oracle(ns=20000, seed=43, Lx=30.0, Ly=15.0, Lz=Lz)
    sim = H.gpu_like(op, orc, 43, precision=precision)
    sim.step(3)
    s = sim.get_state().a
    v, z = np.stack([s["svx"], s["svy"], s["svz"]]), s["sz"]
    n, eps = z.size, 2.0 ** -53
    o = sim.observables()
    tol = n * eps
    lay = np.clip(np.floor(z).astype(int), 0, int(Lz) - 1)
    m = np.bincount(lay, minlength=int(Lz))
    u = np.stack([np.bincount(lay, w, int(Lz)) for w in v]) / np.maximum(m, 1)
    # the layers' means are subtracted from the whole, so errors are the whole's
    whole = np.mean(v ** 2)
    assert abs(o[0] - np.mean((v - u[:, lay]) ** 2)) <= 4 * tol * whole
    assert abs(o[8] - whole) <= tol * whole
    assert abs(o[7] - np.mean(v[0])) <= tol * np.mean(np.abs(v[0]))
    for bins in (1, 20, 256, 257, 300):
        b = np.clip(np.floor(z).astype(int), 0, bins - 1)
        c = np.bincount(b, minlength=bins)
        want = np.bincount(b, v[0], bins) / np.maximum(c, 1)
        bound = tol * np.bincount(b, np.abs(v[0]), bins) / np.maximum(c, 1)
        assert (np.abs(sim.velocity_profile(bins) - want) <= bound).all(), bins


def test_collisions_above_4096_tiles():
    """Two collisions in a box of 4128 tiles (three arrays in one scan) against
    the oracle, and a cohort of two such members against one alone."""
    import irbc_b200 as G
    V, E, T = H.geodesic(2, 3.0)
    op, orc = _mesh_oracle(V, E, T, 12, Ns=20000, Lx=129.0, Ly=128.0, Lz=255.0, dtcd=0.004)
    st = orc.get_state()
    sim = H.gpu_like(op, orc, 43, state=st)
    alone, *members = [H.gpu_like(op, orc, 43, precision=1, state=st) for _ in range(3)]
    orc.step(4)
    sim.step(4)
    assert H.compare(sim.get_state(), orc.get_state()) == {}
    b = G.Batch(nthreads=1)
    for s in members:
        b.add(s)
    b.step(4)
    alone.step(4)
    for s in members:
        assert H.compare(s.get_state(), alone.get_state(), 0.0) == {}
    b.close()


@pytest.mark.parametrize("box", [(16, 16, 3), (31, 11, 2), (41, 5, 4), (3, 1, 1), (128, 128, 64),
                                 (128, 128, 255), (129, 128, 255)])
def test_cell_scan_at_tile_edges(box):
    """Counting sorts over 1024, 1023, 1025, 6 and 1,064,960 cells (a tile of
    the scan has 1024 cells; 1040 tiles are more than a block's threads), over
    4096 tiles, the most that go without a launch for the tiles' sums, and over
    4128, whose sums are scanned in groups of 1024; cells sorted by a thread
    each below four particles a cell, by sixteen lanes from there on."""
    import torch
    import irbc_b200 as G
    Lx, Ly, Lz = box
    p = G.default_params(Lx=float(Lx), Ly=float(Ly), Lz=float(Lz), Ns=0)
    ncell = Lx * Ly * (Lz + 1)
    rng = np.random.default_rng(3)
    for n in (0, 1, 5000) + ((4 * ncell - 1, 4 * ncell) if ncell < 2000 else ()):
        pos = [torch.tensor(rng.uniform(0, L, n), device="cuda") for L in box]
        cell = torch.zeros(max(n, 1), dtype=torch.int32, device="cuda")
        start = torch.full((ncell + 1,), -1, dtype=torch.int32, device="cuda")
        order = torch.zeros(max(n, 1), dtype=torch.int32, device="cuda")
        rc = G.lib().irbc_bin_particles(C.byref(p), *[q.data_ptr() for q in pos], n, 0.25, 0.5, 0.75,
                                        cell.data_ptr(), start.data_ptr(), order.data_ptr())
        assert rc == 0
        f = [np.floor((q.cpu().numpy() - r) % L) for q, r, L in zip(pos[:2], (0.25, 0.5), box)]
        want = ((f[0] * Ly + f[1]) * (Lz + 1) + np.floor(pos[2].cpu().numpy() + 0.25)).astype(np.int64)
        np.testing.assert_array_equal(cell.cpu().numpy()[:n], want)
        np.testing.assert_array_equal(start.cpu().numpy(),
                                      np.concatenate([[0], np.cumsum(np.bincount(want, minlength=ncell))]))
        np.testing.assert_array_equal(order.cpu().numpy()[:n], np.argsort(want, kind="stable"))
