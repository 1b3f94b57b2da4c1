"""Cohorts: FP32 simulations stepped together with one kernel launch per
phase of the step (irbc_schedule.fused), each launch's blocks split among
the members.  Every member must end bit for bit where the same simulation
ends alone on the plain path: uneven boxes, knob counts and bond rates,
two meshes in one cohort, list updates and the physical re-sort inside the
stretch, and members that fall out of phase with the others."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _params(seed, Lx, ns, precision=1, **over):
    import irbc_b200 as G
    p = G.default_params(Lx=float(Lx), Ns=ns, seed=seed, precision=precision, **over)
    return p


def _alone(p, V, E, T, nknobs, steps):
    import irbc_b200 as G
    sim = G.Simulation(p)
    sim.init(V, E, T, nknobs)
    sim.step(steps)
    st = sim.get_state()
    sim.close()
    return st


def _check(sims, cfgs, steps):
    for sim, (p, (V, E, T), nk) in zip(sims, cfgs):
        ref = _alone(p, V, E, T, nk, steps)
        bad = H.compare(sim.get_state(), ref, 0.0)
        assert bad == {}, (p.seed, bad)


def test_fused_batch_equals_members_alone():
    """Five FP32 members (boxes 40..72 long, 300..600 knobs, one with bond
    rates raised so that bonds form and break) stepped 200 steps as one
    cohort, in two calls: 16 collisions (the 16th re-sorts the solvent),
    and list updates at steps 82 and 165."""
    import irbc_b200 as G
    troph = H.troph()
    cfgs = []
    for r, (Lx, nk, over) in enumerate([(60, 500, {}), (40, 300, {}), (72, 600, dict(onrate=300.0, offrate=50.0)),
                                        (48, 400, {}), (56, 350, {})]):
        cfgs.append((_params(700 + r, Lx, int(Lx * 40 * 41 * 3), **over), troph, nk))
    sims = []
    b = G.Batch(nthreads=2)
    assert b.schedule()["fused"] == 1
    for p, (V, E, T), nk in cfgs:
        s = G.Simulation(p)
        s.init(V, E, T, nk)
        sims.append(s)
        b.add(s)
    launches0 = sims[0].launch_count()
    b.step(37)
    b.step(163)
    # one launch per phase: far fewer than five members' own launches
    assert sims[0].launch_count() - launches0 < 200 * 40
    _check(sims, cfgs, 200)
    b.close()
    for s in sims:
        s.close()


def test_fused_cohort_with_two_meshes_and_an_fp64_member():
    """The 600-vertex trophozoite and the 2562-vertex discocyte in one
    cohort, and an FP64 member beside it (stepped by the pool of host
    threads): each equals itself alone."""
    import irbc_b200 as G
    from irbc_b200 import mesh
    troph, disc = H.troph(), mesh.discocyte()
    de = mesh.scaled_elap(disc[0], disc[1])
    cfgs = [(_params(801, 48, 48 * 40 * 41 * 3), troph, 300),
            (_params(802, 40, 40 * 40 * 41 * 3, Nt=len(disc[0]), elap=de, walls=0.4), disc, 800),
            (_params(803, 44, 44 * 40 * 41 * 3, precision=0), troph, 250)]
    sims = []
    b = G.Batch(nthreads=2)
    for p, (V, E, T), nk in cfgs:
        s = G.Simulation(p)
        s.init(V, E, T, nk)
        sims.append(s)
        b.add(s)
    b.step(60)
    b.step(36)
    _check(sims, cfgs, 96)
    b.close()
    for s in sims:
        s.close()


def test_members_out_of_phase_form_their_own_cohorts():
    """A member that has taken 7 steps alone before joining is out of phase
    with the others (its collisions fall on other steps): the batch steps
    it in a cohort of its own, and every member still equals itself alone."""
    import irbc_b200 as G
    troph = H.troph()
    cfgs = [(_params(900 + r, 40 + 4 * r, (40 + 4 * r) * 40 * 41 * 3), troph, 300) for r in range(3)]
    sims = []
    for p, (V, E, T), nk in cfgs:
        s = G.Simulation(p)
        s.init(V, E, T, nk)
        sims.append(s)
    sims[2].step(7)
    b = G.Batch(nthreads=2)
    for s in sims:
        b.add(s)
    b.step(50)
    _check(sims[:2], cfgs[:2], 50)
    _check(sims[2:], cfgs[2:], 57)
    b.close()
    for s in sims:
        s.close()


def test_members_an_odd_number_of_steps_apart_share_a_cohort():
    """Five steps between collisions: a member five steps ahead collides on the
    same steps as another, so both advance in one cohort (as many launches as
    for one member), and each equals itself alone."""
    import irbc_b200 as G
    troph = H.troph()
    cfgs = [(_params(910 + r, 40, 20000, dtcd=0.01), troph, 300) for r in range(3)]
    sims = []
    for p, (V, E, T), nk in cfgs:
        s = G.Simulation(p)
        s.init(V, E, T, nk)
        sims.append(s)
    sims[0].step(5)
    sims[1].step(10)
    launches = []
    for group in ((sims[2],), sims[:2]):
        b = G.Batch(nthreads=2)
        for s in group:
            b.add(s)
        if len(group) == 1:
            b.step(5)
        n0 = sims[0].launch_count()
        b.step(40)
        launches.append(sims[0].launch_count() - n0)
        b.close()
    # (a launch per member sets its draw base)
    assert launches[1] == launches[0] + 1
    for s, c, n in zip(sims, cfgs, (45, 50, 45)):
        _check([s], [c], n)


def test_cohort_reflects_what_rounding_carries_to_the_membrane():
    """A cohort takes 16 steps in one part.  In a box longer than 256 a
    particle at x > 256 moves in units of 2^-15; with v dt = 23.51 of them it is
    rounded to 24 a step, so one that starts 381 to 383 units before the
    membrane, which 16 steps of v dt do not reach, crosses it in the last step.
    The members equal single steps bit for bit."""
    import irbc_b200 as G
    from irbc_b200 import mesh
    # a cube of side 2, each face in 2 x 2 squares
    pts, T = {}, []
    for k in range(3):
        for side in (-1, 1):
            at = {}
            for i in (-1, 0, 1):
                for j in (-1, 0, 1):
                    q = [i, j]
                    q.insert(k, side)
                    at[i, j] = pts.setdefault(tuple(q), len(pts))
            for i in (-1, 0):
                for j in (-1, 0):
                    c = at[i, j], at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]
                    T += [(c[0], c[1], c[2]), (c[0], c[2], c[3])]
    V, T = np.array(list(pts), float), np.array(T, np.int32)
    nv = len(V)
    T = mesh.orient_outward(V, T)
    E = mesh.edges_of(T)
    ulp, face = 2.0 ** -15, 261.0
    units = np.arange(365, 395)
    spots = [(5.3, 6.45), (6.62, 6.55), (6.4, 5.2)]  # (y, z) inside triangles of the face
    ns = len(units) * len(spots)
    # (a heavy membrane stays where it is)
    p = G.default_params(Lx=276.0, Ly=12.0, Lz=12.0, Ns=ns, seed=5, precision=G.FP32, dtcd=0.05, pmass=1e12, Nt=nv)
    ends, sims = [], []
    for _ in range(3):
        s = G.Simulation(p)
        s.init(V, E, T, 0)
        st = s.get_state()
        a = st.a
        a["x"], a["y"], a["z"] = V[:, 0] + face + 1.0, V[:, 1] + 6.0, V[:, 2] + 6.0
        for k in ("vx", "vy", "vz"):
            a[k] = np.zeros(nv)
        st.s.update(para=np.array([20.0, 6.0, 6.0]), paraV=np.zeros(3))
        a["sx"] = np.repeat(face - units * ulp, len(spots))
        a["sy"], a["sz"] = np.tile(np.array(spots).T, len(units))
        a["svx"] = np.full(ns, 23.51 * ulp / p.dtmd)
        a["svy"], a["svz"], a["sindio"] = np.zeros(ns), np.zeros(ns), np.ones(ns, np.int32)
        s.set_state(st)
        s.call("llist_update")
        sims.append(s)
    for _ in range(16):
        sims[2].call("step_part1")
        sims[2].call("step_part2")
    b = G.Batch(nthreads=1)
    b.add(sims[0])
    b.add(sims[1])
    b.step(16)
    ends = [s.get_state() for s in sims]
    hit = (ends[2].a["svx"] < 0).reshape(len(units), len(spots))
    late = (units >= 381) & (units <= 383)
    assert hit[late].any() and not hit[units >= 385].any()
    for k in (0, 1):
        assert H.compare(ends[k], ends[2], 0.0) == {}, k
    b.close()
