"""The many-step kernels (resident on small meshes, streamed on mid-size
ones; the default there) against the two-kernel step -- GPU.

Both compute each triangle with the same arithmetic and sum every node's
contributions in ascending triangle order from zero
(calc_deformation_forces.cpp:185), so they give the same bits."""
from __future__ import annotations

import os

import numpy as np
import pytest

from conftest import deformed_state, make_model

pytestmark = pytest.mark.gpu


def _pair(m, precision=0, a_info=None, b_info=None, protocol=3):
    from morphoshell_b200 import GpuLoop
    s = m.scalars
    if a_info is None:
        a_info, b_info = m.programmed()
    out = []
    for path in (None, 2):
        g = GpuLoop(m, precision=precision)
        g.set_programmed(protocol, a_info, b_info, s.dial_factors_to_hold_at_spacing)
        if path is not None:
            g.set_step_path(path)
        out.append(g)
    return out


def _same(ga, gb):
    return all(np.array_equal(a, b) for a, b in zip(ga.download(), gb.download()))


def _equil(r):
    e = r.equil
    return e.max_force, e.max_speed, e.max_force_node, e.max_speed_node, e.at_equilibrium


# Resident: disk250, a handful of tiles; disk100, disk50, 128 threads; disk18k,
# 256; disk15, 384.  Streamed: disk14, the smallest; disk7; disk6; disk5, near
# the largest in both precisions; disk4, too large for both.
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", ["disk250", "disk100", "disk50", "disk18k", "disk15", "disk14", "disk7", "disk6", "disk5", "disk4"])
def test_resident_equals_two_kernel_bitwise(workdir, name, precision):
    m = make_model(workdir, name)
    s = m.scalars
    x, v = deformed_state(m, seed=41, amp=0.02)
    ga, gb = _pair(m, precision)
    reps = []
    for g in (ga, gb):
        g.upload(x, v)
        g.step_n(1, np.array([0.2]), s.timestep, s.damping_factor_1)
        g.step_n(300, 0.2 + 1e-5 * np.arange(300), s.timestep, s.damping_factor_1)
        g.do_dialling(0.21)
        r1 = g.step_n(2, None, s.timestep, s.damping_factor_2, check_last=True)
        r2 = g.step_n(101, None, s.timestep, s.damping_factor_2, check_last=True)
        reps.append((_equil(r1), _equil(r2)))
    assert reps[0] == reps[1]
    assert _same(ga, gb)


@pytest.mark.parametrize("name,steps", [("disk100", 20001), ("disk12", 300)])
def test_resident_more_than_one_launch_and_gradient_descent(workdir, name, steps):
    m = make_model(workdir, name)
    s = m.scalars
    x, v = deformed_state(m, seed=42, amp=0.02)
    ga, gb = _pair(m)
    for g in (ga, gb):
        g.upload(x, v)
        g.step_n(steps, 0.2 + 1e-7 * np.arange(steps), s.timestep, s.damping_factor_1)
        g.do_dialling(0.2)
        g.step_n(7, None, 1e-3 * s.timestep, s.damping_factor_1, gd=True)
    assert _same(ga, gb)


def test_resident_other_metrics_and_constraints(workdir, tmp_path):
    """Programmed tensors with bbar from the arrays, per-triangle fields and
    materials (which take the general path), constrained nodes, and a mesh
    whose labels follow no curve."""
    from morphoshell_b200 import Model, meshgen
    mesh = meshgen.disk_mesh(0.12, seed=5, reorder=False)
    info = meshgen.lce_abar_info(mesh, meshgen.azimuthal_director, 0.9)
    rng = np.random.default_rng(6)
    T, N = mesh.num_tris, mesh.num_nodes
    st = os.path.join(str(tmp_path), "s.txt")
    meshgen.write_settings(st, protocol=3)
    bbar = 0.3 * rng.standard_normal((T, 3))
    fixed = (rng.random(N) < 0.1).astype(np.uint8)
    varied = info.copy()
    varied[:, 1] = 0.85 + 0.05 * rng.random(T)
    for kw, a, b, protocol in [({}, info, bbar, 3), ({}, varied, bbar, 3),
                               ({}, meshgen.lce_abar_comps(info, 1.0), bbar, 1),
                               ({"shear_modulus": 1 + 0.3 * rng.random(T)}, info, bbar, 3)]:
        m = Model.from_arrays(st, mesh.nodes, mesh.tris, info, bbar, constrained=fixed, **kw)
        s = m.scalars
        x, v = deformed_state(m, seed=43, amp=0.02)
        ga, gb = _pair(m, a_info=a, b_info=b, protocol=protocol)
        for g in (ga, gb):
            g.upload(x, v)
            g.step_n(40, 0.2 + 1e-5 * np.arange(40), s.timestep, s.damping_factor_1)
            g.do_dialling(0.3)
            g.step_n(40, None, s.timestep, s.damping_factor_2)
        assert _same(ga, gb)


@pytest.mark.parametrize("name", ["disk18k", "disk10"])
@pytest.mark.parametrize("at", [0, 3])
def test_resident_guard(workdir, at, name):
    """A trip of the force guard: the same step, dof, force and surviving
    state as the two-kernel step, at the first step and later (a node whose
    speed carries it away)."""
    from morphoshell_b200 import MsError
    m = make_model(workdir, name)
    s = m.scalars
    x, v = deformed_state(m, seed=44, amp=0.02)
    node = 2 * m.num_nodes + 4321
    if at == 0:
        x[node] += 1e6
    else:
        v[node] = 10.0 / s.timestep
    got = []
    for g in _pair(m):
        g.upload(x, v)
        with pytest.raises(MsError) as ei:
            g.step_n(500, None, s.timestep, s.damping_factor_2)
        r = ei.value.report
        got.append((r.error_step, r.offending_dof, r.offending_force, r.steps_done) + tuple(map(bytes, g.download())))
    assert got[0] == got[1]
    assert (got[0][0] == 0) == (at == 0)


def _batch_members(tmp_path, ks, **kw):
    from morphoshell_b200 import ensemble
    # Short dial phases and loose thresholds: whole runs in a few thousand steps.
    fast = dict(dial_factors_to_hold_at_spacing=0.5, dial_phase_time_prefactor=0.02,
                force_to_char_force_ratio_equil_threshold=1e-5, speed_to_char_speed_ratio_equil_threshold=1e-4)
    return ensemble.build_members(ks, str(tmp_path), threads=4, **dict(fast, **kw))[0]


def _batch_state(b):
    out = []
    for i in range(b.n):
        s = b.status(i)
        out.append((s.status, s.equilibria, s.stepcount, s.dial_factor, s.last_equil_dial, s.sim_time, s.max_force_ratio,
                    s.max_speed_ratio, s.max_force_node, s.max_speed_node, s.offending_dof)
                   + tuple(map(bytes, b.download(i))))
    return out


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_stretches_equal_step_by_step(tmp_path, precision):
    """Streamed stretches of a batch against its two-kernel schedule: from the
    start through dial phases, checks, one instance reaching its final
    equilibrium and one failing on the guard; the same states and step
    counts at every stop."""
    from morphoshell_b200 import MS_INST_DONE, MS_INST_FAILED, Batch
    models = _batch_members(tmp_path, [12, 13, 14], spacing_range=(0.07, 0.1))
    bad = models[2].dofs(1).copy()
    vel = np.zeros_like(bad)
    vel[2 * models[2].num_nodes + 5] = 10.0 / models[2].scalars.timestep
    a, b = Batch(models, precision=precision), Batch(models, precision=precision)
    b.set_schedule(0, 256, 64)
    for g in (a, b):
        g.upload(2, bad, vel)
    for steps in (1, 7, 100, 1001, 20_000, 400_000):
        assert a.run(steps) == b.run(steps)
        assert _batch_state(a) == _batch_state(b)
    assert a.status(2).status == MS_INST_FAILED
    assert a.status(0).status == MS_INST_DONE and a.status(1).status == MS_INST_DONE


@pytest.mark.parametrize("ks,lo,hi", [([3], 0.02, 0.021), ([3, 4, 5, 6, 7, 8], 0.012, 0.02), (list(range(40)), 0.08, 0.1)])
def test_batch_stretches_many_sizes(tmp_path, ks, lo, hi):
    """One instance, several per SM, and tiles of several instances; from the
    start and from warm starts in both kinds of phase."""
    from morphoshell_b200 import Batch
    models = _batch_members(tmp_path, ks, spacing_range=(lo, hi))
    a, b = Batch(models), Batch(models)
    b.set_schedule(0, 256, 64)
    for g in (a, b):
        for i, m in enumerate(models):
            if i % 3:
                g.upload(i, *deformed_state(m, seed=50 + i, amp=0.02))
                g.set_start(i, 0.52 if i % 3 == 1 else 1.0, i % 3 == 2)
    assert a.run(700) == b.run(700)
    assert _batch_state(a) == _batch_state(b)


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_node_tiled_stretches_equal_step_by_step(tmp_path, precision):
    """Quiet stretches of the node-tiled schedule (one launch a step) against
    the two-kernel schedule: lengths around the shortest stretch and the
    longest, dial phases, checks, an instance that fails inside a stretch while
    the others go on, one that failed before, and a warm start in each kind of
    phase."""
    from morphoshell_b200 import MS_INST_DONE, MS_INST_FAILED, Batch
    models = _batch_members(tmp_path, [12, 13, 14, 15], spacing_range=(0.07, 0.1))
    bad = models[2].dofs(1).copy()
    vel = np.zeros_like(bad)
    vel[2 * models[2].num_nodes + 5] = 10.0 / models[2].scalars.timestep
    warm = deformed_state(models[3], seed=53, amp=0.02)
    a, b = Batch(models, precision=precision), Batch(models, precision=precision)
    a.set_schedule(-1, 0, 64)
    b.set_schedule(0, 256, 64)
    for g in (a, b):
        g.upload(3, *warm)
        g.set_start(3, 0.52, True)
    for steps in (1, 7, 8, 9, 300, 1001):
        assert a.run(steps) == b.run(steps)
        assert _batch_state(a) == _batch_state(b)
    for g in (a, b):
        g.upload(2, bad, vel)
    for steps in (100, 20_000, 400_000):
        assert a.run(steps) == b.run(steps)
        assert _batch_state(a) == _batch_state(b)
    assert a.status(2).status == MS_INST_FAILED
    assert a.status(0).status == MS_INST_DONE and a.status(1).status == MS_INST_DONE


@pytest.mark.parametrize("sched", [None, (-1, 0)])
def test_batch_steps_reported_when_the_last_instance_fails(tmp_path, sched):
    """A run ends with the chunk of the step at which its last instance fails,
    with and without a stretch before that step."""
    from morphoshell_b200 import MS_INST_FAILED, Batch
    # An unstable timestep: both fail, one sooner.
    models = _batch_members(tmp_path, [12, 13], spacing_range=(0.07, 0.1), timestep_prefactor=1.7)
    out = []
    for choice in (sched, (0, 256)):
        g = Batch(models)
        if choice is not None:
            g.set_schedule(*choice, 64)
        for i, m in enumerate(models):
            g.upload(i, *deformed_state(m, seed=50 + i, amp=(1e-6, 1e-2)[i]))
        done = [g.run(10), g.run(3000)]
        assert all(g.status(i).status == MS_INST_FAILED for i in range(2))
        out.append((done, _batch_state(g)))
    assert out[0] == out[1]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", ["disk100", "disk18k", "disk15", "disk14"])
@pytest.mark.parametrize("launch", [0, 1, 2])
def test_wait_that_runs_out(workdir, name, launch, precision):
    """A launch given up because a tile's wait ran out -- the first of a call,
    the second, which writes the buffer the call began from, or the third, with
    the check -- leaves no trace: the bits and the report of the two-kernel
    step, and so the next call's with waits as they were."""
    m = make_model(workdir, name)
    s = m.scalars
    x, v = deformed_state(m, seed=45, amp=0.02)
    n = 128 + 8192 + 160
    out = []
    for g in _pair(m, precision):
        g.upload(x, v)
        g.set_wait_limit(0, launch)
        r = [_equil(g.step_n(n, 0.2 + 1e-6 * np.arange(n), s.timestep, s.damping_factor_1, check_last=True))]
        noted = g.last_error()
        state = g.download()
        metric = g.programmed()
        g.set_wait_limit(2_000_000_000)
        r.append(_equil(g.step_n(200, None, s.timestep, s.damping_factor_2, check_last=True)))
        out.append((noted, r, [bytes(a) for a in (*state, *metric, *g.download())]))
    assert "waited too long" in out[0][0] and not out[1][0]
    assert out[0][1:] == out[1][1:]


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_wait_that_runs_out(tmp_path, precision):
    """The same for a batch's stretches: step by step instead, from the states
    and counters before."""
    from morphoshell_b200 import Batch
    models = _batch_members(tmp_path, [12, 13, 14, 15, 16, 17], spacing_range=(0.03, 0.05))
    a, b = Batch(models, precision=precision), Batch(models, precision=precision)
    b.set_schedule(0, 256, 64)
    for steps, clocks in [(100, 2_000_000_000), (300, 0), (300, 2_000_000_000), (3000, 0)]:
        a.set_wait_limit(clocks)
        assert a.run(steps) == b.run(steps)
        assert _batch_state(a) == _batch_state(b)
        assert ("waited too long" in a.last_error()) == (steps > 100)


@pytest.mark.parametrize("precision", [0, 1])
def test_varied_materials_keep_the_node_tiled_plan(workdir, tmp_path, precision):
    """A mid-size mesh with a material per triangle, which the many-step
    kernels do not take: node tiles of at least 256 nodes as without those
    kernels, and the two-kernel step's bits on them."""
    from morphoshell_b200 import Model, meshgen
    mesh = meshgen.disk_mesh(0.013, seed=5)
    info = meshgen.lce_abar_info(mesh, meshgen.azimuthal_director, 0.9)
    st = os.path.join(str(tmp_path), "s.txt")
    meshgen.write_settings(st, protocol=3, ref_shear_modulus_if_uniform=-1.0)
    shear = 1 + 0.3 * np.random.default_rng(7).random(mesh.num_tris)
    m = Model.from_arrays(st, mesh.nodes, mesh.tris, info, np.zeros((mesh.num_tris, 3)), shear_modulus=shear)
    assert np.ptp(m.tables()["ref_shear_modulus"]) > 0.2
    s = m.scalars
    ga, gb = _pair(m, precision)
    assert ga.plan_info()["nodes_per_tile"] >= 256
    ga.set_step_path(3)
    for g in (ga, gb):
        g.upload(*deformed_state(m, seed=46, amp=0.02))
        g.step_n(40, 0.2 + 1e-5 * np.arange(40), s.timestep, s.damping_factor_1)
        g.do_dialling(0.3)
        g.step_n(40, None, s.timestep, s.damping_factor_2)
    assert _same(ga, gb)


@pytest.mark.parametrize("name,precision,first", [("disk100", 0, 128), ("disk18k", 1, 128), ("disk5", 0, 128),
                                                  ("disk4", 0, 0), ("disk4", 1, 128)])
def test_many_step_launches(workdir, name, precision, first):
    """The library's own answer whether and in how many launches whole
    stretches run: none on meshes too large for them, with a path by number,
    or for single steps."""
    g = _pair(make_model(workdir, name), precision)[0]
    assert g.many_step_launches(1) == 0
    for n, launches in [(2, 1), (128, 1), (255, 1), (256, 2), (128 + 8192, 2), (128 + 8192 + 128, 3)]:
        assert g.many_step_launches(n) == (launches if first else 0)
    assert g.many_step_launches(8192 + 127, dialling=False) == (1 if first else 0)
    assert g.many_step_launches(8192 + 128, dialling=False) == (2 if first else 0)
    g.set_step_path(2)
    assert g.many_step_launches(1000) == 0


def _without_neighbours(m, first):
    """The model with its first nodes cut off from the rest: triangles on both
    stand for another triangle once more, with no area."""
    import ctypes as C
    import types
    t = m.tables()
    ids, w, area = (t[k].copy() for k in ("patch_ids", "deriv_coeffs", "ref_area"))
    ids = ids.astype(np.int32)
    both = ((ids < first).any(1)) & ((ids >= first).any(1))
    other = np.flatnonzero((ids >= first).all(1))[0]
    ids[both], w[both], area[both] = ids[other], w[other], 0.0
    desc = type(m.desc)()
    C.memmove(C.byref(desc), C.byref(m.desc), C.sizeof(desc))
    desc.patch_ids = ids.ctypes.data_as(C.POINTER(C.c_int32))
    desc.deriv_coeffs = w.ctypes.data_as(C.POINTER(C.c_double))
    desc.ref_area = area.ctypes.data_as(C.POINTER(C.c_double))
    return types.SimpleNamespace(desc=desc, params=m.params, scalars=m.scalars, num_nodes=m.num_nodes,
                                 num_tris=m.num_tris, programmed=m.programmed, dofs=m.dofs, keep=(ids, w, area))


# Nodes cut off: as many as a tile of the mesh without them as neighbours has.
# The meshes have under 256 nodes, so that the check by itself is one block.
@pytest.mark.parametrize("name,first", [("disk125", 32), ("disk135", 37), ("disk145", 36)])
def test_guard_and_wait_in_one_launch(workdir, name, first):
    """A launch in which a node trips the guard, the waits of tiles run out and
    the first, which waits for nobody, reaches the check on its last step:
    reported as the two-kernel step reports it, and the checks after it are of
    the state then."""
    from morphoshell_b200 import MsError
    m = _without_neighbours(make_model(workdir, name), first)
    s = m.scalars
    x, v = deformed_state(m, seed=47, amp=0.02)
    bad = x.copy()
    bad[-3] += 1e6
    out = []
    for g in _pair(m):
        got = []
        for k in range(3):
            g.upload(x, (1.0 + k) * v)
            got.append(_equil(g.step_n(3, None, s.timestep, s.damping_factor_2, check_last=True)))
            g.upload(bad, v)
            g.set_wait_limit(0)
            with pytest.raises(MsError) as ei:
                g.step_n(2, None, s.timestep, s.damping_factor_2, check_last=True)
            r = ei.value.report
            got.append((r.error_step, r.offending_dof, r.offending_force, r.steps_done))
            g.set_wait_limit(2_000_000_000)
            e = g.is_at_equilibrium()
            got.append((e.max_force, e.max_speed, e.max_force_node, e.max_speed_node))
        out.append(got)
    assert out[0] == out[1]
