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
# 256; disk15, 384.  Streamed: disk14, the smallest; disk7; disk6, near the
# largest in FP64; disk5, mixed only; disk4, too large for both.
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
