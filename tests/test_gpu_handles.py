"""Several handles alive together, host threads, and page-locked sources -- GPU.

What one handle or call does must not depend on what another handle did
before or does meanwhile, nor a call's result on what its caller does with
the arrays after it has returned."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import deformed_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [0.05, 0.006])
@pytest.mark.parametrize("pinned", [(True, True), (False, True), (False, False)])
def test_batch_upload_has_read_its_source(tmp_path, pinned, spacing):
    """One staging buffer each for positions and velocities, page-locked or
    not, filled and uploaded member after member while the batch's stream is
    busy: each member gets its own state."""
    import torch
    from morphoshell_b200 import Batch, ensemble
    models, _ = ensemble.build_members([0, 1, 2], str(tmp_path), spacing_range=(spacing, 1.2 * spacing),
                                       threads=4)
    b = Batch(models)
    stream = torch.cuda.ExternalStream(b.stream())
    most = 3 * max(m.num_nodes for m in models)
    stage = [torch.empty(most, dtype=torch.float64, pin_memory=p).numpy() for p in pinned]
    want = [deformed_state(m, seed=60 + i) for i, m in enumerate(models)]
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)  # about 10 ms in front of the copies
    for i, state in enumerate(want):
        part = [a[:3 * models[i].num_nodes] for a in stage]
        for a, src in zip(part, state):
            a[:] = src
        b.upload(i, *part)
        for a in part:
            a[:] = -1.0
    for i, state in enumerate(want):
        assert all(np.array_equal(a, src) for a, src in zip(b.download(i), state))


def _disk_loop(workdir, name, precision=0, path=None):
    from morphoshell_b200 import GpuLoop
    from conftest import make_model
    m = make_model(workdir, name)
    g = GpuLoop(m, precision=precision)
    a, b = m.programmed()
    g.set_programmed(3, a, b, m.scalars.dial_factors_to_hold_at_spacing)
    if path is not None:
        g.set_step_path(path)
    g.upload(*deformed_state(m, seed=61, amp=0.02))
    return m, g


def _steps(m, g, n=20):
    s = m.scalars
    g.step_n(n, 0.2 + 1e-5 * np.arange(n), s.timestep, s.damping_factor_1)
    g.do_dialling(0.3)
    g.step_n(n, None, s.timestep, s.damping_factor_2)
    return g.download()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("path", [3, 4])
def test_larger_mesh_steps_after_a_smaller_one_is_created(workdir, monkeypatch, path, precision):
    """A kernel's shared-memory limit belongs to the process: creating a handle
    whose tiles need less must not take it from one whose tiles need more."""
    if path == 4:
        monkeypatch.setenv("MSB_NODE_TILE_PLAN", "4")
    m, big = _disk_loop(workdir, "disk5", precision, path)
    want = _steps(m, _disk_loop(workdir, "disk5", precision, 2)[1])
    _, small = _disk_loop(workdir, "disk14", precision, path)
    assert small.plan_info()["nodes_per_tile"] < big.plan_info()["nodes_per_tile"]
    assert all(np.array_equal(a, b) for a, b in zip(_steps(m, big), want))


@pytest.mark.parametrize("precision", [0, 1])
def test_larger_batch_steps_after_a_smaller_one_is_created(tmp_path, precision):
    """The same for the batch's node-tiled schedule, in graphs (events) and in
    quiet stretches."""
    from morphoshell_b200 import Batch, ensemble
    big_m, _ = ensemble.build_members([3, 5], str(tmp_path / "big"), spacing_range=(0.006, 0.0061), threads=4)
    small_m, _ = ensemble.build_members([0, 1], str(tmp_path / "small"), spacing_range=(0.05, 0.1), threads=4)
    big, ref = Batch(big_m, precision=precision), Batch(big_m, precision=precision)
    big.set_schedule(-1, 0, 4)
    ref.set_schedule(0, 256, 4)
    small = Batch(small_m, precision=precision)
    assert small.schedule()["nodes_per_tile"] < big.schedule()["nodes_per_tile"]
    for steps in (4, 20):
        assert big.run(steps) == ref.run(steps) == steps
    for i in range(2):
        assert all(np.array_equal(a, b) for a, b in zip(big.download(i), ref.download(i)))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("big,small", [("disk15", "disk16"), ("disk6", "disk14")])
def test_threads_step_meshes_of_different_size(workdir, big, small, precision):
    """Host threads, a handle each, whose launches are of one kernel and need
    different amounts of shared memory: the bits of each alone."""
    import threading
    got, errors = {}, []

    def work(key, m, g):
        s = m.scalars
        lengths = np.random.default_rng(62).integers(2, 12, 3000)
        try:
            for n in lengths:
                g.step_n(int(n), None, s.timestep, s.damping_factor_2)
            got[key] = g.download()
        except Exception as e:  # noqa: BLE001
            errors.append((key, e))

    for name in (big, small):
        work(name, *_disk_loop(workdir, name, precision))
    assert not errors, errors
    loops = [(0, *_disk_loop(workdir, big, precision))]
    loops += [(k, *_disk_loop(workdir, small, precision)) for k in (1, 2, 3)]
    threads = [threading.Thread(target=work, args=x) for x in loops]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(4):
        assert all(np.array_equal(a, b) for a, b in zip(got[k], got[small if k else big]))
