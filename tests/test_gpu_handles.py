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
