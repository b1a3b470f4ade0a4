"""Grids that the resident kernel cuts into thinner bricks in their absorbing
layers (the first fits in shared memory only so), and grids part of whose split
pairs stay in global memory (the last two), give the plain kernel's bits."""
import numpy as np
import pytest

from modelgen import configs
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_pml", [((133, 44, 88), 8), ((55, 140, 47), 8), ((41, 54, 143), 8), ((64, 40, 36), 12),
                                     ((120, 100, 64), 8), ((139, 49, 93), 8)])
def test_equals_plain(engine_lib, n, n_pml):
    s = configs.boxes(n=n, n_pml=n_pml, n_boxes=4, nt=70, n_ports=1, n_probes=4)
    phase = np.exp(-0.1j * np.arange(71)[:, None] * np.arange(1, 3)[None]).astype(np.complex64)
    got = []
    for plain in (False, True):
        sim, nt = _model_sim(s)
        if n[0] in (55, 120):
            sim.add_monitor(1, 0, n[0] // 2, 2, phase=phase)
        if plain:
            sim.set_kernel(0)
        sim.run(nt)
        assert plain or sim.stats()["variant"] == 2
        got.append([sim.probe_values(), sim.dft()] + [sim.monitor(m) for m in range(len(sim.monitors))])
        sim.close()
    assert np.abs(got[1][0]).max() > 0
    assert all(np.array_equal(a, b) for a, b in zip(*got))
