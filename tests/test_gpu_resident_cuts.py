"""Grids that the resident kernel cuts into thinner bricks in their absorbing
layers (the first fits in shared memory only so) give the plain kernel's bits."""
import numpy as np
import pytest

from modelgen import configs
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_pml", [((133, 44, 88), 8), ((55, 140, 47), 8), ((41, 54, 143), 8), ((64, 40, 36), 12)])
def test_equals_plain(engine_lib, n, n_pml):
    s = configs.boxes(n=n, n_pml=n_pml, n_boxes=4, nt=70, n_ports=1, n_probes=4)
    got = []
    for plain in (False, True):
        sim, nt = _model_sim(s)
        if plain:
            sim.set_kernel(0)
        sim.run(nt)
        assert plain or sim.stats()["variant"] == 2
        got.append((sim.probe_values(), sim.dft()))
        sim.close()
    assert np.abs(got[1][0]).max() > 0
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
