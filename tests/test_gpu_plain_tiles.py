"""Grids without absorbing layers, whose tiles are almost all plain, give the
plain kernel's bits at every tile height of the streaming kernels."""
import numpy as np
import pytest

from modelgen import configs
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(94, 62, 41), (70, 97, 33)])
@pytest.mark.parametrize("tile_y", [4, 6, 8, 12])
def test_streaming_equals_plain(engine_lib, n, tile_y):
    s = configs.boxes(n=n, n_pml=0, n_boxes=4, nt=60, n_ports=1, n_probes=3)
    got = []
    for kernel in ((1, tile_y, 6, 0), (0, 0, 4, 0)):
        sim, nt = _model_sim(s)
        sim.set_kernel(*kernel)
        sim.run(nt)
        got.append((sim.probe_values(), sim.dft()))
        sim.close()
    assert np.abs(got[1][0]).max() > 0
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
