"""The far-field transform over the ways its cells are cut into parts: one part
(a pattern that fills the GPU by itself), many, the last one short, one cell.
Tolerance as in test_farfield.py: FP32 phases up to ~10 rad (rounding about
1e-6 rad) and FP32 products summed in FP64, 1e-5 relative L2."""
import numpy as np
import pytest

from helpers import rel_l2
from oracle import nf2ff as nf2ff_oracle
from rfnetwork_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,F,n_theta,n_phi", [
    ((2, 2, 2), 1, 400, 400),     # 1250 direction blocks: one part
    ((1, 1, 1), 3, 1, 1),         # six cells, one direction
    ((9, 7, 5), 2, 3, 43),        # 129 directions, 286 cells: three parts, the last one short
    ((24, 20, 16), 1, 7, 19),     # one block of directions, eighteen parts
    ((40, 1, 33), 2, 13, 9),      # faces of very different size
])
def test_parts_match_oracle(engine_lib, n, F, n_theta, n_phi):
    rng = np.random.default_rng(sum(n) + F)
    w = 1e-3
    J, M, r, ds, pos = [], [], [], [], []
    for axis in range(3):
        f0, f1 = [a for a in range(3) if a != axis]
        r.append([np.ascontiguousarray(v, np.float32) for v in np.meshgrid(
            (np.arange(n[f0]) - n[f0] / 2) * w, (np.arange(n[f1]) - n[f1] / 2) * w, indexing="ij")])
        ds.append(rng.uniform(0.5, 1.5, (n[f0], n[f1])).astype(np.float32) * np.complex64(w * w))
        pos.append([-n[axis] * w / 2, n[axis] * w / 2])
        shape = (3, F, n[f0], n[f1])
        for X, scale in ((J, 1.0), (M, 377.0)):
            X.append([(scale * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))).astype(np.complex64)
                      for _ in range(2)])

    def data():
        return dict(beta=np.linspace(150, 400, F).astype(np.float32),
                    theta=np.linspace(0.1, 3.0, n_theta).astype(np.float32),
                    phi=np.linspace(-3.0, 3.1, n_phi).astype(np.float32),
                    data=np.zeros((2, F, n_theta, n_phi), dtype=np.complex64))

    ref, gpu = data(), data()
    nf2ff_oracle.nf2ff(J, M, r, ds, pos, ref)
    _lib.nf2ff(J, M, r, ds, pos, gpu)
    assert rel_l2(gpu["data"], ref["data"]) <= 1e-5
