"""The gradient's way from the device's order (x fastest) to the caller's (z fastest)."""
import time

import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from rfnetwork_b200.solver_constants import COEFF_NAMES

pytestmark = pytest.mark.gpu


def _sim(n, nt):
    co, pr, mo, mem, Nx, Ny, Nz, Nt = configs.boxes(n=n, n_pml=6, n_boxes=8, nt=nt, n_ports=2,
                                                    n_probes=4).pack_inputs(gpu=True)
    sim = _lib.Simulation(Nx, Ny, Nz)
    sim.set_coefficients(co)
    for p in pr:
        sim.add_probe(p["field"], p["idx"], p["is_source"], p["values"][:Nt] if p["is_source"] else None)
    sim.set_dft([(k % 3, k, 1.0) for k in range(len(pr))], np.linspace(0.01, 0.4, 7))
    return sim, np.array([p["idx"] for p in pr if p["is_source"]])


def _free(sources, want, n):
    """A box of `want` cells without source cells, outside the absorbing layers."""
    for x in range(8, n[0] - 8 - want[0], 3):
        for y in range(8, n[1] - 8 - want[1], 3):
            for z in range(8, n[2] - 8 - want[2], 3):
                lo, hi = np.array((x, y, z)), np.array((x, y, z)) + want
                if not ((sources >= lo - 2) & (sources < hi + 2)).all(axis=1).any():
                    return (x, x + want[0], y, y + want[1], z, z + want[2])
    raise AssertionError("no free box")


def test_parts_of_a_box(engine_lib):
    """A cell's gradient does not depend on the box around it: boxes of one cell, of a
    tile (32) and one cell more and less along x and z are the same bits as their part
    of a large one. (The arrays are turned at once, or three by three when the box is
    larger than a third of the grid.)"""
    n, nt = (96, 90, 88), 240
    sim, sources = _sim(n, nt)
    big = _free(sources, (67, 24, 66), n)
    sim.run_recorded(nt, big)
    dJ = 2 * sim.dft()
    want = sim.adjoint(dJ, big)
    assert np.abs(want).max() > 0 and (np.abs(want) > 0).mean() > 0.5
    for size in ((1, 1, 1), (32, 3, 32), (31, 1, 33), (33, 5, 31), (64, 2, 1), (1, 24, 66), (67, 7, 65)):
        o = (1 if size[0] < 67 else 0, 24 - size[1], 66 - size[2])
        box = tuple(big[2 * a] + o[a] + (size[a] if hi else 0) for a in range(3) for hi in (0, 1))
        sim.run_recorded(nt, box)
        got = sim.adjoint(dJ, box)
        part = want[:, :, o[0]:o[0] + size[0], o[1]:o[1] + size[1], o[2]:o[2] + size[2]]
        assert np.array_equal(got, part), size
    sim.close()


def test_large_boxes_cost_the_host_a_copy(engine_lib):
    """The call's host part for 320,000 cells (23 MB) was three times the sweep's 4 ms
    when the host turned the arrays; a copy is half of it."""
    n, nt = (128, 128, 96), 40
    sim, sources = _sim(n, nt)
    box = _free(sources, (80, 80, 50), n)
    rest = []
    for _ in range(6):
        sim.run_checkpointed(nt, 8)
        g = 2 * sim.dft()
        t0 = time.perf_counter()
        sim.adjoint(g, box)
        wall = (time.perf_counter() - t0) * 1e3
        rest.append((wall - sim.stats()["adjoint_ms"]) / sim.stats()["adjoint_ms"])
    sim.close()
    assert sorted(rest)[2] < 1.2, rest


def test_a_box_of_most_of_the_grid(engine_lib):
    """The box fills more than a third of the grid: the same bits as a part of it by
    itself."""
    n, nt = (24, 26, 30), 50
    rng = np.random.default_rng(7)
    sim = _lib.Simulation(*n)
    for name in COEFF_NAMES:
        a = np.full(n, 0.97) if name[0] + name[1] in ("Ca", "Da") else np.full(n, 0.3)
        sim.set_coefficient(name, a.astype(np.float32))
    sim.add_probe(2, (12, 2, 14), True, rng.standard_normal(nt).astype(np.float32))
    sim.add_probe(2, (12, 23, 14))
    sim.set_dft([(0, 1, 1.0)], [0.1, 0.3])
    big = (1, 23, 4, 25, 1, 29)
    sim.run_recorded(nt, big)
    dJ = 2 * sim.dft()
    want = sim.adjoint(dJ, big)
    assert (np.abs(want) > 0).mean() > 0.5
    box = (3, 4, 6, 20, 2, 29)
    sim.run_recorded(nt, box)
    assert np.array_equal(sim.adjoint(dJ, box), want[:, :, 2:3, 2:16, 1:28])
    sim.close()
