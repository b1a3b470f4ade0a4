"""A batch steps its large members one after the other and its small ones
together; each member keeps the bits of its own run either way."""
import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu

NT = 60
SMALL, MID, LARGE = (20, 18, 16), (40, 36, 34), (74, 64, 56)  # 6k, 49k and 265k cells
BOXES = {SMALL: (8, 11, 6, 10, 5, 7), MID: (16, 24, 14, 20, 9, 11), LARGE: (30, 40, 28, 36, 12, 14)}


@pytest.mark.parametrize("members", [
    [SMALL], [SMALL] * 2, [SMALL] * 3, [MID, SMALL, LARGE, SMALL, SMALL], [LARGE, MID], [MID] * 3 + [LARGE] * 2])
def test_members_keep_their_bits(engine_lib, members):
    single = {}
    for n in set(members):
        m = configs.microstrip(n=n, n_pml=3, nt=NT)
        sim, _ = _model_sim(m)
        sim.run(NT)
        rec = sim.probe_values()
        sim.run_recorded(NT, BOXES[n])
        single[n] = (m, rec, sim.adjoint(2 * sim.dft(), BOXES[n]))
        sim.close()
    sims = [_model_sim(single[n][0])[0] for n in members]
    batch = _lib.Batch(sims)
    boxes = [BOXES[n] for n in members]
    for kind in ("run", "recorded", "checkpointed", "run"):
        if kind == "run":
            batch.run(NT)
        elif kind == "recorded":
            batch.run_recorded(NT, boxes)
        else:
            batch.run_checkpointed(NT, 16, boxes)
        for n, sim in zip(members, sims):
            assert np.abs(single[n][1]).max() > 0 and np.array_equal(sim.probe_values(), single[n][1])
        assert batch.stats()["step_launches"] == NT
        if kind != "run":
            grads = batch.adjoint([2 * sim.dft() for sim in sims])
            assert batch.stats()["adjoint_launches"] == NT
            for n, g in zip(members, grads):
                assert np.abs(g).max() > 0 and np.array_equal(g, single[n][2])
    batch.close()
    for sim in sims:
        sim.close()


@pytest.mark.parametrize("members,together", [
    ([SMALL] * 2, False), ([SMALL] * 3, True), ([MID] * 2, False), ([MID] * 3, True), ([MID] * 8, True),
    ([(46, 40, 33)] * 4, False), ([(46, 40, 33)] * 5, True), ([(52, 44, 37)] * 5, False), ([(52, 44, 37)] * 6, True),
    ([LARGE] * 6, False), ([MID, (52, 44, 37)] * 3 + [LARGE], True)])
def test_the_more_the_larger(engine_lib, members, together):
    """Members of 50k to 90k cells are stepped together only where they are many: the
    first part's kernel is the resident one where each is stepped alone."""
    models = {n: _model_sim(configs.microstrip(n=n, n_pml=3, nt=NT)) for n in set(members)}
    want = {}
    for n, (sim, _) in models.items():
        sim.run(NT)
        want[n] = sim.probe_values()
        sim.close()
    sims = [_model_sim(configs.microstrip(n=n, n_pml=3, nt=NT))[0] for n in members]
    batch = _lib.Batch(sims)
    batch.run(NT)
    tiles = batch.stats()["n_tiles"]
    alone = 0
    for n, sim in zip(members, sims):
        assert np.abs(want[n]).max() > 0 and np.array_equal(sim.probe_values(), want[n])
        sim.run(NT)
        assert sim.stats()["variant"] == 2
        alone += sim.stats()["n_tiles"]
    assert (tiles != alone) == together
    batch.close()
    for sim in sims:
        sim.close()


def test_largest_members_of_a_gradient_share_launches(engine_lib):
    """Two members whose reverse step does not fit in L2: their adjoints together took
    35 ms against 41 one after the other; each keeps the bits of its own."""
    n, nt, box = (200, 180, 128), 60, (100, 116, 150, 166, 53, 57)
    m = configs.boxes(n=n, n_pml=0, n_boxes=8, nt=nt, n_ports=2, n_probes=4)
    packed = m.pack_inputs(gpu=True)
    small = _model_sim(configs.microstrip(n=SMALL, n_pml=3, nt=nt))[0]

    def make():
        sim = _lib.Simulation(*n)
        sim.set_coefficients(packed[0], borrow=True)
        for p in packed[1]:
            sim.add_probe(p["field"], p["idx"], p["is_source"], p["values"][:nt] if p["is_source"] else None)
        sim.set_dft([(k % 3, k, 1.0) for k in range(len(packed[1]))], np.linspace(0.01, 0.4, 7))
        return sim

    sims = [make(), make()]
    alone, grads = [], []
    for sim in sims:
        for _ in range(3):
            sim.run_recorded(nt, box)
            g = sim.adjoint(2 * sim.dft(), box)
        alone.append(sim.stats()["adjoint_ms"])
        grads.append(g)
    assert np.abs(grads[0]).max() > 0
    members = [sims[0], small, sims[1]]
    batch = _lib.Batch(members)
    for _ in range(3):
        batch.run_recorded(nt, [box, BOXES[SMALL], box])
        got = batch.adjoint([2 * sim.dft() for sim in members])
    together = batch.stats()["adjoint_ms"]
    assert np.array_equal(got[0], grads[0]) and np.array_equal(got[2], grads[1])
    small.run_recorded(nt, BOXES[SMALL])
    assert np.array_equal(got[1], small.adjoint(2 * small.dft(), BOXES[SMALL]))
    # (the small member's own part adds its 0.5 ms)
    assert together - small.stats()["adjoint_ms"] < 0.93 * sum(alone), (together, alone)
    batch.close()
    for sim in members:
        sim.close()
