"""What the autotuner remembers: a choice holds for grids of the same sizes with the
same work beside the steps, since the step kernels differ in what that costs them."""
import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu

NT = 40
N = (61, 47, 35)  # (a size of no other test: choices are remembered for the process)
BOX = (24, 36, 18, 28, 15, 19)
PHASE = np.exp(-0.1j * np.arange(NT + 1)[:, None] * np.arange(1, 3)[None]).astype(np.complex64)


def _run(kind, monitors):
    sim, _ = _model_sim(configs.microstrip(n=N, n_pml=5, nt=NT))
    for axis in range(3):
        for field in range(6 if monitors else 0):
            sim.add_monitor(field, axis, N[axis] // 2, 1, phase=PHASE)
    batch = _lib.Batch([sim]) if kind == "batch" else None
    if batch:
        batch.run_recorded(NT, [BOX])
    elif kind == "recorded":
        sim.run_recorded(NT, BOX)
    else:
        sim.run(NT)
    trials = (batch or sim).stats()["tune_trials"]
    out = [sim.probe_values()] + [sim.monitor(m) for m in range(len(sim.monitors))]
    if batch:
        batch.close()
    sim.close()
    return trials, out


def test_choices_are_for_the_same_work(engine_lib):
    rec = None
    for kind in ("run", "recorded"):
        for monitors in (False, True):
            trials, out = _run(kind, monitors)
            assert trials > 0, (kind, monitors)
            again, same = _run(kind, monitors)
            assert again == 0 and all(map(np.array_equal, out, same))
            rec = out[0] if rec is None else rec
            assert np.abs(rec).max() > 0 and np.array_equal(out[0], rec)
            assert all(np.abs(m).max() > 0 for m in out[1:])
            if kind == "run":
                plain = out[1:]
        assert all(map(np.array_equal, out[1:], plain))
    assert _run("batch", True)[0] == 0  # (a batch of one is the same work)


@pytest.mark.parametrize("members", [1, 3])
def test_tuning_after_a_recorded_run(engine_lib, members):
    """A batch keeps its engines from a recorded run to a plain one of a size that is
    tuned there for the first time."""
    n = (33 + members, 31, 27)
    sims = [_model_sim(configs.microstrip(n=n, n_pml=4, nt=NT))[0] for _ in range(members)]
    batch = _lib.Batch(sims)
    out = []
    for _ in range(2):
        batch.run_recorded(NT, [(14, 18, 10, 16, 12, 14)] * members)
        out.append([sim.probe_values() for sim in sims])
        grads = batch.adjoint([2 * sim.dft() for sim in sims])
        assert all(np.abs(g).max() > 0 and np.array_equal(g, grads[0]) for g in grads)
        batch.run(NT)
        out.append([sim.probe_values() for sim in sims])
    assert all(np.abs(r).max() > 0 and np.array_equal(r, out[0][0]) for recs in out for r in recs)
    batch.close()
    for sim in sims:
        sim.close()


def test_tuning_takes_a_few_hundred_steps(engine_lib):
    """A first call on a size that no tuned one shares pays for the trials: the time of
    300 to 350 steps of these grids, and of 680 to 760 when every trial made its index
    of the split cells anew and ran more steps. The bound lies between."""
    cost = []
    for n in ((200, 180, 128), (202, 178, 127), (198, 182, 129)):
        co, pr, mo, mem, Nx, Ny, Nz, Nt = configs.boxes(n=n, n_pml=8, n_boxes=8, nt=100, n_ports=2,
                                                        n_probes=4).pack_inputs(gpu=True)
        sim = _lib.Simulation(Nx, Ny, Nz)
        sim.set_coefficients(co, borrow=True)
        for p in pr:
            sim.add_probe(p["field"], p["idx"], p["is_source"], p["values"][:Nt] if p["is_source"] else None)
        sim.run(Nt)
        st = sim.stats()
        assert st["tune_trials"] > 10
        for _ in range(2):
            sim.run(Nt)
        cost.append(st["tune_ms"] / (sim.stats()["last_run_ms"] / Nt))
        sim.close()
    assert min(cost) < 520, cost
