"""Handles used by several threads at the same time: what one thread builds, captures
or releases must not disturb the runs of another."""
import threading

import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu

NT = 60
# grids for the streaming and half-step kernels, tuned here for the first time
SIZES = [[(112, 104, 96), (128, 100, 90)], [(120, 110, 95), (116, 99, 104)], [(126, 104, 91), (110, 110, 99)]]


def _work(model, n):
    """Plain, recorded and checkpointed runs, each from the host and as a graph."""
    box = (n[0] // 2 - 4, n[0] // 2 + 4, n[1] // 2 - 3, n[1] // 2 + 3, 12, 14)
    sim, _ = _model_sim(model)
    out = []
    for _ in range(3):
        sim.run(NT)
    out.append(sim.probe_values())
    for run in (lambda: sim.run_recorded(NT, box), lambda: sim.run_checkpointed(NT, 16)):
        for _ in range(2):
            run()
            out.append(sim.adjoint(2 * sim.dft(), box))
        out.append(sim.probe_values())
    sim.close()
    return out


def _check(got, models):
    for n, model in models.items():
        want = _work(model, n)
        assert all(np.abs(w).max() > 0 for w in want)
        assert len(got[n]) == len(want) and all(map(np.array_equal, got[n], want)), n


def _run(jobs):
    errors = []

    def guarded(f):
        def g():
            try:
                f()
            except Exception as e:  # noqa: BLE001
                errors.append(e)
        return g

    threads = [threading.Thread(target=guarded(f)) for f in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_threads_that_tune_capture_and_release(engine_lib):
    models = {n: configs.microstrip(n=n, n_pml=8, nt=NT) for group in SIZES for n in group}
    small = configs.microstrip(n=(20, 18, 16), n_pml=3, nt=NT)
    got, busy = {}, [True]

    def group(k):
        for n in SIZES[k]:
            got[n] = _work(models[n], n)

    def churn():  # makes and releases buffers all the while
        for _ in range(300):
            if not busy[0]:
                break
            sim, _ = _model_sim(small)
            sim.run(NT)
            sim.close()

    def all_groups():
        try:
            _run([lambda k=k: group(k) for k in range(3)])
        finally:
            busy[0] = False

    _run([all_groups, churn])
    _check(got, models)
