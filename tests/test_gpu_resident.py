"""The resident step kernel (the engine's own choice for grids whose state fits
in shared memory) gives the plain kernel's bits: every expression is the same
with the same rounding, so records and DFT are compared for equality."""
import threading

import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from test_gpu_edge_cases import _random_sim

pytestmark = pytest.mark.gpu


def _model_sim(s):
    co, pr, mo, mem, Nx, Ny, Nz, Nt = s.pack_inputs(gpu=True)
    sim = _lib.Simulation(Nx, Ny, Nz)
    sim.set_coefficients(co)
    for p in pr:
        sim.add_probe(p["field"], p["idx"], p["is_source"], p["values"][:Nt] if p["is_source"] else None)
    sim.set_dft([(k % 3, k, 1.0 + k) for k in range(len(pr))], np.linspace(0.01, 0.4, 7))
    return sim, Nt


def _both(make, nt):
    """(records, DFT or None) of the engine's choice and of the plain kernel."""
    out = []
    for plain in (False, True):
        sim = make()
        if plain:
            sim.set_kernel(0)
        sim.run(nt)
        if not plain:
            assert sim.stats()["variant"] == 2 and sim.stats()["step_launches"] == nt
        out.append((sim.probe_values(), sim.dft() if sim.n_series else None))
        sim.close()
    return out


# one cell per brick and fewer bricks than cells; one brick; long thin grids;
# rows that stay in global memory (random coefficients: two Db per split)
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 2), (149, 3, 2), (2, 3, 151), (33, 9, 5), (31, 37, 27)])
def test_random_grids_equal_plain(engine_lib, shape):
    (a, _), (b, _) = _both(lambda: _random_sim(shape, 4, 50, 1, tile_y=0), 50)
    assert np.abs(b).max() > 0 and np.array_equal(a, b)


# absorbing layers thicker and thinner than a brick, a graded mesh, more table
# rows than the bricks' local tables hold, no layers at all
@pytest.mark.parametrize("model", [
    lambda: configs.microstrip(n=(64, 64, 48), n_pml=10, nt=300),
    lambda: configs.microstrip(n=(52, 44, 33), n_pml=3, nt=200, graded=True),
    lambda: configs.boxes(n=(97, 60, 51), n_pml=12, n_boxes=8, nt=120, n_ports=2, n_probes=6),
    lambda: configs.boxes(n=(100, 90, 70), n_pml=0, n_boxes=8, nt=100, n_ports=2, n_probes=6),
])
def test_models_equal_plain(engine_lib, model):
    s = model()
    nt = s.pack_inputs(gpu=True)[-1]
    (a, X), (b, Y) = _both(lambda: _model_sim(s)[0], nt)
    assert np.abs(b).max() > 0 and np.array_equal(a, b) and np.array_equal(X, Y)


def test_more_steps_than_one_launch(engine_lib):
    s = configs.microstrip(n=(18, 16, 14), n_pml=3, nt=4096 + 300)
    (a, X), (b, Y) = _both(lambda: _model_sim(s)[0], 4096 + 300)
    assert np.abs(b).max() > 0 and np.array_equal(a, b) and np.array_equal(X, Y)


def test_two_threads(engine_lib):
    """Two simulations stepped by two threads at the same time: each launch
    needs every SM, so they take turns, and both give their own bits."""
    models = [configs.microstrip(n=(40 + 8 * k, 36, 30), n_pml=5, nt=1500) for k in range(2)]
    want = []
    for s in models:
        sim, nt = _model_sim(s)
        sim.run(nt)
        want.append(sim.probe_values())
        sim.close()
    got = [[], []]
    errors = []

    def work(k):
        try:
            sim, nt = _model_sim(models[k])
            for _ in range(6):
                sim.run(nt)
                got[k].append(sim.probe_values())
            sim.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2):
        assert len(got[k]) == 6 and all(np.array_equal(g, want[k]) for g in got[k])


@pytest.mark.parametrize("step", [0, 7, 39])
def test_expired_wait_reports_device_error_and_the_handle_recovers(engine_lib, step):
    """One brick sends no faces in one step: the waits for them run out after a few
    hundred polls, every block ends, and the same handle runs normally again."""
    sim, nt = _model_sim(configs.microstrip(n=(40, 30, 24), n_pml=4, nt=40))
    sim.run(nt)
    ref, X = sim.probe_values(), sim.dft()
    assert sim.stats()["variant"] == 2 and sim.stats()["grid"] > 1 and np.abs(ref).max() > 0
    for _ in range(2):
        sim.set_debug(wait_limit=200, withhold_plane=step)
        with pytest.raises(_lib.FdtdError, match="resident step kernel gave up waiting") as e:
            sim.run(nt)
        assert e.value.code == 5  # FDTD_ERR_DEVICE
        sim.set_debug()
        for _ in range(2):
            sim.run(nt)
            assert np.array_equal(sim.probe_values(), ref) and np.array_equal(sim.dft(), X)
    sim.close()


def test_partition_follows_the_run(engine_lib):
    """A batch of one member is stepped by the resident kernel in a plain run
    and by the streaming kernels when the run records a gradient's history."""
    s = configs.microstrip(n=(30, 26, 22), n_pml=4, nt=120)
    sim, nt = _model_sim(s)
    batch = _lib.Batch([sim])
    batch.run(nt)
    a, X = sim.probe_values(), sim.dft()
    assert batch.stats()["variant"] == 2
    batch.run_recorded(nt, [(12, 16, 8, 12, 8, 10)])
    assert np.array_equal(sim.probe_values(), a) and np.array_equal(sim.dft(), X)
    batch.run(nt)
    assert np.array_equal(sim.probe_values(), a) and np.array_equal(sim.dft(), X)
    batch.close()
    sim.close()


# time samples and phasors, sampled every step and every third, on planes at the
# grid's ends and inside, of split (layer) and unsplit cells
@pytest.mark.parametrize("shape,n_pml", [((34, 30, 26), 4), ((3, 6, 4), 0)])
def test_monitors_equal_plain(engine_lib, shape, n_pml):
    nt = 50
    phase = np.exp(-1j * 0.2 * np.arange(nt + 1)[:, None] * np.arange(1, 4)[None]).astype(np.complex64)

    def make():
        if n_pml:
            sim, _ = _model_sim(configs.microstrip(n=shape, n_pml=n_pml, nt=nt))
        else:
            sim = _random_sim(shape, 8, nt, 1, tile_y=0)
        for axis in range(3):
            for field in range(6):
                for k, pos in enumerate((1, shape[axis] // 2, shape[axis] - 1)):
                    if (field + k) % 2:
                        sim.add_monitor(field, axis, pos, 1 + 2 * (k == 1), phase=phase)
                    elif k == 1:
                        sim.add_monitor(field, axis, pos, 3)
        return sim

    out = []
    for plain in (False, True):
        sim = make()
        if plain:
            sim.set_kernel(0)
        sim.run(nt)
        assert plain or sim.stats()["variant"] == 2
        out.append([sim.monitor(m) for m in range(len(sim.monitors))])
        sim.close()
    assert any(np.abs(b).max() > 0 for b in out[1])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
