"""The half-step kernels (one of the engine's own choices for grids that do not
fit in shared memory; RFN_FDTD_KERNEL=half asks for them) give the plain
kernel's bits in runs, batches and gradients."""
import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from test_gpu_edge_cases import _random_sim
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu


def _pair(make, nt, monkeypatch, run=None):
    out = []
    for kernel in ("half", "plain"):
        monkeypatch.setenv("RFN_FDTD_KERNEL", kernel)
        sim = make()
        if run:
            out.append(run(sim))
        else:
            sim.run(nt)
            out.append((sim.probe_values(), [sim.monitor(m) for m in range(len(sim.monitors))]))
        assert sim.stats()["variant"] == (3 if kernel == "half" else 0)
        sim.close()
    return out


# rows shorter and longer than a block, several rows per block, ragged ends
@pytest.mark.parametrize("n,n_pml", [((18, 16, 14), 3), ((33, 29, 17), 4), ((70, 45, 38), 6), ((290, 20, 18), 3)])
@pytest.mark.parametrize("threads", ["64", "128", "256"])
def test_models_equal_plain(engine_lib, monkeypatch, n, n_pml, threads):
    monkeypatch.setenv("RFN_FDTD_TY", threads)
    nt = 90
    if n[0] < 290:
        s = configs.microstrip(n=n, n_pml=n_pml, nt=nt, graded=n[0] == 33)
    else:
        s = configs.boxes(n=n, n_pml=n_pml, n_boxes=3, nt=nt, n_ports=1, n_probes=3)
    phase = np.exp(-0.1j * np.arange(nt + 1)[:, None] * np.arange(1, 3)[None]).astype(np.complex64)

    def make():
        sim, _ = _model_sim(s)
        sim.add_monitor(0, 2, n[2] // 2, 1, phase=phase)
        sim.add_monitor(4, 0, n[0] // 2, 4)
        return sim

    (a, ma), (b, mb) = _pair(make, nt, monkeypatch)
    assert np.abs(b).max() > 0 and np.array_equal(a, b)
    assert all(np.array_equal(x, y) for x, y in zip(ma, mb))


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 2), (64, 9, 40), (257, 3, 5)])
def test_random_grids_equal_plain(engine_lib, monkeypatch, shape):
    got = []
    for kernel in ("half", "plain"):
        monkeypatch.setenv("RFN_FDTD_KERNEL", kernel)
        monkeypatch.setattr(_lib.Simulation, "set_kernel", lambda self, *a, **k: None)
        sim = _random_sim(shape, 11, 30, 0)
        sim.run(30)
        assert sim.stats()["variant"] == (3 if kernel == "half" else 0)
        got.append(sim.probe_values())
        sim.close()
    assert np.array_equal(*got)


def test_batch_equals_single_runs(engine_lib, monkeypatch):
    nt = 60
    models = [configs.batch_member(3, i, nt=nt, size_range=(20, 70), n_pml=4) for i in range(4)]
    monkeypatch.setenv("RFN_FDTD_KERNEL", "plain")
    want = []
    for s in models:
        sim, _ = _model_sim(s)
        sim.run(nt)
        want.append(sim.probe_values())
        sim.close()
    monkeypatch.setenv("RFN_FDTD_KERNEL", "half")
    sims = [_model_sim(s)[0] for s in models]
    batch = _lib.Batch(sims)
    batch.run(nt)
    assert batch.stats()["variant"] == 3
    for sim, w in zip(sims, want):
        assert np.array_equal(sim.probe_values(), w)
    batch.close()


@pytest.mark.parametrize("mode", ["recorded", "checkpointed", "checkpointed, whole grid"])
def test_gradients_equal_plain(engine_lib, monkeypatch, mode):
    """Histories written by the E launches, segment replays of the cells within
    reach of the box and the half-step reverse, against a plain-kernel run of the
    same mode and the reverse step in one launch."""
    s = configs.microstrip(n=(58, 44, 30), n_pml=5, nt=130)
    box = (24, 33, 18, 26, 12, 15)
    if mode.endswith("grid"):
        monkeypatch.setenv("RFN_REPLAY_FULL", "1")

    halves = iter(("1", "0"))

    def run(sim):
        monkeypatch.setenv("RFN_ADJ_HALF", next(halves))
        if mode == "recorded":
            sim.run_recorded(130, box)
        else:
            sim.run_checkpointed(130, 24)
        rec, X = sim.probe_values(), sim.dft()
        g = sim.adjoint(2 * X, box)
        assert np.array_equal(sim.probe_values(), rec)
        return rec, X, g

    a, b = _pair(lambda: _model_sim(s)[0], 130, monkeypatch, run)
    assert np.abs(b[2]).max() > 0
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


# more threads per block than the kernels take, and a size that is no multiple of a
# warp: replayed regions wide enough to use them all
@pytest.mark.parametrize("threads", ["512", "100"])
def test_replays_of_any_block_size(engine_lib, monkeypatch, threads):
    monkeypatch.setenv("RFN_FDTD_TY", threads)
    test_gradients_equal_plain(engine_lib, monkeypatch, "checkpointed")


def test_batched_gradients_equal_single(engine_lib, monkeypatch):
    models = [configs.microstrip(n=(40, 30, 24), n_pml=4, nt=90), configs.microstrip(n=(46, 34, 22), n_pml=4, nt=90)]
    boxes = [(16, 22, 12, 17, 9, 11), (18, 24, 14, 20, 9, 12)]
    out = {}
    for kernel in ("half", "plain"):
        monkeypatch.setenv("RFN_FDTD_KERNEL", kernel)
        monkeypatch.setenv("RFN_ADJ_HALF", "1" if kernel == "half" else "0")
        sims = [_model_sim(s)[0] for s in models]
        b = _lib.Batch(sims)
        for mode in ("recorded", "checkpointed"):
            if mode == "recorded":
                b.run_recorded(90, boxes)
            else:
                b.run_checkpointed(90, 17, boxes)
            Xs = [sim.dft() for sim in sims]
            out[kernel, mode] = Xs + b.adjoint([2 * X for X in Xs])
        b.close()
        for sim in sims:
            sim.close()
    want = out["plain", "recorded"]
    assert all(np.abs(w).max() > 0 for w in want)
    for got in out.values():
        assert all(np.array_equal(x, y) for x, y in zip(got, want))


# grids large enough for two and four cells per thread along z, with a remainder
@pytest.mark.parametrize("sizes", [[(90, 80, 59)], [(120, 110, 77)], [(90, 80, 59), (92, 70, 61)]])
def test_gradients_of_deep_columns(engine_lib, monkeypatch, sizes):
    nt, out = 50, []
    models = [configs.microstrip(n=n, n_pml=5, nt=nt) for n in sizes]
    boxes = [(n[0] // 2 - 4, n[0] // 2 + 5, n[1] // 2 - 3, n[1] // 2 + 6, 8, 12) for n in sizes]
    monkeypatch.setenv("RFN_FDTD_KERNEL", "half")  # (members of a batch step together)
    for half in ("1", "0"):
        monkeypatch.setenv("RFN_ADJ_HALF", half)
        sims = [_model_sim(s)[0] for s in models]
        b = _lib.Batch(sims)
        b.run_recorded(nt, boxes)
        out.append(b.adjoint([2 * sim.dft() for sim in sims]))
        b.close()
        for sim in sims:
            sim.close()
    assert all(np.abs(g).max() > 0 and np.array_equal(g, w) for g, w in zip(*out))
