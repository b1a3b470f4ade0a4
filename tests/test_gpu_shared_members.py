"""A simulation that runs by itself and as a member of batches: a run of one kind
moves or frees device buffers that the engines of the other kind were built on,
and each of them has to notice. And several engines side by side, each with its own
shape of the same kernels."""
import numpy as np
import pytest

from modelgen import configs
from rfnetwork_b200 import _lib
from test_gpu_resident import _model_sim

pytestmark = pytest.mark.gpu

NT = 60
SIZES = ((40, 36, 34), (20, 18, 16))
PHASE = np.exp(-0.1j * np.arange(2 * NT + 1)[:, None] * np.arange(1, 3)[None]).astype(np.complex64)


def _make(n):
    sim, _ = _model_sim(configs.microstrip(n=n, n_pml=3, nt=2 * NT))
    sim.add_monitor(2, 2, n[2] // 2, 1, phase=PHASE)
    return sim


def _results(sim):
    return sim.probe_values(), sim.dft(), sim.monitor(0)


def _want(n, nt):
    sim = _make(n)
    sim.run(nt)
    out = _results(sim)
    sim.close()
    assert np.abs(out[0]).max() > 0 and np.abs(out[2]).max() > 0
    return out


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("kernel", [(1, 0, 4), (1, 8, 4), (0, 0, 4)])
def test_other_step_counts_in_between(engine_lib, kernel):
    """Runs with another number of steps reallocate the sources, records, sums and
    monitor outputs; the buffers between them keep the old addresses from coming back."""
    want = {(n, nt): _want(n, nt) for n in SIZES for nt in (NT, 2 * NT)}
    sims = [_make(n) for n in SIZES]
    others = []
    batch = _lib.Batch(sims)
    batch.set_kernel(*kernel)
    for sim in sims:
        sim.set_kernel(*kernel)

    def check(nt):
        for n, sim in zip(SIZES, sims):
            assert _same(_results(sim), want[n, nt])
        other = _make(SIZES[1])  # (takes freed blocks of the records' size)
        other.run(nt)
        others.append(other)

    for nt in (NT, NT):  # (the second run replays a graph)
        batch.run(nt)
        check(nt)
    for nt in (2 * NT, NT, NT):  # by themselves
        for sim in sims:
            sim.run(nt)
        check(nt)
    batch.run(NT)  # as before, on moved buffers
    check(NT)
    batch.run(2 * NT)
    check(2 * NT)
    batch.run(NT)
    check(NT)
    for sim in sims:  # the same for the members' own engines
        sim.run(NT)
    check(NT)
    batch.close()
    for sim in sims + others:
        sim.close()


def test_refused_step_count_in_between(engine_lib):
    """A run refused for its step count leaves the results of the run before it, and
    the same run again gives them again."""
    n = SIZES[1]
    want = _want(n, NT)
    sim, _ = _model_sim(configs.microstrip(n=n, n_pml=3, nt=2 * NT))
    sim.add_monitor(2, 2, n[2] // 2, 1, phase=PHASE[:NT + 1])  # too short for 2 NT steps
    for _ in range(2):
        sim.run(NT)
        assert _same(_results(sim), want)
        with pytest.raises(ValueError, match="phase table"):
            sim.run(2 * NT)
        sim.nt = NT
        assert _same(_results(sim), want)
    co = configs.microstrip(n=n, n_pml=3, nt=2 * NT).pack_inputs(gpu=True)[0]
    sim.set_coefficients(co)  # (the refused run then compiles and moves the fields first)
    with pytest.raises(ValueError, match="phase table"):
        sim.run(2 * NT)
    sim.run(NT)
    assert _same(_results(sim), want)
    sim.close()


def test_modes_change_hands(engine_lib):
    """Plain, recorded and checkpointed runs of the members by themselves and in two
    batches, each twice (the second replays a graph) before another kind follows."""
    boxes = [(n[0] // 2 - 4, n[0] // 2 + 4, n[1] // 2 - 3, n[1] // 2 + 3, 5, 7) for n in SIZES]
    want, grads, others = {}, [], []
    for n, box in zip(SIZES, boxes):
        want[n] = _want(n, NT)
        sim = _make(n)
        sim.run_recorded(NT, box)
        grads.append(sim.adjoint(2 * sim.dft(), box))
        assert np.abs(grads[-1]).max() > 0
        sim.close()
    sims = [_make(n) for n in SIZES]
    pair = [_lib.Batch(sims), _lib.Batch(sims)]

    def single(mode):
        for n, sim, box, g in zip(SIZES, sims, boxes, grads):
            if mode == "run":
                sim.run(NT)
            elif mode == "recorded":
                sim.run_recorded(NT, box)
            else:
                sim.run_checkpointed(NT, 16)
            assert _same(_results(sim), want[n])
            if mode != "run":
                assert np.array_equal(sim.adjoint(2 * sim.dft(), box), g)

    def together(batch, mode):
        if mode == "run":
            batch.run(NT)
        elif mode == "recorded":
            batch.run_recorded(NT, boxes)
        else:
            batch.run_checkpointed(NT, 16, boxes)
        assert all(_same(_results(sim), want[n]) for n, sim in zip(SIZES, sims))
        if mode != "run":
            assert all(map(np.array_equal, batch.adjoint([2 * sim.dft() for sim in sims]), grads))

    modes = ("run", "recorded", "checkpointed")
    for a in modes:
        for b in modes:
            for who in (0, 1):  # who comes between: a batch, or the members by themselves
                first = single if who == 0 else lambda m: together(pair[0], m)
                then = (lambda m: together(pair[0], m)) if who == 0 else single
                first(a), first(a)
                then(b), then(b)
                other = _make(SIZES[0])  # takes what they freed
                other.run_recorded(NT, boxes[0])
                others.append(other)
                first(a), first(a)
            together(pair[0], a), together(pair[0], a)
            together(pair[1], b), together(pair[1], b)
            together(pair[0], a), together(pair[1], a)
    for x in pair + sims + others:
        x.close()


def test_kernel_chosen_before_a_refused_call(engine_lib):
    """A batch call refused for one member's box does not forget the kernel chosen
    before it."""
    sims = [_make(n) for n in SIZES]
    batch = _lib.Batch(sims)
    batch.run(NT)
    assert batch.stats()["variant"] != 0
    want = [_results(sim) for sim in sims]
    batch.set_kernel(0)
    with pytest.raises(ValueError, match="box"):
        batch.run_recorded(NT, [(0, 3, 0, 3, 0, 3), (4, 6, 4, 6, 5, 7)])
    batch.run(NT)
    assert batch.stats()["variant"] == 0
    assert all(_same(_results(sim), w) for sim, w in zip(sims, want))
    batch.close()
    for sim in sims:
        sim.close()


def test_handles_with_different_plane_slots(engine_lib):
    """Handles whose launches use different amounts of shared memory take turns; each
    runs from the host first and as a graph later, and a gradient's replays too."""
    n, box = SIZES[0], (16, 24, 14, 20, 9, 11)
    want = _want(n, NT)
    sims = []
    for stages in (8, 4, 6, 3):
        sim = _make(n)
        sim.set_kernel(1, 8, stages)
        sims.append(sim)
    for _ in range(3):
        for sim in sims:
            sim.run(NT)
            assert _same(_results(sim), want)
    grads = []
    for _ in range(2):
        for sim in sims:
            sim.run_checkpointed(NT, 16)
        for sim in sims:
            grads.append(sim.adjoint(2 * sim.dft(), box))
    assert np.abs(grads[0]).max() > 0 and all(np.array_equal(g, grads[0]) for g in grads)
    for sim in sims:
        sim.set_graph(False)
        sim.run(NT)
        assert _same(_results(sim), want)
        sim.close()
