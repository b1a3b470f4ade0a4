"""What a user of this framework has it do, as timed cases.

Every case is one of these kinds, at sizes of the repository's own workloads
and tests or of the same range:

  resident   a model kept on the GPU (``Simulation``): one pass is one time
             loop from zero fields, then the probe records and the device DFT
  solve      the drop-in call on host arrays (``cuda_func``): one pass compiles
             the coefficient arrays, runs the loop and reads the results, with
             phasor plane monitors where a far field is wanted
  farfield   the near-to-far-field transform of surface currents on host arrays
  batch      uneven grids stepped together (``Batch``)
  gradient   one forward and one backward pass through ``FDTDDesign``
  designs    the same for several variants at once (``FDTDDesignBatch``)

The models are dielectric boxes or a strip line over a ground plane, in a
box of metal or with graded split-field absorbing layers on all six faces, on
uniform or graded cells, with resistive ports that carry a pulse. ``exact``
marches the same discretisation in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

E0, U0, C0 = 8.854187817e-12, 4e-7 * math.pi, 299792458.0
INCH = 0.0254
CELL = 2.0 ** -7  # inches
AX = "xyz"
# (field, split axis, sign of the difference) in the engine's split order
E_SPLITS = (("ex", "y", 1), ("ex", "z", -1), ("ey", "z", 1), ("ey", "x", -1), ("ez", "x", 1), ("ez", "y", -1))
H_SPLITS = (("hx", "y", -1), ("hx", "z", 1), ("hy", "z", -1), ("hy", "x", 1), ("hz", "x", -1), ("hz", "y", 1))


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest calls: a model of a few thousand cells while a geometry is sketched; launch latency is all
        dict(name="resident_tiny", kind="resident", nx=24, ny=20, nz=16, pml=4, nt=300, model="line", graded=False,
             freqs=11),
        # the ordinary solve: a strip line, 10-cell absorbing layers, S-parameters from a 101-frequency DFT
        dict(name="resident_line", kind="resident", nx=64, ny=64, nz=48, pml=10, nt=2000, model="line", graded=False,
             freqs=101),
        # the same on a graded mesh with odd sizes that fill no tile
        dict(name="resident_graded", kind="resident", nx=91, ny=71, nz=53, pml=7, nt=1000, model="line", graded=True,
             freqs=101),
        # a shielded resonator: no absorbing layers, every cell an interior cell
        dict(name="resident_cavity", kind="resident", nx=150, ny=130, nz=90, pml=0, nt=400, model="boxes",
             graded=False, freqs=51),
        # the largest grid of the benchmark, larger than the L2 cache (fewer steps; a step costs the same)
        dict(name="resident_large", kind="resident", nx=256, ny=256, nz=128, pml=8, nt=300, model="boxes",
             graded=False, freqs=51),
        # the reference's own call, host arrays in and records out
        dict(name="solve_hostarrays", kind="solve", nx=120, ny=100, nz=64, pml=8, nt=1500, model="line", graded=False,
             freqs=51, ff=0),
        # an antenna: the same call with far-field phasor monitors on the six faces
        dict(name="solve_antenna", kind="solve", nx=72, ny=64, nz=64, pml=5, nt=800, model="boxes", graded=False,
             freqs=0, ff=2),
        # that antenna's pattern: 19 x 91 directions at two frequencies
        dict(name="farfield_pattern", kind="farfield", n0=58, n1=50, n2=50, freqs=2, theta=19, phi=91),
        # port excitations or variants of uneven size in one launch
        dict(name="batch_uneven", kind="batch", members=8, lo=32, hi=160, sizes=7, pml=8, nt=400, freqs=21),
        # a design gradient whose forward history does not fit: field snapshots and recomputation
        dict(name="gradient_checkpointed", kind="gradient", nx=128, ny=128, nz=96, pml=10, nt=480, dx=48, dy=48,
             dz=4, freqs=11, every=32),
        # a small design whose history is recorded
        dict(name="gradient_recorded", kind="gradient", nx=52, ny=44, nz=33, pml=6, nt=400, dx=14, dy=13, dz=2,
             freqs=11, every=0),
        # several variants per optimiser step
        dict(name="designs_batched", kind="designs", variants=6, nx=96, ny=96, nz=64, pml=10, nt=220, dx=32, dy=32,
             dz=4, freqs=5, every=20),
    ]


MOST_CELL_STEPS = 256 * 256 * 128 * 300


def draw(rng: random.Random) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(cells_lo, cells_hi, pml):
        """Three axes whose product is spread over its logarithm; room for the layers and a model."""
        lo = 2 * pml + 12
        while True:
            n = log(cells_lo, cells_hi)
            a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
            s = (n / (a * b)) ** (1 / 3)
            d = [max(lo, int(s * a)), max(lo, int(s * b)), max(lo, int(s))]
            if d[0] * d[1] * d[2] <= 1.3 * cells_hi and max(d) <= 320:
                return d

    kind = rng.choice(["resident", "resident", "resident", "solve", "solve", "farfield", "batch", "gradient",
                       "gradient", "designs"])
    pml = rng.choice([4, 5, 6, 7, 8, 10, 12])
    if kind == "farfield":
        return dict(kind=kind, n0=log(12, 120), n1=log(12, 120), n2=log(12, 120), freqs=rng.randint(1, 4),
                    theta=log(2, 91), phi=log(1, 91))
    if kind == "batch":
        return dict(kind=kind, members=rng.randint(2, 8), lo=rng.randint(32, 40), hi=rng.randint(60, 128),
                    sizes=rng.randint(0, 10 ** 6), pml=rng.choice([4, 6, 8]), nt=rng.randint(60, 300),
                    freqs=rng.randint(1, 51))
    if kind in ("gradient", "designs"):
        pml = min(pml, 10)
        n = grid(4e4, 1.2e6 if kind == "gradient" else 3e5, pml)
        c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], pml=pml, nt=log(80, 400),
                 dx=rng.randint(4, max(4, (n[0] - 2 * pml) // 3)), dy=rng.randint(4, max(4, (n[1] - 2 * pml) // 3)),
                 dz=rng.randint(1, 4), freqs=rng.randint(1, 11), every=rng.choice([0, 0, 13, 20, 32, 50]))
        if kind == "designs":
            c = dict(c, variants=rng.randint(2, 5), every=c["every"] or 20)
        return c
    model = rng.choice(["line", "boxes"])
    if model == "boxes" and rng.random() < 0.25:
        pml = 0
    n = grid(8e3, 6e6 if kind == "resident" else 1.5e6, pml)
    nt = max(60, min(log(100, 2000), MOST_CELL_STEPS // (3 * n[0] * n[1] * n[2])))
    c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], pml=pml, nt=nt, model=model,
             graded=model == "line" and rng.random() < 0.4, freqs=rng.choice([1, 11, 51, 101]))
    if kind == "solve":
        c["ff"] = rng.choice([0, 0, 1, 2, 3]) if pml else 0
    return c


# ---------------------------------------------------------------- the models
def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _widths(case, axis):
    """Cell widths (inches) along an axis; a graded mesh has cells twice as wide away from the strip in y and z."""
    n = case[("nx", "ny", "nz")[axis]]
    w = np.full(n, CELL)
    if case.get("graded") and axis:
        a, b = case["pml"] + 1, n - case["pml"] - 1
        third = (b - a) // 3
        if axis == 1:
            w[a:a + third] *= 2
        w[b - third:b] *= 2
    return w


def _model(case, seed):
    """Engine inputs of one model: coefficient arrays, probe dicts, DFT terms, cell material and widths."""
    rng = np.random.default_rng(seed)
    n = [case["nx"], case["ny"], case["nz"]]
    pml, nt, dev = case["pml"], case["nt"], _device()
    w_in = [_widths(case, a) for a in range(3)]
    d = [torch.tensor(w * INCH, dtype=torch.float64, device=dev) for w in w_in]
    dt = 0.99 / (C0 * math.sqrt(sum(1.0 / float(x.min()) ** 2 for x in d)))
    lo, hi = [pml + 1] * 3, [k - pml - 1 for k in n]
    eps = torch.full(n, E0, dtype=torch.float64, device=dev)
    sig = torch.zeros(n, dtype=torch.float64, device=dev)
    line = case.get("model", "line") == "line"
    zg = lo[2] + max(1, n[2] // 12)
    zs = min(zg + 4, hi[2] - 2)
    if line:
        eps[:, :, zg:zs] = float(rng.uniform(2.2, 4.5)) * E0
    else:
        for _ in range(12):
            size = [int(rng.integers(4, max(5, (hi[a] - lo[a]) // 2))) for a in range(3)]
            at = [int(rng.integers(lo[a], max(lo[a] + 1, hi[a] - size[a]))) for a in range(3)]
            box = tuple(slice(at[a], min(at[a] + size[a], hi[a])) for a in range(3))
            eps[box] = float(rng.uniform(1, 10)) * E0
            sig[box] = float(rng.uniform(0, 0.05))
    smax = [0.8 * 4 / (math.sqrt(U0 / E0) * float(x[0])) for x in d]

    def view(v, axis):
        return v.reshape([-1 if a == axis else 1 for a in range(3)])

    def average(v, axis):
        """Width-weighted mean of a cell and the next one; vacuum past the last cell."""
        m = v.shape[axis] - 1
        a, b = v.narrow(axis, 0, m), v.narrow(axis, 1, m)
        da, db = view(d[axis][:m], axis), view(d[axis][1:], axis)
        last = torch.full_like(v.narrow(axis, 0, 1), E0 if v is not sig else 0.0)
        return torch.cat([(a * da + b * db) / (da + db), last], axis)

    def layers(axis, half):
        """Conductivity of the absorbing layers at the cells (half) or at the planes after them."""
        k = torch.arange(n[axis], dtype=torch.float64, device=dev)
        if half:
            depth = torch.maximum(pml - 0.5 - k, k - (n[axis] - pml) + 0.5)
        else:
            f = k + 1
            depth = torch.maximum(pml - f, f - (n[axis] - pml))
            depth = torch.where(f < n[axis], depth, torch.zeros_like(depth))
        on = depth >= 0 if pml else torch.zeros_like(depth, dtype=torch.bool)
        return view(torch.where(on, smax[axis] * (depth.clamp(min=0) / max(pml, 1)) ** 3, torch.zeros_like(depth)),
                    axis), view(on, axis)

    e_mat, loss = {}, {}
    for c in range(3):
        em, sm = eps, sig
        for a in range(3):
            if a != c:
                em, sm = average(em, a), (average(sm, a) if sm is not sig else _avg_sigma(sig, d, a))
        e_mat["e" + AX[c]], loss["e" + AX[c]] = em, sm
    # resistive ports across the substrate (or a few cells of a box model), driven by a pulse
    ports = []
    if line:
        zp = list(range(zg, zs))
        x0, x1, yc = lo[0] + 2, hi[0] - 3, n[1] // 2
        cols = [(x0, yc - 1), (x0, yc), (x0, yc + 1)], [(x1, yc - 1), (x1, yc), (x1, yc + 1)]
    else:
        z0 = int(rng.integers(lo[2] + 1, hi[2] - 4))
        zp = list(range(z0, z0 + 3))
        cols = [[(int(rng.integers(lo[0] + 1, hi[0] - 1)), int(rng.integers(lo[1] + 1, hi[1] - 2)))]
                for _ in range(2)]
    for group in cols:
        sites = [(x, y, z) for x, y in group for z in zp]
        for x, y, z in sites:  # full-grid ez index; the packed arrays hold it at (x - 1, y - 1, z)
            loss["ez"][x - 1, y - 1, z] += float(d[2][z]) / (50.0 * len(group) / len(zp) * float(d[0][x]) *
                                                             float(d[1][y]))
        ports.append(sites)
    coef, dh = {}, []
    for a in range(3):
        inv = torch.zeros_like(d[a])
        inv[:-1] = 2.0 / (d[a][:-1] + d[a][1:])
        dh.append(view(inv, a))
    for f, ax, sign in E_SPLITS:
        a = AX.index(ax)
        s, on = layers(a, False)
        em, sm = e_mat[f], loss[f]
        se = torch.where(on, s * em / E0, sm)
        den = 2 * em + se * dt
        ca, cb = (2 * em - se * dt) / den, sign * (2 * dt / den) * dh[a]
        if line:  # the ground sheet and the strip are metal
            metal = torch.zeros(n, dtype=torch.bool, device=dev)
            if f != "ez":
                metal[:, :, zg - 1] = True
                metal[lo[0] + 2:hi[0] - 3, n[1] // 2 - 3:n[1] // 2 + 3, zs - 1] = True
            ca, cb = torch.where(metal, -torch.ones_like(ca), ca), torch.where(metal, torch.zeros_like(cb), cb)
        coef["Ca_%s_%s" % (f, ax)], coef["Cb_%s_%s" % (f, ax)] = ca.expand(n), cb.expand(n)
    for f, ax, sign in H_SPLITS:
        a = AX.index(ax)
        s, _ = layers(a, True)
        g = s * dt / E0
        coef["Da_%s_%s" % (f, ax)] = ((2 - g) / (2 + g)).expand(n)
        db = (sign * (2 * dt / (U0 * (2 + g))) / view(d[a], a)).expand(n)
        coef["Db_%s_%s1" % (f, ax)] = coef["Db_%s_%s2" % (f, ax)] = db
    coef = {k: v.to(torch.float32).contiguous().cpu().numpy() for k, v in coef.items()}

    t = np.arange(nt)
    width = 8.0 * 1.5 ** float(rng.uniform(0, 1))
    pulse = np.exp(-((t - 3.2 * width) / width) ** 2) * float(rng.uniform(0.5, 2.0))
    probes, terms = [], []
    for k, sites in enumerate(ports):
        for x, y, z in sites:
            terms.append((k, len(probes), -float(d[2][z]) / max(1, len(cols[k]))))
            probes.append(dict(values=(pulse * (k == 0)).astype(np.float32), field=2, idx=[x, y, z],
                               is_source=int(k == 0)))
    for k in range(12):
        f = k % 6
        at = [int(rng.integers(lo[a] + 1, hi[a] - 1)) for a in range(3)]
        terms.append((2 + k // 4, len(probes), float(rng.uniform(0.5, 1.5))))
        probes.append(dict(values=np.zeros(nt, np.float32), field=f, idx=at, is_source=0))
    omega = 2 * np.pi * np.linspace(1e9, 20e9, max(1, case["freqs"])) * dt
    return dict(coef=coef, probes=probes, terms=terms, omega=omega, n=n, nt=nt, dt=dt, eps=eps.cpu().numpy(),
                sig=sig.cpu().numpy(), d_in=tuple(w_in))


def _avg_sigma(v, d, axis):
    m = v.shape[axis] - 1
    shape = [-1 if a == axis else 1 for a in range(3)]
    da, db = d[axis][:m].reshape(shape), d[axis][1:].reshape(shape)
    mean = (v.narrow(axis, 0, m) * da + v.narrow(axis, 1, m) * db) / (da + db)
    return torch.cat([mean, torch.zeros_like(v.narrow(axis, 0, 1))], axis)


def _monitors(case, m):
    """Far-field phasor monitors: per face two tangential E planes and the H planes either side of it."""
    if not case.get("ff"):
        return []
    freq, n, pad, out = np.linspace(8e9, 20e9, case["ff"]), m["n"], case["pml"] + 2, []
    phase = np.exp(-1j * (2 * np.pi * freq * m["dt"])[None] * np.arange(m["nt"] + 1)[:, None]).astype(np.complex64)
    for axis in range(3):
        shape = tuple(n[a] for a in range(3) if a != axis)
        for at, other in ((pad, pad - 1), (n[axis] - pad, n[axis] - pad + 1)):
            for f in [a for a in range(3) if a != axis]:
                for field, pos in ((f, at), (3 + f, at), (3 + f, other)):
                    out.append(dict(field=field, axis=axis, position=pos, n_step=1, dtft_phase=phase,
                                    n_frequencies=len(freq),
                                    values=np.zeros((len(freq),) + shape, dtype=np.complex64)))
    return out


def _simulation(m):
    from rfnetwork_b200 import _lib

    sim = _lib.Simulation(*m["n"])
    sim.set_coefficients(m["coef"])
    for p in m["probes"]:
        sim.add_probe(p["field"], p["idx"], bool(p["is_source"]), p["values"] if p["is_source"] else None)
    sim.set_dft(m["terms"], m["omega"])
    return sim


def _member_cases(case):
    r = random.Random(case["sizes"])
    return [dict(nx=r.randint(case["lo"], case["hi"]), ny=r.randint(case["lo"], case["hi"]),
                 nz=r.randint(case["lo"], case["hi"]), pml=case["pml"], nt=case["nt"], freqs=case["freqs"],
                 model="boxes") for _ in range(case["members"])]


def _design(case):
    """Cells of the design region: centred in x and y, in the substrate."""
    n, z = [case["nx"], case["ny"], case["nz"]], case["pml"] + 1 + max(1, case["nz"] // 12)
    x, y = (n[0] - case["dx"]) // 2, case["pml"] + 3
    return (x, x + case["dx"], y, min(y + case["dy"], n[1] - case["pml"] - 3), z + 5, min(z + 5 + case["dz"],
                                                                                       n[2] - case["pml"] - 2))


def _theta(case, seed, k=0):
    b = _design(case)
    shape = (b[1] - b[0], b[3] - b[2], b[5] - b[4])
    return torch.from_numpy(np.random.default_rng([seed, 99, k]).standard_normal(shape))


def _output_terms(m):
    """The record of the second port, and one Ez probe: the design's objectives."""
    second = [t for t in m["terms"] if t[0] == 1]
    return [(0, p, w / m["d_in"][2][0]) for _, p, w in second] + [(1, second[-1][1] + 3, 1.0)]


def _packed(m):
    from rfnetwork_b200.adjoint import PackedModel

    return PackedModel(m["coef"], m["probes"], tuple(m["n"]), m["nt"], m["dt"], m["eps"], m["sig"], m["d_in"])


def _currents(case, seed):
    rng = np.random.default_rng(seed)
    n, F = [case["n0"], case["n1"], case["n2"]], case["freqs"]
    w = CELL * INCH
    J, M, r, ds, pos = [], [], [], [], []
    for axis in range(3):
        f0, f1 = [a for a in range(3) if a != axis]
        centre = [(np.arange(n[a]) - (n[a] - 1) / 2) * w for a in (f0, f1)]
        r.append([np.ascontiguousarray(v, dtype=np.float32) for v in np.meshgrid(*centre, indexing="ij")])
        ds.append(np.full((n[f0], n[f1]), w * w, dtype=np.complex64))
        pos.append([-n[axis] * w / 2, n[axis] * w / 2])
        shape = (3, F, n[f0], n[f1])
        J.append([(rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
                  for _ in range(2)])
        M.append([(377 * rng.standard_normal(shape) + 377j * rng.standard_normal(shape)).astype(np.complex64)
                  for _ in range(2)])
    f = dict(beta=(2 * np.pi * np.linspace(8e9, 20e9, F) / C0).astype(np.float32),
             theta=np.linspace(0, np.pi, case["theta"]).astype(np.float32),
             phi=np.linspace(-np.pi, np.pi, case["phi"]).astype(np.float32),
             data=np.zeros((2, F, case["theta"], case["phi"]), dtype=np.complex64))
    return J, M, r, ds, pos, f


# ---------------------------------------------------------------- one pass
def prepare(case, seed):
    kind = case["kind"]
    if kind == "farfield":
        return dict(kind=kind, args=_currents(case, seed))
    if kind == "batch":
        from rfnetwork_b200 import _lib

        sims = [_simulation(_model(c, seed * 1000 + i)) for i, c in enumerate(_member_cases(case))]
        return dict(kind=kind, sims=sims, batch=_lib.Batch(sims), nt=case["nt"])
    if kind in ("gradient", "designs"):
        from rfnetwork_b200.adjoint import FDTDDesign, FDTDDesignBatch

        m = _model(case, seed)
        args = (_design(case), _output_terms(m), m["omega"])
        if kind == "gradient":
            return dict(kind=kind, design=FDTDDesign(_packed(m), *args, checkpoint_every=case["every"] or None),
                        theta=_theta(case, seed))
        pk = _packed(m)
        return dict(kind=kind, design=FDTDDesignBatch([pk] * case["variants"], *args,
                                                      checkpoint_every=case["every"] or None),
                    theta=[_theta(case, seed, k) for k in range(case["variants"])])
    m = _model(case, seed)
    if kind == "solve":
        return dict(kind=kind, m=m, monitors=_monitors(case, m), freqs=case["freqs"])
    return dict(kind=kind, sim=_simulation(m), nt=case["nt"])


def run(state):
    kind = state["kind"]
    if kind == "resident":
        sim = state["sim"]
        sim.run(state["nt"])
        return dict(records=sim.probe_values(), dft=sim.dft())
    if kind == "batch":
        state["batch"].run(state["nt"])
        return [dict(records=s.probe_values(), dft=s.dft()) for s in state["sims"]]
    if kind == "farfield":
        from rfnetwork_b200 import _lib

        _lib.nf2ff(*state["args"])
        return state["args"][-1]["data"]
    if kind == "solve":
        from rfnetwork_b200 import cuda_func

        m, mon = state["m"], state["monitors"]
        probes = [dict(p, values=p["values"].copy()) for p in m["probes"]]  # the call overwrites them in place
        n, out = m["n"], {}
        if state["freqs"]:
            out["dft"] = cuda_func.solver_run_dft(m["coef"], probes, mon, *n, m["nt"], m["terms"], m["omega"])
        else:
            cuda_func.solver_run_cu(m["coef"], probes, mon, np.zeros(0, np.float32), *n, m["nt"], 4, 0)
        out["records"] = np.stack([p["values"] for p in probes])
        if mon:
            out["monitors"] = [q["values"] for q in mon]
        return out
    many = kind == "designs"
    theta = [t.clone().requires_grad_(True) for t in (state["theta"] if many else [state["theta"]])]
    eps = [1 + 9 * torch.sigmoid(t) for t in theta]
    X = state["design"](eps if many else eps[0])
    (X.abs() ** 2).sum().backward()
    return dict(dft=X.detach(), grad=[t.grad for t in theta])


# ---------------------------------------------------------------- what a pass needs
def _step_bytes(n, pml):
    """49 B per interior and 97 B per absorbing-layer cell: fields or split pairs read and written, 1 B of material."""
    total = n[0] * n[1] * n[2]
    inner = max(n[0] - 2 * pml, 0) * max(n[1] - 2 * pml, 0) * max(n[2] - 2 * pml, 0)
    return 49.0 * inner + 97.0 * (total - inner), 36.0 * inner + 42.0 * (total - inner)


def work(case):
    kind = case["kind"]
    if kind == "farfield":
        cells = 2 * (case["n0"] * case["n1"] + case["n0"] * case["n2"] + case["n1"] * case["n2"])
        dirs = case["theta"] * case["phi"]
        # per cell, direction and frequency: a phase (6), its sine and cosine (about 20), six complex products (48)
        return dict(bytes=case["freqs"] * (cells * 48.0 + dirs * 16.0) + cells * 12.0,
                    flops=74.0 * cells * dirs * case["freqs"])
    if kind == "batch":
        w = [_step_bytes((c["nx"], c["ny"], c["nz"]), c["pml"]) for c in _member_cases(case)]
        return dict(bytes=case["nt"] * sum(b for b, _ in w), flops=case["nt"] * sum(f for _, f in w))
    n = (case["nx"], case["ny"], case["nz"])
    b, f = _step_bytes(n, case["pml"])
    times = case["nt"]
    if kind in ("gradient", "designs"):
        box = _design(case)
        hist = 36.0 * 2 * (box[1] - box[0] + 1) * (box[3] - box[2] + 1) * (box[5] - box[4] + 1)
        # a step forward and a step back, and the box's history written and read
        return dict(bytes=times * (2 * b + hist) * case.get("variants", 1), flops=2 * times * f * case.get("variants", 1))
    extra = 0.0
    if kind == "solve":
        extra = 30 * 4.0 * n[0] * n[1] * n[2]  # the coefficient arrays, read once
        extra += case["ff"] * times * 2 * 6 * 12.0 * (n[0] * n[1] + n[0] * n[2] + n[1] * n[2]) / 3
    return dict(bytes=times * b + extra, flops=times * f)


# ---------------------------------------------------------------- the same in 64 bits
def _shift(h, axis):
    """The next cell's value along an axis, zero past the end."""
    return torch.cat([h.narrow(axis, 1, h.shape[axis] - 1), torch.zeros_like(h.narrow(axis, 0, 1))], axis)


def _back(e, axis):
    return torch.cat([torch.zeros_like(e.narrow(axis, 0, 1)), e.narrow(axis, 0, e.shape[axis] - 1)], axis)


def _coef64(m):
    dev = _device()
    c = {k: torch.from_numpy(v).to(dev, torch.float64) for k, v in m["coef"].items()}
    for k in c:  # the last x plane of the y and z electric and the x magnetic coefficients is a wall
        if k[3:5] in ("ey", "ez", "hx"):
            c[k] = c[k].clone()
            c[k][-1] = 0
    return c


def _site(p):
    """Cell of a probe: the engine's shift of each component's index."""
    f, idx = p["field"], list(p["idx"])
    for a, fields in ((0, (1, 2, 3)), (1, (0, 2, 4)), (2, (0, 1, 5))):
        if f in fields:
            idx[a] -= 1
    return tuple(idx)


def _e_difference(H, f, ax):
    """The difference of the magnetic component that drives split (f, ax) of E."""
    other = 3 - AX.index(f[1]) - AX.index(ax)
    h = H[other]
    return _shift(h, AX.index(ax)) - h


def _marcher(m, coef):
    """One step (state, n) -> (state, recorded values) in 64 bits; the state is 12 split arrays."""
    dev = _device()
    sites = [_site(p) for p in m["probes"]]
    at = [torch.tensor([s[a] for s in sites], device=dev) for a in range(3)]
    field = [[k for k, p in enumerate(m["probes"]) if p["field"] == f] for f in range(6)]
    src = {}
    for k, p in enumerate(m["probes"]):
        if p["is_source"]:
            src.setdefault(p["field"], []).append(k)
    amp = {f: torch.from_numpy(np.stack([m["probes"][k]["values"] for k in ks])).to(dev, torch.float64)
           for f, ks in src.items()}
    order = torch.tensor([k for f in range(6) for k in field[f]], device=dev)
    back = torch.argsort(order)

    def step(state, n):
        E, H = list(state[:6]), list(state[6:])
        Ht = [H[0] + H[1], H[2] + H[3], H[4] + H[5]]
        for s, (f, ax, _) in enumerate(E_SPLITS):
            name = "%s_%s" % (f, ax)
            E[s] = coef["Ca_" + name] * E[s] + coef["Cb_" + name] * _e_difference(Ht, f, ax)
        for f, ks in src.items():
            cells = tuple(a[ks] for a in at)
            for s in (2 * f, 2 * f + 1):
                E[s] = E[s].index_put(cells, amp[f][:, n], accumulate=True)
        Et = [E[0] + E[1], E[2] + E[3], E[4] + E[5]]
        for s, (f, ax, _) in enumerate(H_SPLITS):
            name, a = "%s_%s" % (f, ax), AX.index(ax)
            e = Et[3 - AX.index(f[1]) - a]
            H[s] = coef["Da_" + name] * H[s] + (coef["Db_%s2" % name] * e - coef["Db_%s1" % name] * _back(e, a))
        tot = Et + [H[0] + H[1], H[2] + H[3], H[4] + H[5]]
        rec = torch.cat([tot[f][tuple(a[field[f]] for a in at)] for f in range(6)])[back]
        return tuple(E + H), rec, tot

    return step


def _spectrum(rec, terms, omega):
    """X[series, frequency] of records [probes, nt]."""
    dev = rec.device
    nt = rec.shape[1]
    om = torch.tensor(omega, dtype=torch.float64, device=dev)
    ph = torch.exp(-1j * om[:, None] * torch.arange(nt, dtype=torch.float64, device=dev)[None])
    series = []
    for s in range(max(t[0] for t in terms) + 1):
        series.append(sum(w * rec[p] for k, p, w in terms if k == s))
    return torch.stack(series).to(torch.complex128) @ ph.T


def _march(m, monitors=()):
    with torch.no_grad():
        step = _marcher(m, _coef64(m))
        state = tuple(torch.zeros(m["n"], dtype=torch.float64, device=_device()) for _ in range(12))
        rec = []
        mon = [torch.zeros(q["values"].shape, dtype=torch.complex128, device=_device()) for q in monitors]
        for n in range(m["nt"]):
            state, r, tot = step(state, n)
            rec.append(r)
            for q, acc in zip(monitors, mon):
                pos = q["position"] - int(q["field"] in ((3, 1, 2), (4, 0, 2), (5, 0, 1))[q["axis"]])
                v = tot[q["field"]].select(q["axis"], pos)
                acc += v[None] * torch.from_numpy(q["dtft_phase"][n].astype(np.complex128)).to(v.device)[:, None, None]
        return torch.stack(rec, 1), mon


def _affordable(case, times=1):
    cells = case["nx"] * case["ny"] * case["nz"]
    if torch.cuda.is_available():
        return times * case["nt"] * (2.2e-3 + cells * 6e-10) < 16
    return times * case["nt"] * cells * 1e-7 < 16


def _design_coefficients(m, case, theta):
    """The E coefficients with the design cells' permittivity in place, differentiably: {name: array}."""
    dev = _device()
    b = _design(case)
    x = slice(b[0], b[1]), slice(b[2], b[3]), slice(b[4], b[5])
    coef = _coef64(m)
    grow = tuple(slice(s.start - 1, s.stop) for s in x)
    eps = torch.from_numpy(m["eps"]).to(dev).clone()
    new = eps.clone()
    new[x] = E0 * (1 + 9 * torch.sigmoid(theta.to(dev)))
    sig = torch.from_numpy(m["sig"]).to(dev)
    d = [torch.from_numpy(w * INCH).to(dev) for w in m["d_in"]]
    touched = torch.zeros(m["n"], dtype=torch.float64, device=dev)
    touched[x] = 1.0
    for f, ax, _ in E_SPLITS:
        site = []
        for v in (new, eps, sig, touched):
            for a in range(3):
                if AX[a] != f[1]:
                    v = _avg_sigma(v, d, a)
            site.append(v[grow])
        e_new, e_old, s, t = site
        name = "%s_%s" % (f, ax)
        ca = (2 * e_new - s * m["dt"]) / (2 * e_new + s * m["dt"])
        old_ca, old_cb = coef["Ca_" + name][grow], coef["Cb_" + name][grow]
        cb = old_cb * (2 * e_old + s * m["dt"]) / (2 * e_new + s * m["dt"])
        for key, old, val in (("Ca_", old_ca, ca), ("Cb_", old_cb, cb)):
            full = coef[key + name].clone()
            full[grow] = torch.where(t > 0, val, old)
            coef[key + name] = full
    return coef


def _exact_gradient(m, case, theta):
    theta = theta.clone().requires_grad_(True)
    terms = _output_terms(m)
    coef = _design_coefficients(m, case, theta)
    names = list(coef)
    block = 12

    def segment(n0, n1, *args):
        step = _marcher(m, dict(zip(names, args[12:])))
        state, rec = args[:12], []
        for n in range(n0, n1):
            state, r, _ = step(state, n)
            rec.append(r)
        return (*state, torch.stack(rec, 1))

    state = tuple(torch.zeros(m["n"], dtype=torch.float64, device=_device()) for _ in range(12))
    records = []
    for n0 in range(0, m["nt"], block):
        out = checkpoint(segment, n0, min(m["nt"], n0 + block), *state, *coef.values(), use_reentrant=False)
        state = out[:12]
        records.append(out[12])
    X = _spectrum(torch.cat(records, 1), terms, m["omega"])
    (X.abs() ** 2).sum().backward()
    return X.detach().cpu(), theta.grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "farfield":
        return _exact_farfield(*_currents(case, seed))
    if kind == "batch":
        out = []
        members = _member_cases(case)
        if not all(_affordable(c, len(members)) for c in members):
            return None
        for i, c in enumerate(members):
            m = _model(c, seed * 1000 + i)
            rec, _ = _march(m)
            out.append(dict(records=rec.cpu(), dft=_spectrum(rec, m["terms"], m["omega"]).cpu()))
        return out
    many = case.get("variants", 1)
    if kind in ("gradient", "designs"):
        # the graph of a block of steps stays below about 40 GB
        if not _affordable(case, 5 * many) or case["nx"] * case["ny"] * case["nz"] > 2_000_000:
            return None
        m = _model(case, seed)
        got = [_exact_gradient(m, case, _theta(case, seed, k)) for k in range(many)]
        X = got[0][0] if kind == "gradient" else torch.stack([g[0] for g in got])
        return dict(dft=X, grad=[g[1] for g in got])
    if not _affordable(case):
        return None
    m = _model(case, seed)
    mon = _monitors(case, m) if kind == "solve" else []
    rec, acc = _march(m, mon)
    out = dict(records=rec.cpu())
    if kind == "resident" or case["freqs"]:
        out["dft"] = _spectrum(rec, m["terms"], m["omega"]).cpu()
    if mon:
        out["monitors"] = [a.cpu() for a in acc]
    return out


def _exact_farfield(J, M, r, ds, pos, f):
    dev = _device()

    def t(v, kind=torch.float64):
        return torch.from_numpy(np.ascontiguousarray(v)).to(dev, kind)

    th, ph = torch.meshgrid(t(f["theta"]), t(f["phi"]), indexing="ij")
    st, ct, sp, cp = th.sin().reshape(-1), th.cos().reshape(-1), ph.sin().reshape(-1), ph.cos().reshape(-1)
    unit = torch.stack([st * cp, st * sp, ct])
    out = torch.zeros((2, len(f["beta"]), st.numel()), dtype=torch.complex128, device=dev)
    for k, beta in enumerate(f["beta"]):
        S = torch.zeros((6, st.numel()), dtype=torch.complex128, device=dev)
        for axis in range(3):
            o = [a for a in range(3) if a != axis]
            for side in range(2):
                xyz = torch.zeros((3, r[axis][0].size), dtype=torch.float64, device=dev)
                xyz[axis] = float(np.float32(pos[axis][side]))
                xyz[o[0]], xyz[o[1]] = t(r[axis][0]).reshape(-1), t(r[axis][1]).reshape(-1)
                cur = torch.cat([t(v[axis][side][:, k], torch.complex128).reshape(3, -1) for v in (J, M)])
                cur = cur * t(np.real(ds[axis])).reshape(-1)
                for a in range(0, xyz.shape[1], 2048):
                    S += cur[:, a:a + 2048] @ torch.exp(1j * float(beta) * (xyz[:, a:a + 2048].T @ unit))
        N, L = S[:3], S[3:]

        def theta_phi(v):
            return v[0] * ct * cp + v[1] * ct * sp - v[2] * st, -v[0] * sp + v[1] * cp

        (nt_, np_), (lt, lp) = theta_phi(N), theta_phi(L)
        g = float(beta) / (4 * math.pi)
        out[0, k] = -1j * g * (lp + 376.730313 * nt_)
        out[1, k] = 1j * g * (lt - 376.730313 * np_)
    return out.reshape(2, len(f["beta"]), len(f["theta"]), len(f["phi"])).cpu()
