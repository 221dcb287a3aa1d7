"""The work that users of this solver give it, as measurable cases.

A case is one of five kinds of call, all through the package's public entry points:

* ``green``  one application of the spectral Green operator (``evp_green_apply`` and its
  allocation-free form) to a polarization field in device memory, as a caller with a
  fixed-point scheme of its own issues it;
* ``inc``    increments of a solve that is open on the device (``Solve.advance``) and one field
  read back, as a step-by-step caller does: the long middle of every solve;
* ``solve``  a whole short solve through ``Solve``: deck and microstructure read, every
  increment advanced with its row read, one field at the end, closed;
* ``file``   a whole solve as the drop-in executable does it (``run_solver``), scored from its
  ``results.csv``;
* ``batch``  several solves of different grids and materials advanced together
  (``solve_files``), and ``serve`` the same kind of mix through a resident ``Server``.

Grids, materials and loadings are those of the repository's decks (creep, tension, calibration
ramps, the sweep's and the served stream's distributions) on seeded Voronoi polycrystals; the
``work`` of a case counts, per equilibrium iteration and increment, every field that the step
cannot do without once in and once out.
"""
import ctypes
import dataclasses
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from creep_modeling_b200 import Solve, _lib, decks, run_solver, solve_files
from creep_modeling_b200.serve import Server

# bytes per voxel that one equilibrium iteration reads or writes once (12 systems): stress, stress at
# the last increment, velocity gradients, F^-1, weights, three symmetric 6x6 operators, Schmid vectors,
# trial and committed resistances, slip rates, strain rates, the polarization and the correction
ITER_BYTES, ITER_BYTES_PER_SYSTEM = 1160.0, 88.0
# floating-point operations per voxel of one iteration: the local solves (constitutive evaluations,
# Newton steps, hardening) and nine forward and inverse transforms (added in work())
ITER_FLOPS_PER_SYSTEM = 480.0
# bytes per voxel of the updates at the end of an increment (deformation gradients, rotated stiffness,
# operators, averages and the macroscopic tangent)
INC_BYTES = 3600.0


def listed():
    return [
        # the smallest call: the bare operator on the smallest grid in use, where latency is all
        dict(name="green_16", kind="green", n1=16, n2=16, n3=16, alloc=False),
        # the bare operator on a large ragged grid (radices 3 and 5)
        dict(name="green_ragged", kind="green", n1=120, n2=90, n3=80, alloc=True),
        # the smallest solve in daily use: 16^3 creep to its end, plain FP64
        dict(name="creep_16", kind="solve", n1=16, n2=16, n3=16, grains=64, law="creep", nrs=10.0, increments=100),
        # one calibration candidate: stress ramp, then holds with time-step cuts, n = 30, through files
        dict(name="calib_16", kind="file", n1=16, n2=16, n3=16, grains=60, law="ramp", nrs=30.0, increments=24),
        # large-strain tension, the single-solve benchmark's grid and law, in its steady flow
        dict(name="tension_64", kind="inc", n1=64, n2=64, n3=64, grains=500, law="tension", nrs=20.0, systems=12,
             modal=0, phase2="", precision=0, warm=24, increments=4),
        # a fitted (non-integer) exponent on a ragged grid (radices 2, 3 and 5 on unequal axes)
        dict(name="tension_ragged", kind="inc", n1=50, n2=45, n3=36, grains=200, law="tension", nrs=12.6, systems=12,
             modal=0, phase2="", precision=0, warm=24, increments=4),
        # the modified augmented Lagrangian (--modal 1), creep
        dict(name="modal_32", kind="inc", n1=32, n2=32, n3=32, grains=100, law="creep", nrs=10.0, systems=12,
             modal=1, phase2="", precision=0, warm=6, increments=6),
        # a specimen with free side faces (gas layers), as the roughness sweeps run it, whole
        dict(name="surface_32", kind="solve", n1=32, n2=32, n3=20, grains=80, law="creep", nrs=10.0, phase2="gas", increments=3),
        # a BCC law: 24 systems in two modes
        dict(name="bcc_40", kind="inc", n1=40, n2=40, n3=40, grains=150, law="tension", nrs=10.0, systems=24,
             modal=0, phase2="", precision=0, warm=20, increments=4),
        # the largest: two-phase creep at 128^3 in mixed precision
        dict(name="creep_128_mixed", kind="inc", n1=128, n2=128, n3=128, grains=2000, law="creep", nrs=10.0, systems=12,
             modal=0, phase2="stiff", precision=1, warm=4, increments=1),
        # a calibration sweep's batch of uneven grids, results and diagnostics written
        dict(name="sweep_batch", kind="batch", edges="16 32 48 24 40", law="creep", increments=16, precision=0),
        # requests of the served stream through a resident server, mixed precision
        dict(name="served_mix", kind="serve", edges="16 24 40 56", law="stream", increments=20, precision=1),
    ]


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _edge(rng, lo, hi):
    """An edge log-uniform in [lo, hi] whose prime factors the transforms take."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if _smooth(n):
            return n


def draw(rng):
    kind = rng.choice(["green", "solve", "file", "inc", "inc", "inc", "inc", "batch", "serve"])
    if kind == "green":
        alloc = rng.random() < 0.6
        while True:
            n = [_edge(rng, 8, 128 if alloc else 32) for _ in range(3)]
            if (n[0] // 2 + 1) * n[1] * n[2] <= (900000 if alloc else 17408):
                return dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], alloc=alloc)
    # creep decks have cubic grids, as the sweeps' decks do; tension takes any
    if kind in ("solve", "file"):
        law = "ramp" if kind == "file" else rng.choice(["creep", "tension"])
        n = [_edge(rng, 10, 28) for _ in range(3)] if law == "tension" else [_edge(rng, 10, 28)] * 3
        case = dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], grains=rng.randint(20, 100), law=law)
        if kind == "solve" and rng.random() < 0.25:
            return dict(case, nrs=float(rng.randint(5, 10)), phase2="gas", increments=rng.randint(1, 3))
        if kind == "file":
            return dict(case, nrs=float(rng.randint(8, 30)), increments=rng.randint(12, 24))
        return dict(case, nrs=round(rng.uniform(5.0, 20.0 if law == "tension" else 10.0), 2), increments=rng.randint(20, 80))
    if kind in ("batch", "serve"):
        while True:
            edges = [_edge(rng, 16, 40) for _ in range(rng.randint(2, 4))]
            increments = rng.randint(5, 12)
            if sum(e ** 3 for e in edges) * increments <= 600000:
                return dict(kind=kind, edges=" ".join(map(str, edges)), law="stream" if kind == "serve" else "creep",
                            increments=increments, precision=int(rng.random() < 0.5))
    law = rng.choice(["creep", "tension", "tension"])
    while True:
        n = [_edge(rng, 16, 96) for _ in range(3)] if law == "tension" else [_edge(rng, 16, 72)] * 3
        if n[0] * n[1] * n[2] <= 300000:
            break
    nrs = float(rng.randint(5, 20 if law == "tension" else 10))
    if rng.random() < 0.4:
        nrs = round(rng.uniform(5.0, nrs), 2)
    return dict(kind="inc", n1=n[0], n2=n[1], n3=n[2], grains=rng.randint(32, 500), law=law, nrs=nrs,
                systems=24 if rng.random() < 0.2 else 12, modal=int(rng.random() < 0.25),
                phase2=rng.choice(["", "", "stiff"]), precision=int(rng.random() < 0.25), warm=20,
                increments=rng.randint(1, 3))


# ---------------------------------------------------------------- inputs
def _polycrystal(n, grains, seed, phase2):
    """(grain ids, phases) [n1, n2, n3] of a periodic Voronoi tessellation and Bunge angles per grain."""
    rng = np.random.default_rng(seed)
    box = torch.tensor(n, dtype=torch.float32, device="cuda")
    seeds = torch.tensor(rng.uniform(0.0, 1.0, (grains, 3)), dtype=torch.float32, device="cuda") * box
    euler = np.stack([rng.uniform(0.0, 360.0, grains), np.degrees(np.arccos(rng.uniform(-1.0, 1.0, grains))),
                      rng.uniform(0.0, 360.0, grains)], axis=1)
    ax = [torch.arange(m, dtype=torch.float32, device="cuda") + 0.5 for m in n]

    def nearest(points):  # squared periodic distance, an axis at a time, one x plane after the other
        d2, arg = [], []
        per = []
        for a in range(3):
            d = ax[a][:, None] - points[None, :, a]
            per.append((d - box[a] * torch.round(d / box[a])) ** 2)
        for i in range(n[0]):
            m = (per[0][i][None, None] + per[1][:, None] + per[2][None]).min(dim=2)
            d2.append(m.values)
            arg.append(m.indices)
        return torch.stack(d2), torch.stack(arg)

    grain = (nearest(seeds)[1] + 1).cpu().numpy()
    phase = np.ones(n, dtype=np.int64)
    if phase2 == "stiff":  # 5 vol % spheres of 3 voxels' radius
        count = max(1, int(round(0.05 * n[0] * n[1] * n[2] / (4.0 / 3.0 * math.pi * 27.0))))
        centres = torch.tensor(rng.uniform(0.0, 1.0, (count, 3)), dtype=torch.float32, device="cuda") * box
        phase[(nearest(centres)[0] <= 9.0).cpu().numpy()] = 2
    elif phase2 == "gas":  # two layers on the x and y sides
        phase[:2] = phase[-2:] = 2
        phase[:, :2] = phase[:, -2:] = 2
    return grain, phase, euler


def _write_micro(path, grain, phase, euler):
    """``phi1 Phi phi2 i j k grain phase`` lines, x fastest."""
    n1, n2, n3 = grain.shape
    head = ["0.000000 0.000000 0.000000 "] + ["%.6f %.6f %.6f " % tuple(e) for e in euler]
    ij = ["%d %d " % (i + 1, j + 1) for j in range(n2) for i in range(n1)]
    tail = [["", " %d 1\n" % g, " %d 2\n" % g] for g in range(len(euler) + 1)]
    with open(path, "w") as f:
        for k in range(n3):
            g = grain[:, :, k].T.ravel().tolist()
            p = phase[:, :, k].T.ravel().tolist()
            z = str(k + 1)
            f.write("".join([head[a if b == 1 else 0] + c + z + tail[a][b] for a, b, c in zip(g, p, ij)]))


def _material(law, nrs, systems=12):
    if law == "ramp":
        return decks.Material(nrs=nrs, gamd0=1e-4, tau0f=160.0, tau0b=136.0, tau1=2.0, thet0=1000.0, thet1=200.0)
    return decks.Material(nrs=nrs, slip="bcc24" if systems == 24 else "fcc")


def _loading(law, increments):
    creep = decks.Loading(kind="creep", stress33=150.0, udot33=1e-4, tdot=10.0, nsteps=increments)
    if law == "tension":
        return [decks.Loading(kind="tension", udot33=1e-3, tdot=0.5, nsteps=increments)]
    if law == "ramp":  # a stress ramp of one-second steps, then holds whose time step may be cut in half
        ramp = [dataclasses.replace(creep, stress33=s, tdot=1.0, nsteps=1, error=1e-3) for s in
                (56.0, 112.0, 168.0, 224.0, 280.0, 350.0, 375.0, 395.0)]
        hold = dataclasses.replace(creep, stress33=395.0, error=1e-3)
        return ramp + [dataclasses.replace(hold, tdot=t, tdotmin=t / 2, nsteps=max(1, (increments - 8) // 4))
                       for t in (120.0, 1200.0, 4800.0, 20000.0)]
    return [creep]


def _write_deck(root, n, grains, seed, law, nrs, increments, systems=12, phase2="", material=None, loading=None):
    root = Path(root)
    root.mkdir(parents=True, exist_ok=True)
    grain, phase, euler = _polycrystal(n, grains, seed, phase2)
    _write_micro(root / "micro.dat", grain, phase, euler)
    material = material or _material(law, nrs, systems)
    decks.write_cuel(root / "cuel.sx", material)
    decks.write_cupl2(root / "cupl2.sx", material)
    second, complgas = None, 0.0
    if phase2:
        decks.write_cuel(root / "cuel2.sx", iso=1, young=400000.0, nu=0.3)
        decks.write_cupl2(root / "cupl2_2.sx", dataclasses.replace(material, tau0f=1e8, tau0b=1e8))
        second = (int(phase2 == "gas"), root / "cupl2_2.sx", root / "cuel2.sx")
        complgas = 1.0 if phase2 == "gas" else 0.0
    decks.write_fft_in(root / "fft.in", n, root / "micro.dat", root / "cupl2.sx", root / "cuel.sx",
                       loading or _loading(law, increments), phase2=second, complgas=complgas)
    return root / "fft.in"


def _mixed_decks(case, root, seed):
    """The decks of a batch or of a served stream: one grid edge each, material and stress drawn as the
    sweep (tau0, n, theta0) or the stream (temperature-scaled rate, stress) draws them."""
    rng = np.random.default_rng([seed, 17])
    out = []
    for i, e in enumerate(int(x) for x in case["edges"].split()):
        if case["law"] == "stream":
            temp = (475.0, 525.0, 575.0)[i % 3]
            gamd0 = 1e-3 * math.exp(-decks.ARRHENIUS_Q / decks.GAS_R * (1.0 / temp - 1.0 / 525.0))
            mat, stress = decks.Material(nrs=10.0, gamd0=gamd0), float(rng.uniform(140.0, 160.0))
        else:
            tau0 = 80.0 + 15.0 * i
            mat = decks.Material(nrs=float(rng.uniform(8.0, 12.0)), tau0f=tau0, tau0b=tau0, thet0=400.0 + 100.0 * i)
            stress = 120.0
        load = [decks.Loading(kind="creep", stress33=stress, udot33=1e-4, tdot=10.0, nsteps=case["increments"])]
        out.append(_write_deck(Path(root) / str(i), (e, e, e), min(120, e ** 3 // 64), seed * 100 + i, "", 0.0, 0,
                               material=mat, loading=load))
    return out


def _medium():
    """Stiffness and compliance (3x3x3x3) of a cubic reference medium, twice the crystal's stiffness."""
    m = decks.Material()
    c6 = np.zeros((6, 6))
    c6[:3, :3] = m.c12
    c6[[0, 1, 2], [0, 1, 2]] = m.c11
    c6[[3, 4, 5], [3, 4, 5]] = m.c44
    c6 *= 2.0
    s6 = np.linalg.inv(c6)
    ij = {(0, 0): 0, (1, 1): 1, (2, 2): 2, (1, 2): 3, (0, 2): 4, (0, 1): 5}
    at = np.array([[ij[tuple(sorted((i, j)))] for j in range(3)] for i in range(3)])
    c4, s4 = np.zeros((3, 3, 3, 3)), np.zeros((3, 3, 3, 3))
    for i in range(3):
        for j in range(3):
            for k in range(3):
                for q in range(3):
                    a, b = at[i, j], at[k, q]
                    c4[i, j, k, q] = c6[a, b]
                    s4[i, j, k, q] = s6[a, b] / ((2.0 if a > 2 else 1.0) * (2.0 if b > 2 else 1.0))
    return c4, s4


def _polarization(case, seed):
    """A stress polarization: one tensor per grain of a polycrystal, plus a little scatter inside."""
    n = (case["n1"], case["n2"], case["n3"])
    grain, _, _ = _polycrystal(n, 64, seed, "")
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    per = 50.0 * torch.randn(9, 65, dtype=torch.float64, device="cuda", generator=g)
    at = torch.from_numpy(np.ascontiguousarray(grain.transpose(2, 1, 0)).reshape(-1)).cuda()
    return (per[:, at] + torch.randn(9, at.numel(), dtype=torch.float64, device="cuda", generator=g)).contiguous()


class _State(dict):
    """What a program keeps between calls; its files, handles and server go with it."""

    def __del__(self):
        try:
            for key in ("solve", "server"):
                if self.get(key) is not None:
                    self[key].close()
        except TypeError:  # at the interpreter's end, when the modules are gone
            pass


def _results(out):
    """results.csv without its wall-clock column; the text has eight digits, which single precision holds."""
    rows = np.loadtxt(Path(out) / "results.csv", delimiter=",", skiprows=1, ndmin=2)
    return np.delete(rows, 4, axis=1).astype(np.float32)


def prepare(case, seed):
    state = _State(case=case)
    if case["kind"] == "green":
        state["tau"] = _polarization(case, seed)
        state["out"] = torch.empty_like(state["tau"])
        state["c0"], state["s0"] = (np.ascontiguousarray(a.reshape(-1)) for a in _medium())
        return state
    state["dir"] = tempfile.TemporaryDirectory(prefix="evp_case_")
    root = state["dir"].name
    if case["kind"] in ("batch", "serve"):
        state["decks"] = _mixed_decks(case, root, seed)
        state["outs"] = [str(Path(root) / str(i) / "out") + "/" for i in range(len(state["decks"]))]
        if case["kind"] == "serve":
            state["server"] = Server()
        return state
    steps = case["increments"] if case["kind"] != "inc" else 100000
    state["fft"] = _write_deck(root, (case["n1"], case["n2"], case["n3"]), case["grains"], seed, case["law"], case["nrs"],
                               steps, case.get("systems", 12), case.get("phase2", ""))
    state["out"] = str(Path(root) / "out") + "/"
    if case["kind"] == "inc":
        state["solve"] = Solve(state["fft"], mix=1, modal=case["modal"], precision=case["precision"])
        state["solve"].advance(case["warm"])
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "green":
        lib = _lib.load()
        call = lib.evp_green_apply if case["alloc"] else lib.evp_green_apply_noalloc
        dp = ctypes.POINTER(ctypes.c_double)
        _lib.check(call(ctypes.c_void_p(state["tau"].data_ptr()), ctypes.c_void_p(state["out"].data_ptr()), case["n1"],
                        case["n2"], case["n3"], state["c0"].ctypes.data_as(dp), state["s0"].ctypes.data_as(dp),
                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["out"]
    if case["kind"] == "inc":
        s = state["solve"]
        if s.advance(case["increments"]) != case["increments"]:
            raise RuntimeError("the deck has ended")
        row = np.delete(s.rows()[0], 4)  # without the wall-clock column
        sg = s.field("sg")
        # a mixed-precision solve's results have single precision
        return {"row": row, "sg": sg} if not case["precision"] else {"row": row.astype(np.float32), "sg": sg.astype(np.float32)}
    if case["kind"] == "solve":
        with Solve(state["fft"], mix=1, modal=0) as s:
            rows = []
            while s.advance(1) == 1:
                rows.append(np.delete(s.rows()[0], 4))
            return {"rows": np.array(rows), "sg": s.field("sg"), "defgrad": s.field("defgrad")}
    if case["kind"] == "file":
        rep = run_solver(state["fft"], state["out"], mix=1, modal=0)
        return {"results": _results(state["out"]), "macrosteps": rep.macrosteps}
    if case["kind"] == "batch":
        reps = solve_files(state["decks"], state["outs"], csv_only=True, precision=case["precision"])
        status = [r.status for r in reps]
    else:
        srv = state["server"]
        tickets = [srv.submit(f, o, csv_only=True, precision=case["precision"]) for f, o in zip(state["decks"], state["outs"])]
        status = [srv.wait(t)["status"] for t in tickets]
    return {"status": status, "results": [_results(o) for o in state["outs"]]}


# ---------------------------------------------------------------- what a pass cannot do without
def _iterations(law):
    """Equilibrium iterations of one increment, about, of each loading at its tolerance."""
    return {"tension": 18.0, "creep": 19.0, "stream": 22.0, "ramp": 16.0}[law]


def work(case):
    if case["kind"] == "green":
        vox = case["n1"] * case["n2"] * case["n3"]
        return {"bytes": 2 * 9 * 8.0 * vox, "flops": 2 * 9 * 2.5 * vox * math.log2(vox)}
    if case["kind"] in ("batch", "serve"):
        vox = sum(int(e) ** 3 for e in case["edges"].split())
    else:
        vox = case["n1"] * case["n2"] * case["n3"]
    systems = case.get("systems", 12)
    its = _iterations(case["law"]) * case["increments"]
    return {"bytes": vox * (its * (ITER_BYTES + ITER_BYTES_PER_SYSTEM * systems) + case["increments"] * INC_BYTES),
            "flops": vox * its * (ITER_FLOPS_PER_SYSTEM * systems + 2 * 9 * 2.5 * math.log2(vox))}


def exact(case, seed):
    """The Green operator's result in 64 bits by torch's transforms (even grids; the operator of an odd axis
    follows the solver's own frequency convention).  A whole solve has no such value at hand."""
    n = (case.get("n1", 1), case.get("n2", 1), case.get("n3", 1))
    if case["kind"] != "green" or any(m % 2 for m in n):
        return None
    c4, s4 = (torch.from_numpy(a).cuda() for a in _medium())
    tau = _polarization(case, seed).reshape(9, n[2], n[1], n[0])  # [component, z, y, x]
    k = [torch.arange(m, device="cuda") for m in (n[2], n[1], n[0])]
    xi = [2.0 * math.pi * torch.where(a < m // 2, a, a - m).double() / m for a, m in zip(k, (n[2], n[1], n[0]))]
    spec = torch.fft.fftn(tau, dim=(1, 2, 3)).reshape(3, 3, n[2], n[1], n[0])
    z, y, x = torch.meshgrid(*xi, indexing="ij")
    w = torch.stack([x, y, z])
    acoustic = torch.einsum("ijkl,jzyx,lzyx->zyxik", c4, w, w)
    acoustic[0, 0, 0] = torch.eye(3, dtype=torch.float64, device="cuda")
    inv = torch.linalg.inv(acoustic).to(torch.complex128)
    p = torch.einsum("klzyx,lzyx->kzyx", spec, w.to(torch.complex128))
    res = -torch.einsum("zyxik,kzyx,jzyx->ijzyx", inv, p, w.to(torch.complex128))
    nyq = (k[0] == n[2] // 2)[:, None, None] | (k[1] == n[1] // 2)[None, :, None] | (k[2] == n[0] // 2)[None, None, :]
    on_nyq = -torch.einsum("pqij,ijzyx->pqzyx", s4.to(torch.complex128), spec)
    res = torch.where(nyq, on_nyq, res)
    res[:, :, 0, 0, 0] = 0.0
    return torch.fft.ifftn(res.reshape(9, n[2], n[1], n[0]), dim=(1, 2, 3)).real.reshape(9, -1).contiguous()
