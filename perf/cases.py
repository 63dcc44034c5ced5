"""Performance cases of the FDTD stage: the work a user of the library has it
do, through its public entry points.

Kinds (the "kind" of a case):
  echo     rfsyn's drop-in call, fdtd_simulate_echo: one FP64 run of an empty
           box from configuration to series, creation and read-back included.
  sim      a resident session: the scene stays on the device, a pass rewinds
           it, advances "steps" time steps and reads series and spectra
           (with "iq" also the stage's noisy output signal of probe 0).
           FP32 or FP64, any size, CPML on the axes that are not periodic.
  cell     a session of the periodic unit cell: plane wave through a TF/SF
           boundary, smoothed anisotropic slab, Lorentz layer, plane probes.
  fresh    fdtd_b200_run on a scene with boxes and smoothed spheres: host
           set-up, upload, loop and read-back of every call.
  batch    many small scenes advanced together (a resident batch).
  dataset  the surrogate's data generation and fallback path: scenes in,
           transfer functions out, batch creation included.
  train    Adam steps of the surrogate's network, weights read back.
  predict  the network's outputs for rows on the host.

Step counts are cut so that a pass stays short; the work per step is that of
a full-length run.  A session's pass starts from zero fields, and its first
steps spread from the source, but every step of the loop moves the same bytes
and executes the same operations whatever the fields hold.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rfsyn_b200 as rb
from rfsyn_b200 import scenes, surrogate

EPS0, MU0, C0 = rb.EPS0, rb.MU0, rb.C0


def listed():
    return [
        # rfsyn's own unit-test size through the drop-in call: the smallest run
        # a user of rfsyn makes, bound by latency, launches and set-up
        {"name": "echo_50_fp64", "kind": "echo", "n": 50, "steps": 200, "npml": 8},
        # the plain 64^3 vacuum scene in FP64 (the precision rfsyn computes
        # in), with the stage's I/Q output
        {"name": "c1_64_fp64_iq", "kind": "sim", "nx": 64, "ny": 64, "nz": 64, "npml": 10, "periodic": 0, "fp64": True,
         "boxes": 0, "spheres": 0, "debye": 0, "probes": 4, "bins": 64, "steps": 240, "iq": True},
        # a small ragged FP32 scene with a few scatterers, one at a time
        {"name": "small_47x53x61_fp32", "kind": "sim", "nx": 47, "ny": 53, "nz": 61, "npml": 8, "periodic": 0,
         "fp64": False, "boxes": 3, "spheres": 2, "debye": 0, "probes": 8, "bins": 128, "steps": 240, "iq": False},
        # an ordinary FP64 scene with smoothed spheres, ragged
        {"name": "mid_150x131x170_fp64", "kind": "sim", "nx": 150, "ny": 131, "nz": 170, "npml": 10, "periodic": 0,
         "fp64": True, "boxes": 2, "spheres": 8, "debye": 0, "probes": 16, "bins": 128, "steps": 64, "iq": False},
        # an FP32 cell periodic in x and y, odd sizes, CPML in z only
        {"name": "periodic_77x91x203_fp32", "kind": "sim", "nx": 77, "ny": 91, "nz": 203, "npml": 12, "periodic": 3,
         "fp64": False, "boxes": 5, "spheres": 0, "debye": 0, "probes": 16, "bins": 128, "steps": 96, "iq": False},
        # the headline scene: 256^3 FP32, 24 dielectric and 3 Debye spheres
        {"name": "c2_256_fp32", "kind": "sim", "nx": 256, "ny": 256, "nz": 256, "npml": 12, "periodic": 0,
         "fp64": False, "boxes": 0, "spheres": 24, "debye": 3, "probes": 16, "bins": 256, "steps": 96, "iq": False},
        # the periodic unit cell at the benchmark's size
        {"name": "c3_cell_128x128x512", "kind": "cell", "nx": 128, "ny": 128, "nz": 512, "steps": 96},
        # a new scene per call: set-up, sphere rasteriser, upload, loop, read
        {"name": "fresh_96_fp32", "kind": "fresh", "nx": 96, "ny": 96, "nz": 96, "npml": 10, "boxes": 2, "spheres": 6,
         "probes": 4, "bins": 64, "steps": 400},
        # scenes of 32-96 cells per axis advanced together
        {"name": "c4_batch_96", "kind": "batch", "scenes": 96, "lo": 32, "hi": 96, "geometry": 4, "steps": 96},
        # surrogate data generation / fallback on 48^3 scenes
        {"name": "c5_dataset_24", "kind": "dataset", "scenes": 24, "steps": 400},
        # surrogate training and inference at the benchmark's network
        {"name": "c5_train_256", "kind": "train", "rows": 5000, "batch": 256, "steps": 60, "width": 512, "depth": 4},
        {"name": "c5_predict_2000", "kind": "predict", "rows": 2000, "width": 512, "depth": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["echo", "sim", "sim", "sim", "sim", "cell", "fresh", "batch", "dataset", "train", "predict"])
    if kind == "echo":
        n = rng.randint(24, 80)
        return {"kind": kind, "n": n, "steps": rng.randint(50, 300), "npml": rng.randint(4, 10)}
    if kind == "sim":
        fp64 = rng.random() < 0.4
        periodic = rng.choice([0, 0, 0, 3, 1, 4, 6, 7])
        dims = [_log_int(rng, 32, 240) for _ in range(3)]
        cells = dims[0] * dims[1] * dims[2]
        steps = max(16, min(400, int(1.2e9 * (0.4 if fp64 else 1.0) / cells)))
        plain = periodic != 0 or min(dims) < 44
        return {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "npml": rng.randint(4, 12),
                "periodic": periodic, "fp64": fp64, "boxes": rng.randint(0, 6), "spheres": 0 if plain else
                rng.randint(0, 12), "debye": 0 if plain else rng.randint(0, 2), "probes": rng.randint(1, 32),
                "bins": rng.choice([16, 64, 100, 256]), "steps": steps, "iq": rng.random() < 0.3}
    if kind == "cell":
        nx, ny, nz = rng.randint(24, 120), rng.randint(24, 120), rng.randint(200, 500)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(24, 90)}
    if kind == "fresh":
        n = [_log_int(rng, 48, 128) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "npml": rng.randint(6, 10), "boxes": rng.randint(0, 4),
                "spheres": rng.randint(1, 8), "probes": rng.randint(1, 8), "bins": 64, "steps": rng.randint(100, 400)}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 4, 96), "lo": 32, "hi": rng.randint(48, 96),
                "geometry": rng.randint(10, 10000), "steps": rng.randint(24, 96)}
    if kind == "dataset":
        return {"kind": kind, "scenes": rng.randint(4, 24), "steps": rng.randint(100, 400)}
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 600, 5000), "batch": 64 * rng.randint(1, 8),
                "steps": rng.randint(10, 60), "width": 64 * rng.randint(2, 8), "depth": rng.randint(2, 5)}
    return {"kind": kind, "rows": _log_int(rng, 1, 3000), "width": 64 * rng.randint(2, 8), "depth": rng.randint(2, 5)}


# ---- scenes -----------------------------------------------------------------


def _workload(case, seed):
    """The "sim" / "fresh" scene of the case: size, probe count and source
    position from the case, materials and probe positions from the seed."""
    n = (case["nx"], case["ny"], case["nz"])
    npml, periodic = case["npml"], case.get("periodic", 0)
    rng = scenes.Pcg32(seed, 7)
    margin = [2 if (periodic >> a) & 1 else npml + 2 for a in range(3)]
    boxes, spheres = [], []
    for _ in range(case["boxes"]):
        b = []
        for a in range(3):
            side = rng.randint(3, max(4, min(24, n[a] - 2 * margin[a])))
            a0 = rng.randint(margin[a], max(margin[a] + 1, n[a] - margin[a] - side + 1))
            b += [a0, a0 + side]
        boxes.append((*b, rng.range(1.5, 10.0), rng.log_range(1e-4, 1e-1)))
    top = min(n[a] - 2 * margin[a] for a in range(3)) / 2.0 - 1.0
    for q in range(case["spheres"] + case.get("debye", 0)):
        r = rng.range(3.0, max(3.1, min(30.0, top)))
        c = [rng.range(margin[a] + r, n[a] - margin[a] - r) for a in range(3)]
        if q < case["spheres"]:
            spheres.append((*c, r, rng.range(1.5, 12.0), rng.log_range(1e-4, 1e-1), None))
        else:
            spheres.append((*c, r, 1.0, 0.0, (rng.range(2.0, 4.0), 0.0,
                                              [("debye", rng.range(5.0, 60.0), rng.log_range(1e-11, 1e-9))])))
    probes = [dict(i=rng.randint(1, n[0]), j=rng.randint(1, n[1]), k=rng.randint(1, n[2]),
                   component=[rb.FIELD_EZ, rb.FIELD_EX, rb.FIELD_HY][q % 3]) for q in range(case["probes"])]
    # a probe a few cells from the source, where every run records a signal
    probes[0] = dict(i=n[0] // 2 + 3, j=n[1] // 2 - 2, k=n[2] // 2 + 2, component=rb.FIELD_EZ)
    tau = 2.0 / (math.pi * 16e9)
    return scenes.Workload(
        name="case", nx=n[0], ny=n[1], nz=n[2], dx=1e-3, n_steps=case["steps"], npml=npml, periodic=periodic,
        precision=rb.FP64 if case.get("fp64") else rb.FP32,
        sources=[dict(i=n[0] // 2, j=n[1] // 2, k=n[2] // 2, component=rb.FIELD_EZ, mode=0,
                      amplitude=rng.range(0.5, 2.0), waveform=rb.WAVE_MOD_GAUSSIAN, p0=20e9, p1=1.5 * tau, p2=tau)],
        probes=probes, freqs=list(np.linspace(4e9, 36e9, case["bins"])), boxes=boxes, spheres=spheres)


def _cell(case, seed):
    return scenes.c3(seed=seed, nx=case["nx"], ny=case["ny"], nz=case["nz"], n_steps=case["steps"])


def _batch(case, seed):
    """Scene sizes from the case, scatterers and positions from the seed."""
    out = []
    sizes = scenes.c4(seed=case["geometry"], n_scenes=case["scenes"], lo=case["lo"], hi=case["hi"],
                      n_steps=case["steps"])
    for s, w in enumerate(sizes):
        rng = scenes.Pcg32(seed, s)
        dims = (w.nx, w.ny, w.nz)
        w.boxes, w.spheres = scenes.draw_scatterers(rng, dims, w.npml)
        w.sources = [dict(w.sources[0], amplitude=rng.range(0.5, 2.0), p1=0.4 * w.sources[0]["p1"])]
        src = w.sources[0]
        near = dict(i=src["i"] - 2, j=src["j"] + 2, k=src["k"] - 1, component=rb.FIELD_EZ)
        w.probes = [near] + [dict(i=rng.randint(1, w.nx), j=rng.randint(1, w.ny), k=rng.randint(1, w.nz),
                                  component=rb.FIELD_EZ) for _ in range(3)]
        out.append(w)
    return out


def _echo(case, seed):
    rng = scenes.Pcg32(seed, 3)
    c = rb.FdtdSimConfig()
    n = case["n"]
    c.nx = c.ny = c.nz = n
    c.dx, c.courant_safety, c.n_steps, c.npml = 1e-3, 0.99, case["steps"], case["npml"]
    c.src_i = c.src_j = c.src_k = n // 2
    c.src_component = rb.FIELD_EZ
    c.t0_over_dt, c.tau_over_dt = rng.range(20.0, 40.0), rng.range(6.0, 10.0)
    c.probe_i, c.probe_j, c.probe_k = rng.randint(n // 2 + 1, n - 1), n // 2, rng.randint(n // 2, n - 1)
    c.probe_component = rb.FIELD_EZ
    return c


class _Net:
    """The network's parameters, inputs and targets, from the seed."""

    def __init__(self, case, seed):
        r = np.random.RandomState(seed % (1 << 31))
        self.n_in, self.width, self.depth = surrogate.N_FEAT, case["width"], case["depth"]
        self.n_out = 2 * surrogate.N_BINS
        kin = (self.n_in + 63) // 64 * 64
        self.kin = kin
        self.shapes = []
        parts = []
        for q in range(self.depth + 1):
            i, o = (kin if q == 0 else self.width), (self.n_out if q == self.depth else self.width)
            w = (r.uniform(-1, 1, (o, i)) * math.sqrt(6.0 / (self.n_in if q == 0 else i)) *
                 (0.5 if q == self.depth else 1.0)).astype(np.float32)
            if q == 0:
                w[:, self.n_in:] = 0.0
            b = (0.01 * r.randn(o)).astype(np.float32)
            self.shapes.append((o, i))
            parts += [w.ravel(), b]
        self.params = np.concatenate(parts)
        self.X = r.uniform(-1, 1, (case["rows"], self.n_in)).astype(np.float32)
        f = r.randn(self.n_in, self.n_out).astype(np.float32) / math.sqrt(self.n_in)
        self.Y = np.sin(3.0 * (self.X @ f)).astype(np.float32)
        self.seed = int(r.randint(1, 1 << 30))


# ---- what a user's program has in hand, and one pass -------------------------


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "echo":
        st["cfg"] = _echo(case, seed)
    elif kind in ("sim", "cell"):
        w = _cell(case, seed) if kind == "cell" else _workload(case, seed)
        st["setup"] = scenes.scene_setup(w)
        st["sim"] = rb.Sim(scenes.run_config(w), st["setup"].ptr if st["setup"] else None)
        st["noise_seed"] = seed
    elif kind == "fresh":
        w = _workload(case, seed)
        st["setup"] = scenes.scene_setup(w)
        st["rc"] = scenes.run_config(w)
    elif kind == "batch":
        ws = _batch(case, seed)
        st["setups"] = [scenes.scene_setup(w) for w in ws]
        st["batch"] = rb.Batch([scenes.run_config(w) for w in ws], [s.ptr if s else None for s in st["setups"]])
    elif kind == "dataset":
        st["ws"] = surrogate.c5_scenes(seed, case["scenes"], n_steps=case["steps"])
    else:
        net = _Net(case, seed)
        st["net"] = net
        st["mlp"] = rb.Mlp(net.n_in, net.width, net.depth, net.n_out)
        st["mlp"].set_params(net.params)
        if kind == "train":
            st["mlp"].set_data(net.X, net.Y)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "echo":
        rc, td, fs = rb.simulate_echo(state["cfg"])
        if rc != 0:
            raise RuntimeError(rb.last_error())
        return {"td": td, "fs": fs}
    if kind in ("sim", "cell"):
        sim = state["sim"]
        sim.reset()
        sim.advance(case["steps"])
        out = {"td": sim.probes(), "dft": sim.dft()}
        if case.get("iq"):
            out["iq"] = sim.read_iq(0, snr_db=20.0, seed=state["noise_seed"])
        return out
    if kind == "fresh":
        got = rb.run(state["rc"], state["setup"].ptr if state["setup"] else None)
        return {"td": got["td"], "dft": got["dft"], "fs": got["fs"]}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        b.advance(case["steps"])
        n = case["scenes"]
        return {"td": np.concatenate([b.probes(s) for s in range(n)]),
                "dft": np.concatenate([b.dft(s) for s in range(n)])}
    if kind == "dataset":
        X, H = surrogate.transfer_functions(state["ws"])
        return {"X": X, "H": H}
    net, mlp = state["net"], state["mlp"]
    if kind == "train":
        loss = mlp.train(case["steps"], batch=case["batch"], lr=1e-3, seed=net.seed)
        return {"loss": loss, "params": mlp.params()}
    return {"Y": mlp.predict(net.X)}


# ---- the work a pass cannot do without ----------------------------------------


def _loop_work(dims, npml, periodic, esz, steps):
    """Every step reads and writes six components per cell once, reads a
    one-byte material code, and reads and writes four CPML memory values per
    (cell, absorbing axis)."""
    cells = dims[0] * dims[1] * dims[2]
    slab = sum(2 * npml * cells // dims[a] for a in range(3) if npml and not (periodic >> a) & 1)
    return steps * (cells * (12 * esz + 1) + slab * 8 * esz), steps * (cells * 33.0 + slab * 28.0)


def work(case):
    kind = case["kind"]
    if kind == "echo":
        b, f = _loop_work((case["n"],) * 3, case["npml"], 0, 8, case["steps"])
    elif kind in ("sim", "fresh"):
        b, f = _loop_work((case["nx"], case["ny"], case["nz"]), case["npml"], case.get("periodic", 0),
                          8 if case.get("fp64") else 4, case["steps"])
    elif kind == "cell":
        b, f = _loop_work((case["nx"], case["ny"], case["nz"]), 16, 3, 4, case["steps"])
    elif kind == "batch":
        b = f = 0.0
        for w in scenes.c4(seed=case["geometry"], n_scenes=case["scenes"], lo=case["lo"], hi=case["hi"]):
            wb, wf = _loop_work((w.nx, w.ny, w.nz), w.npml, 0, 4, case["steps"])
            b, f = b + wb, f + wf
    elif kind == "dataset":
        b, f = _loop_work((48, 48, 48), 8, 0, 4, case["steps"])
        b, f = b * case["scenes"], f * case["scenes"]
    else:
        w, d, n_out = case["width"], case["depth"], 2 * surrogate.N_BINS
        weights = 64 * w + (d - 1) * w * w + w * n_out
        if kind == "train":
            # per step: weights and both moments read and written, the
            # minibatch's rows read; three products per layer
            rows = case["batch"] * (2 * 64 + 4 * n_out)
            b, f = case["steps"] * (24.0 * weights + rows), case["steps"] * 6.0 * weights * case["batch"]
        else:
            b, f = 2.0 * weights + case["rows"] * 4.0 * (surrogate.N_FEAT + n_out), 2.0 * weights * case["rows"]
    return {"bytes": float(b), "flops": float(f)}


# ---- 64-bit values ------------------------------------------------------------


def _profiles(n, dx, dt, npml, absorbing, dev, m=3.0, ma=1.0, kappa_max=7.0, alpha_max=0.05, r0=1e-6):
    """CPML triples (1/kappa, b, a) at integer (n + 1) and half (n) positions."""
    out = []
    for pos in (np.arange(n + 1) * dx, (np.arange(n) + 0.5) * dx):
        kinv, b, a = np.ones(len(pos)), np.ones(len(pos)), np.zeros(len(pos))
        if absorbing:
            d, length = npml * dx, n * dx
            smax = -(m + 1.0) * math.log(r0) / (2.0 * math.sqrt(MU0 / EPS0) * npml * dx)
            rho = np.where(pos < d, d - pos, np.where(pos > length - d, pos - (length - d), -1.0))
            on = rho >= 0.0
            r = np.clip(rho / d, 0.0, 1.0)
            sig, kap = smax * r ** m, 1.0 + (kappa_max - 1.0) * r ** m
            alp = alpha_max * (1.0 - r) ** ma
            bb = np.exp(-(sig / kap + alp) * dt / EPS0)
            den = np.where(sig > 0, dx * kap * (sig + kap * alp), 1.0)
            aa = np.where(sig > 0, sig * (bb - 1.0) / den, 0.0)
            kinv, b, a = np.where(on, 1.0 / kap, 1.0), np.where(on, bb, 1.0), np.where(on, aa, 0.0)
        out.append([torch.tensor(x, device=dev, dtype=torch.float64) for x in (kinv, b, a)])
    return out


def _fraction(sp, c, lo, hi, dev):
    """Fill fraction (8^3 lattice) of the unit cube around each E_c sample of
    the box [lo, hi] in the sphere, and the squared normal component."""
    pos = []
    for a in range(3):
        q = torch.arange(lo[a], hi[a] + 1, device=dev, dtype=torch.float64) + (0.5 if a == c else 0.0) - sp[a]
        sh = [1, 1, 1]
        sh[a] = -1
        pos.append(q.reshape(sh))
    d = torch.sqrt(pos[0] ** 2 + pos[1] ** 2 + pos[2] ** 2)
    n2 = torch.where(d > 0, (pos[c] / torch.where(d > 0, d, 1.0)) ** 2, 0.0)
    count = torch.zeros_like(d)
    for a in range(8):
        px = (pos[0] + ((a + 0.5) / 8.0 - 0.5)) ** 2
        for b in range(8):
            pxy = px + (pos[1] + ((b + 0.5) / 8.0 - 0.5)) ** 2
            for e in range(8):
                count += (pxy + (pos[2] + ((e + 0.5) / 8.0 - 0.5)) ** 2 <= sp[3] * sp[3])
    h = 0.8660254037844386
    f = torch.where(d + h <= sp[3], 1.0, torch.where(d - h >= sp[3], 0.0, count / 512.0))
    return f, n2


def _materials(w, dev):
    """eps_r and sigma of every E sample (boxes, then spheres smoothed at
    their surfaces), and the dispersive samples as (mask, model) pairs."""
    shape = (3, w.nx + 1, w.ny + 1, w.nz + 1)
    eps = torch.ones(shape, device=dev, dtype=torch.float64)
    sig = torch.zeros(shape, device=dev, dtype=torch.float64)
    bg_e, bg_s = torch.ones(shape[1:], device=dev, dtype=torch.float64), torch.zeros(shape[1:], device=dev,
                                                                                    dtype=torch.float64)
    which = torch.full(shape, -1, device=dev, dtype=torch.int64)
    models = []
    for (i0, i1, j0, j1, k0, k1, e, s) in w.boxes:
        eps[:, i0:i1, j0:j1, k0:k1], sig[:, i0:i1, j0:j1, k0:k1] = e, s
        bg_e[i0:i1, j0:j1, k0:k1], bg_s[i0:i1, j0:j1, k0:k1] = e, s
    n = (w.nx, w.ny, w.nz)
    for sp in w.spheres:
        lo = [max(0, math.floor(sp[a] - sp[3]) - 2) for a in range(3)]
        hi = [min(n[a], math.ceil(sp[a] + sp[3]) + 2) for a in range(3)]
        box = tuple(slice(lo[a], hi[a] + 1) for a in range(3))
        fr = [_fraction(sp, c, lo, hi, dev) for c in range(3)]
        full = (fr[0][0] == 1) & (fr[1][0] == 1) & (fr[2][0] == 1)
        if sp[6] is not None:
            models.append(sp[6])
        for c in range(3):
            f, n2 = fr[c]
            v = which[(c, *box)]
            if sp[6] is not None:
                which[(c, *box)] = torch.where(full | (f >= 0.5), len(models) - 1, v)
                continue
            eb, sb = bg_e[box], bg_s[box]
            mean, minv = f * sp[4] + (1 - f) * eb, f / sp[4] + (1 - f) / eb
            es = 1.0 / (n2 * minv + (1.0 - n2) / mean)
            ss = f * sp[5] + (1 - f) * sb
            touched = f > 0
            eps[(c, *box)] = torch.where(f == 1, sp[4], torch.where(touched, es, eps[(c, *box)]))
            sig[(c, *box)] = torch.where(f == 1, sp[5], torch.where(touched, ss, sig[(c, *box)]))
            which[(c, *box)] = torch.where(touched, -1, v)
        if sp[6] is None:
            bg_e[box] = torch.where(full, sp[4], bg_e[box])
            bg_s[box] = torch.where(full, sp[5], bg_s[box])
    return eps, sig, which, models


def _wave(s, t):
    u = (t - s["p1"]) / s["p2"]
    return s["amplitude"] * math.exp(-u * u) * math.sin(2.0 * math.pi * s["p0"] * (t - s["p1"]))


def _fdtd64(w, source):
    """Series and spectra of the scene: the Yee loop with CPML, scalar lossy
    media and Debye currents, torch in 64 bits.  source(n): the value added
    before the E update of step n."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, dx, dt = (w.nx, w.ny, w.nz), w.dx, w.dt
    per = [bool((w.periodic >> a) & 1) for a in range(3)]
    shape = tuple(x + 1 for x in n)
    F = [torch.zeros(shape, device=dev, dtype=torch.float64) for _ in range(6)]
    prof = [_profiles(n[a], dx, dt, w.npml, w.npml > 0 and not per[a], dev) for a in range(3)]
    eps, sig, which, models = _materials(w, dev)
    loss = sig * dt / (2.0 * eps * EPS0)
    ca, cb = (1 - loss) / (1 + loss), dt / (eps * EPS0 * dx) / (1 + loss)
    cbh = dt / (MU0 * dx)
    # swept ranges: H_c over [0, n) on every axis but its own, where it also
    # has the boundary sample; E_c from 1 on closed axes other than its own
    hr = [tuple(slice(0, n[a] + (1 if a == c and not per[a] else 0)) for a in range(3)) for c in range(3)]
    er = [tuple(slice(0 if a == c or per[a] else 1, n[a]) for a in range(3)) for c in range(3)]

    def diff(f, axis, rng, forward):
        lo, hi = rng[axis].start, rng[axis].stop
        here = list(rng)
        there = list(rng)
        if forward:
            there[axis] = slice(lo + 1, hi + 1)
            if per[axis]:
                q = torch.arange(lo, hi, device=dev)
                return f[tuple(rng[a] if a != axis else slice(None) for a in range(3))].index_select(
                    axis, (q + 1) % n[axis]) - f[tuple(here)]
            return f[tuple(there)] - f[tuple(here)]
        if per[axis]:
            q = torch.arange(lo, hi, device=dev)
            return f[tuple(here)] - f[tuple(rng[a] if a != axis else slice(None) for a in range(3))].index_select(
                axis, (q - 1) % n[axis])
        there[axis] = slice(lo - 1, hi - 1)
        return f[tuple(here)] - f[tuple(there)]

    psi = {}

    def stretched(key, d, axis, rng, half):
        if not w.npml or per[axis]:
            return d
        sh = [1, 1, 1]
        sh[axis] = -1
        kinv, b, a = (p[rng[axis]].reshape(sh) for p in prof[axis][1 if half else 0])
        p = psi.get(key)
        p = a * d if p is None else b * p + a * d
        psi[key] = p
        return d * kinv + dx * p

    disp = []
    for q, (ei, s0, poles) in enumerate(models):
        de, tau = poles[0][1], poles[0][2]
        den = 1.0 + dt / (2.0 * tau)
        beta = (EPS0 * de * dt / tau) / den
        kj, ke, hb = (1.0 - dt / (2.0 * tau)) / den, beta / dt, 0.5 * beta
        A = EPS0 * ei + 0.5 * s0 * dt + hb
        rec = ((EPS0 * ei - 0.5 * s0 * dt + hb) / A, dt / (A * dx), 0.5 * dt * (1.0 + kj) / A, kj, ke)
        for c in range(3):
            mask = which[(c, *er[c])] == q
            if bool(mask.any()):
                disp.append((c, mask, rec, torch.zeros(int(mask.sum()), device=dev, dtype=torch.float64)))
    td = torch.zeros((len(w.probes), w.n_steps), device=dev, dtype=torch.float64)
    src = w.sources[0]
    for step in range(w.n_steps):
        new = []
        for c in range(3):
            p, q = (c + 1) % 3, (c + 2) % 3  # curl: d_p E_q - d_q E_p
            dA = stretched(("h", c, p), diff(F[q], p, hr[c], True), p, hr[c], True)
            dB = stretched(("h", c, q), diff(F[p], q, hr[c], True), q, hr[c], True)
            new.append(F[3 + c][hr[c]] - cbh * (dA - dB))
        for c in range(3):
            F[3 + c][hr[c]] = new[c]
        F[src["component"]][src["i"], src["j"], src["k"]] += source(step)
        for c in range(3):
            p, q = (c + 1) % 3, (c + 2) % 3
            dA = stretched(("e", c, p), diff(F[3 + q], p, er[c], False), p, er[c], False)
            dB = stretched(("e", c, q), diff(F[3 + p], q, er[c], False), q, er[c], False)
            curl, old = dA - dB, F[c][er[c]]
            e = ca[(c, *er[c])] * old + cb[(c, *er[c])] * curl
            for m, (dc, mask, rec, J) in enumerate(disp):
                if dc != c:
                    continue
                v = old[mask]
                en = rec[0] * v + rec[1] * curl[mask] - rec[2] * J
                disp[m] = (dc, mask, rec, rec[3] * J + rec[4] * (en - v))
                e[mask] = en
            F[c][er[c]] = e
        for r, pr in enumerate(w.probes):
            td[r, step] = F[pr["component"]][pr["i"], pr["j"], pr["k"]]
    t = (torch.arange(w.n_steps, device=dev, dtype=torch.float64) + 1.0) * dt
    out = {"td": td.cpu().numpy()}
    if w.freqs:
        ph = 2.0 * math.pi * torch.tensor(w.freqs, device=dev, dtype=torch.float64)[:, None] * t[None, :]
        dft = torch.complex(td @ torch.cos(ph).T * dt, -(td @ torch.sin(ph).T) * dt)
        out["dft"] = dft.cpu().numpy()
    return out


def _gelu(x):
    return 0.5 * x * (1.0 + torch.erf(x / math.sqrt(2.0)))


def _unpack(net, params):
    layers, o = [], 0
    for (r, c) in net.shapes:
        layers.append([params[o:o + r * c].reshape(r, c), params[o + r * c:o + r * c + r]])
        o += r * c + r
    return layers


def _forward(net, layers, x):
    for q, (W, b) in enumerate(layers):
        x = x @ W.T + b
        if q < len(layers) - 1:
            x = _gelu(x)
    return x


def _shuffles(rows, seed):
    """The training permutations, one per pass over the data (Fisher-Yates on
    splitmix64)."""
    mask = (1 << 64) - 1
    state = seed & mask
    while True:
        perm = list(range(rows))
        for q in range(rows - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            r = (z ^ (z >> 31)) % (q + 1)
            perm[q], perm[r] = perm[r], perm[q]
        yield perm


def _train64(case, net, dev):
    X = torch.zeros((case["rows"], net.kin), device=dev, dtype=torch.float64)
    X[:, :net.n_in] = torch.tensor(net.X, device=dev)
    Y = torch.tensor(net.Y, device=dev, dtype=torch.float64)
    p = torch.tensor(net.params, device=dev, dtype=torch.float64, requires_grad=True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    B, steps, n = case["batch"], case["steps"], case["rows"]
    passes = _shuffles(n, net.seed)
    left, loss = 0, 0.0
    for s in range(steps):
        if left == 0:
            perm, left = next(passes), max(1, n // B)
        left -= 1
        rows = torch.tensor([perm[(s * B + q) % n] for q in range(B)], device=dev)
        out = _forward(net, _unpack(net, p), X[rows])
        se = ((out - Y[rows]) ** 2).mean()
        g, = torch.autograd.grad(se, p)
        loss = float(se)
        with torch.no_grad():
            lr = 1e-3 * 0.5 * (1.0 + math.cos(math.pi * s / steps))
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            step = lr * (m / (1 - 0.9 ** (s + 1))) / (torch.sqrt(v / (1 - 0.999 ** (s + 1))) + 1e-8)
            p = (p - step).requires_grad_(True)
    return {"loss": loss, "params": p.detach().cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cell", "dataset", "batch"):
        # the unit cell's plane wave and anisotropic faces, and scene sets
        # whose loops would take minutes one after the other
        return None
    if kind == "echo":
        c = _echo(case, seed)
        w = scenes.Workload(
            name="echo", nx=c.nx, ny=c.ny, nz=c.nz, dx=c.dx, n_steps=c.n_steps, npml=c.npml,
            sources=[dict(i=c.src_i, j=c.src_j, k=c.src_k, component=c.src_component)],
            probes=[dict(i=c.probe_i, j=c.probe_j, k=c.probe_k, component=c.probe_component)])

        def pulse(step):
            u = (step * w.dt - c.t0_over_dt * w.dt) / (c.tau_over_dt * w.dt)
            return -2.0 * u * math.exp(-u * u)

        return {"td": _fdtd64(w, pulse)["td"][0], "fs": 1.0 / w.dt}
    if kind in ("sim", "fresh"):
        w = _workload(case, seed)
        out = _fdtd64(w, lambda step: _wave(w.sources[0], step * w.dt))
        if case.get("iq"):
            out["iq"] = None  # seeded noise
        if kind == "fresh":
            out["fs"] = 1.0 / w.dt
        return out
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    net = _Net(case, seed)
    if kind == "train":
        return _train64(case, net, dev)
    layers = _unpack(net, torch.tensor(net.params, device=dev, dtype=torch.float64))
    X = torch.zeros((case["rows"], net.kin), device=dev, dtype=torch.float64)
    X[:, :net.n_in] = torch.tensor(net.X, device=dev)
    return {"Y": _forward(net, layers, X).cpu().numpy()}
