"""The measured work of the solver: what a user's program has it do, through its public entry points.

Kinds of case (`kind`), each with the use it stands for:
  frame   one frame of the headless loop: two leapfrog steps, then the probes and the flux box read back
  step    a run of steps on one grid, with the port record, the far-field monitor or the multi-frequency
          far-field DFT attached, under the graded absorber or the convolutional one
  batch   one chunk of the batched antenna sweep: scenes of several sizes in one stack, the chunk's port
          series read back; with `freqs`, scenes of one size with their surface DFT and its spectra
  pattern the phased array's pattern over a whole angle grid at every DFT frequency
  report  the single-frequency pattern of the console report: three cuts and two hemisphere maps
  train   one training step of the learned ring-down extrapolator
  radar   the back-projected image of the pulsed radar

Sizes are those of the repository's own workloads (48 to 512 cells per side) and odd ones between.
Fields start as wave packets in flight, so every pass works on non-zero fields everywhere.
"""
import ctypes as C
import math

import numpy as np
import torch

from em_lab_gb300 import SimulationGrid, abi, configs
from em_lab_gb300.batch import FarField
from em_lab_gb300.extrap import AUX, CONV, ENC, HEAD, OUT, T_IN, Net, init_params, layer_shapes
from em_lab_gb300.grid import SceneStack
from em_lab_gb300.instruments import far_field_directions
from em_lab_gb300.phased import angle_grid
from em_lab_gb300.radar import RadarMonitor
from em_lab_gb300.scene import EnvironmentBuilder, FluxSetup, Material, SourceDesc

F64 = torch.float64
DEV = "cuda"


def listed():
    return [
        # the smallest call: one frame of the headless loop on a small scene (latency, launches, read-backs)
        _frame("frame of a 48 cube", 48, 48, 48, pml=8, steps=2),
        # the point-dipole scene's run: a hundred frames' worth of far-field accumulation is 50 of these steps
        _step("128 cube, far-field monitor", 128, 128, 128, pml=10, steps=50, fill=0.01, ntff=1),
        # an odd, ragged grid with lossy blocks and its feed's record, as a ring-down run steps it
        _step("odd grid, port record", 211, 147, 93, pml=12, steps=40, fill=0.05, record=1),
        # the large workload: 512 cube, thin-wire feed, dielectric blocks, port record, 32-frequency DFT
        _step("512 cube, port record and DFT", 512, 512, 512, pml=16, steps=64, fill=0.05, record=1, freqs=32, dirs=1024),
        # the optional absorber
        _step("convolutional absorber", 192, 168, 144, pml=10, steps=20, fill=0.02, cpml=1),
        # a wideband far-field run: one whole DFT block, then the spectra over 650 directions
        _step("wideband far field", 256, 256, 176, pml=12, steps=256, fill=0.02, freqs=32, dirs=650, every=1),
        # the batched sweep's chunk: mixed scene sizes in one stack
        _batch("stack of 16 scenes", scenes=16, lo=48, hi=160, steps=64),
        # the learned sweep's chunk: every scene with its surface DFT, spectra at the snapshot
        _batch("stack with surface DFT", scenes=8, lo=80, hi=80, steps=64, freqs=32),
        # the phased array's pattern: one degree steps over the sphere
        _pattern("pattern 181 x 361 x 32", 184, 184, 120, pml=10, freqs=32, n_theta=181, n_phi=361),
        # the console report's pattern
        _report("report pattern", 128, 128, 128, pml=10),
        # training and inference of the extrapolator share these layers; training has both directions
        _train("extrapolator training step", batch=256, rows=256),
        # the radar's image
        _radar("radar image", elements=36, nr=64, naz=61, nel=41, samples=240),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "step", "step", "step", "batch", "pattern", "report", "train", "radar"])
    pml = rng.choice([6, 8, 10, 12, 16])
    least = 2 * pml + 16
    dims = lambda lo, hi: [max(least, size(lo, hi)) for _ in range(3)]  # noqa: E731
    if kind == "frame":
        return _frame(None, *dims(32, 200), pml=pml, steps=rng.choice([1, 2, 4, 8]))
    if kind == "step":
        n = dims(40, 320)
        steps = max(2, min(200, int(4e8 / (n[0] * n[1] * n[2]))))
        extra = rng.choice([{}, {"record": 1}, {"ntff": 1}, {"cpml": 1}, {"record": 1, "ntff": 1},
                            {"freqs": rng.choice([1, 8, 20, 32, 64]), "dirs": size(20, 1024), "every": rng.choice([0, 1])}])
        return _step(None, *n, pml=pml, steps=steps, fill=rng.choice([0.0, 0.02, 0.05]), **extra)
    if kind == "batch":
        if rng.random() < 0.5:
            lo = rng.choice([48, 64, 80])
            return _batch(None, scenes=rng.randint(2, 16), lo=lo, hi=lo + 16 * rng.randint(0, 3), steps=64)
        edge = rng.choice([48, 64, 80, 96])
        return _batch(None, scenes=rng.randint(1, 8), lo=edge, hi=edge, steps=64, freqs=rng.choice([8, 16, 32]))
    if kind == "pattern":
        return _pattern(None, *dims(56, 184), pml=pml, freqs=rng.choice([1, 4, 16]), n_theta=rng.choice([19, 37, 91, 181]),
                        n_phi=rng.choice([37, 73, 181]))
    if kind == "report":
        return _report(None, *dims(48, 200), pml=pml)
    if kind == "train":
        batch = rng.choice([32, 64, 128, 256])
        return _train(None, batch=batch, rows=rng.randint(1, batch))
    return _radar(None, elements=rng.choice([4, 9, 16, 25, 64]), nr=size(8, 90), naz=2 * size(4, 30) + 1,
                  nel=2 * size(4, 25) + 1, samples=size(60, 400))


def _named(name, case):
    return {"name": name, **case} if name else case


def _frame(name, nx, ny, nz, pml, steps):
    return _named(name, {"kind": "frame", "nx": nx, "ny": ny, "nz": nz, "pml": pml, "steps": steps})


def _step(name, nx, ny, nz, pml, steps, fill, record=0, ntff=0, freqs=0, dirs=0, every=0, cpml=0):
    return _named(name, {"kind": "step", "nx": nx, "ny": ny, "nz": nz, "pml": pml, "steps": steps, "fill": fill,
                         "record": record, "ntff": ntff, "freqs": freqs, "dirs": dirs, "every": every, "cpml": cpml})


def _batch(name, scenes, lo, hi, steps, freqs=0):
    return _named(name, {"kind": "batch", "scenes": scenes, "lo": lo, "hi": hi, "steps": steps, "freqs": freqs})


def _pattern(name, nx, ny, nz, pml, freqs, n_theta, n_phi):
    return _named(name, {"kind": "pattern", "nx": nx, "ny": ny, "nz": nz, "pml": pml, "freqs": freqs, "n_theta": n_theta,
                         "n_phi": n_phi})


def _report(name, nx, ny, nz, pml):
    return _named(name, {"kind": "report", "nx": nx, "ny": ny, "nz": nz, "pml": pml})


def _train(name, batch, rows):
    return _named(name, {"kind": "train", "batch": batch, "rows": rows})


def _radar(name, elements, nr, naz, nel, samples):
    return _named(name, {"kind": "radar", "elements": elements, "nr": nr, "naz": naz, "nel": nel, "samples": samples})


# ---- inputs ------------------------------------------------------------------------------------------
def _scene(case, seed):
    """A thin-wire dipole with its 50-ohm feed at the centre, a continuous point dipole, and seeded
    lossy dielectric blocks over `fill` of the cells."""
    n = (case["nx"], case["ny"], case["nz"])
    L = case["pml"]
    rng = np.random.default_rng([int(seed), 11])
    grid = abi.GridConfig(n, courant=0.5, pml_thickness=L, pml_sigma_max=1.6, pml_grading=3.0)
    wl = 16.0 if min(n) < 256 else 40.0
    b = EnvironmentBuilder("case", grid, wavelength=wl)
    blocks, target = 0, case.get("fill", 0.0) * n[0] * n[1] * n[2]
    while blocks < target:
        e = rng.integers(4, 25, size=3)
        e = np.minimum(e, [max(2, (v - 2 * L) // 4) for v in n])
        p = [int(rng.integers(L // 2, max(L // 2 + 1, n[a] - L // 2 - e[a]))) for a in range(3)]
        m = Material(float(10.0 ** rng.uniform(-4.4, -1.4)), float(rng.uniform(1.0, 10.0)))
        blocks += b.box(p, [p[a] + int(e[a]) for a in range(3)], m)
    c = tuple(v * 0.5 for v in n)
    wave = SourceDesc(wavelength=wl, waveform=abi.WAVE_CW, ramp_periods=1.0, phase=float(rng.uniform(0, 6.2)))
    b.thin_dipole(wave, c, 2, min(0.5 * wl, min(n) - 2 * L - 8), radius=0.05, impedance_ohm=50.0, drive=1.0)
    at = [float(rng.uniform(L + 4, v - L - 4)) for v in n]
    b.scene.sources.append(SourceDesc.dipole(at, (0.6, 0.0, 0.8), wl, float(rng.uniform(1.0, 7.0))))
    return b.build(), wl


def _packets(shape, seed):
    """Six field components (nz, ny, nx) float32: two wave packets each."""
    rng = np.random.default_rng([int(seed), 7])
    out = []
    for _ in range(6):
        total = torch.zeros(shape, dtype=torch.float32, device=DEV)
        for _ in range(2):
            axes = []
            for n in shape:
                r = np.arange(n) - rng.uniform(0.25, 0.75) * n
                k = 2.0 * math.pi / rng.uniform(10.0, 40.0) * rng.choice([-1.0, 1.0])
                axes.append(np.exp(-0.5 * (r / (0.2 * n + 3.0)) ** 2 + 1j * (k * r + rng.uniform(0.0, 6.2))))
            z, y, x = ((torch.from_numpy(a.real.astype(np.float32)).to(DEV), torch.from_numpy(a.imag.astype(np.float32)).to(DEV))
                       for a in axes)
            re = y[0][:, None] * x[0] - y[1][:, None] * x[1]
            im = y[0][:, None] * x[1] + y[1][:, None] * x[0]
            total += z[0][:, None, None] * re
            total -= z[1][:, None, None] * im
        out.append(total)
    return out


class _Fields:
    """The grid's field arrays as torch views, one set for each generation of the state; a view keeps
    its grid, whose memory it shows."""

    def __init__(self, grid):
        self.grid, self.size, self.known = grid, grid.size(), {}

    def __call__(self):
        ptrs, pitch, plane = self.grid.field_pointers()
        key = tuple(ptrs)
        if key not in self.known:
            nx, ny, nz = self.size
            grid = self.grid

            class View:
                def __init__(self, p):
                    self.grid = grid
                    self.__cuda_array_interface__ = {"shape": (nz, ny, nx), "typestr": "<f4", "data": (p, False),
                                                     "strides": (plane * 4, pitch * 4, 4), "version": 2}

            self.known[key] = [torch.as_tensor(View(p), device=DEV) for p in ptrs]
        return self.known[key]


def _far_box(case):
    L = case["pml"]
    n = (case["nx"], case["ny"], case["nz"])
    d = 4 if min(n) < 256 else 20
    d = max(0, min(d, (min(n) - 2 * L - 12) // 3))
    return [L + 1 + d] * 3, [v - L - 2 - d for v in n]


def _wavelengths(wl, nf):
    return [wl / f for f in np.linspace(0.3, 1.7, nf)] if nf > 1 else [wl]


def _sphere(n):
    return configs.fibonacci_directions(n)


def _grid(case, seed, sc):
    g = SimulationGrid(sc.grid)
    if case.get("cpml"):
        g.set_cpml((3.2, 1.0, 0.05, 3.0))
    g.upload_materials(sc.materials.sigma, sc.materials.epsilon_r, sc.edges, sc.wires)
    g.set_sources(sc.sources)
    g.synchronize()
    fields = _Fields(g)
    for view, v in zip(fields(), _packets((case["nz"], case["ny"], case["nx"]), seed)):
        view.copy_(v)
    torch.cuda.synchronize()
    return g, fields


def _batch_scenes(case, seed):
    edges = list(range(case["lo"], case["hi"] + 1, 16))
    return [configs.batched_scene(seed, i, edges=(edges[i % len(edges)],)) for i in range(case["scenes"])]


def _train_data(case, seed):
    rng = np.random.default_rng([int(seed), 3])
    n = case["rows"]
    t = np.arange(T_IN) / T_IN
    x = np.empty((n, T_IN, 2), np.float32)
    for ch in range(2):  # ringing port voltage and current
        f, d, ph = rng.uniform(2, 9, (n, 1)), rng.uniform(1, 6, (n, 1)), rng.uniform(0, 6.2, (n, 1))
        x[:, :, ch] = np.exp(-d * t) * np.sin(6.2832 * f * t + ph)
    aux = rng.standard_normal((n, AUX)).astype(np.float32)
    tgt = rng.standard_normal((n, OUT)).astype(np.float32)
    return x, aux, tgt


def _moments(seed):
    """Adam's state of a run in progress: name -> (mW, vW, mb, vb)."""
    rng = np.random.default_rng([int(seed), 4])
    out = {}
    for name, o, i in layer_shapes():
        out[name] = tuple((rng.standard_normal(s) * 3e-4).astype(np.float32) if k == 0 else
                          (1e-6 * rng.uniform(0.5, 2.0, s)).astype(np.float32) for s in ((o, i), (o,)) for k in range(2))
    return out


T_STEP, LR = 200, 1e-3


def _radar_inputs(case, seed):
    rng = np.random.default_rng([int(seed), 5])
    n, M = case["elements"], case["samples"]
    side = int(math.ceil(math.sqrt(n)))
    wl = 16.0
    tx = np.array([14.2, 80.3, 79.6]) + rng.uniform(-0.5, 0.5, 3)
    yz = [((k % side) - 0.5 * (side - 1), (k // side) - 0.5 * (side - 1)) for k in range(n)]
    ep = np.array([[tx[0], tx[1] + 0.5 * wl * y, tx[2] + 0.5 * wl * z] for y, z in yz]) + rng.uniform(-0.01, 0.01, (n, 3))
    z = (rng.standard_normal((M, n)) + 1j * rng.standard_normal((M, n))).astype(np.complex64)
    g = abi.RadarGeometry()
    for k in range(3):
        g.tx[k], g.interior_min[k], g.interior_max[k] = float(tx[k]), 11.13, 148.77
    for k, v in enumerate([0, -1, 0, 0, 0, 1, 1, 0, 0]):  # right, up, boresight (+x)
        g.axes[k] = float(v)
    g.omega, g.dt, g.sample_dt = 2.0 * math.pi / wl, 0.5, 320.0 / M
    g.r0, g.dr, g.daz, g.del_ = 20.0, 120.0 / case["nr"], 1.5, 1.5
    g.nr, g.naz, g.nel = case["nr"], case["naz"], case["nel"]
    g.az0, g.el0 = -1.5 * (case["naz"] // 2), -1.5 * (case["nel"] // 2)

    class Array:
        elem_pos, weights = ep.astype(np.float32), 0.54 + 0.46 * rng.random(n)
        tx_pos, tx_amp = ep.astype(np.float32), rng.uniform(0.5, 1.5, n)
    return Array(), z, g


# ---- the program's state, and one pass ----------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        net = Net(init_params(seed % 100003), batch=case["batch"])
        for name, (mw, vw, mb, vb) in _moments(seed).items():
            for dst, v in ((net.mW, mw), (net.vW, vw), (net.mb, mb), (net.vb, vb)):
                dst[name].copy_(torch.from_numpy(v))
        net.t_step = T_STEP
        return {"kind": kind, "net": net, "data": _train_data(case, seed)}
    if kind == "radar":
        return {"kind": kind, "args": _radar_inputs(case, seed)}
    if kind == "batch":
        return _prepare_batch(case, seed)
    sc, wl = _scene(case, seed)
    g, fields = _grid(case, seed, sc)
    st = {"kind": kind, "grid": g, "fields": fields, "steps": case.get("steps", 0)}
    if kind == "frame":
        n = (case["nx"], case["ny"], case["nz"])
        lo, hi = [v // 2 - 8 for v in n], [v // 2 + 8 for v in n]
        st["origins"] = [(v[0], v[1], v[2]) for v in (lo, hi, (n[0] // 3, n[1] // 2, n[2] // 2))]
        st["planes"] = [abi.FluxPlane(ax, i, (C.c_int * 2)(*a), (C.c_int * 2)(*b))
                        for _, ax, i, a, b in FluxSetup("box", "box", tuple(lo), tuple(hi)).planes()]
    elif kind == "step":
        if case["record"]:
            g.ports_configure([p.to_c() for p in sc.ports], wl, 4.0, False, case["steps"])
        st["record"] = case["record"]
        if case["ntff"]:
            g.ntff_configure(*_far_box(case), wl, 4.0)
            st["cuts"] = far_field_directions((0.0, 0.0, 1.0))[0][:540]
        if case["freqs"]:
            g.ntff_dft_configure(*_far_box(case), _wavelengths(wl, case["freqs"]))
            st["dirs"], st["every"], st["mid"] = _sphere(case["dirs"]), case["every"], case["freqs"] // 2
        g.synchronize()
    elif kind == "pattern":
        g.ntff_dft_configure(*_far_box(case), _wavelengths(wl, case["freqs"]))
        g.step(64)
        st["dirs"] = angle_grid(case["n_theta"], case["n_phi"])[0]
        g.synchronize()
    elif kind == "report":
        g.ntff_configure(*_far_box(case), wl, 4.0)
        g.step(64)
        st["dirs"] = far_field_directions((0.0, 0.0, 1.0))[0]
        g.synchronize()
    return st


def _prepare_batch(case, seed):
    scenes = _batch_scenes(case, seed)
    first = scenes[0]
    if case["lo"] == case["hi"]:
        g = SceneStack(first.grid, [sc.grid.size[2] for sc in scenes])
    else:
        g = SceneStack(first.grid, scene_dims=[tuple(sc.grid.size) for sc in scenes])
    for k, sc in enumerate(scenes):
        g.upload_scene_materials(k, sc.materials.sigma, sc.materials.epsilon_r, sc.edges, sc.wires)
    g.set_scene_sources([sc.sources for sc in scenes])
    g.commit()
    g.set_graph(case["steps"])
    z0, _ = g.layout()
    ports = []
    for sc, z in zip(scenes, z0):
        p = sc.ports[0].to_c()
        p.z += z
        ports.append(p)
    g.ports_configure(ports, first.wavelength, 4.0, False, case["steps"])
    far = None
    if case["freqs"]:
        far = FarField(case["freqs"])
        g.ntff_dft_configure_boxes([far.box(sc, z) for sc, z in zip(scenes, z0)], far.wavelengths(first), block=far.block)
    g.synchronize()
    fields = _Fields(g)
    for k, (sc, z) in enumerate(zip(scenes, z0)):
        nx, ny, nz = sc.grid.size
        for view, v in zip(fields(), _packets((nz, ny, nx), seed * 64 + k)):
            view[z:z + nz, :ny, :nx].copy_(v)
    torch.cuda.synchronize()
    return {"kind": "batch", "grid": g, "fields": fields, "steps": case["steps"], "far": far, "scenes": len(scenes)}


def run(st):
    kind = st["kind"]
    if kind == "train":
        net, (x, aux, tgt) = st["net"], st["data"]
        net.load(x, aux, tgt)
        net.forward()
        net.backward()
        net.step(lr=LR)
        return {"y": net.y, "loss": net.loss, "gW": net.gW, "gb": net.gb, "W": net.W, "b": net.b, "mW": net.mW, "vW": net.vW,
                "mb": net.mb, "vb": net.vb}
    if kind == "radar":
        array, z, geo = st["args"]
        return RadarMonitor.backproject(array, z, geo)
    g = st["grid"]
    if kind == "frame":
        g.step(st["steps"])
        g.synchronize()
        probes = g.probe_gather(st["origins"])
        return {"probes": probes, "flux": g.flux_planes(st["planes"]), "fields": st["fields"]()}
    if kind == "pattern":
        return g.ntff_dft_pattern_gemm(0, st["dirs"])
    if kind == "report":
        return g.ntff_evaluate(st["dirs"])
    g.step(st["steps"])
    out = {}
    if kind == "batch":
        slot, rows = g.ports_take_series_async()
        out["series"] = g.ports_collect_series(slot, rows)
        if st["far"] is not None:
            out["far"] = [g.ntff_dft_spectra(k, st["far"].dirs) for k in range(st["scenes"])]
    else:
        if st["record"]:
            out["series"] = g.ports_take_series(st["steps"])
        if "cuts" in st:
            out["cuts"] = g.ntff_evaluate(st["cuts"])
        if "dirs" in st:
            out["far"] = g.ntff_dft_spectra(0, st["dirs"]) if st["every"] else g.ntff_dft_evaluate(st["mid"], st["dirs"])
    out["fields"] = st["fields"]()
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------
def _points(lo, hi):
    d = [b - a + 1 for a, b in zip(lo, hi)]
    return 2 * (d[0] * d[1] + d[1] * d[2] + d[0] * d[2])


STEP_BYTES, STEP_FLOPS = 50.0, 33.0  # six fields read and written, a 16-bit material index; the two curls


def work(case):
    kind = case["kind"]
    if kind == "train":
        macs = sum(o * i * (64 * case["batch"] if n == "conv1" else 16 * case["batch"] if n == "conv2" else case["batch"])
                   for n, o, i in layer_shapes())
        params = sum(o * i + o for _, o, i in layer_shapes())
        return {"bytes": params * 28.0 + case["rows"] * 4.0 * (2 * T_IN + AUX + OUT), "flops": 6.0 * macs}
    if kind == "radar":
        pts = case["nr"] * case["naz"] * case["nel"]
        return {"bytes": pts * 8.0 + case["samples"] * case["elements"] * 8.0, "flops": pts * case["elements"] * 80.0}
    if kind == "batch":
        edges = list(range(case["lo"], case["hi"] + 1, 16))
        ns = [edges[i % len(edges)] for i in range(case["scenes"])]
        cells = sum(n ** 3 for n in ns)
        pts = sum(_points([9] * 3, [n - 10] * 3) for n in ns) if case["freqs"] else 0
        return {"bytes": case["steps"] * STEP_BYTES * cells + pts * 6.0 * (8.0 * case["steps"] + 32.0 * case["freqs"]),
                "flops": case["steps"] * (STEP_FLOPS * cells + 24.0 * case["freqs"] * pts) + 650.0 * pts * 60.0 * case["freqs"]}
    pts = _points(*_far_box(case))
    if kind == "report":
        return {"bytes": pts * 64.0, "flops": len(far_field_directions((0.0, 0.0, 1.0))[0]) * pts * 60.0}
    if kind == "pattern":  # per face and frequency one sum factorised over the two lattice axes
        lo, hi = _far_box(case)
        d = [b - a + 1 for a, b in zip(lo, hi)]
        D, F = case["n_theta"] * case["n_phi"], case["freqs"]
        per = sum(32.0 * (d[u] * d[v] + d[u]) for u, v in ((1, 2), (0, 2), (0, 1)) for _ in range(2))
        return {"bytes": pts * 96.0 * F + D * F * 8.0, "flops": per * D * F}
    cells = case["nx"] * case["ny"] * case["nz"]
    out = {"bytes": case["steps"] * STEP_BYTES * cells, "flops": case["steps"] * STEP_FLOPS * cells}
    if case.get("ntff"):
        out["bytes"] += case["steps"] * pts * 256.0
        out["flops"] += case["steps"] * pts * 36.0 + 540.0 * pts * 60.0
    if case.get("freqs"):
        F = case["freqs"]
        out["bytes"] += pts * 6.0 * (8.0 * case["steps"] + 32.0 * F)
        out["flops"] += case["steps"] * 24.0 * F * pts + case["dirs"] * pts * 60.0 * (F if case["every"] else 1)
    return out


# ---- the same in 64 bits ----------------------------------------------------------------------------------
def _profile(n, cfg, half):
    L = cfg.pml_thickness
    i = torch.arange(n, dtype=F64, device=DEV) + half
    u = (torch.maximum(L - i, i - (n - 1 - L)).clamp(min=0) / L).clamp(max=1)
    return float(cfg.pml_sigma_max) * torch.expm1(float(cfg.pml_grading) * u) / math.expm1(float(cfg.pml_grading))


def _phi(x):
    return torch.where(x > 1e-12, -torch.expm1(-x) / x.clamp(min=1e-12), 1.0 - 0.5 * x)


def _shift(f, axis, forward):
    """The neighbour along an axis (0 = x), zero beyond the grid."""
    d = 2 - axis
    out = torch.zeros_like(f)
    n = f.shape[d]
    if forward:
        out.narrow(d, 0, n - 1).copy_(f.narrow(d, 1, n - 1))
    else:
        out.narrow(d, 1, n - 1).copy_(f.narrow(d, 0, n - 1))
    return out


def _signal(s, t):
    wl = float(np.float32(s.wavelength))
    w = 2.0 * math.pi / wl
    if s.waveform == abi.WAVE_CW:
        ramp_t = float(np.float32(s.ramp_periods)) * wl
        r = min(t / ramp_t, 1.0) if ramp_t > 0 else 1.0
        return r ** 3 * (10.0 + r * (-15.0 + 6.0 * r)) * math.sin(w * t + float(np.float32(s.phase)))
    tau = max(float(np.float32(s.ramp_periods)), 0.1) * wl
    u = (t - 3.0 * tau) / tau
    return math.exp(-u * u) * math.sin(w * (t - 3.0 * tau) + float(np.float32(s.phase))) if abs(u) <= 6.0 else 0.0


class _Solver64:
    """The leapfrog of one scene in float64: graded or convolutional absorber, edge-averaged materials
    rounded to binary16, thin wires, volume current sources."""

    def __init__(self, sc, fields, cpml=None):
        self.cfg = cfg = sc.grid
        nx, ny, nz = n = cfg.size
        self.dt, self.n, self.t = float(cfg.courant), n, 0
        self.F = [f.to(F64) for f in fields]
        sig = torch.from_numpy(np.asarray(sc.materials.sigma)).to(DEV)
        eps = torch.from_numpy(np.asarray(sc.materials.epsilon_r)).to(DEV)

        def low(f, axis):  # the lower neighbour, clamped to the edge cell
            d = 2 - axis
            return torch.cat([f.narrow(d, 0, 1), f.narrow(d, 0, f.shape[d] - 1)], d)

        I = [_profile(n[a], cfg, 0.0).reshape([-1 if 2 - a == k else 1 for k in range(3)]) for a in range(3)]
        H = [_profile(n[a], cfg, 0.5).reshape([-1 if 2 - a == k else 1 for k in range(3)]) for a in range(3)]
        if cpml:
            I = H = [torch.zeros_like(v) for v in I]
        self.ca, self.cb, self.da, self.db = [], [], [], []
        for c in range(3):
            u, v = [a for a in range(3) if a != c]
            av = lambda f: 0.25 * (((f + low(f, u)) + low(f, v)) + low(low(f, u), v))  # noqa: E731
            s, e = av(sig).clamp(max=6.0e4).half(), av(eps).half()
            for o in sc.edges:
                if o.axis == c:
                    s[o.z, o.y, o.x] = min(max(o.sigma, 0.0), 6.0e4)
            ce = self.dt / e.to(F64).clamp(min=1.0)
            x = (s.to(F64).clamp(min=0.0) + sum(H[a] if a == c else I[a] for a in range(3))) * ce
            self.ca.append(torch.exp(-x))
            self.cb.append(ce * _phi(x))
            xm = self.dt * sum(I[a] if a == c else H[a] for a in range(3)).expand(nz, ny, nx)
            self.da.append(torch.exp(-xm))
            self.db.append(self.dt * _phi(xm))
        self.wires = {}
        for w in sc.wires:
            if all(0 <= v < m for v, m in zip((w.x, w.y, w.z), n)):
                self.wires.setdefault((w.component, w.term), {})[(w.z, w.y, w.x)] = float(np.float16(w.factor))
        self.wires = {k: (torch.tensor(list(d.keys()), device=DEV).T, torch.tensor(list(d.values()), dtype=F64, device=DEV))
                      for k, d in self.wires.items()}
        self.psi = {}
        self.cpml = None
        if cpml:
            smax, kmax, amax, order = cpml
            self.cpml = {}
            for half in (0, 1):
                for a in range(3):
                    L = cfg.pml_thickness
                    i = torch.arange(n[a], dtype=F64, device=DEV) + 0.5 * half
                    d = (torch.maximum(L - i, i - (n[a] - 1 - L)) / L).clamp(0, 1)
                    s, k, al = smax * d ** order, 1 + (kmax - 1) * d ** order, amax * (1 - d)
                    b = torch.exp(-(s / k + al) * self.dt)
                    cc = torch.where(s > 0, s / (s * k + k * k * al).clamp(min=1e-300) * (b - 1), torch.zeros_like(s))
                    self.cpml[half, a] = [v.reshape([-1 if 2 - a == q else 1 for q in range(3)]) for v in (b, cc, 1 / k)]
        self.src = []
        f32 = lambda v: [float(np.float32(q)) for q in v]  # noqa: E731
        for s in sc.sources:
            ctr, half, soft, pol = f32(s.center), f32(s.half_extent), [max(v, 0.25) for v in f32(s.softness)], f32(s.polarization)
            norm = math.sqrt(sum(v * v for v in pol))
            lo = [min(max(int(math.floor(np.float32(ctr[a] - half[a] - 3.5 * soft[a]))) - 1, 0), n[a] - 1) for a in range(3)]
            hi = [min(max(int(math.ceil(np.float32(ctr[a] + half[a] + 3.5 * soft[a]))), 0), n[a] - 1) for a in range(3)]
            box = tuple(slice(lo[a], hi[a] + 1) for a in (2, 1, 0))
            parts = []
            for c in range(3):
                q = 0
                for a in range(3):
                    r = torch.arange(lo[a], hi[a] + 1, dtype=F64, device=DEV) + (0.5 if a == c else 0.0)
                    d = ((r - ctr[a]).abs() - half[a]).clamp(min=0) / soft[a]
                    q = q + (d * d).reshape([-1 if 2 - a == k else 1 for k in range(3)])
                parts.append(pol[c] / norm * float(np.float32(s.amplitude)) * torch.exp(-q))
            self.src.append((s, box, parts))

    def _term(self, d, half, axis, key):
        if not self.cpml:
            return d
        b, c, ik = self.cpml[half, axis]
        p = self.psi.get(key)
        p = c * d if p is None else b * p + c * d
        self.psi[key] = p
        return d * ik + p

    def step(self):
        F = self.F
        old = F[:3]
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            t0, t1 = _shift(old[v], u, True) - old[v], _shift(old[u], v, True) - old[u]
            for k, t in enumerate((t0, t1)):
                if (c, k) in self.wires:
                    at, f = self.wires[c, k]
                    t[at[0], at[1], at[2]] *= f
            curl = self._term(t0, 1, u, ("B", c, 0)) - self._term(t1, 1, v, ("B", c, 1))
            F[3 + c] = self.da[c] * F[3 + c] - self.db[c] * curl
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            curl = (self._term(F[3 + v] - _shift(F[3 + v], u, False), 0, u, ("E", c, 0))
                    - self._term(F[3 + u] - _shift(F[3 + u], v, False), 0, v, ("E", c, 1)))
            F[c] = self.ca[c] * F[c] + self.cb[c] * curl
        t = (self.t + 0.5) * self.dt
        for s, box, parts in self.src:
            amp = _signal(s, t)
            for c in range(3):
                F[c][box] -= self.cb[c][box] * (amp * parts[c])
        self.t += 1

    def port(self, p):
        a = p.axis
        u, v = (a + 1) % 3, (a + 2) % 3
        at = lambda f, d: f[p.texel[2] - (d == 2), p.texel[1] - (d == 1), p.texel[0] - (d == 0)]  # noqa: E731
        B = self.F[3:]
        i = (at(B[v], -1) - at(B[v], u)) - (at(B[u], -1) - at(B[u], v))
        return torch.stack([at(self.F[a], -1), i]) * (1.0 if p.sign >= 0 else -1.0)

    def nodes(self, faces):
        """Co-located E and H (6, points) at a box's nodes."""
        cols = [[] for _ in range(6)]
        for sl, _, _, _, _ in faces:
            for c in range(3):
                e = self.F[c]
                cols[c].append((0.5 * (e[sl] + e[_moved(sl, c)])).reshape(-1))
                b, (u, v) = self.F[3 + c], [a for a in range(3) if a != c]
                m = _moved(sl, u)
                cols[3 + c].append((0.25 * (b[sl] + b[m] + b[_moved(sl, v)] + b[_moved(m, v)])).reshape(-1))
        return torch.stack([torch.cat(c) for c in cols])


def _moved(sl, axis):
    out = list(sl)
    s = out[2 - axis]
    out[2 - axis] = slice(s.start - 1, s.stop - 1)
    return tuple(out)


def _faces(lo, hi):
    """Per face: the node slices (z, y, x), normal axis, sign, and the trapezoid weights."""
    out = []
    for f in range(6):
        a, side = f >> 1, f & 1
        at = [slice(lo[k], hi[k] + 1) for k in range(3)]
        p = hi[a] if side else lo[a]
        at[a] = slice(p, p + 1)
        w = torch.ones([at[k].stop - at[k].start for k in (2, 1, 0)], dtype=F64, device=DEV)
        for k in range(3):
            if k != a:
                w.narrow(2 - k, 0, 1).mul_(0.5)
                w.narrow(2 - k, w.shape[2 - k] - 1, 1).mul_(0.5)
        out.append(((at[2], at[1], at[0]), a, 1.0 if side else -1.0, w, at))
    return out


def _far64(X, lo, hi, k, dirs, origin=(0, 0, 0)):
    """(directions, 2): |N_perp - r x L|^2 and the radiated power (first direction), from the complex
    phasors X (6, points) of a box, each face summed over one lattice axis after the other."""
    r = torch.from_numpy(np.asarray(dirs, np.float32)).to(DEV).to(F64)
    N = torch.zeros((len(dirs), 3), dtype=torch.complex128, device=DEV)
    Lv = torch.zeros_like(N)
    power, first = 0.0, 0
    mid = [0.5 * (a + b) for a, b in zip(lo, hi)]
    for _, a, sign, w, at in _faces(lo, hi):
        u, v = [q for q in range(3) if q != a]
        nu, nv = hi[u] - lo[u] + 1, hi[v] - lo[v] + 1
        x = X[:, first:first + nu * nv].reshape(6, nv, nu)
        first += nu * nv
        w = w.reshape(nv, nu)
        e, h = x[:3], x[3:]
        # n x V for n = sign e_a
        cross = lambda V: {(a + 1) % 3: -sign * V[(a + 2) % 3], (a + 2) % 3: sign * V[(a + 1) % 3]}  # noqa: E731
        J, M = cross(h), cross(e)
        pos = [torch.arange(lo[q], hi[q] + 1, dtype=F64, device=DEV) - mid[q] for q in range(3)]
        pa = (hi[a] if sign > 0 else lo[a]) - mid[a]
        for d0 in range(0, len(dirs), 8192):
            rr = r[d0:d0 + 8192]
            V = torch.exp(1j * k * rr[:, v:v + 1] * pos[v])
            U = torch.exp(1j * k * (rr[:, u:u + 1] * pos[u] + rr[:, a:a + 1] * pa))
            for out, src, s in ((N, J, 1.0), (Lv, M, -1.0)):
                for q in (u, v):
                    out[d0:d0 + 8192, q] += ((V @ (s * w * src[q])) * U).sum(1)
        s = e[(a + 1) % 3] * h[(a + 2) % 3].conj() - e[(a + 2) % 3] * h[(a + 1) % 3].conj()
        power += float((w * sign * s.real).sum())
    rc = r.to(torch.complex128)
    f = N - (N * rc).sum(1, keepdim=True) * rc - torch.linalg.cross(rc, Lv, dim=1)
    out = torch.zeros((len(dirs), 2), dtype=F64, device=DEV)
    out[:, 0] = f.abs().square().sum(1)
    out[0, 1] = 0.5 * power
    return out


class _Dft64:
    """Samples of a box's co-located fields and their sums at every frequency."""

    def __init__(self, solver, lo, hi, wavelengths):
        self.s, self.lo, self.hi = solver, lo, hi
        self.faces, self.rows, self.times = _faces(lo, hi), [], []
        self.k = [2.0 * math.pi / max(float(np.float32(w)), 2.0) for w in wavelengths]

    def sample(self):
        self.rows.append(self.s.nodes(self.faces))
        self.times.append(self.s.t * self.s.dt)

    def phasors(self, f):
        t = torch.tensor(self.times, dtype=F64, device=DEV)
        rows = torch.stack(self.rows)
        out = []
        for part, lag in ((rows[:, :3], 0.0), (rows[:, 3:], 0.5 * self.s.dt)):
            ph = self.k[f] * (t - lag)
            re, im = (torch.einsum("t,tcp->cp", g, part) for g in (torch.cos(ph), -torch.sin(ph)))
            out.append(torch.complex(re, im))
        return torch.cat(out) * (2.0 / len(self.times))

    def spectra(self, dirs):
        return torch.stack([_far64(self.phasors(f), self.lo, self.hi, self.k[f], dirs) for f in range(len(self.k))])


class _Average64:
    """The single-frequency monitor's two-stage running average."""

    def __init__(self, solver, lo, hi, wl):
        self.s, self.lo, self.hi = solver, lo, hi
        self.faces, self.k = _faces(lo, hi), 2.0 * math.pi / wl
        self.b = -math.expm1(-solver.dt / (0.5 * 4.0 * wl))
        self.one = self.two = 0.0

    def sample(self):
        x = self.s.nodes(self.faces)
        tE = self.s.t * self.s.dt
        rot = torch.tensor([2.0 * np.exp(-1j * self.k * t) for t in [tE] * 3 + [tE - 0.5 * self.s.dt] * 3], device=DEV)
        self.one = self.one + self.b * (rot[:, None] * x - self.one)
        self.two = self.two + self.b * (self.one - self.two)

    def pattern(self, dirs):
        return _far64(self.two, self.lo, self.hi, self.k, dirs)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train64(case, seed)
    if kind == "radar":
        return _radar64(case, seed)
    if kind == "batch":
        return _batch64(case, seed)
    sc, wl = _scene(case, seed)
    s = _Solver64(sc, _packets((case["nz"], case["ny"], case["nx"]), seed), (3.2, 1.0, 0.05, 3.0) if case.get("cpml") else None)
    if kind == "frame":
        return _frame64(case, s, sc)
    lo, hi = _far_box(case)
    monitor = None
    if kind == "pattern" or case.get("freqs"):
        monitor = _Dft64(s, lo, hi, _wavelengths(wl, case["freqs"]))
    elif kind == "report" or case.get("ntff"):
        monitor = _Average64(s, lo, hi, wl)
    series = []
    for _ in range(64 if kind in ("pattern", "report") else case["steps"]):
        s.step()
        if monitor:
            monitor.sample()
        if case.get("record"):
            series.append(s.port(sc.ports[0]))
    if kind == "pattern":
        return monitor.spectra(angle_grid(case["n_theta"], case["n_phi"])[0])
    if kind == "report":
        return monitor.pattern(far_field_directions((0.0, 0.0, 1.0))[0])
    out = {"fields": s.F}
    if case["record"]:
        out["series"] = torch.stack(series)[:, None]
    if case["ntff"]:
        out["cuts"] = monitor.pattern(far_field_directions((0.0, 0.0, 1.0))[0][:540])
    if case["freqs"]:
        dirs, mid = _sphere(case["dirs"]), case["freqs"] // 2
        out["far"] = monitor.spectra(dirs) if case["every"] else _far64(monitor.phasors(mid), lo, hi, monitor.k[mid], dirs)
    return out


def _frame64(case, s, sc):
    for _ in range(case["steps"]):
        s.step()
    n = (case["nx"], case["ny"], case["nz"])
    lo, hi = [v // 2 - 8 for v in n], [v // 2 + 8 for v in n]
    probes = torch.empty((3, 54, 4), dtype=F64, device=DEV)
    mats = [torch.from_numpy(np.asarray(m)).to(DEV).to(F64) for m in (sc.materials.sigma, sc.materials.epsilon_r)]
    for k, o in enumerate((lo, hi, (n[0] // 3, n[1] // 2, n[2] // 2))):
        box = tuple(slice(o[a], o[a] + 3) for a in (2, 1, 0))
        for half in range(2):
            for c, f in enumerate(s.F[3 * half:3 * half + 3] + [mats[half]]):
                probes[k, 27 * half:27 * half + 27, c] = f[box].reshape(-1)
    flux = []
    for _, a, i, rmin, rmax in FluxSetup("box", "box", tuple(lo), tuple(hi)).planes():
        u, v = [q for q in range(3) if q != a]
        at = [None] * 3
        at[a], at[u], at[v] = slice(i, i + 1), slice(rmin[0], rmax[0]), slice(rmin[1], rmax[1])
        x = s.nodes([((at[2], at[1], at[0]), 0, 0, 0, 0)])
        flux.append((x[(a + 1) % 3] * x[3 + (a + 2) % 3] - x[(a + 2) % 3] * x[3 + (a + 1) % 3]).sum())
    return {"probes": probes, "flux": torch.stack(flux), "fields": s.F}


def _batch64(case, seed):
    scenes = _batch_scenes(case, seed)
    far = FarField(case["freqs"]) if case["freqs"] else None
    nx, ny = max(sc.grid.size[0] for sc in scenes), max(sc.grid.size[1] for sc in scenes)
    nz = sum(sc.grid.size[2] for sc in scenes) + len(scenes) - 1
    fields = [torch.zeros((nz, ny, nx), dtype=F64, device=DEV) for _ in range(6)]
    series, spectra, z0 = [], [], 0
    for k, sc in enumerate(scenes):
        mx, my, mz = sc.grid.size
        s = _Solver64(sc, _packets((mz, my, mx), seed * 64 + k))
        if far:
            box = far.box(sc)
            dft = _Dft64(s, box[:3], box[3:], far.wavelengths(scenes[0]))
        rows = []
        for _ in range(case["steps"]):
            s.step()
            rows.append(s.port(sc.ports[0]))
            if far:
                dft.sample()
        series.append(torch.stack(rows))
        if far:
            spectra.append(dft.spectra(far.dirs))
        for f, g in zip(fields, s.F):
            f[z0:z0 + mz, :my, :mx] = g
        z0 += mz + 1
    out = {"series": torch.stack(series, 1), "fields": fields}
    if far:
        out["far"] = spectra
    return out


def _train64(case, seed):
    """The training step with its operands rounded to bfloat16 where the network stores them so, every
    product, sum and update in float64."""
    B, n = case["batch"], case["rows"]
    bf = lambda v: v.to(torch.float32).to(torch.bfloat16).to(F64)  # noqa: E731
    up = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(DEV).to(F64)  # noqa: E731
    P = {k: (up(w), up(b)) for k, (w, b) in init_params(seed % 100003).items()}
    x, aux, tgt = (up(v) for v in _train_data(case, seed))
    pad = lambda v: torch.cat([v, torch.zeros((B - n,) + v.shape[1:], dtype=F64, device=DEV)])  # noqa: E731
    x, aux, tgt = bf(pad(x)), bf(pad(aux)), pad(tgt)

    def im2col(a, k, stride, p, lo):
        a = torch.nn.functional.pad(a, (0, 0, p, p + k))
        return torch.stack([a[:, j:j + stride * lo:stride][:, :lo] for j in range(k)], 2).reshape(a.shape[0] * lo, -1)

    c1, c2 = CONV
    cols1 = im2col(x, c1[3], c1[4], c1[5], c1[7])
    z1 = cols1 @ bf(P["conv1"][0]).T + P["conv1"][1]
    cols2 = im2col(bf(z1.clamp(min=0)).reshape(B, c1[7], c1[2]), c2[3], c2[4], c2[5], c2[7])
    z2 = cols2 @ bf(P["conv2"][0]).T + P["conv2"][1]
    a = torch.cat([bf(z2.clamp(min=0)).reshape(B, ENC), aux], 1)
    ins, zs = {}, {}
    for name, _, _, relu in HEAD:
        ins[name] = a
        zs[name] = a @ bf(P[name][0]).T + P[name][1]
        a = bf(zs[name].clamp(min=0)) if relu else None
    y = zs["out"]
    dy = torch.zeros_like(y)
    dy[:n] = 2.0 * (y[:n] - tgt[:n]) / (n * OUT)
    loss = ((y[:n] - tgt[:n]) ** 2).sum().reshape(1) / (n * OUT)
    gW, gb, d = {}, {}, dy
    for name, _, _, relu in reversed(HEAD):
        dz = d * (zs[name] > 0) if relu else d
        gW[name], gb[name] = bf(dz).T @ ins[name], dz.sum(0)
        d = bf(dz) @ bf(P[name][0])
    dz2 = d[:, :ENC].reshape(-1, c2[2]) * (z2 > 0)
    gW["conv2"], gb["conv2"] = bf(dz2).T @ cols2, dz2.sum(0)
    dc = (bf(dz2) @ bf(P["conv2"][0])).reshape(B, c2[7], c2[3], c2[1])
    da = torch.zeros((B, c2[6] + 2 * c2[5] + c2[3], c2[1]), dtype=F64, device=DEV)
    for j in range(c2[3]):
        da[:, j:j + c2[4] * c2[7]:c2[4]][:, :c2[7]] += dc[:, :, j]
    dz1 = da[:, c2[5]:c2[5] + c2[6]].reshape(-1, c1[2]) * (z1 > 0)
    gW["conv1"], gb["conv1"] = bf(dz1).T @ cols1, dz1.sum(0)
    out = {"y": y, "loss": loss, "gW": gW, "gb": gb, "W": {}, "b": {}, "mW": {}, "vW": {}, "mb": {}, "vb": {}}
    t = T_STEP + 1
    for name, st in _moments(seed).items():
        for key, p, g, m, v in (("W", P[name][0], gW[name], st[0], st[1]), ("b", P[name][1], gb[name], st[2], st[3])):
            m, v = 0.9 * up(m) + 0.1 * g, 0.999 * up(v) + 0.001 * g * g
            out[key][name] = p - LR * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
            out["m" + key][name], out["v" + key][name] = m, v
    return out


def _radar64(case, seed):
    array, z, g = _radar_inputs(case, seed)
    up = lambda v: torch.from_numpy(np.asarray(v, np.float64)).to(DEV)  # noqa: E731
    tx, ax = up(list(g.tx)), up(list(g.axes)).reshape(3, 3)
    az = torch.deg2rad(g.az0 + torch.arange(g.naz, dtype=F64, device=DEV) * g.daz)[None, None, :]
    el = torch.deg2rad(g.el0 + torch.arange(g.nel, dtype=F64, device=DEV) * g.del_)[None, :, None]
    r = (g.r0 + torch.arange(g.nr, dtype=F64, device=DEV) * g.dr)[:, None, None, None]
    d = (torch.sin(az) * torch.cos(el))[..., None] * ax[0] + torch.sin(el)[..., None] * ax[1] + (torch.cos(az) * torch.cos(el))[..., None] * ax[2]
    P = tx + r * d
    inside = ((P >= up(list(g.interior_min))) & (P <= up(list(g.interior_max)))).all(-1)
    ar = torch.zeros(P.shape[:3], dtype=torch.complex128, device=DEV)
    ad, mag = torch.zeros_like(ar), torch.zeros(P.shape[:3], dtype=F64, device=DEV)
    for pos, amp in zip(up(array.tx_pos), array.tx_amp):
        v = P - pos
        dist = v.norm(dim=-1).clamp(min=0.5)
        a = amp * ((v @ ax[2]) / dist).clamp(min=0) / dist
        e = a * torch.exp(-1j * g.omega * dist)
        ar, ad, mag = ar + e, ad + dist * e, mag + a
    out = torch.where(ar.abs() < 1e-3 * mag, (P - tx).norm(dim=-1), (ad / ar).real)
    zt = torch.from_numpy(z).to(DEV).to(torch.complex128)
    total = torch.zeros_like(ar)
    for i, (pos, w) in enumerate(zip(up(array.elem_pos), array.weights)):
        t = out + (P - pos).norm(dim=-1)
        s = (t + 0.5 * g.dt) / g.sample_dt
        ok = (s >= 0) & (s < len(zt) - 1)
        m0 = torch.where(ok, s, torch.zeros_like(s)).long()
        f = torch.where(ok, s - m0, torch.zeros_like(s))
        v = zt[m0, i] * (1 - f) + zt[m0 + 1, i] * f
        total = total + torch.where(ok, float(w) * v * torch.exp(1j * g.omega * t), torch.zeros_like(v))
    return torch.where(inside, total.abs().square(), torch.full_like(mag, -1.0))
