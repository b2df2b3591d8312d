"""Timed cases of the engine's public entry points.

A case is a dict of plain values; ``kind`` names the call a program makes:

* ``stream`` — a host drives the engine step by step: one source amplitude
  in, one step, the probe's newest sample out (a co-simulation loop);
* ``engine`` — ``Engine.run`` over a number of steps, then the recorded
  series; with ``energy`` the last step also takes the energy the run loop's
  end criterion asks for, with ``dft`` the pass reads a running transform,
  with ``fields`` every field component (a program that reads the state or writes field files);
* ``batch`` — ``Batch.run`` over many models, then every port's V and I;
* ``forward`` / ``train`` — the learned early stop's network: predictions of
  a batch of port records, one training step.

Models, grids and tables are built once per case; the seed sets what runs
through them: the field state a pass starts from (cavity modes, so that no
face sees a jump), the source amplitudes, the records and the weights.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import ems_b200 as E
from ems_b200 import learn as L
from ems_b200 import workloads as W

TABLE = 200_000  # steps of tabulated source amplitudes


def listed():
    return [
        # A host-coupled loop on a tiny box: latency of one step.
        {"name": "stream_box_24", "kind": "stream", "nx": 24, "ny": 24, "nz": 24, "medium": "vacuum", "wall": "cpml",
         "layers": 6, "mesh": 0, "curl": 0, "steps": 1},
        # A small lossy PEC resonator, odd sizes, its fields written out after the run.
        {"name": "lossy_cavity_37x52x29", "kind": "engine", "nx": 37, "ny": 52, "nz": 29, "medium": "lossy",
         "wall": "pec", "layers": 0, "mesh": 1, "curl": 0, "steps": 50, "fields": True},
        # The small plain-method configuration: 100^3 vacuum, CPML 8, point source, four probes.
        {"name": "vacuum_box_100", "kind": "engine", "nx": 100, "ny": 100, "nz": 100, "medium": "vacuum",
         "wall": "cpml", "layers": 8, "mesh": 0, "curl": 0, "steps": 100},
        # The patch antenna configuration on its graded, jittered mesh: one check interval of the run loop.
        {"name": "patch_antenna", "kind": "engine", "nx": 194, "ny": 196, "nz": 77, "medium": "patch", "wall": "cpml",
         "layers": 8, "mesh": 1, "curl": 0, "steps": 50, "energy": True},
        # The large dispersive configuration: 512^3, CPML 10, two-pole Lorentz sphere, Drude slab, sheet source.
        {"name": "dispersive_box_512", "kind": "engine", "nx": 512, "ny": 512, "nz": 512, "medium": "dispersive",
         "wall": "cpml", "layers": 10, "mesh": 0, "curl": 0, "steps": 10},
        # An odd box half full of Debye and Lorentz media in the default (trapezoidal) scheme, with its energy check.
        {"name": "trapezoidal_157x203x119", "kind": "engine", "nx": 157, "ny": 203, "nz": 119, "medium": "trapezoidal",
         "wall": "cpml", "layers": 8, "mesh": 0, "curl": 0, "steps": 50, "energy": True},
        # What an openEMS file sets up: openEMS's summation order, its PML, lossy media, f32 current probe; the
        # fields are read at the end of the pass, as that path's energy check does.
        {"name": "openems_pml_131x117x93", "kind": "engine", "nx": 131, "ny": 117, "nz": 93, "medium": "lossy",
         "wall": "upml", "layers": 8, "mesh": 1, "curl": 1, "steps": 50, "fields": True},
        # A voxel body model (a material per blob on a graded mesh, so every row has its own coefficients) with
        # the transform of E over a region of interest at four frequencies.
        {"name": "voxel_dft_171x142x190", "kind": "engine", "nx": 171, "ny": 142, "nz": 190, "medium": "voxels",
         "wall": "cpml", "layers": 8, "mesh": 1, "curl": 0, "steps": 30, "dft": 4},
        # The training-data sweep of the learned stop: 64 small patch variants of uneven size.
        {"name": "batch_64_small", "kind": "batch", "models": 64, "lo": 30, "hi": 50, "graded": False, "steps": 50},
        # A design sweep of graded variants, with the energies the end criteria ask for.
        {"name": "batch_12_graded", "kind": "batch", "models": 12, "lo": 60, "hi": 128, "graded": True, "steps": 25,
         "energy": True},
        # The decision of the learned stop for a sweep's models.
        {"name": "net_forward_32", "kind": "forward", "batch": 32},
        # One training step at the default minibatch.
        {"name": "net_train_64", "kind": "train", "batch": 64},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stream", "engine", "engine", "engine", "engine", "batch", "batch", "forward", "train"])
    if kind in ("forward", "train"):
        return {"kind": kind, "batch": _spread(rng, 1, 256)}
    if kind == "batch":
        graded = rng.random() < 0.4
        lo = _spread(rng, 24, 70)
        return {"kind": "batch", "models": _spread(rng, 2, 12 if graded else 96), "lo": lo,
                "hi": lo + _spread(rng, 4, 60 if graded else 30), "graded": graded, "steps": _spread(rng, 10, 60),
                "energy": rng.random() < 0.5}
    if kind == "stream":
        n = [_spread(rng, 16, 64) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "medium": "vacuum", "wall": "cpml",
                "layers": rng.randint(3, 6), "mesh": rng.randint(0, 1), "curl": 0, "steps": 1}
    medium = rng.choice(["vacuum", "lossy", "dispersive", "trapezoidal", "voxels"])
    n = [_spread(rng, 28, 260) for _ in range(3)]
    wall = rng.choice(["cpml", "cpml", "pec", "upml" if medium in ("vacuum", "lossy") else "cpml"])
    c = {"kind": "engine", "nx": n[0], "ny": n[1], "nz": n[2], "medium": medium, "wall": wall,
         "layers": 0 if wall == "pec" else rng.randint(4, 10), "mesh": rng.randint(0, 1),
         "curl": 1 if wall == "upml" else 0, "steps": _spread(rng, 10, 60)}
    if wall != "upml" and rng.random() < 0.4:
        c["energy"] = True
    if rng.random() < 0.25:
        c["dft"] = rng.randint(1, 6)
    if n[0] * n[1] * n[2] < 200_000 and rng.random() < 0.5:
        c["fields"] = True
    return c


# ---------------------------------------------------------------------------
# Models.

def _lines(n, cell, mesh, rng):
    """n cells of about `cell`; mesh 1: graded by a slow wave and a jitter."""
    if not mesh:
        return np.arange(n + 1) * cell
    h = cell * (1.0 + 0.4 * np.sin(np.arange(n) * (2.0 * math.pi / max(n, 8)))) * rng.uniform(0.92, 1.08, n)
    return np.concatenate([[0.0], np.cumsum(h)])


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "energy", "dft", "fields")))


@functools.lru_cache(maxsize=2)
def _model(key):
    """(model, source op, port op, probe ops) of an engine case."""
    c = dict(key)
    n = [c["nx"], c["ny"], c["nz"]]
    lay = c["layers"]
    if c["medium"] == "patch":
        w = W.patch_antenna(steps=16)
        return w.model, None, w.port, []
    if c["medium"] == "dispersive" and c["nx"] == c["ny"] == c["nz"] >= 256:
        w = W.dispersive_box(n=n[0], cpml=lay, radius=n[0] * 80 / 512, slab=max(4, n[0] * 20 // 512), steps=16)
        return w.model, w.source, None, w.probes
    rng = np.random.default_rng(7 + 13 * n[0] + 17 * n[1] + 19 * n[2])
    cell = 0.5e-3 if c["medium"] in ("dispersive", "trapezoidal") else 1e-3
    m = E.Model(*[_lines(q, cell, c["mesh"], rng) for q in n])
    mid = [q / 2 for q in n]
    ball = m.cells().sphere(mid, 0.3 * min(n))
    if c["medium"] == "lossy":
        lo = [q // 4 for q in n]
        hi = [max(a + 1, 3 * q // 4) for a, q in zip(lo, n)]
        m.fill(m.cells().box(lo, [hi[0], hi[1], max(lo[2] + 1, n[2] // 2)]), m.material(eps_r=4.3, kappa=0.004))
        m.fill(m.cells().box([lo[0], lo[1], n[2] // 2], hi), m.material(eps_r=2.2, kappa=0.02, mu_r=1.1))
    elif c["medium"] == "voxels":
        for _ in range(40):
            at = [rng.uniform(0.25, 0.75) * q for q in n]
            mat = m.material(eps_r=rng.uniform(4.0, 60.0), kappa=rng.uniform(0.05, 2.0))
            m.fill(m.cells().sphere(at, rng.uniform(0.04, 0.16) * min(n)), mat)
    elif c["medium"] == "dispersive":
        m.fill(ball, m.material(eps_r=2.0))
    if c["wall"] == "pec":
        m.faces([E.PEC] * 6)
    m.build(courant=0.99)
    if c["wall"] == "cpml":
        m.add_cpml([min(lay, max(2, q // 4)) for q in n for _ in range(2)])
    elif c["wall"] == "upml":
        m.add_openems_pml([min(lay, max(2, q // 4)) for q in n for _ in range(2)])
    if c["medium"] in ("dispersive", "trapezoidal"):
        d = E.Dispersive()
        z0 = int(n[2] * 0.8)
        slab = m.cells().box([0, 0, z0], [n[0], n[1], min(n[2], z0 + max(2, n[2] // 25))])
        if c["medium"] == "dispersive":
            d.fill_cells(m, ball, W.lorentz_poles(5))
            d.fill_cells(m, slab, [E.Pole.drude(W.TWO_PI * 10e9, W.TWO_PI * 1e9)])
        else:
            half = m.cells().box([n[0] // 5, n[1] // 5, n[2] // 5], [n[0] - n[0] // 5, n[1] - n[1] // 5, n[2] // 2])
            d.fill_cells(m, half, [E.Pole.debye(3.0, 9.4e-12)] + W.lorentz_poles(5)[:1])
            d.fill_cells(m, slab, [E.Pole.drude(W.TWO_PI * 10e9, W.TWO_PI * 1e9)])
        m.add_dispersive(d, E.LEAPFROG if c["medium"] == "dispersive" else E.TRAPEZOIDAL)
    h = [q // 2 for q in n]
    src = m.add_source_table(E.SOFT_E, [(E.Z, (h[0], h[1], h[2]), 1.0)], np.zeros(1))
    pr = []
    for q in range(4):
        node = tuple(int(rng.integers(max(1, s // 5), max(2, s - s // 5))) for s in n)
        pr.append(m.add_probe(E.VOLTAGE, [(q % 3, node, 1.0)]))
    loop = [(E.X, tuple(h), 1.0), (E.X, (h[0], h[1] - 1, h[2]), -1.0), (E.Y, tuple(h), 1.0),
            (E.Y, (h[0] - 1, h[1], h[2]), -1.0)]
    pr.append(m.add_probe(E.CURRENT, loop, f32_sum=c["curl"] == 1))
    return m, src, None, pr


def _amplitude(case, seed, dt):
    """A carrier in the band, switched on over its first periods."""
    rng = np.random.default_rng([seed, 1])
    t = np.arange(TABLE) * dt
    f = rng.uniform(1.5e9, 5e9)
    return rng.uniform(0.5, 2.0) * np.sin(2 * math.pi * f * t + rng.uniform(0, 6)) * -np.expm1(-t * f)


def _modes(nodes, seed, comp):
    """A field component as a sum of cavity modes (f32, on the GPU), zero on every face."""
    rng = np.random.default_rng([seed, 2, comp])
    out = torch.zeros(nodes, dtype=torch.float32, device="cuda")
    for _ in range(3):
        v = []
        for q in nodes:
            x = torch.arange(q, device="cuda", dtype=torch.float64) / (q - 1)
            s = torch.sin(math.pi * int(rng.integers(1, 6)) * x)
            s[-1] = 0.0
            v.append(s.float())
        out += float(rng.uniform(-1e-3, 1e-3)) * v[0][:, None, None] * v[1][None, :, None] * v[2][None, None, :]
    return out


def _freqs(case):
    return np.linspace(1.0e9, 4.0e9, case["dft"])


def _dft_box(case):
    """Nodes lo..hi of the region the transform covers: a slab across the middle."""
    n = [case["nx"], case["ny"], case["nz"]]
    lo = [n[0] // 4, n[1] // 4, n[2] // 2 - 2]
    return lo, [3 * n[0] // 4, 3 * n[1] // 4, n[2] // 2 + 2]


def _batch_models(case, seed):
    rng = np.random.default_rng([seed, 3])
    models, ports = [], []
    for q in range(case["models"]):
        make = W.sweep_variant if case["graded"] else W.patch_variant
        w = make(1000 + q, cells=(case["lo"], case["hi"]), steps=TABLE // 10, cpml=min(8, case["lo"] // 5))
        n = w.model.nodes
        at = (n[0] // 2, n[1] // 2, n[2] // 2)
        t = np.arange(TABLE // 10) * w.model.dt
        amp = rng.uniform(0.5, 2.0) * np.sin(2 * math.pi * rng.uniform(1e9, 3e9) * t + rng.uniform(0, 6))
        w.model.add_source_table(E.SOFT_E, [(E.Z, at, 1.0)], amp)
        models.append(w.model)
        ports.append(w.port)
    return models, ports


def _records(case, seed):
    """Port records as the network reads them, (batch, K_IN, 2), and their
    tails: a band-limited burst that rings down (unit amplitude at the end)."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 1)
    b = case["batch"]
    r = lambda lo, hi: lo + (hi - lo) * torch.rand(b, 2, 1, generator=g, device="cuda")  # noqa: E731
    f, ph, tau = r(1e9, 3e9), r(0.0, 6.3), r(1e-9, 6e-9)

    def at(t):
        pulse = 200.0 * torch.exp(-(((t - 1.2e-9) / 0.4e-9) ** 2)) * torch.sin(2 * math.pi * 2e9 * t)
        ring = torch.exp(-(t - L.K_IN * L.DT_REF) / tau) * torch.sin(2 * math.pi * f * t + ph)
        return pulse + ring

    t = (torch.arange(L.K_IN, device="cuda") + 1.0) * L.DT_REF
    tt = torch.as_tensor(L.tail_times(), device="cuda", dtype=torch.float32)
    x = torch.asinh(at(t)).transpose(1, 2).contiguous()
    return x, at(tt).reshape(b, -1).contiguous()


# ---------------------------------------------------------------------------
# The timed calls.

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        net = L.Net(seed=seed)
        x, y = _records(case, seed)
        return {"case": case, "net": net, "x": x, "y": y}
    if kind == "batch":
        models, ports = _batch_models(case, seed)
        return {"case": case, "batch": E.Batch(models, max_steps=TABLE), "ports": ports}
    m, src, port, probes = _model(_key(case))
    e = E.Engine(m)
    if case["curl"]:
        e.set_curl_order(1)
    amp = _amplitude(case, seed, m.dt)
    st = {"case": case, "engine": e, "source": src, "port": port, "probes": probes, "amp": amp, "at": 0}
    if kind == "engine":
        e.source_amplitude(port if src is None else src, 0, amp)
    if case["medium"] != "patch":  # the antenna starts at rest, driven by its port
        for a in range(3):
            e.set_field(0, a, _modes(e.nodes, seed, a).cpu().numpy())
    if case.get("dft"):
        lo, hi = _dft_box(case)
        st["dump"] = e.add_freq_dump(0, lo, hi, _freqs(case))
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        return state["net"].forward(state["x"])
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["y"])
        return {"loss": loss, "gradient": net.g, "parameters": net.p}
    if kind == "batch":
        b = state["batch"]
        out = {}
        b.run(case["steps"] - (1 if case.get("energy") else 0))
        if case.get("energy"):
            out["energy"] = b.step_with_energy()
        out["v"] = np.stack([b.samples(q, p, 1) for q, p in enumerate(state["ports"])])
        out["i"] = np.stack([b.samples(q, p, 2) for q, p in enumerate(state["ports"])])
        return out
    e = state["engine"]
    if kind == "stream":
        n = state["at"]
        e.source_amplitude(state["source"], n, state["amp"][n:n + 1])
        e.run(1)
        state["at"] = n + 1
        return [e.last_sample(op) for op in state["probes"]]
    out = {}
    e.run(case["steps"] - (1 if case.get("energy") else 0))
    if case.get("energy"):
        out["energy"] = e.step_with_energy()
    if state["port"] is not None:
        out["v"] = e.samples(state["port"], 1)
        out["i"] = e.samples(state["port"], 2)
    if state["probes"]:
        out["series"] = np.stack([e.samples(op) for op in state["probes"]])
    if case.get("dft"):
        out["dft"] = [e.freq_dump(state["dump"], k) for k in range(case["dft"])]
    if case.get("fields"):
        out["fields"] = [e.field(f, a) for f in range(2) for a in range(3)]
    return out


# ---------------------------------------------------------------------------
# What a pass cannot do without.

def _sizes(case):
    """(cells, CPML values, pole edges, poles) of an engine case, estimated from its shapes."""
    n = [case["nx"], case["ny"], case["nz"]]
    cells = n[0] * n[1] * n[2]
    psi = 0
    if case["wall"] != "pec":
        faces = [0, 0] if case["medium"] == "patch" else None
        for a in range(3):
            lay = min(case["layers"], max(2, n[a] // 4)) * (1 if faces and a == 2 else 2)
            psi += 4 * lay * cells // n[a]
    edges = poles = 0
    if case["medium"] in ("dispersive", "trapezoidal"):
        if case["medium"] == "dispersive":
            r = n[0] * 80 / 512 if n[0] == n[1] == n[2] >= 256 else 0.3 * min(n)
            inner = 3 * 4 / 3 * math.pi * r ** 3
        else:
            inner = 3 * (n[0] * 0.6) * (n[1] * 0.6) * max(1, n[2] // 2 - n[2] // 5)
        slab = 3 * n[0] * n[1] * max(2, n[2] // 25)
        edges, poles = inner + slab, 2 * inner + slab
    return cells, psi, edges, poles


def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        shapes, T = L.layer_shapes()
        rows = [case["batch"] * t for t in T[1:]] + [case["batch"]] * 2
        macs = sum(r * co * fi for r, (_, co, fi) in zip(rows, shapes))
        params = sum(co * fi + co for _, co, fi in shapes)
        if kind == "forward":
            return {"bytes": case["batch"] * (8 * L.K_IN + 8 * L.T_OUT) + 2 * params, "flops": 2 * macs}
        first = rows[0] * shapes[0][1] * shapes[0][2]  # the input needs no gradient
        return {"bytes": case["batch"] * (8 * L.K_IN + 8 * L.T_OUT) + 30 * params, "flops": 2 * (3 * macs - first)}
    if kind == "batch":
        mean = (case["lo"] + case["hi"]) / 2
        cells = case["models"] * mean ** 3 * (1.0 if case["graded"] else 0.5)
        psi = case["models"] * mean ** 2 * 8 * 4 * (5 if case["graded"] else 3)
        return {"bytes": case["steps"] * (48 * cells + 24 * cells + 8 * psi), "flops": case["steps"] * 36 * cells}
    cells, psi, edges, poles = _sizes(case)
    # Per step: both fields read and written, the recursive convolution terms, the poles' state (f64) and the
    # coefficients that differ from node to node.
    dense = 24 if case["medium"] == "voxels" or case["mesh"] else 0
    per = (48 + dense) * cells + 8 * psi + 32 * poles + 8 * edges
    return {"bytes": case["steps"] * per, "flops": case["steps"] * (36 * cells + 8 * psi + 10 * poles)}


def tolerance(case):
    # The network multiplies bf16 operands: sums in another order flip roundings of what follows. Against a numpy
    # restatement with the same roundings the outputs differ by 2e-4 to 5e-4 and the gradient by 2e-4 to 6e-4 (largest
    # element 0.04 of the r.m.s.); Adam's first step turns a gradient near zero into a full step of either sign.
    if case["kind"] == "train":
        return {"rel": 5e-3, "max": 0.5}
    if case["kind"] == "forward":
        return {"rel": 2e-3, "max": 0.1}
    if case.get("energy"):
        # Field values and series are exact; the energy is one f64 sum whose order is free.
        return {"rel": 1e-11, "max": 1e-10}
    if case.get("dft"):
        return {"rel": 1e-12, "max": 1e-10}  # f64 accumulators; the phasor's last bit is free
    return "exact"


# ---------------------------------------------------------------------------
# The same results in 64 bits, by plain torch on the tables a case's model holds.

class _Lumped(C.Structure):
    _fields_ = [("axis", C.c_int32), ("n", C.c_size_t), ("node", C.c_void_p), ("cb", C.c_void_p), ("g", C.c_void_p),
                ("series", C.c_uint64), ("in_branch", C.c_int32), ("w", C.c_void_p), ("n_amp", C.c_size_t),
                ("amp", C.c_void_p), ("branch", C.c_int32), ("l", C.c_void_p), ("c", C.c_void_p), ("z", C.c_void_p),
                ("record", C.c_int32), ("rg", C.c_void_p), ("rc", C.c_void_p), ("columns", C.c_uint64)]


class _Source(C.Structure):
    _fields_ = [("kind", C.c_int32), ("n", C.c_size_t), ("axis", C.c_void_p), ("node", C.c_void_p), ("w", C.c_void_p),
                ("n_amp", C.c_size_t), ("amp", C.c_void_p)]


class _Probe(C.Structure):
    _fields_ = [("quantity", C.c_int32), ("n", C.c_size_t), ("axis", C.c_void_p), ("node", C.c_void_p),
                ("w", C.c_void_p), ("interval", C.c_uint64), ("f32", C.c_int32)]


_CT = {"f4": C.c_float, "f8": C.c_double, "u1": C.c_uint8, "u4": C.c_uint32, "u8": C.c_uint64}


def _arr(p, n, t):
    """A copy of n values at address p, as a tensor on the GPU (f64 or int64)."""
    if not n:
        return torch.zeros(0, dtype=torch.float64 if t[0] == "f" else torch.int64, device="cuda")
    a = np.ctypeslib.as_array((_CT[t] * int(n)).from_address(p))
    return torch.from_numpy(a.astype(np.float64 if t[0] == "f" else np.int64)).cuda()


class _Plain:
    """A model's leapfrog in 64 bits; `drive`: amplitudes by op index."""

    def __init__(self, model, drive):
        d = E.EngineDesc.from_address(model.desc)
        self.model = model
        self.N = N = [int(v) for v in d.nodes]
        self.dt = d.dt
        n = N[0] * N[1] * N[2]
        self.c = [_arr(d.coeff[q], n, "f4").view(N) for q in range(12)]
        self.u = [torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(3)]
        self.i = [torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(3)]
        self.ops, self.series, self.n = [], {}, 0
        kinds = (E.OpEntry * d.n_ops).from_address(d.ops) if d.n_ops else []
        for at, op in enumerate(kinds):
            self.ops.append((op.kind, at, self._table(op.kind, op.table, drive.get(at))))

    def _at(self, axis, node):
        """Flat places of edges in the three components joined."""
        return axis * (self.N[0] * self.N[1] * self.N[2]) + node

    def _table(self, kind, p, drive):
        if kind == E.OP_CPML:
            t = E.CpmlTable.from_address(p)
            out = []
            for s in (E.CpmlSlab * t.n_slabs).from_address(t.slabs):
                lo, hi = [int(v) for v in s.lo], [int(v) for v in s.hi]
                n = [h - q for h, q in zip(hi, lo)]
                if min(n) <= 0:
                    continue
                shape = [1, 1, 1]
                shape[s.normal] = n[s.normal]
                k = [_arr(x, n[s.normal], "f4").view(shape) for x in (s.b, s.a, s.k)]
                out.append((s.e_side, s.comp, s.normal, s.other, s.sign, lo, hi, k,
                            torch.zeros(n, dtype=torch.float64, device="cuda")))
            return out
        if kind == E.OP_POLES:
            t = E.PolesTable.from_address(p).electric
            end = _arr(t.pole_end, t.n_edges, "u4")
            count = torch.diff(end, prepend=torch.zeros(1, dtype=torch.int64, device="cuda"))
            axis, node = _arr(t.axis, t.n_edges, "u1"), _arr(t.node, t.n_edges, "u8")
            return {"at": self._at(axis, node), "of": torch.repeat_interleave(count),
                    "siz": _arr(t.sum_inv_z, t.n_edges, "f8"), "kind": _arr(t.kind, t.n_poles, "u1"),
                    "a": _arr(t.a, t.n_poles, "f8"), "ic": _arr(t.inv_c, t.n_poles, "f8"),
                    "iz": _arr(t.inv_z, t.n_poles, "f8"), "hl": _arr(t.half_l, t.n_poles, "f8"),
                    "j": torch.zeros(t.n_poles, dtype=torch.float64, device="cuda"),
                    "q": torch.zeros(t.n_poles, dtype=torch.float64, device="cuda"),
                    "cb": torch.stack(self.c[3:6]).view(-1)[self._at(axis, node)]}
        if kind == E.OP_LUMPED:
            t = _Lumped.from_address(p)
            amp = _arr(t.amp, t.n_amp, "f8").cpu().numpy() if drive is None else drive
            return {"axis": t.axis, "node": _arr(t.node, t.n, "u8"), "cbg": _arr(t.cb, t.n, "f8") * _arr(t.g, t.n, "f8"),
                    "w": _arr(t.w, t.n, "f8"), "rg": _arr(t.rg, t.n, "f8"), "rc": _arr(t.rc, t.n, "f8"),
                    "series": t.series, "columns": t.columns, "amp": amp}
        if kind == E.OP_SOURCE:
            t = _Source.from_address(p)
            amp = _arr(t.amp, t.n_amp, "f4").cpu().numpy() if drive is None else drive.astype(np.float32)
            return {"at": self._at(_arr(t.axis, t.n, "u1"), _arr(t.node, t.n, "u8")), "w": _arr(t.w, t.n, "f4"),
                    "amp": amp.astype(np.float64)}
        if kind == E.OP_PROBE:
            t = _Probe.from_address(p)
            return {"current": t.quantity == E.CURRENT, "w": _arr(t.w, t.n, "f8"),
                    "at": self._at(_arr(t.axis, t.n, "u1"), _arr(t.node, t.n, "u8"))}
        if kind == E.OP_UPML:
            t = E.UpmlTable.from_address(p)
            out = []
            for s in range(2):
                n = t.n[s]
                z = torch.zeros(n, dtype=torch.float64, device="cuda")
                out.append({"at": self._at(_arr(t.axis[s], n, "u1"), _arr(t.node[s], n, "u8")),
                            "co": _arr(t.co[s], 4 * n, "f4").view(-1, 4), "f": z, "v": z.clone()})
            return out
        raise ValueError("operator kind %d" % kind)

    def _get(self, f, at):
        n = self.N[0] * self.N[1] * self.N[2]
        out = torch.zeros(len(at), dtype=torch.float64, device="cuda")
        for a in range(3):
            m = at // n == a
            out[m] = f[a].view(-1)[at[m] - a * n]
        return out

    def _put(self, f, at, v):
        n = self.N[0] * self.N[1] * self.N[2]
        for a in range(3):
            m = at // n == a
            f[a].view(-1)[at[m] - a * n] = v[m]

    def _slabs(self, slabs, e_side):
        for es, comp, normal, other, sign, lo, hi, (b, a, k), psi in slabs:
            if es != e_side:
                continue
            box = tuple(slice(q, h) for q, h in zip(lo, hi))
            F = self.i[other] if e_side else self.u[other]
            if e_side:
                low = F[box].clone()
                prev = [slice(q, h) for q, h in zip(lo, hi)]
                prev[normal] = slice(max(lo[normal] - 1, 0), hi[normal] - 1)
                low.narrow(normal, 1 if lo[normal] == 0 else 0, prev[normal].stop - prev[normal].start).copy_(F[tuple(prev)])
                if lo[normal] == 0:
                    low.narrow(normal, 0, 1).zero_()
                s = sign * (F[box] - low)
                t, coef = self.u[comp], self.c[3 + comp][box]
            else:
                up = [slice(q, h) for q, h in zip(lo, hi)]
                up[normal] = slice(lo[normal] + 1, hi[normal] + 1)
                s = sign * (F[tuple(up)] - F[box])
                t, coef = self.i[comp], -self.c[9 + comp][box]
            psi.mul_(b).add_(a * s)
            t[box] += coef * (k * s + psi)

    def _upml(self, sides, done):
        """After the update of side `done`: the other side's start values, then this side's layer update."""
        F = (self.u, self.i)
        other, me = sides[1 - done], sides[done]
        if len(other["at"]):
            other["v"] = self._get(F[1 - done], other["at"])
        if len(me["at"]):
            f1 = me["co"][:, 0] * me["f"] + self._get(F[done], me["at"])
            me["v"] = me["co"][:, 1] * me["v"] - me["co"][:, 3] * me["f"] + me["co"][:, 2] * f1
            me["f"] = f1
            self._put(F[done], me["at"], me["v"])

    def step(self, energy=False):
        u, i, c, dt = self.u, self.i, self.c, self.dt
        w = torch.zeros((), dtype=torch.float64, device="cuda")
        if energy:
            for kind, _, t in self.ops:
                if kind == E.OP_POLES:
                    w += (t["hl"] * t["j"] ** 2 + 0.5 * t["ic"] * t["q"] ** 2).sum()
            old = [x.clone() for x in i]
        i[0][:, :-1, :-1] = (c[6] * i[0])[:, :-1, :-1] - c[9][:, :-1, :-1] * (
            (u[2][:, 1:, :-1] - u[2][:, :-1, :-1]) - (u[1][:, :-1, 1:] - u[1][:, :-1, :-1]))
        i[1][:-1, :, :-1] = (c[7] * i[1])[:-1, :, :-1] - c[10][:-1, :, :-1] * (
            (u[0][:-1, :, 1:] - u[0][:-1, :, :-1]) - (u[2][1:, :, :-1] - u[2][:-1, :, :-1]))
        i[2][:-1, :-1] = (c[8] * i[2])[:-1, :-1] - c[11][:-1, :-1] * (
            (u[1][1:, :-1] - u[1][:-1, :-1]) - (u[0][:-1, 1:] - u[0][:-1, :-1]))
        if energy:
            for a in range(3):
                for x, ca, cb in ((u[a] * u[a], c[a], c[3 + a]), (old[a] * i[a], c[6 + a], c[9 + a])):
                    if x is not None:
                        ok = cb != 0
                        w += 0.25 * dt * ((1 + ca[ok]) * x[ok] / cb[ok]).sum()
            del old
        for kind, _, t in self.ops:
            if kind == E.OP_CPML:
                self._slabs(t, 0)
            elif kind == E.OP_UPML:
                self._upml(t, 1)
        for kind, at, t in self.ops:
            if kind == E.OP_PROBE and t["current"]:
                self.series.setdefault(at, []).append((t["w"] * self._get(i, t["at"])).sum())
        prev = {at: self._get(u, t["at"]) for kind, at, t in self.ops if kind == E.OP_POLES}
        u0 = {at: u[t["axis"]].view(-1)[t["node"]].clone() for kind, at, t in self.ops if kind == E.OP_LUMPED}
        dx = lambda x: torch.diff(x, dim=0, prepend=torch.zeros_like(x[:1]))  # noqa: E731
        dy = lambda x: torch.diff(x, dim=1, prepend=torch.zeros_like(x[:, :1]))  # noqa: E731
        dz = lambda x: torch.diff(x, dim=2, prepend=torch.zeros_like(x[:, :, :1]))  # noqa: E731
        u[0][:-1] = (c[0] * u[0] + c[3] * (dy(i[2]) - dz(i[1])))[:-1]
        u[1][:, :-1] = (c[1] * u[1] + c[4] * (dz(i[0]) - dx(i[2])))[:, :-1]
        u[2][:, :, :-1] = (c[2] * u[2] + c[5] * (dx(i[1]) - dy(i[0])))[:, :, :-1]
        for kind, at, t in self.ops:
            if kind == E.OP_CPML:
                self._slabs(t, 1)
            elif kind == E.OP_UPML:
                self._upml(t, 0)
            elif kind == E.OP_POLES:
                p = prev[at][t["of"]]
                leap = t["kind"] == E.LEAPFROG
                kk = t["a"] * t["j"] - t["q"] * t["ic"] + 0.5 * p
                jn = t["a"] * t["j"] + t["iz"] * (p - t["q"] * t["ic"])
                s = torch.zeros(len(t["at"]), dtype=torch.float64, device="cuda")
                s.index_add_(0, t["of"], torch.where(leap, jn, kk * t["iz"]))
                x = (self._get(u, t["at"]) - t["cb"] * s) / (1 + 0.5 * t["cb"] * t["siz"])
                self._put(u, t["at"], x)
                jb = (kk + 0.5 * x[t["of"]]) * t["iz"]
                t["q"] += dt * torch.where(leap, jn, jb)
                t["j"] = torch.where(leap, jn, 2 * jb - t["j"])
        for kind, at, t in self.ops:
            if kind == E.OP_LUMPED:
                f = u[t["axis"]].view(-1)
                v = t["w"] * (float(t["amp"][self.n]) if self.n < len(t["amp"]) else 0.0)
                f[t["node"]] += t["cbg"] * v
                u1 = f[t["node"]]
                rec = (t["rg"] * (0.5 * (u0[at] + u1) - v) + t["rc"] * (u1 - u0[at]) / dt).sum() / t["series"]
                self.series.setdefault(at, []).append(torch.stack([u1.sum() / t["columns"], -rec]))
            elif kind == E.OP_SOURCE:
                a = float(t["amp"][self.n]) if self.n < len(t["amp"]) else 0.0
                self._put(u, t["at"], self._get(u, t["at"]) + t["w"] * a)
            elif kind == E.OP_PROBE and not t["current"]:
                self.series.setdefault(at, []).append((t["w"] * self._get(u, t["at"])).sum())
        self.n += 1
        return float(w) if energy else 0.0

    def of(self, op):
        return torch.stack(self.series[op]).cpu().numpy()


def _exact_engine(case, seed):
    if case["nx"] * case["ny"] * case["nz"] * case["steps"] > 400_000_000:
        return None
    m, src, port, probes = _model(_key(case))
    p = _Plain(m, {port if src is None else src: _amplitude(case, seed, m.dt)})
    if case["medium"] != "patch":
        for a in range(3):
            p.u[a].copy_(_modes(p.N, seed, a).double())
    acc = None
    if case.get("dft"):
        lo, hi = _dft_box(case)
        box = tuple(slice(q, h + 1) for q, h in zip(lo, hi))
        inv = [torch.from_numpy(m.inv_edge_lengths(a)).cuda() for a in range(3)]
        shape = [[-1, 1, 1], [1, -1, 1], [1, 1, -1]]
        acc = [0.0] * case["dft"]

        def sample(k):
            x = torch.stack([(p.u[a] * inv[a].view(shape[a]))[box] for a in range(3)], dim=-1)
            for q, f in enumerate(_freqs(case)):
                acc[q] = acc[q] + x * (complex(np.exp(-2j * math.pi * ((f * k * m.dt) % 1.0))) * m.dt)

        sample(0)
    w = 0.0
    for k in range(case["steps"]):
        w = p.step(energy=bool(case.get("energy")) and k == case["steps"] - 1)
        if acc is not None:
            sample(k + 1)
    if case["kind"] == "stream":
        return [float(p.of(op)[-1]) for op in probes]
    out = {}
    if case.get("energy"):
        out["energy"] = w
    if port is not None:
        vi = p.of(port)
        out["v"], out["i"] = vi[:, 0].copy(), vi[:, 1].copy()
    if probes:
        out["series"] = np.stack([p.of(op) for op in probes])
    if acc is not None:
        out["dft"] = [x.cpu().numpy() for x in acc]
    if case.get("fields"):
        out["fields"] = [x.cpu().numpy() for x in p.u + p.i]
    return out


def _exact_net(case, seed):
    x, y = _records(case, seed)
    flat = torch.from_numpy(L.init_params(seed)).double().cuda().requires_grad_(True)
    p = L.param_views(flat)
    a = x.double().transpose(1, 2)
    for (W_, b), (ci, co, k, s) in zip(p, L.CONVS):
        w = W_.view(co, k, ci).permute(0, 2, 1)
        cols = a.unfold(2, k, s)  # (batch, ci, out, k)
        a = torch.nn.functional.silu(torch.einsum("bitk,oik->bot", cols, w) + b[None, :, None])
    h = torch.nn.functional.silu(a.transpose(1, 2).reshape(x.shape[0], -1) @ p[3][0].T + p[3][1])
    out = h @ p[4][0].T + p[4][1]
    if case["kind"] == "forward":
        return out.detach()
    loss = ((out - y.double()) ** 2).mean()
    g, = torch.autograd.grad(loss, flat)
    step = 1e-3 * g / (g.abs() + 1e-8)  # the first Adam step: m / (1 - b1) = g, sqrt(v / (1 - b2)) = |g|
    return {"loss": loss.detach().reshape(1), "gradient": g, "parameters": flat.detach() - step}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        return _exact_net(case, seed)
    if kind != "batch":
        return _exact_engine(case, seed)
    models, ports = _batch_models(case, seed)
    v, i, w = [], [], []
    for m, port in zip(models, ports):
        p = _Plain(m, {})
        e = 0.0
        for k in range(case["steps"]):
            e = p.step(energy=bool(case.get("energy")) and k == case["steps"] - 1)
        w.append(e)
        vi = p.of(port)
        v.append(vi[:, 0])
        i.append(vi[:, 1])
    out = {"v": np.stack(v), "i": np.stack(i)}
    if case.get("energy"):
        out["energy"] = np.array(w)
    return out
