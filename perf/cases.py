"""The calls whose speed matters to a user of this framework, with inputs, minimal work and 64-bit results.

Four kinds of use, each through the package's public entry points:

* ``source``: one evaluation of the right-hand side on the device (``Workspace.source_device``), as a program
  with a stepper of its own calls it, on the capillary's field grid or the graded-index fibre's envelope grid;
* ``run``: a run's first attempts from a host field (``Workspace.start``, ``Session.advance``,
  ``Session.export``): exponential Adams on the field grid, Runge-Kutta on the envelope grid;
* ``scan``: batch steps of many uneven runs and the read-back of their states (``Scan.advance``, ``Scan.run``);
* ``infer`` / ``train``: the scan surrogate's ensemble inference and one member's training step.

Sizes are those of the package's workload builders (``scan.draw_points``, ``grin.grin_record``,
``surrogate.HIDDEN``) and of the committed four-mode gradient capillary under ``tests/golden``.
"""

from __future__ import annotations

import dataclasses
import json
import math
import random
from pathlib import Path

import numpy as np
import torch

from solprop_b200 import _lib, grin, scan, surrogate
from solprop_b200.record import load_record

EPS0 = 8.8541878188e-12
CAP = 2e-5  # the mixed scans' largest step over their length
GOLDEN = Path(__file__).resolve().parents[1] / "tests" / "golden"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a one-mode capillary on the shortest scan grid, where launches and latency count
        {"name": "source_one_mode", "kind": "source", "grid": "capillary", "modes": 1, "n_to": 4096,
         "precision": "fp64"},
        # the largest capillary of the scan's distribution: eight modes on 64 nodes and the longest rows
        {"name": "source_eight_modes", "kind": "source", "grid": "capillary", "modes": 8, "n_to": 32768,
         "precision": "fp64"},
        # an odd mode count in the mixed form, the ordinary grid of a few-cycle run
        {"name": "source_five_modes_mixed", "kind": "source", "grid": "capillary", "modes": 5, "n_to": 16384,
         "precision": "mixed"},
        # soliton-driven wave generation in a pressure gradient (four modes, band-rule plasma integrals, an
        # 18-term operator expansion): the start of the adaptive run, host field in and host field out
        {"name": "run_gradient", "kind": "run", "grid": "gradient", "attempts": 48, "precision": "fp64"},
        # a one-mode run in the mixed form
        {"name": "run_one_mode_mixed", "kind": "run", "grid": "capillary", "modes": 1, "n_to": 8192,
         "attempts": 48, "precision": "mixed"},
        # a parameter scan with part of its runs left, stepped together, its states read back now and then
        {"name": "scan_mixed", "kind": "scan", "runs": 96, "steps": 24, "precision": "mixed"},
        # the envelope grid's ordinary GNLSE: one mode, a delayed Raman response, Runge-Kutta steps
        {"name": "run_gnlse", "kind": "run", "grid": "gnlse", "n_to": 4096, "attempts": 4, "precision": "fp64"},
        # the graded-index fibre at full size: 30 vector modes, 128 x 128 nodes, two components, tensor Raman
        {"name": "source_fibre_mixed", "kind": "source", "grid": "fibre", "nodes": 128, "n_to": 16384,
         "precision": "mixed"},
        # the fibre in the plain form on an odd quadrature
        {"name": "source_fibre", "kind": "source", "grid": "fibre", "nodes": 45, "n_to": 8192,
         "precision": "fp64"},
        # a coarse fibre run, the first thing a user tries: short rows, few nodes, Runge-Kutta steps
        {"name": "run_fibre_mixed", "kind": "run", "grid": "fibre", "nodes": 24, "n_to": 4096, "attempts": 3,
         "precision": "mixed"},
        # screening a scan: five members over a chunk of points
        {"name": "infer_chunk", "kind": "infer", "rows": 16384},
        # one optimiser step of one member on the training's batch
        {"name": "train_step", "kind": "train", "rows": 256},
    ]


def draw(rng: random.Random):
    kind = rng.choices(["source", "fibre", "run", "fibre_run", "scan", "infer", "train"],
                       [4, 4, 3, 2, 1, 2, 2])[0]
    precision = rng.choice(["fp64", "mixed"])
    if kind == "source":
        return {"kind": "source", "grid": "capillary", "modes": rng.randint(1, 8), "n_to": 2 ** rng.randint(12, 15),
                "precision": precision}
    if kind == "fibre":
        n_to = 2 ** rng.randint(10, 14)
        most = 128 if precision == "mixed" else 64
        return {"kind": "source", "grid": "fibre", "nodes": round(math.exp(rng.uniform(math.log(5), math.log(most)))),
                "n_to": n_to, "precision": precision}
    if kind == "run":
        return {"kind": "run", "grid": "capillary", "modes": rng.randint(1, 8), "n_to": 2 ** rng.randint(12, 15),
                "attempts": rng.randint(16, 64), "precision": precision}
    if kind == "fibre_run":
        if rng.random() < 0.3:
            return {"kind": "run", "grid": "gnlse", "n_to": 2 ** rng.randint(10, 12), "attempts": rng.randint(1, 8),
                    "precision": "fp64"}
        return {"kind": "run", "grid": "fibre", "nodes": rng.randint(7, 40), "n_to": 2 ** rng.randint(10, 13),
                "attempts": rng.randint(1, 3), "precision": precision}
    if kind == "scan":
        return {"kind": "scan", "runs": rng.randint(8, 96), "steps": rng.randint(4, 24), "precision": precision}
    if kind == "infer":
        return {"kind": "infer", "rows": round(math.exp(rng.uniform(math.log(128), math.log(16384))))}
    return {"kind": "train", "rows": round(math.exp(rng.uniform(math.log(32), math.log(1024))))}


# ------------------------------------------------------------------ the problems
def _point(case, seed):
    """A capillary run of the case's size: argon at a bar, a hundred microjoules in ten femtoseconds, drawn
    around these from the seed."""
    rng = np.random.default_rng(seed)
    return scan.ScanPoint(radius=125e-6, length=1.0, gas="Ar", pressure=1.0,
                          energy=float(rng.uniform(80e-6, 120e-6)), fwhm=float(rng.uniform(9.5e-15, 10.5e-15)),
                          modes=case["modes"], n_to=case["n_to"], seed=int(seed))


def _points(case, seed):
    """A scan's points: the distribution's sizes, the same for every seed, and the seed's physics.  The mixed
    scans are of helium and at most fifty microjoules (see ``_march``)."""
    sizes = scan.draw_points(case["runs"], 2024)
    mixed = case["precision"] == "mixed"
    return [dataclasses.replace(p, modes=q.modes, n_to=q.n_to, gas="He" if mixed else p.gas,
                                energy=min(p.energy, 5e-5) if mixed else p.energy)
            for p, q in zip(scan.draw_points(case["runs"], seed), sizes)]


def _gnlse(n_to, seed):
    """One scalar mode of the graded-index fibre: its axial field alone, no collar."""
    rec, policy = grin.grin_record(n_to=n_to, grid=4, seed=seed)
    peak = 1.0 / math.sqrt(0.5 * EPS0 * grin.C0 * 1.2e-10)  # a 120 um^2 effective area, one watt
    one = slice(0, 1)
    rec = dataclasses.replace(
        rec, n_modes=1, n_nodes=1, n_pol_transform=1, phi_terms=rec.phi_terms[:, one],
        prefactor_terms=rec.prefactor_terms[:, one], synthesis=np.array([[peak]]), projection=np.array([[1.0 / peak]]),
        projection_coarse=np.array([[1.0 / peak]]), raman_tensor_weights=None, absorber_scheme="none",
        temporal_absorber_fine=None, field0=rec.field0[one] * 0.5)
    return rec, policy


def _problem(case, seed):
    if case["grid"] == "capillary":
        return scan.capillary_record(_point(case, seed))
    if case["grid"] == "gnlse":
        return _gnlse(case["n_to"], seed)
    if case["grid"] == "fibre":
        return grin.grin_record(n_to=case["n_to"], grid=case["nodes"], seed=seed)
    rec = load_record(GOLDEN / "config2.problem.npz")
    with np.load(GOLDEN / "config2.golden.npz") as data:
        policy = json.loads(bytes(data["adaptive.policy"]).decode())
    return rec, policy


def _march(policy, precision):
    """A scan's march policy: as it stands in the plain form.  In the mixed form its steps are capped (a march's
    largest step is the user's to set) below what the error control would take: the error norms' 32-bit noise
    would otherwise choose other steps, and two correct implementations would stand at different places after as
    many attempts."""
    if precision == "fp64":
        return policy
    cap = CAP * policy["z_end"]
    return dict(policy, dz_max=cap, proposal=cap)


def _field(rec, seed):
    """A field part of the way down the guide: the launch, its energy leaked into every mode with seeded phases."""
    rng = np.random.default_rng(seed + 17)
    field = rec.launch_field()
    mixed = field + 0.1 * np.exp(2j * np.pi * rng.uniform(size=(rec.n_modes, 1, 1))) * field[:1]
    return np.ascontiguousarray(mixed * rec.active_mask)


def _schedule(case, rec):
    """A run's fixed steps, or None for the adaptive march.  The envelope runs and the mixed form take fixed
    steps, so that every implementation takes the same ones: the plain form's error norms are exact enough to
    choose the same steps again, 32-bit noise in them is not."""
    if rec.grid_kind == "field":
        return np.full(case["attempts"], 5e-5 * rec.z_end) if case["precision"] == "mixed" else None
    return np.geomspace(2e-5, 1e-4, case["attempts"]) if case["attempts"] > 1 else np.array([5e-5])


def _features(rows, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, (rows, surrogate.N_IN)).astype(np.float32)


def _targets(x, seed):
    """Standardised log spectra that depend smoothly on the features, with noise."""
    rng = np.random.default_rng(seed + 5)
    lines = np.linspace(0.0, 6.0, surrogate.N_OUT)
    y = np.sin(x[:, :1] * lines + x[:, 1:2]) + 0.5 * np.cos(x[:, 3:4] + x[:, 4:5] * lines)
    return (y + 0.1 * rng.standard_normal(y.shape)).astype(np.float32)


def _moments(shape, seed):
    """Adam's moments in the middle of a training run."""
    rng = np.random.default_rng(seed)
    return ((1e-5 * rng.standard_normal(shape)).astype(np.float32),
            (1e-10 * rng.uniform(0.5, 2.0, shape)).astype(np.float32))


# ------------------------------------------------------------------ the measured calls
def prepare(case, seed):
    kind = case["kind"]
    if kind == "source":
        rec, _ = _problem(case, seed)
        ws = _lib.Workspace(_lib.Problem(rec), 0, case["precision"])
        lab = torch.from_numpy(_field(rec, seed)).cuda()
        return {"kind": kind, "ws": ws, "lab": lab, "out": torch.empty_like(lab)}
    if kind == "run":
        rec, policy = _problem(case, seed)
        ws = _lib.Workspace(_lib.Problem(rec), 0, case["precision"])
        field = rec.launch_field() if case["grid"] != "gradient" else _field(rec, seed)
        return {"kind": kind, "ws": ws, "policy": policy, "field": field, "steps": _schedule(case, rec),
                "attempts": case["attempts"]}
    if kind == "scan":
        built = [scan.capillary_record(p) for p in _points(case, seed)]
        batch = _lib.Scan([b[0] for b in built], [_march(b[1], case["precision"]) for b in built], 0,
                          case["precision"])
        batch.set_alone(0)  # a run that goes on alone makes as many attempts as the clock lets it
        return {"kind": kind, "scan": batch, "steps": case["steps"], "runs": case["runs"]}
    x = _features(case["rows"], seed)
    if kind == "infer":
        ensemble = surrogate.Ensemble(seed=int(seed))
        for member in ensemble.members:
            member.refresh_bf16()
        return {"kind": kind, "ensemble": ensemble, "x": torch.from_numpy(x).cuda()}
    member = surrogate.Perceptron(int(seed))
    for i, (m1, m2) in enumerate(zip(member.m1, member.m2)):
        first, second = _moments(tuple(m1.shape), seed + i)
        m1.copy_(torch.from_numpy(first))
        m2.copy_(torch.from_numpy(second))
    member.step = 100
    return {"kind": kind, "member": member, "x": torch.from_numpy(x).cuda(),
            "y": torch.from_numpy(_targets(x, seed)).cuda()}


def run(state):
    kind = state["kind"]
    if kind == "source":
        state["ws"].source_device(state["lab"].data_ptr(), 0.0, state["out"].data_ptr())
        return state["out"]
    if kind == "run":
        session = state["ws"].start(state["policy"], field0=state["field"], schedule=state["steps"])
        session.advance(state["attempts"])
        out = session.export()
        session.close()
        return out
    if kind == "scan":
        state["scan"].advance(state["steps"])
        return np.concatenate([state["scan"].run(i)[0].ravel() for i in range(state["runs"])])
    if kind == "infer":
        return state["ensemble"].infer(state["x"])[0]
    member = state["member"]
    out, cache, status = member.forward_tc(state["x"], keep=True)
    loss, dy = surrogate.mse(out, state["y"])
    grads, status = member.gradients_tc(cache, dy, status=status)
    member.adam(grads, 1e-3)
    return {"out": out, "loss": loss, "grads": grads, "params": member.params}


# ------------------------------------------------------------------ minimal work and tolerances
def _source_work(modes, nodes, n_to, n_omega, envelope):
    """Bytes and operations of one source evaluation: the field in and the source out, with the operator's
    arrays; the transforms' 5 n log n (2.5 for real rows), the modal products' 2 per term, the node responses."""
    fft = lambda n: 5.0 * n * math.log2(n)  # noqa: E731
    bytes_ = 16.0 * modes * n_omega * 3 + 16.0 * n_to + 16.0 * modes * nodes
    if envelope:
        components = 2 if modes > 1 else 1
        rows = components * nodes
        convolutions = 3 if components == 2 else 1
        flops = modes * 3 * fft(n_to) + 4.0 * 2 * rows * modes * n_to / components
        flops += nodes * (convolutions * 2 * 0.5 * fft(2 * n_to) + 40.0 * convolutions * n_to)
    else:
        flops = modes * (0.5 * fft(n_to) * 5) + 2.0 * 4 * modes * nodes * n_to + 80.0 * nodes * n_to
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind in ("infer", "train"):
        sizes = (surrogate.N_IN,) + surrogate.HIDDEN + (surrogate.N_OUT,)
        weights = sum(a * b + b for a, b in zip(sizes[:-1], sizes[1:]))
        rows = case["rows"]
        if kind == "infer":
            return {"bytes": 5 * (2.0 * weights + 4.0 * rows * surrogate.N_OUT) + 4.0 * rows * surrogate.N_IN,
                    "flops": 5 * 2.0 * rows * weights}
        return {"bytes": 4.0 * weights * 7 + 4.0 * rows * 2 * surrogate.N_OUT, "flops": 6.0 * rows * weights}
    if kind == "scan":
        bytes_ = flops = 0.0
        for p in _points(case, 1):
            b, f = _source_work(p.modes, max(8, 8 * p.modes), p.n_to, p.n_to // 4 + 1, False)
            bytes_, flops = bytes_ + b, flops + f
        return {"bytes": case["steps"] * bytes_, "flops": case["steps"] * flops}
    if case["grid"] == "gradient":
        b, f = _source_work(4, 64, 16384, 4097, False)
    elif case["grid"] == "capillary":
        b, f = _source_work(case["modes"], 8 * case["modes"], case["n_to"], case["n_to"] // 4 + 1, False)
    elif case["grid"] == "gnlse":
        b, f = _source_work(1, 1, case["n_to"], case["n_to"], True)
    else:
        b, f = _source_work(30, case["nodes"] ** 2, case["n_to"], case["n_to"], True)
    if kind == "source":
        return {"bytes": b, "flops": f}
    evaluations = case["attempts"] * (7 if case["grid"] in ("gnlse", "fibre") else 1)
    return {"bytes": evaluations * b, "flops": evaluations * f}


def tolerance(case):
    """About four times what a perturbation of the inputs by one rounding, or the 64-bit result, shows."""
    kind, mixed = case["kind"], case.get("precision") == "mixed"
    if kind in ("infer", "train"):
        return {"rel": 2e-2}
    if kind == "scan":
        return {"rel": 1e-7 if mixed else 2e-10}  # mixed: 32-bit sources over the share of the field they change
    if case["grid"] in ("capillary", "gradient"):
        if kind == "run":
            return {"rel": 3e-7 if mixed else 2e-10}
        return {"rel": 1e-6 if mixed else 1e-13}
    if kind == "run":
        return {"rel": 2e-6 if mixed else 1e-13}
    return {"rel": 2e-5 if mixed else 1e-13}


# ------------------------------------------------------------------ the same results in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _constant(table):
    return 1.0 if table is None else float(table.coefficients[0, 0, 0])


def _rate(rec, magnitude):
    c = _t(rec.rate_coefficients, magnitude.device)
    inside = (magnitude >= rec.field_min) & (magnitude <= rec.field_max)
    lf = torch.log(torch.where(inside, magnitude, torch.full_like(magnitude, rec.field_min)))
    index = ((lf - rec.log_field_min) / rec.d_log_field).long().clamp(0, c.shape[1] - 1)
    local = lf - (rec.log_field_min + index.double() * rec.d_log_field)
    value = torch.exp(((c[0][index] * local + c[1][index]) * local + c[2][index]) * local + c[3][index])
    value = torch.where(inside, value, torch.zeros_like(value))
    return torch.where(magnitude > rec.field_max, torch.full_like(value, rec.rate_max), value)


def _running(values, dt):
    out = torch.zeros_like(values)
    out[:, 1:] = torch.cumsum(0.5 * dt * (values[:, 1:] + values[:, :-1]), dim=1)
    return out


def _field_source(rec, lab):
    """The field grid's source (Kerr, plasma with the trapezoid rule, the in-stage collar)."""
    dev, n_to, n_omega = lab.device, rec.n_to, rec.n_omega
    fine = torch.zeros((rec.n_modes, n_to // 2 + 1), dtype=torch.complex128, device=dev)
    fine[:, :n_omega] = lab[:, 0]
    modal = torch.fft.irfft(fine, n=n_to)
    gate, gate_d = _t(rec.t_window, dev), _t(rec.t_window_derivative, dev)
    field = _t(rec.synthesis, dev) @ modal
    magnitude = field.abs()
    rate = _rate(rec, magnitude)
    f0 = _constant(rec.preionisation)
    fraction = 1.0 - (1.0 - f0) * torch.exp(-_running(rate, rec.dt_fine))
    free = _running(fraction * rec.charge_mass_ratio * field, rec.dt_fine)
    loss = torch.where(rate > 0, rec.ionisation_potential * rate * (1.0 - fraction) / magnitude.clamp_min(1e-300) ** 2,
                       torch.zeros_like(rate))
    current = _constant(rec.plasma_density) * (free + loss * field)
    kerr = rec.kerr_coefficient * _constant(rec.kerr_density) * field ** 3
    projection = _t(rec.projection, dev)
    spectrum = torch.fft.rfft(projection @ (kerr * gate))[:, :n_omega]
    gated = torch.fft.rfft(projection @ (gate * current))[:, :n_omega]
    edge = torch.fft.rfft(projection @ (gate_d * current))[:, :n_omega]
    active = _t(rec.active_mask, dev)
    iw = 1j * torch.where(active, _t(rec.omega, dev), torch.ones(n_omega, dtype=torch.float64, device=dev))
    spectrum = spectrum + torch.where(active, gated / iw - edge / iw ** 2, torch.zeros_like(gated))
    absorber = torch.fft.rfft(-0.5 * _t(rec.temporal_absorber_fine, dev) * modal)[:, :n_omega] * active
    out = _t(rec.prefactor_terms[0][:, 0], dev) * _t(rec.omega_window, dev) * spectrum + absorber
    return out[:, None, :]


def _fibre_source(rec, lab):
    """The envelope grid's source: the analytic Kerr cubic, scalar or tensor Raman, the collar."""
    dev, n = lab.device, rec.n_to
    modal = torch.fft.ifft(lab[:, 0])
    pols = rec.n_pol_transform
    t = torch.arange(2 * n, dtype=torch.float64, device=dev) * rec.dt_fine
    damped = _t(rec.raman_undamped[0], dev) * torch.exp(-_constant(rec.raman_rates[0]) * t)
    kernel = torch.fft.rfft(rec.raman_fraction * damped) * rec.dt_fine
    rho = _constant(rec.raman_density)
    factor = rec.kerr_coefficient * _constant(rec.kerr_density)
    gate = _t(rec.t_window, dev)
    synthesis, projection = _t(rec.synthesis, dev), _t(rec.projection, dev)
    weights = (1.0, 0.0) if rec.raman_tensor_weights is None else rec.raman_tensor_weights[0]

    def convolve(weight, drive):
        return float(weight) * torch.fft.irfft(kernel * torch.fft.rfft(drive, n=2 * n), n=2 * n)[:, :n]

    projected = torch.zeros_like(modal)
    chunk = max(1, 2 ** 22 // n)
    for i in range(0, rec.n_nodes, chunk):
        rows = slice(i * pols, min(i + chunk, rec.n_nodes) * pols)
        field = torch.complex(synthesis[rows] @ modal.real, synthesis[rows] @ modal.imag)
        comps = [field[p::pols] for p in range(pols)]
        intensities = [0.5 * (c.real ** 2 + c.imag ** 2) for c in comps]
        squares = sum(c * c for c in comps)
        moduli = 2.0 * sum(intensities)
        u = convolve(weights[0], sum(intensities))
        if pols == 2:
            v = convolve(weights[1], intensities[0] - intensities[1])
            w = convolve(weights[1], comps[0].real * comps[1].real + comps[0].imag * comps[1].imag)
            raman = [(u + v) * comps[0] + w * comps[1], w * comps[0] + (u - v) * comps[1]]
        else:
            raman = [u * comps[0]]
        for p in range(pols):
            total = factor * (rec.kerr_self * moduli * comps[p] + rec.kerr_conjugate * squares * comps[p].conj())
            total = (total + EPS0 * rho * raman[p]) * gate
            part = projection[:, rows][:, p::pols]
            projected += torch.complex(part @ total.real, part @ total.imag)
    out = _t(rec.prefactor_terms[0][:, 0], dev) * _t(rec.omega_window, dev) * torch.fft.fft(projected)
    if rec.absorber_scheme == "nonlinear":
        term = -0.5 * _t(rec.temporal_absorber_fine, dev) * modal
        out = out + torch.fft.fft(term) * _t(rec.active_mask, dev)
    return out[:, None, :]


_MATRIX = ((), (1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
           (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
           (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
           (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
_NODES = (0.0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1.0, 1.0)


def _runge_kutta(rec, field, steps):
    """Interaction-picture Dormand-Prince steps with the operator D of a uniform guide (the last weights row is
    the solution's)."""
    dev = field.device
    operator = _t(rec.phi_terms[0], dev)
    active = _t(rec.active_mask, dev)
    state = field * active
    for dz in steps:
        stages = []
        for node, row in zip(_NODES, _MATRIX):
            inner = state + dz * sum(a * k for a, k in zip(row, stages)) if row else state
            there = torch.exp(node * dz * operator)
            stages.append(_fibre_source(rec, there * inner) / there)
        solution = sum(a * k for a, k in zip(_MATRIX[6], stages))
        state = torch.exp(dz * operator) * (state + dz * solution) * active
    return state


def _member(seed):
    """A freshly initialised member's weights and biases, in 64 bits."""
    m = surrogate.Perceptron(int(seed))
    return [w.double() for w in m.weights], [b.double() for b in m.biases]


def _perceptron(weights, biases, x):
    for w, b in zip(weights[:-1], biases[:-1]):
        x = torch.nn.functional.gelu(x @ w.T + b)
    return x @ weights[-1].T + biases[-1]


def exact(case, seed):
    kind, dev = case["kind"], _device()
    if kind == "source":
        rec, _ = _problem(case, seed)
        lab = _t(_field(rec, seed), dev)
        out = _field_source(rec, lab) if rec.grid_kind == "field" else _fibre_source(rec, lab)
        return out
    if kind == "run" and case["grid"] in ("gnlse", "fibre"):
        rec, _ = _problem(case, seed)
        return _runge_kutta(rec, _t(rec.launch_field(), dev), _schedule(case, rec)).cpu().numpy()
    if kind in ("run", "scan"):
        return None  # adaptive multistep runs: the sources above are their 64-bit check
    x = _t(_features(case["rows"], seed), dev).double()
    if kind == "infer":
        return torch.stack([_perceptron(*_member(seed + 1000 * k), x) for k in range(5)])
    weights, biases = _member(seed)
    params = [t.requires_grad_() for pair in zip(weights, biases) for t in pair]
    out = _perceptron(weights, biases, x)
    loss = ((out - _t(_targets(_features(case["rows"], seed), seed), dev)) ** 2).mean()
    grads = torch.autograd.grad(loss, params)
    updated = []
    for i, (p, g) in enumerate(zip(params, grads)):
        m1, m2 = (_t(m, dev).double() for m in _moments(tuple(p.shape), seed + i))
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        step = (m1 / (1.0 - 0.9 ** 101)) / (torch.sqrt(m2 / (1.0 - 0.999 ** 101)) + 1e-8)
        updated.append((p - 1e-3 * step).detach())
    return {"out": out.detach(), "loss": loss.detach()[None], "grads": list(grads), "params": updated}
