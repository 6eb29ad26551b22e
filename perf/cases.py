"""Workloads of the framework, each through its public entry points.

``listed()`` names them, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes a
workload's inputs (and the plan or batch that a program keeps between calls), ``run`` is one pass,
``work`` its least traffic and arithmetic, and ``exact`` the same outputs in float64 from plain torch.

The kinds:

* ``call``      one drop-in call ``kspaceFirstOrder2D/3D(kgrid, source, sensor, medium, options)`` from
                host arrays to host results;
* ``plan``      one more simulation on a plan that is kept: a new initial pressure, all time steps,
                the recorded results (parameter studies, training data);
* ``batch``     transmit events of different sizes advanced together, new source signals each pass;
* ``recon``     one iteration's passes of a reconstruction: forward, residual, adjoint;
* ``gradient``  misfit and its gradients with respect to initial pressure and sound speed;
* ``conv``      one 3x3 convolution layer of the warm-start network, forward or backward.
"""
import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "k-wave-python_gb300"))

import kwave_gb300  # noqa: E402
from kwave_gb300 import unet_ops  # noqa: E402
from kwave_gb300.adjoint import LinearP0, misfit_gradients  # noqa: E402
from kwave_gb300.solver import Simulation, SimulationBatch  # noqa: E402

_CONV_LAYERS = {  # (input channels, upsampled input channels, output channels) of the network, image size / its grid
    (32, 0, 32): 1, (64, 0, 64): 2, (128, 0, 128): 4, (128, 0, 256): 8, (256, 0, 256): 8,
    (128, 256, 128): 4, (64, 128, 64): 2, (32, 64, 32): 1,
}


def listed():
    return [
        # the reference's own first example: a small homogeneous 2-D run with a circle of sensors
        {"name": "water_2d_128", "kind": "call", "nx": 128, "ny": 128, "nz": 0, "nt": 604, "tissue": False,
         "source": "p0", "sensor": "circle", "record_u": False, "pml": 20},
        # one ultrasound transmit in speckled tissue, pressure and velocity recorded, sizes of no power of two
        {"name": "transmit_2d_375x324", "kind": "call", "nx": 375, "ny": 324, "nz": 0, "nt": 600, "tissue": True,
         "source": "array", "sensor": "plane", "record_u": True, "pml": 20},
        # the headline: heterogeneous, absorbing, nonlinear tissue on 256^3
        {"name": "tissue_3d_256", "kind": "call", "nx": 256, "ny": 256, "nz": 256, "nt": 250, "tissue": True,
         "source": "p0", "sensor": "plane", "record_u": False, "pml": 10},
        # a phantom study on a small volume: launches and latency
        {"name": "water_3d_64", "kind": "plan", "nx": 64, "ny": 64, "nz": 64, "nt": 300, "tissue": False,
         "source": "p0", "sensor": "plane", "record_u": False, "pml": 10},
        # tissue volumes of sizes that users pick (small prime factors), ordinary and large
        {"name": "tissue_3d_216x180x150", "kind": "plan", "nx": 216, "ny": 180, "nz": 150, "nt": 100, "tissue": True,
         "source": "p0", "sensor": "plane", "record_u": False, "pml": 10},
        {"name": "tissue_3d_432x384x320", "kind": "plan", "nx": 432, "ny": 384, "nz": 320, "nt": 40, "tissue": True,
         "source": "p0", "sensor": "plane", "record_u": False, "pml": 10},
        # transmit events of uneven sizes in one batch
        {"name": "batch_32_transmits", "kind": "batch", "members": 32, "low": 192, "high": 512, "nt": 500, "pml": 20},
        # one iteration of the 512^2 photoacoustic reconstruction
        {"name": "recon_2d_512", "kind": "recon", "nx": 512, "ny": 512, "nt": 1500, "points": 256, "pml": 20},
        # a sound-speed inversion's gradient on an uneven grid
        {"name": "gradient_2d_300x240", "kind": "gradient", "nx": 300, "ny": 240, "nt": 500, "points": 100, "pml": 20},
        # the network's layers: full resolution and decoder in training, the bottom level at inference
        {"name": "conv_back_32to32_256", "kind": "conv", "c1": 32, "c2": 0, "cout": 32, "size": 256, "images": 16,
         "backward": True},
        {"name": "conv_back_384to128_64", "kind": "conv", "c1": 128, "c2": 256, "cout": 128, "size": 64, "images": 16,
         "backward": True},
        {"name": "conv_fwd_256to256_32", "kind": "conv", "c1": 256, "c2": 0, "cout": 256, "size": 32, "images": 4,
         "backward": False},
    ]


def _smooth_sizes(low, high):
    """Lengths the transforms take: products of 2, 3, 5 and 7."""
    out = []
    for n in range(low, high + 1):
        m = n
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        if m == 1:
            out.append(n)
    return out


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["call", "call", "plan", "plan", "plan", "batch", "recon", "gradient", "conv", "conv"])

    def size(low, high):
        return min(_smooth_sizes(low, high), key=lambda n, t=_log_int(rng, low, high): abs(n - t))

    if kind in ("call", "plan"):
        if rng.random() < 0.45:
            nx, ny, nz, pml = size(72, 1024), size(72, 1024), 0, rng.choice([10, 20])
            nt = min(_log_int(rng, 100, 1200), int(2.5e8 / (nx * ny)))
        else:
            nx, ny, nz, pml = size(40, 400), size(40, 400), size(40, 400), 10
            nt = max(10, min(_log_int(rng, 50, 400), int(1.0e9 / (nx * ny * nz))))
        source = "array" if kind == "call" and ny >= 96 and rng.random() < 0.5 else "p0"
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "nt": nt, "tissue": rng.random() < 0.6, "source": source,
                "sensor": rng.choice(["plane", "circle"]) if nz == 0 else "plane",
                "record_u": kind == "call" and rng.random() < 0.3, "pml": pml}
    if kind == "batch":
        low = size(128, 256)
        return {"kind": kind, "members": _log_int(rng, 4, 32), "low": low, "high": size(low + 64, 512),
                "nt": _log_int(rng, 200, 500), "pml": 20}
    if kind == "recon":
        nx, ny = size(96, 512), size(96, 512)
        return {"kind": kind, "nx": nx, "ny": ny, "nt": _log_int(rng, 200, 1200), "points": rng.randrange(50, 257),
                "pml": 20}
    if kind == "gradient":
        nx, ny = size(80, 360), size(80, 360)
        return {"kind": kind, "nx": nx, "ny": ny, "nt": _log_int(rng, 150, 500), "points": rng.randrange(40, 130),
                "pml": rng.choice([10, 20])}
    c1, c2, cout = rng.choice(sorted(_CONV_LAYERS))
    full = rng.choice([96, 128, 160, 192, 256])
    return {"kind": kind, "c1": c1, "c2": c2, "cout": cout, "size": full // _CONV_LAYERS[(c1, c2, cout)],
            "images": rng.randrange(1, 17), "backward": rng.random() < 0.6}


# ---------------------------------------------------------------------------
# problems, as plain dicts of host arrays
# ---------------------------------------------------------------------------
def _blobs(shape, rng, pml, count, sigma, amplitude):
    """Gaussian blobs inside the absorbing layer, each added on its own box."""
    p0 = np.zeros(shape)
    for _ in range(count):
        s, a = rng.uniform(*sigma), rng.uniform(*amplitude)
        c = [rng.uniform(pml, n - pml) for n in shape]
        r = int(math.ceil(5 * s)) + 1
        box = tuple(slice(max(0, int(x) - r), min(n, int(x) + r + 1)) for x, n in zip(c, shape))
        r2 = sum((g - x) ** 2 for g, x in zip(np.ogrid[box], c))
        p0[box] += a * np.exp(-r2 / (2 * s * s))
    return p0


def _tissue(shape, rng, pml):
    """Sound speed and density: speckle in 2-D, homogeneous in 3-D, with ellipsoidal inclusions."""
    c, rho = np.full(shape, 1540.0), np.full(shape, 1000.0)
    if len(shape) == 2:
        c *= 1 + 0.02 * rng.standard_normal(shape)
        rho *= 1 + 0.02 * rng.standard_normal(shape)
    for _ in range(3 if len(shape) == 2 else 8):
        centre = [rng.uniform(pml, n - pml) for n in shape]
        semi = [rng.uniform(0.03, 0.12) * n for n in shape]
        box = tuple(slice(max(0, int(x - s) - 1), min(n, int(x + s) + 2)) for x, s, n in zip(centre, semi, shape))
        inside = sum(((g - x) / s) ** 2 for g, x, s in zip(np.ogrid[box], centre, semi)) <= 1.0
        c[box] = np.where(inside, c[box] * rng.uniform(0.91, 1.16), c[box])
        rho[box] = np.where(inside, rho[box] * rng.uniform(0.9, 1.2), rho[box])
    return c, rho


def _circle(points, radius):
    angle = 2 * np.pi * np.arange(points) / points
    return np.stack([radius * np.cos(angle), radius * np.sin(angle)])


def _array_source(problem, rng, f0=1.5e6, cycles=3):
    """A steered linear array behind the absorbing layer, each element's points driven by a tone burst."""
    shape, dx, dt, pml = problem["shape"], problem["spacing"][0], problem["dt"], problem["pml_size"][0]
    ny = shape[1]
    elements = min(32, (ny - 2 * pml - 8) // 4)
    element_of = np.full(shape, -1)
    first = (ny - 4 * elements) // 2
    for e in range(elements):
        rows = slice(first + 4 * e, first + 4 * e + 3)
        if len(shape) == 2:
            element_of[pml + 2, rows] = e
        else:
            element_of[pml + 2, rows, shape[2] // 2] = e
    mask = element_of >= 0
    y = np.arange(elements) * 4 * dx
    delay = (y - y.mean()) * math.sin(math.radians(rng.uniform(-30, 30))) / 1540.0
    delay -= delay.min()
    burst = cycles / f0
    time = np.arange(int(math.ceil((burst + delay.max()) / dt)) + 1) * dt
    local = time[None, :] - delay[element_of[mask]][:, None]
    envelope = np.exp(-((local - burst / 2) / (burst / 4)) ** 2) * ((local >= 0) & (local <= burst))
    return mask, 1e4 * rng.uniform(0.5, 2.0) * envelope * np.sin(2 * np.pi * f0 * local)


def _simulation(case, seed, smooth):
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())
    dx, pml = (1e-4 if case["source"] == "p0" else 5e-5), case["pml"]
    problem = dict(shape=shape, spacing=(dx,) * len(shape), Nt=case["nt"], pml_size=(pml,) * len(shape),
                   pml_alpha=(2.0,) * len(shape), use_sg=True, use_kspace=True, smooth_p0=smooth)
    if case["tissue"]:
        c, rho = _tissue(shape, rng, pml)
        problem.update(sound_speed=c, density=rho, alpha_coeff=0.75, alpha_power=1.5, BonA=6.0)
    else:
        problem.update(sound_speed=1500.0, density=1000.0)
    problem["dt"] = 0.3 * dx / float(np.max(problem["sound_speed"]))
    if case["source"] == "p0":
        problem["p0"] = _blobs(shape, rng, pml, 12 if len(shape) == 2 else 40, (2, 6), (1, 10))
    else:
        problem["p_mask"], problem["p"] = _array_source(problem, rng)
        problem["p_mode"] = "additive"
    if case["sensor"] == "circle":
        problem["sensor_mask"] = _circle(50, 0.3 * min(shape) * dx)
    else:
        mask = np.zeros(shape, bool)
        mask[..., shape[-1] // 2] = True
        problem["sensor_mask"] = mask
    problem["record"] = ("p", "p_max") + (("u",) if case["record_u"] else ())
    return problem


def _transmits(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.array(_smooth_sizes(case["low"], case["high"]))
    layout = np.random.default_rng(case["members"] * 1000 + case["low"])  # the batch's grids stay as they are
    problems = []
    for _ in range(case["members"]):
        shape = tuple(int(n) for n in layout.choice(sizes, 2))
        c, rho = _tissue(shape, layout, case["pml"])
        p = dict(shape=shape, spacing=(5e-5, 5e-5), Nt=case["nt"], sound_speed=c, density=rho, alpha_coeff=0.5,
                 alpha_power=1.1, pml_size=(case["pml"],) * 2, pml_alpha=(2.0, 2.0), use_sg=True, use_kspace=True,
                 smooth_p0=False, dt=0.3 * 5e-5 / float(c.max()), p_mode="additive", record=("p",))
        p["p_mask"], p["p"] = _array_source(p, layout)
        p["sensor_mask"] = p["p_mask"].copy()
        p["p"] = p["p"] * rng.uniform(0.5, 2.0, (p["p"].shape[0], 1))  # this pass's apodisation
        problems.append(p)
    return problems


def _inversion(case, seed):
    """A reconstruction's problem, its present estimate, and the noisy data of the true phantom."""
    rng = np.random.default_rng(seed)
    shape, dx = (case["nx"], case["ny"]), 5e-5
    problem = dict(shape=shape, spacing=(dx, dx), Nt=case["nt"], dt=0.3 * dx / 1500.0, sound_speed=1500.0,
                   density=1000.0, pml_size=(case["pml"],) * 2, pml_alpha=(2.0, 2.0), use_sg=True, use_kspace=True,
                   smooth_p0=False, record=("p",),
                   sensor_mask=_circle(case["points"], (0.5 * min(shape) - case["pml"] - 4) * dx))
    true = _blobs(shape, rng, case["pml"], 12, (1, 4), (0.5, 2))
    estimate = 0.5 * true + 0.2 * _blobs(shape, rng, case["pml"], 12, (1, 4), (0.5, 2))
    data = _Exact(dict(problem, p0=true)).run()["p"].cpu().numpy()
    data += 0.01 * data.std() * rng.standard_normal(data.shape)
    return problem, estimate, data


def _conv_inputs(case, seed):
    """A layer's tensors in NHWC bf16: activations after ReLU, their output gradient, He-scaled weights."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    n, s, c1, c2, cout = case["images"], case["size"], case["c1"], case["c2"], case["cout"]
    t = {"x1": torch.relu(normal(n, s, s, c1)).to(torch.bfloat16),
         "x2": torch.relu(normal(n, s // 2, s // 2, c2)).to(torch.bfloat16) if c2 else None,
         "w": (normal(cout, 9, c1 + c2) * math.sqrt(2 / (9 * (c1 + c2)))).to(torch.bfloat16),
         "b": 0.1 * normal(cout)}
    if case["backward"]:
        t["y"] = torch.relu(normal(n, s, s, cout)).to(torch.bfloat16)
        t["dy"] = (1e-3 * normal(n, s, s, cout)).to(torch.bfloat16)
    return t


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "call":
        p = _simulation(case, seed, smooth=True)
        names = ("shape", "spacing", "Nt", "dt")
        shape, spacing, nt, dt = (p[k] for k in names)
        return {"kind": kind, "simulate": kwave_gb300.kspaceFirstOrder3D if case["nz"] else kwave_gb300.kspaceFirstOrder2D,
                "kgrid": SimpleNamespace(N=np.array(shape), spacing=np.array(spacing), Nt=nt, dt=dt, dim=len(shape)),
                "medium": SimpleNamespace(**{k: p.get(k) for k in ("sound_speed", "density", "alpha_coeff", "alpha_power",
                                                                   "BonA")}),
                "source": SimpleNamespace(**{k: p.get(k) for k in ("p0", "p_mask", "p", "p_mode")}),
                "sensor": SimpleNamespace(mask=p["sensor_mask"], record=p["record"], record_start_index=1),
                "options": SimpleNamespace(pml_size=p["pml_size"], pml_alpha=p["pml_alpha"], use_sg=True, use_kspace=True,
                                           smooth_p0=True)}
    if kind == "plan":
        p = _simulation(case, seed, smooth=False)
        return {"kind": kind, "sim": Simulation.from_problem(p).setup(), "p0": p["p0"]}
    if kind == "batch":
        problems = _transmits(case, seed)
        return {"kind": kind, "batch": SimulationBatch.from_problems(problems), "problems": problems}
    if kind == "recon":
        problem, estimate, data = _inversion(case, seed)
        return {"kind": kind, "map": LinearP0(problem), "estimate": estimate, "data": data}
    if kind == "gradient":
        problem, estimate, data = _inversion(case, seed)
        rng = np.random.default_rng(seed + 1)
        return {"kind": kind, "problem": problem, "estimate": estimate, "data": data,
                "c": 1500.0 - _blobs(problem["shape"], rng, case["pml"], 6, (4, 10), (2, 10))}
    t = _conv_inputs(case, seed)
    if case["backward"]:
        t["dw"] = torch.zeros(t["w"].shape, device="cuda")
        t["db"] = torch.zeros(t["b"].shape, device="cuda")
    return {"kind": kind, **t}


def run(state):
    kind = state["kind"]
    if kind == "call":
        return state["simulate"](state["kgrid"], state["source"], state["sensor"], state["medium"], state["options"])
    if kind == "plan":
        sim = state["sim"]
        sim._plan.update_p0(state["p0"])
        sim._plan.run(sim.Nt)
        sim._plan.sync()
        return sim.results()
    if kind == "batch":
        batch = state["batch"]
        for sim, problem in zip(batch.sims, state["problems"]):
            sim._plan.update_sources(problem)
            sim.t = 0
        return [r["p"] for r in batch.run()]
    if kind == "recon":
        d = state["map"].forward(state["estimate"])
        return {"p": d, "gradient": state["map"].adjoint(d - state["data"])}
    if kind == "gradient":
        misfit, g_p0, g_c = misfit_gradients(state["problem"], state["estimate"], state["data"], c=state["c"])
        return {"misfit": misfit, "g_p0": g_p0, "g_c": g_c}
    if "dy" not in state:
        return unet_ops.conv3x3(state["x1"], state["w"], state["b"], relu=True, x2=state["x2"])[0]
    # a training step's backward pass of the layer
    dz = unet_ops.relu_grad(state["dy"], state["y"])
    unet_ops.conv3x3_wgrad(state["x1"], dz, state["dw"].zero_(), x2=state["x2"])
    unet_ops.bias_grad(dz, state["db"].zero_())
    dx, _ = unet_ops.conv3x3(dz, unet_ops.flip_weights(state["w"]))
    return {"dw": state["dw"], "db": state["db"], "dx": dx}


def work(case):
    """Time steps: the wave field read and written and the medium read once a step, and the transforms."""
    kind = case["kind"]
    if kind == "conv":
        n, s, c1, c2, cout = case["images"], case["size"], case["c1"], case["c2"], case["cout"]
        x = n * s * s * c1 + n * (s // 2) ** 2 * c2
        macs = n * s * s * 9 * (c1 + c2) * cout
        weights, y = 9 * (c1 + c2) * cout, n * s * s * cout
        if not case["backward"]:
            return {"bytes": 2 * (x + weights + y), "flops": 2 * macs}
        return {"bytes": 2 * (x + 2 * y + weights + n * s * s * (c1 + c2)) + 4 * (weights + cout), "flops": 4 * macs}

    def steps(shape, nt, fields, grids, transforms):
        cells = math.prod(shape)
        return nt * cells * 4 * (2 * fields + grids), nt * transforms * 2.5 * cells * math.log2(cells)

    if kind in ("call", "plan"):
        shape = (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())
        dim = len(shape)
        # pressure, velocity and split density; c0, rho0, tau, eta, B/A where the medium is tissue
        b, f = steps(shape, case["nt"], 2 * dim + 1, 5 if case["tissue"] else 0, 1 + 3 * dim + (4 if case["tissue"] else 0))
        return {"bytes": b, "flops": f}
    if kind == "batch":
        got = [steps(p["shape"], case["nt"], 5, 5, 11) for p in _transmits(case, 0)]
        return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}
    # forward and transposed steps; the gradient reruns the forward steps from its checkpoints
    b, f = steps((case["nx"], case["ny"]), case["nt"], 5, 0, 7)
    return {"bytes": (2 if kind == "recon" else 3) * b, "flops": (2 if kind == "recon" else 3) * f}


# ---------------------------------------------------------------------------
# the same in float64, from plain torch
# ---------------------------------------------------------------------------
class _Exact:
    """The k-space first-order time loop and its transpose, on real half-spectrum transforms in float64."""

    def __init__(self, p):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.shape, self.dim = p, tuple(p["shape"]), len(p["shape"])
        self.dt, self.nt = p["dt"], p["Nt"]
        self.c, self.rho0 = self._grid(p["sound_speed"]), self._grid(p["density"])
        c_ref = float(p["c_ref"]) if p.get("c_ref") is not None else float(np.max(np.asarray(p["sound_speed"], np.float32)))
        k = [2 * np.pi * np.fft.fftfreq(n, d) for n, d in zip(self.shape, p["spacing"])]
        half = self.shape[-1] // 2 + 1

        def along(values, a, spectrum=True):
            values = values[:half] if spectrum and a == self.dim - 1 else values
            size = [1] * self.dim
            size[a] = len(values)
            return torch.as_tensor(np.ascontiguousarray(values), device=self.device).reshape(size)

        k_mag = sum(along(x, a) ** 2 for a, x in enumerate(k)).sqrt()
        phase = 0.5 * c_ref * self.dt * k_mag
        kappa = torch.where(phase == 0, torch.ones_like(phase), torch.sin(phase) / phase.clamp_min(1e-300))
        self.source_kappa = torch.cos(phase)

        def shifted(a, sign, derivative=True):
            t = np.exp(sign * 0.5j * k[a] * p["spacing"][a]) * (1j * k[a] if derivative else 1.0)
            # the part that maps real fields to real fields (it differs at an even length's last frequency)
            return along(0.5 * (t + np.conj(t[-np.arange(len(t))])), a)

        self.grad = [shifted(a, 1) * kappa for a in range(self.dim)]
        self.div = [shifted(a, -1) * kappa for a in range(self.dim)]
        self.back = [shifted(a, -1, False) for a in range(self.dim)]
        self.pml, self.pml_sg = ([along(self._layer(a, c_ref, s), a, False) for a in range(self.dim)] for s in (0.0, 0.5))
        self.dt_rho = [self.dt / self._between(self.rho0, a) for a in range(self.dim)]
        self.tau = None
        if p.get("alpha_coeff"):
            y = p["alpha_power"]
            alpha = 100.0 * p["alpha_coeff"] * (1e-6 / (2 * np.pi)) ** y / (20 * np.log10(np.e))
            self.tau, self.eta = -2 * alpha * self.c ** (y - 1), 2 * alpha * self.c ** y * math.tan(math.pi * y / 2)
            safe = torch.where(k_mag == 0, torch.ones_like(k_mag), k_mag)
            self.nabla = [torch.where(k_mag == 0, torch.zeros_like(k_mag), safe ** (y + e)) for e in (-2, -1)]
        self._sensor()

    def _grid(self, v):
        return torch.as_tensor(np.asarray(v, np.float64), device=self.device)

    def _layer(self, a, c_ref, shift):
        n, size, alpha, dx = self.shape[a], self.p["pml_size"][a], self.p["pml_alpha"][a], self.p["spacing"][a]
        x = np.arange(1, size + 1) + shift
        out = np.ones(n)
        out[:size] = np.exp(-alpha * c_ref / dx * ((size + 1 - x) / size) ** 4 * self.dt / 2)
        out[n - size:] = np.exp(-alpha * c_ref / dx * (x / size) ** 4 * self.dt / 2)
        return out

    def _between(self, f, a):
        """Neighbour mean along an axis, the last plane kept."""
        if f.dim() == 0:
            return f
        n = f.shape[a]
        return torch.cat([0.5 * (f.narrow(a, 0, n - 1) + f.narrow(a, 1, n - 1)), f.narrow(a, n - 1, 1)], a)

    def _sensor(self):
        m = np.asarray(self.p["sensor_mask"])
        if m.dtype == bool:
            self.at = torch.as_tensor(np.flatnonzero(m), device=self.device)[:, None]
            self.weight = torch.ones_like(self.at, dtype=torch.float64)
            return
        at, weight = np.zeros((m.shape[1], 1), np.int64), np.ones((m.shape[1], 1))
        for a in range(self.dim):  # multilinear interpolation between grid points
            x = m[a] / self.p["spacing"][a] + self.shape[a] // 2
            i = np.clip(np.floor(x).astype(np.int64), 0, self.shape[a] - 2)
            f = (x - i)[:, None]
            at = np.concatenate([at * self.shape[a] + i[:, None], at * self.shape[a] + i[:, None] + 1], 1)
            weight = np.concatenate([weight * (1 - f), weight * f], 1)
        self.at, self.weight = torch.as_tensor(at, device=self.device), torch.as_tensor(weight, device=self.device)

    def sample(self, f):
        return (f.reshape(-1)[self.at] * self.weight).sum(1)

    def spread(self, r):
        out = torch.zeros(math.prod(self.shape), dtype=torch.float64, device=self.device)
        return out.index_add_(0, self.at.reshape(-1), (self.weight * r[:, None]).reshape(-1)).reshape(self.shape)

    def fft(self, f):
        return torch.fft.rfftn(f)

    def real(self, f):
        return torch.fft.irfftn(f, s=self.shape)

    def smoothed(self, p0):
        """Radially symmetric Blackman filter, scaled back to the largest value."""
        sizes = [n + 1 - n % 2 for n in self.shape]
        length = max(sizes)
        x = np.arange(length) / (length - 1)
        window = 0.42 - 0.5 * np.cos(2 * np.pi * x) + 0.08 * np.cos(4 * np.pi * x)
        radius = (length - 1) / 2
        axes = [np.fft.ifftshift(np.linspace(-radius, radius, m)[:n]) ** 2 for m, n in zip(sizes, self.shape)]
        r = np.sqrt(sum(np.reshape(x, [-1 if i == a else 1 for i in range(self.dim)]) for a, x in enumerate(axes)))
        w = np.abs(np.interp(np.minimum(r, radius), np.linspace(-radius, radius, length), window))
        s = torch.fft.ifftn(torch.fft.fftn(p0) * torch.as_tensor(w, device=self.device)).real
        return s * (p0.abs().max() / s.abs().max())

    def start(self, p0):
        rho = [p0 / (self.c ** 2 * self.dim) for _ in range(self.dim)]
        pk = self.fft(p0)
        return p0, [0.5 * self.dt_rho[i] * self.real(self.grad[i] * pk) for i in range(self.dim)], rho

    def run(self, keep=None):
        """Recorded series and the largest pressure of each point; ``keep`` collects each step's density."""
        p = self.p
        zero = torch.zeros(self.shape, dtype=torch.float64, device=self.device)
        pr, u, rho = zero, [zero] * self.dim, [zero] * self.dim
        out = {k: [] for k in ["p"] + ["u" + a for a in "xyz"[: self.dim]]}
        if p.get("p0") is not None:
            p0 = self._grid(p["p0"])
            pr, u, rho = self.start(self.smoothed(p0) if p["smooth_p0"] else p0)
        signal = None
        if p.get("p_mask") is not None:
            where = torch.as_tensor(np.flatnonzero(p["p_mask"]), device=self.device)
            c = self.c.reshape(-1)[where] if self.c.dim() else self.c
            signal = torch.as_tensor(p["p"], device=self.device) * (2 * self.dt / (self.dim * c)).reshape(-1, 1)
        for t in range(self.nt):
            if t > 0 or p.get("p0") is None:
                pk = self.fft(pr)
                sg, pml = self.pml_sg, self.pml
                u = [sg[i] * (sg[i] * u[i] - self.dt_rho[i] * self.real(self.grad[i] * pk)) for i in range(self.dim)]
                total = sum(rho)
                b = self.dt * (2 * total + self.rho0) if p.get("BonA") else self.dt * self.rho0
                du = [self.real(self.div[i] * self.fft(u[i])) for i in range(self.dim)]
                rho = [pml[i] * (pml[i] * rho[i] - b * du[i]) for i in range(self.dim)]
                if signal is not None and t < signal.shape[1]:
                    s = torch.zeros_like(zero).reshape(-1).index_copy_(0, where, signal[:, t]).reshape(self.shape)
                    s = self.real(self.source_kappa * self.fft(s))
                    rho = [rho[i] + s / p["spacing"][i] for i in range(self.dim)]
                total = sum(rho)
                if keep is not None:
                    keep.append(total)
                eos = total
                if self.tau is not None:
                    eos = eos + self.tau * self.real(self.nabla[0] * self.fft(self.rho0 * sum(du)))
                    eos = eos - self.eta * self.real(self.nabla[1] * self.fft(total))
                if p.get("BonA"):
                    eos = eos + p["BonA"] * total ** 2 / (2 * self.rho0)
                pr = self.c ** 2 * eos
            out["p"].append(self.sample(pr))
            if "u" in p["record"]:
                for i in range(self.dim):
                    out["u" + "xyz"[i]].append(self.sample(self.real(self.back[i] * self.fft(u[i]))))
        out = {k: torch.stack(v, 1) for k, v in out.items() if v}
        if "p_max" in p["record"]:
            out["p_max"] = out["p"].amax(1)
        return out

    def transposed(self, r, totals=None, p0=None):
        """Gradients with respect to the initial pressure, and to the sound speed where ``totals`` are given."""
        zero = torch.zeros(self.shape, dtype=torch.float64, device=self.device)
        lp, lu, lr, gc2 = zero, [zero] * self.dim, [zero] * self.dim, zero
        c2, b = self.c ** 2, self.dt * self.rho0

        def derivative(op, f):
            return self.real(op * self.fft(f))

        for t in range(self.nt - 1, 0, -1):
            lp = lp + self.spread(r[:, t])
            if totals is not None:
                gc2 = gc2 + totals[t - 1] * lp
            for i in range(self.dim):
                m, sg = self.pml[i], self.pml_sg[i]
                lr[i] = lr[i] + c2 * lp
                lu[i] = lu[i] + derivative(self.grad[i], b * m * lr[i])
                lr[i] = m * m * lr[i]
            lp = sum(derivative(self.div[i], self.dt_rho[i] * self.pml_sg[i] * lu[i]) for i in range(self.dim))
            lu = [self.pml_sg[i] ** 2 * lu[i] for i in range(self.dim)]
        g = lp + self.spread(r[:, 0])
        for i in range(self.dim):
            g = g + lr[i] / (c2 * self.dim) - derivative(self.div[i], 0.5 * self.dt_rho[i] * lu[i])
            if totals is not None:
                gc2 = gc2 - p0 * lr[i] / (c2 * c2 * self.dim)
        return g, 2 * self.c * gc2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("call", "plan"):
        return _Exact(_simulation(case, seed, smooth=kind == "call")).run()
    if kind == "batch":
        return [_Exact(p).run()["p"] for p in _transmits(case, seed)]
    if kind == "recon":
        problem, estimate, data = _inversion(case, seed)
        e = _Exact(dict(problem, p0=estimate))
        d = e.run()["p"]
        return {"p": d, "gradient": e.transposed(d - e._grid(data))[0]}
    if kind == "gradient":
        problem, estimate, data = _inversion(case, seed)
        c = 1500.0 - _blobs(problem["shape"], np.random.default_rng(seed + 1), case["pml"], 6, (4, 10), (2, 10))
        e = _Exact(dict(problem, p0=estimate, sound_speed=c, c_ref=1500.0))
        totals = []
        r = e.run(totals)["p"] - e._grid(data)
        g_p0, g_c = e.transposed(r, totals, e._grid(estimate))
        return {"misfit": float(0.5 * (r * r).sum()), "g_p0": g_p0, "g_c": g_c}
    t = {k: v.double() if v is not None else None for k, v in _conv_inputs(case, seed).items()}
    x = t["x1"].permute(0, 3, 1, 2)
    if t["x2"] is not None:
        up = t["x2"].repeat_interleave(2, 1).repeat_interleave(2, 2)
        x = torch.cat([x, up.permute(0, 3, 1, 2)], 1)
    cin, cout = x.shape[1], case["cout"]
    w = t["w"].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
    if not case["backward"]:
        y = torch.relu(torch.nn.functional.conv2d(x, w, padding=1) + t["b"].reshape(1, -1, 1, 1))
        return y.permute(0, 2, 3, 1)
    dz = torch.where(t["y"] > 0, t["dy"], torch.zeros_like(t["dy"]))
    flat, s = dz.reshape(-1, cout), x.shape[2]
    padded = torch.nn.functional.pad(x, (1, 1, 1, 1))
    dw = torch.stack([flat.t() @ padded[:, :, i:i + s, j:j + s].permute(0, 2, 3, 1).reshape(-1, cin)
                      for i in range(3) for j in range(3)], 1)
    dx = torch.nn.functional.conv_transpose2d(dz.permute(0, 3, 1, 2), w, padding=1)
    return {"dw": dw, "db": flat.sum(0), "dx": dx.permute(0, 2, 3, 1)}
