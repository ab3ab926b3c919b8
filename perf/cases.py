"""The work a program gives this library, as cases that can be timed and checked.

Each case goes through the Python entry points, on inputs made from a seed:

  velocity   one residual evaluation (explicit time integrators, error estimates)
  jacobian   residual and CSR Jacobian together (implicit solvers, LSPG, linear stability)
  ssprk3     explicit time steps of one problem (graph replay)
  batch      explicit time steps of many small problems (parameter studies, snapshots)
  implicit   Crank-Nicolson steps, Newton with BiCGSTAB
  lspg       steps of the hyper-reduced learned-manifold reduced-order model
  train      Adam steps of the reduced-order model's autoencoder

`exact` restates the same operations in 64-bit torch."""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The library's Python package (its folder's name is no identifier)."""
    if "pda_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "pda_gb300", os.path.join(_ROOT, "pressio-demoapps_gb300", "__init__.py"))
        module = importlib.util.module_from_spec(spec)
        sys.modules["pda_gb300"] = module
        spec.loader.exec_module(module)
    return sys.modules["pda_gb300"]


# problem: (family enum, member, IC flag, dimensions, dofs, bounds of one axis, periodic)
_PROBLEMS = {
    "sod1d": ("Euler1d", "Sod", 1, 1, 3, (-0.5, 0.5), False),
    "riemann2d": ("Euler2d", "Riemann", 2, 2, 4, (0.0, 1.0), False),
    "kh2d": ("Euler2d", "KelvinHelmholtz", 1, 2, 4, (-5.0, 5.0), True),
    "smooth3d": ("Euler3d", "PeriodicSmooth", 1, 3, 5, (-1.0, 1.0), True),
    "swe2d": ("Swe2d", "SlipWall", 1, 2, 3, (-5.0, 5.0), False),
}
_GAMMA = 1.4
_SWE = {"gravity": 9.8, "coriolis": -3.0, "pulseMagnitude": 0.125}
# reduced-order model: hidden widths and latent size of the shallow-water network
_HIDDEN, _LATENT, _ROM_DT = (256, 1024), 12, 0.025
_TRAIN_LR, _TRAIN_ROWS = 1e-3, 128


def listed():
    return [
        # the smallest call: a 1D shock tube's residual, bound by launch and latency
        {"name": "velocity_sod1d", "kind": "velocity", "problem": "sod1d", "scheme": 2, "nx": 1000, "ny": 1, "nz": 1},
        # the benchmark's residual: 2D Riemann problem at 1024^2
        {"name": "velocity_riemann2d", "kind": "velocity", "problem": "riemann2d", "scheme": 2,
         "nx": 1024, "ny": 1024, "nz": 1},
        # an ordinary mesh with odd sizes, periodic, third order
        {"name": "velocity_kh2d", "kind": "velocity", "problem": "kh2d", "scheme": 1, "nx": 401, "ny": 203, "nz": 1},
        # a large 3D residual
        {"name": "velocity_smooth3d", "kind": "velocity", "problem": "smooth3d", "scheme": 2,
         "nx": 160, "ny": 160, "nz": 160},
        # residual and Jacobian of a 2D mesh, transmissive boundaries
        {"name": "jacobian_riemann2d", "kind": "jacobian", "problem": "riemann2d", "scheme": 2,
         "nx": 512, "ny": 512, "nz": 1, "sample": 0.0},
        # residual and Jacobian of a 3D mesh with odd sizes, third order (the reference's 3D scheme)
        {"name": "jacobian_smooth3d", "kind": "jacobian", "problem": "smooth3d", "scheme": 1,
         "nx": 41, "ny": 37, "nz": 43, "sample": 0.0},
        # residual and Jacobian on a 1 % sample mesh, as a hyper-reduced solver calls them
        {"name": "jacobian_sample_swe2d", "kind": "jacobian", "problem": "swe2d", "scheme": 2,
         "nx": 256, "ny": 256, "nz": 1, "sample": 0.01},
        # explicit steps of a small problem
        {"name": "ssprk3_sod1d", "kind": "ssprk3", "problem": "sod1d", "scheme": 2, "nx": 1000, "ny": 1, "nz": 1,
         "steps": 50, "dt": 1e-4},
        # explicit steps of a parameter study: instances of uneven sizes
        {"name": "batch_swe2d", "kind": "batch", "scheme": 2, "instances": 24, "smallest": 64, "largest": 256,
         "steps": 2, "dt": 0.005},
        # Crank-Nicolson steps of the 2D Riemann problem
        {"name": "implicit_riemann2d", "kind": "implicit", "problem": "riemann2d", "scheme": 1,
         "nx": 64, "ny": 64, "nz": 1, "steps": 2, "dt": 0.01},
        # the online phase of the reduced-order model
        {"name": "lspg_swe2d", "kind": "lspg", "nx": 256, "ny": 256, "sample": 0.01, "steps": 20, "jacobian_bits": 32},
        # its offline phase: Adam steps of the autoencoder
        {"name": "train_autoencoder", "kind": "train", "outputs": 3 * 128 * 128, "steps": 6},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["velocity"] * 4 + ["jacobian"] * 3 + ["ssprk3", "batch", "implicit", "lspg", "train"])
    if kind == "batch":
        return {"kind": kind, "scheme": rng.choice([1, 2]), "instances": rng.randint(2, 24), "smallest": 32,
                "largest": log_int(48, 256), "steps": rng.randint(1, 3), "dt": 0.005}
    if kind == "lspg":
        return {"kind": kind, "nx": log_int(64, 256), "ny": log_int(64, 256), "sample": rng.uniform(0.005, 0.02),
                "steps": rng.randint(5, 20), "jacobian_bits": rng.choice([32, 64])}
    if kind == "train":
        return {"kind": kind, "outputs": 192 * log_int(16, 256), "steps": rng.randint(2, 6)}
    if kind == "implicit":
        n = log_int(16, 64)
        return {"kind": kind, "problem": "riemann2d", "scheme": rng.choice([0, 1]), "nx": n, "ny": log_int(16, 64),
                "nz": 1, "steps": rng.randint(1, 2), "dt": 0.01}
    problem = rng.choice(sorted(_PROBLEMS))
    dim = _PROBLEMS[problem][3]
    if kind == "ssprk3":
        most = {1: 4000, 2: 256, 3: 32}[dim]
    elif kind == "velocity":
        most = {1: 20000, 2: 1024, 3: 128}[dim]
    else:
        most = {1: 4000, 2: 400, 3: 40}[dim]
    size = [log_int(16, most) if a < dim else 1 for a in range(3)]
    case = {"kind": kind, "problem": problem, "scheme": rng.choice([0, 1, 2, 2]),
            "nx": size[0], "ny": size[1], "nz": size[2]}
    if kind == "ssprk3":
        case.update(steps=rng.randint(2, 30), dt=1e-4)
    if kind == "jacobian":
        # a sample mesh where the mesh is large enough for its stencils to be a part of it
        case["sample"] = rng.uniform(0.01, 0.05) if dim == 2 and min(size[:2]) >= 64 and rng.random() < 0.4 else 0.0
    return case


# ------------------------------------------------------------------- inputs
def _shape(case):
    return [case["nx"], case.get("ny", 1), case.get("nz", 1)][: _dim(case)]


def _dim(case):
    return _PROBLEMS[case["problem"]][3]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _noise(shape, seed, size=1e-3):
    return (2 * torch.rand(shape, generator=_generator(seed), device="cuda", dtype=torch.float64) - 1) * size


def _conserved(rho, velocities, p):
    """Euler state [dof, z, y, x] from density, velocities and pressure."""
    e = p / (_GAMMA - 1) + 0.5 * rho * sum(v * v for v in velocities)
    return torch.stack([rho] + [rho * v for v in velocities] + [e])


def _grid(shape, lo, hi):
    """Cell centres, one tensor per axis, broadcast to [z, y, x]."""
    dim, out = len(shape), []
    for a, n in enumerate(shape):
        x = lo + (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * (hi - lo) / n
        view = [1] * dim
        view[dim - 1 - a] = n
        out.append(x.view(view).expand(shape[::-1]))
    return out


def _state(problem, shape, seed):
    """A state of the problem, [dof, z, y, x]: the flow its runs start from and seeded noise."""
    lo, hi = _PROBLEMS[problem][5]
    g = _grid(shape, lo, hi)
    one = torch.ones_like(g[0])
    if problem == "sod1d":
        left = g[0] < 0.0
        u = _conserved(torch.where(left, one, 0.125 * one), [0 * one], torch.where(left, one, 0.1 * one))
        # the ends stay at rest: the gas there is the tube's undisturbed gas
        return u * (1 + _noise(u.shape, seed) * (g[0].abs() < 0.4))
    if problem == "riemann2d":
        right, top = g[0] >= 0.8, g[1] >= 0.8
        rho = torch.where(right & top, 1.5 * one, torch.where(right | top, 0.5323 * one, 0.138 * one))
        p = torch.where(right & top, 1.5 * one, torch.where(right | top, 0.3 * one, 0.029 * one))
        u = torch.where(right, 0.0 * one, 1.206 * one)
        v = torch.where(top, 0.0 * one, 1.206 * one)
        w = _conserved(rho, [u, v], p)
    elif problem == "kh2d":
        band = g[1].abs() < 2.0 + 0.1 * torch.sin(2 * math.pi * g[0] / 10.0)
        w = _conserved(torch.where(band, 2 * one, one), [torch.where(band, 0.5 * one, -0.5 * one), 0 * one], 2.5 * one)
    elif problem == "smooth3d":
        w = _conserved(1 + 0.2 * torch.sin(math.pi * (g[0] + g[1] + g[2])), [one, one, one], one)
    else:
        w = torch.stack([1 + 0.125 * torch.exp(-(g[0] - 1) ** 2 - (g[1] - 1) ** 2), 0 * one, 0 * one])
    return w + _noise(w.shape, seed)


def _flat(u):
    """[dof, z, y, x] to the library's cell-major vector."""
    return u.movedim(0, -1).reshape(-1).contiguous()


def _full_mesh(shape, problem, scheme):
    lo, hi = _PROBLEMS[problem][5]
    periodic = _PROBLEMS[problem][6]
    return _package().create_full_mesh(shape, [lo, hi] * len(shape), 2 * scheme + 3, [periodic] * len(shape))


def _make_problem(mesh, problem, scheme, params=None, stream=None):
    pda = _package()
    family, member, ic = _PROBLEMS[problem][:3]
    return pda.create_problem(mesh, getattr(getattr(pda, family), member), scheme, ic,
                              params or (_SWE if problem == "swe2d" else None), stream=stream)


def _sample_cells(shape, fraction):
    """The sample mesh's cells: a fixed choice for each mesh, as in a trained reduced-order model."""
    n = int(np.prod(shape))
    return np.sort(np.random.default_rng(7).choice(n, max(1, round(fraction * n)), replace=False))


def _batch_members(case, seed):
    rng = np.random.default_rng(512)  # the sizes of the study; its parameters come from the seed
    sizes = rng.integers(case["smallest"], case["largest"] + 1, case["instances"])
    rng = np.random.default_rng(seed)
    return [((int(n), int(n)), {"gravity": float(rng.uniform(5, 10)), "coriolis": float(rng.uniform(-4, -1)),
                                "pulseMagnitude": float(rng.uniform(0.05, 0.2))}) for n in sizes]


def _decoder(n, seed):
    """Weights of a decoder (weights hold bf16 values, as trained ones do) and a starting latent vector."""
    g = _generator(seed)

    def weight(rows, cols, size):
        w = torch.randn(rows, cols, generator=g, device="cuda") * size
        return w.to(torch.bfloat16).float()

    hb, ha = _HIDDEN
    w = (weight(hb, _LATENT, 0.3), torch.randn(hb, generator=g, device="cuda") * 0.1,
         weight(ha, hb, 0.05), torch.randn(ha, generator=g, device="cuda") * 0.1,
         weight(n, ha, 0.02), torch.randn(n, generator=g, device="cuda") * 0.1)
    return w, torch.randn(_LATENT, generator=g, device="cuda", dtype=torch.float64) * 0.3


def _reference_water(n):
    u = torch.zeros(n, device="cuda", dtype=torch.float64)
    u[0::3] = 1.0
    return u


def _training_inputs(case, seed):
    """Snapshot rows (smooth, low-dimensional, scaled to [-1, 1]) and initial weights and biases."""
    n, g = case["outputs"], _generator(seed)
    x = torch.arange(n, device="cuda", dtype=torch.float32) / n
    waves = torch.sin(2 * math.pi * torch.arange(1, 13, device="cuda")[:, None] * x[None, :])
    rows = torch.randn(_TRAIN_ROWS, 12, generator=g, device="cuda") @ waves / 4
    widths = (n, _HIDDEN[1], _HIDDEN[0], _LATENT, _HIDDEN[0], _HIDDEN[1], n)
    layers = []
    for i, o in zip(widths[:-1], widths[1:]):
        w = (2 * torch.rand(o, i, generator=g, device="cuda") - 1) / math.sqrt(i)
        layers.append((w, torch.randn(o, generator=g, device="cuda") * 0.1))
    return torch.tanh(rows).to(torch.bfloat16).contiguous(), layers


# ---------------------------------------------------------- prepare and run
def prepare(case, seed):
    pda = _package()
    kind = case["kind"]
    s = {"case": case}
    if kind == "train":
        s["data"], layers = _training_inputs(case, seed)
        s["net"] = pda.AutoEncoder(case["outputs"], _LATENT, _HIDDEN[1], _HIDDEN[0], seed=0)
        for l, (w, b) in enumerate(layers):
            # the library pads the latent dimension
            o, i = s["net"].layer_shape(l)
            wp, bp = torch.zeros(o, i, device="cuda"), torch.zeros(o, device="cuda")
            wp[: w.shape[0], : w.shape[1]] = w
            bp[: b.shape[0]] = b
            s["net"].set_layer(l, wp, bp)
        torch.cuda.synchronize()
        return s
    s["stream"] = None if kind in ("velocity", "jacobian", "implicit") else torch.cuda.Stream()
    if kind == "batch":
        members = _batch_members(case, seed)
        meshes = {m: _full_mesh(m, "swe2d", case["scheme"]) for m in {m for m, _ in members}}
        s["batch"] = pda.create_batch([_make_problem(meshes[m], "swe2d", case["scheme"], p, s["stream"])
                                       for m, p in members], stream=s["stream"])
        s["start"] = s["batch"].initialCondition()
        s["u"] = s["batch"].createState()
        torch.cuda.synchronize()
        return s
    if kind == "lspg":
        shape = (case["nx"], case["ny"])
        mesh = _full_mesh(shape, "swe2d", 2)
        cells = _sample_cells(shape, case["sample"])
        sample, stencil = pda.create_sample_mesh(mesh, cells)
        n = 3 * len(stencil)
        (w1, b1, w2, b2, w3, b3), s["start"] = _decoder(n, seed)
        s["x"] = torch.empty_like(s["start"])
        s["rom"] = pda.LspgRom.mlp(_make_problem(sample, "swe2d", 2, stream=s["stream"]),
                                   np.searchsorted(stencil, cells), _reference_water(n),
                                   torch.full((n,), 0.05, device="cuda", dtype=torch.float64),
                                   w1, b1, w2, b2, w3, b3, tensor_cores=True)
        s["rom"].set_jacobian_precision(case["jacobian_bits"])
        torch.cuda.synchronize()
        return s
    shape = _shape(case)
    u = _flat(_state(case["problem"], shape, seed))
    mesh = _full_mesh(shape, case["problem"], case["scheme"])
    if case.get("sample"):
        mesh, stencil = pda.create_sample_mesh(mesh, _sample_cells(shape, case["sample"]))
        nd = _PROBLEMS[case["problem"]][4]
        u = u.view(-1, nd)[torch.from_numpy(stencil).cuda()].reshape(-1).contiguous()
    p = s["problem"] = _make_problem(mesh, case["problem"], case["scheme"], stream=s["stream"])
    s["start"] = u
    if kind in ("ssprk3", "implicit"):
        s["u"] = torch.empty_like(u)
    else:
        s["v"] = p.createVelocity()
    if kind == "jacobian":
        s["j"] = p.createJacobian()
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "velocity":
        s["problem"].velocity(s["start"], 0.0, s["v"])
        return s["v"]
    if kind == "jacobian":
        s["problem"].rightHandSideAndJacobian(s["start"], 0.0, s["v"], s["j"])
        return [s["v"], s["j"].values, s["j"].rowptr, s["j"].colidx]
    if kind == "implicit":
        s["u"].copy_(s["start"])
        s["problem"].advance_implicit(s["u"], 0.0, case["dt"], case["steps"], scheme="cn")
        return s["u"]
    if kind == "ssprk3":
        with torch.cuda.stream(s["stream"]):
            s["u"].copy_(s["start"])
        s["problem"].advance_ssprk3(s["u"], 0.0, case["dt"], case["steps"])
        return s["u"]
    if kind == "batch":
        with torch.cuda.stream(s["stream"]):
            s["u"].copy_(s["start"])
        s["batch"].advance_ssprk3(s["u"], 0.0, case["dt"], case["steps"])
        return [s["batch"].instance(s["u"], i) for i in range(s["batch"].size)]
    if kind == "lspg":
        with torch.cuda.stream(s["stream"]):
            s["x"].copy_(s["start"])
        # the reduced-order model's setting: BDF2, one Gauss-Newton iteration a step
        s["rom"].advance(s["x"], _ROM_DT, case["steps"], 1, 1e-9, order=2)
        return s["rom"].decode(s["x"])
    losses = s["net"].train(s["data"], batch=_TRAIN_ROWS, epochs=case["steps"], lr=_TRAIN_LR, seed=3)
    out = [torch.from_numpy(losses)]
    for l in range(s["net"].LAYERS):
        out += list(s["net"].layer(l))
    return out


# ------------------------------------------------------------ work and floor
def work(case):
    """Bytes: every input read once and every output written once.  Operations: those of
    the scheme's formulas with each face evaluated once (a division or root as one)."""
    kind = case["kind"]
    if kind == "train":
        n, (hb, ha) = case["outputs"], _HIDDEN
        params = 2 * (n * ha + ha * hb + hb * _LATENT)
        # weights and both Adam moments read and written each step; forward and two backward products
        return {"bytes": case["steps"] * (24 * params + 2 * n * _TRAIN_ROWS),
                "flops": case["steps"] * 6 * params * _TRAIN_ROWS}
    side = {0: 0, 1: 22, 2: 75}
    if kind == "lspg":
        cells = max(1, round(case["sample"] * case["nx"] * case["ny"]))
        rows = 3 * 12 * cells  # decoder rows: the stencil cells, about 12 to a sample cell
        step = {"bytes": 2 * rows * _HIDDEN[1] + 8 * rows, "flops": 2 * rows * _HIDDEN[1] * (_LATENT + 1)
                + cells * 4 * (6 * 200 + 12 * 120)}
        return {k: case["steps"] * v for k, v in step.items()}
    if kind == "batch":
        cells = sum(m[0] * m[1] for m, _ in _batch_members(case, 0))
        evals, nd, dim = 3 * case["steps"], 3, 2
    else:
        dim, nd = _dim(case), _PROBLEMS[case["problem"]][4]
        cells = int(np.prod(_shape(case)))
        evals = {"velocity": 1, "jacobian": 1, "ssprk3": 3 * case.get("steps", 1),
                 "implicit": 3 * case.get("steps", 1)}[kind]
        if case.get("sample"):
            cells = max(1, round(case["sample"] * cells))
    flops = cells * dim * nd * (2 * side[case["scheme"]] + 20)
    bytes_ = cells * nd * 16
    if kind in ("jacobian", "implicit"):
        h = case["scheme"] + 1
        nnz = cells * nd * nd * (1 + 2 * dim * h)
        bytes_ += 8 * nnz
        flops += 6 * nnz
    return {"bytes": evals * bytes_, "flops": evals * flops}


# -------------------------------------------------------------------- exact
def _weno(q, scheme):
    """Left- and right-biased values of the face in the middle of the cells q[0..2h-1]."""
    if scheme == 0:
        return q[0], q[1]

    def third(a, b, c):
        w0, w1 = (1 / 3) / (1e-6 + (a - b) ** 2) ** 2, (2 / 3) / (1e-6 + (b - c) ** 2) ** 2
        return (w0 * (3 * b - a) + w1 * (b + c)) / (2 * (w0 + w1))

    def fifth(a, b, c, d, e):
        b0 = 13 / 12 * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4
        b1 = 13 / 12 * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4
        b2 = 13 / 12 * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4
        w0, w1, w2 = 0.1 / (1e-6 + b0) ** 2, 0.6 / (1e-6 + b1) ** 2, 0.3 / (1e-6 + b2) ** 2
        return (w0 * (2 * a - 7 * b + 11 * c) + w1 * (5 * c - b + 2 * d) + w2 * (2 * c + 5 * d - e)) / (6 * (w0 + w1 + w2))

    if scheme == 1:
        return third(*q[:3]), third(*q[:0:-1])
    return fifth(*q[:5]), fifth(*q[:0:-1])


def _flux(l, r, axis, swe, gravity):
    """Rusanov flux of the states l | r across a face normal to the axis."""
    def side(u):
        v = [c / u[0] for c in u[1:]] if swe else [c / u[0] for c in u[1:-1]]
        if swe:
            p, h = 0.5 * gravity * u[0] ** 2, None
        else:
            p = (_GAMMA - 1) * (u[-1] - 0.5 * u[0] * sum(c * c for c in v))
            h = (u[-1] + p) / u[0]
        f = [u[0] * v[axis]] + [u[0] * v[axis] * c + (p if a == axis else 0) for a, c in enumerate(v)]
        return v, h, torch.stack(f if swe else f + [u[0] * v[axis] * h])

    (vl, hl, fl), (vr, hr, fr) = side(l), side(r)
    if swe:
        sl, sr = torch.sqrt(l[0]), torch.sqrt(r[0])
        m = (vl[axis] * sl + vr[axis] * sr) / (sl + sr)
        speed = torch.where(m >= 0, m, -m) + torch.sqrt(gravity * 0.5 * (l[0] + r[0]))
    else:
        t = torch.sqrt(r[0] / l[0])
        v = [(a + t * b) / (1 + t) for a, b in zip(vl, vr)]
        k = sum(c * c for c in v)
        speed = torch.sqrt(k + 1e-300) + torch.sqrt((_GAMMA - 1) * ((hl + t * hr) / (1 + t) - 0.5 * k))
    return 0.5 * (fl + fr + speed * (l - r))


def _padded(u, axis, h, problem):
    """u with h ghost layers on both ends of the axis: wrapped, or mirrored (walls reflect the normal momentum)."""
    d, n = u.dim() - 1 - axis, u.shape[u.dim() - 1 - axis]
    at = torch.arange(-h, n + h, device=u.device)
    if _PROBLEMS[problem][6]:
        return u.index_select(d, at % n)
    out = torch.where(at < 0, -1 - at, torch.where(at >= n, 2 * n - 1 - at, at))
    e = u.index_select(d, out)
    if problem == "swe2d":
        sign = torch.ones([u.shape[0]] + [1] * (u.dim() - 1), device=u.device, dtype=u.dtype)
        sign[1 + axis] = -1
        view = [1] * u.dim()
        view[d] = n + 2 * h
        e = torch.where(((at < 0) | (at >= n)).view(view), e * sign, e)
    return e


def _face_cells(u, axis, scheme, problem):
    """The 2h cell states around every face normal to the axis."""
    h = scheme + 1
    e, d = _padded(u, axis, h, problem), u.dim() - 1 - axis
    faces = u.shape[d] + 1
    return [e.narrow(d, s, faces) for s in range(2 * h)]


def _face_flux(q, axis, scheme, problem, gravity):
    l, r = _weno(q, scheme)
    return _flux(l, r, axis, problem == "swe2d", gravity)


def _velocity(u, problem, scheme, params=_SWE):
    lo, hi = _PROBLEMS[problem][5]
    total = 0
    for axis in range(u.dim() - 1):
        d = u.dim() - 1 - axis
        f = _face_flux(_face_cells(u, axis, scheme, problem), axis, scheme, problem, params["gravity"])
        n = u.shape[d]
        total = total + (f.narrow(d, 0, n) - f.narrow(d, 1, n)) * (n / (hi - lo))
    if problem == "swe2d":
        c = params["coriolis"]
        total = total + torch.stack([0 * u[0], -c * u[2] / u[0], c * u[1] / u[0]])
    return total


def _jacobian(u, problem, scheme, cells, columns):
    """CSR values, row pointers and columns for the rows of the given cells; columns: cell to column block.
    Rows whose stencil leaves the mesh take the first-order flux, as the library documents."""
    nd, dim = u.shape[0], u.dim() - 1
    shape = list(u.shape[1:])[::-1]
    lo, hi = _PROBLEMS[problem][5]
    periodic, h = _PROBLEMS[problem][6], scheme + 1
    pos = [cells // int(np.prod(shape[:a])) % shape[a] for a in range(dim)]
    near = torch.zeros_like(cells, dtype=torch.bool)
    if not periodic:
        for a in range(dim):
            near |= (pos[a] < h) | (pos[a] >= shape[a] - h)
    rows, cols, vals = [], [], []
    block = torch.arange(len(cells), device=u.device)

    def put(which, k, j, column_cell, value):
        rows.append(block[which] * nd + k)
        cols.append(columns[column_cell] * nd + j)
        vals.append(value)

    for axis in range(dim):
        stride, n = int(np.prod(shape[:axis])), shape[axis]
        for order, which in ((scheme, (~near).nonzero()[:, 0]), (0, near.nonzero()[:, 0])):
            if not len(which):
                continue
            q = _face_cells(u, axis, order, problem)
            f = pos[axis][which]
            others = [pos[a][which] for a in range(dim)]
            for s in range(2 * order + 2):
                for j in range(nd):
                    t = [torch.zeros_like(x) for x in q]
                    t[s][j] = 1
                    _, df = torch.func.jvp(lambda *z: _face_flux(list(z), axis, order, problem, _SWE["gravity"]),
                                           tuple(q), tuple(t))
                    for face, sign in ((0, 1.0), (1, -1.0)):
                        at = [o + face if a == axis else o for a, o in enumerate(others)]
                        value = df[(slice(None),) + tuple(at[::-1])] * (sign * n / (hi - lo))
                        c = f + face - (order + 1) + s
                        ghost = (c < 0) | (c >= n)
                        c = c % n if periodic else torch.where(ghost, f, c)
                        if problem == "swe2d" and j == 1 + axis:
                            value = torch.where(ghost, -value, value)
                        for k in range(nd):
                            put(which, k, j, cells[which] + (c - f) * stride, value[k])
    if problem == "swe2d":
        w, c, every = u.reshape(nd, -1)[:, cells], _SWE["coriolis"], block
        for k, j, v in ((1, 0, c * w[2] / w[0] ** 2), (1, 2, -c / w[0]), (2, 0, -c * w[1] / w[0] ** 2), (2, 1, c / w[0])):
            put(every, k, j, cells, v)
    ncol = int(columns.max()) + 1
    m = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals),
                                (len(cells) * nd, ncol * nd)).coalesce()
    count = torch.bincount(m.indices()[0], minlength=len(cells) * nd)
    rowptr = torch.cat([torch.zeros(1, device=u.device, dtype=torch.int64), count.cumsum(0)])
    return m.values(), rowptr.int(), m.indices()[1].int()


def _ssprk3(u, f, dt, steps):
    for _ in range(steps):
        a = u + dt * f(u)
        a = 0.75 * u + 0.25 * (a + dt * f(a))
        u = u / 3 + 2 / 3 * (a + dt * f(a))
    return u


def _krylov(apply, b, tol=1e-13, most=300):
    """GMRES without restart."""
    beta = b.norm()
    basis, hess = [b / beta], torch.zeros(most + 1, most, dtype=b.dtype, device=b.device)
    for k in range(most):
        w = apply(basis[k])
        for _ in range(2):  # orthogonalised twice
            for i, v in enumerate(basis):
                c = torch.dot(v, w)
                hess[i, k] += c
                w = w - c * v
        hess[k + 1, k] = w.norm()
        basis.append(w / hess[k + 1, k])
        rhs = torch.zeros(k + 2, 1, dtype=b.dtype, device=b.device)
        rhs[0] = beta
        if k % 5 == 4 or k == most - 1:
            y = torch.linalg.lstsq(hess[: k + 2, : k + 1], rhs).solution
            if (hess[: k + 2, : k + 1] @ y - rhs).norm() <= tol * beta:
                break
    return (torch.stack(basis[: k + 1], 1) @ y)[:, 0]


def _crank_nicolson(u, f, dt, steps):
    shape = u.shape
    for _ in range(steps):
        start, y = u + dt / 2 * f(u), u
        for _ in range(12):
            r = (y - dt / 2 * f(y) - start).reshape(-1)
            d = _krylov(lambda z: z - dt / 2 * torch.func.jvp(f, (y,), (z.view(shape),))[1].reshape(-1), r)
            y = y - d.view(shape)
            if d.norm() < 1e-12 * y.norm():
                break
        u = y
    return u


def _lspg(case, seed):
    shape = (case["nx"], case["ny"])
    cells = torch.from_numpy(_sample_cells(shape, case["sample"])).cuda()
    # the sample mesh's cells: the samples and their stencils
    x, y = cells % shape[0], cells // shape[0]
    around = [cells]
    for k in (-3, -2, -1, 1, 2, 3):
        around += [cells[(x + k >= 0) & (x + k < shape[0])] + k]
        around += [cells[(y + k >= 0) & (y + k < shape[1])] + k * shape[0]]
    stencil = torch.unique(torch.cat(around))
    own = torch.searchsorted(stencil, cells)
    n = 3 * len(stencil)
    w, z = _decoder(n, seed)
    w1, b1, w2, b2, w3, b3 = (t.double() for t in w)
    base, elu = _reference_water(3 * shape[0] * shape[1]).view(-1, 3), torch.nn.functional.elu

    def decode(z):
        y = w3 @ elu(w2 @ elu(w1 @ z + b1) + b2) + b3
        return _reference_water(n) + 0.05 * y

    def parts(z):
        """The decoded state and the velocity on the sample cells."""
        state = decode(z).view(-1, 3)
        full = base.index_copy(0, stencil, state).view(shape[1], shape[0], 3).movedim(-1, 0)
        v = _velocity(full, "swe2d", 2).movedim(0, -1).reshape(-1, 3)
        return state[own].reshape(-1), v[cells].reshape(-1)

    old, older = parts(z)[0], None
    for step in range(case["steps"]):
        def residual(z):
            s, v = parts(z)
            if step == 0:
                return s - old - _ROM_DT * v
            return s - 4 / 3 * old + older / 3 - 2 / 3 * _ROM_DT * v

        r = residual(z)
        j = torch.stack([torch.func.jvp(residual, (z,), (e,))[1] for e in torch.eye(_LATENT, device="cuda").double()], 1)
        z = z - torch.linalg.solve(j.T @ j, j.T @ r)
        older, old = old, parts(z)[0]
    return decode(z)


def _train(case, seed):
    data, layers = _training_inputs(case, seed)
    data = data.double()
    params = [t.double().requires_grad_() for pair in layers for t in pair]
    m, v = [torch.zeros_like(t) for t in params], [torch.zeros_like(t) for t in params]
    losses = []
    for step in range(1, case["steps"] + 1):
        y = data
        for l in range(6):
            y = y @ params[2 * l].T + params[2 * l + 1]
            if l not in (2, 5):
                y = torch.nn.functional.elu(y)
        loss = ((y - data) ** 2).mean()
        losses.append(float(loss.detach()))
        grads = torch.autograd.grad(loss, params)
        with torch.no_grad():
            for t, g, a, b in zip(params, grads, m, v):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).addcmul_(g, g, value=0.001)
                t -= _TRAIN_LR * (a / (1 - 0.9 ** step)) / ((b / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return losses, [t.detach() for t in params]


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        losses, params = _train(case, seed)
        out = [torch.tensor(losses, dtype=torch.float64)]
        net = _package().AutoEncoder(case["outputs"], _LATENT, _HIDDEN[1], _HIDDEN[0], seed=0)
        for l in range(6):  # laid out as the library's layers: the latent dimension padded
            o, i = net.layer_shape(l)
            w = torch.zeros(o, i, device="cuda", dtype=torch.float64)
            b = torch.zeros(o, device="cuda", dtype=torch.float64)
            w[: params[2 * l].shape[0], : params[2 * l].shape[1]] = params[2 * l]
            b[: params[2 * l + 1].shape[0]] = params[2 * l + 1]
            out += [w, b]
        return out
    if kind == "lspg":
        return _lspg(case, seed)
    if kind == "batch":
        out = []
        for shape, p in _batch_members(case, seed):
            g = _grid(shape, -5.0, 5.0)
            u = torch.stack([1 + p["pulseMagnitude"] * torch.exp(-((g[0] - 1) ** 2 + (g[1] - 1) ** 2)), 0 * g[0], 0 * g[0]])
            out.append(_flat(_ssprk3(u, lambda w: _velocity(w, "swe2d", case["scheme"], p), case["dt"], case["steps"])))
        return out
    problem, scheme, shape = case["problem"], case["scheme"], _shape(case)
    u = _state(problem, shape, seed)
    f = lambda w: _velocity(w, problem, scheme)  # noqa: E731
    if kind == "ssprk3":
        return _flat(_ssprk3(u, f, case["dt"], case["steps"]))
    if kind == "implicit":
        return _flat(_crank_nicolson(u, f, case["dt"], case["steps"]))
    v = _flat(f(u))
    if kind == "velocity":
        return v
    n, nd = int(np.prod(shape)), u.shape[0]
    cells = torch.arange(n, device="cuda")
    columns = cells
    if case["sample"]:
        cells = torch.from_numpy(_sample_cells(shape, case["sample"])).cuda()
        h, around = scheme + 1, [cells]
        for a in range(_dim(case)):
            stride = int(np.prod(shape[:a]))
            at = cells // stride % shape[a]
            for k in list(range(-h, 0)) + list(range(1, h + 1)):
                c = at + k
                c = c % shape[a] if _PROBLEMS[problem][6] else c
                inside = (c >= 0) & (c < shape[a])
                around.append((cells + (c - at) * stride)[inside])
        columns = torch.searchsorted(torch.unique(torch.cat(around)), torch.arange(n, device="cuda"))
        v = v.view(-1, nd)[cells].reshape(-1)
    values, rowptr, colidx = _jacobian(u, problem, scheme, cells, columns)
    return [v, values, rowptr, colidx]
