"""The calls that users of this framework make, as cases that can be timed and checked.

Every case goes through the Python surface (``ktt_b200``) as a program on PyTorch tensors calls it:
potential maps on 3D grids (``CoulombContext.forward_3d``, and ``forward_3d_host`` on host arrays),
2D slices (``slice_atoms`` + ``forward_2d``), many molecules at once (``Batch``), the gradient of a
loss on a map (``adjoint_3d``) and a charge-fitting step (``coulomb_map`` and its backward), and the
N-body step (``nbody_step``).  ``form`` says how the call chooses its kernel:

* ``default``   no configuration given, the plain call
* ``fast``      FP32 sums with 2/8 of the reciprocal square roots on the FMA pipe
* ``accurate``  the shipped tuned configuration (``tuned("b200_map3d")``: FP64 merge of FP32 partials)
* ``exact``     every pair in FP64
* ``split``     (slices) the balanced atom-split configuration that INTEGRATION.md recommends
"""
import math
import random

import torch

import ktt_b200

_context = None


def _ctx():
    """One context for the whole program, as a user keeps it."""
    global _context
    if _context is None:
        _context = ktt_b200.CoulombContext(torch.cuda.current_device())
    return _context


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # One z slice of the KTT 2D example's kind at the benchmark's size (ktt_b200/run_slice2d.py),
        # atoms converted to the 2D convention on the device, then the recommended slice form.
        {"name": "slice 256x256x4000", "kind": "slice", "form": "split", "nx": 256, "ny": 256, "atoms": 4000, "h": 0.5},
        # A slice of odd size by the plain call: what a plotting or inspection program asks for.
        {"name": "slice plain 250x187", "kind": "slice", "form": "default", "nx": 250, "ny": 187, "atoms": 1501,
         "h": 0.5},
        # The smallest map: a ligand on its own grid, where launches and latency count.
        {"name": "map ligand", "kind": "map", "form": "default", "nx": 37, "ny": 41, "nz": 33, "atoms": 211, "h": 0.5},
        # An ordinary protein map by the plain call.
        {"name": "map plain 96", "kind": "map", "form": "default", "nx": 96, "ny": 96, "nz": 96, "atoms": 4096,
         "h": 0.5},
        # A map of odd sides, FP32 sums with the FMA-pipe share.
        {"name": "map fast odd", "kind": "map", "form": "fast", "nx": 131, "ny": 117, "nz": 125, "atoms": 5003,
         "h": 0.5},
        # The benchmark's map (bench.py): 256^3 points, 65,536 atoms, the shipped tuned form.
        {"name": "map accurate 256", "kind": "map", "form": "accurate", "nx": 256, "ny": 256, "nz": 256,
         "atoms": 65536, "h": 0.5},
        # A map every pair of which is evaluated in FP64 (reference values for another program).
        {"name": "map exact 96", "kind": "map", "form": "exact", "nx": 96, "ny": 96, "nz": 96, "atoms": 8192, "h": 0.5},
        # Host arrays in and out, the whole call with its copies (KTT's Tuner::Run semantics).
        {"name": "host 128", "kind": "host", "form": "accurate", "nx": 128, "ny": 128, "nz": 128, "atoms": 8192,
         "h": 0.5},
        # Uneven molecules, 200 to 20,000 atoms, grids with an 8 A margin, one persistent launch.
        {"name": "batch of 32", "kind": "batch", "form": "default", "molecules": 32, "lo": 200, "hi": 20000,
         "mix": 4, "h": 0.5},
        # Charge fitting (ktt_b200/run_adjoint.py): forward map, weighted least-squares loss, backward.
        {"name": "fit step 128", "kind": "fit", "form": "accurate", "nx": 128, "ny": 128, "nz": 128, "atoms": 8192,
         "h": 0.5},
        # The gradient alone for a small molecule on a grid of odd sides (inside somebody's own loop).
        {"name": "gradient small", "kind": "gradient", "form": "default", "nx": 61, "ny": 57, "nz": 50, "atoms": 777,
         "h": 0.5},
        # KTT's N-body example at its size, plain call.
        {"name": "nbody 131072", "kind": "nbody", "form": "default", "bodies": 131072},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["slice", "slice", "map", "map", "map", "map", "host", "batch", "fit", "gradient", "nbody"])
    h = rng.choice([0.25, 0.5, 0.5, 1.0])
    if kind == "slice":
        return {"kind": kind, "form": rng.choice(["default", "split"]), "nx": _log(rng, 64, 1024),
                "ny": _log(rng, 64, 1024), "atoms": _log(rng, 200, 20000), "h": h}
    if kind == "nbody":
        return {"kind": kind, "form": "default", "bodies": _log(rng, 1000, 131072)}
    if kind == "batch":
        return {"kind": kind, "form": "default", "molecules": rng.randint(2, 48), "lo": 200,
                "hi": _log(rng, 1000, 20000), "mix": rng.randint(0, 1 << 30), "h": 0.5}
    top = {"map": 224, "host": 160, "fit": 128, "gradient": 128}[kind]
    side = [_log(rng, 24, top) for _ in range(3)]
    most = {"map": 40000, "host": 20000, "fit": 10000, "gradient": 10000}[kind]
    atoms = _log(rng, 200, most)
    if kind == "map":
        form = rng.choice(["default", "default", "fast", "accurate", "accurate", "exact"])
        if form == "exact":
            atoms = min(atoms, 16384)
    else:
        form = "default" if kind == "gradient" else "accurate"
    return {"kind": kind, "form": form, "nx": side[0], "ny": side[1], "nz": side[2], "atoms": atoms, "h": h}


# ---- configurations, inputs -------------------------------------------------------------------

def _tune(case):
    form = case["form"]
    if form == "accurate":
        return ktt_b200.tuned("b200_map3d")
    if form == "fast":
        return ktt_b200.Tune(block_x=64, block_y=1, z_iterations=8, x_points=2, unroll=2, rsqrt_soft=2)
    if form == "exact":
        return ktt_b200.Tune(block_x=64, block_y=1, z_iterations=8, x_points=4, unroll=1,
                             precision=ktt_b200.PREC_FP64_PAIRS)
    if form == "split":
        return ktt_b200.Tune(block_x=32, block_y=1, z_iterations=4, x_points=4, unroll=2, rsqrt_soft=2, atom_split=32,
                             split_form=2)
    return None


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _atoms(gen, n, box):
    """n atoms uniform in the box (three sides, A), charges uniform in [-1, 1]."""
    a = torch.rand((n, 4), generator=gen, device="cuda", dtype=torch.float32)
    return torch.cat([a[:, :3] * torch.tensor(box, device="cuda", dtype=torch.float32), a[:, 3:] * 2.0 - 1.0],
                     dim=1).contiguous()


def _box(case):
    return [case["h"] * case[k] for k in ("nx", "ny", "nz")]


def _molecules(case):
    """Atom count and grid side of each molecule: counts log-uniform, a cube of side
    (n / 0.1)^(1/3) A with an 8 A margin all round."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["molecules"]):
        n = _log(rng, case["lo"], case["hi"])
        side = (n / 0.1) ** (1.0 / 3.0)
        out.append((n, side, int((side + 16.0) / case["h"]) + 1))
    return out


def _fit_inputs(case, gen):
    """Atoms, the target map's charges, and the loss weights (0 within 1.5 A of an atom, else 1)."""
    nx, ny, nz = _dims(case)
    atoms = _atoms(gen, case["atoms"], _box(case))
    target = atoms.clone()
    target[:, 3] += 0.1 * torch.randn(case["atoms"], generator=gen, device="cuda")
    reach = int(math.ceil(1.5 / case["h"]))
    o = torch.arange(-reach, reach + 1, device="cuda")
    off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), dim=-1).reshape(-1, 3)
    cell = torch.floor(atoms[:, :3] / case["h"]).to(torch.int64)
    at = cell[:, None, :] + off[None]
    near = ((at * case["h"] - atoms[:, None, :3]) ** 2).sum(-1) < 1.5 ** 2
    size = torch.tensor([nx, ny, nz], device="cuda")
    near &= ((at >= 0) & (at < size)).all(-1)
    at = at[near]
    weight = torch.ones((nz, ny, nx), device="cuda")
    weight[at[:, 2], at[:, 1], at[:, 0]] = 0.0
    return atoms, target, weight


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    s = {"case": case, "ctx": _ctx(), "tune": _tune(case)}
    if kind == "nbody":
        s["pos"] = torch.rand((case["bodies"], 4), generator=gen, device="cuda") * 20.0
        s["vel"] = torch.rand((case["bodies"], 4), generator=gen, device="cuda") * 20.0
        s["vel"][:, 3] = 0.0
    elif kind == "batch":
        mols = []
        for n, side, points in _molecules(case):
            mols.append((_atoms(gen, n, [side] * 3), (points,) * 3, case["h"], (-8.0, -8.0, -8.0)))
        s["batch"] = ktt_b200.Batch(s["ctx"], mols)
    elif kind == "slice":
        s["atoms"] = _atoms(gen, case["atoms"], [case["h"] * case["nx"], case["h"] * case["ny"], 32.0])
    elif kind == "host":
        s["atoms"] = _atoms(gen, case["atoms"], _box(case)).cpu().numpy()
    elif kind == "fit":
        atoms, target, s["weight"] = _fit_inputs(case, gen)
        s["target"] = s["ctx"].forward_3d(target, _dims(case), case["h"], tune=s["tune"])
        s["atoms"] = atoms.requires_grad_(True)
    else:
        s["atoms"] = _atoms(gen, case["atoms"], _box(case))
        if kind == "gradient":
            nx, ny, nz = _dims(case)
            s["grad_map"] = torch.randn((nz, ny, nx), generator=gen, device="cuda")
    return s


def run(s):
    case, ctx, tune = s["case"], s["ctx"], s["tune"]
    kind = case["kind"]
    if kind == "slice":
        sliced = ctx.slice_atoms(s["atoms"], 16.0)
        return ctx.forward_2d(sliced, case["h"], case["nx"], case["ny"], tune=tune)
    if kind == "map":
        return ctx.forward_3d(s["atoms"], _dims(case), case["h"], tune=tune)
    if kind == "host":
        return ctx.forward_3d_host(s["atoms"], _dims(case), case["h"], tune=tune)
    if kind == "batch":
        s["batch"].run()
        return s["batch"].outputs
    if kind == "gradient":
        return ktt_b200.adjoint_3d(ctx, s["atoms"], _dims(case), case["h"], s["grad_map"])
    if kind == "fit":
        v = ktt_b200.coulomb_map(s["atoms"], ctx, _dims(case), case["h"], None, tune)
        loss = 0.5 * (s["weight"] * (v - s["target"]) ** 2).sum()
        (grad,) = torch.autograd.grad(loss, s["atoms"])
        return {"map": v.detach(), "loss": loss.detach(), "grad": grad}
    return ktt_b200.nbody_step(ctx, s["pos"], s["vel"], 0.001, 0.5, 0.01)


# ---- what a pass cannot do without ----------------------------------------------------------

def work(case):
    """Forward: 5 operations a pair (r^2 and the sum as FMAs, one reciprocal square root; the
    per-axis differences are shared).  Gradient: 13 a pair (r^2, the square root, its square and cube,
    three FMA sums).  N-body: 20 an interaction."""
    kind = case["kind"]
    if kind == "nbody":
        n = case["bodies"]
        return {"bytes": 64.0 * n, "flops": 20.0 * n * n}
    if kind == "batch":
        mols = _molecules(case)
        return {"bytes": float(sum(16 * n + 4 * p ** 3 for n, _, p in mols)),
                "flops": 5.0 * sum(n * p ** 3 for n, _, p in mols)}
    points = case["nx"] * case["ny"] * case.get("nz", 1)
    n = case["atoms"]
    pairs = float(points) * n
    if kind == "gradient":
        return {"bytes": 4.0 * points + 32.0 * n, "flops": 13.0 * pairs}
    if kind == "fit":
        return {"bytes": 16.0 * points + 32.0 * n, "flops": 18.0 * pairs}
    return {"bytes": 4.0 * points + 16.0 * n, "flops": 5.0 * pairs}


# ---- the same in 64 bits -----------------------------------------------------------------------

def _axis(count, h, origin=0.0):
    """The grid's own coordinates along one axis: FP32 values, widened."""
    x = torch.arange(count, device="cuda", dtype=torch.float64) * h + origin
    return x.to(torch.float32).to(torch.float64)


def _exact_map(atoms, dims, h, origin=0.0):
    a = atoms.detach().to(torch.float64)
    gx, gy, gz = (_axis(d, h, origin) for d in dims)
    out = torch.zeros((dims[2], dims[1] * dims[0]), device="cuda", dtype=torch.float64)
    step = max(1, min(a.shape[0], (1 << 27) // (dims[0] * dims[1])))
    for j in range(0, a.shape[0], step):
        b = a[j:j + step]
        dxy = (((gy[:, None, None] - b[:, 1]) ** 2) + ((gx[None, :, None] - b[:, 0]) ** 2)).reshape(-1, b.shape[0])
        r = torch.empty_like(dxy)
        for k in range(dims[2]):
            torch.add(dxy, (gz[k] - b[:, 2]) ** 2, out=r)
            out[k] += r.rsqrt_() @ b[:, 3]
    return out.reshape(dims[2], dims[1], dims[0])


def _exact_gradient(atoms, dims, h, grad_map):
    a = atoms.detach().to(torch.float64)
    g = grad_map.to(torch.float64).reshape(dims[2], -1)
    gx, gy, gz = (_axis(d, h) for d in dims)
    out = torch.zeros((a.shape[0], 4), device="cuda", dtype=torch.float64)
    x, y = gx.repeat(dims[1]), gy.repeat_interleave(dims[0])
    step = max(1, min(a.shape[0], (1 << 27) // (dims[0] * dims[1])))
    for j in range(0, a.shape[0], step):
        b = a[j:j + step]
        dxy = (x - b[:, :1]) ** 2 + (y - b[:, 1:2]) ** 2
        r = torch.empty_like(dxy)
        for k in range(dims[2]):
            dz = gz[k] - b[:, 2]
            torch.add(dxy, (dz ** 2)[:, None], out=r)
            r.rsqrt_()
            out[j:j + step, 3] += r @ g[k]
            r.pow_(3)
            s, sx, sy = r @ g[k], r @ (g[k] * x), r @ (g[k] * y)
            out[j:j + step, 0] += sx - b[:, 0] * s
            out[j:j + step, 1] += sy - b[:, 1] * s
            out[j:j + step, 2] += dz * s
    out[:, :3] *= a[:, 3:]
    return out


def exact(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "nbody":
        pos = (torch.rand((case["bodies"], 4), generator=gen, device="cuda") * 20.0).to(torch.float64)
        vel = (torch.rand((case["bodies"], 4), generator=gen, device="cuda") * 20.0).to(torch.float64)
        acc = torch.zeros((case["bodies"], 3), device="cuda", dtype=torch.float64)
        for i in range(0, case["bodies"], 512):
            d = [pos[None, :, c] - pos[i:i + 512, None, c] for c in range(3)]
            f = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + 0.01) ** -1.5 * pos[None, :, 3]
            for c in range(3):
                acc[i:i + 512, c] = (f * d[c]).sum(1)
        dt, damping = 0.001, 0.5
        new_pos = torch.cat([pos[:, :3] + dt * vel[:, :3] + damping * dt * dt * acc, pos[:, 3:]], dim=1)
        return new_pos, torch.cat([vel[:, :3] + dt * acc, torch.zeros_like(vel[:, 3:])], dim=1)
    if kind == "batch":
        return [_exact_map(_atoms(gen, n, [side] * 3), (points,) * 3, case["h"], -8.0)
                for n, side, points in _molecules(case)]
    if kind == "slice":
        a = _atoms(gen, case["atoms"], [case["h"] * case["nx"], case["h"] * case["ny"], 32.0])
        a[:, 2] -= 16.0
        return _exact_map(a, (case["nx"], case["ny"], 1), case["h"]).reshape(case["ny"], case["nx"])
    if kind == "host":
        a = _atoms(gen, case["atoms"], _box(case))
        return _exact_map(a, _dims(case), case["h"]).cpu().numpy()
    if kind == "fit":
        atoms, target, weight = _fit_inputs(case, gen)
        v = _exact_map(atoms, _dims(case), case["h"])
        diff = weight.to(torch.float64) * (v - _exact_map(target, _dims(case), case["h"]))
        return {"map": v, "loss": 0.5 * (diff ** 2).sum(),
                "grad": _exact_gradient(atoms, _dims(case), case["h"], diff)}
    atoms = _atoms(gen, case["atoms"], _box(case))
    if kind == "gradient":
        nx, ny, nz = _dims(case)
        return _exact_gradient(atoms, _dims(case), case["h"],
                               torch.randn((nz, ny, nx), generator=gen, device="cuda"))
    return _exact_map(atoms, _dims(case), case["h"])
