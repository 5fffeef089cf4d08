"""Timed cases of the public entry points: Vext fields (forward, forward +
adjoint, batches of frameworks), poses and String paths, and the drop-in CSR
kernel.

A case is a dict of plain values.  ``prepare`` makes what a user's program
holds before the call (frameworks, system or batch handles, device buffers),
``run`` is one call through the public API, ``exact`` the same result from a
plain 64-bit sum over every image, ``work`` the bytes and operations a pass
cannot do without: the inputs and outputs once, and 16 operations per
in-cutoff (site, image) pair forward, 28 forward + adjoint, with the pair
count taken from the framework's atom density.

Frameworks are seeded draws of the shapes and sizes of the benchmark's five
workloads (``string_vext_b200.synth``): a layered cell with a short c axis
(37 x 37 x 3.6 A, 600 atoms), a strongly skewed dense cell (28 x 31 x 24 A,
3000 atoms), a small cell of per-atom parameters (15 x 15 x 10 A, 64 atoms),
and uneven frameworks of 100-4000 atoms in 10-45 A cells.  The seed draws atom
positions and types; the case fixes the cell and the counts.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from string_vext_b200 import _lib, synth
from string_vext_b200.autograd import pose_energy
from string_vext_b200.cell import valid_cell
from string_vext_b200.orientation import normalized_directors, regular_pose_grid
from string_vext_b200.string_path import run_string
from string_vext_b200.system import VextBatch, VextPoseBatch, VextSystem
from string_vext_b200.vext import calculate_vext

GUESTS = {"A": synth.GUEST_A, "B": synth.GUEST_B}

#: cell lengths, angles, atoms, cutoff of the three named frameworks
CELLS = {"layered": ([37.0, 37.0, 3.6], [90.0, 90.0, 119.993], 600, 12.8),
         "skewed": ([28.0, 31.0, 24.0], [75.0, 85.0, 110.0], 3000, 12.8),
         "small": ([15.0, 15.0, 10.0], [90.0, 90.0, 120.0], 64, 12.0)}


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest whole call: one small framework, all pairs in FP64
        # (the CLI's --fp64), system set-up and output copies included
        {"name": "calculate_small_fp64", "kind": "calculate", "frame": "small", "guest": "A",
         "size": 20, "dirs": 64, "fp64": True},
        # the reference's default call on the full-size layered framework:
        # a new system, its lists, the field and every channel back on the host
        {"name": "calculate_layered", "kind": "calculate", "frame": "layered", "guest": "B",
         "size": 60, "dirs": 64, "fp64": False},
        # forward field into device tensors of a kept system, odd grid and
        # director count (partial blocks on every axis)
        {"name": "field_skewed_ragged", "kind": "field", "frame": "skewed", "guest": "A",
         "size": 47, "dirs": 50, "fp64": False},
        # the headline: forward + adjoint of every pose of the 60^3 x 64 field
        {"name": "adjoint_layered", "kind": "adjoint", "frame": "layered", "guest": "B",
         "size": 60, "dirs": 64},
        # forward + adjoint into page-locked host arrays, medium framework,
        # more directors than one work item holds
        {"name": "adjoint_host", "kind": "adjoint_host", "frame": "mix", "mix": 11, "guest": "A",
         "size": 24, "dirs": 96},
        # uneven frameworks x both guests in one launch, forward, full grids
        {"name": "batch_forward", "kind": "batch", "mix": 4, "frameworks": 4, "size": 60,
         "dirs": 64, "adjoint": False},
        # the same forward + adjoint, odd grids
        {"name": "batch_adjoint", "kind": "batch", "mix": 7, "frameworks": 4, "size": 35,
         "dirs": 64, "adjoint": True},
        # random poses through torch autograd, forward and backward
        {"name": "poses_random", "kind": "poses", "frame": "layered", "guest": "B",
         "poses": 1 << 20},
        # one String path's images: the smallest call, latency and launches
        {"name": "poses_path", "kind": "poses", "frame": "small", "guest": "A", "poses": 64},
        # String paths of many systems in one launch
        {"name": "path_batch", "kind": "paths", "mix": 5, "frameworks": 12, "paths": 100},
        # 200 String iterations with reparametrisation on one path
        {"name": "string_run", "kind": "string", "frame": "small", "guest": "A", "images": 64,
         "iterations": 200},
        # the reference driver's own kernel call: 512 centers with their CSR
        {"name": "dropin_csr", "kind": "dropin", "frame": "layered", "guest": "B",
         "centers": 512, "dirs": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calculate", "field", "field", "adjoint", "adjoint", "adjoint_host",
                       "batch", "batch", "poses", "poses", "paths", "string", "dropin"])
    case = {"kind": kind}
    if kind not in ("batch", "paths"):
        case["frame"] = rng.choice(["layered", "skewed", "small", "mix"])
        if case["frame"] == "mix":
            case["mix"] = rng.randrange(1 << 20)
        case["guest"] = rng.choice("AB")
    if kind == "calculate":
        fp64 = rng.random() < 0.3
        case.update(size=rng.randint(8, 24 if fp64 else 60), dirs=rng.randint(16, 96), fp64=fp64)
    elif kind == "field":
        case.update(size=rng.randint(16, 60), dirs=rng.randint(16, 96),
                    fp64=rng.random() < 0.15)
        if case["fp64"]:
            case["size"] = min(case["size"], 40)
    elif kind == "adjoint":
        case.update(size=rng.randint(16, 60), dirs=rng.randint(16, 96))
    elif kind == "adjoint_host":
        case.update(size=rng.randint(8, 40), dirs=rng.randint(16, 130))
    elif kind == "batch":
        adjoint = rng.random() < 0.5
        case.update(mix=rng.randrange(1 << 20), frameworks=rng.randint(1, 4),
                    size=rng.randint(16, 35 if adjoint else 45), dirs=rng.randint(32, 64),
                    adjoint=adjoint)
    elif kind == "poses":
        case.update(poses=_log_int(rng, 16, 1 << 20))
    elif kind == "paths":
        case.update(mix=rng.randrange(1 << 20), frameworks=rng.randint(1, 12),
                    paths=_log_int(rng, 4, 100))
    elif kind == "string":
        case.update(images=rng.randint(24, 128), iterations=rng.randint(50, 250))
    else:
        case.update(centers=_log_int(rng, 16, 512), dirs=rng.randint(16, 96))
    return case


# ------------------------------------------------------------------ inputs

def _mix_shapes(mix, count):
    """`count` (lengths, angles, atoms) of the uneven framework distribution."""
    rng = np.random.default_rng(mix)
    shapes = []
    for _ in range(count):
        n = int(round(math.exp(rng.uniform(math.log(100.0), math.log(4000.0)))))
        lengths = rng.uniform(10.0, 45.0, 3)
        angles = rng.uniform(60.0, 120.0, 3)
        while not valid_cell(lengths, angles):
            angles = rng.uniform(60.0, 120.0, 3)
        shapes.append((lengths.tolist(), angles.tolist(), n, 12.8))
    return shapes


def _shape(case):
    return _mix_shapes(case["mix"], 1)[0] if case["frame"] == "mix" else CELLS[case["frame"]]


def _framework(frame, shape, rng):
    lengths, angles, n, cutoff = shape
    if frame == "layered":
        z = 0.5 * rng.integers(0, 2, n) + rng.normal(0.0, 0.02, n)
        frac = np.column_stack([rng.random((n, 2)), z])
    else:
        frac = rng.random((n, 3))
    if frame == "small":
        eps, sig = rng.uniform(20.0, 60.0, n), rng.uniform(2.5, 3.8, n)
    else:
        kind = rng.integers(0, 4, n)
        eps, sig = synth.TYPE_TABLE[kind, 0], synth.TYPE_TABLE[kind, 1]
    return lambda guest: synth.make_case(lengths, angles, frac, sig, eps, GUESTS[guest], cutoff)


def _case_of(case, seed):
    rng = np.random.default_rng([seed, 1])
    return _framework(case["frame"], _shape(case), rng)(case["guest"]), rng


def _cases_of(case, seed):
    rng = np.random.default_rng([seed, 2])
    made = [_framework("mix", s, rng) for s in _mix_shapes(case["mix"], case["frameworks"])]
    return [m(g) for m in made for g in "AB"], rng


def _axes(dirs):
    return normalized_directors(regular_pose_grid(2, dirs)[1])


def _cuda(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _path(rng, frame_case, images):
    """A straight path along c at a random (a, b), random orientations."""
    path = np.empty((images, 6))
    path[:, :2] = rng.random(2)
    path[:, 2] = np.linspace(0.0, 1.0, images)
    path[:, 3:] = rng.uniform(0.0, 2 * np.pi, (images, 3))
    return path


def _images(frame_case, radius):
    """Every image (Cartesian) within `radius` of the cell [0, 1]^3, with its
    atom: the reference driver's image list."""
    cell = np.asarray(frame_case["cell"], dtype=float)
    inv = np.linalg.inv(cell)
    reach = radius * np.linalg.norm(inv, axis=0)
    lo, hi = np.floor(-reach).astype(int), np.ceil(reach).astype(int)
    frac = np.mod(np.asarray(frame_case["frame_frac"], dtype=float), 1)
    out, atom = [], []
    for i in range(lo[0], hi[0] + 1):
        for j in range(lo[1], hi[1] + 1):
            for k in range(lo[2], hi[2] + 1):
                f = frac + (i, j, k)
                keep = np.flatnonzero(((f > -reach) & (f < 1 + reach)).all(1))
                out.append(f[keep] @ cell)
                atom.append(keep)
    return np.concatenate(out), np.concatenate(atom)


def _coefficients(frame_case):
    """c12, c6, shift, floor^2 per framework atom (Lorentz-Berthelot mixing)."""
    sig = (np.asarray(frame_case["frame_sigma"]) + float(frame_case["guest_sigma"][0])) / 2
    eps = np.sqrt(np.asarray(frame_case["frame_epsilon"]) * float(frame_case["guest_epsilon"][0]))
    s6 = sig ** 6
    cut6 = (sig / frame_case["cutoff"]) ** 6
    return (4 * eps * s6 * s6, 4 * eps * s6, -4 * eps * (cut6 * cut6 - cut6), (0.1 * sig) ** 2)


def _offsets(frame_case):
    xyz, mass = np.asarray(frame_case["guest_xyz"]), np.asarray(frame_case["guest_mass"])
    return xyz[:, 0] - (xyz[:, 0] * mass).sum() / mass.sum()


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind in ("batch", "paths"):
        cases, rng = _cases_of(case, seed)
        systems = [VextSystem(c) for c in cases]
        if kind == "batch":
            shape = (case["dirs"],) + (case["size"],) * 3
            energy = [torch.empty(shape, device="cuda") for _ in systems]
            grad = [torch.empty(shape + (6,), device="cuda") for _ in systems] \
                if case["adjoint"] else None
            state["batch"] = VextBatch(systems, case["size"], _axes(case["dirs"]), energy,
                                       gradients=grad)
        else:
            counts, centers, quats = _path_poses(case, cases, rng)
            n = len(centers)
            state["batch"] = VextPoseBatch(systems, counts)
            state["in"] = (_cuda(centers), _cuda(quats))
            state["out"] = tuple(torch.empty((n,) + s, dtype=torch.float64, device="cuda")
                                 for s in ((), (3,), (4,), (3,)))
        return state
    frame_case, rng = _case_of(case, seed)
    state["frame"] = frame_case
    if kind == "calculate":
        return state
    if kind == "dropin":
        return {**state, **_csr(case, frame_case, rng)}
    state["system"] = VextSystem(frame_case)
    if kind in ("field", "adjoint", "adjoint_host"):
        state["axes"] = _axes(case["dirs"])
        shape = (case["dirs"],) + (case["size"],) * 3
        if kind == "field":
            state["out"] = (torch.empty(shape, device="cuda"),
                            torch.empty(shape[1:], device="cuda"),
                            torch.empty((2,) + shape[1:], device="cuda"),
                            torch.empty(shape[1:], device="cuda"))
        elif kind == "adjoint":
            state["out"] = (torch.empty(shape, device="cuda"),
                            torch.empty(shape + (6,), device="cuda"))
    elif kind == "poses":
        state["in"] = (_cuda(rng.random((case["poses"], 3)) @ frame_case["cell"]),
                       _cuda(synth.random_quaternions(rng, case["poses"])))
    else:
        state["path"] = _path(rng, frame_case, case["images"])
    return state


def _path_poses(case, cases, rng):
    """Random straight paths of 32-96 images, path p on system p % systems,
    the poses stacked system by system."""
    per = [[] for _ in cases]
    lengths = np.random.default_rng(case["mix"]).integers(32, 97, case["paths"])
    for p, n in enumerate(lengths):
        ends = rng.random((2, 3))
        t = np.linspace(0.0, 1.0, n)[:, None]
        per[p % len(cases)].append((ends[0] + t * (ends[1] - ends[0]),
                                    synth.random_quaternions(rng, n)))
    counts = [sum(len(f) for f, _ in rows) for rows in per]
    centers = [f @ c["cell"] for c, rows in zip(cases, per) for f, _ in rows]
    quats = [q for rows in per for _, q in rows]
    return counts, np.concatenate(centers), np.concatenate(quats)


def _csr(case, frame_case, rng):
    """One batch of the reference driver: consecutive grid centers with the
    image indices within cutoff + max|offset| of each."""
    offsets = np.ascontiguousarray(_offsets(frame_case))
    radius = frame_case["cutoff"] + np.abs(offsets).max()
    images, atom = _images(frame_case, radius)
    coeff = [np.ascontiguousarray(c[atom]) for c in _coefficients(frame_case)]
    grid = (np.arange(60) + .5) / 60
    first = int(rng.integers(0, 60 ** 3 - case["centers"]))
    at = np.arange(first, first + case["centers"])
    frac = np.column_stack([grid[at // 3600], grid[at // 60 % 60], grid[at % 60]])
    centers = np.ascontiguousarray(frac @ frame_case["cell"])
    near = [np.flatnonzero(((images - c) ** 2).sum(1) <= radius * radius) for c in centers]
    starts = np.concatenate([[0], np.cumsum([len(n) for n in near])]).astype(np.int64)
    axes = _axes(case["dirs"])
    output = np.empty((len(centers), len(axes)))
    return {"csr": (centers, axes, np.ascontiguousarray(images), offsets, *coeff, starts,
                    np.concatenate(near).astype(np.int32), output),
            "lib": _lib.load()}


# ------------------------------------------------------------------ one pass

def run(state):
    kind, case = state["kind"], state["case"]
    mode = _lib.VEXT_MODE_FP64 if case.get("fp64") else _lib.VEXT_MODE_MIXED
    if kind == "calculate":
        return calculate_vext(state["frame"], case["size"], case["dirs"], mode=mode)
    if kind == "field":
        orientation, marginal, site, grid = state["out"]
        state["system"].field_device(case["size"], state["axes"], orientation, mode=mode,
                                     out_marginal=marginal, out_site=site, out_grid=grid,
                                     stream=torch.cuda.current_stream())
        return state["out"]
    if kind == "adjoint":
        state["system"].field_adjoint_device(case["size"], state["axes"], *state["out"],
                                             stream=torch.cuda.current_stream())
        return state["out"]
    if kind == "adjoint_host":
        return state["system"].field_adjoint(case["size"], state["axes"], pinned=True)
    if kind == "batch":
        batch = state["batch"]
        batch.run(torch.cuda.current_stream())
        return batch.outputs + (batch.gradients or [])
    if kind == "poses":
        centers, quats = (t.detach().requires_grad_() for t in state["in"])
        energy = pose_energy(state["system"], centers, quats)
        gc, gq = torch.autograd.grad(energy.sum(), (centers, quats))
        return energy.detach(), gc, gq
    if kind == "paths":
        state["batch"].run(*state["in"], *state["out"], stream=torch.cuda.current_stream())
        return state["out"]
    if kind == "string":
        path, energy, result = run_string(state["system"], state["path"], direction=3,
                                          max_iterations=case["iterations"])
        return path, energy, result["iterations"]
    arrays = state["csr"]
    cutoff = state["frame"]["cutoff"]
    _lib.check(state["lib"].evaluate_reused_neighbors(
        len(arrays[0]), len(arrays[1]), len(arrays[2]), ctypes.c_double(cutoff * cutoff),
        *(_lib.ptr(a) for a in arrays)))
    return arrays[-1]


# ------------------------------------------------------------------ work

def _pairs(shape, poses):
    lengths, angles, n, cutoff = shape
    ca, cb, cg = (math.cos(math.radians(a)) for a in angles)
    volume = math.prod(lengths) * math.sqrt(1 - ca * ca - cb * cb - cg * cg + 2 * ca * cb * cg)
    return 2 * poses * n / volume * 4 / 3 * math.pi * cutoff ** 3


def work(case):
    kind = case["kind"]
    if kind in ("batch", "paths"):
        shapes = [s for s in _mix_shapes(case["mix"], case["frameworks"]) for _ in "AB"]
        atoms = sum(s[2] for s in shapes)
        if kind == "batch":
            poses = case["size"] ** 3 * case["dirs"]
            flops = sum(_pairs(s, poses) for s in shapes) * (28 if case["adjoint"] else 16)
            return {"bytes": 40 * atoms + len(shapes) * poses * (28 if case["adjoint"] else 4),
                    "flops": flops}
        lengths = np.random.default_rng(case["mix"]).integers(32, 97, case["paths"])
        flops = sum(28 * _pairs(shapes[p % len(shapes)], int(n)) for p, n in enumerate(lengths))
        return {"bytes": 40 * atoms + 144 * int(lengths.sum()), "flops": flops}
    shape = _shape(case)
    atoms = 40 * shape[2]
    if kind in ("calculate", "field", "adjoint", "adjoint_host"):
        s3 = case["size"] ** 3
        poses = s3 * case["dirs"]
        adjoint = kind.startswith("adjoint")
        return {"bytes": atoms + poses * (28 if adjoint else 4) + (0 if adjoint else 16 * s3),
                "flops": _pairs(shape, poses) * (28 if adjoint else 16)}
    if kind == "poses":
        return {"bytes": atoms + 120 * case["poses"], "flops": 28 * _pairs(shape, case["poses"])}
    if kind == "string":
        evaluations = case["images"] * case["iterations"]
        return {"bytes": atoms + 104 * case["images"],
                "flops": (28 + 16) * _pairs(shape, evaluations)}
    poses = case["centers"] * case["dirs"]
    pairs = _pairs(shape, poses)
    return {"bytes": 24 * case["centers"] + 8 * poses + 4 * pairs / 2 / case["dirs"],
            "flops": 16 * pairs}


# ------------------------------------------------------------------ 64-bit values

#: above this many pairs the plain 64-bit sum takes too long
MOST_PAIRS = 8e10


def _site_sums(frame_case, points, gradient):
    """Plain 64-bit pair sums at Cartesian points [M, 3]: energy [M] and, with
    `gradient`, its derivative [M, 3].  The points are wrapped into the cell
    and taken by bins; a bin's candidates are all images within the cutoff
    plus the bin's radius of its middle."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cell = torch.tensor(np.asarray(frame_case["cell"], dtype=float), device=dev)
    cut = float(frame_case["cutoff"])
    points = torch.as_tensor(points, device=dev)
    frac = points @ torch.linalg.inv(cell)
    frac = frac - torch.floor(frac)
    width = 2.0
    n = [max(1, int(round(1 / np.linalg.norm(np.linalg.inv(frame_case["cell"])[:, k]) / width)))
         for k in range(3)]
    scale = torch.tensor(n, device=dev, dtype=torch.float64)
    at = torch.minimum((frac * scale).long(), (scale - 1).long())
    where = (at[:, 0] * n[1] + at[:, 1]) * n[2] + at[:, 2]
    order = torch.argsort(where)
    number, count = torch.unique_consecutive(where[order], return_counts=True)
    number, count = number.tolist(), count.tolist()
    images, atom = _images(frame_case, cut + 1e-6)
    images = torch.tensor(images, device=dev)
    coeff = torch.tensor(np.stack(_coefficients(frame_case))[:, atom], device=dev)
    cart = frac @ cell
    corner = torch.tensor([[i, j, k] for i in (-.5, .5) for j in (-.5, .5) for k in (-.5, .5)],
                          device=dev, dtype=torch.float64) / scale
    radius = float((corner @ cell).norm(dim=1).max())
    energy = torch.zeros(len(points), dtype=torch.float64, device=dev)
    force = torch.zeros((len(points), 3), dtype=torch.float64, device=dev) if gradient else None
    first = 0
    for b, c in zip(number, count):
        mid = (torch.tensor([b // (n[1] * n[2]), b // n[2] % n[1], b % n[2]], device=dev)
               + 0.5) / scale @ cell
        keep = ((images - mid) ** 2).sum(1) < (cut + radius + 1e-6) ** 2
        x, (c12, c6, shift, floor2) = images[keep], coeff[:, keep]
        step = max(1, (1 << 25) // max(1, len(x)))
        for k in range(first, first + c, step):
            rows = order[k:min(k + step, first + c)]
            d = [cart[rows, j:j + 1] - x[:, j] for j in range(3)]
            d2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            inside = d2 < cut * cut
            i2 = 1 / torch.maximum(d2, floor2)
            i6 = i2 * i2 * i2
            energy[rows] = torch.where(inside, (c12 * i6 - c6) * i6 + shift, 0.0).sum(1)
            if gradient:
                w = torch.where(inside & (d2 >= floor2), (6 * c6 - 12 * c12 * i6) * i6 * i2, 0.0)
                for j in range(3):
                    force[rows, j] = (w * d[j]).sum(1)
        first += c
    return energy, force


def _pose_sums(frame_case, centers, directors, gradient):
    """Energy, dE/dcenter and dE/ddirector of poses (Cartesian centers)."""
    energy, gc, gu = 0.0, 0.0, 0.0
    for o in _offsets(frame_case):
        e, f = _site_sums(frame_case, centers + o * directors, gradient)
        energy = energy + e
        if gradient:
            gc, gu = gc + f, gu + o * f
    return energy, gc, gu


def _field_poses(case, frame_case):
    s, dirs = case["size"], case["dirs"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = (torch.arange(s, dtype=torch.float64, device=dev) + .5) / s
    frac = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    cart = frac @ torch.tensor(np.asarray(frame_case["cell"], dtype=float), device=dev)
    k = np.arange(dirs)
    z = 1 - 2 * (k + .5) / dirs
    phi = k * np.pi * (3 - np.sqrt(5))
    axes = np.stack([np.sqrt(1 - z * z) * np.cos(phi), np.sqrt(1 - z * z) * np.sin(phi), z], 1)
    u = torch.tensor(axes, device=dev)
    u = u / u.norm(dim=1, keepdim=True)
    centers = cart[None].expand(dirs, -1, 3).reshape(-1, 3)
    return axes, cart, centers, u[:, None].expand(-1, s ** 3, 3).reshape(-1, 3)


def _exact_adjoint(case, frame_case):
    _, _, centers, u = _field_poses(case, frame_case)
    e, gc, gu = _pose_sums(frame_case, centers, u, True)
    gu = gu - (gu * u).sum(1, keepdim=True) * u
    shape = (case["dirs"],) + (case["size"],) * 3
    return e.reshape(shape), torch.cat([gc, gu], 1).reshape(shape + (6,))


def _exact_field(case, frame_case):
    axes, cart, centers, u = _field_poses(case, frame_case)
    s, dirs, temp = case["size"], case["dirs"], float(frame_case["temperature"])
    e = _pose_sums(frame_case, centers, u, False)[0].reshape(dirs, -1)
    marginal = -temp * (torch.logsumexp(-e / temp, 0) - math.log(dirs))
    site = _site_sums(frame_case, cart, False)[0].reshape(s, s, s)
    return (axes, e.reshape(dirs, s, s, s), marginal.reshape(s, s, s), torch.stack([site, site]),
            torch.asinh(marginal / 1000).reshape(s, s, s))


def _exact_quaternions(quats, e, gc, gu):
    q = quats / quats.norm(dim=1, keepdim=True)
    w, x, y, z = q.T
    g = torch.stack([2 * z * gu[:, 1] - 2 * y * gu[:, 2], 2 * y * gu[:, 1] + 2 * z * gu[:, 2],
                     -4 * y * gu[:, 0] + 2 * x * gu[:, 1] - 2 * w * gu[:, 2],
                     -4 * z * gu[:, 0] + 2 * w * gu[:, 1] + 2 * x * gu[:, 2]], 1)
    return (g - (g * q).sum(1, keepdim=True) * q) / quats.norm(dim=1, keepdim=True)


def _director(quats):
    w, x, y, z = (quats / quats.norm(dim=1, keepdim=True)).T
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)], 1)


def exact(case, seed):
    kind = case["kind"]
    # a String run is 200 dependent steps with truncations and branches; its
    # poses are the "poses" cases
    if kind == "string" or work(case)["flops"] / 16 > MOST_PAIRS:
        return None
    if kind in ("batch", "paths"):
        cases, rng = _cases_of(case, seed)
        if kind == "batch":
            if case["adjoint"]:
                both = [_exact_adjoint(case, c) for c in cases]
                return [e for e, _ in both] + [g for _, g in both]
            return [_exact_field(case, c)[1] for c in cases]
        counts, centers, quats = _path_poses(case, cases, rng)
        centers, quats = _cuda(centers), _cuda(quats)
        parts, first = [], 0
        for c, n in zip(cases, counts):
            if n:
                rows = slice(first, first + n)
                parts.append(_pose_sums(c, centers[rows], _director(quats[rows]), True))
            first += n
        e, gc, gu = (torch.cat(v) for v in zip(*parts))
        return e, gc, _exact_quaternions(quats, e, gc, gu), gu
    frame_case, rng = _case_of(case, seed)
    if kind == "calculate":
        axes, e, marginal, site, grid = _exact_field(case, frame_case)
        return {"orientation_K": e, "marginal_K": marginal, "site_K": site, "axes": axes,
                "cell_matrix": np.asarray(frame_case["cell"]),
                "atom_fractional": np.asarray(frame_case["frame_frac"]),
                "framework_sigma_A": np.asarray(frame_case["frame_sigma"]),
                "framework_epsilon_K": np.asarray(frame_case["frame_epsilon"]), "grid": grid}
    if kind == "field":
        return _exact_field(case, frame_case)[1:]
    if kind in ("adjoint", "adjoint_host"):
        return _exact_adjoint(case, frame_case)
    if kind == "poses":
        centers = _cuda(rng.random((case["poses"], 3)) @ frame_case["cell"])
        quats = _cuda(synth.random_quaternions(rng, case["poses"]))
        e, gc, gu = _pose_sums(frame_case, centers, _director(quats), True)
        return e, gc, _exact_quaternions(quats, e, gc, gu)
    csr = _csr(case, frame_case, rng)["csr"]
    centers, axes = _cuda(csr[0]), _cuda(csr[1])
    n, m = len(centers), len(axes)
    e = _pose_sums(frame_case, centers[:, None].expand(n, m, 3).reshape(-1, 3),
                   axes[None].expand(n, m, 3).reshape(-1, 3), False)[0]
    return e.reshape(n, m)
