"""Performance cases of the signed-distance framework, each one pass through a public entry point.

The cases cover what a program does with the library: the signed distance field of a new mesh held
on the GPU (mesh build, distances in every mode, signs, combine), the reference's two-result
distance call on host arrays, a batch of uneven meshes from page-locked host memory, and the stages
that follow the field (artifact removal, RBF smoothing).  Sizes run from the 5,120-triangle
icosphere on a 53-node grid, where launches and host waits count, to 1.4M triangles on a 256-node
grid and a thin sheet of several million triangles on a 320-node grid.

Meshes are closed surfaces with float32-rounded coordinates, as an STL import gives them:
icospheres and tori with radial noise, and iso-surfaces of Gaussian blobs and of a thin gyroid
sheet, extracted on the GPU by surface nets (one vertex per mixed lattice cell, one quad per lattice
edge that crosses the surface).
"""

from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stl2sdf.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from stl2sdf import _native  # noqa: E402

MODES = {"ref": _native.MODE_REF_RULE, "exact": _native.MODE_EXACT, "unbounded": _native.MODE_UNBOUNDED,
         "learned": _native.MODE_LEARNED}


def listed():
    return [
        # A small part at a coarse cell size: the shortest call, bound by launches and host waits.
        {"name": "icosphere_ref", "job": "field", "mesh": "icosphere", "level": 4, "nodes": 53, "mode": "ref"},
        # The same part with the learned-radius form (training included): many short launches.
        {"name": "icosphere_learned", "job": "field", "mesh": "icosphere", "level": 4, "nodes": 53, "mode": "learned"},
        # An ordinary part: 131k triangles, 128 nodes, the reference's truncated distance.
        {"name": "torus_ref", "job": "field", "mesh": "torus", "nu": 512, "nv": 128, "nodes": 128, "mode": "ref"},
        # The same with the true (unclamped) distance.
        {"name": "torus_unbounded", "job": "field", "mesh": "torus", "nu": 512, "nv": 128, "nodes": 128,
         "mode": "unbounded"},
        # What evalDistancesOnTriMesh does for a new mesh: host arrays in, distances and closest
        # points out (of every node, so the 3-nearest-vertex fallback runs too).
        {"name": "torus_closest", "job": "closest", "mesh": "torus", "nu": 512, "nv": 128, "nodes": 128},
        # A large scan-like surface: 1.4M triangles, 256 nodes, in the three distance forms.
        {"name": "blobs_ref", "job": "field", "mesh": "blobs", "blobs": 64, "cells": 512, "nodes": 256, "mode": "ref"},
        {"name": "blobs_unbounded", "job": "field", "mesh": "blobs", "blobs": 64, "cells": 512, "nodes": 256,
         "mode": "unbounded"},
        {"name": "blobs_learned", "job": "field", "mesh": "blobs", "blobs": 64, "cells": 512, "nodes": 256,
         "mode": "learned"},
        # A thin double-walled sheet on the largest grid, the true minimum clamped at the cell size:
        # many triangles per node, many grazing rays.
        {"name": "sheet_exact", "job": "field", "mesh": "sheet", "cells": 384, "thickness": 0.04, "nodes": 320,
         "mode": "exact"},
        # Uneven meshes in one call, end to end from page-locked host memory.
        {"name": "batch_ref", "job": "batch", "count": 32, "mode": "ref"},
        # Small-component removal on a large device-resident field.
        {"name": "artifacts", "job": "artifacts", "blobs": 64, "nodes": 256, "noise": 0.001},
        # RBF interpolation of a truncated field, refined twice (host arrays, as stl_to_sdf calls it).
        {"name": "smoothing", "job": "smoothing", "nodes": 128, "interpolation": True, "refine": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    job = rng.choice(["field"] * 8 + ["closest", "batch", "artifacts", "smoothing"])
    if job == "batch":
        return {"job": "batch", "count": rng.randint(3, 32), "mode": rng.choice(["ref", "exact"])}
    if job == "artifacts":
        return {"job": "artifacts", "blobs": rng.randint(8, 64), "nodes": _log_int(rng, 20, 256),
                "noise": math.exp(rng.uniform(math.log(1e-4), math.log(1e-2)))}
    if job == "smoothing":
        return {"job": "smoothing", "nodes": _log_int(rng, 16, 128), "interpolation": rng.random() < 0.7,
                "refine": rng.choice([1, 2])}
    kind = rng.choice(["icosphere", "torus", "blobs", "blobs", "sheet"])
    case = {"job": job, "mesh": kind}
    if kind == "icosphere":
        case.update(level=rng.randint(2, 6))
    elif kind == "torus":
        case.update(nu=_log_int(rng, 24, 1024), nv=_log_int(rng, 12, 256))
    elif kind == "blobs":
        case.update(blobs=rng.randint(8, 64), cells=_log_int(rng, 32, 512))
    else:
        cells = _log_int(rng, 64, 384)  # walls of one to four lattice cells
        case.update(cells=cells, thickness=round(15.4 / cells * rng.uniform(1.0, 4.0), 4))
    if job == "closest":
        case.update(nodes=_log_int(rng, 20, 96))
        return case
    case["mode"] = rng.choice(["ref", "exact", "unbounded", "learned"])
    full = case["mode"] in ("ref", "exact")
    case["nodes"] = _log_int(rng, 24, 256 if full else 160)
    return case


# ---- meshes ------------------------------------------------------------------------------------

def _icosphere(level, rng):
    p = (1.0 + 5.0 ** 0.5) / 2.0
    V = np.array([[-1, p, 0], [1, p, 0], [-1, -p, 0], [1, -p, 0], [0, -1, p], [0, 1, p],
                  [0, -1, -p], [0, 1, -p], [p, 0, -1], [p, 0, 1], [-p, 0, -1], [-p, 0, 1]], np.float64)
    V /= np.linalg.norm(V, axis=1, keepdims=True)
    F = np.array([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                  [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5],
                  [2, 4, 11], [6, 2, 10], [8, 6, 7], [9, 8, 1]], np.int64)
    for _ in range(level):
        E = np.sort(np.concatenate([F[:, [0, 1]], F[:, [1, 2]], F[:, [2, 0]]]), axis=1)
        u, inv = np.unique(E[:, 0] * len(V) + E[:, 1], return_inverse=True)
        M = V[u // len(V)] + V[u % len(V)]
        M /= np.linalg.norm(M, axis=1, keepdims=True)
        ab, bc, ca = (inv.reshape(3, -1) + len(V))
        V = np.concatenate([V, M])
        a, b, c = F.T
        F = np.stack([np.stack(t, 1) for t in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))], 1).reshape(-1, 3)
    return V * (1.0 + rng.normal(0.0, 0.01, (len(V), 1))), F


def _torus(nu, nv, rng):
    u, v = np.meshgrid(2 * np.pi * np.arange(nu) / nu, 2 * np.pi * np.arange(nv) / nv, indexing="ij")
    r = 0.3 * (1.0 + rng.uniform(-0.02, 0.02, u.shape))
    X = np.stack([(1 + r * np.cos(v)) * np.cos(u), (1 + r * np.cos(v)) * np.sin(u), r * np.sin(v)], -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
    a, b = i * nv + j, (i + 1) % nu * nv + j
    c, d = (i + 1) % nu * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    return X, np.stack([np.stack([a, b, c], -1), np.stack([a, c, d], -1)], 2).reshape(-1, 3)


def _blob_field(axes, n, rng, device="cuda"):
    """Sum of n unit-amplitude Gaussians (centres U[-1,1]^3, sigma U[0.1,0.3]) on a lattice."""
    C, S = rng.uniform(-1.0, 1.0, (n, 3)), rng.uniform(0.1, 0.3, n)
    f = torch.zeros([len(a) for a in axes], dtype=torch.float32, device=device)
    for c, s in zip(C, S):
        g = [torch.exp(-0.5 * ((a - float(x)) / float(s)) ** 2).float() for a, x in zip(axes, c)]
        f.addcmul_(g[0][:, None, None], g[1][:, None] * g[2][None, :])
    return f


def _surface_nets(f, lo, step):
    """Closed quad surface of f > 0, split into triangles: (vertices float64, triangles int64)."""
    inside = f > 0
    n = [s - 1 for s in f.shape]

    def corner(t, i, j, k):
        return t[i:i + n[0], j:j + n[1], k:k + n[2]]

    corners = [(i, j, k) for i in (0, 1) for j in (0, 1) for k in (0, 1)]
    some, every = corner(inside, 0, 0, 0).clone(), corner(inside, 0, 0, 0).clone()
    for c in corners[1:]:
        some |= corner(inside, *c)
        every &= corner(inside, *c)
    cell = torch.nonzero(some & ~every)
    del some, every
    vid = torch.full(n, -1, dtype=torch.int32, device=f.device)
    vid[cell[:, 0], cell[:, 1], cell[:, 2]] = torch.arange(len(cell), dtype=torch.int32, device=f.device)
    val = {c: f[cell[:, 0] + c[0], cell[:, 1] + c[1], cell[:, 2] + c[2]].double() for c in corners}
    total = torch.zeros(len(cell), 3, dtype=torch.float64, device=f.device)
    count = torch.zeros(len(cell), 1, dtype=torch.float64, device=f.device)
    for a in range(3):
        for c in corners:
            if c[a]:
                continue
            e = tuple(1 if x == a else c[x] for x in range(3))
            hit = (val[c] > 0) != (val[e] > 0)
            t = torch.where(hit, val[c] / torch.where(hit, val[c] - val[e], 1.0), 0.0)
            p = torch.tensor(c, dtype=torch.float64, device=f.device).repeat(len(cell), 1)
            p[:, a] = t
            total += torch.where(hit[:, None], p, 0.0)
            count += hit[:, None]
    X = (cell.double() + total / count) * step + torch.tensor(lo, dtype=torch.float64, device=f.device)
    tris = []
    for a in range(3):
        b, c = (a + 1) % 3, (a + 2) % 3
        s0 = [slice(1, -1)] * 3
        s1 = list(s0)
        s0[a], s1[a] = slice(0, -1), slice(1, None)
        one, two = inside[tuple(s0)], inside[tuple(s1)]
        at = torch.nonzero(one != two)
        up = one[at[:, 0], at[:, 1], at[:, 2]]
        at = at + torch.tensor([0 if x == a else 1 for x in range(3)], device=f.device)
        quad = []
        for db, dc in ((1, 1), (0, 1), (0, 0), (1, 0)):
            q = at.clone()
            q[:, b] -= db
            q[:, c] -= dc
            quad.append(vid[q[:, 0], q[:, 1], q[:, 2]].long())
        q0, q1, q2, q3 = quad
        q1, q3 = torch.where(up, q1, q3), torch.where(up, q3, q1)
        tris.append(torch.stack([torch.stack([q0, q2, q3], 1), torch.stack([q0, q1, q2], 1)], 1).reshape(-1, 3))
    return X, torch.cat(tris)


def _mesh(case, rng):
    """(X float64 (nnp, 3) rounded through float32, IEN int64 (nel, 3) 1-based), both on the GPU."""
    kind = case["mesh"]
    if kind in ("icosphere", "torus"):
        V, F = _icosphere(case["level"], rng) if kind == "icosphere" else _torus(case["nu"], case["nv"], rng)
        V, F = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    elif kind == "blobs":
        x = torch.linspace(-2.0, 2.0, case["cells"] + 1, dtype=torch.float64, device="cuda")
        V, F = _surface_nets(_blob_field([x, x, x], case["blobs"], rng) - 0.5, [-2.0] * 3, 4.0 / case["cells"])
    else:
        # |gyroid| <= thickness over two periods, shifted by a random phase, closed at the border
        m = case["cells"]
        s = 4.0 * math.pi / m
        g = [torch.arange(m + 1, dtype=torch.float64, device="cuda") * s + float(q) for q in rng.uniform(0, 2 * math.pi, 3)]
        sn, cs = [torch.sin(t).float() for t in g], [torch.cos(t).float() for t in g]
        f = sn[0][:, None, None] * cs[1][None, :, None] + sn[1][None, :, None] * cs[2][None, None, :]
        f = f + sn[2][None, None, :] * cs[0][:, None, None]
        f = case["thickness"] - f.abs()
        f = torch.nn.functional.pad(f, (1,) * 6, value=-1.0)
        V, F = _surface_nets(f, [-2.0 * math.pi - s] * 3, s)
    return V.float().double().contiguous(), (F + 1).contiguous()


# The box each kind of mesh lies in (a blob surface can reach past its box by a little), so that a
# case's grid does not depend on its seed.
BOX = {"icosphere": (1.03, 1.03, 1.03), "torus": (1.31, 1.31, 0.31), "blobs": (1.45, 1.45, 1.45),
       "sheet": (2 * math.pi, 2 * math.pi, 2 * math.pi)}


def _grid(kind, nodes):
    """Grid of about `nodes` nodes on the longest axis of the kind's box, padded by 3 cells: (origin, h, N)."""
    hi = np.array(BOX[kind])
    o, _, N, h, _ = _native.grid_setup(-hi, hi, max(nodes - 7, 1))
    return o, h, N


# ---- cases -------------------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    job = case["job"]
    s = {"case": case}
    if job in ("field", "closest"):
        X, IEN = _mesh(case, rng)
        s["X"], s["IEN"] = X, IEN
        s["grid"] = o, h, N = _grid(case["mesh"], case["nodes"])
        s["ctx"] = _native.Context(0)
        if job == "closest":
            s["X"], s["IEN"] = X.cpu().numpy(), IEN.cpu().numpy()
        else:
            ngp = int(np.prod(N + 1))
            s["sdf"] = torch.empty(ngp, dtype=torch.float64, device="cuda")
            s["conf"] = torch.empty(ngp, dtype=torch.float64, device="cuda")
    elif job == "batch":
        s["meshes"], s["out"] = [], []
        sizes = np.random.default_rng(case["count"])
        for k in range(case["count"]):
            # half icospheres of level 2..6, half iso-surfaces of 8..32 blobs; grids of 32..160 nodes
            c = ({"mesh": "icosphere", "level": int(sizes.integers(2, 7))} if k % 2 == 0 else
                 {"mesh": "blobs", "blobs": int(sizes.integers(8, 33)),
                  "cells": int(round(32 * 10 ** sizes.uniform(0, 1)))})
            X, IEN = _mesh(c, rng)
            o, h, N = _grid(c["mesh"], int(sizes.integers(32, 161)))
            s["meshes"].append((X.cpu().pin_memory().numpy(), IEN.cpu().pin_memory().numpy(), o, h, N))
            s["out"].append(torch.empty(int(np.prod(N + 1)), dtype=torch.float64).pin_memory().numpy())
        s["ctx"] = _native.Context(0)
    elif job == "artifacts":
        n = case["nodes"]
        N = np.array([n - 1, n - 1 - n // 16, n - 1 - n // 10], np.int64)
        ax = [torch.linspace(-1.6, 1.6, int(m) + 1, dtype=torch.float64, device="cuda") for m in N[::-1]]
        f = _blob_field(ax, case["blobs"], rng).double().reshape(-1) - 0.5
        # stray sign errors, the islands the stage is there to remove
        flip = torch.from_numpy(rng.random(f.numel()) < case["noise"]).cuda()
        s["field"] = torch.where(flip, -f, f).contiguous()
        s["sdf"] = torch.empty_like(s["field"])
        s["N"] = N
        s["ctx"] = _native.Context(0)
        s["stream"] = torch.cuda.ExternalStream(s["ctx"].stream_ptr())
    else:
        o, h, N = _grid("torus", case["nodes"])
        x, y, z = np.meshgrid(*[o[a] + h * np.arange(N[a] + 1) for a in range(3)], indexing="ij")
        d = 0.3 - np.sqrt((np.sqrt(x * x + y * y) - 1.0) ** 2 + z * z) + rng.uniform(-0.05, 0.05) * h
        d = d + rng.normal(0.0, 0.02 * h, d.shape)
        s["dist"] = np.ascontiguousarray(np.clip(d, -h, h).transpose(2, 1, 0)).reshape(-1)
        s["grid"] = o, h, N
        s["ctx"] = _native.Context(0)
    torch.cuda.synchronize()
    return s


def run(state):
    case = state["case"]
    job = case["job"]
    if job == "field":
        ctx, (o, h, N), X, IEN = state["ctx"], state["grid"], state["X"], state["IEN"]
        ctx.set_mesh_device(X.data_ptr(), X.shape[0], IEN.data_ptr(), IEN.shape[0])
        if case["mode"] == "learned":
            ctx.train_radius()
        ctx.sdf_device(o, h, N, state["sdf"].data_ptr(), MODES[case["mode"]], conf_ptr=state["conf"].data_ptr())
        return state["sdf"], state["conf"]
    if job == "closest":
        state["ctx"].set_mesh(state["X"], state["IEN"])
        return state["ctx"].distances(*state["grid"], want_xp=True)
    if job == "batch":
        return state["ctx"].sdf_batch(state["meshes"], MODES[case["mode"]], out=state["out"])
    if job == "artifacts":
        ctx, sdf = state["ctx"], state["sdf"]
        with torch.cuda.stream(state["stream"]):  # the field's copy runs on the library's own stream
            sdf.copy_(state["field"])
        counts = [ctypes.c_int64() for _ in range(3)]
        rc = _native.lib().sdfgpu_remove_artifacts_device(
            ctx.handle, state["N"].ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), ctypes.c_void_p(sdf.data_ptr()),
            0.0, 0.01, *[ctypes.byref(c) for c in counts])
        if rc:
            raise _native.SdfGpuError(rc, "remove_artifacts")
        return (sdf, *[c.value for c in counts])
    o, h, N = state["grid"]
    fine, _, _, _ = state["ctx"].rbf_smoothing(o, o + h * N, N, h, state["dist"], case["interpolation"], case["refine"])
    return fine


def _sizes(case):
    """(triangles, grid nodes) of a field or closest case, estimated from its recipe."""
    kind, n = case["mesh"], case["nodes"]
    if kind == "icosphere":
        return 20 * 4 ** case["level"], n ** 3
    if kind == "torus":
        return 2 * case["nu"] * case["nv"], int(0.28 * n ** 3)
    if kind == "blobs":
        return int(5.4 * case["cells"] ** 2), n ** 3
    return int(37 * case["cells"] ** 2), n ** 3


def work(case):
    """Bytes: the mesh (24 B per vertex and per triangle), fields and results once.  Operations: per
    node one FP32 point-triangle distance (162) and, for a sign, the ray tests of its three rows
    (three of 52 per node at the least); per triangle its record (about 200)."""
    job = case["job"]
    if job in ("field", "closest"):
        nel, ngp = _sizes(case)
        out = 16 if job == "field" else 32
        return {"bytes": 36 * nel + out * ngp, "flops": 200 * nel + ngp * (162 + (156 if job == "field" else 0))}
    if job == "batch":
        nel, ngp = 40_000 * case["count"], 850_000 * case["count"]
        return {"bytes": 36 * nel + 8 * ngp, "flops": 200 * nel + 318 * ngp}
    if job == "artifacts":
        ngp = int(0.84 * case["nodes"] ** 3)
        return {"bytes": 24 * ngp, "flops": 6 * ngp}  # the copy (16 B per node) and the pass (8)
    n = case["nodes"]
    ngp = int(0.28 * n ** 3)
    fine = ngp * case["refine"] ** 3
    # the fine evaluation (81 terms a point); interpolation: about 30 products of 81 terms as well
    return {"bytes": 8 * ngp + 4 * fine, "flops": 4 * 81 * fine + (30 * 2 * 81 * ngp if case["interpolation"] else 0)}


# ---- 64-bit values -----------------------------------------------------------------------------

def _exact_field(X, IEN, o, h, N):
    """Distance to the nearest triangle and inside (+1) / outside (-1) by the winding number, float64."""
    ax = [torch.from_numpy(o[a] + h * np.arange(N[a] + 1)).cuda() for a in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    P = torch.stack([x, y, z], -1).reshape(-1, 3)
    T = X[IEN - 1]
    a, b, c = (T[:, k][None] for k in range(3))
    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(-1)
    best = torch.empty(len(P), dtype=torch.float64, device="cuda")
    wind = torch.empty_like(best)
    chunk = max(1, 20_000_000 // T.shape[0])
    for i in range(0, len(P), chunk):
        p = P[i:i + chunk, None, :]
        d2, ins = None, None
        for u, v in ((a, b), (b, c), (c, a)):
            e, w = v - u, p - u
            t = ((w * e).sum(-1) / (e * e).sum(-1)).clamp(0, 1)
            q = w - t[..., None] * e
            s = (q * q).sum(-1)
            k = (torch.linalg.cross(e.expand_as(w), w) * n).sum(-1) >= 0
            d2, ins = (s, k) if d2 is None else (torch.minimum(d2, s), ins & k)
        pl = ((p - a) * n).sum(-1) ** 2 / nn
        best[i:i + chunk] = torch.where(ins, torch.minimum(d2, pl), d2).min(1).values.sqrt()
        ra, rb, rc = a - p, b - p, c - p
        la, lb, lc = ra.norm(dim=-1), rb.norm(dim=-1), rc.norm(dim=-1)
        num = (ra * torch.linalg.cross(rb, rc)).sum(-1)
        den = la * lb * lc + (ra * rb).sum(-1) * lc + (rb * rc).sum(-1) * la + (rc * ra).sum(-1) * lb
        wind[i:i + chunk] = 2 * torch.atan2(num, den).sum(1) / (4 * math.pi)
    return best, torch.where(wind.abs() > 0.5, 1.0, -1.0)


def _exact_smoothing(case, seed):
    """The Gaussian interpolant (or approximant) in float64: conjugate gradients run to 1e-13."""
    s = prepare(case, seed)
    o, h, N = s["grid"]
    n = [int(v) + 1 for v in N]
    d = torch.from_numpy(s["dist"]).cuda().reshape(n[2], n[1], n[0])
    cut = -math.log(1e-3)

    def gather(w, m, shape, shift):
        """Sum over coarse nodes within the cut-off of the points at (m index + shift) / m cells."""
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
        pad = torch.nn.functional.pad(w, (3,) * 6)
        for oz in range(-3, 4):
            for oy in range(-3, 4):
                for ox in range(-3, 4):
                    r2 = sum((k - f / m) ** 2 for k, f in zip((oz, oy, ox), shift))
                    if r2 < cut:
                        out += math.exp(-r2) * pad[3 + oz:3 + oz + shape[0], 3 + oy:3 + oy + shape[1],
                                                   3 + ox:3 + ox + shape[2]]
        return out

    w = d
    if case["interpolation"]:
        x, r = torch.zeros_like(d), d.clone()
        u, rr = r.clone(), (r * r).sum()
        stop = 1e-26 * rr
        for _ in range(400):
            c = gather(u, 1, n[::-1], (0, 0, 0))
            al = rr / (u * c).sum()
            x += al * u
            r -= al * c
            new = (r * r).sum()
            if new <= stop:
                break
            u, rr = r + (new / rr) * u, new
        w = x
    m = case["refine"]
    fine = torch.empty([(k - 1) * m + 1 for k in n[::-1]], dtype=torch.float64, device="cuda")
    for z in range(m):
        for y in range(m):
            for x in range(m):
                part = fine[z::m, y::m, x::m]
                part.copy_(gather(w, m, list(part.shape), (z, y, x)))
    return fine.reshape(-1).cpu().numpy()


def exact(case, seed):
    """float64 values where the result is defined by its inputs alone: true-distance fields small
    enough for all pairs (the reference rule's truncated distance depends on the order of its
    candidates), and the smoothed field."""
    if case["job"] == "smoothing":
        return _exact_smoothing(case, seed)
    if case["job"] == "field" and case["mode"] != "ref":
        X, IEN = _mesh(case, np.random.default_rng(seed))
        o, h, N = _grid(case["mesh"], case["nodes"])
        if IEN.shape[0] * int(np.prod(N + 1)) <= 4_000_000_000 and case["mesh"] != "sheet":
            d, sign = _exact_field(X, IEN, o, h, N)
            if case["mode"] == "exact":
                d = d.clamp(max=h)
            return d * sign, None
    return None
