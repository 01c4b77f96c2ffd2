"""Workloads of the RMSD library, for timing and for comparing results.

``listed()`` names the workloads, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call
(frames, references and, where the API has one, the prepared handle),
``run(state)`` is one pass through the public entry points (the plans, the
torch functions, the batched launch, the C ABI), ``work(case)`` the bytes and
operations a pass cannot do without, and ``exact(case, seed)`` the same results
from plain torch in 64 bits.

Trajectories are random-walk chains (3.8 A steps) that tumble and diffuse, with
0.2 to 3 A of noise per atom, or chains that drift from frame to frame for the
all-pairs and clustering workloads.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warp-md_b200"))

from warp_md import RmsdPlan, System, Trajectory  # noqa: E402
from warp_md import _native as N  # noqa: E402
from warp_md import torch_ops  # noqa: E402
from warp_md.batched import BatchedRmsd  # noqa: E402

DEV = "cuda:0"
PAIR_MODE = {"fp64": N.MODE_FP64, "i8x3": N.MODE_I8X3}


# ---------------------------------------------------------------- cases --

def listed():
    return [
        # the smallest call a script makes: RmsdPlan on a short in-memory trajectory of a small protein
        {"name": "plan_small", "kind": "plan", "frames": 100, "atoms": 500, "sel": "all", "align": True},
        # RmsdPlan on an in-memory trajectory of a solvated system, fitted on every tenth atom (CA-like)
        {"name": "plan_ca", "kind": "plan", "frames": 1000, "atoms": 20000, "sel": "tenth", "align": True},
        # streaming per-frame RMSD of a large system with the frames on the GPU (the headline workload, shortened)
        {"name": "frames_large", "kind": "frames", "frames": 4000, "atoms": 100000, "stride": 3, "sel": "all",
         "align": True},
        # a mid-sized protein whose frames are not a multiple of 16 bytes
        {"name": "frames_odd", "kind": "frames", "frames": 5001, "atoms": 3001, "stride": 3, "sel": "all",
         "align": True},
        # one step of a small restrained fit: RMSD under autograd and its backward
        {"name": "autograd_small", "kind": "autograd", "frames": 64, "atoms": 250, "sel": "all"},
        # differentiable RMSD over a batch of conformations, value and gradient at once
        {"name": "value_grad", "kind": "value_grad", "frames": 4096, "atoms": 2000},
        # all-pairs matrix in the plans' default arithmetic (PairwiseRmsdPlan, the DBSCAN distances)
        {"name": "pair_fp64", "kind": "pair", "frames": 4000, "atoms": 500, "mode": "fp64", "metric": "rms"},
        # all-pairs matrix of a long trajectory on the tensor cores
        {"name": "pair_i8x3", "kind": "pair", "frames": 20000, "atoms": 1000, "mode": "i8x3", "metric": "rms"},
        # k-means over the superposed frames of a trajectory
        {"name": "kmeans", "kind": "cluster", "method": "kmeans", "frames": 10000, "atoms": 600, "clusters": 8},
        # SuperposePlan: mass-weighted fit on every tenth atom, every atom of every frame moved
        {"name": "superpose", "kind": "superpose", "frames": 1000, "atoms": 100000, "sel": "tenth", "mass": True},
        # RmsdPerResPlan: fit on every tenth atom, ten-atom residues
        {"name": "per_residue", "kind": "residue", "frames": 1000, "atoms": 100000, "sel": "tenth"},
        # RMSD and gradients of many trajectories of uneven size in one launch
        {"name": "batched", "kind": "batched", "trajectories": 30, "min_atoms": 50, "max_atoms": 20000,
         "min_frames": 100, "max_frames": 5000, "grad": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "frames", "frames", "autograd", "value_grad", "pair", "pair", "cluster", "superpose",
                       "residue", "batched"])
    if kind == "plan":
        return {"kind": kind, "frames": _log(rng, 20, 1000), "atoms": _log(rng, 100, 20000),
                "sel": rng.choice(["all", "tenth", "half"]), "align": rng.random() < 0.8}
    if kind == "frames":
        atoms = _log(rng, 100, 100000)
        return {"kind": kind, "frames": max(1, min(20000, _log(rng, 2e6, 4e8) // atoms)), "atoms": atoms,
                "stride": rng.choice([3, 3, 4]), "sel": rng.choice(["all", "all", "tenth"]),
                "align": rng.random() < 0.8}
    if kind == "autograd":
        return {"kind": kind, "frames": _log(rng, 16, 4096), "atoms": _log(rng, 50, 2500),
                "sel": rng.choice(["all", "all", "half"])}
    if kind == "value_grad":
        return {"kind": kind, "frames": _log(rng, 64, 6000), "atoms": _log(rng, 100, 4000)}
    if kind == "pair":
        mode = rng.choice(["fp64", "i8x3"])
        return {"kind": kind, "frames": _log(rng, 100, 4000 if mode == "fp64" else 12000),
                "atoms": _log(rng, 50, 1200), "mode": mode, "metric": rng.choice(["rms", "rms", "nofit"])}
    if kind == "cluster":
        method = rng.choice(["kmeans", "dbscan"])
        return {"kind": kind, "method": method, "frames": _log(rng, 200, 10000 if method == "kmeans" else 3000),
                "atoms": _log(rng, 50, 800), "clusters": rng.choice([4, 8, 13])}
    if kind == "superpose":
        return {"kind": kind, "frames": _log(rng, 50, 2000), "atoms": _log(rng, 2000, 60000),
                "sel": rng.choice(["all", "tenth"]), "mass": rng.random() < 0.5}
    if kind == "residue":
        return {"kind": kind, "frames": _log(rng, 50, 2000), "atoms": _log(rng, 2000, 60000),
                "sel": rng.choice(["all", "tenth"])}
    return {"kind": kind, "trajectories": rng.randint(3, 30), "min_atoms": 50, "max_atoms": _log(rng, 500, 20000),
            "min_frames": 20, "max_frames": _log(rng, 200, 5000), "grad": rng.random() < 0.7}


# --------------------------------------------------------------- inputs --

def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _chain(atoms, g):
    d = torch.randn(atoms, 3, generator=g, device=DEV, dtype=torch.float64)
    d /= d.norm(dim=1, keepdim=True)
    d[0] = 0
    return torch.cumsum(3.8 * d, dim=0)


def _rotations(m, g):
    q = torch.randn(m, 4, generator=g, device=DEV, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).reshape(m, 3, 3)


def _rows(atoms):
    """Frames handled at a time: about 10 million atoms."""
    return max(1, 10_000_000 // max(atoms, 1))


def _tumbling(frames, atoms, g, drift=0.0, stride=3):
    """frames x atoms x stride float32 and the chain they fluctuate about."""
    ref = _chain(atoms, g)
    out = torch.empty(frames, atoms, stride, device=DEV, dtype=torch.float32)
    cur = ref.clone()
    for f0 in range(0, frames, _rows(atoms)):
        m = min(_rows(atoms), frames - f0)
        if drift:
            walk = cur + torch.cumsum(drift * torch.randn(m, atoms, 3, generator=g, device=DEV), dim=0).double()
            cur = walk[-1].clone()
        else:
            s = 0.2 + 2.8 * torch.rand(m, 1, 1, generator=g, device=DEV)
            walk = ref + (s * torch.randn(m, atoms, 3, generator=g, device=DEV)).double()
        t = 10.0 * torch.randn(m, 1, 3, generator=g, device=DEV, dtype=torch.float64)
        out[f0:f0 + m, :, :3] = torch.matmul(walk, _rotations(m, g).transpose(1, 2)) + t
        if stride == 4:
            out[f0:f0 + m, :, 3] = 0
    return out, ref.float()


def _selection(sel, atoms):
    if sel == "tenth":
        return np.arange(1, atoms, 10, dtype=np.uint32)
    if sel == "half":
        return np.arange(0, atoms, 2, dtype=np.uint32)
    return None


def _batch_sizes(case, seed):
    rng = np.random.default_rng(7)  # sizes belong to the case, not to the seed
    lo, hi = math.log(case["min_atoms"]), math.log(case["max_atoms"])
    n = case["trajectories"]
    return [(int(round(math.exp(a))), int(f)) for a, f in
            zip(rng.uniform(lo, hi, n), rng.integers(case["min_frames"], case["max_frames"] + 1, n))]


def _inputs(case, seed):
    """The arrays of a case: coords, ref, sel (numpy or None), weights (or None); lists for a batch."""
    g = _gen(seed)
    k = case["kind"]
    if k == "batched":
        made = [_tumbling(f, n, g) for n, f in _batch_sizes(case, seed)]
        return {"coords": [m[0] for m in made], "ref": [m[1] for m in made]}
    drift = 0.1 if k in ("pair", "cluster") else 0.0
    coords, ref = _tumbling(case["frames"], case["atoms"], g, drift, case.get("stride", 3))
    sel = _selection(case.get("sel", "all"), case["atoms"])
    w = None
    if case.get("mass"):
        kinds = torch.tensor([1.008, 12.011, 14.007, 15.999], device=DEV)
        w = kinds[torch.randint(0, 4, (case["atoms"],), generator=g, device=DEV)]
        w = w if sel is None else w[torch.from_numpy(sel.astype(np.int64)).to(DEV)]
    return {"coords": coords, "ref": ref, "sel": sel, "w": w}


def prepare(case, seed):
    d = _inputs(case, seed)
    k = case["kind"]
    s = {"kind": k, "case": case}
    if k == "plan":
        n = case["atoms"]
        coords = d["coords"].cpu().numpy()
        table = {"name": ["CA"] * n, "resname": ["ALA"] * n, "resid": list(range(1, n + 1)), "mass": [12.011] * n}
        system = System.from_arrays(table, positions0=d["ref"].cpu().numpy())
        pick = system.select("all") if d["sel"] is None else system.select_indices(d["sel"])
        s.update(traj=Trajectory.from_numpy(coords), system=system, plan=RmsdPlan(pick, align=case["align"]))
        return s
    if k == "batched":
        s["batch"] = BatchedRmsd(d["coords"], d["ref"], with_grad=case["grad"])
        return s
    s["x"] = d["coords"]
    sel = d["sel"]
    s["n_sel"] = case["atoms"] if sel is None else int(sel.size)
    s["sel"] = None if sel is None else torch.from_numpy(sel.astype(np.int32)).to(DEV)
    ref_sel = d["ref"] if sel is None else d["ref"][s["sel"].long()].contiguous()
    if k == "autograd":
        s["x"].requires_grad_(True)
        s["ref"] = ref_sel
    elif k == "value_grad":
        s["ref"] = ref_sel
    elif k in ("frames", "superpose", "residue"):
        ctx = N.context(0)
        w = None if d["w"] is None else d["w"].cpu().numpy()
        s["handle"] = N.Reference.from_numpy(ctx, ref_sel.cpu().numpy(), weights=w)
        if k == "residue":
            n = case["atoms"]
            off = np.append(np.arange(0, n, 10), n).astype(np.uint32)
            s["groups"] = N.GroupRef(ctx, d["ref"].cpu().numpy(), off, np.arange(n, dtype=np.uint32))
    return s


# ---------------------------------------------------------------- calls --

def _ptr(t):
    return None if t is None else t.data_ptr()


def run(state):
    k, c = state["kind"], state["case"]
    if k == "plan":
        return state["plan"].run(state["traj"], state["system"])
    if k == "batched":
        b = state["batch"]
        return {"rmsd": b.run(), "grad": b.grads} if c["grad"] else {"rmsd": b.run()}
    x = state["x"]
    if k == "autograd":
        x.grad = None
        r = torch_ops.rmsd(x, state["ref"], state["sel"])
        r.sum().backward()
        return {"rmsd": r.detach(), "grad": x.grad}
    if k == "value_grad":
        r, g = torch_ops.rmsd_value_and_grad(x, state["ref"])
        return {"rmsd": r, "grad": g}
    if k == "pair":
        return torch_ops.pairwise(x, c["metric"], c["mode"])
    ctx = N.context(0)
    stream = torch.cuda.current_stream().cuda_stream
    F, n, sel, m = c["frames"], c["atoms"], _ptr(state["sel"]), state["n_sel"]
    if k == "frames":
        out = torch.empty(F, dtype=torch.float64, device=DEV)
        ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x.data_ptr(), F, n, c["stride"], sel, m, state["handle"].handle,
                                          int(c["align"]), out.data_ptr(), stream))
        return out
    if k == "superpose":
        out = torch.empty(F, n, 3, dtype=torch.float32, device=DEV)
        rows = torch.empty(F, 12, dtype=torch.float32, device=DEV)
        ctx.check(ctx.lib.wmd_superpose(ctx.handle, x.data_ptr(), F, n, 3, sel, m, state["handle"].handle, 0,
                                        out.data_ptr(), rows.data_ptr(), stream))
        return {"coords": out, "transforms": rows}
    if k == "residue":
        out = torch.empty(F, state["groups"].n_groups, dtype=torch.float32, device=DEV)
        ctx.check(ctx.lib.wmd_rmsd_per_group(ctx.handle, x.data_ptr(), F, n, 3, sel, m, state["handle"].handle,
                                             state["groups"].handle, 1, out.data_ptr(), stream))
        return out
    labels, cent, sizes = np.empty(F, np.int32), np.empty(F, np.uint32), np.empty(F, np.uint32)
    found = ctypes.c_int64(0)
    if c["method"] == "kmeans":
        ctx.check(ctx.lib.wmd_cluster_kmeans(ctx.handle, x.data_ptr(), F, n, 3, None, n, c["clusters"], 20, 1e-4, 7,
                                             labels.ctypes.data, cent.ctypes.data, sizes.ctypes.data, found, stream))
    else:
        eps = 0.1 * math.sqrt(3 * 4 * F / 100.0)  # about F / 25 frames of drift
        ctx.check(ctx.lib.wmd_cluster_dbscan(ctx.handle, x.data_ptr(), F, n, 3, None, n, N.MODE_FP64, eps, 5,
                                             labels.ctypes.data, cent.ctypes.data, sizes.ctypes.data, found, stream))
    kk = int(found.value)
    return {"labels": labels, "centroids": cent[:kk].copy().astype(np.int64), "sizes": sizes[:kk].copy().astype(np.int64)}


# ----------------------------------------------------------------- work --

def work(case):
    k = case["kind"]
    if k == "batched":
        sizes = _batch_sizes(case, 0)
        af = sum(n * f for n, f in sizes)
        per = 24 if case["grad"] else 12
        return {"bytes": per * af + sum(12 * n + 8 * f for n, f in sizes), "flops": (60 if case["grad"] else 30) * af}
    F, n = case["frames"], case["atoms"]
    sel = _selection(case.get("sel", "all"), n)
    m = n if sel is None else int(sel.size)
    if k == "plan":
        return {"bytes": F * m * 12 + m * 12 + F * 4, "flops": 30 * F * m}
    if k == "frames":
        return {"bytes": F * m * 12 + m * 12 + F * 8, "flops": 30 * F * m}
    if k == "autograd":
        return {"bytes": F * (m + n) * 12 + m * 12 + F * 8, "flops": 60 * F * m}
    if k == "value_grad":
        return {"bytes": F * n * 24 + n * 12 + F * 8, "flops": 60 * F * n}
    if k == "pair":
        return {"bytes": F * n * 12 + F * F * 4, "flops": 18 * n * (F * (F - 1) // 2)}
    if k == "superpose":
        return {"bytes": F * n * 24 + m * 16 + F * 48, "flops": 30 * F * m + 18 * F * n}
    if k == "residue":
        return {"bytes": F * n * 12 + n * 12 + F * (n // 10) * 4, "flops": 30 * F * m + 27 * F * n}
    if case["method"] == "kmeans":  # features once per iteration at least; up to 20 iterations
        return {"bytes": F * n * 12 + F * 4, "flops": 20 * F * 3 * n * (3 * case["clusters"] + 1)}
    return {"bytes": F * n * 12 + F * 4, "flops": 18 * n * (F * (F - 1) // 2)}


# ---------------------------------------------------------------- exact --

def _kabsch(x, y, w=None):
    """Centroids, rotations R (R (x - cx) ~ y - cy) and residual sums of frames x [m, n, 3] on y [n, 3], float64."""
    ww = torch.ones(y.shape[0], dtype=torch.float64, device=y.device) if w is None else w.double()
    cx = (x * ww[None, :, None]).sum(1) / ww.sum()
    cy = (y * ww[:, None]).sum(0) / ww.sum()
    dx, dy = x - cx[:, None], y - cy
    h = torch.matmul(dx.transpose(1, 2), dy * ww[:, None])
    u, _, vt = torch.linalg.svd(h.cpu())
    d = torch.det(torch.matmul(u, vt)).sign()
    fix = torch.ones(x.shape[0], 3, dtype=torch.float64)
    fix[:, 2] = d
    r = torch.matmul(vt.transpose(1, 2) * fix[:, None, :], u.transpose(1, 2)).to(x.device)
    return cx, cy, r, dx, dy


def _frame_rmsd(x, y, align, want_grad=False):
    if not align:
        return (x - y).square().sum((1, 2)).div(y.shape[0]).sqrt(), None
    cx, cy, r, dx, dy = _kabsch(x, y)
    back = dx - torch.matmul(dy, r)  # x - cx - R^T (y - cy)
    v = back.square().sum((1, 2)).div(y.shape[0]).sqrt()
    return v, (back / (y.shape[0] * v)[:, None, None] if want_grad else None)


def _pair_exact(x, metric):
    F, n = x.shape[0], x.shape[1]
    xd = x.double()
    cen = xd.mean(1)
    c = xd - cen[:, None]
    g = c.square().sum((1, 2))
    b = c.permute(1, 0, 2).reshape(n, 3 * F)  # [atom][frame, component]
    out = torch.empty(F, F, dtype=torch.float64, device=x.device)
    rows = max(1, 4_000_000 // F)
    for i0 in range(0, F, rows):
        i1 = min(F, i0 + rows)
        h = torch.matmul(b[:, 3 * i0:3 * i1].t(), b).reshape(i1 - i0, 3, F, 3).permute(1, 3, 0, 2)
        e = g[i0:i1, None] + g[None]
        if metric == "nofit":
            d = (cen[i0:i1, None] - cen[None]).square().sum(2)
            ss = e - 2 * (h[0, 0] + h[1, 1] + h[2, 2]) + n * d
        else:
            ss = e - 2 * _top_root(h, 0.5 * e)
        out[i0:i1] = (ss.clamp_min(0) / n).sqrt()
    out.fill_diagonal_(0)
    return out


def _top_root(h, e0):
    """Largest eigenvalue of the quaternion key matrices of the 3x3 covariances h[a][b]: Newton's method down from the
    bound e0 on the characteristic polynomial t^4 + p t^2 + q t + r (Horn 1987; Theobald 2005), scaled by e0."""
    h = h / e0
    sxx, sxy, sxz, syx, syy, syz, szx, szy, szz = (h[a, b] for a in range(3) for b in range(3))
    k = [[sxx + syy + szz, syz - szy, szx - sxz, sxy - syx],
         [None, sxx - syy - szz, sxy + syx, szx + sxz],
         [None, None, syy - sxx - szz, syz + szy],
         [None, None, None, szz - sxx - syy]]
    p = -2 * h.square().sum((0, 1))
    det3 = (sxx * (syy * szz - syz * szy) - sxy * (syx * szz - syz * szx) + sxz * (syx * szy - syy * szx))
    q = -8 * det3
    m = lambda i, j: k[min(i, j)][max(i, j)]  # noqa: E731
    low = {(a, b): m(2, a) * m(3, b) - m(2, b) * m(3, a) for a in range(4) for b in range(a + 1, 4)}
    top = {(a, b): m(0, a) * m(1, b) - m(0, b) * m(1, a) for a in range(4) for b in range(a + 1, 4)}
    r = (top[0, 1] * low[2, 3] - top[0, 2] * low[1, 3] + top[0, 3] * low[1, 2]
         + top[1, 2] * low[0, 3] - top[1, 3] * low[0, 2] + top[2, 3] * low[0, 1])
    t = torch.ones_like(e0)
    for _ in range(60):
        f = ((t * t + p) * t + q) * t + r
        d = (4 * t * t + 2 * p) * t + q
        step = torch.where(d.abs() > 0, f / d, torch.zeros_like(f))
        t = t - step
        if float(step.abs().max()) < 1e-15:
            break
    return t * e0


def exact(case, seed):
    k = case["kind"]
    if k == "cluster":
        return None  # labels and indices are whole numbers
    d = _inputs(case, seed)
    if k == "batched":
        res = {"rmsd": [], "grad": []}
        for x, y in zip(d["coords"], d["ref"]):
            parts = [_frame_rmsd(x[f0:f0 + _rows(x.shape[1])].double(), y.double(), True, case["grad"])
                     for f0 in range(0, x.shape[0], _rows(x.shape[1]))]
            res["rmsd"].append(torch.cat([p[0] for p in parts]))
            if case["grad"]:
                res["grad"].append(torch.cat([p[1] for p in parts]))
        return res if case["grad"] else {"rmsd": res["rmsd"]}
    x = d["coords"][:, :, :3]
    if k == "pair":
        return _pair_exact(x, case["metric"])
    sel = slice(None) if d["sel"] is None else torch.from_numpy(d["sel"].astype(np.int64)).to(DEV)
    ref = d["ref"].double()
    y = ref[sel]
    step = _rows(case["atoms"])
    blocks = [x[f0:f0 + step].double() for f0 in range(0, x.shape[0], step)] if x.shape[1] * x.shape[0] < 5e7 else None
    block = (lambda f0: x[f0:f0 + step].double()) if blocks is None else (lambda f0: blocks[f0 // step])
    if k in ("plan", "frames"):
        return torch.cat([_frame_rmsd(block(f0)[:, sel], y, case["align"])[0] for f0 in range(0, x.shape[0], step)])
    if k in ("autograd", "value_grad"):
        v, g = [], torch.zeros(x.shape, dtype=torch.float64, device=DEV)
        for f0 in range(0, x.shape[0], step):
            b = block(f0)
            r, gr = _frame_rmsd(b[:, sel], y, True, True)
            v.append(r)
            g[f0:f0 + b.shape[0], sel] = gr
        return {"rmsd": torch.cat(v), "grad": g}
    rows, moved, per = [], [], []
    for f0 in range(0, x.shape[0], step):
        b = block(f0)
        cx, cy, r, _, _ = _kabsch(b[:, sel], y, d["w"])
        t = cy - torch.matmul(r, cx[:, :, None])[:, :, 0]
        at = torch.matmul(b, r.transpose(1, 2)) + t[:, None]
        if k == "superpose":
            rows.append(torch.cat([r.reshape(-1, 9), t], dim=1))
            moved.append(at)
        else:
            off = (at - ref).square().sum(2)
            n = off.shape[1]
            full = torch.nn.functional.pad(off, (0, -n % 10)).reshape(off.shape[0], -1, 10).sum(2)
            size = torch.full((full.shape[1],), 10.0, dtype=torch.float64, device=DEV)
            if n % 10:
                size[-1] = n % 10
            per.append((full / size).sqrt())
    if k == "superpose":
        return {"coords": torch.cat(moved), "transforms": torch.cat(rows)}
    return torch.cat(per)
