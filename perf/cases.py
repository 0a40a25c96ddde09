"""The work that programs built on stkfmm_b200 ask of it, as cases that can be timed.

Every case goes through a public entry point: the direct sum on host arrays, the
differentiable regularized Stokeslet, the FMM with its geometry set up once and
evaluated many times (an iterative solver), the FMM of a time step whose points
moved, the near field alone, and the no-slip wall.  The listed sizes are those of
the repository's benchmark and tests; draw() spreads over the ranges between them.

prepare() makes what a program holds before the call: points and values from the
seed, the FMM handle with its tree, and the far field's operators, which the
library builds at the first evaluation of a handle.  run() is one call.
"""
import math

import numpy as np
import torch

import stkfmm_b200 as S
from stkfmm_b200.autograd import UListPlan, stokes_regvel

KERNELS = {"LapPGrad": S.KERNEL.LapPGrad, "Stokes": S.KERNEL.Stokes, "RPY": S.KERNEL.RPY,
           "StokesRegVel": S.KERNEL.StokesRegVel, "PVel": S.KERNEL.PVel}
PRECISIONS = {"fp64": S.PRECISION.FP64, "mixed": S.PRECISION.MIXED}
PBCS = {"none": S.PAXIS.NONE, "pxy": S.PAXIS.PXY, "pxyz": S.PAXIS.PXYZ}
# operations of one (target, source) pair, without the reciprocal square root
PAIR_FLOPS = {("LapPGrad", "sl"): 17, ("LapPGrad", "dl"): 30, ("LapPGrad", "both"): 33, ("Stokes", "sl"): 24,
              ("RPY", "sl"): 43, ("StokesRegVel", "sl"): 28, ("PVel", "sl"): 29, ("PVel", "dl"): 38,
              ("PVel", "both"): 52}


def listed():
    return [
        # a direct sum of a few hundred points: a check, a small cluster; latency is all of it
        {"name": "kernel_stokes_host_small", "do": "kernel", "kernel": "Stokes", "layer": "sl", "nsrc": 400,
         "ntrg": 300, "precision": "fp64"},
        # the direct sum used to validate an FMM or for a boundary of this size
        {"name": "kernel_pvel_dl_host_30k", "do": "kernel", "kernel": "PVel", "layer": "dl", "nsrc": 20011,
         "ntrg": 30011, "precision": "fp64"},
        # value and gradient of a loss through the all-pairs regularized Stokeslet
        {"name": "grad_regvel_direct_4k", "do": "grad", "plan": "direct", "n": 4096, "max_pts": 0,
         "precision": "fp64"},
        # the same through the near field of an octree, forward and adjoint passes
        {"name": "grad_regvel_ulist_262k", "do": "grad", "plan": "ulist", "n": 262144, "max_pts": 256,
         "precision": "fp64"},
        # the smallest FMM that has levels: launches and host work of the whole chain
        {"name": "fmm_lappgrad_host_4k", "do": "fmm", "kernel": "LapPGrad", "layer": "sl", "pbc": "none",
         "points": "clustered", "n": 4000, "p": 8, "max_pts": 64, "precision": "fp64", "arrays": "host"},
        # Stokeslets of an ordinary boundary-integral solve
        {"name": "fmm_stokes_32k", "do": "fmm", "kernel": "Stokes", "layer": "sl", "pbc": "none",
         "points": "uniform", "n": 32768, "p": 8, "max_pts": 128, "precision": "fp64", "arrays": "device"},
        # the near field alone (U list, single and double layer) of strongly clustered points
        {"name": "near_lappgrad_1m", "do": "near", "kernel": "LapPGrad", "layer": "both", "pbc": "none",
         "points": "clustered", "n": 1048576, "p": 10, "max_pts": 256, "precision": "fp64", "arrays": "device"},
        # the whole FMM of the same points, mixed precision
        {"name": "fmm_lappgrad_1m_mixed", "do": "fmm", "kernel": "LapPGrad", "layer": "both", "pbc": "none",
         "points": "clustered", "n": 1048576, "p": 10, "max_pts": 256, "precision": "mixed", "arrays": "device"},
        # a triply periodic suspension; the far field is most of it
        {"name": "fmm_rpy_pxyz_2m", "do": "fmm", "kernel": "RPY", "layer": "sl", "pbc": "pxyz",
         "points": "uniform", "n": 2097152, "p": 8, "max_pts": 256, "precision": "fp64", "arrays": "device"},
        # surface points of many spheres, doubly periodic, single and double layer
        {"name": "fmm_pvel_pxy_spheres_524k", "do": "fmm", "kernel": "PVel", "layer": "both", "pbc": "pxy",
         "points": "spheres", "n": 524288, "p": 10, "max_pts": 256, "precision": "fp64", "arrays": "device"},
        # particles above a no-slip wall
        {"name": "wall_stokes_131k", "do": "wall", "kernel": "Stokes", "n": 131072, "p": 8, "max_pts": 256,
         "precision": "fp64"},
        # one step of a simulation: the points moved, so tree and lists are set up again (host arrays)
        {"name": "step_stokes_100k_mixed", "do": "step", "kernel": "Stokes", "layer": "sl", "pbc": "none",
         "points": "uniform", "n": 100000, "p": 8, "max_pts": 256, "precision": "mixed", "arrays": "host"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["kernel", "grad", "fmm", "fmm", "fmm", "periodic", "near", "wall", "step"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    if do == "kernel":
        kernel, layer = rng.choice([("Stokes", "sl"), ("LapPGrad", "sl"), ("LapPGrad", "dl"), ("RPY", "sl"),
                                    ("StokesRegVel", "sl"), ("PVel", "sl"), ("PVel", "dl")])
        return {"do": do, "kernel": kernel, "layer": layer, "nsrc": _log(rng, 100, 50000),
                "ntrg": _log(rng, 100, 50000), "precision": precision}
    if do == "grad":
        if rng.random() < 0.5:
            return {"do": do, "plan": "direct", "n": _log(rng, 300, 16000), "max_pts": 0, "precision": precision}
        return {"do": do, "plan": "ulist", "n": _log(rng, 5000, 500000), "max_pts": rng.choice([64, 128, 256]),
                "precision": precision}
    if do == "wall":
        return {"do": do, "kernel": rng.choice(["Stokes", "RPY"]), "n": _log(rng, 4000, 250000), "p": 8,
                "max_pts": rng.choice([128, 256]), "precision": precision}
    kernel, layer = rng.choice([("LapPGrad", "sl"), ("LapPGrad", "both"), ("Stokes", "sl"), ("RPY", "sl"),
                                ("StokesRegVel", "sl"), ("PVel", "sl"), ("PVel", "both")])
    case = {"do": do, "kernel": kernel, "layer": layer, "pbc": "none", "points": rng.choice(["uniform", "clustered"]),
            "n": _log(rng, 2000, 500000), "p": 8, "max_pts": rng.choice([64, 128, 256]), "precision": precision,
            "arrays": rng.choice(["host", "device", "device"])}
    if kernel == "LapPGrad":
        case["p"] = rng.choice([8, 10])
    if do == "periodic":
        case.update(do="fmm", pbc=rng.choice(["pxy", "pxyz"]), points=rng.choice(["uniform", "spheres"]),
                    n=_log(rng, 8000, 1000000), max_pts=rng.choice([128, 256]))
    elif do == "step":
        case.update(n=_log(rng, 2000, 60000), arrays="host")
    elif do == "near":
        case["n"] = _log(rng, 5000, 1000000)
    if case["points"] == "clustered":
        case["max_pts"] = max(case["max_pts"], 128)
    return case


# ------------------------------------------------------------------ inputs ----
def _points(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "clustered":  # 64 Gaussian clusters: very uneven leaves
        centres = rng.uniform(0.1, 0.9, size=(64, 3))
        pts = centres[rng.integers(0, 64, size=n)] + rng.normal(0.0, 0.02, size=(n, 3))
        return np.clip(pts, 0.0, np.nextafter(1.0, 0.0))
    if kind == "spheres":  # surfaces of spheres of radius 0.01, about 1024 points each
        nsph = max(1, n // 1024)
        centres = np.concatenate([rng.uniform(0.05, 0.95, (nsph, 2)), rng.uniform(0.05, 0.5, (nsph, 1))], axis=1)
        u = rng.normal(size=(n, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        return centres[np.arange(n) % nsph] + 0.01 * u
    return rng.random((n, 3))


def _values(kernel, layer, n, seed, periodic):
    """Single- and double-layer values (None where the case has no such layer)."""
    rng = np.random.default_rng([seed, 1])
    sl = dl = None
    if layer in ("sl", "both"):
        if kernel == "LapPGrad":
            sl = rng.uniform(-0.5, 0.5, size=(n, 1))
        else:
            sl = rng.normal(size=(n, 3))
        if periodic:
            sl -= sl.mean(0)  # a periodic sum wants neutral sources
        if kernel == "RPY":
            sl = np.concatenate([sl, rng.uniform(1e-4, 5e-4, (n, 1))], axis=1)
        elif kernel == "StokesRegVel":
            sl = np.concatenate([sl, np.full((n, 1), 1e-3)], axis=1)
        elif kernel == "PVel":
            sl = np.concatenate([sl, np.zeros((n, 1))], axis=1)
    if layer in ("dl", "both"):
        dl = rng.normal(size=(n, 3 if kernel == "LapPGrad" else 9))
        if kernel == "PVel" and periodic:
            dl[:, [0, 4, 8]] -= (dl[:, 0] + dl[:, 4] + dl[:, 8]).mean() / 3
    return sl, dl


_operators = {}


def _keep_operators(kernel, p, pbc):
    """A small handle per configuration, kept as a program keeps its FMM object: the
    library's level-independent operators live as long as one handle that uses them."""
    key = (kernel, p, pbc)
    if key not in _operators:
        K = KERNELS[kernel]
        fmm = S.Stk3DFMM(p, 64, PBCS[pbc], K)
        fmm.set_box(np.zeros(3), 1.0)
        pts = np.random.default_rng(0).random((256, 3))
        fmm.set_points(pts, pts, None)
        fmm.setup_tree(K)
        sd, _, td = S.get_kernel_dimension(K)
        fmm.evaluate_fmm(K, np.ones((256, sd)), np.zeros((256, td)), None)
        _operators[key] = fmm
    return _operators[key]


def _make_fmm(case, pts, dl):
    K = KERNELS[case["kernel"]]
    fmm = S.Stk3DFMM(case["p"], case["max_pts"], PBCS[case["pbc"]], K, PRECISIONS[case["precision"]])
    fmm.set_box(np.zeros(3), 1.0)
    fmm.set_points(pts, pts, pts if dl is not None else None)
    fmm.setup_tree(K)
    return fmm


def _gpu(a):
    return None if a is None else torch.as_tensor(a, device="cuda")


def prepare(case, seed):
    do = case["do"]
    s = {"case": case}
    if do == "kernel":
        s["src"] = _points("uniform", case["nsrc"], seed)
        s["trg"] = _points("uniform", case["ntrg"], seed + 7919)
        sl, dl = _values(case["kernel"], case["layer"], case["nsrc"], seed, False)
        s["val"] = sl if dl is None else dl
        return s
    if do == "grad":
        n = case["n"]
        pts = _points("uniform", n, seed)
        rng = np.random.default_rng([seed, 2])
        s["x"] = _gpu(pts).requires_grad_(True)
        s["v"] = _gpu(np.concatenate([rng.normal(size=(n, 3)), np.full((n, 1), 1e-3)], axis=1)).requires_grad_(True)
        s["w"] = _gpu(rng.normal(size=(n, 3)))
        s["plan"] = UListPlan(pts, max_pts=case["max_pts"]) if case["plan"] == "ulist" else None
        if s["plan"] is not None:
            s["plan"].pairs()  # uploads the list
        return s
    if do == "wall":
        K = KERNELS[case["kernel"]]
        _keep_operators("Stokes", case["p"], "none")
        _keep_operators("LapPGrad", case["p"], "none")
        pts, val = _wall_inputs(case, seed)
        s["fmm"] = S.StkWallFMM(case["p"], case["max_pts"], S.PAXIS.NONE, K, PRECISIONS[case["precision"]])
        s["fmm"].set_box(np.zeros(3), 1.0)
        s["fmm"].set_points(pts, pts, None)
        s["fmm"].setup_tree(K)
        s["sl"], s["dl"] = _gpu(val), None
    else:
        pts = _points(case["points"], case["n"], seed)
        sl, dl = _values(case["kernel"], case["layer"], case["n"], seed, case["pbc"] != "none")
        if do != "near":
            _keep_operators(case["kernel"], case["p"], case["pbc"])
        s["fmm"] = _make_fmm(case, pts, dl)
        s["pts"] = pts
        s["sl"], s["dl"] = (sl, dl) if case["arrays"] == "host" else (_gpu(sl), _gpu(dl))
    td = S.get_kernel_dimension(KERNELS[case["kernel"]])[2]
    if case.get("arrays") == "host":
        s["out"] = np.zeros((case["n"], td))
    else:
        s["out"] = torch.zeros((case["n"], td), dtype=torch.float64, device="cuda")
        s["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()
    run(s)  # the first evaluation of a handle lays out the far field of its tree
    return s


def _wall_inputs(case, seed):
    pts = _points("clustered", case["n"], seed)
    pts[:, 2] = 0.01 + 0.48 * np.minimum(pts[:, 2], 0.999)
    pts[:, :2] = np.minimum(pts[:, :2], 0.999)
    sl, _ = _values(case["kernel"], "sl", case["n"], seed, False)
    return pts, sl


# -------------------------------------------------------------------- runs ----
def run(s):
    case = s["case"]
    do = case["do"]
    if do == "kernel":
        K = KERNELS[case["kernel"]]
        out = np.zeros((case["ntrg"], S.get_kernel_dimension(K)[2]))
        return S.evaluate_kernel(K, S.PPKERNEL.DLS2T if case["layer"] == "dl" else S.PPKERNEL.SLS2T, s["src"],
                                 s["val"], s["trg"], out, PRECISIONS[case["precision"]])
    if do == "grad":
        x, v = s["x"], s["v"]
        x.grad = v.grad = None
        u = stokes_regvel(x, v, plan=s["plan"], precision=PRECISIONS[case["precision"]])
        u.backward(s["w"])
        return {"u": u.detach(), "x": x.grad, "v": v.grad}
    K = KERNELS[case["kernel"]]
    fmm = s["fmm"]
    if do == "step":
        fmm.set_points(s["pts"], s["pts"], s["pts"] if s["dl"] is not None else None)
        fmm.setup_tree(K)
    if case.get("arrays") == "host":
        s["out"][:] = 0.0
        evaluate = fmm.evaluate_near if do == "near" else fmm.evaluate_fmm
        return evaluate(K, s["sl"], s["out"], s["dl"]).copy()
    stream = s["stream"]
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        s["out"].zero_()
        if do == "wall":
            fmm.evaluate_fmm_device(K, s["sl"].data_ptr(), s["out"].data_ptr(), stream.cuda_stream)
        else:
            evaluate = fmm.evaluate_near_device if do == "near" else fmm.evaluate_fmm_device
            evaluate(K, s["sl"].data_ptr(), s["out"].data_ptr(), s["dl"].data_ptr() if s["dl"] is not None else 0,
                     stream.cuda_stream)
    torch.cuda.current_stream().wait_stream(stream)
    return s["out"]


def work(case):
    """Bytes: coordinates and values read once, outputs written once.  Flops: of every
    pair of a direct sum; of an FMM the near field's alone, with leaves half full and
    27 neighbours (the far field's count is a choice of method)."""
    if case["do"] == "kernel":
        K = KERNELS[case["kernel"]]
        sd, dd, td = (int(v) for v in S.get_kernel_dimension(K))
        return {"bytes": 8.0 * (case["nsrc"] * (3 + (dd if case["layer"] == "dl" else sd)) + case["ntrg"] * (3 + td)),
                "flops": float(case["nsrc"]) * case["ntrg"] * PAIR_FLOPS[case["kernel"], case["layer"]]}
    n = float(case["n"])
    if case["do"] == "grad":
        # x, v and the upstream gradient in; u and the gradients of x and v out; three passes over the pairs
        pairs = n * n if case["plan"] == "direct" else n * min(n, 27 * case["max_pts"] / 2)
        return {"bytes": 8.0 * n * (3 + 4 + 3 + 3 + 3 + 4), "flops": 3 * pairs * PAIR_FLOPS["StokesRegVel", "sl"]}
    sd, dd, td = (int(v) for v in S.get_kernel_dimension(KERNELS[case["kernel"]]))
    layer = case.get("layer", "sl")
    pairs = n * min(n, 27 * case["max_pts"] / 2)
    dims = (sd if layer != "dl" else 0) + (dd if layer != "sl" else 0)
    return {"bytes": 8.0 * n * (3 + dims + td), "flops": pairs * PAIR_FLOPS[case["kernel"], layer]}


# ------------------------------------------------------------- exact values ----
def _pair_sum(kernel, src, sl, dl, trg):
    """sum over all sources at every target in FP64, plain torch on the GPU."""
    n = len(src)
    sx, sy, sz = src.T.contiguous()
    rows = max(1, (1 << 25) // n)
    out = []
    for a in range(0, len(trg), rows):
        t = trg[a:a + rows]
        dx, dy, dz = t[:, 0:1] - sx, t[:, 1:2] - sy, t[:, 2:3] - sz
        r2 = dx * dx + dy * dy + dz * dz
        if kernel == "StokesRegVel":
            e2 = sl[:, 3] ** 2
            R3 = (r2 + e2) ** -1.5
            fr = (sl[:, 0] * dx + sl[:, 1] * dy + sl[:, 2] * dz) * R3
            al = (r2 + 2 * e2) * R3
            out.append(torch.stack([al @ sl[:, k] + (fr * d).sum(1) for k, d in enumerate((dx, dy, dz))], 1)
                       / (8 * math.pi))
            continue
        ri = torch.where(r2 > 0, r2, math.inf) ** -0.5
        ri2 = ri * ri
        ri3 = ri2 * ri
        D = (dx, dy, dz)
        if kernel == "LapPGrad":
            res = 0.0
            if sl is not None:
                w = ri3 * sl[:, 0]
                res = torch.stack([ri @ sl[:, 0]] + [-(w * d).sum(1) for d in D], 1)
            if dl is not None:
                dr = (dl[:, 0] * dx + dl[:, 1] * dy + dl[:, 2] * dz) * ri2
                res = res + torch.stack([(dr * ri).sum(1)]
                                        + [ri3 @ dl[:, k] - 3 * (dr * ri3 * d).sum(1) for k, d in enumerate(D)], 1)
            out.append(res / (4 * math.pi))
            continue
        res = 0.0
        if sl is not None:
            fr = sl[:, 0] * dx + sl[:, 1] * dy + sl[:, 2] * dz
            u = [ri @ sl[:, k] + (fr * ri3 * d).sum(1) for k, d in enumerate(D)]
            if kernel == "RPY":  # (1 + b^2/6 lap) G f and lap G f
                third = sl[:, 3] ** 2 / 3
                fr3 = -3 * fr * ri2 * ri3
                C = [ri3 * sl[:, k] + fr3 * d for k, d in enumerate(D)]
                u = [v + c @ third for v, c in zip(u, C)] + [2 * c.sum(1) for c in C]
            if kernel == "PVel":
                u = [2 * (fr * ri3).sum(1)] + [v - (sl[:, 3] * ri3 * d).sum(1) for v, d in zip(u, D)]
            res = torch.stack(u, 1)
        if dl is not None:
            m = sum(dl[:, 3 * i + j] * D[i] * D[j] for i in range(3) for j in range(3)) * ri2
            m = -3 * m * ri3
            tr = dl[:, 0] + dl[:, 4] + dl[:, 8]
            res = res + torch.stack([2 * (m.sum(1) + ri3 @ tr)] + [(m * d).sum(1) for d in D], 1)
        out.append(res / (8 * math.pi))
    return torch.cat(out)


def _wall_sum(pts, f):
    """Stokeslets above a no-slip wall at z = 0: Blake's image tensor."""
    n = len(pts)
    u = _pair_sum("Stokes", pts, f, None, pts)
    img = pts * pts.new_tensor([1.0, 1.0, -1.0])
    u -= _pair_sum("Stokes", img, f, None, pts)
    g = f * f.new_tensor([1.0, 1.0, -1.0])
    h = pts[:, 2]
    rows = max(1, (1 << 25) // n)
    for a in range(0, n, rows):
        t = pts[a:a + rows]
        R = [t[:, k:k + 1] - img[:, k] for k in range(3)]
        ri2 = 1.0 / (R[0] * R[0] + R[1] * R[1] + R[2] * R[2])
        ri3 = ri2 * ri2.sqrt() * (2 * h)
        gr = g[:, 0] * R[0] + g[:, 1] * R[1] + g[:, 2] * R[2]
        away = ri3 * (h - R[2])
        back = 3 * gr * ri2 * (R[2] - h) * ri3 - g[:, 2] * ri3
        add = [away @ g[:, k] + (back * R[k]).sum(1) for k in range(3)]
        add[2] = add[2] + (gr * ri3).sum(1)
        u[a:a + rows] += torch.stack(add, 1) / (8 * math.pi)
    return u


def exact(case, seed):
    do = case["do"]
    if do == "kernel":
        sl, dl = _values(case["kernel"], case["layer"], case["nsrc"], seed, False)
        u = _pair_sum(case["kernel"], _gpu(_points("uniform", case["nsrc"], seed)), _gpu(sl), _gpu(dl),
                      _gpu(_points("uniform", case["ntrg"], seed + 7919)))
        return u.cpu().numpy()
    if do == "grad":
        if case["plan"] != "direct":
            return None  # a sum over the library's own octree lists
        x = _gpu(_points("uniform", case["n"], seed))
        rng = np.random.default_rng([seed, 2])
        v = _gpu(np.concatenate([rng.normal(size=(case["n"], 3)), np.full((case["n"], 1), 1e-3)], axis=1))
        return _grad_exact(x, v, _gpu(rng.normal(size=(case["n"], 3))))
    if do == "near" or case.get("pbc", "none") != "none":
        return None  # the library's own lists; an Ewald sum over all of these points takes minutes
    if case["n"] > (150000 if do == "wall" else 300000):
        return None  # over 20 seconds of direct sums
    if do == "wall":
        if case["kernel"] != "Stokes":
            return None  # no closed image tensor in plain terms: six sub-sums of the library's own composition
        pts, f = _wall_inputs(case, seed)
        return _wall_sum(_gpu(pts), _gpu(f))
    pts = _gpu(_points(case["points"], case["n"], seed))
    sl, dl = _values(case["kernel"], case["layer"], case["n"], seed, False)
    u = _pair_sum(case["kernel"], pts, _gpu(sl), _gpu(dl), pts)
    return u.cpu().numpy() if case["arrays"] == "host" else u


def _grad_exact(x, v, w):
    """Velocity and the gradients of sum(w . u) for x (as sources and as targets) and v."""
    n = len(x)
    gx, gv = torch.zeros_like(x), torch.zeros_like(v)
    u = _pair_sum("StokesRegVel", x, v, None, x)
    rows = max(1, (1 << 24) // n)
    e = v[:, 3]
    for a in range(0, n, rows):
        t, wt = x[a:a + rows], w[a:a + rows]
        R = [t[:, k:k + 1] - x[:, k] for k in range(3)]
        r2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2]
        q = 1.0 / (r2 + e * e)
        q3 = q * q.sqrt() / (8 * math.pi)
        wf = wt @ v[:, :3].T
        fr = sum(v[:, k] * R[k] for k in range(3))
        wr = sum(wt[:, k:k + 1] * R[k] for k in range(3))
        al = (r2 + 2 * e * e) * q3
        m = ((r2 + 2 * e * e) * wf + wr * fr) * q
        c = (2 * wf - 3 * m) * q3
        gv[:, 3] += (e * (4 * wf - 3 * m) * q3).sum(0)
        for k in range(3):
            gv[:, k] += al.T @ wt[:, k] + (wr * q3 * R[k]).sum(0)
            F = c * R[k] + wt[:, k:k + 1] * fr * q3 + v[:, k] * wr * q3
            gx[a:a + rows, k] += F.sum(1)
            gx[:, k] -= F.sum(0)
    return {"u": u, "x": gx, "v": gv}
