"""The work that users of this framework have it do, as timed cases.

Kinds of a case, each through the public entry point named:

  solve     computeCovariances of one reconstruction: on device-resident arrays
            (compute_covariances_device) or on the host arrays of the drop-in
            boundary (compute_covariances)
  batch     many uneven reconstructions in one call (Batch.compute, host arrays)
  inverse   the SPD inverse building block (dense_inverse_device)
  pinv      the PSD pseudo-inverse of the SVD algorithms (pinv_psd_device)
  product   the int8-sliced symmetric product (gemm_mixed_device)
  eigen     eigen-decompositions of covariance blocks behind the Uncertainty
            accessors (unc_block_eigen_device)
  jacobian  the Jacobian of a scene (unc_jacobian_device)

Scenes have the distributions of uncertaintyte_b200.scenes: cameras on a sphere
cap looking at the origin, points in a box, 2 + Poisson(views) observations per
point among the cameras nearest to it in azimuth, two of them half that window
apart (pipelines drop points of a small triangulation angle before this step).
They are made here with torch, so that the inputs depend on the seed alone; how
many cameras see each point is the same for every seed of a case, so that all its
inputs have one size.

lam is the regulariser of the Taylor inverse; -1 is the automatic one. A .jacob
file carries its own value. Small scenes take the automatic one; larger scenes
a given one of about 1e-5, since at the automatic value (4.7e-9 for 2000
cameras) the rounding of the Schur complement, divided by lam, already moves the
results of a 64-bit computation in the eighth digit.
"""
import ctypes
import math

import numpy as np
import torch

from uncertaintyte_b200 import native, scenes
from uncertaintyte_b200.jacob import Jacobian

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _solve(name, cams, points_per_cam, views, window, precision, lam, host):
    return {"name": name, "kind": "solve", "cams": cams, "points_per_cam": points_per_cam, "views": views,
            "window": window, "precision": precision, "lam": lam, "host": host}


def listed():
    return [
        # the smallest reconstruction, called as the reference's users call it: latency and launches
        _solve("solve_small_host", 10, 50, 4.0, 10, "fp64", -1.0, True),
        # a 200-camera / 50k-point scene resident on the device, default and plain FP64 products
        _solve("solve_medium_mixed", 200, 250, 5.0, 200, "mixed", 1e-5, False),
        _solve("solve_medium_fp64", 200, 250, 5.0, 200, "fp64", 1e-5, False),
        # the headline scene: 2000 cameras, 500k points, about 3.5M observations
        _solve("solve_large_mixed", 2000, 250, 5.0, 96, "mixed", 1e-5, False),
        # uneven small reconstructions packed into one call, as the request server packs them
        {"name": "batch_uneven", "kind": "batch", "scenes": 24, "median": 60.0, "sigma": 1.0, "low": 8, "high": 200,
         "points_per_cam": 150, "views": 4.0, "precision": "mixed", "lam": 1e-5},
        # the dense inverse alone: a mid-sized odd order, and one past the tile-task limit
        {"name": "inverse_1351", "kind": "inverse", "n": 1351},
        {"name": "inverse_5401", "kind": "inverse", "n": 5401},
        # the SVD algorithms' inverse step on the full J^T J of a small scene (9 * 10 + 3 * 500)
        {"name": "pinv_1590", "kind": "pinv", "n": 1590, "remove": 7},
        # one Taylor product of a 400-camera scene, five slices
        {"name": "product_3600", "kind": "product", "n": 3600, "slices": 5},
        # accessors: every point's 3 x 3 block of the headline scene, every camera's 9 x 9 block of a medium one
        {"name": "eigen_points", "kind": "eigen", "blocks": 500_000, "params": 3, "offset": 0, "dim": 3, "vectors": True},
        {"name": "eigen_cameras", "kind": "eigen", "blocks": 200, "params": 9, "offset": 0, "dim": 9, "vectors": True},
        # the headline scene's Jacobian from its cameras and points
        {"name": "jacobian_large", "kind": "jacobian", "cams": 2000, "points_per_cam": 250, "views": 5.0, "window": 96},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "inverse", "inverse", "pinv", "product", "eigen", "jacobian"])
    if kind == "solve":
        cams = _log_int(rng, 6, 900)
        small = cams <= 24
        return {"kind": kind, "cams": cams, "points_per_cam": _log_int(rng, 40, 250),
                "views": rng.choice([3.0, 4.0, 5.0]), "window": rng.choice([24, 48, 96, cams]),
                "precision": rng.choice(["mixed", "mixed", "fp64"]),
                "lam": -1.0 if small else 10.0 ** rng.uniform(-5.2, -4.3), "host": small or rng.random() < 0.25}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 24), "median": rng.uniform(20.0, 80.0), "sigma": 1.0, "low": 8,
                "high": rng.randint(60, 200), "points_per_cam": rng.randint(60, 150), "views": 4.0,
                "precision": "mixed", "lam": 10.0 ** rng.uniform(-5.2, -4.3)}
    if kind == "inverse":
        return {"kind": kind, "n": _log_int(rng, 20, 6000)}
    if kind == "pinv":
        return {"kind": kind, "n": _log_int(rng, 60, 2200), "remove": rng.choice([3, 7, 7])}
    if kind == "product":
        return {"kind": kind, "n": _log_int(rng, 60, 6000), "slices": rng.choice([3, 4, 5, 5])}
    if kind == "eigen":
        params = rng.choice([3, 3, 9])
        sub = params == 9 and rng.random() < 0.5  # the camera centre
        return {"kind": kind, "blocks": _log_int(rng, 10, 500_000 if params == 3 else 4000), "params": params,
                "offset": 3 if sub else 0, "dim": 3 if sub else params, "vectors": rng.random() < 0.7}
    cams = _log_int(rng, 10, 1800)
    return {"kind": kind, "cams": cams, "points_per_cam": _log_int(rng, 40, 250), "views": rng.choice([3.0, 4.0, 5.0]),
            "window": rng.choice([24, 48, 96])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(g, shape, lo, hi):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device=DEV, dtype=F64)


def _normal(g, shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=F64)


def _look_at_angle_axis(centers):
    """Angle-axis of the world-to-camera rotations whose +z axis points at the origin."""
    z = -centers / centers.norm(dim=1, keepdim=True)
    up = torch.tensor([0.0, 0.0, 1.0], device=DEV, dtype=F64).expand_as(z)
    x = torch.linalg.cross(up, z)
    x = x / x.norm(dim=1, keepdim=True)
    y = torch.linalg.cross(z, x)
    R = torch.stack([x, y, z], dim=1)
    angle = torch.arccos(((R.diagonal(dim1=1, dim2=2).sum(1) - 1) / 2).clamp(-1.0, 1.0))
    w = torch.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1]], dim=1)
    return w * (angle / (2 * torch.sin(angle)))[:, None]


def _scene(cams, points_per_cam, views, window, seed):
    """(cameras (C, 9), points (P, 3), observation camera ids, observation point ids), observations by point."""
    g = _generator(seed)
    C, P = int(cams), int(cams) * int(points_per_cam)
    theta = torch.arccos(_uniform(g, (C,), math.cos(math.radians(60)), math.cos(math.radians(15))))
    phi = _uniform(g, (C,), 0.0, 2 * math.pi)
    centers = 20 * torch.stack([torch.sin(theta) * torch.cos(phi), torch.sin(theta) * torch.sin(phi),
                                torch.cos(theta)], dim=1)
    camera = torch.cat([_look_at_angle_axis(centers), centers, _uniform(g, (C, 1), 800.0, 1200.0),
                        1e-2 * _normal(g, (C, 2))], dim=1)
    box = torch.tensor([2.0, 2.0, 1.0], device=DEV, dtype=F64)
    points = _uniform(g, (P, 3), -1.0, 1.0) * box
    w = min(int(window), C)
    counts = (2 + torch.poisson(torch.full((P,), float(views), device=DEV), generator=_generator(0)).long()).clamp(max=w)
    azimuth, order = torch.sort(phi)
    at = torch.searchsorted(azimuth, torch.remainder(torch.atan2(points[:, 1], points[:, 0]), 2 * math.pi))
    start = (at - w // 2).clamp(0, C - w)
    most = int(counts.max())
    keys = torch.rand((P, w), generator=g, device=DEV, dtype=F64)
    pair = torch.randint(w - w // 2, (P, 1), generator=g, device=DEV)
    keys.scatter_(1, torch.cat([pair, pair + w // 2], dim=1), 2.0)  # the two that every point has
    chosen = keys.topk(most, dim=1).indices
    seen = order[start[:, None] + chosen]
    taken = torch.arange(most, device=DEV)[None, :] < counts[:, None]
    seen = torch.where(taken, seen, C).sort(dim=1).values  # ascending cameras, unused places last
    obs_pt = torch.repeat_interleave(torch.arange(P, device=DEV), counts)
    return camera, points, seen[taken].to(torch.int32), obs_pt.to(torch.int32)


def _skew(v):
    zero = torch.zeros_like(v[:, 0])
    return torch.stack([zero, -v[:, 2], v[:, 1], v[:, 2], zero, -v[:, 0], -v[:, 1], v[:, 0], zero], dim=1).view(-1, 3, 3)


def _observation_blocks(camera, points, obs_cam, obs_pt):
    """The analytic 2 x 12 reprojection blocks (9 camera, 3 point columns), (n, 2, 12)."""
    oc, op = obs_cam.long(), obs_pt.long()
    aa = camera[:, :3]
    t = aa.norm(dim=1)[:, None, None]
    K = _skew(aa)
    K2 = K @ K
    eye = torch.eye(3, device=DEV, dtype=F64)
    R = (eye + torch.sin(t) / t * K + (1 - torch.cos(t)) / t ** 2 * K2)[oc]
    Jr = (eye - (1 - torch.cos(t)) / t ** 2 * K + (t - torch.sin(t)) / t ** 3 * K2)[oc]
    f, k1, k2 = (camera[oc, i] for i in (6, 7, 8))
    ray = points[op] - camera[oc, 3:6]
    p = torch.einsum("nij,nj->ni", R, ray)
    z = p[:, 2]
    x = p[:, :2] / z[:, None]
    r2 = (x * x).sum(1)
    d = 1 + k1 * r2 + k2 * r2 * r2
    grad = k1 + 2 * k2 * r2
    M = f[:, None, None] * (d[:, None, None] * eye[:2, :2] + 2 * grad[:, None, None] * x[:, :, None] * x[:, None, :])
    Q = torch.cat([eye[:2, :2].expand(len(z), 2, 2), -x[:, :, None]], dim=2) / z[:, None, None]
    to_point = M @ Q
    out = torch.empty((len(z), 2, 12), device=DEV, dtype=F64)
    out[:, :, 9:12] = to_point @ R
    out[:, :, 0:3] = -out[:, :, 9:12] @ _skew(ray) @ Jr
    out[:, :, 3:6] = -out[:, :, 9:12]
    out[:, :, 6] = d[:, None] * x
    out[:, :, 7] = (f * r2)[:, None] * x
    out[:, :, 8] = (f * r2 * r2)[:, None] * x
    return out


def _columns(C, obs_cam, obs_pt):
    nine, three = torch.arange(9, device=DEV), torch.arange(3, device=DEV)
    row = torch.cat([9 * obs_cam.long()[:, None] + nine, 9 * C + 3 * obs_pt.long()[:, None] + three], dim=1)
    return row[:, None, :].expand(-1, 2, -1).reshape(-1).to(torch.int32)


def _reconstruction(cams, points_per_cam, views, window, lam, seed, host):
    """A Jacobian in the reference's layout, its arrays on the host (numpy) or on the device (torch)."""
    camera, points, oc, op = _scene(cams, points_per_cam, views, window, seed)
    n, C, P = len(oc), len(camera), len(points)
    values = _observation_blocks(camera, points, oc, op).reshape(-1)
    cols = _columns(C, oc, op)
    rows = (12 * torch.arange(2 * n + 1, device=DEV)).to(torch.int32)
    fixed = scenes.farthest_triple(points.cpu().numpy())
    if host:
        rows, cols, values = rows.cpu().numpy(), cols.cpu().numpy(), values.cpu().numpy()
    return Jacobian(C, 9, P, n, 2 * n, 9 * C + 3 * P, rows, cols, values, lam, fixed, algorithm=2, epsilon=1e-10,
                    svd_remove_n=7)


def _batch_cameras(case, seed):
    rng = np.random.default_rng(int(seed))
    c = np.round(case["median"] * np.exp(case["sigma"] * rng.standard_normal(case["scenes"])))
    return np.clip(c, case["low"], case["high"]).astype(int)


def _batch_jacobians(case, seed):
    return [_reconstruction(c, case["points_per_cam"], case["views"], 48, case["lam"], 1000 * int(seed) + i, True)
            for i, c in enumerate(_batch_cameras(case, 0))]  # one set of sizes: seeds change the scenes


def _spd(n, seed, low, high, null=0):
    """(matrix, orthogonal Q, eigenvalues): log-uniform spectrum in [low, high] after `null` zeros."""
    g = _generator(seed)
    Q, _ = torch.linalg.qr(_normal(g, (n, n)))
    w = torch.exp(_uniform(g, (n,), math.log(low), math.log(high)))
    w[:null] = 0.0
    A = (Q * w) @ Q.T
    return (A + A.T) / 2, Q, w


def _padded(A):
    """The columns of a symmetric A at a leading dimension that is a multiple of 8."""
    n = len(A)
    out = torch.zeros((n, (n + 7) // 8 * 8), device=DEV, dtype=F64)
    out[:, :n] = A
    return out


def _product_operands(case, seed):
    X, _, _ = _spd(case["n"], seed, 1e-3, 1.0)
    return _padded(X @ X), _padded(X)


def _eigen_blocks(case, seed):
    """Covariance blocks: positive definite, their axes' lengths a factor of ten to some hundred apart."""
    g = _generator(seed)
    n, p = case["blocks"], case["params"]
    B = _normal(g, (n, p, p)) * torch.exp(_uniform(g, (n, 1, p), -3.0, 3.0))
    return B @ B.transpose(1, 2)


_handles = {}


def _context():
    """The context that a program keeps for all its reconstructions."""
    if "context" not in _handles:
        _handles["context"] = native.Context(0)
    return _handles["context"]


def _batch():
    if "batch" not in _handles:
        _handles["batch"] = native.Batch(0)
    return _handles["batch"]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "solve":
        jac = _reconstruction(case["cams"], case["points_per_cam"], case["views"], case["window"], case["lam"], seed,
                              case["host"])
        state.update(jac=jac, context=_context())
        if not case["host"]:
            state.update(options=native.make_options(jac, precision=case["precision"]),
                         cam=torch.zeros(jac.num_cams * 45, device=DEV, dtype=F64),
                         pt=torch.zeros(jac.num_points * 6, device=DEV, dtype=F64))
    elif kind == "batch":
        state.update(jacs=_batch_jacobians(case, seed), batch=_batch())
    elif kind == "inverse":
        state["a"] = _padded(_spd(case["n"], seed, 1e-4, 1.0)[0])
    elif kind == "pinv":
        state["a"] = _padded(_spd(case["n"], seed, 1.0, 1e3, case["remove"])[0])
    elif kind == "product":
        state["p"], state["x"] = _product_operands(case, seed)
        state["out"] = torch.zeros_like(state["p"])
    elif kind == "eigen":
        n, p, d = case["blocks"], case["params"], case["dim"]
        i, j = torch.triu_indices(p, p, device=DEV)
        state["packed"] = _eigen_blocks(case, seed)[:, i, j].contiguous()
        state["values"] = torch.zeros((n, d), device=DEV, dtype=F64)
        state["vectors"] = torch.zeros((n, d, d), device=DEV, dtype=F64) if case["vectors"] else None
    elif kind == "jacobian":
        camera, points, oc, op = _scene(case["cams"], case["points_per_cam"], case["views"], case["window"], seed)
        n = len(oc)
        state.update(cameras=camera.contiguous(), points=points, obs_cam=oc, obs_pt=op,
                     rows=torch.zeros(2 * n + 1, device=DEV, dtype=torch.int32),
                     cols=torch.zeros(24 * n, device=DEV, dtype=torch.int32),
                     values=torch.zeros(24 * n, device=DEV, dtype=F64))
    torch.cuda.synchronize()  # the library's streams do not wait for torch's
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ok(status):
    if status != 0:
        raise native.UncError(status, native.lib().unc_last_error().decode())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve" and case["host"]:
        cam, pt, stats = native.compute_covariances(state["jac"], state["context"], precision=case["precision"])
        return {"cam": cam, "pt": pt, "iterations": stats["te_iterations"]}
    if kind == "solve":
        jac = state["jac"]
        stats = native.compute_covariances_device(
            state["context"], state["options"], jac.num_rows, jac.num_cols, jac.rows.data_ptr(), jac.cols.data_ptr(),
            jac.values.data_ptr(), state["cam"].data_ptr(), state["pt"].data_ptr())
        return {"cam": state["cam"], "pt": state["pt"], "iterations": stats["te_iterations"]}
    if kind == "batch":
        out = state["batch"].compute(state["jacs"], precision=case["precision"])
        return [{"cam": cam, "pt": pt} for cam, pt, _, _ in out]
    if kind in ("inverse", "pinv"):
        a = state["a"].clone()  # in place, and the caller keeps its matrix
        n, ld = a.shape
        if kind == "inverse":
            native.dense_inverse_device(a.data_ptr(), n, ld)
        else:
            native.pinv_psd_device(a.data_ptr(), n, ld, case["remove"])
        return a[:, :n]
    if kind == "product":
        n, ld = state["p"].shape
        native.gemm_mixed_device(n, state["p"].data_ptr(), state["x"].data_ptr(), ld, state["out"].data_ptr(),
                                 case["slices"])
        return state["out"][:, :n]
    if kind == "eigen":
        v = state["vectors"]
        _ok(native.lib().unc_block_eigen_device(
            state["packed"].data_ptr(), case["blocks"], case["params"], case["offset"], case["dim"],
            state["values"].data_ptr(), v.data_ptr() if v is not None else None, None))
        return {"values": state["values"], "vectors": v}
    _ok(native.lib().unc_jacobian_device(
        len(state["cameras"]), len(state["points"]), len(state["obs_cam"]), state["cameras"].data_ptr(),
        state["points"].data_ptr(), state["obs_cam"].data_ptr(), state["obs_pt"].data_ptr(), state["rows"].data_ptr(),
        state["cols"].data_ptr(), state["values"].data_ptr(), ctypes.c_void_p()))
    return {"rows": state["rows"], "cols": state["cols"], "values": state["values"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _solve_work(cams, points_per_cam, views):
    """Input and output bytes; the sparse stages' flops, the dense inverse (n^3) and five symmetric products."""
    n, points = 9 * cams, cams * points_per_cam
    obs = points * (2 + views)
    pairs = points * (2 + views) * (3 + views) / 2
    dense = n ** 3 + 5 * n * n * (n + 1)
    return 296 * obs + 360 * cams + 48 * points, dense + 486 * pairs + 1300 * obs


def work(case):
    kind = case["kind"]
    if kind == "solve":
        b, f = _solve_work(case["cams"], case["points_per_cam"], case["views"])
    elif kind == "batch":
        per = [_solve_work(int(c), case["points_per_cam"], case["views"]) for c in _batch_cameras(case, 0)]
        b, f = sum(p[0] for p in per), sum(p[1] for p in per)
    elif kind == "inverse":
        b, f = 16 * case["n"] ** 2, case["n"] ** 3
    elif kind == "pinv":
        b, f = 16 * case["n"] ** 2, 2 * case["n"] ** 3
    elif kind == "product":
        b, f = 24 * case["n"] ** 2, 2 * case["n"] ** 3
    elif kind == "eigen":
        p, d = case["params"], case["dim"]
        b = 8 * case["blocks"] * (p * (p + 1) // 2 + d + (d * d if case["vectors"] else 0))
        f = case["blocks"] * 25 * d ** 3
    else:
        obs = case["cams"] * case["points_per_cam"] * (2 + case["views"])
        b, f = 304 * obs + 24 * case["cams"] * case["points_per_cam"] + 72 * case["cams"], 350 * obs
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
def _wrapped_factorial(n):
    """32-bit signed factorial, wrapping from 13! on, as the Taylor coefficients use it."""
    f = math.factorial(n) & 0xFFFFFFFF
    return f - (1 << 32) if f >= 1 << 31 else f


def _taylor_inverse(Z, lam):
    """X + sum_i lam^i / (i-1)! X^(i+1), X = (Z + lam I)^-1, with the reference's stop rule."""
    n = len(Z)
    if lam == -1:
        lam = 10.0 ** (-1.2653 * math.log10(n) - 2.9415)
    Z.diagonal().add_(lam)
    e = 1 / torch.sqrt(Z.diagonal())
    X = torch.linalg.inv(Z * e[:, None] * e[None, :]) * e[:, None] * e[None, :]
    X = (X + X.T) / 2
    total, power, before, steps = X.clone(), X, math.inf, 0
    for i in range(1, 20):
        power = power @ X
        k = lam ** i / _wrapped_factorial(i - 1)
        change = abs(k * float(power.abs().max()))
        if change < 1e-5 or change > before:
            break
        before, steps = change, steps + 1
        total += k * power
    return total, steps


def _exact_solve(jac):
    """Camera and point covariances of a Jacobian whose arrays are torch tensors on the device."""
    C, P, N = jac.num_cams, jac.num_points, 9 * jac.num_cams
    J = jac.values.view(-1, 2, 12)
    first = jac.cols.view(-1, 24)
    oc, op = first[:, 0].long() // 9, (first[:, 9].long() - N) // 3
    keep = torch.ones(P, dtype=torch.bool, device=DEV)
    keep[torch.as_tensor(jac.pts2fix, device=DEV).long()] = False
    kept = keep[op]
    J, oc, op = J[kept], oc[kept], op[kept]
    Jc, Jp = J[:, :, :9], J[:, :, 9:]
    U = torch.zeros((C, 9, 9), device=DEV, dtype=F64).index_add_(0, oc, Jc.transpose(1, 2) @ Jc)
    V = torch.zeros((P, 3, 3), device=DEV, dtype=F64).index_add_(0, op, Jp.transpose(1, 2) @ Jp)
    sc = U.diagonal(dim1=1, dim2=2).sqrt()
    sp = V.diagonal(dim1=1, dim2=2).sqrt()
    sc, sp = torch.where(sc > 0, sc, 1.0), torch.where(sp > 0, sp, 1.0)
    W = Jc.transpose(1, 2) @ Jp
    Ws = W / sc[oc][:, :, None] / sp[op][:, None, :]
    Vs = V / sp[:, :, None] / sp[:, None, :]
    seen = torch.bincount(op, minlength=P) > 0
    Vs[~seen] = torch.eye(3, device=DEV, dtype=F64)
    Y = Ws @ torch.linalg.inv(Vs)[op]
    # Z as C x C blocks, one pass for each distance of two observations of a point in its list
    Z = torch.zeros((C * C, 9, 9), device=DEV, dtype=F64)
    diag = torch.arange(C, device=DEV) * (C + 1)
    Z.index_add_(0, diag, U / sc[:, :, None] / sc[:, None, :])
    lag = 0
    while lag < len(op):
        a = torch.nonzero(op[lag:] == op[:len(op) - lag])[:, 0]
        if not len(a):
            break
        for part in a.split(1 << 20):
            block = Y[part] @ Ws[part + lag].transpose(1, 2)
            Z.index_add_(0, oc[part] * C + oc[part + lag], block, alpha=-1)
            if lag:
                Z.index_add_(0, oc[part + lag] * C + oc[part], block.transpose(1, 2).contiguous(), alpha=-1)
        lag += 1
    Z = Z.view(C, C, 9, 9).permute(0, 2, 1, 3).reshape(N, N)
    iZ, steps = _taylor_inverse(Z, jac.lam)
    del Z
    blocks = iZ.view(C, 9, C, 9).diagonal(dim1=0, dim2=2).permute(2, 0, 1) / sc[:, :, None] / sc[:, None, :]
    i, j = torch.triu_indices(9, 9, device=DEV)
    cam = (blocks + blocks.transpose(1, 2) / 2)[:, i, j].reshape(-1)
    inner = torch.zeros((P, 3, 3), device=DEV, dtype=F64).index_add_(0, op, W.transpose(1, 2) @ blocks[oc] @ W)
    w, Q = torch.linalg.eigh(V.cpu())  # many small blocks: the host's routine
    w = torch.where(w > 64 * 2.220446049250313e-16 * w.abs().amax(1, keepdim=True), 1 / w, 0.0)
    D = ((Q * w[:, None, :]) @ Q.transpose(1, 2)).to(DEV)
    full = D + D @ inner @ D
    full[~seen] = 0.0
    i, j = torch.triu_indices(3, 3, device=DEV)
    return {"cam": cam, "pt": full[:, i, j].reshape(-1), "iterations": steps}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        out = _exact_solve(_reconstruction(case["cams"], case["points_per_cam"], case["views"], case["window"],
                                           case["lam"], seed, False))
        if case["host"]:
            out["cam"], out["pt"] = out["cam"].cpu().numpy(), out["pt"].cpu().numpy()
        return out
    if kind == "batch":
        outs = []
        for i, c in enumerate(_batch_cameras(case, 0)):
            jac = _reconstruction(c, case["points_per_cam"], case["views"], 48, case["lam"], 1000 * int(seed) + i, False)
            one = _exact_solve(jac)
            outs.append({"cam": one["cam"].cpu().numpy(), "pt": one["pt"].cpu().numpy()})
        return outs
    if kind == "inverse":
        return torch.linalg.inv(_spd(case["n"], seed, 1e-4, 1.0)[0])
    if kind == "pinv":
        _, Q, w = _spd(case["n"], seed, 1.0, 1e3, case["remove"])
        keep = Q[:, case["remove"]:]
        return (keep / w[case["remove"]:]) @ keep.T
    if kind == "product":
        P, X = _product_operands(case, seed)
        n = case["n"]
        return P[:, :n] @ X[:, :n]
    if kind == "eigen":
        o, d = case["offset"], case["dim"]
        values = torch.linalg.eigvalsh(_eigen_blocks(case, seed)[:, o:o + d, o:o + d].cpu())
        return {"values": values.flip(1).contiguous(), "vectors": None}  # a vector's sign is arbitrary
    camera, points, oc, op = _scene(case["cams"], case["points_per_cam"], case["views"], case["window"], seed)
    n = len(oc)
    return {"rows": (12 * torch.arange(2 * n + 1, device=DEV)).to(torch.int32), "cols": _columns(len(camera), oc, op),
            "values": _observation_blocks(camera, points, oc, op).reshape(-1)}
