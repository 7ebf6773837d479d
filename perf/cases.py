"""What is timed when this solver is made faster: the calls its users make,
from one tracked frame to a 1,200-camera map, through the public entry points
(visloc_ba.solver.CudaSolver and the C ABI of include/visloc_ba_cuda.h).

Problems are synthetic and made from a seed with torch, on the GPU when there
is one.  `exact` solves the same problems again with plain torch in FP64: the
Levenberg-Marquardt loop of the reference (right-perturbed poses, IRLS
weights, lambda on the diagonal, x10 / x0.1) over an explicitly formed reduced
system, with block-Jacobi conjugate gradients under the same stopping rule.
"""

from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "visloc-rs_b200"))

from visloc_ba import _abi  # noqa: E402
from visloc_ba.problem import (  # noqa: E402
    SE3,
    BaConfig,
    Camera,
    CameraModel,
    GncConfig,
    PackedProblem,
    RobustKernel,
)
from visloc_ba.solver import CudaSolver  # noqa: E402

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64

# LM settings of the solves: the stopping rules a mapping program uses, and
# the PCG controls of this repository's benchmark.
RELATIVE_COST_TOLERANCE = 1e-6
PCG_TOLERANCE = 1e-6
MAX_PCG = 200


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # Per-frame pose refinement of a tracker: 2D-3D matches of one image
        # against fixed landmarks, 30% of them wrong.  The smallest call.
        {"name": "pose_487", "kind": "pose", "matches": 487, "iterations": 10},
        # The cost of a map that is already on the device (the gate before a
        # tracking thread accepts an update), no allocation.
        {"name": "cost_200k", "kind": "cost", "cameras": 333, "observations": 200_001},
        # Local window of a stereo rig as monocular observations of two
        # sensors (the second through its extrinsic), Huber.
        {"name": "window_20", "kind": "window", "keyframes": 20, "points": 2000,
         "stereo": "rig", "weighted": False, "robust": "huber", "iterations": 10},
        # Local window of rectified stereo observations (three residual rows)
        # with external weights per observation, Cauchy, odd sizes.
        {"name": "window_13_rectified", "kind": "window", "keyframes": 13, "points": 1107,
         "stereo": "rectified", "weighted": True, "robust": "cauchy", "iterations": 10},
        # A small map with a SIMPLE_RADIAL camera per image (unordered photos).
        {"name": "ring_50", "kind": "ring", "cameras": 50, "points": 5000, "track": 6.0,
         "per_camera": True, "robust": "huber", "iterations": 20, "call": "optimize"},
        # Many uneven local windows as one batch in a captured graph (a
        # backend that refines the windows of many agents), from host to host
        # state on the uploaded batch.
        {"name": "batch_48", "kind": "batch", "windows": 48, "max_keyframes": 40,
         "max_points": 5000, "iterations": 6},
        # Global adjustment of a mid-sized map, host arrays in and out.
        {"name": "ring_300", "kind": "ring", "cameras": 300, "points": 60_000, "track": 7.0,
         "per_camera": False, "robust": "huber", "iterations": 15, "call": "optimize"},
        # The benchmark's map: 1,200 cameras with nearly every pair covisible
        # (the reduced system is dense), solved from the uploaded state.
        {"name": "ring_1200", "kind": "ring", "cameras": 1200, "points": 500_000, "track": 8.5,
         "per_camera": False, "robust": "huber", "iterations": 8, "call": "uploaded"},
        # A closed street loop: consecutive views, a banded reduced system.
        {"name": "street_1400", "kind": "street", "cameras": 1400, "points": 250_000,
         "iterations": 6, "call": "uploaded"},
        # Graduated non-convexity against gross outliers, truncated least
        # squares.
        {"name": "gnc_60", "kind": "gnc", "cameras": 60, "points": 4000, "track": 10.0,
         "outliers": 0.2},
        # ReducedSolveAccelerator::solve on blocks that the caller formed
        # (f32, as the reference hands them over), block-Jacobi.
        {"name": "reduced_1500", "kind": "reduced", "nodes": 1500, "band": 100, "cross": 40},
        # One damping trial of the rig solver: eliminate the points with new
        # inverses, then solve on the resident blocks with run inverses and
        # the coarse level.
        {"name": "trial_900", "kind": "trial", "frames": 900, "per_frame": 1500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pose", "cost", "window", "window", "ring", "ring", "batch", "street", "gnc",
                       "reduced", "trial"])
    if kind == "pose":
        return {"kind": kind, "matches": _log_int(rng, 60, 4000), "iterations": 10}
    if kind == "cost":
        return {"kind": kind, "cameras": _log_int(rng, 2, 1200),
                "observations": _log_int(rng, 500, 4_000_000)}
    if kind == "window":
        return {"kind": kind, "keyframes": rng.randint(5, 40), "points": _log_int(rng, 200, 5000),
                "stereo": rng.choice(["rig", "rectified"]), "weighted": rng.random() < 0.5,
                "robust": rng.choice(["huber", "cauchy", "none"]), "iterations": 10}
    if kind == "ring":
        cams = _log_int(rng, 12, 1100)
        per = rng.choice([60, 90, 140]) if cams > 100 else rng.randint(60, 200)
        return {"kind": kind, "cameras": cams, "points": int(cams * per * rng.uniform(0.9, 1.1)),
                "track": round(rng.uniform(5.5, 8.5), 2), "per_camera": rng.random() < 0.4,
                "robust": rng.choice(["huber", "cauchy"]), "iterations": 15 if cams < 400 else 8,
                "call": rng.choice(["optimize", "uploaded"])}
    if kind == "batch":
        return {"kind": kind, "windows": rng.randint(3, 60), "max_keyframes": rng.randint(8, 40),
                "max_points": _log_int(rng, 400, 5000), "iterations": 6}
    if kind == "street":
        cams = _log_int(rng, 400, 1400)
        return {"kind": kind, "cameras": cams, "points": int(cams * rng.uniform(100, 170)),
                "iterations": 6, "call": rng.choice(["optimize", "uploaded"])}
    if kind == "gnc":
        cams = _log_int(rng, 20, 120)
        return {"kind": kind, "cameras": cams, "points": cams * rng.randint(50, 80),
                "track": round(rng.uniform(9.0, 11.0), 2), "outliers": round(rng.uniform(0.05, 0.22), 2)}
    if kind == "reduced":
        n = _log_int(rng, 40, 1500)
        return {"kind": kind, "nodes": n, "band": min(rng.randint(10, 100), n // 3),
                "cross": min(rng.randint(0, 40), n // 8)}
    return {"kind": "trial", "frames": _log_int(rng, 150, 900), "per_frame": rng.randint(300, 1500)}


# ---------------------------------------------------------------- the problems
# A problem is a dict of FP64 / int64 tensors: q (N,4) (w,i,j,k), t (N,3), X
# (M,3), fixed (N) and pfixed (M) flags, op / ol (K) pose and landmark of each
# observation (landmark order), xy (K,2), oc (K) camera, cams (C,6) fx fy cx cy
# k1 k2, ext (C,3) sensor translation; optionally w (K) and ur (K) with
# baseline for rectified stereo.
class _Draws:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device=DEVICE, dtype=F64)

    def normal(self, sigma, *shape):
        return sigma * torch.randn(*shape, generator=self.g, device=DEVICE, dtype=F64)

    def integers(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device=DEVICE)


def _rotation(q):
    w, i, j, k = q.unbind(-1)
    return torch.stack([w * w + i * i - j * j - k * k, 2 * (i * j - w * k), 2 * (w * j + i * k),
                        2 * (w * k + i * j), w * w - i * i + j * j - k * k, 2 * (j * k - w * i),
                        2 * (i * k - w * j), 2 * (w * i + j * k), w * w - i * i - j * j + k * k],
                       -1).reshape(q.shape[:-1] + (3, 3))


def _quat_mul(a, b):
    aw, ai, aj, ak = a.unbind(-1)
    bw, bi, bj, bk = b.unbind(-1)
    return torch.stack([aw * bw - ai * bi - aj * bj - ak * bk, aw * bi + ai * bw + aj * bk - ak * bj,
                        aw * bj - ai * bk + aj * bw + ak * bi, aw * bk + ai * bj - aj * bi + ak * bw], -1)


def _axis_angle(v):
    th = v.norm(dim=-1, keepdim=True)
    s = torch.where(th > 1e-12, torch.sin(th / 2) / th.clamp_min(1e-300), torch.full_like(th, 0.5))
    return torch.cat([torch.cos(th / 2), v * s], -1)


def _looking(centers, targets):
    """Quaternions of world->camera rotations at `centers` towards `targets`
    (upright cameras: a turn about the vertical, then a tilt)."""
    f = targets - centers
    yaw = torch.atan2(f[:, 0], f[:, 2])
    pitch = torch.atan2(f[:, 1], torch.hypot(f[:, 0], f[:, 2]))
    zero = torch.zeros_like(yaw)
    turn = _axis_angle(torch.stack([zero, -yaw, zero], -1))
    tilt = _axis_angle(torch.stack([pitch, zero, zero], -1))
    return _quat_mul(tilt, turn)


def _project(P, q, t, X):
    """Pixels and depths of every observation at a state."""
    xs = torch.einsum("kij,kj->ki", _rotation(q)[P["op"]], X[P["ol"]]) + t[P["op"]] + P["ext"][P["oc"]]
    c = P["cams"][P["oc"]]
    x, y = xs[:, 0] / xs[:, 2], xs[:, 1] / xs[:, 2]
    r2 = x * x + y * y
    d = 1 + c[:, 4] * r2 + c[:, 5] * r2 * r2
    return torch.stack([c[:, 0] * x * d + c[:, 2], c[:, 1] * y * d + c[:, 3]], -1), xs[:, 2]


def _finish(P, d, size, *, outliers=0.02, rotation=0.005, translation=0.03, point=0.03, per_point=2,
            spread=50, outliers_every=1):
    """Measures the observations (those that fall in an image of `size`, of
    points that have `per_point` of them; the others stay unobserved), and
    perturbs the state that is handed over."""
    uv, z = _project(P, P["q"], P["t"], P["X"])
    if size:
        keep = (z > 0.3) & (uv >= 0).all(1) & (uv[:, 0] < size[0]) & (uv[:, 1] < size[1])
        seen = torch.bincount(P["ol"][keep], minlength=P["X"].shape[0])
        keep &= (seen >= per_point)[P["ol"]]
        P["op"], P["oc"], P["ol"], uv, z = P["op"][keep], P["oc"][keep], P["ol"][keep], uv[keep], z[keep]
    K = uv.shape[0]
    uv = uv + d.normal(0.7, K, 2)
    wrong = d.uniform(0, 1, K) < outliers
    if outliers_every > 1:  # so that every point keeps enough good observations
        first = torch.searchsorted(P["ol"], P["ol"])
        wrong = d.uniform(0, 1, K) < outliers * outliers_every
        wrong &= (torch.arange(K, device=DEVICE) - first) % outliers_every == 0
    uv = torch.where(wrong[:, None], uv + d.uniform(-spread, spread, K, 2), uv)
    P["xy"] = uv
    if P.get("baseline"):
        c = P["cams"][P["oc"]]
        P["ur"] = uv[:, 0] - c[:, 0] * P["baseline"] / z + d.normal(0.7, K)
    free = ~P["fixed"]
    n = P["q"].shape[0]
    turn = _axis_angle(d.normal(rotation, n, 3))
    move = d.normal(translation, n, 3)
    centre = -torch.einsum("nji,nj->ni", _rotation(P["q"]), P["t"])
    q1 = _quat_mul(P["q"], turn)
    t1 = -torch.einsum("nij,nj->ni", _rotation(q1), centre + move)
    P["q"] = torch.where(free[:, None], q1, P["q"])
    P["t"] = torch.where(free[:, None], t1, P["t"])
    moved = P["X"] + d.normal(point, P["X"].shape[0], 3)
    P["X"] = torch.where(P["pfixed"][:, None], P["X"], moved)
    return P


def _flags(n, first):
    f = torch.zeros(n, dtype=torch.bool, device=DEVICE)
    f[:first] = True
    return f


def _ring(case, seed, outliers=0.02):
    """Cameras on a circle around a cube of points, each point in a random
    set of at least four images (geometric count); the first two cameras
    fixed."""
    d = _Draws(seed)
    n, m = case["cameras"], case["points"]
    ang = torch.arange(n, device=DEVICE, dtype=F64) * (2 * math.pi / n)
    centers = torch.stack([20 * torch.cos(ang), d.uniform(-1, 1, n), 20 * torch.sin(ang)], 1)
    q = _looking(centers, d.normal(0.15, n, 3))
    t = -torch.einsum("nij,nj->ni", _rotation(q), centers)
    X = d.uniform(-5, 5, m, 3) * torch.tensor([1.0, 0.7, 1.0], device=DEVICE, dtype=F64)
    # Track lengths follow the law's quantiles, so that every seed has as many
    # observations; a point's images are distinct.
    mean, least = case["track"], case.get("least", 4)
    u = torch.frac((torch.arange(m, device=DEVICE, dtype=F64) + 0.5) * 0.6180339887498949)
    T = least + torch.floor(torch.log(u.clamp_min(1e-12)) / math.log(1 - 1 / (mean - least + 1))).long()
    T = T.clamp(max=min(60, n))
    ol = torch.repeat_interleave(torch.arange(m, device=DEVICE), T)
    pick = torch.floor(d.uniform(0, 1, ol.shape[0]) * (n + 1 - T)[ol]).long()
    pick = torch.sort(ol * n + pick).values % n
    op = pick + torch.arange(ol.shape[0], device=DEVICE) - (torch.cumsum(T, 0) - T)[ol]
    if case["per_camera"]:
        f, k1 = d.uniform(2400, 3600, n), d.uniform(-0.05, 0.05, n)
        cams = torch.stack([f, f, torch.full_like(f, 2000), torch.full_like(f, 1500), k1,
                            torch.zeros_like(f)], 1)
    else:
        cams = torch.tensor([[3000.0, 3000.0, 2000.0, 1500.0, 0.0, 0.0]], device=DEVICE, dtype=F64)
    P = {"q": q, "t": t, "X": X, "fixed": _flags(n, 2), "pfixed": _flags(m, 0), "op": op, "ol": ol,
         "oc": op.clone() if case["per_camera"] else torch.zeros_like(op),
         "cams": cams, "ext": torch.zeros(cams.shape[0], 3, device=DEVICE, dtype=F64)}
    return _finish(P, d, None, outliers=outliers, outliers_every=case.get("every", 1))


def _street(case, seed):
    """Forward cameras along a closed loop, facade points on both sides, each
    seen by a run of consecutive cameras; every 100th camera fixed (surveyed
    positions), so the loop has no free long-wavelength drift."""
    d = _Draws(seed)
    n, m = case["cameras"], case["points"]
    radius = n / (2 * math.pi)
    ang = torch.arange(n, device=DEVICE, dtype=F64) / radius
    centers = torch.stack([radius * torch.cos(ang), torch.full_like(ang, 1.6), radius * torch.sin(ang)], 1)
    q = _looking(centers, centers + torch.stack([-torch.sin(ang), torch.zeros_like(ang), torch.cos(ang)], 1))
    t = -torch.einsum("nij,nj->ni", _rotation(q), centers)
    s = d.uniform(0, n, m)
    side = torch.where(d.uniform(0, 1, m) < 0.5, -1.0, 1.0)
    rad = radius + side * (8 + d.normal(0.2, m))
    X = torch.stack([rad * torch.cos(s / radius), d.uniform(-6, 8, m), rad * torch.sin(s / radius)], 1)
    lo, hi = torch.floor(s - 24).long(), torch.floor(s - 9).long()
    T = (4 + torch.floor(torch.log(d.uniform(1e-12, 1, m)) / math.log(1 - 1 / 3.7)).long()).clamp(4, 16)
    T = torch.minimum(T, hi - lo + 1)
    start = lo + torch.floor(d.uniform(0, 1, m) * (hi - lo + 2 - T)).long()
    ol = torch.repeat_interleave(torch.arange(m, device=DEVICE), T)
    rank = torch.arange(ol.shape[0], device=DEVICE) - (torch.cumsum(T, 0) - T)[ol]
    op = (start[ol] + rank) % n
    cams = torch.tensor([[1000.0, 1000.0, 960.0, 540.0, 0.0, 0.0]], device=DEVICE, dtype=F64)
    fixed = torch.arange(n, device=DEVICE) % 100 < 2
    P = {"q": q, "t": t, "X": X, "fixed": fixed, "pfixed": _flags(m, 0), "op": op, "ol": ol,
         "oc": torch.zeros_like(op), "cams": cams, "ext": torch.zeros(1, 3, device=DEVICE, dtype=F64)}
    return _finish(P, d, (1920, 1080), rotation=0.002, translation=0.02, per_point=4, spread=8)


def _window(keyframes, points, stereo, weighted, seed):
    """A local window moving forward; the first tenth of its keyframes is
    anchored.  Each point is taken by up to 5 to 12 of the sensors that see it."""
    d = _Draws(seed)
    n, m, b = keyframes, points, 0.11
    s = torch.arange(n, device=DEVICE, dtype=F64) * 0.35
    centers = torch.stack([0.3 * torch.sin(s / 3), d.normal(0.02, n), s], 1)
    zero = torch.zeros_like(s)
    q = _axis_angle(torch.stack([zero, -0.05 * torch.sin(s / 2), zero], 1))
    t = -torch.einsum("nij,nj->ni", _rotation(q), centers)
    # Points beside the path (ahead of it there is no parallax).
    aside = torch.where(d.uniform(0, 1, m) < 0.5, -1.0, 1.0) * d.uniform(1, 5, m)
    X = torch.stack([aside, d.uniform(-3, 3, m),
                     d.uniform(3, 10, m) + float(s.max()) * d.uniform(0, 1, m)], 1)
    sides = 2 if stereo == "rig" else 1
    cam = [458.0, 458.0, 376.0, 240.0, 0.0, 0.0]
    cams = torch.tensor([cam] * sides, device=DEVICE, dtype=F64)
    ext = torch.tensor([[0.0, 0, 0], [-b, 0, 0]][:sides], device=DEVICE, dtype=F64)
    want = d.integers(5, 13, m)
    pick = torch.argsort(d.uniform(0, 1, m, n * sides), 1)
    pick = torch.argsort(pick, 1) < want[:, None]
    ol, sensor = torch.nonzero(pick, as_tuple=True)
    P = {"q": q, "t": t, "X": X, "fixed": _flags(n, max(1, round(0.1 * n))), "pfixed": _flags(m, 0),
         "op": sensor // sides, "oc": sensor % sides, "ol": ol, "cams": cams, "ext": ext}
    if stereo == "rectified":
        P["baseline"] = b
    P = _finish(P, d, (752, 480), rotation=0.003, translation=0.01, point=0.03,
                per_point=4, spread=15)
    if weighted:
        P["w"] = d.uniform(0.2, 1.5, P["op"].shape[0])
    return P


def _pose(case, seed):
    d = _Draws(seed)
    m = case["matches"]
    z = d.uniform(2, 20, m)
    uv = torch.stack([d.uniform(0, 752, m), d.uniform(0, 480, m)], 1)
    X = torch.cat([(uv - torch.tensor([376.0, 240.0], device=DEVICE, dtype=F64)) / 458.0 * z[:, None],
                   z[:, None]], 1)
    P = {"q": torch.tensor([[1.0, 0, 0, 0]], device=DEVICE, dtype=F64),
         "t": torch.zeros(1, 3, device=DEVICE, dtype=F64), "X": X, "fixed": _flags(1, 0),
         "pfixed": _flags(m, m), "op": torch.zeros(m, dtype=torch.long, device=DEVICE),
         "ol": torch.arange(m, device=DEVICE), "oc": torch.zeros(m, dtype=torch.long, device=DEVICE),
         "cams": torch.tensor([[458.0, 458.0, 376.0, 240.0, 0.0, 0.0]], device=DEVICE, dtype=F64),
         "ext": torch.zeros(1, 3, device=DEVICE, dtype=F64)}
    return _finish(P, d, (752, 480), outliers=0.3, rotation=0.02, translation=0.1, per_point=1)


def _problems(case, seed):
    kind = case["kind"]
    if kind == "pose":
        return [_pose(case, seed)]
    if kind == "window":
        return [_window(case["keyframes"], case["points"], case["stereo"], case["weighted"], seed)]
    if kind == "batch":
        sizes = np.random.default_rng(case["windows"])  # other contents, the same sizes
        nk = sizes.integers(5, case["max_keyframes"] + 1, case["windows"])
        npt = sizes.integers(200, case["max_points"] + 1, case["windows"])
        return [_window(int(a), int(b), "rig", False, seed + 7919 * (1 + i))
                for i, (a, b) in enumerate(zip(nk, npt))]
    if kind == "street":
        return [_street(case, seed)]
    if kind == "cost":
        track = 6.0
        return [_ring({"cameras": case["cameras"], "points": int(case["observations"] / track) + 1,
                       "track": track, "per_camera": False}, seed)]
    # Under GNC a point may lose its outliers: enough images stay to hold it.
    gnc = {"least": 7, "every": 4} if kind == "gnc" else {}
    return [_ring({"per_camera": False, **gnc, **case}, seed,
                  outliers=case.get("outliers", 0.02))]


def _config(case):
    robust = {"huber": RobustKernel.huber(1.0), "cauchy": RobustKernel.cauchy(2.0),
              "none": RobustKernel.none()}[case.get("robust", "huber")]
    return BaConfig(max_iterations=case.get("iterations", 10), robust_kernel=robust,
                    relative_cost_tolerance=RELATIVE_COST_TOLERANCE, max_pcg_iterations=MAX_PCG,
                    pcg_relative_tolerance=PCG_TOLERANCE, graph=case["kind"] == "batch")


def _packed(P):
    h = {k: v.cpu().numpy() for k, v in P.items() if isinstance(v, torch.Tensor)}
    cameras = []
    for c, e in zip(h["cams"], h["ext"]):
        if c[4] != 0.0:
            cam = Camera(CameraModel.SIMPLE_RADIAL, 4000, 3000, [c[0], c[2], c[3], c[4]])
        else:
            cam = Camera.pinhole(int(2 * c[2]), int(2 * c[3]), c[0], c[1], c[2], c[3])
        cameras.append((cam, SE3((1.0, 0.0, 0.0, 0.0), tuple(e))))
    K = h["op"].shape[0]
    stereo = "ur" in h
    return PackedProblem(
        h["q"], h["t"], h["X"], h["op"], h["ol"], h["xy"], cameras, h["fixed"], h["pfixed"],
        h["oc"] if len(cameras) > 1 else None, h.get("w"),
        np.full(K, _abi.OBS_STEREO, np.uint8) if stereo else None,
        np.stack([h["ur"], np.zeros(K)], 1) if stereo else None, None, P.get("baseline") or 0.0)


# ------------------------------------------------------ reduced camera systems
def _reduced(case, seed):
    """A reduced camera system of a city block passed several times: each node
    tied to its capture-order neighbours and to nodes of the other passes by
    random positive semidefinite couplings, lightly damped."""
    d = _Draws(seed)
    n, band, cross = case["nodes"], case["band"], case["cross"]
    i = torch.arange(n, device=DEVICE)
    a = i[:, None].expand(n, band)
    b = a + torch.arange(1, band + 1, device=DEVICE)
    key = (a * n + b)[b < n]
    if cross:
        other = (i[:, None] + n // 4 + d.integers(0, max(1, n // 2), n, cross)) % n
        lo, hi = torch.minimum(i[:, None], other), torch.maximum(i[:, None], other)
        key = torch.cat([key, (lo * n + hi)[lo != hi]])
    key = torch.unique(key)
    a, b = key // n, key % n
    ne = key.shape[0]
    eye = torch.eye(6, device=DEVICE, dtype=F64)
    ga, gb = eye + d.normal(0.15, ne, 6, 6), eye + d.normal(0.15, ne, 6, 6)
    w = d.uniform(0.5, 1.5, ne)[:, None, None]
    diag = torch.zeros(n, 6, 6, device=DEVICE, dtype=F64)
    # Sums over at most a few hundred edges a node, in edge order on the host
    # (the same inputs on every run).
    for idx, g in ((a, ga), (b, gb)):
        diag += _ordered_sum(idx, (w * (g.transpose(1, 2) @ g)).reshape(ne, 36), n).reshape(n, 6, 6)
    diag += 0.05 * eye
    off = (-w * (gb.transpose(1, 2) @ ga)).float()
    return {"diag": diag, "a": a, "b": b, "off": off, "rhs": d.normal(1.0, n, 6)}


def _ordered_sum(idx, v, n):
    """Rows of v summed by idx in row order: the same result on every run."""
    order = torch.argsort(idx, stable=True)
    lengths = torch.bincount(idx, minlength=n)
    return torch.segment_reduce(v[order], "sum", lengths=lengths, axis=0, initial=0.0)


def _elimination(case, seed):
    """The points of a street capture: frames along a line, each point in a
    run of consecutive frames (95% 3-15, 5% 40-120), random Jacobians."""
    d, layout = _Draws(seed), _Draws(case["frames"])  # other contents, the same structure
    n = case["frames"]
    m = max(8, int(n * case["per_frame"] / 12.5))
    long = layout.uniform(0, 1, m) < 0.05
    T = torch.where(long, layout.integers(40, 121, m), layout.integers(3, 16, m)).clamp(max=n)
    start = torch.floor(layout.uniform(0, 1, m) * (n + 1 - T)).long()
    ol = torch.repeat_interleave(torch.arange(m, device=DEVICE), T)
    off = torch.cat([torch.zeros(1, dtype=torch.long, device=DEVICE), torch.cumsum(T, 0)])
    nodes = start[ol] + torch.arange(ol.shape[0], device=DEVICE) - off[:-1][ol]
    K = ol.shape[0]
    A, B = d.normal(1.0, K, 3, 6), d.normal(1.0, K, 3, 3)
    hcp = A.transpose(1, 2) @ B
    eye3, eye6 = torch.eye(3, device=DEVICE, dtype=F64), torch.eye(6, device=DEVICE, dtype=F64)
    V = torch.segment_reduce((B.transpose(1, 2) @ B).reshape(K, 9), "sum", lengths=T, axis=0
                             ).reshape(m, 3, 3) + eye3
    vinv, before = torch.linalg.inv(V), torch.linalg.inv(V + 0.5 * eye3)
    U = _ordered_sum(nodes, (A.transpose(1, 2) @ A).reshape(K, 36), n).reshape(n, 6, 6)
    W = _ordered_sum(nodes, (hcp @ vinv[ol] @ hcp.transpose(1, 2)).reshape(K, 36), n).reshape(n, 6, 6)
    reach = torch.full((n,), -1, dtype=torch.long, device=DEVICE)
    reach.scatter_reduce_(0, start, start + T - 1, "amax")
    reach = torch.cummax(reach, 0).values
    cnt = (reach - torch.arange(n, device=DEVICE)).clamp_min(0)
    s = torch.repeat_interleave(torch.arange(n, device=DEVICE), cnt)
    t = s + 1 + torch.arange(s.shape[0], device=DEVICE) - (torch.cumsum(cnt, 0) - cnt)[s]
    first = torch.cumsum(cnt, 0) - cnt
    E = {"n": n, "off": off, "ol": ol, "nodes": nodes, "hcp": hcp, "vinv": vinv, "before": before,
         "diag": U + 0.3 * eye6 - W, "a": s, "b": t, "first": first, "rhs": d.normal(1.0, n, 6)}
    E["blocks"] = _eliminated(E, vinv)
    run, group = 32, max(32, -(-n // 256))
    E["run_edges"] = torch.nonzero(s // run == t // run).reshape(-1)
    E["group"], E["run"] = group, run
    E["runs"] = []
    dense = _dense_blocks(E["diag"], s, t, E["blocks"])
    for f in range(0, n, run):
        e = min(n, f + run)
        sub = dense[f:e, f:e].permute(0, 2, 1, 3).reshape(6 * (e - f), 6 * (e - f))
        E["runs"].append((f, torch.linalg.inv(sub)))
    g = torch.arange(n, device=DEVICE) // group
    mg = int(g[-1]) + 1
    fold = torch.zeros(mg, n, device=DEVICE, dtype=F64)
    fold[g, torch.arange(n, device=DEVICE)] = 1.0
    agg = torch.einsum("gi,hj,ijab->gahb", fold, fold, dense).reshape(6 * mg, 6 * mg)
    E["coarse"] = torch.linalg.inv(agg)
    return E


def _pairs(off, chunk):
    """(first, second) rows of every ordered pair k <= j of each segment, in
    pieces of about `chunk` pairs."""
    T = off[1:] - off[:-1]
    total = torch.cumsum(T * T, 0)
    p, m = 0, T.shape[0]
    while p < m:
        base = int(total[p - 1]) if p else 0
        e = max(p + 1, int(torch.searchsorted(total, base + chunk)))
        e = min(e, m)
        cnt = T[p:e] * T[p:e]
        pt = torch.repeat_interleave(torch.arange(p, e, device=off.device), cnt)
        r = torch.arange(pt.shape[0], device=off.device) - (torch.cumsum(cnt, 0) - cnt)[pt - p]
        k, j = off[pt] + r // T[pt], off[pt] + r % T[pt]
        yield k, j
        p = e


def _eliminated(E, vinv):
    ne = E["a"].shape[0]
    blocks = torch.zeros(ne, 6, 6, device=DEVICE, dtype=F64)
    sk = E["hcp"] @ vinv[E["ol"]]
    for k, j in _pairs(E["off"], 1 << 21):
        keep = k < j
        k, j = k[keep], j[keep]
        s, t = E["nodes"][k], E["nodes"][j]
        blocks.index_add_(0, E["first"][s] + t - s - 1, E["hcp"][j] @ sk[k].transpose(1, 2), alpha=-1)
    return blocks


def _dense_blocks(diag, a, b, off):
    n = diag.shape[0]
    S = torch.zeros(n, n, 6, 6, device=DEVICE, dtype=F64)
    S[b, a] = off.to(F64)
    S[a, b] = off.to(F64).transpose(1, 2)
    i = torch.arange(n, device=DEVICE)
    S[i, i] = diag
    return S


def _doubles(x):
    return np.ascontiguousarray(x.cpu().numpy(), dtype=np.float64)


def _column_major(x):
    return np.ascontiguousarray(x.transpose(-1, -2).cpu().numpy())


def _ptr(a, ctype):
    return a.ctypes.data_as(C.POINTER(ctype))


# ---------------------------------------------------------- prepare, run, work
_SOLVER = []


def _solver():
    """The one context that a program's solves share."""
    if not _SOLVER:
        _SOLVER.append(CudaSolver(0))
    return _SOLVER[0]


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case, kind = case, case["kind"]
    if kind in ("reduced", "trial"):
        return _prepare_reduced(st, case, seed)
    problems = [_packed(P) for P in _problems(case, seed)]
    st.cfg = _config(case)
    st.problems = problems
    if kind == "cost":
        return _prepare_cost(st)
    uploaded = kind == "batch" or case.get("call") == "uploaded"
    st.solver = CudaSolver(0) if uploaded else _solver()
    if kind == "batch":
        st.solver.batch_upload(problems, st.cfg)
    elif uploaded:
        if st.solver.upload(problems[0], st.cfg) != _abi.OK:
            raise RuntimeError(st.solver.last_error())
    else:
        p = problems[0]
        st.initial = (p.pose_q.copy(), p.pose_t.copy(), p.landmarks.copy())
        st.gnc = GncConfig(kernel=_abi.GNC_TRUNCATED_LEAST_SQUARES, c=3.0, anneal_factor=2.0,
                           inner_iterations=3)
    return st


def _prepare_cost(st):
    p = st.problems[0]
    st.keep = []
    st.abi = p.abi()
    for name, ctype in (("pose_q", C.c_double), ("pose_t", C.c_double), ("landmarks", C.c_double),
                        ("obs_pose", C.c_uint32), ("obs_landmark", C.c_uint32), ("obs_xy", C.c_double)):
        t = torch.from_numpy(getattr(p, name)).to(DEVICE)
        st.keep.append(t)
        setattr(st.abi, name, C.cast(C.c_void_p(t.data_ptr()), C.POINTER(ctype)))
    st.abi_cfg = st.cfg.to_abi()
    st.cost = torch.zeros(1, dtype=F64, device=DEVICE)
    st.counts = torch.zeros(2, dtype=torch.int64, device=DEVICE)
    st.error = C.create_string_buffer(256)
    st.lib = _abi.load_solver_library()
    return st


def _prepare_reduced(st, case, seed):
    trial = case["kind"] == "trial"
    D = _elimination(case, seed) if trial else _reduced(case, seed)
    n = D["diag"].shape[0]
    st.diag, st.rhs = _column_major(D["diag"]), _doubles(D["rhs"])
    st.edges = np.ascontiguousarray(torch.stack([D["a"], D["b"]], 1).cpu().numpy().astype(np.uint32))
    st.x = np.zeros((n, 6))
    st.its, st.rr = C.c_uint32(), C.c_double()
    s = st.system = _abi.ReducedSystem()
    s.num_nodes, s.num_edges = n, len(st.edges)
    s.diag, s.rhs, s.edges = _ptr(st.diag, C.c_double), _ptr(st.rhs, C.c_double), _ptr(st.edges, C.c_uint32)
    s.tol, s.max_iterations = PCG_TOLERANCE, 500
    st.solver = CudaSolver(0)
    if not trial:
        st.off = _column_major(D["off"])
        s.offdiag = _ptr(st.off, C.c_float)
        return st
    pre = st.pre = _abi.ReducedPreconditioner()
    st.first = np.array([f for f, _ in D["runs"]], np.uint32)
    st.size = np.array([r.shape[0] // 6 for _, r in D["runs"]], np.uint32)
    st.inv = np.concatenate([_column_major(r).reshape(-1) for _, r in D["runs"]])
    st.cinv = _column_major(D["coarse"])
    pre.num_clusters = len(st.first)
    pre.cluster_first, pre.cluster_size = _ptr(st.first, C.c_uint32), _ptr(st.size, C.c_uint32)
    pre.cluster_inverse = _ptr(st.inv, C.c_double)
    pre.coarse_group, pre.coarse_nodes, pre.coarse_inverse = D["group"], n, _ptr(st.cinv, C.c_double)
    el = st.el = _abi.PointElimination()
    st.off = np.ascontiguousarray(D["off"].cpu().numpy().astype(np.uint64))
    st.nodes = np.ascontiguousarray(D["nodes"].cpu().numpy().astype(np.uint32))
    st.hcp, st.vinv, st.before = _column_major(D["hcp"]), _column_major(D["vinv"]), _column_major(D["before"])
    st.run_edges = np.ascontiguousarray(D["run_edges"].cpu().numpy().astype(np.uint32))
    el.structure_id, el.linearization_id = 1, 1
    el.num_nodes, el.num_points, el.num_edges = n, len(st.off) - 1, len(st.edges)
    el.edges, el.point_off = _ptr(st.edges, C.c_uint32), _ptr(st.off, C.c_uint64)
    el.point_nodes, el.hcp = _ptr(st.nodes, C.c_uint32), _ptr(st.hcp, C.c_double)
    el.num_run_edges, el.run_edges = len(st.run_edges), _ptr(st.run_edges, C.c_uint32)
    el.coarse_group, el.coarse_nodes = D["group"], n
    m = -(-n // D["group"])
    st.run_blocks, st.sums = np.zeros((len(st.run_edges), 36)), np.zeros((m * m, 36))
    # The trial before this one: the structure is indexed and the
    # linearisation uploaded.
    el.point_inverse = _ptr(st.before, C.c_double)
    _eliminate(st)
    el.point_inverse = _ptr(st.vinv, C.c_double)
    return st


def _eliminate(st):
    rc = st.solver.lib.visloc_ba_cuda_reduced_eliminate(
        st.solver.ctx, C.byref(st.el), _ptr(st.run_blocks, C.c_double), _ptr(st.sums, C.c_double))
    if rc != _abi.OK:
        raise RuntimeError(st.solver.last_error())


def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "cost":
        rc = st.lib.visloc_ba_cuda_cost_noalloc(
            C.byref(st.abi), C.byref(st.abi_cfg), C.c_void_p(torch.cuda.current_stream().cuda_stream),
            C.c_void_p(st.cost.data_ptr()), C.c_void_p(st.counts.data_ptr()), st.error, len(st.error))
        if rc != _abi.OK:
            raise RuntimeError(st.error.value.decode())
        return {"cost": st.cost, "counts": st.counts}
    if kind == "reduced":
        rc = st.solver.lib.visloc_ba_cuda_reduced_solve(
            st.solver.ctx, C.byref(st.system), _ptr(st.x, C.c_double), C.byref(st.its), C.byref(st.rr))
        if rc != _abi.OK:
            raise RuntimeError(st.solver.last_error())
        return {"x": st.x}
    if kind == "trial":
        _eliminate(st)
        rc = st.solver.lib.visloc_ba_cuda_reduced_solve_preconditioned(
            st.solver.ctx, C.byref(st.system), C.byref(st.pre), _ptr(st.x, C.c_double),
            C.byref(st.its), C.byref(st.rr))
        if rc != _abi.OK:
            raise RuntimeError(st.solver.last_error())
        return {"x": st.x, "run_blocks": st.run_blocks, "coarse_sums": st.sums}
    if kind == "batch":
        results = st.solver.batch_solve_uploaded()
        st.solver.batch_download(st.problems)
        return {"initial": np.array([r.initial_cost for r in results]),
                "final": np.array([r.final_cost for r in results]),
                "q": np.concatenate([p.pose_q for p in st.problems]),
                "t": np.concatenate([p.pose_t for p in st.problems]),
                "X": np.concatenate([p.landmarks for p in st.problems])}
    p = st.problems[0]
    if case.get("call") == "uploaded":
        rc, res = st.solver.solve_uploaded(st.cfg)
        if rc == _abi.OK:
            rc = st.solver.download(p)
    else:
        for a, b in zip((p.pose_q, p.pose_t, p.landmarks), st.initial):
            np.copyto(a, b)
        if kind == "gnc":
            rc, res = st.solver.optimize_gnc(p, st.cfg, st.gnc)
        else:
            rc, res = st.solver.optimize(p, st.cfg)
    if rc != _abi.OK:
        raise RuntimeError(st.solver.last_error())
    out = {"initial": res.initial_cost, "final": res.final_cost, "q": p.pose_q, "t": p.pose_t}
    if kind != "pose":
        out["X"] = p.landmarks
    if kind == "gnc":
        out["weights"] = res.observation_weights
    return out


def work(case):
    """Bytes: the caller's arrays once in and the state once out (what any
    solve must move).  Operations: each LM iteration linearises every
    observation and forms the Schur terms, and each PCG iteration (taken as
    ten per LM iteration) multiplies by the reduced system."""
    kind = case["kind"]
    if kind == "cost":
        k = case["observations"]
        return {"bytes": 24 * k + 24 * (k / 6) + 56 * case["cameras"], "flops": 80 * k}
    if kind == "reduced":
        ne = case["nodes"] * (case["band"] + case["cross"])
        return {"bytes": 152 * ne + 384 * case["nodes"], "flops": 30 * 144 * ne}
    if kind == "trial":
        k = case["frames"] * case["per_frame"]
        pairs, ne = 19 * k, 100 * case["frames"]
        return {"bytes": 144 * k + 72 * k / 12.5 + 288 * ne, "flops": 216 * pairs + 30 * 144 * ne}
    if kind == "pose":
        sizes = [(1, case["matches"], case["matches"], 0)]
    elif kind == "window":
        sizes = [(case["keyframes"], case["points"], 6 * case["points"], 21)]
    elif kind == "batch":
        n, m = (5 + case["max_keyframes"]) / 2, (200 + case["max_points"]) / 2
        sizes = [(case["windows"] * n, case["windows"] * m, case["windows"] * 6 * m, 21)]
    elif kind == "street":
        sizes = [(case["cameras"], case["points"], 6.5 * case["points"], 25)]
    else:
        T = case["track"]
        sizes = [(case["cameras"], case["points"], T * case["points"], T * T)]
    n, m, k, pairs = sizes[0]
    its = {"gnc": 40}.get(kind, min(case.get("iterations", 6), 6))
    flops = its * (300 * k + 250 * m * pairs)
    return {"bytes": 24 * k + 2 * (24 * m + 56 * n), "flops": flops}


def tolerance(case):
    """About four times what FP32 Jacobians, Schur blocks and PCG vectors (this
    solver's precision) were seen to move the results, by comparison with
    `exact` over drawn cases: the worst landmarks 2.3e-6 (weakly held depths),
    a reduced solve 1.5e-7.  Costs alone are FP64 sums."""
    return {"cost": {"rel": 1e-12},
            "reduced": {"rel": 1e-6},
            "trial": {"rel": 1e-6}}.get(case["kind"], {"rel": 1e-5})


# --------------------------------------------------------------- exact results
def _weights(kernel, p, s):
    if kernel == "huber":
        return torch.where(s <= p * p, torch.ones_like(s), p / s.clamp_min(1e-300).sqrt())
    if kernel == "cauchy":
        return 1 / (1 + s / (p * p))
    return torch.ones_like(s)


def _robust(kernel, p, s):
    if kernel == "huber":
        return torch.where(s <= p * p, s, 2 * p * s.clamp_min(1e-300).sqrt() - p * p)
    if kernel == "cauchy":
        return p * p * torch.log1p(s / (p * p))
    return s


def _residuals(P, q, t, X, jacobians=False):
    """Residual rows r (K,m), d r / d X (K,m,3), and whether the point is in
    front of the sensor."""
    R = _rotation(q)[P["op"]]
    xs = torch.einsum("kij,kj->ki", R, X[P["ol"]]) + t[P["op"]] + P["ext"][P["oc"]]
    c = P["cams"][P["oc"]]
    x, y, z = xs[:, 0] / xs[:, 2], xs[:, 1] / xs[:, 2], xs[:, 2]
    r2 = x * x + y * y
    d, g = 1 + c[:, 4] * r2 + c[:, 5] * r2 * r2, c[:, 4] + 2 * c[:, 5] * r2
    rows = [c[:, 0] * x * d + c[:, 2] - P["xy"][:, 0], c[:, 1] * y * d + c[:, 3] - P["xy"][:, 1]]
    stereo = "ur" in P
    if stereo:
        rows.append(c[:, 0] * x + c[:, 2] - c[:, 0] * P["baseline"] / z - P["ur"])
    r, ok = torch.stack(rows, -1), z > 0
    if not jacobians:
        return r, None, ok
    d11, d12, d22 = d + 2 * x * x * g, 2 * x * y * g, d + 2 * y * y * g
    j = [torch.stack([c[:, 0] * d11, c[:, 0] * d12, -c[:, 0] * (d11 * x + d12 * y)], -1),
         torch.stack([c[:, 1] * d12, c[:, 1] * d22, -c[:, 1] * (d12 * x + d22 * y)], -1)]
    if stereo:
        zero = torch.zeros_like(z)
        j.append(torch.stack([c[:, 0], zero, -c[:, 0] * (x - P["baseline"] / z)], -1))
    return r, (torch.stack(j, 1) / z[:, None, None]) @ R, ok


def _cost(P, q, t, X, kernel, p):
    r, _, ok = _residuals(P, q, t, X)
    rho = _robust(kernel, p, (r * r).sum(1))
    if "w" in P:
        rho = rho * P["w"]
    return float(rho[ok].sum()), int((~ok).sum())


class _System:
    """The normal equations of a problem: index lists once per problem, the
    damped reduced system of each linearisation and lambda."""

    def __init__(self, P):
        self.P = P
        self.slot = torch.where(P["fixed"], -1, torch.cumsum(~P["fixed"], 0) - 1)
        self.nv, self.m = int((~P["fixed"]).sum()), P["X"].shape[0]
        var = (self.slot[P["op"]] >= 0) & ~P["pfixed"][P["ol"]]
        self.obs = torch.nonzero(var).reshape(-1)          # landmark order
        pts = P["ol"][self.obs]
        self.off = torch.cat([torch.zeros(1, dtype=torch.long, device=DEVICE),
                              torch.cumsum(torch.bincount(pts, minlength=self.m), 0)])

    def linearise(self, q, t, X, kernel, p):
        P = self.P
        r, J, ok = _residuals(P, q, t, X, True)
        w = _weights(kernel, p, (r * r).sum(1))
        if "w" in P:
            w = w * P["w"]
        w = torch.where(ok, w, torch.zeros_like(w))
        H = torch.einsum("kma,kmb->kab", J, J) * w[:, None, None]
        e = torch.einsum("kma,km->ka", J, r) * w[:, None]
        bad = ~ok
        H[bad], e[bad] = 0.0, 0.0
        x = X[P["ol"]]
        zero = torch.zeros_like(x[:, 0])
        cross = torch.stack([zero, -x[:, 2], x[:, 1], x[:, 2], zero, -x[:, 0], -x[:, 1], x[:, 0], zero],
                            -1).reshape(-1, 3, 3)
        eye = torch.eye(3, device=DEVICE, dtype=F64).expand(x.shape[0], 3, 3)
        self.B = torch.cat([eye, -cross], 2)               # J_p = J_l [I | -[X]x]
        self.H, self.e = H, e
        self.Hl = torch.zeros(self.m, 3, 3, device=DEVICE, dtype=F64).index_add_(0, P["ol"], H)
        self.gl = torch.zeros(self.m, 3, device=DEVICE, dtype=F64).index_add_(0, P["ol"], e)

    def solve(self, lam):
        P, nv = self.P, self.nv
        eye3, eye6 = torch.eye(3, device=DEVICE, dtype=F64), torch.eye(6, device=DEVICE, dtype=F64)
        Hinv = torch.linalg.inv(self.Hl + lam * eye3)
        free = ~P["pfixed"]
        v = torch.where(free[:, None], torch.einsum("mab,mb->ma", Hinv, self.gl), torch.zeros_like(self.gl))
        dp = torch.zeros(nv, 6, device=DEVICE, dtype=F64)
        if nv:
            on = torch.nonzero(self.slot[P["op"]] >= 0).reshape(-1)
            slot = self.slot[P["op"][on]]
            B, H = self.B[on], self.H[on]
            W = B.transpose(1, 2) @ H                      # (K,6,3)
            diag = torch.zeros(nv, 6, 6, device=DEVICE, dtype=F64).index_add_(0, slot, W @ B)
            diag += lam * eye6
            rhs = torch.zeros(nv, 6, device=DEVICE, dtype=F64)
            rhs.index_add_(0, slot, torch.einsum("kab,kb->ka", W, v[P["ol"][on]])
                           - torch.einsum("kba,kb->ka", B, self.e[on]))
            S = torch.zeros(nv * nv, 6, 6, device=DEVICE, dtype=F64)
            Wv = self.B[self.obs].transpose(1, 2) @ self.H[self.obs]
            Y = Wv @ Hinv[P["ol"][self.obs]]
            so = self.slot[P["op"][self.obs]]
            for k, j in _pairs(self.off, 1 << 21):
                keep = so[k] >= so[j]
                k, j = k[keep], j[keep]
                S.index_add_(0, so[k] * nv + so[j], Y[k] @ Wv[j].transpose(1, 2), alpha=-1)
            S = S.reshape(nv, nv, 6, 6)
            i = torch.arange(nv, device=DEVICE)
            S[i, i] += diag
            diag = S[i, i].clone()
            S[i, i] = 0.0
            S = S.permute(0, 2, 1, 3).reshape(6 * nv, 6 * nv)
            S = S + S.T
            S.view(nv, 6, nv, 6)[i, :, i, :] = diag
            inv = torch.linalg.inv(diag)
            dp = _pcg(S, rhs.reshape(-1),
                      lambda r: torch.einsum("nab,nb->na", inv, r.reshape(nv, 6)).reshape(-1),
                      MAX_PCG).reshape(nv, 6)
        u = self.gl.clone()
        if nv:
            u.index_add_(0, P["ol"][on], torch.einsum("kab,kb->ka", W.transpose(1, 2), dp[slot]))
        dl = -torch.einsum("mab,mb->ma", Hinv, u)
        return dp, torch.where(free[:, None], dl, torch.zeros_like(dl))


def _pcg(S, b, precondition, cap):
    x, r = torch.zeros_like(b), b.clone()
    z = precondition(r)
    p, rz, bnorm = z.clone(), r @ z, float(b.norm())
    if not bnorm > 0:
        return x
    for _ in range(cap):
        q = S @ p
        pq = p @ q
        if not float(pq) > 0:
            break
        alpha = rz / pq
        x, r = x + alpha * p, r - alpha * q
        if float(r.norm()) <= PCG_TOLERANCE * bnorm:
            break
        z = precondition(r)
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x


def _moved(P, slot, q, t, dp):
    full = torch.zeros(q.shape[0], 6, device=DEVICE, dtype=F64)
    full[slot >= 0] = dp
    rho, w = full[:, :3], full[:, 3:]
    th = w.norm(dim=1, keepdim=True)
    a = torch.where(th > 1e-5, (1 - torch.cos(th)) / (th * th).clamp_min(1e-300), torch.full_like(th, 0.5))
    b = torch.where(th > 1e-5, (th - torch.sin(th)) / (th ** 3).clamp_min(1e-300), torch.full_like(th, 1 / 6))
    wr = torch.linalg.cross(w, rho)
    te = rho + a * wr + b * torch.linalg.cross(w, wr)
    return _quat_mul(q, _axis_angle(w)), torch.einsum("nij,nj->ni", _rotation(q), te) + t


def _lm(P, q, t, X, kernel, p, iterations, relative=RELATIVE_COST_TOLERANCE, system=None):
    """(initial cost, final cost, q, t, X) of the reference's LM control."""
    system = system or _System(P)
    cost, bad = _cost(P, q, t, X, kernel, p)
    initial, lam, fresh = cost, 1e-4, True
    for _ in range(iterations):
        if fresh:
            system.linearise(q, t, X, kernel, p)
        dp, dl = system.solve(lam)
        q1, t1 = _moved(P, system.slot, q, t, dp)
        X1 = X + dl
        new, bad1 = _cost(P, q1, t1, X1, kernel, p)
        fresh = new < cost and bad1 <= bad
        if not fresh:
            lam = min(lam * 10, 1e12)
            if lam >= 1e12:
                break
            continue
        before, cost, bad, q, t, X = cost, new, bad1, q1, t1, X1
        lam = max(lam * 0.1, 1e-9)
        pose = float(dp.norm(dim=1).max()) if dp.numel() else 0.0
        land = float(dl.norm(dim=1).max())
        if (pose < 1e-7 and land < 1e-7) or abs(before - cost) < 1e-9:
            break
        if relative is not None and (before - cost) / max(abs(before), 2.2e-16) < relative:
            break
    return initial, cost, q, t, X


def _gnc(P, c=3.0, factor=2.0, inner=3):
    q, t, X, system = P["q"], P["t"], P["X"], _System(P)

    def squared():
        r, _, ok = _residuals(P, q, t, X)
        return torch.where(ok, (r * r).sum(1), torch.full_like(r[:, 0], float("nan")))

    def weight(s, mu):
        lo, hi = mu / (mu + 1) * c * c, (mu + 1) / mu * c * c
        w = (c * c * mu * (mu + 1) / s.clamp_min(1e-300)).sqrt() - mu
        return torch.where(s <= lo, torch.ones_like(s), torch.where(s >= hi, torch.zeros_like(s), w))

    s = squared()
    initial, top = float(s.nansum()), float(s.nan_to_num(0.0).max())
    mu = min(max(c * c / max(2 * top - c * c, 1e-300), 2.3e-308), 200.0)
    for _ in range(100):
        s, last = squared(), mu >= 200.0
        P["w"] = torch.where(s.isnan(), torch.ones_like(s), weight(s, mu))
        _, _, q, t, X = _lm(P, q, t, X, "none", 0.0, inner, system=system)
        if last:
            break
        mu = min(mu * factor, 200.0)
    s = squared()
    w = torch.where(s.isnan(), s, weight(s, mu))
    return {"initial": initial, "final": float((w * s).nansum()), "q": q, "t": t, "X": X, "weights": w}


def exact(case, seed):
    kind = case["kind"]
    if kind == "reduced":
        D = _reduced(case, seed)
        S = _dense_blocks(D["diag"], D["a"], D["b"], D["off"])
        return {"x": _reduced_pcg(S, D["rhs"], torch.linalg.inv(D["diag"]))}
    if kind == "trial":
        E = _elimination(case, seed)
        blocks, n, g = E["blocks"], E["n"], E["group"]
        m = -(-n // g)
        sums = torch.zeros(m * m, 6, 6, device=DEVICE, dtype=F64)
        sums.index_add_(0, E["a"] // g * m + E["b"] // g, blocks)
        S = _dense_blocks(E["diag"], E["a"], E["b"], blocks)
        return {"x": _reduced_pcg(S, E["rhs"], None, E),
                "run_blocks": blocks[E["run_edges"]].transpose(1, 2).reshape(-1, 36),
                "coarse_sums": sums.transpose(1, 2).reshape(-1, 36)}
    problems = _problems(case, seed)
    if kind == "cost":
        P = problems[0]
        c, bad = _cost(P, P["q"], P["t"], P["X"], "huber", 1.0)
        return {"cost": torch.tensor([c], dtype=F64), "counts": torch.tensor([bad, 0])}
    if kind == "gnc":
        return _gnc(problems[0])
    robust = case.get("robust", "huber")
    p = {"huber": 1.0, "cauchy": 2.0, "none": 0.0}[robust]
    got = [_lm(P, P["q"], P["t"], P["X"], robust, p, case["iterations"]) for P in problems]
    if kind == "batch":
        col = list(zip(*got))
        return {"initial": torch.tensor(col[0], dtype=F64), "final": torch.tensor(col[1], dtype=F64),
                "q": torch.cat(col[2]), "t": torch.cat(col[3]), "X": torch.cat(col[4])}
    out = dict(zip(("initial", "final", "q", "t", "X"), got[0]))
    if kind == "pose":
        del out["X"]
    return out


def _reduced_pcg(S, rhs, jacobi, E=None):
    n = S.shape[0]

    def precondition(r):
        r = r.reshape(n, 6)
        if jacobi is not None:
            return torch.einsum("nab,nb->na", jacobi, r).reshape(-1)
        z = torch.empty_like(r)
        for f, inv in E["runs"]:
            k = inv.shape[0] // 6
            z[f:f + k] = (inv @ r[f:f + k].reshape(-1)).reshape(k, 6)
        g = torch.arange(n, device=DEVICE) // E["group"]
        rc = torch.zeros(int(g[-1]) + 1, 6, device=DEVICE, dtype=F64).index_add_(0, g, r)
        return (z + (E["coarse"] @ rc.reshape(-1)).reshape(-1, 6)[g]).reshape(-1)

    dense = S.permute(0, 2, 1, 3).reshape(6 * n, 6 * n)
    return _pcg(dense, rhs.reshape(-1), precondition, 500).reshape(n, 6)
