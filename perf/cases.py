"""The work this framework is used for, as measurable cases.

The cases follow HI-SLAM2's runtime: the frontend builds correlation volumes for new
edges, looks them up and solves a 25-keyframe window; the backend correlates chunks of
edges on the fly and solves all keyframes at once (SE3 ``ba`` or Sim3 ``pgba``); keyframe
decisions need ``frame_distance`` over many pairs; the mono prior is aligned by ``JDSA``;
training differentiates the lookup and one bundle-adjustment step; and many independent
windows are solved as one batch.  Shapes are those of :mod:`hislam2_b200.synth`
(1/8-resolution grids of 344x616, 384x512 and 240x320 images, 128 feature channels, 4
levels) and generic ragged ones.  Disparities are smooth per-frame fields, camera poses
scatter by a few centimetres and degrees, flow targets carry half a pixel of noise.
"""

import math
import os
import random
import sys

import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hi-slam2_b200"))

import droid_backends  # noqa: E402
from hislam2_b200 import autotune, backends, corr, diff, mono  # noqa: E402

DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}
LEVELS = 4
CHANNELS = 128
MIN_DEPTH = 0.25


def listed():
    return [
        # the smallest solve: a starting clip of 8 keyframes, where launches and latency count
        dict(name="ba_clip8", kind="ba", keyframes=8, ht=48, wd=64, edges=24, t0=2, iters=2, lm=1e-4, ep=0.1,
             outliers=0.0, motion_only=False),
        # the frontend's window, solved after every update of the recurrent network
        dict(name="ba_frontend25", kind="ba", keyframes=25, ht=43, wd=77, edges=258, t0=2, iters=4, lm=1e-4, ep=0.1,
             outliers=0.0, motion_only=False),
        # global bundle adjustment of a long sequence (the backend, and the largest solve)
        dict(name="ba_backend300", kind="ba", keyframes=300, ht=43, wd=77, edges=6000, t0=10, iters=8, lm=1e-5,
             ep=1e-2, outliers=0.05, motion_only=False),
        # many independent windows of uneven sizes solved together (offline reconstruction, evaluation)
        dict(name="ba_batch64", kind="ba_batch", windows=64, iters=4, lm=1e-4, ep=0.1),
        # one differentiable step on a training clip, forward and backward
        dict(name="ba_train7", kind="ba_train", keyframes=7, ht=48, wd=64, edges=42, t0=2, lm=1e-4, ep=0.1),
        # one Sim3 step with relative-pose factors after a loop closure
        dict(name="pgba_backend300", kind="pgba", keyframes=300, ht=43, wd=77, edges=6000, t0=10, factors=600,
             lm=1e-5, ep=1e-2),
        # the frontend's correlation volumes for the edges a keyframe brings
        dict(name="corr_build48", kind="corr_build", keyframes=25, ht=43, wd=77, edges=48, dtype="float16"),
        # the frontend's lookup of all its edges, once per update
        dict(name="corr_lookup258", kind="corr_lookup", keyframes=25, ht=43, wd=77, edges=258, radius=4,
             dtype="float16"),
        # the backend's on-the-fly correlation of one chunk (the edges of two source keyframes)
        dict(name="altcorr_chunk40", kind="altcorr", keyframes=300, ht=43, wd=77, edges=40, radius=3,
             dtype="float16"),
        # the differentiable lookup on two training clips of 7 frames, forward and backward
        dict(name="corr_train84", kind="corr_train", keyframes=7, ht=48, wd=64, edges=84, radius=4, dtype="float16"),
        # keyframe proximity: every ordered pair of a long sequence
        dict(name="distance300", kind="distance", keyframes=300, ht=43, wd=77, pairs=90000, beta=0.3),
        # mono-prior depth and scale alignment of the frontend's window
        dict(name="jdsa_frontend25", kind="jdsa", keyframes=25, ht=43, wd=77, edges=258, grid=2, alpha=0.01),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng):
    wd = rng.randint(32, 80)
    return dict(ht=min(rng.randint(24, 60), 3400 // wd), wd=wd)


def draw(rng):
    kind = rng.choice(["ba", "ba", "ba_batch", "ba_train", "pgba", "corr_build", "corr_lookup", "altcorr",
                       "corr_train", "distance", "jdsa"])
    dtype = rng.choice(["float16", "bfloat16"])
    c = dict(kind=kind)
    if kind == "ba":
        K = _log(rng, 6, 300)
        c.update(_grid(rng), keyframes=K, edges=min(6000, K * (K - 1), int(K * rng.uniform(4, 20))),
                 t0=rng.randint(1, max(1, K // 5)), iters=rng.randint(1, 8), lm=1e-4, ep=rng.choice([0.1, 1e-2]),
                 outliers=rng.choice([0.0, 0.05]), motion_only=rng.random() < 0.15)
    elif kind == "ba_batch":
        c.update(windows=_log(rng, 4, 64), iters=rng.randint(1, 4), lm=1e-4, ep=0.1)
    elif kind == "ba_train":
        K = rng.randint(5, 16)
        c.update(_grid(rng), keyframes=K, edges=min(K * (K - 1), K * rng.randint(4, 8)), t0=rng.randint(1, 2),
                 lm=1e-4, ep=0.1)
    elif kind == "pgba":
        K = _log(rng, 30, 300)
        c.update(_grid(rng), keyframes=K, edges=int(K * rng.uniform(6, 20)), t0=rng.randint(1, K // 5),
                 factors=rng.randint(K // 2, 2 * K), lm=1e-5, ep=1e-2)
    elif kind == "corr_build":
        c.update(_grid(rng), keyframes=25, edges=_log(rng, 4, 96), dtype=dtype)
    elif kind == "corr_lookup":
        c.update(_grid(rng), keyframes=25, edges=_log(rng, 12, 258), radius=rng.choice([3, 4]), dtype=dtype)
    elif kind == "altcorr":
        c.update(_grid(rng), keyframes=_log(rng, 30, 300), edges=_log(rng, 8, 200), radius=rng.choice([3, 4]),
                 dtype=dtype)
    elif kind == "corr_train":
        c.update(_grid(rng), keyframes=7, edges=rng.randint(16, 84), radius=rng.choice([3, 4]), dtype=dtype)
    elif kind == "distance":
        K = _log(rng, 12, 300)
        c.update(_grid(rng), keyframes=K, pairs=rng.randint(K, K * K), beta=rng.choice([0.3, 0.5, 0.7]))
    else:
        K = _log(rng, 8, 60)
        c.update(_grid(rng), keyframes=K, edges=min(K * (K - 1), K * rng.randint(5, 12)), grid=rng.choice([2, 3]),
                 alpha=rng.choice([0.01, 0.001]))
    return c


# ------------------------------------------------------------------------- inputs
def _cross(a, b):
    return torch.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                        a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _rot(q, X):
    uv = 2.0 * _cross(q[..., :3].expand(X.shape), X)
    return X + q[..., 3:4] * uv + _cross(q[..., :3].expand(X.shape), uv)


def _qmul(a, b):
    return torch.cat([a[..., 3:4] * b[..., :3] + b[..., 3:4] * a[..., :3] + _cross(a[..., :3], b[..., :3]),
                      a[..., 3:4] * b[..., 3:4] - (a[..., :3] * b[..., :3]).sum(-1, keepdim=True)], -1)


def _exp(xi):
    tau, phi = xi[..., :3], xi[..., 3:]
    th = phi.norm(dim=-1, keepdim=True)
    small = th < 1e-6
    s = torch.where(small, torch.ones_like(th), th)
    k = torch.where(small, 0.5 - th ** 2 / 48, torch.sin(0.5 * s) / s)
    a = torch.where(small, 0.5 - th ** 2 / 24, (1 - torch.cos(s)) / s ** 2)
    b = torch.where(small, 1.0 / 6 - th ** 2 / 120, (s - torch.sin(s)) / s ** 3)
    c = _cross(phi, tau)
    return torch.cat([tau + a * c + b * _cross(phi, c), k * phi, torch.cos(0.5 * th)], -1)


def _compose(a, b):
    return torch.cat([_rot(a[..., 3:7], b[..., :3]) + a[..., :3], _qmul(a[..., 3:7], b[..., 3:7])], -1)


def _intrinsics(ht, wd):
    # the Replica pinhole (600, 600, 599.5, 339.5 at 1200x680) at the grid's resolution
    return torch.tensor([wd / 2.0, 600.0 * ht / 680.0, 599.5 * wd / 1200.0, 339.5 * ht / 680.0], dtype=torch.float64,
                        device="cuda")


def _relative(poses, ii, jj):
    """t, q, s of Gj Gi^-1 for poses [N, 7] (SE3) or [N, 8] (Sim3)."""
    pi, pj = poses[ii], poses[jj]
    q = _qmul(pj[:, 3:7], torch.cat([-pi[:, 3:6], pi[:, 6:7]], -1))
    s = pj[:, 7:8] / pi[:, 7:8] if poses.shape[1] == 8 else torch.ones_like(q[:, :1])
    return pj[:, :3] - s * _rot(q, pi[:, :3]), q, s


def _rays(intr, ht, wd):
    v, u = torch.meshgrid(torch.arange(ht, dtype=torch.float64, device="cuda"),
                          torch.arange(wd, dtype=torch.float64, device="cuda"), indexing="ij")
    u, v = u.reshape(-1), v.reshape(-1)
    return u, v, torch.stack([(u - intr[2]) / intr[0], (v - intr[3]) / intr[1], torch.ones_like(u)], -1)


def _project(poses, disps, intr, ii, jj):
    """Where the pixels of frames ii fall in frames jj: [E, HW, 2] in 64 bits, 256 edges at a time."""
    K, ht, wd = disps.shape
    _, _, X = _rays(intr, ht, wd)
    out = []
    for s in range(0, len(ii), 256):
        t, q, sc = _relative(poses, ii[s:s + 256], jj[s:s + 256])
        Y = sc[:, None] * _rot(q[:, None], X[None].expand(len(t), -1, 3)) \
            + disps.reshape(K, -1)[ii[s:s + 256], :, None] * t[:, None]
        out.append(intr[:2] * Y[..., :2] / Y[..., 2:3] + intr[2:])
    return torch.cat(out)


def _edges(K, count, radius, rnd):
    """`count` ordered pairs: neighbours up to `radius` first, then loop pairs in both directions."""
    e = [(i, j) for d in range(1, radius + 1) for i in range(K) for j in (i + d, i - d) if 0 <= j < K][:count]
    seen = set(e)
    while len(e) < min(count, K * (K - 1)):
        i, j = rnd.randrange(K), rnd.randrange(K)
        for p in ((i, j), (j, i)):
            if i != j and p not in seen and len(e) < count:
                seen.add(p)
                e.append(p)
    ij = torch.tensor(e, dtype=torch.int64, device="cuda")
    return ij[:, 0].contiguous(), ij[:, 1].contiguous()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")


def _smooth(g, K, ht, wd, lo, hi):
    field = lo + (hi - lo) * _rand(g, K, 1, ht // 8 + 2, wd // 8 + 2)
    return F.interpolate(field, size=(ht, wd), mode="bilinear", align_corners=True)[:, 0].contiguous()


def _scene(c, seed, edges=True):
    g, rnd = _gen(seed), random.Random(seed)
    K, ht, wd = c["keyframes"], c["ht"], c["wd"]
    s = dict(g=g, intr=_intrinsics(ht, wd), poses=_exp(0.05 * _randn(g, K, 6)), disps=_smooth(g, K, ht, wd, 0.1, 2.0))
    if edges:
        s["ii"], s["jj"] = _edges(K, c["edges"], 3 if K < 100 else 2, rnd)
    return s


def _solve_inputs(c, seed):
    """The arguments of a bundle adjustment: poses off by a hundredth, targets off by half a pixel."""
    s = _scene(c, seed)
    g, ii, jj, t0 = s["g"], s["ii"], s["jj"], c["t0"]
    K, ht, wd = s["disps"].shape
    E = len(ii)
    xy = _project(s["poses"], s["disps"], s["intr"], ii, jj)
    targets = (xy + 0.5 * _randn(g, *xy.shape)).float()
    weights = _rand(g, *xy.shape).float()
    if c.get("outliers"):
        bad = _rand(g, E, ht * wd, 1) < c["outliers"]
        targets = torch.where(bad, targets + (40 * _rand(g, *xy.shape) - 20).float(), targets)
        weights = torch.where(bad, torch.zeros_like(weights), weights)
    del xy
    poses = s["poses"].clone()
    poses[t0:] = _compose(_exp(0.01 * _randn(g, K - t0, 6)), s["poses"][t0:])
    M = len(torch.unique(torch.cat([torch.arange(t0, K, device="cuda"), ii])))
    return dict(g=g, poses=poses.float().contiguous(), disps=s["disps"].float().contiguous(),
                intrinsics=s["intr"].float(), targets=targets.transpose(1, 2).reshape(E, 2, ht, wd).contiguous(),
                weights=weights.transpose(1, 2).reshape(E, 2, ht, wd).contiguous(),
                eta=(2e-3 * _rand(g, M, ht, wd) + 1e-4).float(), ii=ii, jj=jj, t0=t0, t1=K)


def _features(g, K, ht, wd, dtype):
    return (_randn(g, K, CHANNELS, ht, wd) / math.sqrt(CHANNELS)).to(DTYPES[dtype])


def _corr_inputs(c, seed, source=None):
    """Features and the coordinates that an update looks up: the reprojection, off by a pixel."""
    s = _scene(c, seed, edges=source is None)
    K, ht, wd = s["disps"].shape
    if source is not None:
        s["ii"], s["jj"] = source(s["g"], K)
    coords = _project(s["poses"], s["disps"], s["intr"], s["ii"], s["jj"])
    coords = (coords + _randn(s["g"], *coords.shape)).float().reshape(-1, ht, wd, 2)
    return dict(g=s["g"], fmaps=_features(s["g"], K, ht, wd, c["dtype"]), ii=s["ii"], jj=s["jj"], coords=coords)


def _chunk(c):
    """The edges of a backend chunk: two neighbouring source keyframes, any targets."""
    def source(g, K):
        i = int(torch.randint(0, K - 1, (1,), generator=g, device="cuda"))
        ii = i + torch.arange(c["edges"], device="cuda") * 2 // c["edges"]
        jj = torch.randint(0, K, (c["edges"],), generator=g, device="cuda")
        return ii, jj
    return source


def _windows(c, seed):
    """Windows of uneven sizes; the sizes belong to the case, the values to the seed."""
    rnd = random.Random(c["windows"])
    out = []
    for k in range(c["windows"]):
        ht, wd = rnd.choice([(43, 77), (30, 40)])
        K = rnd.randint(8, 40)
        E = min(K * (K - 1), max(rnd.randint(20, 500), K))
        out.append(dict(keyframes=K, ht=ht, wd=wd, edges=E, t0=1))
    return [(w, _solve_inputs(w, seed * 1000 + k) if seed is not None else None) for k, w in enumerate(out)]


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("ba", "pgba"):
        s = _solve_inputs(c, seed)
        if kind == "pgba":
            g, K, N = s["g"], c["keyframes"], c["factors"]
            s["poses"] = torch.cat([s["poses"], torch.exp(0.05 * _randn(g, K, 1)).float()], 1).contiguous()
            s["iip"] = torch.randint(0, K, (N,), generator=g, device="cuda")
            s["jjp"] = torch.randint(c["t0"], K, (N,), generator=g, device="cuda")
            J, W = _randn(g, 2, N, 7, 7), torch.diag_embed(10.0 ** (3 + 3 * _rand(g, N, 7)))
            wJ = 1e-3 * J.transpose(2, 3) @ W
            r = 0.01 * _randn(g, N, 7, 1)
            s["Hsp"] = torch.stack([wJ[0] @ J[0], wJ[0] @ J[1], wJ[1] @ J[0], wJ[1] @ J[1]])[:, None].float().contiguous()
            s["vsp"] = -torch.stack([wJ[0] @ r, wJ[1] @ r]).squeeze(-1)[:, None].float().contiguous()
    elif kind == "ba_batch":
        s = dict(windows=[w for _, w in _windows(c, seed)])
        ws = s["windows"]
        s["poses0"], s["disps0"] = [w["poses"].clone() for w in ws], [w["disps"].clone() for w in ws]
        s["plan"] = backends.BABatch(ws, c["lm"], c["ep"], **autotune.best("batch64"))
    elif kind == "ba_train":
        s = _solve_inputs(c, seed)
        for k in ("targets", "weights", "eta"):
            s[k].requires_grad_(True)
        s["grad_dx"] = _randn(s["g"], c["keyframes"] - c["t0"], 6).float()
        s["grad_dz"] = _randn(s["g"], len(s["eta"]), c["ht"] * c["wd"]).float()
    elif kind == "corr_build":
        s = _corr_inputs(c, seed)
        s["f1"], s["f2"] = s["fmaps"][s["ii"]][None], s["fmaps"][s["jj"]][None]
    elif kind == "corr_lookup":
        s = _corr_inputs(c, seed)
        s["block"] = corr.CorrBlock(s["fmaps"][s["ii"]][None], s["fmaps"][s["jj"]][None], LEVELS, c["radius"])
        s["coords"] = s["coords"][None]
    elif kind == "altcorr":
        s = _corr_inputs(c, seed, _chunk(c))
        s["block"] = corr.AltCorrBlock(s["fmaps"][None], LEVELS, c["radius"])
        s["coords"] = s["coords"][None]
    elif kind == "corr_train":
        s = _corr_inputs(dict(c, edges=min(c["edges"], 42)), seed)
        again = torch.arange(c["edges"], device="cuda") % len(s["ii"])
        s["ii"], s["jj"] = s["ii"][again], s["jj"][again]
        s["coords"] = (s["coords"][again] + 0.5 * _randn(s["g"], c["edges"], c["ht"], c["wd"], 2).float())[None]
        s["f1"] = s["fmaps"][s["ii"]][None].requires_grad_(True)
        s["f2"] = s["fmaps"][s["jj"]][None].requires_grad_(True)
        s["grad"] = _randn(s["g"], 1, c["edges"], LEVELS * (2 * c["radius"] + 1) ** 2, c["ht"], c["wd"]).to(
            DTYPES[c["dtype"]])
    elif kind == "distance":
        s = _scene(c, seed, edges=False)
        K, N = c["keyframes"], c["pairs"]
        at = torch.arange(N, device="cuda") if N == K * K else torch.randperm(K * K, generator=s["g"], device="cuda")[:N]
        s = dict(poses=s["poses"].float().contiguous(), disps=s["disps"].float().contiguous(),
                 intrinsics=s["intr"].float(), ii=(at // K).contiguous(), jj=(at % K).contiguous())
    else:
        s = _solve_inputs(dict(c, t0=0), seed)
        g, K, ht, wd = s["g"], c["keyframes"], c["ht"], c["wd"]
        prior = s["disps"].double() / _smooth(g, K, ht, wd, 0.6, 1.4) * (1 + 0.02 * _randn(g, K, ht, wd))
        s["prior"] = torch.where(_rand(g, K, ht, wd) < 0.1, torch.zeros_like(prior), prior).float().contiguous()
        s["scales"] = (1 + 0.05 * _randn(g, K, c["grid"], c["grid"])).float().contiguous()
    s.pop("g", None)
    s["case"] = c
    return s


# ---------------------------------------------------------------------------- run
def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "ba":
        # ba moves poses and disparities in place: each pass starts from the same ones.  A caller reads those; the last
        # increment is what convergence left over.
        poses, disps = s["poses"].clone(), s["disps"].clone()
        droid_backends.ba(poses, disps, s["intrinsics"], s["targets"], s["weights"], s["eta"], s["ii"], s["jj"],
                          s["t0"], s["t1"], c["iters"], c["lm"], c["ep"], c["motion_only"])
        return poses, disps
    if kind == "ba_batch":
        torch._foreach_copy_([w["poses"] for w in s["windows"]], s["poses0"])
        torch._foreach_copy_([w["disps"] for w in s["windows"]], s["disps0"])
        s["plan"].run(c["iters"])
        s["plan"].check()
        return (torch.cat([w["poses"] for w in s["windows"]]),
                torch.cat([w["disps"].reshape(-1) for w in s["windows"]]))
    if kind == "ba_train":
        dx, dz = diff.ba_step(s["targets"], s["weights"], s["eta"], s["poses"], s["disps"], s["intrinsics"], s["ii"],
                              s["jj"], s["t0"], s["t1"], c["lm"], c["ep"])
        grads = torch.autograd.grad([dx, dz], [s["targets"], s["weights"], s["eta"]], [s["grad_dx"], s["grad_dz"]])
        return dx, dz, list(grads)
    if kind == "pgba":
        disps = s["disps"].clone()
        dx, dz = droid_backends.pgba(s["poses"], disps, s["intrinsics"], s["targets"], s["weights"], s["eta"],
                                     s["Hsp"], s["vsp"], s["ii"], s["jj"], s["iip"], s["jjp"], s["t0"], s["t1"],
                                     c["lm"], c["ep"])
        return disps, dx, dz
    if kind == "corr_build":
        return corr.CorrBlock(s["f1"], s["f2"], LEVELS).corr_pyramid
    if kind == "corr_lookup":
        return s["block"](s["coords"])
    if kind == "altcorr":
        return s["block"](s["coords"], s["ii"], s["jj"])
    if kind == "corr_train":
        out = corr.CorrLookup.apply(s["f1"], s["f2"], s["coords"], c["radius"], LEVELS)
        return out, list(torch.autograd.grad(out, [s["f1"], s["f2"]], s["grad"]))
    if kind == "distance":
        return droid_backends.frame_distance(s["poses"], s["disps"], s["intrinsics"], s["ii"], s["jj"], c["beta"])
    return list(mono.JDSA(s["targets"], s["weights"], s["eta"], s["poses"], s["disps"], s["intrinsics"], s["prior"],
                          s["scales"].clone(), s["ii"], s["jj"], c["alpha"]))


# --------------------------------------------------------------------------- work
def _solve_work(K, E, HW, P, iters, D, motion_only=False):
    rows = E / K + 1                                  # pose rows coupled to one depth frame
    gram = 0 if motion_only else K * (D * rows) * (D * rows + 2) * HW
    flops = iters * (E * HW * (160 if motion_only else 250) + gram + (D * P) ** 3 / 3)
    return dict(bytes=E * HW * 16 + K * HW * 12 + K * 56 + E * 16, flops=flops)


def work(case):
    c, kind = case, case["kind"]
    if kind == "ba_batch":
        each = [_solve_work(w["keyframes"], w["edges"], w["ht"] * w["wd"], w["keyframes"] - 1, c["iters"], 6)
                for w, _ in _windows(c, None)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    K, HW = c["keyframes"], c["ht"] * c["wd"]
    if kind in ("ba", "ba_train", "pgba"):
        w = _solve_work(K, c["edges"], HW, K - c["t0"], c.get("iters", 1), 7 if kind == "pgba" else 6,
                        c.get("motion_only", False))
        if kind == "ba_train":
            w = dict(bytes=2 * w["bytes"] + c["edges"] * HW * 16, flops=3 * w["flops"])
        return w
    if kind == "distance":
        return dict(bytes=K * (HW * 4 + 28) + c["pairs"] * 20, flops=c["pairs"] * HW * 60)
    E = c["edges"]
    if kind == "jdsa":
        return dict(bytes=E * HW * 16 + K * HW * 20, flops=E * HW * 60 + K * HW * 8 * c["grid"] ** 2)
    areas = [(c["ht"] >> i) * (c["wd"] >> i) for i in range(LEVELS)]
    if kind == "corr_build":
        return dict(bytes=2 * E * HW * CHANNELS * 2 + E * HW * sum(areas) * 2, flops=2 * CHANNELS * E * HW * HW)
    r, out = c["radius"], E * HW * LEVELS * (2 * c["radius"] + 1) ** 2
    taps = E * HW * LEVELS * (2 * r + 2) ** 2
    if kind == "corr_lookup":
        return dict(bytes=taps * 2 + out * 2 + E * HW * 8, flops=out * 8)
    if kind == "altcorr":
        frames = min(K, E) * sum(areas) + 2 * HW
        return dict(bytes=frames * CHANNELS * 2 + out * 2 + E * HW * 8, flops=taps * CHANNELS * 2)
    return dict(bytes=4 * E * HW * CHANNELS * 2 + out * 4 + E * HW * 8, flops=3 * taps * CHANNELS * 2)


# -------------------------------------------------- the same results in 64 bits, from plain torch
def _exact_step(poses, disps, intr, targets, weights, eta, ii, jj, t0, t1, lm, ep, motion_only=False, prior=None):
    """One damped Gauss-Newton step on poses [K, 7] or [K, 8] and disparities -> dx, dz, kx."""
    K, ht, wd = disps.shape
    HW, E, P = ht * wd, len(ii), t1 - t0
    D = poses.shape[1] - 1
    fx, fy = intr[0], intr[1]
    _, _, X = _rays(intr, ht, wd)
    ii_exp = torch.cat([torch.arange(t0, t1, device="cuda"), ii])
    jj_exp = torch.cat([torch.arange(t0, t1, device="cuda"), jj])
    kx, kk = torch.unique(ii_exp, return_inverse=True)
    M = len(kx)
    A = torch.zeros(P * P, D, D, dtype=torch.float64, device="cuda")
    b = torch.zeros(P, D, dtype=torch.float64, device="cuda")
    C = torch.zeros(M, HW, dtype=torch.float64, device="cuda")
    w = torch.zeros_like(C)
    Ei = torch.zeros(P, D, HW, dtype=torch.float64, device="cuda")
    Eij = []

    def add(rows, cols, blocks, A):
        ok = (rows >= 0) & (cols >= 0)
        return A.index_add(0, rows[ok] * P + cols[ok], blocks[ok])

    for s in range(0, E, 256):
        ie, je = ii[s:s + 256], jj[s:s + 256]
        n = len(ie)
        t, q, sc = _relative(poses, ie, je)
        d = disps.reshape(K, HW)[ie]
        Y = sc[:, None] * _rot(q[:, None], X[None].expand(n, HW, 3)) + d[..., None] * t[:, None]
        x, y, z = Y.unbind(-1)
        ok = z >= MIN_DEPTH
        zs = torch.where(ok, z, torch.ones_like(z))
        g = torch.where(ok, 1 / zs, torch.zeros_like(z))
        tw, ww = targets[s:s + 256].reshape(n, 2, HW), weights[s:s + 256].reshape(n, 2, HW)
        res = [tw[:, 0] - (fx * x * g + intr[2]), tw[:, 1] - (fy * y * g + intr[3])]
        wt = [torch.where(ok, 0.001 * ww[:, k], torch.zeros_like(z)) for k in (0, 1)]
        o = torch.zeros_like(g)
        z0 = torch.where(ok, z, o)
        Jp = [(fx * g, o, -fx * x * g * g), (o, fy * g, -fy * y * g * g)]
        live = (ie != je).double()[:, None]
        H = Hv = Eii_c = Eij_c = 0
        for (p0, p1, p2), r, wk in zip(Jp, res, wt):
            J = [p0 * d, p1 * d, p2 * d, -p1 * z0 + p2 * y, p0 * z0 - p2 * x, -p0 * y + p1 * x]
            if D == 7:
                J.append(p0 * x + p1 * y + p2 * z0)
            J = torch.stack(J, -1)
            Jz = p0 * t[:, 0:1] + p1 * t[:, 1:2] + p2 * t[:, 2:3]
            C = C.index_add(0, kk[P + s:P + s + n], wk * Jz * Jz)
            w = w.index_add(0, kk[P + s:P + s + n], wk * r * Jz)
            qi = torch.cat([-q[:, :3], q[:, 3:]], -1)[:, None]
            a, tb = J[..., :3], t[:, None].expand(n, HW, 3)
            parts = [sc[:, None] * _rot(qi, a), sc[:, None] * _rot(qi, J[..., 3:6] - _cross(tb, a))]
            if D == 7:
                parts[1] = parts[1] + J[..., 6:7] * tb
                parts.append(J[..., 6:7])
            Jx = torch.cat([-torch.cat(parts, -1), J], -1)
            wl = (wk * live)[..., None]
            H = H + (Jx * wl).transpose(1, 2) @ Jx
            Hv = Hv + ((Jx * wl) * r[..., None]).sum(1)
            Eii_c = Eii_c + (wl * Jz[..., None] * Jx[..., :D]).transpose(1, 2)
            Eij_c = Eij_c + (wl * Jz[..., None] * Jx[..., D:]).transpose(1, 2)
        ri, rj = ie - t0, je - t0
        for rows, cols, blk in ((ri, ri, H[:, :D, :D]), (ri, rj, H[:, :D, D:]), (rj, ri, H[:, D:, :D]),
                                (rj, rj, H[:, D:, D:])):
            A = add(rows, cols, blk, A)
        b = b.index_add(0, ri[ri >= 0], Hv[ri >= 0, :D]).index_add(0, rj[rj >= 0], Hv[rj >= 0, D:])
        Ei = Ei.index_add(0, ri[ri >= 0], Eii_c[ri >= 0])
        Eij.append(Eij_c)
    if prior is not None:
        Hs, vs, ip, jp = prior
        for rows, cols, blk in ((ip, ip, Hs[0]), (ip, jp, Hs[1]), (jp, ip, Hs[2]), (jp, jp, Hs[3])):
            A = add(rows - t0, cols - t0, blk, A)
        for rows, v in ((ip - t0, vs[0]), (jp - t0, vs[1])):
            b = b.index_add(0, rows[rows >= 0], v[rows >= 0])
    Er = torch.cat([Ei] + Eij)
    Q = 1 / (C + eta.reshape(-1, HW))
    if not motion_only:
        order = kk.argsort(stable=True)
        for k, rows in enumerate(torch.split(order, torch.bincount(kk, minlength=M).tolist())):
            rows = rows[jj_exp[rows] >= t0]
            p = jj_exp[rows] - t0
            G = Er[rows].reshape(-1, HW)
            S = ((G * Q[k]) @ G.T).reshape(len(rows), D, len(rows), D).transpose(1, 2)
            A = A.index_add(0, (p[:, None] * P + p[None]).reshape(-1), -S.reshape(-1, D, D))
            b = b.index_add(0, p, -((G * (Q[k] * w[k])).sum(1)).reshape(-1, D))
    A = A.reshape(P, P, D, D).transpose(1, 2).reshape(P * D, P * D)
    if prior is not None:
        A = A.tril() + A.tril(-1).T                   # the solver reads the lower triangle
    dg = A.diagonal()
    L = torch.linalg.cholesky(A + torch.diag(ep + lm * dg))
    dx = torch.cholesky_solve(b.reshape(-1, 1), L).reshape(P, D)
    if motion_only:
        return dx, None, kx
    ix = jj_exp - t0
    dw = torch.zeros_like(C)
    for s in range(0, len(ix), 512):
        keep = (ix[s:s + 512] > 0).nonzero()[:, 0] + s
        dw = dw.index_add(0, kk[keep], (Er[keep] * dx[ix[keep]][..., None]).sum(1))
    return dx, Q * (w - dw), kx


def _exact_ba(s, c, motion_only=False):
    p, d = s["poses"].double(), s["disps"].double()
    args = [s["intrinsics"].double(), s["targets"].double(), s["weights"].double(), s["eta"].double()]
    t0, t1 = s["t0"], s["t1"]
    for _ in range(c["iters"]):
        dx, dz, kx = _exact_step(p, d, *args, s["ii"], s["jj"], t0, t1, c["lm"], c["ep"], motion_only)
        p = torch.cat([p[:t0], _compose(_exp(dx), p[t0:t1]), p[t1:]])
        if not motion_only:
            d = d.index_add(0, kx, dz.reshape(-1, *d.shape[1:]))
    return p, d


def _window_sample(vol, coords, r):
    """Bilinear (2r+1)^2 lookup around coords [2, HW] of vol [HW, h, w], x slowest -> [(2r+1)^2, HW]."""
    N, h, w = vol.shape
    x0, y0 = torch.floor(coords)
    fx, fy = (coords[0] - x0)[:, None, None], (coords[1] - y0)[:, None, None]
    k = torch.arange(-r, r + 2, device="cuda")
    x, y = (x0.long()[:, None] + k)[:, :, None], (y0.long()[:, None] + k)[:, None, :]
    ok = (x >= 0) & (x < w) & (y >= 0) & (y < h)
    at = (y.clamp(0, h - 1) * w + x.clamp(0, w - 1)).reshape(N, -1)
    V = torch.gather(vol.reshape(N, -1), 1, at).reshape(N, len(k), len(k)) * ok
    out = ((1 - fx) * (1 - fy) * V[:, :-1, :-1] + (1 - fx) * fy * V[:, :-1, 1:] + fx * (1 - fy) * V[:, 1:, :-1]
           + fx * fy * V[:, 1:, 1:])
    return out.reshape(N, -1).T


def _exact_levels(f1, f2):
    """All-pairs pyramid of one edge in 64 bits: [HW, h, w] for each level."""
    C, h, w = f1.shape
    vol = ((f1.reshape(C, -1) / 4).T @ (f2.reshape(C, -1) / 4)).reshape(-1, h, w)
    out = [vol]
    for _ in range(1, LEVELS):
        vol = F.avg_pool2d(vol[:, None], 2, stride=2)[:, 0]
        out.append(vol)
    return out


def _exact_lookup(f1, f2, coords, r):
    """[L (2r+1)^2, H, W] of one edge; coords [H, W, 2]."""
    H, W, _ = coords.shape
    xy = coords.double().reshape(-1, 2).T
    return torch.cat([_window_sample(v, xy / 2 ** i, r) for i, v in enumerate(_exact_levels(f1, f2))]).reshape(-1, H, W)


def _exact_jdsa(s, c):
    disps, prior, scales = s["disps"].double(), s["prior"].double(), s["scales"].double()
    K, ht, wd = disps.shape
    HW, n, a = ht * wd, c["grid"], c["alpha"]
    intr = s["intrinsics"].double()
    _, _, X = _rays(intr, ht, wd)
    ii, jj = s["ii"], s["jj"]
    C = torch.zeros(K, HW, dtype=torch.float64, device="cuda")
    w = torch.zeros_like(C)
    t, q, _ = _relative(s["poses"].double(), ii, jj)
    Y = _rot(q[:, None], X[None].expand(len(ii), HW, 3)) + disps.reshape(K, HW)[ii][..., None] * t[:, None]
    ok = Y[..., 2] >= MIN_DEPTH
    g = torch.where(ok, 1 / torch.where(ok, Y[..., 2], torch.ones_like(Y[..., 2])), torch.zeros_like(Y[..., 2]))
    for k in (0, 1):
        J = intr[k] * g * (t[:, k:k + 1] - Y[..., k] * g * t[:, 2:3])
        r = s["targets"].double()[:, k].reshape(-1, HW) - (intr[k] * Y[..., k] * g + intr[2 + k])
        wk = torch.where(ok, 0.001 * s["weights"].double()[:, k].reshape(-1, HW), torch.zeros_like(g))
        C.index_add_(0, ii, wk * J * J)
        w.index_add_(0, ii, wk * r * J)
    # bilinear weights of the n x n scale grid at each pixel; the grid's axes are made in 32 bits
    lin = [torch.linspace(0, n - 1 - 1e-6, m).double().cuda() for m in (ht, wd)]
    B = torch.zeros(ht, wd, n, n, dtype=torch.float64, device="cuda")
    gy, gx = torch.meshgrid(lin[0], lin[1], indexing="ij")
    y0, x0 = torch.floor(gy), torch.floor(gx)
    v, u = torch.meshgrid(torch.arange(ht, device="cuda"), torch.arange(wd, device="cuda"), indexing="ij")
    for dy in (0, 1):
        for dx in (0, 1):
            wy = gy - y0 if dy else y0 + 1 - gy
            wx = gx - x0 if dx else x0 + 1 - gx
            B[v, u, y0.long() + dy, x0.long() + dx] = wy * wx
    B = B.reshape(HW, n * n)
    pr = prior.reshape(K, HW)
    m = (pr > 0).double()
    rd = disps.reshape(K, HW) - pr * (scales.reshape(K, -1) @ B.T)
    J = -(m * pr)[..., None] * B[None]
    Cf = C + m * a + (1 - m) * s["eta"].double().reshape(K, HW)
    wf = w - m * a * rd
    Q = 1 / Cf
    H = a * J.transpose(1, 2) @ J
    E = (a * J).transpose(1, 2)
    H = H + torch.diag_embed(0.1 + 1e-4 * H.diagonal(dim1=1, dim2=2))
    S = H - (E * Q[:, None]) @ E.transpose(1, 2)
    rhs = -(E @ rd[..., None]) - E @ (Q * wf)[..., None]
    L = torch.linalg.cholesky(S)
    dso = torch.cholesky_solve(rhs, L)
    dz = Q * (wf - (E.transpose(1, 2) @ dso)[..., 0])
    cov = (torch.linalg.solve_triangular(L, E * Q[:, None], upper=False) ** 2).sum(1) + Q
    d = disps + dz.reshape(K, ht, wd)
    d = torch.where(d > 10, torch.zeros_like(d), d).clamp(min=0.001)
    return [d, scales + dso.reshape(scales.shape), cov]


def _exact_distance(s, c):
    disps, intr, beta = s["disps"].double(), s["intrinsics"].double(), c["beta"]
    K, ht, wd = disps.shape
    u, v, X = _rays(intr, ht, wd)
    out = []
    for k in range(0, c["pairs"], 1500):
        ii, jj = s["ii"][k:k + 1500], s["jj"][k:k + 1500]
        t, q, _ = _relative(s["poses"].double(), ii, jj)
        shift = disps.reshape(K, -1)[ii][..., None] * t[:, None]
        total = valid = 0
        for share, Y in ((beta, _rot(q[:, None], X[None].expand(len(ii), -1, 3)) + shift), (1 - beta, X[None] + shift)):
            xy = intr[:2] * Y[..., :2] / Y[..., 2:3] + intr[2:]
            ok = Y[..., 2] > MIN_DEPTH
            far = ((xy[..., 0] - u) ** 2 + (xy[..., 1] - v) ** 2).sqrt()
            total = total + share * torch.where(ok, far, torch.zeros_like(far)).sum(1)
            valid = valid + share * ok.sum(1)
        out.append(torch.where(valid / (ht * wd) < 0.75, torch.full_like(valid, 1000.0), total / valid))
    return torch.cat(out)


def exact(case, seed):
    c, kind = case, case["kind"]
    with torch.no_grad():
        if kind == "ba_batch":
            each = [_exact_ba(w, c) for _, w in _windows(c, seed)]
            return torch.cat([p for p, _ in each]), torch.cat([d.reshape(-1) for _, d in each])
        s = prepare(case, seed)
        if kind == "ba":
            return _exact_ba(s, c, c["motion_only"])
        if kind == "pgba":
            d = s["disps"].double()
            prior = (s["Hsp"].double()[:, 0], s["vsp"].double()[:, 0], s["iip"], s["jjp"])
            dx, dz, kx = _exact_step(s["poses"].double(), d, s["intrinsics"].double(), s["targets"].double(),
                                     s["weights"].double(), s["eta"].double(), s["ii"], s["jj"], s["t0"], s["t1"],
                                     c["lm"], c["ep"], prior=prior)
            return d.index_add(0, kx, dz.reshape(-1, *d.shape[1:])), dx, dz
        if kind == "corr_build":
            each = [_exact_levels(a.double(), b.double()) for a, b in zip(s["f1"][0], s["f2"][0])]
            return [torch.stack([e[i] for e in each]).reshape(len(each), c["ht"], c["wd"], c["ht"] >> i, c["wd"] >> i)
                    for i in range(LEVELS)]
        if kind in ("corr_lookup", "altcorr"):
            return torch.stack([_exact_lookup(s["fmaps"][i].double(), s["fmaps"][j].double(), xy, c["radius"])
                                for i, j, xy in zip(s["ii"].tolist(), s["jj"].tolist(), s["coords"][0])])[None]
        if kind == "distance":
            return _exact_distance(s, c)
        if kind == "jdsa":
            return _exact_jdsa(s, c)
    if kind == "ba_train":
        leaves = [s[k].detach().double().requires_grad_(True) for k in ("targets", "weights", "eta")]
        dx, dz, _ = _exact_step(s["poses"].double(), s["disps"].double(), s["intrinsics"].double(), *leaves, s["ii"],
                                s["jj"], s["t0"], s["t1"], c["lm"], c["ep"])
        grads = torch.autograd.grad([dx, dz], leaves, [s["grad_dx"].double(), s["grad_dz"].double()])
        return dx.detach(), dz.detach(), list(grads)
    out, grads = [], []
    for k in range(c["edges"]):
        f1, f2 = (s[f][0, k].detach().double().requires_grad_(True) for f in ("f1", "f2"))
        o = _exact_lookup(f1, f2, s["coords"][0, k], c["radius"])
        out.append(o.detach())
        grads.append(torch.autograd.grad(o, [f1, f2], s["grad"][0, k].double()))
    return torch.stack(out)[None], [torch.stack([g[i] for g in grads])[None] for i in (0, 1)]
