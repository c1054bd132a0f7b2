"""Performance cases: the work that a user of the engine has it do, through its public entry points.

listed()        the cases; draw(rng) gives one more of the same ranges
prepare(c, s)   what a program holds before the call (inputs from seed s, on the GPU, and its engine handle)
run(state)      one pass, as a program calls it
work(c)         the bytes and operations the path cannot do without
exact(c, s)     the outputs in 64 bits, in plain torch, without the engine's code (None where it would take too long)

Sizes and settings are those of the benchmark, the tests and the trainer: RenderSession's default tolerances and the
benchmark's 1e-8; thin disk, 1 to 32 frequency bins; 24^2 to 1024^2 frames, odd sides among them; one to a million
network rows; training batches of 128 to 32768 rows.
"""
import math
import os

import numpy as np
import torch

from sirius_b200 import abi
from sirius_b200.engine import Engine, frames_array

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(abi.__file__)), "data", "surrogate_kerr.npy")
DEV = torch.device("cuda", 0)


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # an interactive preview: one small thin-disk frame at RenderSession's tolerances, where latency counts
        dict(name="frame_preview", kind="frame", w=160, h=90, precision="mixed", tol=5e-6, bins=0),
        # the benchmark's frame: thin disk and 16-bin volumetric transfer at 1e-8, image and spectra on the device
        dict(name="frame_spectra", kind="frame", w=1024, h=1024, precision="mixed", tol=1e-8, bins=16),
        # the library's default precision and settings, ragged sides
        dict(name="frame_fp64", kind="frame", w=717, h=405, precision="fp64", tol=5e-6, bins=0),
        # FP64 with volumetric transfer: the reference image a user checks a mixed one against
        dict(name="frame_fp64_spectra", kind="frame", w=384, h=384, precision="fp64", tol=1e-8, bins=16),
        # GeodesicTracer::trace for a batch of host camera rays with full per-ray records, through host memory
        dict(name="rays_host", kind="rays", n=777, tol=1e-8),
        # a heterogeneous batch: Kerr-Newman, Kerr-de Sitter, wormhole and warp-drive frames in one call
        dict(name="batch_families", kind="batch", n=12, lo=64, hi=320, tol=1e-8),
        # an all-sky map with the symplectic integrator and 32 bins (the benchmark's stress configuration, small)
        dict(name="sky_symplectic", kind="sky", w=128, h=64, order=4, bins=32),
        # the surrogate network alone: a small query, and a large one with a ragged last tile
        dict(name="infer_small", kind="infer", n=1000),
        dict(name="infer_large", kind="infer", n=1048576 + 333),
        # a whole surrogate-gated frame: features, gate, network, gated integration, shading, audit
        dict(name="surrogate_frame", kind="surrogate", w=1024, h=1024),
        # the network's training: optimiser steps over a device-resident set (gradients inside), weights read back
        dict(name="train_steps", kind="train", batch=32768, rows=1 << 20, steps=8),
        # lensing magnification of the sky around the hole (no disk): a beam per pixel
        dict(name="beams", kind="beams", w=120, h=68, tol=1e-8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "rays", "batch", "sky", "infer", "infer", "surrogate", "train",
                       "gradient", "beams"])
    if kind == "frame":
        bins = rng.choice([0, 0, 1, 7, 16, 32])
        w = _log(rng, 24, 800)
        h = max(1, int(w * rng.uniform(0.4, 1.2)))
        return dict(kind="frame", w=w, h=h, precision=rng.choice(["mixed", "fp64"]),
                    tol=rng.choice([5e-6, 1e-7, 1e-8]), bins=bins)
    if kind == "rays":
        return dict(kind="rays", n=_log(rng, 1, 20000), tol=rng.choice([5e-6, 1e-8]))
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(2, 16), lo=32, hi=rng.randint(64, 320), tol=rng.choice([1e-7, 1e-8]))
    if kind == "sky":
        w = 2 * rng.randint(8, 64)
        return dict(kind="sky", w=w, h=w // 2, order=rng.choice([4, 4, 6]), bins=rng.choice([0, 16, 32]))
    if kind == "infer":
        return dict(kind="infer", n=_log(rng, 1, 1 << 20))
    if kind == "surrogate":
        w = _log(rng, 96, 1000)
        return dict(kind="surrogate", w=w, h=max(8, int(w * rng.uniform(0.5, 1.1))))
    if kind == "train":
        return dict(kind="train", batch=128 * rng.randint(16, 256), rows=1 << 18, steps=rng.randint(1, 8))
    if kind == "gradient":
        return dict(kind="gradient", batch=128 * _log(rng, 1, 256))
    return dict(kind="beams", w=_log(rng, 12, 120), h=_log(rng, 8, 68), tol=rng.choice([1e-7, 1e-8]))


# --------------------------------------------------------------------------- inputs
def _config(c):
    kind = c["kind"]
    base = dict(min_step=1e-9, max_step=2.0, initial_step=0.1, escape_radius=200.0, horizon_factor=1.01,
                max_steps=10000)
    if kind == "frame":
        prec = abi.PRECISION_MIXED if c["precision"] == "mixed" else abi.PRECISION_FP64
        if c["tol"] > 1e-6:  # RenderSession's settings
            base = {}
        return abi.default_config(abs_tolerance=c["tol"], rel_tolerance=c["tol"], precision=prec,
                                  enable_volumetric=1 if c["bins"] else 0, n_bins=c["bins"], **base)
    if kind == "rays":
        return abi.default_config(abs_tolerance=c["tol"], rel_tolerance=c["tol"], **base)
    if kind == "batch":
        return abi.default_config(abs_tolerance=c["tol"], rel_tolerance=c["tol"], precision=abi.PRECISION_MIXED, **base)
    if kind == "sky":
        return abi.default_config(integrator=abi.INTEGRATOR_SYMPLECTIC, symplectic_order=c["order"],
                                  symplectic_step=0.01, projection_period=8, max_steps=50000, escape_radius=60.0,
                                  horizon_factor=1.01, min_step=1e-9, enable_volumetric=1 if c["bins"] else 0,
                                  n_bins=c["bins"], precision=abi.PRECISION_MIXED, watchdog_ms=300000)
    if kind == "surrogate":  # the surrogate workload's integration settings
        return abi.default_config(abs_tolerance=1e-8, rel_tolerance=1e-8, precision=abi.PRECISION_MIXED,
                                  critical_band=0.0, island_factor=0.0, **base)
    if kind == "beams":
        base.update(escape_radius=1000.0, max_steps=20000)
        return abi.default_config(abs_tolerance=c["tol"], rel_tolerance=c["tol"], enable_disk=0, **base)
    return abi.default_config()


def _frames(c, seed):
    """The frames of a case: spin, inclination and (for a batch) distance and metric from the seed; a batch's families
    in turn, its sides spread over [lo, hi]."""
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    if kind == "batch":
        out = []
        for i in range(c["n"]):
            side = int(round(c["lo"] * (c["hi"] / c["lo"]) ** ((i * 7 % c["n"] + 0.5) / c["n"])))
            r, th = float(rng.uniform(20.0, 150.0)), float(rng.uniform(10.0, 89.0))
            a = float(rng.uniform(0.0, 0.998))
            if i % 4 == 0:
                m = abi.make_metric(a=a, Q=float(rng.uniform(0.0, 0.9 * math.sqrt(1.0 - a * a))))
            elif i % 4 == 1:
                m = abi.make_metric(a=a, Lambda=float(10 ** rng.uniform(-6.0, -4.0)))
            elif i % 4 == 2:
                m = abi.make_metric(family=abi.MORRIS_THORNE, b0=float(rng.uniform(0.5, 2.0)))
            else:
                m = abi.make_metric(family=abi.ALCUBIERRE, vs=float(rng.uniform(0.1, 2.0)), sigma=8.0, R=1.0)
            out.append(abi.make_frame(m, abi.make_camera(r=r, theta_deg=th, width=side, height=side, fov=30.0), 0.0, 30.0))
        return out
    if kind == "sky":
        cam = abi.make_camera(r=15.0, theta_deg=float(rng.uniform(60.0, 85.0)), width=c["w"], height=c["h"],
                              projection=abi.CAMERA_EQUIRECTANGULAR)
        return [abi.make_frame(abi.make_metric(a=0.998, Q=0.05), cam, 0.0, 30.0)]
    cam = abi.make_camera(r=100.0, theta_deg=float(rng.uniform(30.0, 80.0)), width=c["w"], height=c["h"], fov=30.0)
    return [abi.make_frame(abi.make_metric(M=1.0, a=float(rng.uniform(0.5, 0.95))), cam, 0.0, 30.0)]


def _rays(c, seed):
    """Camera rays as GeodesicTracer's callers build them: one origin, directions over a 30 degree field."""
    rng = np.random.default_rng(seed)
    n = c["n"]
    origin = np.array([0.0, 60.0, math.radians(rng.uniform(40.0, 85.0)), 0.0])
    t = math.tan(math.radians(15.0))
    d = np.stack([-np.ones(n), rng.uniform(-t, t, n), rng.uniform(-t, t, n)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    spin = float(rng.uniform(0.5, 0.95))
    return spin, origin, np.concatenate([np.zeros((n, 1)), d], 1)


def _features(n, gen):
    """Rows as the feature kernel writes them: spin, inclination, alpha / 20, beta / 20 and distance, normalised."""
    f = torch.rand(n, 5, device=DEV, generator=gen) * 2 - 1
    f[:, 2:4] *= 1.4
    return f


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _training_set(rows, seed):
    g = _gen(seed)
    x = _features(rows, g)
    rho = torch.hypot(x[:, 2], x[:, 3])
    hit = (rho > 0.3).float()
    t = torch.stack([hit, hit * (0.9 * rho - 0.5 + 0.1 * x[:, 0]), hit * (0.7 + 0.3 * x[:, 2] * x[:, 1]),
                     0.2 * torch.rand(rows, device=DEV, generator=g) * (rho < 0.5)], 1).contiguous()
    w = 0.05 + torch.rand(rows, device=DEV, generator=g) ** 4
    return x, t, w


def _weights(seed):
    """The shipped weights, each moved by up to 1 %: the seed's network."""
    p = np.load(WEIGHTS).astype(np.float32).ravel()
    u = np.random.default_rng(seed).uniform(-0.01, 0.01, p.size).astype(np.float32)
    return p * (1 + u)


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    s = {"case": c, "eng": Engine(0, _config(c))}
    if kind in ("frame", "batch", "sky"):
        arr, total = frames_array(_frames(c, seed))
        s["n_frames"], s["total"] = len(arr), total
        s["frames"] = torch.from_numpy(np.frombuffer(bytes(arr), dtype=np.uint8).copy()).to(DEV)
        s["image"] = torch.zeros(total, dtype=torch.float32, device=DEV)
        bins = c.get("bins", 0)
        s["spectra"] = torch.zeros(total, bins, dtype=torch.float32, device=DEV) if bins else None
    elif kind == "rays":
        spin, origin, dirs = _rays(c, seed)
        s["metric"] = abi.make_metric(a=spin)
        s["rays"] = []
        for d in dirs:
            r = abi.CameraRay()
            r.origin[:] = list(origin)
            r.direction[:] = list(d)
            s["rays"].append(r)
    elif kind == "infer":
        s["eng"].surrogate_load(_weights(seed))
        s["x"] = _features(c["n"], _gen(seed))
        s["y"] = torch.empty(c["n"], 4, dtype=torch.float32, device=DEV)
    elif kind == "surrogate":
        s["eng"].surrogate_load(np.load(WEIGHTS))
        s["frames"] = _frames(c, seed)
        n = c["w"] * c["h"]
        s["image"] = torch.empty(n, dtype=torch.float32, device=DEV)
        s["gate"] = torch.empty(n, dtype=torch.uint8, device=DEV)
    elif kind in ("train", "gradient"):
        rows = c.get("rows", c["batch"])
        s["set"] = _training_set(rows, seed)
        s["rows"] = rows
        s["eng"].train_init(_weights(seed), abi.train_config(batch=c["batch"], total_steps=4096, max_lr=1e-3))
    else:
        s["frames"] = _frames(c, seed)
    return s


# --------------------------------------------------------------------------- one pass
# Fields of a ray record that a caller of GeodesicTracer::trace reads. The two residuals of the null condition are left
# out: they are rounding residues, which say how good the record is and have no value of their own.
RAY_INTS = ("outcome", "steps", "rejected", "n_crossings", "equatorial_crossings", "image_order", "flags")
RAY_FLOATS = ("final_x", "final_p", "final_k", "disk_r", "disk_phi", "disk_g", "disk_flux", "total_phi_change",
              "min_radius", "intensity", "E", "Lz", "Carter", "impact_parameter", "magnification")


def run(s):
    c, eng = s["case"], s["eng"]
    kind = c["kind"]
    if kind in ("frame", "batch", "sky"):
        spc = s["spectra"]
        eng.trace_frames_device(s["frames"].data_ptr(), s["n_frames"], s["total"], None, s["image"].data_ptr(),
                                spc.data_ptr() if spc is not None else None, torch.cuda.current_stream().cuda_stream)
        return {"image": s["image"], "spectra": spc} if spc is not None else {"image": s["image"]}
    if kind == "rays":
        r = eng.trace_rays(s["metric"], s["rays"], disk_outer=30.0)
        return {f: r[f] for f in RAY_INTS + RAY_FLOATS}
    if kind == "infer":
        eng.surrogate_infer(s["x"].data_ptr(), c["n"], s["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return s["y"]
    if kind == "surrogate":
        eng.render_surrogate_device(s["frames"], s["image"].data_ptr(), None, s["gate"].data_ptr(),
                                    stream=torch.cuda.current_stream().cuda_stream)
        return {"image": s["image"], "gate": s["gate"]}
    if kind == "train":
        x, t, w = s["set"]
        eng.train_steps(x.data_ptr(), t.data_ptr(), w.data_ptr(), s["rows"], c["steps"])
        params, steps = eng.train_params()
        return {"params": params, "steps": steps}
    if kind == "gradient":
        x, t, w = s["set"]
        parts, grad = eng.train_gradient(x.data_ptr(), t.data_ptr(), w.data_ptr(), s["rows"])
        return {"loss_parts": parts, "grad": grad}
    b = eng.trace_beams(s["frames"])
    return {k: np.ascontiguousarray(b[k]) for k in ("outcome", "steps", "magnification", "parity", "final_dir")}


# --------------------------------------------------------------------------- the least work
# Operations of one accepted Dormand-Prince step: six right-hand sides of about 80 operations each, the stage sums (434)
# and the projection onto the null cone (136). Steps per ray: what the tolerance asks for over a 100 M to 200 M path.
STEP_FLOPS = 6 * 80 + 434 + 136
ROW_FLOPS = 2 * 198912


def work(case):
    c = case
    kind = c["kind"]
    if kind == "frame":
        n, steps = c["w"] * c["h"], 170 if c["tol"] < 1e-6 else 150
        return {"bytes": n * 4.0 * (1 + c["bins"]), "flops": float(n) * steps * STEP_FLOPS}
    if kind == "rays":
        return {"bytes": c["n"] * (64.0 + 256.0), "flops": float(c["n"]) * 150 * STEP_FLOPS}
    if kind == "batch":
        side2 = (c["hi"] ** 2 - c["lo"] ** 2) / (2 * math.log(c["hi"] / c["lo"])) if c["hi"] > c["lo"] else c["hi"] ** 2
        return {"bytes": 4.0 * c["n"] * side2, "flops": c["n"] * side2 * 130 * STEP_FLOPS}
    if kind == "sky":  # per step and Yoshida substep: the metric once, two kicks and a drift
        n, sub = c["w"] * c["h"], {4: 3, 6: 7, 8: 15}[c["order"]]
        return {"bytes": n * 4.0 * (1 + c["bins"]), "flops": float(n) * 6200 * sub * 140}
    if kind == "infer":
        return {"bytes": c["n"] * 36.0 + 4e5, "flops": float(c["n"]) * ROW_FLOPS}
    if kind == "surrogate":  # about 60 % of the pixels through the network, 5 % integrated
        n = c["w"] * c["h"]
        return {"bytes": 5.0 * n, "flops": n * (0.6 * ROW_FLOPS + 0.05 * 200 * STEP_FLOPS)}
    if kind in ("train", "gradient"):
        n = c["batch"] * c.get("steps", 1)
        return {"bytes": n * 40.0 + 5.6e6 * c.get("steps", 1), "flops": 3.0 * n * ROW_FLOPS}
    return {"bytes": 32.0 * c["w"] * c["h"], "flops": float(c["w"] * c["h"]) * 600 * 3 * STEP_FLOPS}


# --------------------------------------------------------------------------- the outputs in 64 bits
def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "infer":
        W = _layers(_weights(seed))
        x = _features(c["n"], _gen(seed)).double()
        return torch.cat([_net(W, part) for part in x.split(1 << 17)])
    if kind == "gradient":
        x, t, w = (v.double() for v in _training_set(c["batch"], seed))
        p = torch.from_numpy(_weights(seed)).to(DEV).double()
        parts, grad = _loss_gradient(p, x, t, w)
        return {"loss_parts": parts, "grad": grad}
    if kind == "train":
        return {"params": _adam(c, seed), "steps": c["steps"]}
    if kind == "frame" and c["w"] * c["h"] * max(1, c["bins"]) <= 1 << 22:
        f = _frames(c, seed)[0]
        cam = f.camera
        x, p = _start(cam.r, cam.theta, f.metric.a, _pixel_dirs(cam))
        o = _trace(x, p, f.metric.a, _config(c), f.disk_outer, _sqrt_m_gtt(cam.r, cam.theta, f.metric.a))
        out = {"image": o["intensity"]}
        if c["bins"]:
            out["spectra"] = o["spectra"]
        return out
    if kind == "rays":
        spin, origin, dirs = _rays(c, seed)
        x, p = _start(origin[1], origin[2], spin, torch.from_numpy(dirs[:, 1:]).to(DEV).T)
        o = _trace(x, p, spin, _config(c), 30.0, _sqrt_m_gtt(origin[1], origin[2], spin))
        fields = {f: None for f in RAY_INTS + RAY_FLOATS}
        fields.update({"intensity": o["intensity"], "final_x": o["x"].T, "final_p": o["p"].T, "E": -o["p"][0],
                       "Lz": o["x"][1] * o["p"][2] - o["x"][2] * o["p"][1], "min_radius": o["min_r"],
                       "disk_r": o["disk_r"].T, "disk_g": o["disk_g"].T})
        return fields
    # The rest would take minutes in plain torch: the full-size spectra, the symplectic map (10^5 sequential
    # right-hand sides), the beams (24 equations to R = 1000 M), and frames of four families or a gated one, which
    # mix several programs.
    return None


def _layers(p):
    p = torch.as_tensor(p).to(DEV).double()
    out, off = [], 0
    for o, i in ((256, 5), (256, 256), (256, 256), (256, 256), (4, 256)):
        out.append((p[off:off + o * i].reshape(o, i), p[off + o * i:off + o * i + o]))
        off += o * i + o
    return out


def _net(W, x):
    for k, (w, b) in enumerate(W):
        x = x @ w.T + b
        if k < 4:
            x = x * torch.sigmoid(x)
    return x


def _loss_gradient(p, x, t, w):
    p = p.clone().requires_grad_(True)
    o = _net(_layers_grad(p), x)
    hit = t[:, 0]
    bce = torch.nn.functional.binary_cross_entropy_with_logits(o[:, 0], hit)
    shw, sw = (hit * w).sum(), w.sum()
    lr = (hit * w * (o[:, 1] - t[:, 1]) ** 2).sum() / shw
    lg = (hit * w * (o[:, 2] - t[:, 2]) ** 2).sum() / shw
    lh = (w * (o[:, 3] - t[:, 3]) ** 2).sum() / sw
    (bce + 100 * (lr + lg) + 10 * lh).backward()
    return torch.stack([bce, lr, lg, lh]).detach(), p.grad


def _layers_grad(p):
    out, off = [], 0
    for o, i in ((256, 5), (256, 256), (256, 256), (256, 256), (4, 256)):
        out.append((p[off:off + o * i].reshape(o, i), p[off + o * i:off + o * i + o]))
        off += o * i + o
    return out


def _epoch_rows(n, epoch, lo, hi):
    """Rows [lo, hi) of the first epochs' keyed permutation of [0, n) (seed 0): a 4-round Feistel network on the next
    power of four, cycle-walked."""
    half = 1
    while (1 << (2 * half)) < n:
        half += 1
    mask = np.uint64((1 << half) - 1)
    key = (epoch * 0xC2B2AE35 + 1) & 0xFFFFFFFF

    def mix(x, k):
        x = x ^ np.uint32(k)
        x = x * np.uint32(0x7FEB352D)
        x = x ^ (x >> np.uint32(15))
        x = x * np.uint32(0x846CA68B)
        return x ^ (x >> np.uint32(16))

    def once(i):
        left, right = i >> np.uint64(half), i & mask
        for rnd in range(4):
            f = mix(right.astype(np.uint32), (key + 0x9E3779B9 * (rnd + 1)) & 0xFFFFFFFF).astype(np.uint64) & mask
            left, right = right, left ^ f
        return (left << np.uint64(half)) | right

    x = once(np.arange(lo, hi, dtype=np.uint64))
    while (x >= n).any():
        x = np.where(x >= n, once(x), x)
    return torch.from_numpy(x.astype(np.int64)).to(DEV)


def _adam(c, seed):
    x, t, w = (v.double() for v in _training_set(c["rows"], seed))
    p = torch.from_numpy(_weights(seed)).to(DEV).double()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    per_epoch = c["rows"] // c["batch"]
    for k in range(c["steps"]):
        epoch, pos = divmod(k, per_epoch)
        rows = _epoch_rows(c["rows"], epoch, pos * c["batch"], (pos + 1) * c["batch"])
        _, g = _loss_gradient(p, x[rows], t[rows], w[rows])
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        lr = 1e-3 * (0.04 + 0.96 * k / (0.05 * 4096))
        p = p - lr * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return p


# ---- Kerr geodesics (Kerr-Schild coordinates, M = 1) in plain torch, FP64 -----------------------------------------
def _geometry(x, a):
    X, Y, Z = x[1], x[2], x[3]
    d = X * X + Y * Y + Z * Z - a * a
    sig = (d * d + 4 * a * a * Z * Z).sqrt()
    r = ((d + sig) / 2).sqrt()
    den = r * r + a * a
    return r, sig, den, 2 * r / sig, (r * X + a * Y) / den, (r * Y - a * X) / den, Z / r


def _rhs(x, p, a):
    """dx/dl = g^-1 p and dp/dl = (1/2) (d g) k k with g = eta + H l l."""
    X, Y, Z = x[1], x[2], x[3]
    r, sig, den, H, l1, l2, l3 = _geometry(x, a)
    lp = -p[0] + l1 * p[1] + l2 * p[2] + l3 * p[3]
    k = torch.stack([-p[0] + H * lp, p[1] - H * l1 * lp, p[2] - H * l2 * lp, p[3] - H * l3 * lp])
    lk = k[0] + l1 * k[1] + l2 * k[2] + l3 * k[3]
    rx, ry, rz = r * X / sig, r * Y / sig, Z * den / (r * sig)
    # l_i and H as functions of (r, x, y, z): the chain rule through r and the explicit part
    dl_dr = k[1] * (X - 2 * r * l1) / den + k[2] * (Y - 2 * r * l2) / den - k[3] * Z / (r * r)
    dH_dr = (2 - 4 * H * r + 4) / sig
    ex = (r * k[1] - a * k[2]) / den
    ey = (a * k[1] + r * k[2]) / den
    ez = k[3] / r
    hz = -H * 2 * a * a * Z / (r * r * sig)
    c = 0.5 * dH_dr * lk + H * dl_dr
    f = torch.stack([torch.zeros_like(lk), lk * (c * rx + H * ex), lk * (c * ry + H * ey),
                     lk * (c * rz + H * ez + 0.5 * hz * lk)])
    return torch.cat([k, f])


_A = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
      (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
      (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
      (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
_E = (35 / 384 - 5179 / 57600, 0.0, 500 / 1113 - 7571 / 16695, 125 / 192 - 393 / 640, -2187 / 6784 + 92097 / 339200,
      11 / 84 - 187 / 2100, -1 / 40)


def _attempt(y, k1, h, a, cfg):
    """One Dormand-Prince 5(4) step: (candidate, f at it, scaled error of the position)."""
    ks = [k1]
    for row in _A:
        s = sum(c * k for c, k in zip(row, ks) if c != 0.0)
        yn = y + h * s
        ks.append(_rhs(yn[:4], yn[4:], a))
    e = h * sum(c * k[:4] for c, k in zip(_E, ks) if c != 0.0)
    e = e / (cfg.abs_tolerance + cfg.rel_tolerance * yn[:4].abs())
    return yn, ks[-1], (e * e).mean(0).sqrt()


def _project(y, a):
    """p + alpha dr back onto the null cone; also r and the null value before."""
    r, sig, den, H, l1, l2, l3 = _geometry(y, a)
    d = torch.stack([r * y[1] / sig, r * y[2] / sig, y[3] * den / (r * sig)])
    p = y[5:8]
    ld, lp = l1 * d[0] + l2 * d[1] + l3 * d[2], -y[4] + l1 * p[0] + l2 * p[1] + l3 * p[2]
    A, B = (d * d).sum(0) - H * ld * ld, 2 * ((p * d).sum(0) - H * lp * ld)
    C = -y[4] ** 2 + (p * p).sum(0) - H * lp * lp
    disc = B * B - 4 * A * C
    q = -0.5 * (B + torch.where(B >= 0, 1.0, -1.0) * disc.clamp_min(0).sqrt())
    alpha = torch.where((disc >= 0) & (A.abs() >= 1e-15) & (q != 0), C / q, torch.zeros_like(C))
    return torch.cat([y[:5], p + alpha * d]), r


def _pixel_dirs(cam):
    """Pinhole directions in the camera's single-precision arithmetic (yaw = pitch = roll = 0)."""
    w, h, one = cam.width, cam.height, torch.float32
    px, py = torch.arange(w, device=DEV, dtype=one), torch.arange(h, device=DEV, dtype=one)
    t = float(np.float32(math.tan(np.float32(cam.fov) * np.float32(math.pi) / np.float32(360))))
    x = ((2 * (px + 0.5)) / w - 1) * float(np.float32(w) / np.float32(h)) * t
    y = (1 - (2 * (py + 0.5)) / h) * t
    x, y = x[None, :].expand(h, w).reshape(-1), y[:, None].expand(h, w).reshape(-1)
    n = ((x * x + y * y) + 1).sqrt()
    return torch.stack([-1 / n, -y / n, x / n]).double()


def _start(r, th, a, d):
    """State of camera rays with directions d (r, theta, phi components) at spherical (r, th, 0)."""
    st, ct = math.sin(th), math.cos(th)
    n = d.shape[1]
    x = torch.zeros(4, n, device=DEV, dtype=torch.float64)
    x[1], x[3] = r * st, r * ct
    k = torch.stack([d[0] * st + d[1] * ct, d[2], d[0] * ct - d[1] * st])
    _, _, _, H, l1, l2, l3 = _geometry(x, a)
    lk = l1 * k[0] + l2 * k[1] + l3 * k[2]
    A, B, C = H - 1, 2 * H * lk, (k * k).sum(0) + H * lk * lk
    k0 = (-B - (B * B - 4 * A * C).sqrt()) / (2 * A)
    s = H * (k0 + lk)
    return x, torch.stack([-k0 + s, k[0] + s * l1, k[1] + s * l2, k[2] + s * l3])


def _sqrt_m_gtt(r, th, a):
    x = torch.zeros(4, 1, dtype=torch.float64)
    x[1], x[3] = r * math.sin(th), r * math.cos(th)
    return math.sqrt(1 - float(_geometry(x, a)[3]))


def _kepler_g(X, Y, Z, r, a, E, L, norm):
    """Redshift of a Keplerian emitter at radius r."""
    den = r * r + a * a
    l1, l2 = (r * X + a * Y) / den, (r * Y - a * X) / den
    H = 2 * r * r * r / (r ** 4 + a * a * Z * Z)
    lxi = X * l2 - Y * l1
    om = 1 / (r * r.sqrt() + a)
    n = 1 - H - 2 * om * H * lxi - om * om * (X * X + Y * Y + H * lxi * lxi)
    return n.clamp_min(1e-300).sqrt() / (norm * (1 - om * L / E)) * (n > 0)


def _isco(a):
    z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
    z2 = math.sqrt(3 * a * a + z1 * z1)
    return 3 + z2 - math.sqrt((3 - z1) * (3 + z1 + 2 * z2))


def _flux(r, a, rin):
    """Page-Thorne flux with 16-point Gauss-Legendre quadrature from the ISCO, and the simplified form where the full
    expression is not used."""
    def circ(q):
        s = q.sqrt()
        D = (q * q - 3 * q + 2 * a * s).clamp_min(1e-300)
        d = q * D.sqrt()
        return (q * q - 2 * q + a * s) / d, (q * q - 2 * a * s + a * a) / d, 1 / (q * s + a), D

    def dL(q):
        s = q.sqrt()
        _, _, _, D = circ(q)
        N, w = q * q - 2 * a * s + a * a, a / s
        rs = q * D.sqrt()
        return ((2 * q - w) * rs - N * (2 * D + q * (2 * q - 3 + w)) / (2 * D.sqrt())) / (rs * rs)

    gx, gw = np.polynomial.legendre.leggauss(16)
    hw, mid = 0.5 * (r - rin), 0.5 * (r + rin)
    I = torch.zeros_like(r)
    for g, wt in zip(gx, gw):
        q = mid + hw * g
        e, l, o, _ = circ(q)
        I = I + wt * (e - o * l) * dL(q)
    e, l, o, _ = circ(r)
    fn = 3 / (8 * math.pi * r ** 3)
    full = fn * (1.5 * r.sqrt() / (r * r.sqrt() + a) ** 2 / (e - o * l) ** 2) * I * hw
    y = r.sqrt()
    den = y ** 3 * (y - 3 / y + 2 * a / (y * y))
    Q = torch.where(den.abs() > 1e-10, 1 / den, torch.ones_like(den))
    Q = torch.where(Q > 0, Q, torch.ones_like(Q)).clamp(0.1, 10.0)
    simple = fn * (1 - (rin / r).sqrt()).clamp_min(0) * Q
    return torch.where((r > 1.5 * rin) & (full > 0), full, simple)


def _hermite(s, h, y0, y1, k0, k1):
    s2, s3 = s * s, s * s * s
    return ((2 * s3 - 3 * s2 + 1) * y0 + (s3 - 2 * s2 + s) * h * k0 + (3 * s2 - 2 * s3) * y1 + (s3 - s2) * h * k1)


def _cap(y, k, r, hz, rin, rout):
    """The step cap near the emitting volume."""
    Hs = hz * r.clamp(rin, rout)
    dist = torch.maximum(torch.maximum(rin - r, r - rout), y[3].abs() - 6 * Hs)
    return torch.maximum(0.5 * Hs, dist) / (k[1:4] ** 2).sum(0).sqrt().clamp_min(1e-3)


_GL = np.polynomial.legendre.leggauss(4)


def _segment(I, T, y0, y1, k0, k1, h, r0, r1, a, cfg, nu, rin, rout, norm):
    """Emission and absorption of one accepted step, 4 Gauss-Legendre points on its cubic interpolant between the
    edges of the emitting annulus."""
    def point(q):
        X, Y, Z = (_hermite(q, h, y0[i], y1[i], k0[i], k1[i]) for i in (1, 2, 3))
        d = X * X + Y * Y + Z * Z - a * a
        return X, Y, Z, ((d + (d * d + 4 * a * a * Z * Z).sqrt()) / 2).sqrt()

    E, L = -y1[4], y1[1] * y1[6] - y1[2] * y1[5]
    in0, in1 = (r0 >= rin) & (r0 <= rout), (r1 >= rin) & (r1 <= rout)
    other = torch.where(in0, r1, r0)
    edge = torch.where(other < rin, rin, rout)
    mixed = in0 != in1
    lo, hi = torch.zeros_like(h), torch.ones_like(h)
    g0 = r0 - edge
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        same = (point(mid)[3] - edge > 0) == (g0 > 0)
        lo, hi = torch.where(same, mid, lo), torch.where(same, hi, mid)
    fa = torch.where(mixed & ~in0, lo, torch.zeros_like(h))
    fb = torch.where(mixed & in0, lo, torch.ones_like(h))
    for g, wt in zip(*_GL):
        X, Y, Z, r = point(fa + (fb - fa) * 0.5 * (1 + g))
        zr = Z / (cfg.vol_height_ratio * r)
        gg = _kepler_g(X, Y, Z, r, a, E, L, norm)
        on = (r >= rin) & (r <= rout) & (zr.abs() <= 6) & (gg > 0)
        gs = torch.where(on, gg, torch.ones_like(gg))
        j = cfg.vol_j0 / (r * r) * torch.exp(-0.5 * zr * zr) * gs ** cfg.vol_spectral_index
        dt = torch.where(on, cfg.vol_alpha_over_j * j * (E / norm / gs) * h * (fb - fa) * 0.5 * wt, torch.zeros_like(j))
        om = -torch.expm1(-dt[:, None] * nu[None, :])
        I += T * (gs ** 3 / cfg.vol_alpha_over_j)[:, None] * om
        T -= T * om


def _trace(x, p, a, cfg, rout, norm):
    """The rays' images: Dormand-Prince with retry, projection, horizon and escape tests, disk crossings located on
    the equator, and the volumetric bins."""
    n = x.shape[1]
    rin = _isco(a)
    rhor = (1 + math.sqrt(1 - a * a)) * cfg.horizon_factor
    bins = cfg.n_bins if cfg.enable_volumetric else 0
    Y = torch.cat([x, p])
    K = _rhs(x, p, a)
    Hh = torch.full((n,), cfg.initial_step, device=DEV, dtype=torch.float64)
    R0 = _geometry(x, a)[0].clone()
    out = {"intensity": torch.zeros(n, device=DEV, dtype=torch.float64), "x": x.clone(), "p": p.clone(),
           "min_r": torch.full((n,), 1e10, device=DEV, dtype=torch.float64),
           "disk_r": torch.zeros(4, n, device=DEV, dtype=torch.float64),
           "disk_g": torch.ones(4, n, device=DEV, dtype=torch.float64),
           "spectra": torch.zeros(n, bins, device=DEV, dtype=torch.float64)}
    T = torch.ones(n, bins, device=DEV, dtype=torch.float64)
    if bins:
        nu = torch.tensor(cfg.nu_min, device=DEV, dtype=torch.float64) * (cfg.nu_max / cfg.nu_min) ** (
            torch.arange(bins, device=DEV, dtype=torch.float64) / max(1, bins - 1))
        nu = nu ** -cfg.vol_spectral_index
    ncross = torch.zeros(n, device=DEV, dtype=torch.int64)
    steps = torch.zeros(n, device=DEV, dtype=torch.int64)
    live = torch.arange(n, device=DEV)
    while live.numel():
        y, k, h = Y[:, live], K[:, live], Hh[live]
        yn, kn, err = _attempt(y, k, h, a, cfg)
        fac = (cfg.safety_factor * err.clamp_min(1e-15) ** -0.2).clamp(cfg.step_shrink_min, cfg.step_grow_max)
        hn = torch.where(err < 1e-15, (h * cfg.step_grow_max).clamp_max(cfg.max_step),
                         (h * fac).clamp(cfg.min_step, cfg.max_step))
        ok = err <= 1
        no = live[~ok]
        if no.numel():
            hr = hn[~ok]
            if bins:
                ro = _geometry(y[:, ~ok], a)[0]
                hr = torch.minimum(hr, _cap(y[:, ~ok], k[:, ~ok], ro, cfg.vol_height_ratio, rin, rout)).clamp_min(cfg.min_step)
            Hh[no] = hr
        dead = torch.zeros(n, device=DEV, dtype=torch.bool)
        dead[no] = Hh[no] <= cfg.min_step
        i = live[ok]
        if i.numel():
            y0, k0, h0, yn, kn, h1 = y[:, ok], k[:, ok], h[ok], yn[:, ok], kn[:, ok], hn[ok]
            y1, r = _project(yn, a)
            moved = (y1 - yn)[4:].abs().amax(0) > 1e-10 * y1[4:].abs().amax(0)
            if moved.any():
                kn = kn.clone()
                kn[:, moved] = _rhs(y1[:4, moved], y1[4:, moved], a)
            steps[i] += 1
            out["min_r"][i] = torch.minimum(out["min_r"][i], r)
            if bins:
                h1 = torch.minimum(h1, _cap(y1, kn, r, cfg.vol_height_ratio, rin, rout)).clamp_min(cfg.min_step)
            end = r < rhor
            end |= ((y1[1:4] ** 2).sum(0) > cfg.escape_radius ** 2) & ((y1[1:4] * kn[1:4]).sum(0) > 0)
            go = ~end
            if bins:
                z0, z1, r0 = y0[3].abs(), y1[3].abs(), R0[i]
                far = ((r0 > rout) & (r > rout)) | ((y0[3] * y1[3] > 0) &
                                                   (z0 > 6 * cfg.vol_height_ratio * r0.clamp(rin, rout)) &
                                                   (z1 > 6 * cfg.vol_height_ratio * r.clamp(rin, rout)))
                v = go & ~far
                if v.any():
                    I, Tv = out["spectra"][i[v]], T[i[v]]
                    _segment(I, Tv, y0[:, v], y1[:, v], k0[:, v], kn[:, v], h0[v], r0[v], r[v], a, cfg, nu, rin, rout, norm)
                    out["spectra"][i[v]], T[i[v]] = I, Tv
            x = go & (y0[3] * y1[3] < 0) & (ncross[i] < 4) if cfg.enable_disk else torch.zeros_like(go)
            if x.any():
                ya, ka, ha, yb, kb, j = y0[:, x], k0[:, x], h0[x], yn[:, x], kn[:, x], i[x]
                lo, hi = torch.zeros_like(ha), torch.ones_like(ha)
                for _ in range(50):
                    mid = 0.5 * (lo + hi)
                    same = (_hermite(mid, ha, ya[3], yb[3], ka[3], kb[3]) < 0) == (ya[3] < 0)
                    lo, hi = torch.where(same, mid, lo), torch.where(same, hi, mid)
                s = 0.5 * (lo + hi) * ha
                yc, kc, _ = _attempt(ya, ka, s, a, cfg)
                s = s - yc[3] / kc[3]
                yc, kc, _ = _attempt(ya, ka, s, a, cfg)
                d = -yc[3] / kc[3]
                X, Yc = yc[1] + d * kc[1], yc[2] + d * kc[2]
                rc = (X * X + Yc * Yc - a * a).clamp_min(1e-10).sqrt()
                hit = (rc >= rin) & (rc <= rout)
                if hit.any():
                    j, X, Yc, rc, e = j[hit], X[hit], Yc[hit], rc[hit], y1[:, x][:, hit]
                    g = _kepler_g(X, Yc, torch.zeros_like(X), rc, a, -e[4], e[1] * e[6] - e[2] * e[5], norm)
                    out["disk_r"][ncross[j], j], out["disk_g"][ncross[j], j] = rc, g
                    out["intensity"][j] += torch.exp(-cfg.crossing_weight_decay * ncross[j]) * g ** 4 * _flux(rc, a, rin)
                    ncross[j] += 1
            end |= (ncross[i] >= 4) & go
            end |= steps[i] >= cfg.max_steps
            Y[:, i], K[:, i], Hh[i], R0[i] = y1, kn, h1, r
            dead[i] = end
        live = live[~dead[live]]
    out["x"], out["p"] = Y[:4], Y[4:]
    return out
