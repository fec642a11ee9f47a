"""The work that is timed: calibration filters stepped through the package's public classes.

A case is one filter (or a batch of filters) on a seeded synthetic stereo scene
(`scene.make_scene`: landmarks 2..12 m ahead, Poisson clutter, frames of the fixed camera
and of the camera being calibrated in turn).  `prepare` creates the filter and runs it
over the scene's first frames, so that its maps have grown to what they are in use; `run`
takes the next frame.  The frames after the first ones are walked forwards and backwards,
so a state can be stepped for as long as wanted and the camera always moves smoothly.

Kinds:
  step     one frame through step() from host measurements; `wait` reads the parents back
           and waits for them each frame (a rig that acts on each estimate), otherwise the
           copy is queued into page-locked buffers (a recording worked off at full rate)
  loop     the reference driver's frame: predict, update, the dump of the parents and of
           the most likely parent's map, the NaN check, resample
  batch    many filters in one batched, graph-replayed step from host measurements
  restore  update() of a filter whose state was loaded with set_state (a resumed run): the
           per-measurement normalisers and the parents' log-likelihoods and weights
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("scphd-camera-calibration_b200")

# Frames before the first timed one: past the updates on which a filter tunes its launch
# shapes (the last after 16 + 6 frames) and long enough for the maps to fill.
PREFILL = 30
CYCLE = 16


def _case(name, kind, parents, landmarks, clutter, gaussians, samples=100, dim=3, fp64=False, wait=False,
          filters=1, slam=False):
    return {"name": name, "kind": kind, "parents": parents, "landmarks": landmarks, "clutter": float(clutter),
            "gaussians": gaussians, "samples": samples, "dim": dim, "fp64": fp64, "wait": wait, "filters": filters,
            "slam": slam}


def listed():
    return [
        # The reference's own size and mode: 100 parents, 100 samples, (u,v), double precision,
        # its driver's loop with the dump after each update.
        _case("loop_100_uv_fp64", "loop", 100, 50, 10, 128, dim=2, fp64=True),
        # A live rig with the smallest benchmark filter, a result wanted after each frame.
        _case("live_256", "step", 256, 50, 10, 64, wait=True),
        # The same filter in double precision, a recording.
        _case("rec_256_fp64", "step", 256, 50, 10, 64, fp64=True),
        # An odd size with a sample count other than the configurations' 100.
        _case("live_777_p50", "step", 777, 80, 20, 96, samples=50, wait=True),
        # SLAM frames only (no fixed camera), (u,v) measurements, single precision.
        _case("slam_1500_uv", "step", 1500, 90, 25, 160, dim=2, slam=True),
        # A middle-sized recording.
        _case("rec_1024", "step", 1024, 100, 30, 128),
        # The benchmark's single filter: 4096 parents, 200 landmarks, at most 256 Gaussians.
        _case("rec_4096", "step", 4096, 200, 50, 256),
        # The same in double precision.
        _case("rec_4096_fp64", "step", 4096, 200, 50, 256, fp64=True),
        # The densest scene: 400 landmarks, clutter 100, at most 512 Gaussians.
        _case("rec_8192_dense", "step", 8192, 400, 100, 512),
        # Many small rigs stepped together.
        _case("batch_64x256", "batch", 256, 50, 10, 64, filters=64),
        # A few larger rigs of different sizes stepped together.
        _case("batch_6_mixed", "batch", 1300, 120, 40, 192, filters=6),
        # A run resumed from a loaded state: one update of a map of sample clouds.
        _case("restore_512", "restore", 512, 60, 15, 64),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "loop", "batch", "restore"])
    gaussians = log_int(48, 512)
    landmarks = max(20, int(gaussians * rng.uniform(0.5, 0.8)))
    case = _case("", kind, 0, landmarks, round(rng.uniform(5, 80), 1), gaussians,
                 samples=rng.choice([100, 100, 100, log_int(32, 200)]), dim=rng.choice([3, 3, 3, 2]),
                 fp64=rng.random() < 0.15, wait=rng.random() < 0.5, slam=rng.random() < 0.2)
    # (u,v) measurements leave depth unobserved: such filters run in double precision
    case["fp64"] = case["fp64"] or case["dim"] == 2
    # parents of one filter, or of all the filters of a batch; Gaussians in all are bounded
    # so that no case costs more than the largest listed one
    most = (1 << 19) if case["fp64"] else (1 << 21)
    most //= max(1, -(-case["samples"] // 100))
    if kind == "loop":
        case["parents"] = log_int(64, min(1024, most // gaussians))
    elif kind == "restore":
        case["parents"], case["gaussians"] = log_int(64, 512), min(gaussians, 72)
        case["landmarks"] = min(landmarks, 72)
    elif kind == "batch":
        case["filters"] = log_int(2, 48)
        case["parents"] = log_int(64, max(65, min(2048, most // gaussians // case["filters"])))
    else:
        case["parents"] = log_int(64, max(65, min(8192, most // gaussians)))
    del case["name"]
    return case


# ------------------------------------------------------------------ preparation
def _filter(case, seed, parents, landmarks, clutter):
    sc = pkg.scene.make_scene(landmarks, PREFILL + CYCLE, clutter, seed, slam=case["slam"])
    most = max(z.shape[0] for z in sc.frames)
    cfg = pkg.scene.filter_config(parents, case["gaussians"], (most + 31) // 32 * 32, clutter, int(case["fp64"]),
                                  calib=sc.calib, seed=seed, particles_per_feature=case["samples"],
                                  meas_dim=case["dim"])
    cfg.max_survivors = 3 * case["gaussians"] + cfg.max_measurements
    if case["dim"] == 2:
        # depth is not measured: the clutter density is over the image alone, and new
        # features start in the scene's range of disparities (8 to 50)
        cfg.kappa = clutter / (pkg.scene.IMG_W * pkg.scene.IMG_H)
        cfg.w0 = cfg.kappa / 10.0
        cfg.d0, cfg.var_d0, cfg.var_vu0, cfg.var_vv0 = 22.0, 16.0, 1.0, 1.0
    frames = [(np.ascontiguousarray(z[:, 0]), np.ascontiguousarray(z[:, 1]),
               np.ascontiguousarray(z[:, 2]) if case["dim"] == 3 else None, bool(fx))
              for z, fx in zip(sc.frames, sc.fixed)]
    return pkg.SCPHDCameraCalibration(cfg), frames


def _pinned(filters):
    """Page-locked parent states and log-weights of all the filters, and each filter's rows."""
    n = sum(f.n_parents for f in filters)
    states = torch.zeros(n, 12, dtype=torch.float64, pin_memory=True)
    lw = torch.zeros(n, dtype=torch.float64, pin_memory=True)
    rows, at = [], 0
    for f in filters:
        rows.append((states[at:].data_ptr(), lw[at:].data_ptr()))
        at += f.n_parents
    return {"states": states, "lw": lw}, rows


def _restored(case, seed):
    """A map of sample clouds about points in view, as a checkpoint holds them."""
    rng = np.random.default_rng(seed)
    sc = pkg.scene.make_scene(case["landmarks"], 1, case["clutter"], seed, slam=True)
    n, g, p = case["parents"], case["gaussians"], case["samples"]
    # the detections, and clutter up to a fixed number of measurements
    z = sc.frames[0][:case["landmarks"]]
    more = case["landmarks"] + int(case["clutter"]) - z.shape[0]
    z = np.concatenate([z, rng.random((more, 3)) * [pkg.scene.IMG_W, pkg.scene.IMG_H, 60.0] + [0.0, 0.0, 1.0]])
    cfg = pkg.scene.filter_config(n, g, (z.shape[0] + 31) // 32 * 32, case["clutter"], int(case["fp64"]),
                                  calib=sc.calib, seed=seed, particles_per_feature=p, meas_dim=case["dim"])
    cfg.max_survivors = 3 * g + cfg.max_measurements
    states = np.asarray(cfg.prior_a[:]) + rng.random((n, 12)) * (np.asarray(cfg.prior_b[:]) - np.asarray(cfg.prior_a[:]))
    # features 3 to 8 m ahead, well inside the image; samples some centimetres about them
    depth = rng.uniform(3.0, 8.0, (n, g))
    centre = np.stack([rng.uniform(-0.35, 0.35, (n, g)) * depth, rng.uniform(-0.25, 0.25, (n, g)) * depth, depth,
                       *rng.normal(0, 0.02, (3, n, g))], axis=2)
    # the first of them are the scene's landmarks well inside the image
    at, seen = pkg.scene.project(sc.landmarks, sc.calib)
    seen &= (np.abs(at[:, 0] - pkg.scene.U0) < 190) & (np.abs(at[:, 1] - pkg.scene.V0) < 110)
    near = sc.landmarks[seen][:g]
    centre[:, :len(near), :3] = near[None] + rng.normal(0, 0.02, (n, len(near), 3))
    spread = np.array([0.03, 0.03, 0.06, 0.02, 0.02, 0.02])
    clouds = centre[..., None] + spread[:, None] * rng.standard_normal((n, g, 6, p))
    state = {"states": states, "log_weights": np.full(n, -math.log(n)), "sizes": np.full(n, g, np.int32),
             "weights": rng.uniform(0.05, 1.0, n * g), "clouds": clouds.reshape(n * g, 6, p),
             "omega": np.full((n * g, p), 1.0 / p)}
    return cfg, state, z


def prepare(case, seed):
    kind = case["kind"]
    if kind == "restore":
        cfg, state, z = _restored(case, seed)
        f = pkg.SCPHDCameraCalibration(cfg)
        f.set_state(**state)
        zd = np.ascontiguousarray(z[:, 2]) if case["dim"] == 3 else None
        return {"case": case, "f": f, "z": (np.ascontiguousarray(z[:, 0]), np.ascontiguousarray(z[:, 1]), zd)}
    filters, frames = [], []
    for i in range(case["filters"]):
        # the members of a batch differ in size: from 1/2 to 3/2 of the case's in a mixed
        # batch, the same filter for many small rigs
        scale = 0.5 + i / max(1, case["filters"] - 1) if kind == "batch" and case["filters"] <= 16 else 1.0
        f, fr = _filter(case, seed + 7919 * i, max(1, int(case["parents"] * scale)), case["landmarks"],
                        case["clutter"])
        filters.append(f)
        frames.append(fr)
    out, rows = _pinned(filters)
    state = {"case": case, "filters": filters, "frames": frames, "k": 0, "out": out, "rows": rows}
    if kind == "batch":
        state["batch"] = pkg.SCPHDBatch(filters, use_graph=True)
        for k in range(PREFILL):
            state["batch"].step(pkg.scene.DT, [fr[k] for fr in frames])
    else:
        for k in range(PREFILL):
            u, v, d, fixed = frames[0][k]
            filters[0].step(pkg.scene.DT, u, v, fixed, d)
    filters[0].synchronize()
    return state


# ------------------------------------------------------------------ one pass
def _next(state):
    k = state["k"] % (2 * CYCLE - 2)
    state["k"] += 1
    return PREFILL + (k if k < CYCLE else 2 * CYCLE - 2 - k)


def run(state):
    case = state["case"]
    kind, dt = case["kind"], pkg.scene.DT
    if kind == "restore":
        f, (u, v, d) = state["f"], state["z"]
        f.update(u, v, False, d)
        ell, loglik = f.normalizers(len(u))
        states, lw = f.particles()
        # the normalisers of a single-precision filter are single-precision values
        return {"ell": ell if case["fp64"] else ell.astype(np.float32), "loglik": loglik, "states": states, "lw": lw}
    at = _next(state)
    if kind == "batch":
        state["batch"].step(dt, [fr[at] for fr in state["frames"]])
        for f, (st, lw) in zip(state["filters"], state["rows"]):
            f.particles_async(st, lw)
        return state["out"]
    f = state["filters"][0]
    u, v, d, fixed = state["frames"][0][at]
    if kind == "loop":
        f.predict(dt)
        f.update(u, v, fixed, d)
        st, lw = f.particles()
        best = int(np.argmax(lw))
        # the dump's arrays hold the largest map; rows past the parent's map stay zero
        dump = [np.zeros((case["gaussians"], *shape)) for shape in ((), (6, case["samples"]), (case["samples"],))]
        for to, part in zip(dump, (f.map_weights(best), *f.map_clouds(best))):
            to[:len(part)] = part
        f.checkStuff()
        resampled = f.resample()
        return {"states": st, "lw": lw, "weights": dump[0], "clouds": dump[1], "omega": dump[2],
                "resampled": resampled}
    f.step(dt, u, v, fixed, d)
    if case["wait"]:
        st, lw = f.particles()
        return {"states": st, "lw": lw, "sizes": f.map_sizes()}
    f.particles_async(*state["rows"][0])
    return state["out"]


# ------------------------------------------------------------------ what a pass needs
def _visible(case):
    """Measurements of a frame: the landmarks in view that are detected, and clutter."""
    return 0.55 * case["landmarks"] + case["clutter"]


def work(case):
    s = 8 if case["fp64"] else 4
    n = case["parents"] * case["filters"]
    g, p, m = case["gaussians"], case["samples"], _visible(case)
    # a map entry is a weight, a mean and a covariance; the clouds of the components that
    # were not detected (nearly half of a map) are carried from frame to frame as samples
    carried = 1.0 if case["kind"] == "restore" else 0.46
    bytes_ = n * (2 * 8 * 13 + 2 * g * (28 * s + 4) + 2 * carried * g * 7 * p * s)
    # about 250 operations to draw, move, project and accumulate a sample; 1000 for a
    # Gaussian's Kalman terms; 20 for a (Gaussian, measurement) pair
    flops = n * g * (250.0 * p + 1000.0 + 20.0 * m)
    return {"bytes": float(bytes_), "flops": float(flops)}


# ------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    """The loaded state's update in 64 bits (the only case whose pass draws no samples and
    takes no threshold decisions that feed its outputs): every cloud projected into the
    parent's camera, fitted, and its Kalman likelihood of each measurement summed."""
    if case["kind"] != "restore":
        return None
    cfg, state, z = _restored(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dim, n, g, p = case["dim"], case["parents"], case["gaussians"], case["samples"]

    def t64(x):
        return torch.as_tensor(np.asarray(x), dtype=torch.float64, device=dev)

    ext = t64(state["states"])
    st, ct, sf, cf, sp, cp = (fn(ext[:, 6 + i]) for i in range(3) for fn in (torch.sin, torch.cos))
    rot = torch.stack([cf * cp, ct * sp + st * sf * cp, st * sp - ct * sf * cp,
                       -cf * sp, ct * cp - st * sf * sp, st * cp + ct * sf * sp,
                       sf, -st * cf, ct * cf], dim=1).reshape(n, 3, 3)
    zm, weights = t64(z[:, :dim]), t64(state["weights"]).reshape(n, g)
    omega = t64(state["omega"]).reshape(n, g, p)
    clouds = torch.as_tensor(state["clouds"]).reshape(n, g, 6, p)
    m = zm.shape[0]
    ell = torch.empty(n, m, dtype=torch.float64, device=dev)
    noise = torch.diag(t64([cfg.std_u ** 2, cfg.std_v ** 2, cfg.std_d ** 2][:dim]))
    other = math.log(m * cfg.w0 + cfg.kappa)
    for a in range(n):
        x = clouds[a].to(dev)
        pos = torch.einsum("ij,gjp->gip", rot[a], x[:, :3] - ext[a, :3, None])
        vel = torch.einsum("ij,gjp->gip", rot[a], x[:, 3:])
        iz = 1.0 / pos[:, 2]
        y = torch.stack([cfg.u0 - cfg.fx * pos[:, 0] * iz, cfg.v0 - cfg.fy * pos[:, 1] * iz,
                         -cfg.fx * cfg.baseline * iz,
                         -cfg.fx * (vel[:, 0] * pos[:, 2] - vel[:, 2] * pos[:, 0]) * iz * iz,
                         -cfg.fy * (vel[:, 1] * pos[:, 2] - vel[:, 2] * pos[:, 1]) * iz * iz,
                         cfg.fx * cfg.baseline * vel[:, 2] * iz * iz], dim=1)
        seen = ((y[:, 0] >= 0) & (y[:, 0] <= 2 * cfg.u0) & (y[:, 1] >= 0) & (y[:, 1] <= 2 * cfg.v0) & (y[:, 2] >= 0))
        w = omega[a] * cfg.pd * seen
        total = w.sum(1)
        fit = total > 0
        w = w / torch.where(fit, total, torch.ones_like(total))[:, None]
        mean = (w[:, None] * y).sum(2)
        dev_y = y - mean[:, :, None]
        cov = torch.einsum("gp,gip,gjp->gij", w, dev_y, dev_y) * (1 + (w * w).sum(1))[:, None, None]
        s = cov[:, :dim, :dim] + noise
        # the posterior's covariance has to be positive definite for a term to count
        gain = torch.linalg.solve(s, cov[:, :dim, :]).transpose(1, 2)
        post = cov - gain @ cov[:, :dim, :]
        fit = fit & (torch.linalg.cholesky_ex(post + 0.0)[1] == 0)
        nu = zm[None] - mean[:, None, :dim]
        quad = torch.einsum("gmi,gij,gmj->gm", nu, torch.linalg.inv(s), nu)
        pd_mean = cfg.pd * seen.double().mean(1)
        log_w = (torch.log(pd_mean * weights[a]) - 0.5 * dim * math.log(2 * math.pi) - 0.5 * torch.logdet(s))[:, None]
        term = torch.where(fit[:, None], log_w - 0.5 * quad, torch.full_like(quad, -math.inf))
        ell[a] = torch.logaddexp(torch.logsumexp(term, 0), t64(other))
    loglik = ell.sum(1) + weights.sum(1)
    lw = t64(state["log_weights"]) + loglik
    lw = lw - torch.logsumexp(lw, 0)
    return {"ell": ell, "loglik": loglik, "states": ext, "lw": lw}
