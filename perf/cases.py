"""The engine's work as its users call it: frames, batches of observers, gradients, caller rays and
scene rebuilds, each one pass through the public entry points of `specrel_b200`.

A case is a dict of plain values. `listed()` names the standing cases, `draw()` gives another of the
same ranges, `prepare()` makes what a program holds before the call (an engine with its scene
uploaded, the observers' uniform blocks and cameras, the output buffers), `run()` is one pass and
`work()` what a pass cannot do without. The scenes are the repository's synthetic workloads; the
observers, rays, flashes and targets come from the seed.
"""
import math

import numpy as np
import torch

import specrel_b200 as sr

FIRST_SIZE, LAST_SIZE = (64, 40), (1920, 1200)
MIXED = ((320, 200), (640, 400), (1280, 800), (1920, 1200))


def listed():
    return [
        # The drop-in call of an interactive host at its smallest: one frame of the cube scene into
        # host memory, blocking. Latency and launches.
        dict(name="frame_cubes_320x200", kind="host_frame", scene="cubes", bodies=64, width=320, height=200,
             slice=0, shadow=0),
        # One observer's frame of the 7.9M-tetrahedron scene, FP64 camera, null shadows, the pixels
        # staying on the device (a viewer that presents from there).
        dict(name="frame_accel_1280x800", kind="device_frame", scene="accel", bodies=64, width=1280, height=800,
             slice=0, shadow=1),
        # The headline: eight observers of the 7.9M-tetrahedron scene in one batch.
        dict(name="batch8_accel_1280x800", kind="batch", scene="accel", bodies=64, n=8, width=1280, height=800,
             mixed=False),
        # Many observers of mixed sizes, half past light cone and half God's-eye, in one batch: a
        # sweep of views over a small scene.
        dict(name="batch64_cubes_mixed", kind="batch", scene="cubes", bodies=64, n=64, width=1920, height=1200,
             mixed=True),
        # A ragged batch: odd sizes, every slice mode, every shadow mode, f32 cameras as the
        # reference's host has them.
        dict(name="batch5_accel_ragged", kind="ragged", scene="accel", bodies=16, n=5, width=1279, height=797),
        # A frame with the 100k-star sky behind the cubes.
        dict(name="frame_stars_1280x800", kind="device_frame", scene="stars", bodies=64, width=1280, height=800,
             slice=0, shadow=1),
        # A game frame with flashes, haze and a decision frontier, every side output read back
        # (picking, exports, physics probes).
        dict(name="frame_flash_801x501", kind="flash_frame", scene="accel", bodies=16, width=801, height=501,
             slice=0, shadow=1),
        # One step of a descent on the observer: loss and gradient at full resolution, and at the
        # coarse level a coarse-to-fine descent begins with.
        dict(name="grad_stars_1280x800_l0", kind="gradient", scene="stars", bodies=64, width=1280, height=800, level=0),
        dict(name="grad_stars_320x200_l3", kind="gradient", scene="stars", bodies=64, width=320, height=200, level=3),
        # Caller rays: probes, picking and aiming, from host arrays to host arrays.
        dict(name="rays_4096", kind="rays", scene="accel", bodies=8, n=4096),
        # An edited scene rebuilt from its worldtubes and looked at: the reference's dynamic scale
        # (12,672 tetrahedra), and one of 2M tetrahedra.
        dict(name="rebuild_13k", kind="rebuild", scene="cubes", bodies=11, steps=32, width=320, height=200),
        dict(name="rebuild_2m", kind="rebuild", scene="accel", bodies=16, steps=128, width=640, height=400),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["host_frame", "device_frame", "batch", "ragged", "flash_frame", "gradient", "rays", "rebuild"])
    w = _log_int(rng, FIRST_SIZE[0], LAST_SIZE[0])
    h = max(FIRST_SIZE[1], min(LAST_SIZE[1], int(w * rng.uniform(0.45, 0.85))))
    case = dict(kind=kind, width=w, height=h)
    if kind in ("host_frame", "device_frame"):
        case["scene"] = rng.choice(["cubes", "accel"] if kind == "host_frame" else ["cubes", "accel", "stars"])
        case["bodies"] = 64 if case["scene"] == "stars" else rng.choice([8, 16, 64])
        case["slice"] = 0 if case["scene"] == "stars" else rng.randrange(4)
        case["shadow"] = rng.randrange(3)
    elif kind == "batch":
        case["mixed"] = rng.random() < 0.5
        case["scene"] = "cubes" if case["mixed"] else rng.choice(["cubes", "accel"])
        case["bodies"] = rng.choice([16, 64])
        most = 64 if case["mixed"] else max(2, min(64, 8_000_000 // (w * h)))
        case["n"] = _log_int(rng, 2, most)
    elif kind == "ragged":
        case["scene"], case["bodies"] = rng.choice(["cubes", "accel"]), 16
        case["n"] = _log_int(rng, 2, max(2, min(24, 6_000_000 // (w * h))))
    elif kind == "flash_frame":
        case["width"], case["height"] = min(w, 1280), min(h, 800)
        case["scene"], case["bodies"] = rng.choice(["cubes", "accel"]), rng.choice([8, 16])
        case["slice"], case["shadow"] = rng.randrange(3), rng.randrange(3)
    elif kind == "gradient":
        case["width"], case["height"] = min(w, 1280), min(h, 800)
        case["scene"], case["bodies"], case["level"] = rng.choice(["cubes", "stars"]), 64, rng.randrange(7)
    elif kind == "rays":
        case["scene"], case["bodies"], case["n"] = rng.choice(["cubes", "accel"]), 8, _log_int(rng, 1, 16384)
    else:
        case["width"], case["height"] = min(w, 1280), min(h, 800)
        case["scene"] = rng.choice(["cubes", "accel"])
        case["bodies"] = rng.choice([3, 8, 16])
        case["steps"] = _log_int(rng, 16, 128)
    return case


# ---- scenes: the workloads' own, made once per process (what a program loads from disk) ----
_CONFIG = {"cubes": 1, "accel": 2, "stars": 5}
_scenes = {}


def _scene(case):
    key = (case["scene"], case["bodies"], case.get("steps"))
    if key not in _scenes:
        _scenes[key] = sr.synth_scene(_CONFIG[case["scene"]], 1, n_bodies=case["bodies"], steps=case.get("steps"))
    return _scenes[key]


def _ball(rng, radius):
    while True:
        v = rng.uniform(-1.0, 1.0, 3)
        if v @ v < 1.0:
            return tuple(float(radius * x) for x in v)


def _observer(case, rng):
    """An event and a rapidity: the accelerated bodies are seen from near the origin at t = 0, the
    cubes from anywhere among them at t in [-50, 0]."""
    if case["scene"] == "accel":
        return (0.0,) + _ball(rng, 1.0), _ball(rng, 2.0)
    if case["scene"] == "stars":
        return (0.0, 0.0, 0.0, 0.0), _ball(rng, 0.9)
    return (float(rng.uniform(-50.0, 0.0)),) + _ball(rng, 30.0), _ball(rng, 2.0)


def _uniforms(scene, pos, rapidity, w, h, **kw):
    kw.setdefault("num_stars", scene.num_stars)
    return sr.uniforms(sr.camera(pos, 90.0, rapidity=rapidity), w, h, num_nodes=scene.num_nodes,
                       light_pos=scene.light_pos, **kw)


def _view(case, scene, rng, **kw):
    pos, rap = _observer(case, rng)
    kw.setdefault("slice_mode", case.get("slice", 0))
    kw.setdefault("shadow_mode", case.get("shadow", 0))
    return _uniforms(scene, pos, rap, case["width"], case["height"], **kw), sr.cam64(pos, rap)


def _rays(case, seed):
    """Rays from one event along its past light cone in every direction (t, x, y, z; direction; range)."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    pos, _ = _observer(case, rng)
    d = rng.normal(size=(n, 3))
    rays = np.zeros((n, 10))
    rays[:, 0:4] = pos
    rays[:, 4] = -1.0
    rays[:, 5:8] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 8], rays[:, 9] = 1e-3, 180.0
    return rays


def _sizes(case):
    """The frame sizes of a batch's observers, the case's own (not the seed's)."""
    w, h, n = case["width"], case["height"], case["n"]
    if case["kind"] == "ragged":
        rng = np.random.default_rng([w, h, n])
        return [(int(w * rng.uniform(0.2, 1.0)) | 1, int(h * rng.uniform(0.2, 1.0)) | 1) for _ in range(n)]
    return [MIXED[i % 4] if case["mixed"] else (w, h) for i in range(n)]


def _pixels(n):
    return torch.zeros(n, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    scene = _scene(case)
    eng = sr.Engine(torch.cuda.current_device())
    state = dict(kind=kind, eng=eng, scene=scene)
    if kind == "rebuild":
        pos, rap = _observer(case, rng)
        state["u"] = _uniforms(scene, pos, rap, case["width"], case["height"], mode=0, shadow_mode=1)
        return state
    eng.build_tubes(0, scene)
    if kind == "rays":
        state["rays"] = _rays(case, seed)
        return state
    if kind in ("host_frame", "device_frame"):
        u, cam = _view(case, scene, rng)
        state.update(u=u, cam=cam)
        n = case["width"] * case["height"]
        if kind == "host_frame":
            state["fb"] = np.zeros(n, np.uint32)
        else:
            state["out"] = _pixels(n)
    elif kind == "flash_frame":
        pos, rap = _observer(case, rng)
        t = pos[0]
        # Shells whose fronts cross what the observer sees (a flash lights the past light cone at
        # twice its distance), one remote frontier and a decision frontier.
        flashes = [((t - float(rng.uniform(4.0, 40.0)),) + _ball(rng, 12.0), float(rng.uniform(0.5, 8.0)),
                    float(rng.uniform(1.0, 4.0)), tuple(float(x) for x in rng.uniform(0.2, 1.0, 3))) for _ in range(4)]
        remote = [(t - float(rng.uniform(1.0, 10.0)),) + _ball(rng, 8.0)]
        state["u"] = _uniforms(scene, pos, rap, case["width"], case["height"], slice_mode=case["slice"],
                               shadow_mode=case["shadow"], flashes=flashes, remote_origins=remote,
                               frontier=(pos, 0.0))
    elif kind in ("batch", "ragged"):
        us, cams = [], []
        for i, (w, h) in enumerate(_sizes(case)):
            pos, rap = _observer(case, rng)
            slice_mode, shadow = 0, 1
            if kind == "ragged":
                slice_mode, shadow = i % 4, int(rng.integers(0, 3))
            elif case["mixed"]:
                slice_mode = i // 4 % 2
                shadow = 2 if slice_mode else 1
                rap = tuple(1.5 * x for x in rap)
            us.append(_uniforms(scene, pos, rap, w, h, slice_mode=slice_mode, shadow_mode=shadow))
            cams.append(sr.cam64(pos, rap))
        n = sum(u.size[0] * u.size[1] for u in us)
        state.update(us=us, cams=None if kind == "ragged" else cams, n=n, out=_pixels(n))
    elif kind == "gradient":
        w, h = case["width"], case["height"]
        at = (0.0, 0.0, 0.0, 0.0) if case["scene"] == "stars" else _observer(case, rng)[0]
        u = _uniforms(scene, at, (0.0, 0.0, 0.0), w, h, shadow_mode=1)
        target = eng.render(0, u, hdr=True, cam=sr.cam64(at, _ball(rng, 1.0))).hdr
        state.update(u=u, cam=sr.cam64(at, _ball(rng, 0.3)), level=case["level"], target=torch.tensor(target).cuda())
    else:
        raise ValueError(kind)
    return state


def run(state):
    eng, kind = state["eng"], state["kind"]
    if kind == "host_frame":
        eng.render_host(0, state["u"], state["fb"])
        return state["fb"]
    if kind == "device_frame":
        eng.render_into(0, state["u"], state["out"].data_ptr(), cam=state["cam"])
        return state["out"]
    if kind in ("batch", "ragged"):
        eng.render_batch(0, state["us"], state["out"].data_ptr(), state["n"], cams=state["cams"])
        return state["out"]
    if kind == "flash_frame":
        f = eng.render(0, state["u"], aux=True, hdr=True)
        return dict(rgb=f.rgb, hit_id=f.hit_id, lam=f.lam, tau=f.tau, hdr=f.hdr)
    if kind == "gradient":
        r = eng.adjoint(0, state["u"], state["cam"], state["target"].data_ptr(), level=state["level"])
        return dict(loss=r.loss, grad=[r.grad[k] for k in range(7)])
    if kind == "rays":
        h = eng.trace_rays(0, state["rays"])
        return {k: np.ascontiguousarray(h[k]) for k in h.dtype.names if k != "pad"}
    if kind == "rebuild":
        eng.build_tubes(0, state["scene"])
        f = eng.render(0, state["u"], aux=True)
        return dict(rgb=f.rgb, hit_id=f.hit_id, lam=f.lam, tau=f.tau)
    raise ValueError(kind)


_TETS = {"cubes": lambda b, s: b * 36 * (s or 64), "accel": lambda b, s: b * 960 * (s or 128),
         "stars": lambda b, s: b * 36 * (s or 64)}


def work(case):
    """What a pass cannot do without: every output written once, and of the scene the records that the
    rays end on (80 bytes hot and 192 cold, at most one of each per ray and tetrahedron). Per ray two
    box tests (24 operations each) per level of a balanced binary tree and one tetrahedron test, and
    about 200 operations of shading; a rebuild reads and writes every record once."""
    tets = _TETS[case["scene"]](case["bodies"], case.get("steps"))
    kind = case["kind"]
    if kind == "rays":
        rays, out = case["n"], case["n"] * (56 + 80)
    else:
        sizes = _sizes(case) if "n" in case else [(case["width"], case["height"])]
        rays = sum(w * h for w, h in sizes)
        out = rays * {"flash_frame": 32, "gradient": 48, "rebuild": 16}.get(kind, 4)
    per_ray = 2 * 24 * math.log2(max(2, tets / 3)) + 60 + 200
    byte, flop = out + min(rays, tets) * (80 + 192), rays * per_ray
    if case["scene"] == "stars":
        byte += 100000 * 64
        flop += 100000 * 100
    if kind == "rebuild":
        byte += tets * (80 + 192 + 48)
        flop += tets * 300
    return {"bytes": byte, "flops": flop}


def exact(case, seed):
    """The caller rays in 64 bits: every ray against every tetrahedron of the scene's records, the
    nearest hit kept. Frames pass through texture lookups and 8-bit packing, a gradient through a
    whole frame; neither has a plain 64-bit form."""
    if case["kind"] != "rays":
        return None
    names = ("id", "slot", "lambda_", "proper_time", "event", "tet_bary", "uv", "material")
    packed = _scene(case).packed()
    g = torch.from_numpy(np.ascontiguousarray(packed.geoms).view(np.float32).reshape(-1, 5, 4).copy()).cuda().double()
    r = torch.from_numpy(_rays(case, seed)).cuda()
    o, d = r[:, 0:4].float().double(), r[:, 4:8].float().double()
    t0, t1 = r[:, 8:9].float().double(), r[:, 9:10].float().double()
    best = torch.full((len(r),), math.inf, dtype=torch.float64, device="cuda")
    chunk = max(1, 40_000_000 // len(r))
    eps = -1e-5
    for a in range(0, len(g), chunk):
        v0, n, b = g[a:a + chunk, 0], g[a:a + chunk, 1], g[a:a + chunk, 2:5]
        den = d @ n.T
        lam = ((v0 * n).sum(1)[None, :] - o @ n.T) / den
        ok = (den.abs() >= 1e-9) & (lam > t0) & (lam < t1)
        total = torch.zeros_like(lam)
        for k in range(3):
            c = o @ b[:, k].T + lam * (d @ b[:, k].T) - (v0 * b[:, k]).sum(1)[None, :]
            total += c
            ok &= (c >= eps) & (total <= 1.0 - eps)
        best = torch.minimum(best, torch.where(ok, lam, math.inf).min(1).values)
    lam = torch.where(best.isfinite(), best, 0.0).cpu().numpy()
    out = dict.fromkeys(names)
    out["lambda_"] = lam
    out["event"] = np.where((lam > 0.0)[:, None], o.cpu().numpy() + d.cpu().numpy() * lam[:, None], 0.0)
    return out
