"""The work this library is used for, as measurable cases.

Each case is one call (or one short sequence of calls) of the public entry
points, as a simulator, a surrogate's training program or a reinforcement-
learning rollout makes it:

  ``body``     one body through host buffers (the reference's per-body call
               of a simulator tick, where latency is all);
  ``batch``    a batch of bodies resident on the device: sphere states, the
               mixed batch of distinct meshes, torpedoes over waves;
  ``host``     a vehicle fleet in pageable host arrays, with jet and pipe
               currents and FP64 cut points;
  ``cables``   cables in host arrays;
  ``sea``      the FFT ocean advanced to a time, then depth queries on it;
  ``mlp``      the surrogate network alone;
  ``predict``  the gated two-network surrogate with its exact fallback;
  ``train``    an epoch of the surrogate's training;
  ``rollout``  hulls stepped on the device in a captured graph.

``exact`` restates every one in 64 bits with plain torch and numpy.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from stonefish_gb300 import abi, meshes, rollout as RO, scenarios
from stonefish_gb300 import surrogate as S
from stonefish_gb300.hydro import FftOcean, HydroContext, fft_ocean_params

DEV = "cuda"


def listed() -> list[dict]:
    return [
        # one sphere of a simulator's scene, 1280 faces, per-body host call
        {"name": "body_sphere", "kind": "body", "shape": "sphere", "faces": 1280, "waves": False},
        # one detailed hull on waves, per-body host call
        {"name": "body_hull_waves", "kind": "body", "shape": "torpedo", "faces": 20000, "waves": True},
        # 1000 states of one sphere in one call (a trajectory evaluated at once)
        {"name": "sphere_states", "kind": "batch", "scene": "spheres", "n": 1000, "faces": 1280, "centred": True},
        # the headline batch: 4096 bodies with meshes of their own, 37.8M faces, flat sea
        {"name": "mixed_flat", "kind": "batch", "scene": "mixed", "n": 4096, "faces": 50000, "centred": True},
        # 1024 torpedoes of 20000 faces straddling a wave field
        {"name": "torpedo_waves", "kind": "batch", "scene": "torpedoes", "n": 1024, "faces": 20000, "centred": True},
        # a fleet stepped from a host program: numpy arrays, world frame, currents that vary in space, FP64 cuts
        {"name": "fleet_host", "kind": "host", "n": 200, "faces": 12288},
        # moorings and tethers of a scene, from a host program
        {"name": "cables", "kind": "cables", "n": 300, "nodes": 400},
        # the sea state advanced by one tick and sampled by sensors
        {"name": "sea_tick", "kind": "sea", "passes": 8, "points": 4096},
        # the surrogate network alone, the largest inference batch
        {"name": "mlp_65536", "kind": "mlp", "n": 65536},
        # gated surrogate prediction of 65536 hull states, about 2% of them sent to the exact step
        {"name": "predict_65536", "kind": "predict", "n": 65536},
        # training: one epoch of 64 batches of 4096
        {"name": "train_4096", "kind": "train", "batch": 4096, "steps": 64},
        # 16384 hulls rolled out with the surrogate, 20 steps per replay
        {"name": "rollout_16384", "kind": "rollout", "n": 16384, "mode": "surrogate", "steps": 20},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["body", "batch", "batch", "batch", "host", "cables", "sea", "mlp", "predict", "train", "rollout"])
    if kind == "body":
        return {"kind": kind, "shape": rng.choice(["sphere", "torpedo"]), "faces": _log_int(rng, 320, 20480),
                "waves": rng.random() < 0.5}
    if kind == "batch":
        scene = rng.choice(["spheres", "mixed", "torpedoes"])
        n = {"spheres": _log_int(rng, 3, 4000), "mixed": _log_int(rng, 5, 3000), "torpedoes": _log_int(rng, 2, 1000)}[scene]
        faces = {"spheres": _log_int(rng, 80, 5120), "mixed": _log_int(rng, 1000, 50000),
                 "torpedoes": _log_int(rng, 500, 20000)}[scene]
        return {"kind": kind, "scene": scene, "n": n, "faces": faces, "centred": rng.random() < 0.5}
    if kind == "host":
        return {"kind": kind, "n": _log_int(rng, 2, 300), "faces": _log_int(rng, 500, 12288)}
    if kind == "cables":
        return {"kind": kind, "n": _log_int(rng, 1, 600), "nodes": _log_int(rng, 8, 400)}
    if kind == "sea":
        return {"kind": kind, "passes": rng.randint(5, 9), "points": _log_int(rng, 1, 65536)}
    if kind == "mlp":
        return {"kind": kind, "n": _log_int(rng, 1, 65536)}
    if kind == "predict":
        return {"kind": kind, "n": _log_int(rng, 33, 65536)}
    if kind == "train":
        batch = 64 * _log_int(rng, 4, 128)
        return {"kind": kind, "batch": batch, "steps": rng.randint(8, min(64, 262144 // batch))}
    mode = rng.choice(["exact", "surrogate"])
    return {"kind": kind, "n": _log_int(rng, 17, 16384 if mode == "surrogate" else 1024), "mode": mode,
            "steps": rng.randint(2, 20)}


# ------------------------------------------------------------------ scenes
def _sphere_mesh(faces: int):
    """Icosphere with the subdivision nearest to ``faces`` (20 * 4^s)."""
    s = max(1, min(5, int(round(math.log(max(faces, 20) / 20.0, 4)))))
    return meshes.build_icosphere(0.5, s)


@functools.lru_cache(maxsize=3)
def _wave_field(k: int) -> dict:
    return scenarios.wave_grid(seed=7 + k)


def _waves(seed: int) -> dict:
    """One of three wave fields (each takes a second to build)."""
    return _wave_field(seed % 3)


def _torpedoes(n: int, seed: int, faces: int, at_surface: bool) -> dict:
    """Torpedo hulls over the wave field, CG depth U(-0.5, 0.2) m (about the
    local surface with ``at_surface``)."""
    rng = np.random.default_rng(seed)
    r, L, size = 0.25, 2.0, 102.4
    R, pos, v, w = scenarios.random_states(rng, n, (-0.5, 0.2))
    pos[:, :2] = rng.uniform(0.0, size, (n, 2))
    if at_surface:
        ij = (pos[:, :2] / size * 1024).astype(int) % 1024
        pos[:, 2] = 0.4 * pos[:, 2] - _waves(seed)["data"][ij[:, 1], ij[:, 0]]
    bodies = scenarios.fill_bodies(n, R, pos, v, w, np.tile([0.5 * L + r, r, r], (n, 1)),
                                   meshes.capped_cylinder_volume(r, L), meshes.capped_cylinder_surface(r, L),
                                   (1.0, 0.5, 0.5), (0.1, 0.05, 0.05), 0)
    return {"meshes": [meshes.capped_cylinder_for_faces(r, L, faces)], "bodies": bodies, "ocean": scenarios.flat_ocean()}


def _scene(case: dict, seed: int) -> dict:
    """Host inputs of an exact-step case: meshes, bodies, ocean, wave grid."""
    if case["kind"] == "body":
        n, scene = 1, "spheres" if case["shape"] == "sphere" else "torpedoes"
        waves = case["waves"]
    else:
        n, scene = case["n"], case.get("scene", "mixed")
        waves = scene == "torpedoes"
    rng = np.random.default_rng(1000 + seed)
    if scene == "spheres":
        sc = scenarios.single_sphere(steps=n, seed=seed, depth=(-0.4, 0.2) if case["kind"] == "body" else (-1.0, 0.3))
        sc["meshes"] = [_sphere_mesh(case["faces"])]
    elif scene == "torpedoes":
        sc = _torpedoes(n, seed, case["faces"], at_surface=case["kind"] == "body" and waves)
    else:
        sc = scenarios.mixed_batch(n, seed=seed, scale_faces=case["faces"] / 50000.0)
    sc["waves"] = _waves(seed) if waves else None
    sc["ocean"].waves = int(waves)
    if case["kind"] == "host":   # a jet and a pipe next to the uniform current
        o = sc["ocean"]
        o.n_currents = 3
        j, p = o.currents[1], o.currents[2]
        j.type, j.enabled, j.radius, j.speed = abi.CURRENT_JET, 1, 0.5, 1.5
        p.type, p.enabled, p.radius, p.radius2, p.length, p.speed, p.gamma = abi.CURRENT_PIPE, 1, 6.0, 9.0, 60.0, 0.8, 1.0 / 7.0
        for k in range(3):
            j.point[k] = (-60.0, rng.uniform(-5, 5), 0.3)[k]
            j.dir[k] = (1.0, 0.0, 0.0)[k]
            p.point[k] = (rng.uniform(-5, 5), -30.0, 0.2)[k]
            p.dir[k] = (0.0, 1.0, 0.0)[k]
    return sc


def _bytes(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.frombuffer(a.tobytes(), dtype=np.uint8).copy()).to(DEV)


def _cable_scene(case: dict, seed: int) -> dict:
    """``n`` cables of up to ``nodes`` nodes sagging across the surface, some
    wholly under water, some dry."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    cables = np.zeros(n, dtype=abi.CABLE_DTYPE)
    counts = np.random.default_rng(n).integers(max(2, case["nodes"] // 4), case["nodes"] + 1, n)
    xs, vs, first = [], [], 0
    for c in range(n):
        m = int(counts[c])
        t = np.linspace(0.0, 1.0, m)
        x0 = rng.uniform(-20, 20, 3)
        kind = c % 4
        z = {0: 2.0 + np.sin(3 * t), 1: -3.0 - t}.get(kind)
        if z is None:
            z = rng.uniform(-1.0, 0.3) + rng.uniform(0.2, 3.0) * (1 - (2 * t - 1) ** 2)
        xs.append(np.stack([x0[0] + rng.uniform(2, 10) * t, x0[1] + rng.uniform(-1, 1) * t, z], axis=1))
        vs.append(rng.uniform(-1.0, 1.0, (m, 3)))
        cables[c] = (first, m, rng.uniform(0.01, 0.08), abi.MODE_SUBMERGED, 1)
        first += m
    return {"cables": cables, "x": np.concatenate(xs), "v": np.concatenate(vs),
            "ocean": scenarios.flat_ocean(current=(0.3, -0.1, 0.0))}


def _sea_scene(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    pts = np.zeros((case["points"], 3), dtype=np.float32)
    pts[:, :2] = rng.uniform(-200, 200, (case["points"], 2))
    pts[:, 2] = rng.uniform(-1, 5, case["points"])
    return {"params": fft_ocean_params(float(rng.uniform(0.3, 1.5)), case["passes"]), "t": float(rng.uniform(0, 60)),
            "points": pts, "ocean": S.wave_ocean()}


def _set_net(net: S.Surrogate, F: torch.Tensor, T: torch.Tensor, scales) -> None:
    """A working network without a training run: the hidden layers as they are
    initialised (random features), the last one fitted to the labels by ridge
    regression in 64 bits."""
    net.fit_normalisation(F, T, target_scales=scales)
    x = (F.double() - net.f_mean.double()) * net.f_istd.double()
    t = (T.double() - net.t_mean.double()) * net.t_istd.double()
    for l in range(3):
        k = S.N_FEAT if l == 0 else net.layers[l]["k"]
        x = torch.nn.functional.silu(x @ net.layers[l]["w"][:k].double() + net.layers[l]["b"].double())
    x = torch.cat([x, torch.ones_like(x[:, :1])], dim=1).cpu()
    A = x.T @ x + 1e-2 * torch.eye(x.shape[1], dtype=torch.float64)
    w = torch.linalg.solve(A, x.T @ t.cpu())
    net.layers[3]["w"][:, :S.N_OUT] = w[:-1].float().to(DEV)
    net.layers[3]["b"][:S.N_OUT] = w[-1].float().to(DEV)


def _nets(seed: int, faces: int, ranges: dict, count: int = 12288) -> dict:
    """A context with the hull and its wave field, and two networks fitted on
    states labelled by the exact step."""
    h = HydroContext(0)
    mid = h.upload_mesh(*S.hull_mesh(faces))
    waves = _waves(seed)
    h.set_wave_grid(waves)
    ocean, st = S.wave_ocean(), scenarios.settings()
    if "surface" in ranges:
        ranges = dict(ranges, surface=RO.surface_z(h, ocean))
    lab = S.Labeller(h, mid, ocean, st, chunk=count)
    F, T = S.generate(lab, count, seed=300 + seed, **ranges)
    fs, ts = S.hull_scales(ocean)
    scales = (fs, ts) if faces == S.HULL_FACES else (fs, fs, fs, ts / 10.0, ts, ts)
    nets = [S.Surrogate(h, seed=2 * seed + k) for k in (0, 1)]
    for net in nets:
        _set_net(net, F, T, scales)
    lab.close()
    return {"h": h, "mid": mid, "waves": waves, "ocean": ocean, "st": st, "nets": nets, "F": F, "T": T}


PREDICT_RANGES = {}                        # the hull states' own ranges
ROLLOUT_RANGES = {"depth": (-0.5, 0.6), "v_range": 3.0, "w_body": (10.0, 2.5, 2.5), "surface": True}


def _tau(d: dict) -> float:
    """The disagreement that 1% of the labelled states exceed."""
    fs, ts = S.hull_scales(d["ocean"])
    z = torch.zeros((d["F"].shape[0], 16), dtype=torch.float32, device=DEV)
    a, b = (net.infer_tc(d["F"], z, net.tc_weights())[:, :6].double().clone() for net in d["nets"])
    dis = torch.maximum((a - b)[:, :3].norm(dim=1) / fs, (a - b)[:, 3:].norm(dim=1) / ts)
    return float(np.quantile(dis.cpu().numpy(), 0.99).astype(np.float32))


def _train_rows(case: dict, seed: int):
    """Features over the training ranges and smooth wrench-like targets."""
    n = case["batch"] * case["steps"] + seed % 61
    g = torch.Generator(device=DEV).manual_seed(seed)
    F = torch.rand((n, S.N_FEAT), generator=g, device=DEV) * 2.0 - 1.0
    F[:, 1:3] *= 1.5
    W = torch.randn((S.N_FEAT, S.N_OUT), generator=g, device=DEV)
    T = torch.tanh(F @ W) * 800.0 + 300.0 * F[:, 3:9] * F[:, 3:9].abs()
    return F.contiguous(), T.contiguous()


def _rollout_start(d: dict, case: dict, seed: int) -> np.ndarray:
    return RO.initial_states(np.random.default_rng(404 + seed), case["n"], surface=RO.surface_z(d["h"], d["ocean"]))


# ------------------------------------------------------------------ prepare
def _wrench_views(io: torch.Tensor, n: int) -> dict:
    """hydro_wrench records as (n, 20) FP64 values and (n, 2) position/status words."""
    return {"wrench": io.view(torch.float64).view(n, 21)[:, :20], "flags": io.view(torch.int32).view(n, 42)[:, 40:]}


def _host_views(io: np.ndarray) -> dict:
    return {"wrench": io.view(np.float64).reshape(-1, 21)[:, :20], "flags": io.view(np.int32).reshape(-1, 42)[:, 40:]}


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("body", "batch", "host"):
        sc = _scene(case, seed)
        frame = abi.FRAME_CENTRED if case.get("centred") else abi.FRAME_WORLD
        h = HydroContext(0, frame=frame, cut_precision=abi.CUT_FP64 if kind == "host" else abi.CUT_FP32)
        ids = np.array([h.upload_mesh(*m) for m in sc["meshes"]], dtype=np.uint32)
        if sc["waves"] is not None:
            h.set_wave_grid(sc["waves"])
        bodies = sc["bodies"].copy()
        bodies["mesh"] = ids[bodies["mesh"]]
        n = bodies.size
        s = {"kind": kind, "h": h, "ocean": sc["ocean"], "st": scenarios.settings()}
        if kind == "batch":
            # the headline batch in chunks of 24 tiles, as its tuned runs are
            s["b"] = h.batch(bodies["mesh"], chunk_faces=10752 if case["scene"] == "mixed" and n > 1024 else 0)
            s["bodies"] = _bytes(bodies)
            s["io"] = torch.zeros(n * abi.WRENCH_DTYPE.itemsize, dtype=torch.uint8, device=DEV)
            s["out"] = _wrench_views(s["io"], n)
        else:
            s["bodies"], s["io"] = bodies, scenarios.new_wrenches(n)
            s["out"] = _host_views(s["io"])
            s["b"] = h.batch(bodies["mesh"]) if kind == "host" else None
        return s
    if kind == "cables":
        sc = _cable_scene(case, seed)
        out = np.zeros(sc["x"].shape[0], dtype=abi.CABLE_FORCES_DTYPE)
        return {"kind": kind, "h": HydroContext(0), "st": scenarios.settings(), "io": out,
                "out": out.view(np.float64).reshape(-1, 9), **sc}
    if kind == "sea":
        sc = _sea_scene(case, seed)
        h = HydroContext(0)
        return {"kind": kind, "h": h, "sea": FftOcean(h, sc["params"]), **sc}
    if kind == "mlp":
        d = _nets(seed, S.HULL_FACES, PREDICT_RANGES, 4096)
        n = case["n"]
        F = d["F"].repeat((n + 4095) // 4096, 1)[:n]
        g = torch.Generator(device=DEV).manual_seed(seed)
        F = (F + 0.05 * torch.randn(F.shape, generator=g, device=DEV)).contiguous()
        net = d["nets"][0]
        return {"kind": kind, "d": d, "net": net, "F": F, "tcw": net.tc_weights(),
                "out": torch.zeros((n, 16), dtype=torch.float32, device=DEV)}
    if kind == "predict":
        d = _nets(seed, S.HULL_FACES, PREDICT_RANGES)
        b = S.sample_states(np.random.default_rng(202 + seed), case["n"])
        b["mesh"] = d["mid"]
        gp = S.GatedPredictor(d["nets"][0], d["h"], d["mid"], case["n"], d["ocean"], d["st"], second=d["nets"][1],
                              tau=_tau(d), gate_inside=True, audit_stride=1024)
        return {"kind": kind, "d": d, "gp": gp, "bodies": _bytes(b)}
    if kind == "train":
        h = HydroContext(0)
        F, T = _train_rows(case, seed)
        net = S.Surrogate(h, batch=case["batch"], seed=seed)
        net.fit_normalisation(F, T, sample=65536)
        return {"kind": kind, "h": h, "net": net, "F": F, "T": T}
    # rollout
    d = _nets(seed, 8000, ROLLOUT_RANGES)
    start = _rollout_start(d, case, seed)
    gp = None
    if case["mode"] == "surrogate":
        gp = S.GatedPredictor(d["nets"][0], d["h"], d["mid"], case["n"], d["ocean"], d["st"], second=d["nets"][1])
    ro = RO.Rollout(d["h"], d["mid"], case["n"], d["ocean"], d["st"], case["mode"], predictor=gp)
    ro.reset(start)
    ro.capture(case["steps"], snap_every=case["steps"])
    return {"kind": kind, "d": d, "gp": gp, "ro": ro, "start": _bytes(start),
            "out": ro.states.view(torch.float64).view(case["n"], 27)}


# ---------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "body":
        s["h"].body_forces(s["bodies"], s["ocean"], s["st"], s["io"])
        return s["out"]
    if kind == "batch":
        s["b"].compute_device(s["bodies"].data_ptr(), s["ocean"], s["st"], s["io"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
        return s["out"]
    if kind == "host":
        s["b"].compute(s["bodies"], s["ocean"], s["st"], s["io"])
        return s["out"]
    if kind == "cables":
        s["h"].cable_forces(s["cables"], s["x"], s["v"], s["ocean"], s["st"], s["io"])
        return s["out"]
    if kind == "sea":
        s["sea"].update(s["t"])
        torch.cuda.current_stream().synchronize()   # depth() works on a stream of its own
        return s["h"].depth(s["ocean"], s["points"])
    if kind == "mlp":
        return s["net"].infer_tc(s["F"], s["out"], s["tcw"])
    if kind == "predict":
        return s["gp"].predict(s["bodies"])
    if kind == "train":
        info = s["net"].fit(s["F"], s["T"], epochs=1, lr=3e-3)
        return {"loss": info["loss"][-1], "w": [L["w"] for L in s["net"].layers], "b": [L["b"] for L in s["net"].layers],
                "gw": [L["gw"] for L in s["net"].layers], "gb": [L["gb"] for L in s["net"].layers]}
    ro = s["ro"]
    # a new episode: the start states and the body records they imply, then the captured steps
    ro.states.copy_(s["start"])
    ro.lib.hydro_rigid_write_bodies(ro.h.ctx, C.c_void_p(ro.states.data_ptr()), C.c_void_p(ro.bodies.data_ptr()), ro.n,
                                    torch.cuda.current_stream().cuda_stream)
    ro.replay()
    return s["out"]


# --------------------------------------------------------------------- work
FACE_FLOPS, WAVE_FLOPS = 170, 90      # one submerged face on a flat sea; more for its surface lookups on waves
MLP_FLOPS = 2 * (16 * 256 + 256 * 256 * 2 + 256 * 6)


def _face_work(n_faces_each: float, n: float, distinct: float, waves: bool, grid: int = 1024) -> dict:
    """``n`` bodies: the faces of ``distinct`` meshes read once (three indices
    and half a vertex a face), body records in, wrenches in and out."""
    return {"bytes": 18.0 * n_faces_each * distinct + n * (464 + 2 * 168) + (4.0 * grid * grid if waves else 0.0),
            "flops": 0.65 * n * n_faces_each * (FACE_FLOPS + (WAVE_FLOPS if waves else 0))}


def work(case: dict) -> dict:
    kind, n = case["kind"], case.get("n", 1)
    if kind == "body":
        return _face_work(case["faces"], 1, 1, False)
    if kind == "batch" and case["scene"] != "mixed":
        return _face_work(case["faces"], n, 1, case["scene"] == "torpedoes")
    if kind in ("batch", "host"):
        return _face_work(9235.0 * min(1.0, case["faces"] / 50000.0), n, n, False)
    if kind == "cables":
        nodes = 0.625 * n * case["nodes"]
        return {"bytes": nodes * (48 + 72), "flops": nodes * 250}
    if kind == "sea":
        N = 1 << case["passes"]
        return {"bytes": N * N * (32 + 16) + 16.0 * case["points"], "flops": N * N * (120 + 2 * case["passes"] * 16)}
    if kind == "mlp":
        return {"bytes": n * (64 + 64) + 303104.0, "flops": n * MLP_FLOPS}
    if kind in ("predict", "rollout"):
        steps = case.get("steps", 1)
        faces = S.HULL_FACES if kind == "predict" else 8000
        if case.get("mode") == "exact":
            one, share = {"bytes": 0.0, "flops": 0.0}, 1.0
        else:
            one, share = {"bytes": n * 24.0 + 2 * 303104.0, "flops": 2.0 * n * MLP_FLOPS}, 0.02 if kind == "predict" else 0.005
        ex = _face_work(faces, n * share, 1, True)
        return {"bytes": steps * (one["bytes"] + ex["bytes"] + n * (464 + (2 * 216 if kind == "rollout" else 0))),
                "flops": steps * (one["flops"] + ex["flops"])}
    B, k = case["batch"], case["steps"]
    params = 64 * 256 + 2 * 256 * 256 + 256 * 64
    return {"bytes": k * (B * (128 + 24) + params * 4.0 * 8), "flops": k * 6.0 * B * params}


# -------------------------------------------------------------------- exact
def _t64(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)


class _Wave:
    """The periodic bilinear surface of a texel-centred height grid (layers
    summed), and the flat sea when there is none."""

    def __init__(self, layers):
        self.layers = layers              # [(grid [N, N] FP64 elevation, size)]

    def elevation(self, x, y):
        e = torch.zeros_like(x)
        for g, size in self.layers:
            N = g.shape[0]
            u, v = x / size - 0.5 / N, y / size - 0.5 / N
            u, v = (u - torch.floor(u)) * N, (v - torch.floor(v)) * N
            i, j = torch.floor(u), torch.floor(v)
            a, b = u - i, v - j
            i0, j0 = i.long() % N, j.long() % N
            i1, j1 = (i0 + 1) % N, (j0 + 1) % N
            e = e + (1 - a) * (1 - b) * g[j0, i0] + a * (1 - b) * g[j0, i1] + (1 - a) * b * g[j1, i0] + a * b * g[j1, i1]
        return e

    def depth(self, x, y, z):
        return z + self.elevation(x, y) if self.layers else z


def _grid_wave(waves) -> _Wave:
    return _Wave([] if waves is None else [(_t64(waves["data"]), waves["layers"][0][1])])


def _fluid_velocity(ocean, p):
    """Sum of the ocean's currents at points p [..., 3]."""
    u = torch.zeros_like(p)
    for i in range(ocean.n_currents if ocean.currents_enabled else 0):
        c = ocean.currents[i]
        if not c.enabled:
            continue
        if c.type == abi.CURRENT_UNIFORM:
            u = u + _t64(c.vel[:])
            continue
        d, r = _t64(c.dir[:]), p - _t64(c.point[:])
        dist = torch.linalg.cross(r, d.expand_as(r)).norm(dim=-1)
        t = (r * d).sum(-1)
        if c.type == abi.CURRENT_JET:
            on = (t >= 0) & (dist < (t + 5.0 * c.radius) / 5.0)
            s = 10.0 * c.radius / (t + 5.0 * c.radius) * c.speed * torch.exp(-50.0 * dist * dist / (t * t))
        else:
            R = c.radius + (c.radius2 - c.radius) * t / c.length
            on = (t >= 0) & (t <= c.length) & (dist < R)
            s = c.radius / R * c.speed * (1.0 - dist / R).clamp(min=0).pow(c.gamma)
        u = u + torch.where(on, s, torch.zeros_like(s))[..., None] * d
    return u


def _polygons(acc, b, corners, B, ocean, wave, volume):
    """Adds the terms of planar polygons (``corners`` a list of [m, 3], ``b``
    the body of each) to acc [bodies, 23]: Fb Tb Fdq Tdq Fdf Tdf Swet V6 CB6."""
    if b.numel() == 0:
        return
    add = (lambda k, t: acc[0, k:k + t.shape[1]].add_(t.sum(0))) if acc.shape[0] == 1 else \
        (lambda k, t: acc[:, k:k + t.shape[1]].index_add_(0, b, t))
    p, v, w = B["p"][b], B["v"][b], B["w"][b]
    if volume:
        p0 = p * torch.tensor([1.0, 1.0, 0.0], dtype=torch.float64, device=DEV)
        for k in range(1, len(corners) - 1):
            x, y, z = corners[0] - p0, corners[k] - p0, corners[k + 1] - p0
            v6 = (x * torch.linalg.cross(y, z)).sum(1, keepdim=True)
            add(19, torch.cat([v6, (x + y + z) * 0.25 * v6], 1))
    vec = torch.zeros_like(corners[0])
    for k in range(1, len(corners) - 1):
        vec = vec + torch.linalg.cross(corners[k] - corners[0], corners[k + 1] - corners[0])
    len2 = (vec * vec).sum(1, keepdim=True)
    ok = len2 >= 1e-12
    ln = len2.sqrt()
    nrm = torch.where(ok, vec / ln, torch.zeros_like(vec))
    A = torch.where(ok, 0.5 * ln, torch.zeros_like(ln))
    fc = sum(corners) / len(corners)
    r = fc - p
    if volume:
        add(18, A)
        if wave.layers:
            F = -nrm * A * wave.depth(fc[:, 0], fc[:, 1], fc[:, 2])[:, None]
            add(0, torch.cat([F, torch.linalg.cross(r, F)], 1))
    vc = _fluid_velocity(ocean, fc) - (v + torch.linalg.cross(w, r))
    vn = (vc * nrm).sum(1, keepdim=True)
    vt = vc - vn * nrm
    q = torch.where(vn < -1e-12, vc * vc.norm(dim=1, keepdim=True) * -vn * A, torch.zeros_like(vc))
    f = torch.where((vt * vt).sum(1, keepdim=True) > 1e-9, vt * A, torch.zeros_like(vt))
    add(6, torch.cat([q, torch.linalg.cross(r, q), f, torch.linalg.cross(r, f)], 1))


def _wrenches(mesh_list, bodies: np.ndarray, ocean, wave: _Wave):
    """SolidEntity::ComputeHydrodynamicForces in 64 bits for records with
    zeroed in-out wrenches: (n, 20) values and the fluid position."""
    n = bodies.size
    mn, mx = _t64(bodies["aabb_min"].astype(np.float32)), _t64(bodies["aabb_max"].astype(np.float32))
    under = torch.zeros(n, dtype=torch.long, device=DEV)
    for k in range(8):
        c = [mx[:, a] if k >> a & 1 else mn[:, a] for a in range(3)]
        under += wave.depth(*c) > 0
    pos = torch.where(under == 0, 1, torch.where(under == 8, 0, 2)).cpu().numpy()
    acc = torch.zeros((n, 23), dtype=torch.float64, device=DEV)
    mesh = bodies["mesh"]
    order = np.argsort(mesh, kind="stable")
    cuts = np.flatnonzero(np.diff(mesh[order])) + 1
    for group in np.split(order, cuts):
        xyz, faces = mesh_list[int(mesh[group[0]])]
        V, Fi = _t64(xyz), torch.as_tensor(np.asarray(faces, dtype=np.int64).reshape(-1, 3), device=DEV)
        group = group[pos[group] != abi.OUTSIDE]
        step = max(1, 2_000_000 // Fi.shape[0])
        for at in range(0, len(group), step):
            g = group[at:at + step]
            R = _t64(bodies["T_C"]["basis"][g]).view(-1, 3, 3)
            X = torch.einsum("bij,vj->bvi", R, V) + _t64(bodies["T_C"]["origin"][g])[:, None]
            B = {"p": _t64(bodies["T_CG"]["origin"][g]), "v": _t64(bodies["v"][g]), "w": _t64(bodies["omega"][g])}
            a = torch.zeros((len(g), 23), dtype=torch.float64, device=DEV)
            inside = torch.as_tensor(pos[g] == abi.INSIDE, device=DEV)
            d = wave.depth(X[..., 0], X[..., 1], X[..., 2])
            wet = (d >= 0)[:, Fi].sum(-1)
            for volume in (False, True):
                sel = ~inside if volume else inside
                b, f = torch.nonzero(sel[:, None] & ((wet == 3) | ~torch.as_tensor(volume, device=DEV)), as_tuple=True)
                _polygons(a, b, [X[b, Fi[f, k]] for k in range(3)], B, ocean, wave, volume)
            for count in (1, 2):
                b, f = torch.nonzero(~inside[:, None] & (wet == count), as_tuple=True)
                if b.numel() == 0:
                    continue
                # turn each face so that its odd corner (the wet one of one, the dry one of two) comes first
                odd = ((d[b[:, None], Fi[f]] >= 0) == (count == 1)).to(torch.int8).argmax(1)
                i = [Fi[f, (odd + k) % 3] for k in range(3)]
                P, D = [X[b, k] for k in i], [d[b, k] for k in i]
                cut = [P[0] + (P[k] - P[0]) * (D[0].abs() / (D[0].abs() + D[k].abs()))[:, None] for k in (1, 2)]
                corners = [P[0], cut[0], cut[1]] if count == 1 else [cut[0], P[1], P[2], cut[1]]
                _polygons(a, b, corners, B, ocean, wave, True)
            acc[torch.as_tensor(g, device=DEV)] = a
    out = torch.zeros((n, 20), dtype=torch.float64, device=DEV)
    ins, cro = (torch.as_tensor(pos == k, device=DEV) for k in (abi.INSIDE, abi.CROSSING_SURFACE))
    rho, grav = ocean.density, ocean.gravity
    up = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=DEV)
    og, V6 = _t64(bodies["T_CG"]["origin"]), acc[:, 19:20]
    floats = cro & (V6[:, 0] > 1e-9)
    if wave.layers:
        fb, tb = acc[:, 0:3] * rho * grav, acc[:, 3:6] * rho * grav
    else:
        fb = -V6 / 6.0 * rho * grav * up
        cb = acc[:, 20:23] / V6 + og * torch.tensor([1.0, 1.0, 0.0], dtype=torch.float64, device=DEV)
        tb = torch.linalg.cross(cb - og, fb)
    fi = -_t64(bodies["volume"])[:, None] * rho * grav * up
    arm = torch.einsum("bij,bj->bi", _t64(bodies["T_CG"]["basis"]).view(-1, 3, 3), _t64(bodies["P_CB"]))
    out[floats, 0:3], out[floats, 3:6] = fb[floats], tb[floats]
    out[ins, 0:3], out[ins, 3:6] = fi[ins], torch.linalg.cross(arm, fi)[ins]
    Ro = _t64(bodies["R_O"]).view(-1, 3, 3)
    for k, (c, scale) in enumerate((("Cd", 0.5 * rho), ("Cd", 0.5 * rho), ("Cf", rho), ("Cf", rho))):
        x = acc[:, 6 + 3 * k:9 + 3 * k]
        loc = torch.linalg.solve(Ro, x[..., None])[..., 0]
        nn = loc.norm(dim=1, keepdim=True)
        loc = torch.where(nn > 2.3e-16, loc / nn, torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64, device=DEV))
        out[:, 6 + 3 * k:9 + 3 * k] = x * scale * (loc.abs() * _t64(bodies[c])).sum(1, keepdim=True)
    out[:, 18] = torch.where(ins, _t64(bodies["surface"]), acc[:, 18])
    out[floats, 19] = V6[floats, 0] / 6.0
    out[torch.as_tensor(pos == abi.OUTSIDE, device=DEV)] = 0.0
    return out, pos


def _cable_forces(sc) -> np.ndarray:
    """CableEntity::ComputeHydrodynamicForces on a flat sea, numpy FP64."""
    x, v, o = sc["x"], sc["v"], sc["ocean"]
    seg = np.zeros((x.shape[0], 9))
    out = np.zeros((x.shape[0], 9))
    dep = x[:, 2].astype(np.float32).astype(np.float64)
    U = np.array(o.currents[0].vel[:])

    def circ(h, r):
        hh = np.clip(np.where(h > r, 2 * r - h, h), 0.0, None)
        th = 2.0 * np.arccos(np.clip((r - hh) / r, -1, 1))
        small = r * r / 2.0 * (th - np.sin(th))
        a = np.where(h > r, np.pi * r * r - small, small)
        return np.where(h <= 0, 0.0, np.where(h >= 2 * r, np.pi * r * r, a))

    for cb in sc["cables"]:
        f, n, r = int(cb["first_node"]), int(cb["n_nodes"]), float(cb["radius"])
        a, b = np.arange(f, f + n - 1), np.arange(f + 1, f + n)
        swap = dep[a] > dep[b]
        lo, hi = np.where(swap, b, a), np.where(swap, a, b)
        d1, d2 = dep[lo], dep[hi]
        dz, s = d2 - d1, x[hi] - x[lo]
        dxy, L = np.hypot(s[:, 0], s[:, 1]), np.linalg.norm(s, axis=1)
        with np.errstate(all="ignore"):
            al = np.arctan(dz / dxy)
            ca, sa = np.cos(al), np.sin(al)
            m = r * ca
            full = np.pi * r * r * L
            eps = 2.220446049250313e-16
            V = np.select(
                [d2 < -m, d1 > m, dxy < eps, dz < eps, (np.abs(d1) <= m) & (np.abs(d2) <= m), (d1 < -m) & (d2 > m), d2 <= m],
                [0.0 * L, full, np.pi * r * r * np.minimum(d2, dz), circ(d1 + r, r) * L,
                 (circ(d1 / ca + r, r) + circ(d2 / ca + r, r)) / 2 * L, np.pi * r * r * ((d2 - m) / sa + m),
                 circ(r + d2 / ca, r) * (r + d2 / ca) / sa / 2],
                full - circ(r - d1 / ca, r) * (r - d1 / ca) / sa / 2)
        wet = ~(d2 < -m) & (V > 0)
        seg[a, 2] = np.where(~(d2 < -m), -V * o.density * o.gravity, 0.0)
        rv = (v[a] + v[b]) / 2 - U
        share = V / full
        q = -(1.0 - np.abs((s * rv).sum(1))) * share * 0.5 * o.density * 0.5 * 2 * r * L * np.linalg.norm(rv, axis=1)
        seg[a, 3:6] = np.where(wet, q, 0.0)[:, None] * rv
        seg[a, 6:9] = np.where(wet, -share * 2 * np.pi * r * L, 0.0)[:, None] * rv
        out[a] += seg[a] / 2
        out[b] += seg[a] / 2
        out[f] *= 2
        out[f + n - 1] *= 2
    return out


def _sea_depths(sc) -> np.ndarray:
    """The FFT ocean's two height layers at time t in 64 bits from its
    spectrum and butterfly tables, then the depths of the points."""
    p = sc["params"]
    N, passes = 1 << p.passes, int(p.passes)
    s12, s34 = (np.zeros((N, N, 4), dtype=np.float32) for _ in range(2))
    idx, wt = np.zeros((passes, N, 2), dtype=np.int32), np.zeros((passes, N, 2), dtype=np.float32)
    abi.load_library().hydro_debug_fft_ocean_tables(C.byref(p), s12.ctypes.data, s34.ctypes.data, idx.ctypes.data,
                                                    wt.ctypes.data)
    k = np.arange(N)
    sg = np.where((k + 0.5) / N > 0.5, k / N - 1.0, k / N)
    X, Y = sg[None, :], sg[:, None]
    neg = (N - k) % N
    h = []
    for g in (0, 1):
        z = (s12[..., 2 * g] + 1j * s12[..., 2 * g + 1]).astype(np.complex128) * 1.414213562
        zc = z[neg][:, neg]
        inv = 2.0 * np.pi * N / p.grid_sizes[g]
        K = np.hypot(X * inv, Y * inv)
        w = np.sqrt(9.81 * K * (1.0 + K * K / (370.0 * 370.0))) * sc["t"]
        h.append(((z.real + zc.real) * np.cos(w) - (z.imag + zc.imag) * np.sin(w)) +
                 1j * ((z.real - zc.real) * np.sin(w) + (z.imag - zc.imag) * np.cos(w)))
    a = h[0] + 1j * h[1]
    tw = (wt[..., 0] + 1j * wt[..., 1]).astype(np.complex128)
    for axis in (1, 0):
        a = np.moveaxis(a, axis, 1)
        for q in range(passes):
            a = a[:, idx[q, :, 0]] + tw[q][None, :] * a[:, idx[q, :, 1]]
        a = np.moveaxis(a, 1, axis)
    wave = _Wave([(_t64(a.real), p.grid_sizes[0]), (_t64(a.imag), p.grid_sizes[1])])
    x, y, z = _t64(sc["points"]).T
    return wave.depth(x, y, z).cpu().numpy()


def _mlp(net, F):
    """The network in 64 bits on its FP32 weights: body-frame wrenches."""
    x = (F.double() - net.f_mean.double()) * net.f_istd.double()
    for l in range(4):
        L = net.layers[l]
        k = S.N_FEAT if l == 0 else L["k"]
        x = x @ L["w"][:k].double() + L["b"].double()
        if l < 3:
            x = torch.nn.functional.silu(x)
    return x[:, :S.N_OUT] / net.t_istd.double() + net.t_mean.double()


def _features(bodies: np.ndarray, ocean, wave: _Wave):
    R, p = _t64(bodies["T_CG"]["basis"]).view(-1, 3, 3), _t64(bodies["T_CG"]["origin"])
    ux, uy = R[:, 0, 0], R[:, 1, 0]
    hn = torch.hypot(ux, uy)
    ux, uy = torch.where(hn > 1e-6, ux / hn, torch.ones_like(hn)), torch.where(hn > 1e-6, uy / hn, torch.zeros_like(hn))
    x, y = p[:, 0], p[:, 1]
    h = wave.elevation(x, y)
    ef, eb = wave.elevation(x + ux, y + uy), wave.elevation(x - ux, y - uy)
    el, er = wave.elevation(x - uy, y + ux), wave.elevation(x + uy, y - ux)
    loc = lambda u: torch.einsum("bji,bj->bi", R, u)  # noqa: E731
    U = _t64(ocean.currents[0].vel[:]).expand_as(p)
    cols = [p[:, 2] + h, torch.atan2(R[:, 2, 1], R[:, 2, 2]), torch.asin(-R[:, 2, 0].clamp(-1, 1))]
    return torch.cat([torch.stack(cols, 1), loc(_t64(bodies["v"])), loc(_t64(bodies["omega"])), loc(U),
                      torch.stack([h, (ef - eb) / 2, (el - er) / 2, ef + eb - 2 * h], 1)], 1)


def _predict(d: dict, bodies: np.ndarray, faces: int, tau: float, inside: bool, audit: int):
    """GatedPredictor.predict's first call in 64 bits."""
    wave = _grid_wave(d["waves"])
    a, b = d["nets"]
    F = _features(bodies, d["ocean"], wave)
    za, zb = _mlp(a, F), _mlp(b, F)
    g, fs_ts = a.gate, S.hull_scales(d["ocean"])
    e = F - g["mean"].double()
    ok = ((F >= g["lo"].double()) & (F <= g["hi"].double())).all(1) & (((e @ g["P"].double()) * e).sum(1) <= g["thr"])
    if inside:
        mn, mx = (_t64(bodies[k].astype(np.float32)) for k in ("aabb_min", "aabb_max"))
        deep = torch.ones_like(ok)
        for k in range(8):
            deep &= wave.depth(*[mx[:, c] if k >> c & 1 else mn[:, c] for c in range(3)]) > 0
        ok &= ~deep
    dis = torch.maximum((za - zb)[:, :3].norm(dim=1) / fs_ts[0], (za - zb)[:, 3:].norm(dim=1) / fs_ts[1])
    ok &= dis <= tau
    if audit:
        ok[::audit] = False
    out = 0.5 * (za + zb)
    rows = torch.nonzero(~ok)[:, 0].cpu().numpy()
    if rows.size:
        sub = bodies[rows].copy()
        sub["mesh"] = 0
        w, _ = _wrenches([S.hull_mesh(faces)], sub, d["ocean"], wave)
        out[torch.as_tensor(rows, device=DEV)] = _body_frame(sub, w)
    return out


def _body_frame(bodies, w):
    R = _t64(bodies["T_CG"]["basis"]).view(-1, 3, 3)
    F, T = w[:, 0:3] + w[:, 6:9] + w[:, 12:15], w[:, 3:6] + w[:, 9:12] + w[:, 15:18]
    return torch.cat([torch.einsum("bji,bj->bi", R, F), torch.einsum("bji,bj->bi", R, T)], 1)


def _rotation(q):
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)


def _roll(d: dict, case: dict, start: np.ndarray):
    """The rollout in 64 bits: wrench, implicit gyroscopic step, semi-implicit Euler."""
    s = _t64(start.view(np.float64).reshape(-1, 27).copy())
    dt, n = 0.01, case["n"]
    # a record: p 0..2, q 3..6, v 7..9, w 10..12, thrust force 13..15, thrust torque 16..18, mass, inertial mass, inertia
    mass, im, I, half = s[:, 19:20], s[:, 20:21], s[:, 21:24], start["half_extents"]
    rec = RO.static_bodies(n, 0)
    for _ in range(case["steps"]):
        R = _rotation(s[:, 3:7])
        Rn, p = R.cpu().numpy(), s[:, 0:3].cpu().numpy()
        rec["T_CG"]["basis"] = rec["T_C"]["basis"] = rec["R_O"] = Rn.reshape(n, 9)
        rec["T_CG"]["origin"] = rec["T_C"]["origin"] = p
        rec["v"], rec["omega"] = s[:, 7:10].cpu().numpy(), s[:, 10:13].cpu().numpy()
        rec["aabb_min"], rec["aabb_max"] = scenarios.compound_aabb(Rn, p, half)
        if case["mode"] == "exact":
            bw = _body_frame(rec, _wrenches([S.hull_mesh(8000)], rec, d["ocean"], _grid_wave(d["waves"]))[0])
        else:
            bw = _predict(d, rec, 8000, math.inf, False, 0)
        F = torch.einsum("bij,bj->bi", R, bw[:, :3] + s[:, 13:16])
        F[:, 2:3] += mass * d["ocean"].gravity
        tb = bw[:, 3:] + s[:, 16:19]
        wb = torch.einsum("bji,bj->bi", R, s[:, 10:13])
        skew = lambda a: torch.stack([0 * a[:, 0], -a[:, 2], a[:, 1], a[:, 2], 0 * a[:, 0], -a[:, 0],  # noqa: E731
                                      -a[:, 1], a[:, 0], 0 * a[:, 0]], 1).view(-1, 3, 3)
        J = torch.diag_embed(I) + dt * (skew(wb) @ torch.diag_embed(I) - skew(I * wb))
        wb = wb + dt * tb / I - torch.linalg.solve(J, dt * torch.linalg.cross(wb, I * wb))
        w = torch.einsum("bij,bj->bi", R, wb)
        v = s[:, 7:10] + dt * F / im
        wn = w.norm(dim=1, keepdim=True)
        sc = torch.where(wn > 1e-12, torch.sin(0.5 * wn * dt) / wn, torch.full_like(wn, 0.5 * dt))
        a, b = torch.cat([torch.cos(0.5 * wn * dt), sc * w], 1), s[:, 3:7]
        q = torch.cat([a[:, :1] * b[:, :1] - (a[:, 1:] * b[:, 1:]).sum(1, keepdim=True),
                       a[:, :1] * b[:, 1:] + b[:, :1] * a[:, 1:] + torch.linalg.cross(a[:, 1:], b[:, 1:])], 1)
        s[:, 0:3] += dt * v
        s[:, 3:7], s[:, 7:10], s[:, 10:13] = q / q.norm(dim=1, keepdim=True), v, w
    return s


def _train(case: dict, seed: int, net, F, T):
    """One epoch of AdamW with warm-up and cosine decay in 64 bits."""
    B, lr, end = case["batch"], 3e-3, 2e-5
    X = (F.double() - net.f_mean.double()) * net.f_istd.double()
    Y = (T.double() - net.t_mean.double()) * net.t_istd.double()
    Ls = net.layers
    W = [L["w"].double().clone() for L in Ls]
    b = [L["b"].double().clone() for L in Ls]
    X = torch.nn.functional.pad(X, (0, Ls[0]["k"] - S.N_FEAT))
    mom = [[torch.zeros_like(t) for t in W + b] for _ in range(2)]
    total, loss = F.shape[0] // B, 0.0
    for i in range(total):
        x, y = X[i * B:(i + 1) * B], Y[i * B:(i + 1) * B]
        xs, zs = [x], []
        for l in range(4):
            zs.append(xs[l] @ W[l] + b[l])
            xs.append(torch.nn.functional.silu(zs[l]))
        e = zs[3][:, :S.N_OUT] - y
        loss = loss + (e * e).mean()
        g = torch.nn.functional.pad(2.0 * e / e.numel(), (0, Ls[3]["n"] - S.N_OUT))
        gw, gb = [None] * 4, [None] * 4
        for l in range(3, -1, -1):
            gw[l], gb[l] = xs[l].T @ g, g.sum(0)
            if l:
                sg = torch.sigmoid(zs[l - 1])
                g = (g @ W[l].T) * (sg + zs[l - 1] * sg * (1 - sg))
        cur = (end + 0.5 * (lr - end) * (1 + math.cos(math.pi * i / max(total - 1, 1)))) * min(1.0, (i + 1) / 200)
        for k, (t, gr) in enumerate(zip(W + b, gw + gb)):
            m, v = mom[0][k], mom[1][k]
            m.mul_(0.9).add_(0.1 * gr)
            v.mul_(0.999).add_(0.001 * gr * gr)
            t.mul_(1.0 - cur * (1e-5 if k < 4 else 0.0))
            t.sub_(cur * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8))
    return {"loss": float(loss) / total, "w": W, "b": b, "gw": gw, "gb": gb}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("body", "batch", "host"):
        sc = _scene(case, seed)
        w, pos = _wrenches(sc["meshes"], sc["bodies"], sc["ocean"], _grid_wave(sc["waves"]))
        w = w.cpu().numpy()
        return {"wrench": w, "flags": np.stack([pos, np.zeros_like(pos)], 1).astype(np.int32)}
    if kind == "cables":
        return _cable_forces(_cable_scene(case, seed))
    if kind == "sea":
        return _sea_depths(_sea_scene(case, seed))
    s = prepare(case, seed)
    if kind == "mlp":
        return torch.nn.functional.pad(_mlp(s["net"], s["F"]), (0, 10))
    if kind == "predict":
        b = S.sample_states(np.random.default_rng(202 + seed), case["n"])
        return _predict(s["d"], b, S.HULL_FACES, s["gp"].tau, True, 1024)
    if kind == "train":
        return _train(case, seed, s["net"], s["F"], s["T"])
    return _roll(s["d"], case, _rollout_start(s["d"], case, seed))
