"""Performance cases of the backend: what a user has it compute, through its public entry points.

Kinds of case, and the calls that they time:

* ``dropin``   ``backend.trace_energy_field``: one trace inside a running Acoustic Agent, host result dict out.  The
               smallest calls, where launches and host latency count, in float32 and in the float64 parity mode.
* ``render``   ``batching.RIRRenderer``: every channel of one scene, trace plus band synthesis, resident.
* ``mixed``    the same renderer over scenes of very different sizes, replayed as a CUDA graph (dataset generation).
* ``service``  ``runtime.TraceService``: a burst of jobs handed to the continuously fed launch and awaited (serving).
* ``synth``    ``runtime.synthesize_batch``: echograms to six band impulse responses.
* ``late``     ``late_reverb.LateReverbRenderer``: FDN late tails crossfaded into traced band signals.
* ``direct``   ``direct.direct_results``: direct sound (occlusion, transmission) of source/listener pairs.
* ``bvh``      ``bvh.DeviceBvhBuilder``: the scene BVH of a large model.

Geometry and sizes belong to the case; materials, random streams and signals come from the seed.
"""
from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch

from acoustic_agent_b200 import backend, batching, bvh, direct, late_reverb, runtime, scene, workloads

BANDS = 6
AIR = (0.0, 0.00011513, 0.00034539, 0.00057565, 0.0011513, 0.0034539)   # Np/m per band
CROSSOVERS = (176.78, 353.55, 707.11, 1414.2, 2828.4)
C = 343.0


def listed():
    return [
        # one room response of a quick interactive preview: the shoebox of the reference's first configuration
        {"name": "dropin_shoebox_f32", "kind": "dropin", "room": "shoebox", "geometry": 1729, "rays": 10000,
         "bounces": 50, "precision": "float32", "ambisonics": True, "visual": True},
        # the same call in the float64 parity mode, on the furnished U room
        {"name": "dropin_u_room_f64", "kind": "dropin", "room": "u_room", "geometry": 1729, "rays": 20000,
         "bounces": 100, "precision": "float64", "ambisonics": False, "visual": False},
        # one 8-microphone array response at full quality
        {"name": "render_u_room_8ch", "kind": "render", "room": "u_room", "geometry": 1729, "rays": 200000,
         "bounces": 100, "channels": 8, "fs": 48000, "duration": 2.0, "bin": 0.001},
        # one response across an 8-room apartment, the largest ray budget of the configurations
        {"name": "render_apartment", "kind": "render", "room": "apartment", "geometry": 1729, "rays": 1000000,
         "bounces": 200, "channels": 1, "fs": 48000, "duration": 2.0, "bin": 0.001},
        # a slice of a training-set batch: scenes from one room to eight, uneven ray budgets
        {"name": "mixed_8_scenes", "kind": "mixed", "geometry": 1729, "scenes": 8, "ray_bounces": 2000000000},
        # a server's burst: jobs of uneven size handed to the running launch
        {"name": "service_burst", "kind": "service", "geometry": 5, "scenes": 6, "ray_bounces": 500000000},
        # the band synthesis of a single short response
        {"name": "synth_one_16k", "kind": "synth", "rirs": 1, "fs": 16000, "seconds": 1.0, "bin": 0.01,
         "noise": "philox"},
        # the band synthesis of a whole batch, ragged lengths, two sample rates
        {"name": "synth_192_ragged", "kind": "synth", "rirs": 192, "fs": 0, "seconds": 1.37, "bin": 0.01,
         "noise": "philox"},
        # late tails of one array response
        {"name": "late_8_48k", "kind": "late", "tails": 8, "fs": 48000, "seconds": 2.0},
        # late tails of a batch
        {"name": "late_256_16k", "kind": "late", "tails": 256, "fs": 16000, "seconds": 1.37},
        # direct sound of a batch of pairs in one scene
        {"name": "direct_1024", "kind": "direct", "room": "u_room", "geometry": 1729, "pairs": 1024,
         "volumetric": True, "samples": 32, "layers": 8},
        # the BVH of a warehouse-sized model
        {"name": "bvh_1m", "kind": "bvh", "surfaces": 1 << 20, "leaf": 4, "layout": "warehouse"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("dropin", "dropin", "render", "render", "mixed", "service", "synth", "synth", "late", "late",
                       "direct", "bvh"))
    geometry = rng.randrange(1, 1 << 20)
    if kind == "dropin":
        precision = rng.choice(("float32", "float32", "float64"))
        top = 200000 if precision == "float32" else 20000
        return {"kind": kind, "room": rng.choice(("shoebox", "u_room", "apartment")), "geometry": geometry,
                "rays": log_int(500, top), "bounces": rng.randint(12, 100), "precision": precision,
                "ambisonics": rng.random() < 0.5, "visual": rng.random() < 0.5}
    if kind == "render":
        channels = rng.randint(1, 8)
        bounces = rng.randint(20, 200)
        fs, step = rng.choice(((16000, 0.01), (48000, 0.001)))
        return {"kind": kind, "room": rng.choice(("shoebox", "u_room", "apartment")), "geometry": geometry,
                "rays": log_int(5000, 160000000 // (channels * bounces)), "bounces": bounces, "channels": channels,
                "fs": fs, "duration": round(rng.uniform(0.5, 2.0), 2), "bin": step}
    if kind in ("mixed", "service"):
        return {"kind": kind, "geometry": geometry, "scenes": rng.randint(2, 8),
                "ray_bounces": log_int(50000000, 2000000000 if kind == "mixed" else 500000000)}
    if kind == "synth":
        return {"kind": kind, "rirs": log_int(1, 192), "fs": rng.choice((0, 16000, 16000, 44100, 48000)),
                "seconds": round(rng.uniform(0.2, 1.37), 3), "bin": rng.choice((0.001, 0.01)),
                "noise": rng.choice(("philox", "white"))}
    if kind == "late":
        fs = rng.choice((8000, 16000, 44100, 48000))
        return {"kind": kind, "tails": log_int(1, 256 if fs <= 16000 else 32), "fs": fs,
                "seconds": round(rng.uniform(0.5, 1.37), 3)}
    if kind == "direct":
        return {"kind": kind, "room": rng.choice(("shoebox", "u_room", "apartment")), "geometry": geometry,
                "pairs": log_int(1, 1024), "volumetric": rng.random() < 0.7, "samples": rng.choice((16, 32, 45)),
                "layers": rng.randint(1, 8)}
    return {"kind": kind, "surfaces": log_int(50, 1 << 20), "leaf": rng.choice((1, 2, 4, 8)),
            "layout": rng.choice(("warehouse", "random"))}


# ---- inputs ------------------------------------------------------------------

def _room(case, seed):
    """The case's geometry as a workload, with the seed's materials and random stream."""
    rays, bounces = case.get("rays", 10000), case.get("bounces", 50)
    if case["room"] == "shoebox":
        w = workloads.shoebox(1729, rays=rays, bounces=bounces)
    elif case["room"] == "u_room":
        w = workloads.u_furnished(case["geometry"], rays=rays, bounces=bounces, channels=case.get("channels", 1))
    else:
        w = workloads.apartment(case["geometry"], rays=rays, bounces=bounces)
    spec = workloads.with_surface_materials(w.spec, seed, scattering=(0.05, 0.5))
    duration = case.get("duration", 1.0)
    config = replace(w.config, seed=int(seed), fs=case.get("fs", 16000), duration_s=duration, rt_duration_s=duration,
                     rt_bin_duration_s=case.get("bin", 0.01))
    channels = case.get("channels", 1)
    listeners = w.listeners if len(w.listeners) == channels else workloads.circular_array(w.listeners[0], 8)[:channels]
    return replace(w, spec=spec, config=config, listeners=listeners)


def _population(case, seed):
    """Scenes of very different sizes whose ray budgets add up to the case's ray-bounces."""
    pool = workloads.mixed_batch(case["geometry"], case["scenes"])
    nominal = sum(w.num_traces * w.config.rt_num_rays * w.config.rt_num_bounces for w in pool)
    out = []
    for k, w in enumerate(pool):
        rays = max(64, int(w.config.rt_num_rays * case["ray_bounces"] / nominal))
        spec = workloads.with_surface_materials(w.spec, seed + k, scattering=(0.05, 0.5))
        out.append(replace(w, spec=spec, config=replace(w.config, rt_num_rays=rays, seed=int(seed) + k)))
    return out


def _direct_config(case):
    class Config:
        direct_occlusion = True
        direct_occlusion_mode = "volumetric" if case["volumetric"] else "raycast"
        direct_occlusion_radius_m = 0.1
        direct_occlusion_samples = case["samples"]
        direct_transmission = True
        num_transmission_rays = case["layers"]
        min_distance_m = 1.0
        c = C
        rt_cuda_device = 0
    return Config


def _synth_shapes(case):
    """(rate, bins, samples per bin) of each response: the listed length and down to half of it."""
    out = []
    for k in range(case["rirs"]):
        fs = case["fs"] or (48000 if k % 4 == 3 else 16000)
        seconds = case["seconds"] * (1.0 - 0.5 * ((k * 0.6180339887) % 1.0 if k else 0.0))
        out.append((fs, max(1, int(math.ceil(seconds / case["bin"]))), max(1, int(math.ceil(case["bin"] * fs)))))
    return out


def _synth_inputs(case, seed):
    """Decaying echograms over some five decades, empty before the direct delay and below the audible floor."""
    rng = np.random.default_rng(seed)
    echo, delays, seeds, white = [], [], [], []
    for fs, bins, spb in _synth_shapes(case):
        rt60 = rng.uniform(0.2, 1.2, (BANDS, 1))
        t = (np.arange(bins) + 0.5)[None] * (spb / fs)
        e = 1e-2 * np.exp(-13.8 * t / rt60) * rng.exponential(1.0, (BANDS, bins))
        delay = float(rng.uniform(0.002, 0.03))
        e[:, : int(delay * fs / spb)] = 0.0
        echo.append(e.astype(np.float32))
        delays.append(delay)
        seeds.append(int(rng.integers(1, 1 << 31)))
        white.append(rng.uniform(-1.0, 1.0, bins * spb) if case["noise"] == "white" else None)
    return echo, delays, seeds, white


def _bvh_bounds(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = case["surfaces"]
    u = torch.rand((n, 8), dtype=torch.float64, device="cuda", generator=g)
    if case["layout"] == "random":
        lo = u[:, :3] * torch.tensor([50.0, 50.0, 6.0], dtype=torch.float64, device="cuda")
        return lo, lo + 2.0 * u[:, 3:6]
    # rotated boxes on a warehouse floor and, one in eight, wall pieces on a 2 m grid (many equal centroids)
    half = 0.15 + 0.85 * u[:, 2:4]
    angle = u[:, 4] * (math.pi / 2)
    c, s = angle.cos(), angle.sin()
    ext = torch.stack([half[:, 0] * c + half[:, 1] * s, half[:, 0] * s + half[:, 1] * c], 1)
    centre = 400.0 * u[:, :2]
    lo = torch.cat([centre - ext, torch.zeros_like(ext[:, :1])], 1)
    hi = torch.cat([centre + ext, 0.4 + 2.6 * u[:, 5:6]], 1)
    wall = u[:, 6] < 0.125
    a = torch.floor(200.0 * u[:, :2]) * 2.0
    along = (u[:, 7:8] < 0.5).double() * torch.tensor([[2.0, -2.0]], dtype=torch.float64, device="cuda")
    b = a + torch.where(along >= 0, along, torch.zeros_like(along)) + torch.where(
        u[:, 7:8] < 0.5, torch.zeros_like(a), torch.tensor([[0.0, 2.0]], dtype=torch.float64, device="cuda"))
    lo_w = torch.cat([torch.minimum(a, b), torch.zeros_like(a[:, :1])], 1)
    hi_w = torch.cat([torch.maximum(a, b), torch.full_like(a[:, :1], 3.0)], 1)
    lo = torch.where(wall[:, None], lo_w, lo) - 2e-6
    hi = torch.where(wall[:, None], hi_w, hi) + 2e-6
    return lo.contiguous(), hi.contiguous()


_SERVICE = {}   # a serving process keeps one trace service


def prepare(case, seed):
    kind = case["kind"]
    device = torch.device("cuda", 0)
    state = {"kind": kind, "case": case}
    if kind == "dropin":
        w = _room(case, seed)
        state["scene"] = scene.compile_scene(w.spec)
        state["source"], state["listener"] = np.asarray(w.sources[0]), np.asarray(w.listeners[0])
        state["config"] = replace(w.config, rt_precision=case["precision"], collect_visual_paths=case["visual"])
        state["model"] = w.source_model
    elif kind in ("render", "mixed", "service"):
        ws = [_room(case, seed)] if kind == "render" else _population(case, seed)
        specs, jobs = batching.workload_jobs(ws)
        renderer = batching.RIRRenderer(0)
        plan = renderer.plan([scene.compile_scene(s) for s in specs], jobs)
        state["renderer"], state["plan"] = renderer, plan
        if kind == "mixed":
            renderer.capture(plan)
        if kind == "service":
            if not _SERVICE:
                _SERVICE["service"] = runtime.TraceService(0, idle_timeout_s=0.002)
            state["jobs"] = [(plan.scenes[j.scene_index], j.spec, b) for j, b in zip(plan.jobs, plan.buffers)]
    elif kind == "synth":
        echo, delays, seeds, white = _synth_inputs(case, seed)
        shapes = _synth_shapes(case)
        state["store"] = torch.empty(sum(BANDS * b * s for _, b, s in shapes), dtype=torch.float32, device=device)
        jobs, off = [], 0
        for k, (fs, bins, spb) in enumerate(shapes):
            n = BANDS * bins * spb
            out = state["store"][off:off + n].view(BANDS, bins * spb)
            off += n
            w = torch.as_tensor(white[k], device=device) if white[k] is not None else None
            jobs.append(runtime.SynthJob(torch.as_tensor(echo[k], device=device), out, fs, case["bin"], seeds[k],
                                         delays[k], C, "reference" if w is not None else "philox", w))
        state["jobs"], state["workspace"] = jobs, runtime.SynthBatchWorkspace(device)
    elif kind == "late":
        rng = np.random.default_rng(seed)
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        J, fs = case["tails"], case["fs"]
        n = int(round(case["seconds"] * fs))
        rt60 = rng.uniform(0.3, 1.4, (J, BANDS))
        t = torch.arange(n, dtype=torch.float64, device=device) / fs
        traced = torch.randn((J, BANDS, n), dtype=torch.float64, device=device, generator=g)
        traced *= 1e-2 * torch.exp(-6.9 * t / torch.as_tensor(rt60, device=device)[:, :, None])
        state["out"] = torch.empty((J, BANDS, n), dtype=torch.float32, device=device)
        state["component"] = torch.empty_like(state["out"])
        state["renderer"] = late_reverb.LateReverbRenderer(0)
        transition = 0.6 * case["seconds"]
        state["jobs"] = [late_reverb.LateReverbJob(traced[k], state["out"][k], state["component"][k], fs,
                                                   int(seed) + k // 8, rt60[k].tolist(), 0.001, transition, 0.25)
                         for k in range(J)]
    elif kind == "direct":
        w = _room(case, seed)
        rng = np.random.default_rng(seed)
        arrays = scene.compile_scene(w.spec)
        state["scene"] = runtime.DeviceScene(arrays)
        state["tables"] = direct.DirectTables(arrays.names, rng.uniform(0.0, 0.3, (arrays.num_surfaces, BANDS)), device)
        corners = np.asarray(w.spec["corners"], dtype=float)
        lo = np.r_[corners.min(axis=0), 0.3]
        hi = np.r_[corners.max(axis=0), float(w.spec["height"]) - 0.3]
        state["pairs"] = list(rng.uniform(lo, hi, (case["pairs"], 2, 3)))
        state["config"] = _direct_config(case)
        state["row"] = {name: k for k, name in enumerate(arrays.names)}
    else:
        state["bounds"] = _bvh_bounds(case, seed)
        state["builder"] = bvh.DeviceBvhBuilder(0)
    return state


def _counts(named, names):
    return np.asarray([named.get(n, 0) for n in names])


def run(state):
    kind = state["kind"]
    if kind == "dropin":
        field = backend.trace_energy_field(state["scene"], state["source"], state["listener"], state["config"],
                                           state["model"], render_ambisonics=state["case"]["ambisonics"])
        names = state["scene"].names
        visual = field["visual_candidates"]
        return {"echogram": field["echogram"], "ambisonic": field["ambisonic_echogram"],
                "rays": [field["active_ray_count"], field["actual_bounces"], field["last_energy_time_s"]],
                "hits": _counts(field["surface_hit_count"], names),
                "contributions": _counts(field["surface_contribution_count"], names),
                "energy": _counts(field["surface_energy"], names),
                "visual": None if visual is None else {k: visual[k] for k in (
                    "hit_points", "surface_indices", "ray_indices", "orders", "distances", "gains")}}
    if kind in ("render", "mixed"):
        plan = state["plan"]
        state["renderer"].launch(plan)
        out = {"echograms": plan.echo_store, "irs": plan.ir_store}
        for k, b in enumerate(plan.buffers[:8]):
            out["rir%d" % k] = [b.hit_counts, b.contrib_counts, b.surface_energy, b.counters[:4]]
        return out
    if kind == "service":
        service = _SERVICE["service"]
        waiting = set(service.submit(state["jobs"]))
        while waiting:
            waiting.difference_update(service.poll())
        out = {"echograms": state["plan"].echo_store}
        for k, b in enumerate(state["plan"].buffers[:8]):
            out["rir%d" % k] = [b.hit_counts, b.contrib_counts, b.surface_energy, b.counters[:4]]
        return out
    if kind == "synth":
        runtime.synthesize_batch(state["jobs"], state["workspace"])
        return {"irs": state["store"]}
    if kind == "late":
        stats, _, _ = state["renderer"].render(state["jobs"])
        return {"out": state["out"], "component": state["component"], "stats": stats}
    if kind == "direct":
        res = direct.direct_results(state["scene"], state["tables"], state["pairs"], state["config"], "cardioid")
        return {"gains": np.asarray([list(r["band_gains"].values()) for r in res]),
                "transmission": np.stack([r["transmission"] for r in res]),
                "scalars": np.asarray([[r["distance_m"], r["delay_s"], r["distance_attenuation"], r["occlusion"],
                                        r["source_directivity_gain"]] for r in res]),
                "air": np.stack([r["air_absorption"] for r in res]),
                "surface": np.asarray([state["row"].get(r["occlusion_surface"], -1) for r in res])}
    tree = state["builder"].build(*state["bounds"], leaf_size=state["case"]["leaf"])
    return [tree.bounds_min, tree.bounds_max, tree.start, tree.count, tree.escape, tree.primitives,
            tree.node_count, tree.leaf_count, tree.max_depth]


# ---- what a pass cannot do without ---------------------------------------------

def _bounces(w, surfaces):
    """Ray-bounces of a workload and float operations of its queries, from the mean free path of its hull: two
    queries per bounce, each through about log2(surfaces) levels of box tests (two boxes of 18 operations) and one
    surface test (30), and about 150 operations of shading."""
    corners = np.asarray(w.spec["corners"], dtype=float)
    x, y = corners[:, 0], corners[:, 1]
    area = 0.5 * abs(float(np.dot(x, np.roll(y, -1)) - np.dot(y, np.roll(x, -1))))
    edge = float(np.sum(np.hypot(*(corners - np.roll(corners, -1, axis=0)).T)))
    h = float(w.spec["height"])
    free = 4.0 * area * h / (2.0 * area + edge * h)
    per_ray = min(float(w.config.rt_num_bounces), w.config.max_path_length / free)
    total = w.num_traces * w.config.rt_num_rays * per_ray
    return total, total * (2.0 * (36.0 * math.log2(max(2, surfaces)) + 30.0) + 150.0)


def work(case):
    kind = case["kind"]
    if kind in ("dropin", "render"):
        w = _room(case, 1)
        surfaces = workloads.count_surfaces(w.spec)
        _, flops = _bounces(w, surfaces)
        cells = BANDS * w.config.num_bins * 4
        if kind == "dropin":
            return {"bytes": cells * (5 if case["ambisonics"] else 1) + 100 * surfaces, "flops": flops}
        n = w.config.num_bins * max(1, math.ceil(case["bin"] * case["fs"]))
        rirs = w.num_traces
        return {"bytes": rirs * (2 * cells + BANDS * n * 4) + 100 * surfaces, "flops": flops + rirs * n * 450.0}
    if kind in ("mixed", "service"):
        size = flops = 0.0
        for w in _population(case, 1):
            surfaces = workloads.count_surfaces(w.spec)
            n = w.config.num_bins * max(1, math.ceil(w.config.rt_bin_duration_s * w.config.fs))
            size += 100 * surfaces + w.num_traces * BANDS * 4 * (2 * w.config.num_bins + (n if kind == "mixed" else 0))
            flops += _bounces(w, surfaces)[1] + (w.num_traces * n * 450.0 if kind == "mixed" else 0.0)
        return {"bytes": size, "flops": flops}
    if kind == "synth":
        # ten low-pass chains of four sections (9 operations each) and six envelopes per sample
        shapes = _synth_shapes(case)
        n = sum(b * s for _, b, s in shapes)
        return {"bytes": BANDS * 4 * (n + sum(b for _, b, _ in shapes)) + (8 * n if case["noise"] == "white" else 0),
                "flops": n * (40 * 9 + 60.0)}
    if kind == "late":
        # 96 absorptive and six tone sections and the mix per sample; the band split of the result; the crossfade
        n = case["tails"] * int(round(case["seconds"] * case["fs"]))
        return {"bytes": n * BANDS * (8 + 4 + 4), "flops": n * (1047.0 + 360.0 + 60.0)}
    if kind == "direct":
        surfaces = workloads.count_surfaces(_room(case, 1).spec)
        legs = (2 * case["samples"] if case["volumetric"] else 0) + 1
        return {"bytes": case["pairs"] * (48 + 140) + 100 * surfaces, "flops": case["pairs"] * legs * surfaces * 30.0}
    # bounds read once; the tree (about surfaces / leaf * 2 nodes of 72 bytes) and the leaf order written once
    n = case["surfaces"]
    leaves = 1
    while n > leaves * case["leaf"]:
        leaves *= 2
    return {"bytes": 48 * n + 8 * n + 72 * (2 * leaves - 1), "flops": 3.0 * n * math.log2(max(2, leaves))}


# ---- the same outputs in 64 bits -----------------------------------------------

def _philox_noise(seed, count):
    """Uniform noise in [-1, 1) of the counter-based stream: Philox4x32-10 (Salmon et al., SC'11), two 53-bit values
    per counter, key = the 64-bit seed, counter = (pair, 1 << 24, 0, 0)."""
    pairs = (count + 1) // 2
    mask = np.uint64(0xFFFFFFFF)
    c = [np.arange(pairs, dtype=np.uint64), np.full(pairs, 1 << 24, np.uint64), np.zeros(pairs, np.uint64),
         np.zeros(pairs, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = np.empty(2 * pairs)
    for j in range(2):
        bits = ((c[2 * j] >> np.uint64(5)) << np.uint64(26)) | (c[2 * j + 1] >> np.uint64(6))
        u[j::2] = bits.astype(np.float64) / 9007199254740992.0
    return -1.0 + 2.0 * u[:count]


def _lowpass(x, fs):
    """Five eight-pole Butterworth low-passes (four sections each) of every row of x [signals, 6, N]; only the
    chains that the bands need: returns [signals, 10, N] (upper of bands 0-4, then lower of bands 1-4 and of 5)."""
    rows, coef = [], []
    for band, cut in [(b, b) for b in range(5)] + [(b, b - 1) for b in range(1, 6)]:
        rows.append(band)
        sections = []
        for s in range(4):
            q = 1.0 / (2.0 * math.cos((2.0 * s + 1.0) * math.pi / 16.0))
            w0 = 2.0 * math.pi * CROSSOVERS[cut] / fs
            alpha = math.sin(w0) / (2.0 * q)
            a0 = 1.0 + alpha
            b1 = (1.0 - math.cos(w0)) / a0
            sections.append((b1 / 2.0, b1, b1 / 2.0, -2.0 * math.cos(w0) / a0, (1.0 - alpha) / a0))
        coef.append(sections)
    coef = np.asarray(coef)                       # [10, 4, 5]
    y = np.ascontiguousarray(np.moveaxis(x[:, rows, :], 2, 0))   # [N, signals, 10]
    for s in range(4):
        b0, b1, b2, a1, a2 = (np.broadcast_to(coef[:, s, k], y.shape[1:]).copy() for k in range(5))
        forced = b0 * y
        forced[1:] += b1 * y[:-1]
        forced[2:] += b2 * y[:-2]
        y1 = y2 = np.zeros(y.shape[1:])
        for n in range(y.shape[0]):
            y0 = forced[n] - a1 * y1 - a2 * y2
            forced[n] = y0
            y1, y2 = y0, y1
        y = forced
    return np.moveaxis(y, 0, 2)


def _exact_synth(case, seed):
    shapes = _synth_shapes(case)
    if sum(b * s for _, b, s in shapes) > 600000:
        return None
    echo, delays, seeds, white = _synth_inputs(case, seed)
    out = []
    for k, (fs, bins, spb) in enumerate(shapes):
        n = bins * spb
        noise = white[k] if white[k] is not None else _philox_noise(seeds[k], n)
        e = echo[k].astype(np.float64)
        amp = np.where(echo[k] < np.float32(1e-9), 0.0, np.sqrt(np.maximum(e, 0.0) / (4.0 * math.pi)))
        prev = np.concatenate([amp[:, :1], amp[:, :-1]], axis=1)
        w = np.arange(spb) / spb
        t = delays[k] + (np.arange(bins) + 0.5) * spb / fs
        air = np.exp(-np.asarray(AIR)[:, None] * (t * C)[None])
        env = ((1.0 - w) * prev[:, :, None] + w * amp[:, :, None]) * air[:, :, None]
        x = env.reshape(BANDS, n) * noise
        y = _lowpass(x[None], fs)[0]
        b = np.concatenate([y[:1], y[1:5] - y[5:9], x[5:6] - y[9:10]])
        out.append(b.reshape(-1))
    return {"irs": np.concatenate(out)}


class _Surfaces:
    """Vectorised float64 ray queries against a compiled scene's surfaces."""

    def __init__(self, a):
        self.a = a
        self.kinds = np.asarray(a["kinds"])
        self.corners = np.asarray(a["corners"])[:, :2]

    def inside(self, x, y):
        r = np.zeros(x.shape, dtype=bool)
        n = len(self.corners)
        for i in range(n):
            (xi, yi), (xj, yj) = self.corners[i], self.corners[i - 1]
            if abs(yj - yi) > 1e-12:
                cross = (yi > y) != (yj > y)
                r ^= cross & (x < (xj - xi) * (y - yi) / (yj - yi) + xi)
        return r

    def hit(self, s, o, d):
        """(t, normal [rays, 3] or [3]) of surface s; t = 1e30 where it is missed."""
        a, kind = self.a, self.kinds[s]
        miss = np.full(len(o), 1e30)
        if kind == 0:
            (ax, ay), (sx, sy) = a["wall_a"][s], a["wall_delta"][s]
            z0, z1 = a["wall_z"][s]
            det = sx * d[:, 1] - sy * d[:, 0]
            rx, ry = o[:, 0] - ax, o[:, 1] - ay
            t, u = (rx * sy - ry * sx) / det, (rx * d[:, 1] - ry * d[:, 0]) / det
            z = o[:, 2] + t * d[:, 2]
            ok = ((np.abs(det) > 1e-12) & (t > 1e-6) & (u >= -1e-6) & (u <= 1.0 + 1e-6) & (z >= z0 - 1e-6)
                  & (z <= z1 + 1e-6))
            return np.where(ok, t, miss), a["normals"][s]
        if kind == 1:
            t = (a["z_values"][s] - o[:, 2]) / d[:, 2]
            ok = (np.abs(d[:, 2]) > 1e-12) & (t > 1e-6)
            ok &= self.inside(np.where(ok, o[:, 0] + t * d[:, 0], 0.0), np.where(ok, o[:, 1] + t * d[:, 1], 0.0))
            return np.where(ok, t, miss), a["normals"][s]
        u3 = np.r_[a["box_axis_u"][s], 0.0]
        v3 = np.r_[a["box_axis_v"][s], 0.0]
        rel = o - np.r_[a["box_center"][s], 0.0]
        hw, hd = a["box_half"][s]
        t0, t1 = np.full(len(o), -1e30), np.full(len(o), 1e30)
        n0, n1 = np.zeros_like(o), np.zeros_like(o)
        ok = np.ones(len(o), dtype=bool)
        for axis, lo, hi in ((u3, -hw, hw), (v3, -hd, hd), (np.r_[0.0, 0.0, 1.0], *a["box_z"][s])):
            oo, dd = rel @ axis, d @ axis
            flat = np.abs(dd) <= 1e-12
            ok &= ~flat | ((oo >= lo) & (oo <= hi))
            ta, tb = (lo - oo) / dd, (hi - oo) / dd
            enter, leave = np.minimum(ta, tb), np.maximum(ta, tb)
            sign = np.sign(dd)[:, None] * axis
            first, last = ~flat & (enter > t0), ~flat & (leave < t1)
            t0, n0 = np.where(first, enter, t0), np.where(first[:, None], -sign, n0)
            t1, n1 = np.where(last, leave, t1), np.where(last[:, None], sign, n1)
        ok &= (t0 <= t1) & (t1 > 1e-6)
        front = t0 > 1e-6
        t = np.where(front, t0, t1)
        return np.where(ok & (t < 1e29), t, miss), np.where(front[:, None], n0, n1)

    def closest(self, o, d):
        best_t, best, normal = np.full(len(o), 1e30), np.full(len(o), -1), np.zeros_like(o)
        for s in range(len(self.kinds)):
            t, n = self.hit(s, o, d)
            nearer = t < best_t
            best_t, best = np.where(nearer, t, best_t), np.where(nearer, s, best)
            normal = np.where(nearer[:, None], n, normal)
        back = np.sum(normal * d, axis=1) > 0.0
        return best_t, best, np.where(back[:, None], -normal, normal)

    def blocked(self, o, d, limit):
        r = np.zeros(len(o), dtype=bool)
        for s in range(len(self.kinds)):
            left = ~r
            r[left] = self.hit(s, o[left], d[left])[0] < limit[left]
        return r


def _unit(v):
    n = np.linalg.norm(v, axis=1, keepdims=True)
    return np.where(n > 1e-12, v / np.maximum(n, 1e-300), 0.0)


def _sphere_before(o, d, centre, radius, t):
    rel = o - centre
    b = np.sum(rel * d, axis=1)
    disc = b * b - (np.sum(rel * rel, axis=1) - radius * radius)
    root = -b - np.sqrt(np.maximum(disc, 0.0))
    return (disc >= 0.0) & (root >= 0.0) & (root < t)


def _exact_trace(case, seed):
    """The drop-in's random stream and its path tracer in numpy: jittered Fibonacci directions, one uniform and one
    bank index per (bounce, ray), a 128-sample cosine bank, next-event estimation toward the source."""
    w = _room(case, seed)
    R, B, cfg = case["rays"], case["bounces"], w.config
    if R * B * workloads.count_surfaces(w.spec) > 70e6:
        return None
    a = scene.compile_scene(w.spec).arrays
    surfaces = _Surfaces(a)
    src, lst = np.asarray(w.sources[0]), np.asarray(w.listeners[0])
    i = np.arange(R) + 0.5
    z = 1.0 - 2.0 * i / R
    theta = i * (math.pi * (3.0 - math.sqrt(5.0))) + np.random.default_rng(cfg.seed).uniform(-0.02, 0.02, R)
    r = np.sqrt(np.clip(1.0 - z * z, 0.0, 1.0))
    d0 = np.stack([np.cos(theta) * r, np.sin(theta) * r, z], axis=1)
    k = np.arange(128)
    inverse = sum(((k >> j) & 1) * 0.5 ** (j + 1) for j in range(7))
    u = (k + 0.5) / 128
    bank = np.stack([np.sqrt(u) * np.cos(2 * math.pi * inverse), np.sqrt(u) * np.sin(2 * math.pi * inverse),
                     np.sqrt(1.0 - u)], axis=1)
    draws = np.random.default_rng(cfg.seed + 1)
    weight, power = {"cardioid": (0.5, 1.0), None: (0.0, 1.0)}[w.source_model]
    forward = np.r_[1.0, 0.0, 0.0]
    bins, names = cfg.num_bins, a["names"]
    echo, amb, energy = np.zeros((BANDS, bins)), np.zeros((BANDS, 4, bins)), np.zeros(len(names))
    delay = float(np.linalg.norm(src - lst)) / cfg.c
    o, d, acc, path = np.repeat(lst[None], R, 0), d0.copy(), np.ones((R, BANDS)), np.zeros(R)
    ray = np.arange(R)
    with np.errstate(divide="ignore", invalid="ignore"):
        for bounce in range(B):
            uniform = draws.random(R)
            index = draws.integers(0, 128, size=R, dtype=np.int32)
            if not len(ray):
                continue
            t, surf, n = surfaces.closest(o, d)
            dead = (surf < 0) | (t <= cfg.rt_listener_radius) | (path > cfg.max_path_length)
            if bounce > 0:
                dead |= _sphere_before(o, d, lst, cfg.rt_listener_radius, t)
                if np.linalg.norm(lst - src) > cfg.rt_source_radius:
                    dead |= _sphere_before(o, d, src, cfg.rt_source_radius, t)
            keep = ~dead
            ray, o, d, acc, path, t, surf, n = (v[keep] for v in (ray, o, d, acc, path, t, surf, n))
            h = o + t[:, None] * d + 1e-2 * n
            to = src - h
            dist = np.linalg.norm(to, axis=1)
            sd = to / dist[:, None]
            facing = np.sum(n * sd, axis=1)
            refl, scat = a["reflection"][surf], a["scattering"][surf]
            lit = np.flatnonzero((dist > cfg.rt_irradiance_min_distance) & (facing > 0.0))
            lit = lit[~surfaces.blocked(h[lit], sd[lit], dist[lit] - 1e-6)]
            cos_half = np.maximum(np.sum(_unit(sd[lit] - d[lit]) * n[lit], axis=1), 0.0)
            m = cfg.rt_specular_exponent
            brdf = (scat[lit] * facing[lit] / math.pi
                    + (m + 2.0) / (8.0 * math.pi) * (1.0 - scat[lit]) * cos_half ** m)
            gain = np.abs((1.0 - weight) + weight * -(sd[lit] @ forward)) ** power
            q = np.floor(((path[lit] + t[lit] + dist[lit]) / cfg.c - delay) / cfg.rt_bin_duration_s)
            fits = (q >= 0) & (q < bins)
            e = (4.0 * math.pi / R * gain * brdf / (4.0 * math.pi * dist[lit] ** 2))[:, None] * refl[lit] * acc[lit]
            lit, e, q = lit[fits], e[fits], q[fits].astype(int)
            for b in range(BANDS):
                np.add.at(echo[b], q, e[:, b])
                np.add.at(amb[b, 0], q, e[:, b])
                for axis in range(3):
                    np.add.at(amb[b, 1 + axis], q, e[:, b] * d0[ray[lit], axis])
            np.add.at(energy, surf[lit], e.sum(axis=1))
            acc = acc * refl
            path = path + t
            diffuse = uniform[ray] < scat
            s = bank[index[ray]]
            side = np.where((np.abs(n[:, :1]) >= 0.9), np.array([[0.0, 1.0, 0.0]]), np.array([[1.0, 0.0, 0.0]]))
            tangent = _unit(np.cross(side, n))
            scattered = s[:, :1] * tangent + s[:, 1:2] * np.cross(n, tangent) + s[:, 2:] * n
            mirrored = d - 2.0 * np.sum(d * n, axis=1, keepdims=True) * n
            d = _unit(np.where(diffuse[:, None], scattered, mirrored))
            o = h
            keep = path <= cfg.max_path_length
            ray, o, d, acc, path = (v[keep] for v in (ray, o, d, acc, path))
    # surfaces that share a name are reported under it once, the last one's value
    last = {n: k for k, n in enumerate(names)}
    return {"echogram": echo, "ambisonic": amb if case["ambisonics"] else None, "rays": None, "hits": None,
            "contributions": None, "energy": np.asarray([energy[last[n]] for n in names]), "visual": None}


def exact(case, seed):
    if case["kind"] == "dropin":
        return _exact_trace(case, seed)
    if case["kind"] == "synth":
        return _exact_synth(case, seed)
    return None
