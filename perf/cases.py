"""The calls that users of the tracer make, as timed cases.

A case is a dict of plain values.  `prepare` loads the scene and gives it
what a program holds before the call (sample pools, facet offsets, a batch, a
differentiable pair, an image); `run` is one pass through the package's public
entry points; `exact` is what the same inputs give in 64-bit arithmetic, by a
tracer of plain torch operations without a grid (every heliostat that a cone
around the rays can reach is tested); `work` counts what a pass cannot do
without.

Scenes are the package's seeded synthetic fields (small, large, uneven, huge,
two receivers) in their own configurations: 128 groups x 2048 lights, 2 or 2.9
mrad slope error, 0.02-0.25 m micro-facets.  "own" sample sets are the caller's
(a pillbox sun, Gaussian slope errors, random facet offsets), as a parity run
or a measured sun shape brings them; "seeded" ones are the package's.
"""
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

import solarenergy_chier_b200 as q
from solarenergy_chier_b200 import synth

PILLBOX = 0.00465
SIGMA_PX = 2.0
# exact() traces ray by ray in torch: beyond these it takes over about 20 seconds
EXACT_RAYS = 2.5e8
EXACT_HELIOSTATS = 3000


def listed():
    return [
        # the smallest call: one heliostat of a small plant at a few lights, image and power read back
        {"name": "one heliostat", "kind": "trace", "field": "small", "px": 0.05, "rpx": 0.05, "heliostats": 1,
         "lights": 64, "calls": "one", "pools": "own", "mode": 0},
        # the reference's loop over rayTracing(scene, heliostat), one call each
        {"name": "heliostat by heliostat", "kind": "trace", "field": "small", "px": 0.05, "rpx": 0.05,
         "heliostats": 50, "lights": 256, "calls": "each", "pools": "own", "mode": 0},
        # a small plant at its full sample count in one call
        {"name": "small plant, all lights", "kind": "trace", "field": "small", "px": 0.05, "rpx": 0.05,
         "heliostats": 50, "lights": 2048, "calls": "one", "pools": "seeded", "mode": 0},
        # the benchmark's plant (624 focus-flat heliostats, cylinder), the largest single trace
        {"name": "large plant", "kind": "trace", "field": "large", "px": 0.02, "rpx": 0.02, "heliostats": 624,
         "lights": 32, "calls": "one", "pools": "seeded", "mode": 0},
        # the build that rounds as the reference's host code, two receivers and grids, an odd light count
        {"name": "two receivers, exact build", "kind": "trace", "field": "two", "px": 0.05, "rpx": 0.05,
         "heliostats": 24, "lights": 117, "calls": "one", "pools": "own", "mode": 1},
        # new sample sets from the host before every trace, as a measured sun shape or a replicate does
        {"name": "new sample set", "kind": "resample", "field": "small", "px": 0.1, "rpx": 0.05, "lights": 33,
         "pools": "own", "mode": 0},
        # hours of a day, one sun after another, few lights each
        {"name": "suns in turn", "kind": "suns", "field": "uneven", "index": 13, "px": 0.2, "rpx": 0.05, "suns": 4,
         "lights": 4, "pools": "own", "mode": 0},
        # a year's suns and a second plant in one batch: new suns, one graph launch, all images and powers
        {"name": "batch of suns", "kind": "batch", "keep": 4, "index": 8, "px": 0.1, "rpx": 0.05, "suns": 12,
         "lights": 4, "pools": "seeded", "mode": 0},
        # one step of aim-point optimisation on a slice of the benchmark's plant
        {"name": "aim step", "kind": "diff", "field": "large", "keep": 13, "px": 0.02, "rpx": 0.02, "suns": 1,
         "lights": 32, "pools": "seeded"},
        # the same over several suns of the 10,000-heliostat plant, few lights on coarse facets
        {"name": "aim step, huge plant", "kind": "diff", "field": "huge", "keep": 1, "px": 0.25, "rpx": 0.05,
         "suns": 4, "lights": 4, "pools": "seeded"},
        # the pipeline's smoother (radius 5, ratio 0.05) on the benchmark's flux map
        {"name": "smooth 11x11", "kind": "smooth", "width": 1257, "height": 600, "radius": 5, "ratio": 0.05},
        # the 3x3 window trimmed by one at each end, on the small plant's flux map
        {"name": "smooth 3x3", "kind": "smooth", "width": 160, "height": 120, "radius": 1, "ratio": 0.17},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "resample", "suns", "batch", "diff", "smooth"])
    mode = rng.choice([0, 0, 0, 1])
    if kind == "smooth":
        radius = rng.randint(1, 6)
        return {"kind": kind, "width": int(_log(rng, 40, 1500)), "height": int(_log(rng, 30, 1200)), "radius": radius,
                "ratio": round(rng.uniform(0.12, 0.3) if radius == 1 else rng.uniform(0.03, 0.25), 3)}
    if kind == "resample":
        return {"kind": kind, "field": "small", "px": rng.choice([0.05, 0.1, 0.2]), "rpx": 0.05,
                "lights": int(_log(rng, 5, 500)), "pools": "own", "mode": mode}
    if kind == "suns":
        return {"kind": kind, "field": "uneven", "index": rng.choice([8, 10, 13]), "px": rng.choice([0.1, 0.2, 0.25]),
                "rpx": 0.05, "suns": rng.randint(2, 4), "lights": int(_log(rng, 2, 24)), "pools": "own", "mode": mode}
    if kind == "batch":
        return {"kind": kind, "keep": rng.randint(3, 9), "index": rng.choice([8, 10, 13]),
                "px": rng.choice([0.1, 0.2, 0.25]), "rpx": 0.05, "suns": rng.randint(3, 16),
                "lights": int(_log(rng, 2, 16)), "pools": "seeded", "mode": 0}
    if kind == "diff":
        field = rng.choice(["small", "large", "huge"])
        px = {"small": 0.05, "large": rng.choice([0.02, 0.05]), "huge": 0.25}[field]
        return {"kind": kind, "field": field, "keep": {"small": 1, "large": rng.randint(8, 20), "huge": 1}[field],
                "px": px, "rpx": 0.05 if field != "large" else 0.02, "suns": rng.randint(1, 4),
                "lights": int(_log(rng, 3, 10 if field == "huge" else 40)),
                "pools": "own" if field == "small" else "seeded"}
    field = rng.choice(["small", "uneven", "two", "large"])
    if field == "large":  # part of the plant: at most a few 1e9 rays
        n = int(_log(rng, 5, 624))
        return {"kind": kind, "field": field, "px": 0.02, "rpx": 0.02, "heliostats": n,
                "lights": int(_log(rng, 3, min(300, 32 * 624 / n))), "calls": "one", "pools": "seeded", "mode": 0}
    case = {"kind": kind, "field": field, "px": rng.choice([0.05, 0.1, 0.17]), "rpx": rng.choice([0.05, 0.08]),
            "heliostats": int(_log(rng, 1, {"small": 50, "two": 24, "uneven": 490}[field])),
            "lights": int(_log(rng, 3, 700 if field != "uneven" else 60)),
            "calls": rng.choice(["one", "one", "each"]) if field == "small" else "one", "pools": "own", "mode": mode}
    if field == "uneven":
        case.update(index=rng.choice([8, 10, 13]), px=rng.choice([0.1, 0.17, 0.25]))
    return case


# ---- inputs ------------------------------------------------------------------
def _files(case, out, seed, field=None):
    field = field or case["field"]
    px = {"helio_pixel": case["px"], "receiver_pixel": case["rpx"]}
    if field == "small":
        return synth.small_field(out, seed, **px)
    if field == "large":
        return synth.large_field(out, seed, keep_every=case.get("keep", 1), **px)
    if field == "uneven":
        return synth.uneven_field(out, case["index"], **px)
    if field == "huge":
        return synth.huge_field(out, seed, **px)
    return synth.two_receiver_field(out, seed, groups=128, per_group=2048, **px)


def _suns(n, seed):
    """n sun directions spread over the daylight hours of a day of the year."""
    day = synth.sun_positions(days=12, hours=max(n, 2)).reshape(12, -1, 3)
    return day[seed % 12][:n]


def _ids(case, total):
    """The heliostats that a case traces: all, or some spread over the plant."""
    n = min(case.get("heliostats", total), total)
    return [k * total // n for k in range(n)]


def _sample_set(groups, lights, sigma, seed):
    """A caller's own pools: a pillbox sun and Gaussian slope errors, as unit vectors."""
    g = torch.Generator().manual_seed(seed)
    u = torch.rand((groups * lights, 2), generator=g, dtype=torch.float64)
    th = 2.0 * torch.asin(torch.sqrt(u[:, 0]) * math.sin(0.5 * PILLBOX))
    ph = 2.0 * math.pi * u[:, 1]
    dirs = torch.stack([th.sin() * ph.cos(), th.cos(), th.sin() * ph.sin()], 1)
    n = sigma * torch.randn((groups * lights, 2), generator=g, dtype=torch.float64).clamp(-5.0, 5.0)
    pert = torch.stack([n[:, 0], torch.ones(len(n), dtype=torch.float64), n[:, 1]], 1)
    pert /= pert.norm(dim=1, keepdim=True)
    return dirs.float().numpy(), pert.float().numpy()


def _offsets(counts, pool, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, pool, n + 1, dtype=np.int32) for n in counts]


def _scene(case, seed, field=None):
    with tempfile.TemporaryDirectory() as tmp:
        files = _files(case, tmp, seed, field)
        scene = q.Scene(files.scene, files.config, device=0, seed=seed)
    scene.set_math_mode(case.get("mode", 0))
    scene.set_light_range(0, case["lights"])
    if case["pools"] == "own":
        scene.set_sample_pool(*_sample_set(scene.info.num_sunshape_groups, scene.lights_per_group,
                                           scene.info.helio_disturb_std, seed))
        counts = [scene.heliostat(h)["num_facets"] for h in range(scene.num_heliostats)]
        for h, o in enumerate(_offsets(counts, scene.pool_size, seed)):
            scene.set_facet_offsets(h, o)
    return scene


def _flux_map(case, seed):
    """A flux map as a trace leaves it: a few overlapping spots with the rays' counting noise, dark at the edges."""
    h, w = case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    y, x = torch.meshgrid(torch.linspace(0, 1, h, device="cuda"), torch.linspace(0, 1, w, device="cuda"),
                          indexing="ij")
    r = torch.rand((6, 3), generator=g, device="cuda")
    mean = sum(40 * torch.exp(-((x - 0.2 - 0.6 * a) ** 2 + (y - 0.3 - 0.4 * b) ** 2) / (0.005 + 0.02 * c))
               for a, b, c in r)
    return torch.poisson(mean, generator=g) * 3.7


def _params(n, seed):
    rng = np.random.default_rng([seed, 1])
    return (rng.uniform(-0.5, 0.5, (n, 2)).astype(np.float32), rng.uniform(-5e-4, 5e-4, (n, 2)).astype(np.float32))


def _target(shape, seed):
    h, w = shape
    ph = np.random.default_rng([seed, 2]).uniform(0, 2 * np.pi, 2)
    rows, cols = np.mgrid[0:h, 0:w]
    return (1000.0 * (1.0 + 0.5 * np.cos(6 * np.pi * cols / w + ph[0]) *
                      np.cos(np.pi * rows / h + ph[1]))).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "smooth":
        src = _flux_map(case, seed)
        return {"case": case, "src": src, "img": torch.empty_like(src)}
    if kind == "batch":
        scenes = [_scene(case, seed, "large"), _scene(case, seed + 1, "uneven")]
        suns = _suns(case["suns"], seed)
        inst = [(k, d) for k in (0, 1) for d in suns]
        batch = q.Batch(scenes, inst)
        batch.set_light_range(0, case["lights"])
        batch.capture_graph(clear_first=True)
        return {"case": case, "batch": batch, "suns": np.stack([d for _, d in inst])}
    scene = _scene(case, seed)
    state = {"case": case, "scene": scene}
    if kind == "trace":
        state.update(tracer=q.QuasiMonteCarloRayTracer(), ids=_ids(case, scene.num_heliostats))
    elif kind == "resample":
        state.update(pools=_sample_set(scene.info.num_sunshape_groups, scene.lights_per_group,
                                       scene.info.helio_disturb_std, seed + 7),
                     ids=list(range(scene.num_heliostats)))
    elif kind == "suns":
        state.update(suns=_suns(case["suns"], seed), ids=list(range(scene.num_heliostats)))
    else:
        diff = q.Diff(scene, sigma_px=SIGMA_PX, suns=None if case["suns"] == 1 else _suns(case["suns"], seed))
        diff.set_light_range(0, case["lights"])
        shape = diff.flux(0).shape
        for k in range(case["suns"]):
            diff.set_target(_target(shape, seed), k)
        state.update(diff=diff, params=_params(scene.num_heliostats, seed))
    return state


# ---- one pass ------------------------------------------------------------------
def _read(scene):
    per, total = scene.power()
    return {"images": [scene.image(r) for r in range(scene.num_receivers)], "power": per, "total": total}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "smooth":
        img = state["img"]
        img.copy_(state["src"])  # the smoother works in place
        q.ImageSmoother.image_smooth(img.data_ptr(), case["radius"], case["ratio"], case["width"], case["height"])
        return img
    if kind == "batch":
        b = state["batch"]
        b.set_suns(state["suns"])
        b.graph_launch()
        n = case["suns"]
        return {"images": [np.stack([b.image(k * n + i) for i in range(n)]) for k in (0, 1)],
                "power": [np.stack([b.power(k * n + i)[0] for i in range(n)]) for k in (0, 1)]}
    scene = state["scene"]
    if kind == "diff":
        d = state["diff"]
        d.set_params(*state["params"])
        loss = d.forward()
        grad = d.backward()
        # The parameters are float32, and so is the gradient that an optimiser over them takes.
        return {"loss": loss, "grad": grad.astype(np.float32), "flux": [d.flux(k) for k in range(case["suns"])]}
    if kind == "suns":
        out = []
        for sun in state["suns"]:
            scene.set_sun(sun)
            scene.clear()
            scene.clear_power()
            scene.trace(state["ids"])
            out.append(_read(scene))
        return out
    scene.clear()
    scene.clear_power()
    if kind == "resample":
        scene.set_sample_pool(*state["pools"])
    if case.get("calls") == "each":
        for h in state["ids"]:
            state["tracer"].rayTracing(scene, h)
    else:
        scene.trace(state["ids"])
    return _read(scene)


# ---- what a pass cannot do without ---------------------------------------------
def _field_numbers(case):
    """(heliostats, micro-facets of one, image pixels) of a case's field, to a percent."""
    px, rpx = case["px"], case["rpx"]
    if case["kind"] == "batch" or case.get("field") == "large":
        keep = case.get("keep", 1)
        return -(-624 // keep), 12.84 * 9.45 / px ** 2, 25.1 * 12 / rpx ** 2
    if case["field"] == "uneven":
        n, side = {8: (692, 7.38), 10: (493, 10.76), 13: (648, 9.83)}[case["index"]]
        return n, side ** 2 / px ** 2, 400.0 / rpx ** 2
    if case["field"] == "huge":
        return 10000, 100.0 / px ** 2, 62.8 * 20 / rpx ** 2
    if case["field"] == "two":
        return 24, 24.5 / px ** 2, 2 * 40.0 / rpx ** 2
    return 50, 16.0 / px ** 2, 48.0 / rpx ** 2


# Per ray: the slope-error normal in the facet's frame (15) and normalised (9), the reflection (14), the receiver's
# intersection (45) and the energy (12); the adjoint's reverse pass over the same chain costs about twice that again.
RAY_FLOPS = 95.0
# Streamed once per pass: a pool offset per micro-facet, both sample pools, the image.
POOL_BYTES = 2 * 12 * 128 * 2048


def work(case):
    kind = case["kind"]
    if kind == "smooth":
        n = case["width"] * case["height"]
        return {"bytes": 8.0 * n, "flops": float(n * (2 * case["radius"] + 1) ** 2)}
    n, facets, pixels = _field_numbers(case)
    if kind == "trace":
        n = min(case["heliostats"], n)
    suns = case.get("suns", 1)
    rays = n * facets * case["lights"] * suns
    total = n * facets
    if kind == "batch":
        n2, f2, _ = _field_numbers(dict(case, kind="suns", field="uneven"))
        rays += n2 * f2 * case["lights"] * suns
        total += n2 * f2
    flops = RAY_FLOPS * rays * (3.0 if kind == "diff" else 1.0)
    return {"bytes": 4.0 * total * suns + POOL_BYTES + 4.0 * pixels * suns * (3 if kind == "diff" else 1),
            "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------
class _Field:
    """A scene file's heliostats and receivers, and the geometry of a sun, in 64 bits."""

    def __init__(self, scene_text, config_text):
        import json

        cfg = json.loads(config_text)
        self.cfg = cfg
        f32 = np.float32
        self.px = float(f32(cfg["helio_pixel_length"]))
        self.ppm = int(f32(1.0) / f32(cfg["receiver_pixel_length"]))
        self.recv, self.grids, self.helio = [], [], []
        vec = lambda w: np.array([float(f32(x)) for x in w])  # noqa: E731
        matrix, lines = (1, 1), scene_text.splitlines()
        section, k = None, 0
        while k < len(lines):
            w = lines[k].split()
            k += 1
            if not w or w[0].startswith("#"):
                continue
            if w[0] == "Recv":
                section = {"type": int(w[1])}
                self.recv.append(section)
            elif w[0] == "Grid":
                section = {"recv": len(self.recv) - 1}
                self.grids.append(section)
            elif w[0] in ("pos", "size", "norm"):
                section[w[0]] = vec(w[1:4])
            elif w[0] == "type":
                section["helio"] = int(w[1])
            elif w[0] == "matrix":
                matrix = (int(w[1]), int(w[2]))
            elif w[0] == "helio":
                self.helio.append({"pos": vec(w[1:4]), "size": vec(lines[k].split()), "matrix": matrix,
                                   "grid": len(self.grids) - 1, "type": section["helio"]})
                k += 1
        for h in self.helio:
            rows, cols = h["matrix"]
            h["len"] = (f32(h["size"][2]) / f32(rows), f32(h["size"][0]) / f32(cols))  # (along z, along x), no gaps
            h["sub"] = tuple(int(v / f32(cfg["helio_pixel_length"])) for v in h["len"])
            h["facets"] = rows * cols * h["sub"][0] * h["sub"][1]
            h["len"] = tuple(float(v) for v in h["len"])
            h["focus"] = self._focus(self.recv[self.grids[h["grid"]]["recv"]], h["pos"])
            h["focal"] = float(np.linalg.norm(h["focus"] - h["pos"]))

    @staticmethod
    def _focus(r, pos):
        if r["type"] == 0:  # every rectangle here faces +z: the centre of its front
            return r["pos"] + np.array([0.0, 0.0, r["size"][2] / 2])
        d = pos - r["pos"]
        return r["pos"] + np.array([d[0], 0.0, d[2]]) * (r["size"][0] / math.hypot(d[0], d[2]))

    def shape(self, r):
        w = self.recv[r]["size"]
        x = w[0] if self.recv[r]["type"] == 0 else 2 * math.pi * w[0]
        return int(w[1] * self.ppm), (int(x * self.ppm) if self.recv[r]["type"] == 0 else math.ceil(x * self.ppm))

    def orient(self, sun, aim=None, turn=None):
        for i, h in enumerate(self.helio):
            focus = h["focus"]
            if aim is not None:
                r = self.recv[self.grids[h["grid"]]["recv"]]
                d = focus - r["pos"]
                au = np.array([-d[2], 0.0, d[0]]) / math.hypot(d[0], d[2]) if r["type"] else np.array([1.0, 0.0, 0.0])
                focus = focus + au * float(aim[i][0]) + np.array([0.0, 1.0, 0.0]) * float(aim[i][1])
            n = _unit(_unit(focus - h["pos"]) - sun)
            if turn is not None:
                u, n0, v = _frame(n, False)
                n = _unit(n0 + u * float(turn[i][0]) + v * float(turn[i][1]))
            h["normal"] = n
            F = _frame(n, h["type"] == 1)
            sx, sy, sz = h["size"]
            rows, cols = h["matrix"]
            subs = []
            if h["type"] == 0:
                subs.append((np.array([0.0, sy / 2, 0.0]), np.array([0.0, 1.0, 0.0])))
            else:
                for r_ in range(rows):
                    for c in range(cols):
                        x, z = (c + 0.5) * h["len"][1] - sx / 2, (r_ + 0.5) * h["len"][0] - sz / 2
                        subs.append((np.array([x, sy / 2 + (x * x + z * z) / (4 * h["focal"]), z]),
                                     _unit(np.array([-x / (2 * h["focal"]), 1.0, -z / (2 * h["focal"])]))))
            h["subs"], h["para"], h["spread"] = subs, [], 0.0
            for c, ln in subs:
                G = _frame(ln, True) if h["type"] == 1 else _frame(np.array([0.0, 1.0, 0.0]), False)
                lz, lx = h["len"] if h["type"] == 1 else (sz, sx)
                ab, ac = _turn(F, _turn(G, np.array([0.0, 0.0, lz]))), _turn(F, _turn(G, np.array([lx, 0.0, 0.0])))
                self_c = _turn(F, c) + h["pos"]
                h["para"].append((self_c - 0.5 * ab - 0.5 * ac, ab, ac))
                h["spread"] = max(h["spread"], math.acos(min(1.0, ln[1])))
            h["radius"] = 0.5 * float(np.linalg.norm(h["size"])) + 0.3

    def facets(self, h):
        """Centres and normals of a heliostat's micro-facets, row by row, on the GPU."""
        rows, cols = h["matrix"]
        sr, sc = h["sub"]
        f = torch.arange(h["facets"], device="cuda")
        row, col = f // (cols * sc), f % (cols * sc)
        F = _frame(h["normal"], h["type"] == 1)
        if h["type"] == 0:
            p = torch.stack([(col + 0.5) * self.px - h["size"][0] / 2, torch.full_like(f, 0).double() + h["size"][1] / 2,
                             (row + 0.5) * self.px - h["size"][2] / 2], 1)
            return _turn(F, p) + _t(h["pos"]), _t(h["normal"]).expand(len(f), 3)
        o = torch.empty((len(f), 3), dtype=torch.float64, device="cuda")
        n = torch.empty_like(o)
        block = (row // sr) * cols + col // sc
        for b, (c, ln) in enumerate(h["subs"]):
            m = block == b
            lp = torch.stack([(col[m] % sc + 0.5) * self.px - h["len"][1] / 2, torch.zeros_like(col[m]).double(),
                              (row[m] % sr + 0.5) * self.px - h["len"][0] / 2], 1)
            o[m] = _turn(F, _turn(_frame(ln, True), lp) + _t(c)) + _t(h["pos"])
            n[m] = _t(_turn(F, ln))
        return o, n


def _t(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def _unit(v):
    return v / np.linalg.norm(v)


def _frame(n, flip):
    """(u, n, v): the axes that local x, y, z turn into about a normal."""
    if abs(n[0]) < 1e-5 and abs(n[2]) < 1e-5:
        return np.array([1.0, 0, 0]), np.array([0, 1.0, 0]), np.array([0, 0, 1.0])
    u = _unit(np.cross([0.0, 1.0, 0.0], n))
    v = _unit(np.cross(u, n))
    return (-u, n, -v) if flip and n[2] < 0 else (u, n, v)


def _turn(F, p):
    if isinstance(p, torch.Tensor):
        return p @ torch.stack([_t(a) for a in F])
    return p[0] * F[0] + p[1] * F[1] + p[2] * F[2]


def _dot(a, b):
    return (a * b).sum(-1)


def _plane(o, d, a, ab, ac):
    """Rays against a parallelogram: (hit, t, u, v)."""
    a, ab, ac = _t(a), _t(ab), _t(ac)
    p = torch.linalg.cross(d, ac.expand_as(d))
    det = _dot(p, ab)
    tv = o - a
    inv = 1.0 / torch.where(det.abs() < 1e-5, torch.ones_like(det), det)
    u = _dot(tv, p) * inv
    w = torch.linalg.cross(tv, ab.expand_as(tv))
    v, t = _dot(d, w) * inv, _dot(w, ac) * inv
    return (det.abs() >= 1e-5) & (u >= 0) & (u <= 1) & (v >= 0) & (v <= 1) & (t >= 1e-5), t, u, v


def _receiver(r, o, d):
    """Rays against a receiver: (hit, t, row fraction, column fraction)."""
    if r["type"] == 0:
        x, y, z = r["size"]
        return _plane(o, d, r["pos"] + np.array([-x / 2, -y / 2, z / 2]), np.array([0, y, 0]), np.array([x, 0, 0]))
    c, rad, height = _t(r["pos"]), r["size"][0], r["size"][1]
    lx, lz = o[:, 0] - c[0], o[:, 2] - c[2]
    ln = torch.hypot(d[:, 0], d[:, 2])
    tp = -(lx * d[:, 0] + lz * d[:, 2]) / ln
    delta = ((lx * d[:, 2] - lz * d[:, 0]) / ln) ** 2
    t = (tp - torch.sqrt((rad * rad - delta).clamp_min(0.0))) / ln
    p = o + d * t[:, None]
    u = (p[:, 1] - c[1]) / height + 0.5
    phi = torch.atan2(p[:, 2] - c[2], p[:, 0] - c[0]) / (2 * math.pi)
    ok = (lx * lx + lz * lz > rad * rad) & (tp >= -1e-5) & (delta <= rad * rad) & (u >= 0) & (u <= 1)
    return ok, t, u, torch.where(phi < 0, phi + 1.0, phi)


def _reach(F, i, axis, spread):
    """The other heliostats of i's grid that rays within `spread` radians of an axis can meet."""
    h = F.helio[i]
    a, out = _unit(axis), []
    for j in F.members[h["grid"]]:
        g = F.helio[j]
        e = g["pos"] - h["pos"]
        s = float(e @ a)
        R = h["radius"] + g["radius"]
        if j != i and s > -R and float(np.linalg.norm(e - s * a)) <= R + max(s + R, 0.0) * math.tan(spread):
            out.append(j)
    return out


def _blocked(F, near, o, d):
    hit = torch.zeros(len(o), dtype=torch.bool, device="cuda")
    for j in near:
        for a, ab, ac in F.helio[j]["para"]:
            hit |= _plane(o, d, a, ab, ac)[0]
    return hit


def _trace64(F, ids, sun, pools, offsets, lights, images, power, splat=False):
    """Adds the flux of heliostats `ids` to images (64 bits, one per receiver) and sets their powers."""
    cfg = F.cfg
    dirs, pert = (_t(p) for p in pools)
    P, L = len(dirs), cfg["num_per_sunshape_group"]
    th = float(torch.acos(dirs[:, 1].min().clamp(max=1.0))) + 1e-4
    sl = float(torch.acos(pert[:, 1].min().clamp(max=1.0))) + 1e-4
    world = _turn(_frame(-sun, False), dirs)
    if not hasattr(F, "members"):
        F.members = [[i for i, h in enumerate(F.helio) if h["grid"] == g] for g in range(len(F.grids))]
    for i in ids:
        h = F.helio[i]
        rid = F.grids[h["grid"]]["recv"]
        r = F.recv[rid]
        H, W = F.shape(rid)
        factor = cfg["dni"] * (F.px * F.ppm) ** 2 * cfg["helio_reflected_rate"] / L
        origins, normals = F.facets(h)
        g = torch.as_tensor(offsets[i].astype(np.int64), device="cuda")
        mirror = sun - 2.0 * h["normal"] * float(sun @ h["normal"])
        shade = _reach(F, i, -sun, th)
        block = _reach(F, i, mirror, th + 2 * sl + 2 * h["spread"] + 1e-3)
        step = max(1, 2_000_000 // lights)
        lab = torch.arange(lights, device="cuda")
        for f0 in range(0, h["facets"], step):
            f = torch.arange(f0, min(f0 + step, h["facets"]), device="cuda").repeat_interleave(lights)
            l = lab.repeat(len(f) // lights)
            o = origins[f]
            d = world[(g[f] + l) % P]
            if shade:
                keep = ~_blocked(F, shade, o, d)
                f, l, o, d = f[keep], l[keep], o[keep], d[keep]
            # the slope error turns about the facet normal's frame
            n = normals[f]
            u = torch.stack([n[:, 2], torch.zeros_like(n[:, 0]), -n[:, 0]], 1)
            u = u / u.norm(dim=1, keepdim=True)
            v = torch.linalg.cross(u, n)
            e = pert[(g[(f + 1) % P] + l) % P]
            n = u * e[:, :1] + n * e[:, 1:2] + v * e[:, 2:]
            n = n / n.norm(dim=1, keepdim=True)
            rd = -d + n * (2.0 * _dot(n, d))[:, None]
            if block:
                keep = ~_blocked(F, block, o, rd)
                n, o, rd = n[keep], o[keep], rd[keep]
            ok, t, fu, fv = _receiver(r, o, rd)
            n, rd, t, fu, fv = n[ok], rd[ok], t[ok], fu[ok], fv[ok]
            eta = torch.where(t <= 1000.0, 0.99331 - 0.0001176 * t + 1.97e-8 * t * t, torch.exp(-0.0001106 * t))
            en = _dot(rd, n).abs() * eta * factor
            power[i] += float(en.sum())
            if not splat:
                pix = (fu * H).long().clamp(0, H - 1) * W + (fv * W).long().clamp(0, W - 1)
                images[rid].view(-1).index_add_(0, pix, en)
                continue
            x, y = fv * W - 0.5, fu * H - 0.5
            for k in range(4):
                c, w_ = torch.floor(x).long() + (k & 1), torch.floor(y).long() + (k >> 1)
                wx, wy = x - torch.floor(x), y - torch.floor(y)
                wt = (wx if k & 1 else 1 - wx) * (wy if k >> 1 else 1 - wy)
                if r["type"] == 1:
                    c = c % W
                m = (c >= 0) & (c < W) & (w_ >= 0) & (w_ < H)
                images[rid].view(-1).index_add_(0, (w_ * W + c)[m], (en * wt)[m])


def _smooth64(img, radius, ratio):
    """The reference's streaming trimmed mean: the k smallest and k largest of a window as its two heaps hold them."""
    h, w = img.shape
    src = img.double()
    row, col = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    span = lambda a, n: (a + radius).clamp(max=n - 1) - (a - radius).clamp(min=0) + 1  # noqa: E731
    cnt = span(row, h)[:, None] * span(col, w)[None, :]
    k = (cnt.float() * torch.tensor(ratio, dtype=torch.float32, device="cuda")).int()
    K = max(int(k.max()), 1)
    slot = torch.arange(K, device="cuda")[:, None, None]
    inf = torch.tensor(float("inf"), dtype=torch.float64, device="cuda")
    used = slot < k
    lo, hi = torch.where(used, inf, -inf), torch.where(used, -inf, inf)
    seen = torch.zeros_like(k)
    total = torch.zeros_like(src)
    for dy in range(-radius, radius + 1):
        for dx in range(-radius, radius + 1):
            ok = ((row + dy >= 0) & (row + dy < h))[:, None] & ((col + dx >= 0) & (col + dx < w))[None, :]
            cur = torch.roll(src, (-dy, -dx), (0, 1))
            total += torch.where(ok, cur, torch.zeros_like(cur))
            lt, li = lo.max(0)
            ht, hj = hi.min(0)
            fill, some = seen < k, ok & (k > 0)
            low = some & (fill | (cur < lt))
            high = some & (fill | (~(cur < lt) & (cur > ht)))
            lo = torch.where(low & (slot == li), cur, lo)
            hi = torch.where(high & (slot == hj), cur, hi)
            seen += ok.int()
    zero = torch.zeros_like(lo)
    return (total - torch.where(used, lo, zero).sum(0) - torch.where(used, hi, zero).sum(0)) / (cnt - 2 * k)


def _gauss64(img, wrap):
    r = math.ceil(3 * SIGMA_PX)
    w = torch.exp(-0.5 * (torch.arange(-r, r + 1, dtype=torch.float64, device="cuda") / SIGMA_PX) ** 2)
    w = (w / w.sum()).view(1, 1, 1, -1)
    x = torch.nn.functional.pad(img[None, None], (r, r, 0, 0), mode="circular" if wrap else "constant")
    x = torch.nn.functional.conv2d(x, w)
    return torch.nn.functional.conv2d(torch.nn.functional.pad(x, (0, 0, r, r)), w.view(1, 1, -1, 1))[0, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "smooth":
        return _smooth64(_flux_map(case, seed), case["radius"], case["ratio"])
    n, facets, _ = _field_numbers(case)
    if kind == "trace":
        n = min(n, case["heliostats"])
    suns = case.get("suns", 1)
    if case["pools"] != "own" or n * facets * case["lights"] * suns > EXACT_RAYS or n * suns > EXACT_HELIOSTATS:
        return None
    with tempfile.TemporaryDirectory() as tmp:
        files = _files(case, tmp, seed)
        F = _Field(Path(files.scene).read_text(), Path(files.config).read_text())
    cfg = F.cfg
    groups, lights = cfg["num_of_sunshape_groups"], cfg["num_per_sunshape_group"]
    pools = _sample_set(groups, lights, float(np.float32(cfg["helio_disturb_std"])),
                        seed + 7 if kind == "resample" else seed)
    offsets = _offsets([h["facets"] for h in F.helio], groups * lights, seed)
    ids = _ids(case, len(F.helio))
    own_sun = np.float32(cfg["sun_dir"]).astype(np.float64)

    def traced(sun, splat=False, **params):
        F.orient(sun, **params)
        images = [torch.zeros(F.shape(r), dtype=torch.float64, device="cuda") for r in range(len(F.recv))]
        power = np.zeros(len(F.helio))
        _trace64(F, ids, sun, pools, offsets, case["lights"], images, power, splat)
        return {"images": images, "power": power, "total": float(power.sum())}

    if kind == "diff":
        aim, turn = _params(len(F.helio), seed)
        sun_list = [own_sun] if suns == 1 else _suns(suns, seed).astype(np.float64)
        flux = [_gauss64(traced(s, True, aim=aim, turn=turn)["images"][0], F.recv[0]["type"] == 1) for s in sun_list]
        target = _t(_target(tuple(flux[0].shape), seed))
        # the gradient adds estimates of the receiver's edge terms, which no derivative of the forward holds
        return {"loss": float(sum(((f - target) ** 2).sum() for f in flux)), "grad": None, "flux": flux}
    if kind == "suns":
        return [traced(s.astype(np.float64)) for s in _suns(suns, seed)]
    return traced(own_sun)
