"""The work users have this framework do, as timed cases.

A pass goes through the public Python API with host images, as a caller's
program does: build a session (input upload, pyramids), run it, read the
result back.  Sessions are consumed by their run, so every pass builds its
own.  Inputs are the repository's synthetic textures (workloads.py), seeded.

Kinds of case:
  session  one synthesis: Session.builder() .. build().run() and its result
  batch    sessions of the batched mix run together (Batch)
  serve    a burst of requests, 70% batched mix and 30% inpainting, through a
           Server the program keeps (continuous batching)
  apply    a saved CoordinateTransform applied to other images (the normal
           or roughness map of a texture whose colours were synthesised)
"""
import importlib
import math
import random

import numpy as np

ts = importlib.import_module("texture-synthesis_gb300")
wl = importlib.import_module("texture-synthesis_gb300.workloads")

SIDE_MIN, SIDE_MAX = 48, 2048


def _session(name, w, h, ex_w, ex_h, n_ex=1, k=50, m=50, tiling=False, guide="none", init=-1, alpha=False,
             mask=False, inpaint=False, maps=False):
    """A synthesis.  guide: "none", "given" (a guide per example) or "auto" (a
    target guide only: style transfer, the examples' guides are made by the
    framework); init: random-init pixels (-1: none); alpha: examples with a
    transparent background; mask: the last example has a sample mask;
    inpaint: the first example is inpainted at the output size; maps: the
    caller also reads the coordinate and id maps and the resolve scores."""
    return {"name": name, "kind": "session", "w": w, "h": h, "ex_w": ex_w, "ex_h": ex_h, "n_ex": n_ex, "k": k, "m": m,
            "tiling": tiling, "guide": guide, "init": init, "alpha": alpha, "mask": mask, "inpaint": inpaint,
            "maps": maps}


def listed():
    return [
        # an icon or sprite with transparency: the smallest call, latency only
        _session("icon_64", 64, 64, 48, 48, k=20, m=20, alpha=True),
        # a sprite at the fast setting, odd sizes
        _session("sprite_203x117", 203, 117, 90, 131, k=8, m=8),
        # the single-example texture of the benchmark
        _session("single_256", 256, 256, 128, 128, init=0),
        # the builder's default output size, examples of a photo's shape, one of them masked
        _session("default_500", 500, 500, 320, 213, n_ex=2, mask=True),
        # the benchmark's headline: a seamless remix of four examples, with its maps
        _session("remix_512", 512, 512, 300, 300, n_ex=4, tiling=True, init=10, maps=True),
        # the benchmark's guided synthesis
        _session("guided_512", 512, 512, 256, 256, guide="given"),
        # style transfer to a photo's shape: the framework makes the guides
        _session("style_613x409", 613, 409, 350, 257, guide="auto", k=20, m=50),
        # an edit request: a 512^2 picture with rectangles to fill
        _session("inpaint_512", 512, 512, 512, 512, inpaint=True, maps=True),
        # a large seamless ground texture for a game
        _session("ground_2048", 2048, 2048, 512, 512, n_ex=2, tiling=True),
        # many small and large jobs at once: 24 sessions of the batched mix
        {"name": "batch_24", "kind": "batch", "n": 24, "side_max": 1024},
        # a server under a burst of 16 requests
        {"name": "serve_16", "kind": "serve", "n": 16, "side_max": 512},
        # a saved transform applied to two other maps of the same material
        {"name": "apply_1024", "kind": "apply", "w": 1024, "h": 1024, "ex_w": 512, "ex_h": 512, "n_ex": 2,
         "scale": 1.0},
    ]


def _logi(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["session", "batch", "serve", "apply"], [14, 2, 2, 2])[0]
    if kind == "batch":
        return {"kind": "batch", "n": rng.randint(2, 24), "side_max": rng.choice([256, 512, 1024])}
    if kind == "serve":
        return {"kind": "serve", "n": rng.randint(2, 16), "side_max": rng.choice([128, 256, 512])}
    if kind == "apply":
        return {"kind": "apply", "w": _logi(rng, 64, 2048), "h": _logi(rng, 64, 2048), "ex_w": _logi(rng, 48, 512),
                "ex_h": _logi(rng, 48, 512), "n_ex": rng.randint(1, 4), "scale": rng.choice([1.0, 1.0, 0.5, 2.0])}
    w = _logi(rng, SIDE_MIN, SIDE_MAX)
    h = min(SIDE_MAX, max(SIDE_MIN, int(w * rng.choice([1.0, rng.uniform(0.5, 2.0)]))))
    if rng.random() < 0.3:  # powers of two are what textures are mostly made at
        w = h = 1 << rng.randint(6, 10)
    inpaint = rng.random() < 0.2
    n_ex = rng.randint(1, 4)
    if inpaint:
        n_ex = 1
        w, h = min(w, 1024), min(h, 1024)
    c = _session("", w, h, _logi(rng, 48, 512), _logi(rng, 48, 512), n_ex=n_ex, k=rng.choice([8, 20, 50, 50]),
                 m=rng.choice([8, 20, 50, 50]), tiling=not inpaint and rng.random() < 0.4,
                 guide="none" if inpaint else rng.choice(["none", "none", "none", "given", "auto"]),
                 init=-1 if inpaint else rng.choice([-1, 0, 10]), alpha=rng.random() < 0.15,
                 mask=not inpaint and rng.random() < 0.2, inpaint=inpaint, maps=rng.random() < 0.3)
    if w * h > 1024 * 1024 and c["guide"] != "none":
        c["guide"] = "none"  # a drawn case costs no more than the largest listed one
    del c["name"]
    return c


def _example(seed, w, h, alpha):
    img = wl.texture(seed, h, w)
    if alpha:
        # a soft round cut-out: alpha falls from 255 to 0 towards the border
        yy, xx = np.mgrid[0:h, 0:w]
        r = np.hypot((xx + 0.5) / w - 0.5, (yy + 0.5) / h - 0.5)
        img[..., 3] = np.clip((0.55 - r) * 1500.0, 0, 255).astype(np.uint8)
    return img


def _session_spec(case, seed):
    w, h, ew, eh = case["w"], case["h"], case["ex_w"], case["ex_h"]
    base = 16 * seed
    params = dict(wl.DEFAULTS, nearest_neighbors=case["k"], random_sample_locations=case["m"],
                  seed=1000 + seed, tiling_mode=case["tiling"], random_init=None if case["init"] < 0 else case["init"])
    spec = {"name": "case", "out_w": w, "out_h": h, "params": params, "examples": [], "target_guide": None,
            "inpaint_mask": None, "inpaint_index": -1}
    for i in range(case["n_ex"]):
        if case["inpaint"] and i == 0:
            ew, eh = w, h
        e = {"image": _example(base + i, ew, eh, case["alpha"])}
        if case["guide"] == "given":
            e["guide"] = wl.example_guide(base + 8 + i, eh, ew, sigma=max(1.0, 8.0 * min(ew, eh) / 256))
        if case["mask"] and i == case["n_ex"] - 1:
            m = np.full((eh, ew, 4), 255, np.uint8)
            m[: eh // 3, : ew // 2, :3] = 0  # a corner that must not be copied from
            e["sample"], e["mask"] = "image", m
        spec["examples"].append(e)
    if case["guide"] != "none":
        spec["target_guide"] = wl.target_guide(base + 15, h, w)
    if case["inpaint"]:
        rng = np.random.default_rng(base + 14)
        mask = np.full((h, w, 4), 255, np.uint8)
        n = int(rng.integers(1, 6))
        a = rng.uniform(0.10, 0.40) * w * h / n
        for _ in range(n):
            rw = int(np.clip(math.sqrt(a) * rng.uniform(0.6, 1.6), 2, w))
            rh = int(np.clip(a / rw, 2, h))
            x0, y0 = int(rng.integers(0, w - rw + 1)), int(rng.integers(0, h - rh + 1))
            mask[y0:y0 + rh, x0:x0 + rw, :3] = 0
        spec["inpaint_mask"], spec["inpaint_index"] = mask, 0
    return spec


def _mix_shapes(n, side_max):
    """Sizes and settings of the batched mix: example sides 64-512, output
    sides 128 (or half the largest) to side_max, both log-uniform, k and m
    from {8, 20, 50}, a quarter guided."""
    rng = random.Random(3)
    out = []
    for i in range(n):
        es, side = _logi(rng, 64, 512), _logi(rng, min(128, side_max // 2), side_max)
        out.append((es, side, rng.choice([8, 20, 50]), rng.choice([8, 20, 50]), i % 4 == 3))
    return out


def _mix_specs(n, side_max, seed):
    specs = []
    for i, (es, side, k, m, guided) in enumerate(_mix_shapes(n, side_max)):
        c = _session("", side, side, es, es, k=k, m=m, guide="given" if guided else "none")
        specs.append(_session_spec(c, 1000 * seed + i))
    return specs


def _serve_shapes(n, side_max):
    """Request i of a burst: an inpainting picture (3 of 10) or a job of the mix."""
    mix = _mix_shapes(n, side_max)
    return [("inpaint", side_max) if i % 10 in (2, 5, 8) else ("mix", mix[i]) for i in range(n)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "session":
        return {"case": case, "spec": _session_spec(case, seed)}
    if kind == "batch":
        return {"case": case, "specs": _mix_specs(case["n"], case["side_max"], seed)}
    if kind == "serve":
        specs = []
        for i, (what, shape) in enumerate(_serve_shapes(case["n"], case["side_max"])):
            if what == "inpaint":
                c = _session("", shape, shape, shape, shape, inpaint=True)
            else:
                es, side, k, m, guided = shape
                c = _session("", side, side, es, es, k=k, m=m, guide="given" if guided else "none")
            specs.append(_session_spec(c, 1000 * seed + i))
        return {"case": case, "specs": specs, "server": ts.Server()}
    # apply: a transform as its file holds it (u32 words: magic, sizes, then
    # x, y, map per pixel), patches of neighbouring source texels as a
    # synthesis leaves them
    rng = np.random.default_rng(seed)
    w, h, ew, eh, n = case["w"], case["h"], case["ex_w"], case["ex_h"], case["n_ex"]
    p = 8  # patch side
    ph, pw = -(-h // p), -(-w // p)

    def spread(v):
        return np.kron(v, np.ones((p, p), np.int64))[:h, :w]

    yy, xx = np.mgrid[0:h, 0:w]
    xym = np.empty((h, w, 3), np.uint32)
    xym[..., 0] = (spread(rng.integers(0, ew, (ph, pw))) + xx % p) % ew
    xym[..., 1] = (spread(rng.integers(0, eh, (ph, pw))) + yy % p) % eh
    xym[..., 2] = spread(rng.integers(0, n, (ph, pw)))
    words = np.concatenate([np.array([0x12340001, w, h, n] + [ew, eh] * n, np.uint32), xym.reshape(-1)])
    sw, sh = max(1, int(ew * case["scale"])), max(1, int(eh * case["scale"]))
    return {"case": case, "transform": ts.CoordinateTransform.read(words.astype("<u4").tobytes()),
            "sources": [wl.texture(16 * seed + i, sh, sw) for i in range(n)]}


def run(state):
    kind = state["case"]["kind"]
    if kind == "session":
        g = ts.builder_from_spec(state["spec"]).build().run()
        if not state["case"]["maps"]:
            return {"image": g.into_image()}
        flat, score = g.resolved()
        return {"image": g.into_image(), "coord": g.coord_map(), "id": g.id_map(), "resolved": flat, "score": score}
    if kind == "batch":
        b = ts.Batch()
        for spec in state["specs"]:
            b.add(ts.builder_from_spec(spec).build())
        return [g.into_image() for g in b.run()]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(ts.builder_from_spec(spec).build()) for spec in state["specs"]]
        return [server.wait(t)[0].into_image() for t in tickets]
    return {"image": state["transform"].apply(state["sources"])}


def _session_work(w, h, ex_px, n_ex, k, m, guided, fill=1.0, maps=False):
    """Inputs read and outputs written once; the cost sums that cannot be
    left out: per item the winner's k terms and one term of each other
    candidate, a term being 4 differences, 4 table terms, a product and a sum
    (twice the differences and terms with a guide).  Items: stage s of 5..0
    resolves half of stage s - 1's pixels anew and again what it redoes."""
    n = w * h
    items = sum(int(0.5 ** s * n * fill) for s in range(6))
    inputs = 4 * (n_ex * ex_px * (2 if guided else 1) + (n if guided else 0))
    outputs = 4 * n + (4 * n * 7 if maps else 0)
    per_term = 18 if guided else 10
    return {"bytes": float(inputs + outputs), "flops": float(items * (2 * k + m) * per_term)}


def work(case):
    kind = case["kind"]
    if kind == "session":
        w, h = case["w"], case["h"]
        ex_px = w * h if case["inpaint"] else case["ex_w"] * case["ex_h"]
        return _session_work(w, h, ex_px, case["n_ex"], case["k"], case["m"], case["guide"] != "none",
                             0.25 if case["inpaint"] else 1.0, case["maps"])
    total = {"bytes": 0.0, "flops": 0.0}
    if kind == "apply":
        sources = case["n_ex"] * int(case["ex_w"] * case["scale"]) * int(case["ex_h"] * case["scale"])
        return {"bytes": float(case["w"] * case["h"] * 16 + 4 * sources), "flops": 0.0}
    if kind == "batch":
        parts = [("mix", s) for s in _mix_shapes(case["n"], case["side_max"])]
    else:
        parts = _serve_shapes(case["n"], case["side_max"])
    for what, s in parts:
        if what == "inpaint":
            one = _session_work(s, s, s * s, 1, 50, 50, False, 0.25)
        else:
            one = _session_work(s[1], s[1], s[0] * s[0], 1, s[2], s[3], s[4])
        total = {q: total[q] + one[q] for q in total}
    return total


def exact(case, seed):
    """No value: images and maps are bytes and whole numbers, and the scores
    are sums over the candidates that the whole seeded synthesis picks, which
    takes minutes in plain numpy."""
    return None
