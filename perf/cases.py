"""The work that programs have this renderer do, as cases that a timing harness can prepare and run.

A case is a dict of plain values; `kind` says which entry points it goes through:

  scan     exclusive_scan_i32 on device memory (the reference's standalone scan kernel)
  frame    one ScanlineVGRasterizer frame of a resident scene into a device framebuffer
  reload   loadVG of a scene, then a frame into pinned host memory: a scene that changes every frame
  view     setMVP, then a frame of a resident RVG file: zooming and turning a drawing
  aa       an antialiased frame (render_aa) into pinned host memory
  batch    many uneven scenes in one resident SceneBatch, replayed as a captured graph
  serve    requests submitted together to a RenderServer, and waited for
  predict  the sizing network's inference over paths
  train    the sizing network fitted from a given state
"""
import lzma
import math
import os
import tempfile

import numpy as np
import torch

import vkscanlinepr_gb300 as sr

HERE = os.path.dirname(os.path.abspath(__file__))
RVG_DIR = os.path.join(os.path.dirname(HERE), "tests", "golden", "rvg")
RVG_NAMES = ["car", "chord", "chord-black", "drops", "embrace", "reschart", "test", "tiger"]
LR, BETA1, BETA2, EPS = 1e-3, 0.9, 0.999, 1e-8


def listed():
    return [
        # a short scan: what a caller pays for a call that has almost no work
        dict(name="scan-10007", kind="scan", n=10007),
        # a scan of tens of millions of counts: bandwidth
        dict(name="scan-50m", kind="scan", n=50000017),
        # the small configuration: 500 star paths of cubics at 1024 x 1024
        dict(name="frame-star-1024", kind="frame", preset=0, width=1024, height=1024, paths=500, mode=1),
        # the configuration at scale: 20,000 mixed paths at 4096 x 4096
        dict(name="frame-mixed-4096", kind="frame", preset=1, width=4096, height=4096, paths=20000, mode=1),
        # the reference's own look (2-pixel cells, no blending) on a ragged canvas
        dict(name="frame-reference-1000x750", kind="frame", preset=1, width=1000, height=750, paths=1200, mode=0),
        # a scene that is new every frame, host to host
        dict(name="reload-mixed-2048", kind="reload", preset=1, width=2048, height=2048, paths=5000, mode=1),
        # a drawing from an RVG file under a new matrix every frame
        dict(name="view-tiger-900", kind="view", file="tiger", full=False, side=900, mode=1),
        # four samples a pixel
        dict(name="aa4-star-1024", kind="aa", preset=0, width=1024, height=1024, paths=500, samples=4),
        # a resident batch of uneven scenes (sides 256 to 2048, 10 to some thousands of paths)
        dict(name="batch-64", kind="batch", scenes=64, mode=1),
        # a burst of requests at the server
        dict(name="serve-16", kind="serve", requests=16),
        # sizing a batch's paths, and fitting the network that does it
        dict(name="predict-200k", kind="predict", n=200003),
        dict(name="train-32k", kind="train", n=32768, batch=4096, epochs=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    s = _log_int(rng, lo, hi)
    return s + 1 if s % 2 == 0 and s < hi and rng.random() < 0.5 else s


def draw(rng):
    kind = rng.choice(["scan", "frame", "frame", "frame", "reload", "view", "aa", "batch", "serve", "predict", "train"])
    if kind == "scan":
        return dict(kind=kind, n=_log_int(rng, 1, 50000017))
    if kind in ("frame", "reload"):
        top = 4096 if kind == "frame" else 2048
        w, h = _side(rng, 96, top), _side(rng, 96, top)
        most = min(20000 if kind == "frame" else 5000, w * h // 200)   # four times the listed ones' density
        return dict(kind=kind, preset=rng.randint(0, 1), width=w, height=h, paths=_log_int(rng, 10, most),
                    mode=rng.choice([0, 1, 1]))
    if kind == "view":
        return dict(kind=kind, file=rng.choice(RVG_NAMES), full=rng.random() < 0.5, side=_side(rng, 200, 1800),
                    mode=rng.choice([0, 1, 1]))
    if kind == "aa":
        samples = rng.choice([2, 4, 8, 16])
        return dict(kind=kind, preset=rng.randint(0, 1), width=_side(rng, 96, 1024), height=_side(rng, 96, 1024),
                    paths=_log_int(rng, 10, 2000 // samples), samples=samples)
    if kind == "batch":
        return dict(kind=kind, scenes=_log_int(rng, 2, 64), mode=rng.choice([0, 1, 1]))
    if kind == "serve":
        return dict(kind=kind, requests=_log_int(rng, 1, 16))
    if kind == "predict":
        return dict(kind=kind, n=_log_int(rng, 10, 200003))
    return dict(kind=kind, n=_log_int(rng, 500, 32768), batch=rng.choice([512, 1024, 4096]), epochs=rng.randint(1, 2))


# ------------------------------------------------------------ inputs -----

def _scene(case, seed):
    return sr.synth_scene(case["preset"], seed, width=case["width"], height=case["height"], n_paths=case["paths"])


def _shapes(count):
    """Sides and path counts of `count` uneven scenes, the same for every seed: sides uniform over 256 to 2048, paths
    lognormal around 200."""
    rng = np.random.RandomState(20)
    return [(int(rng.choice([256, 512, 1024, 2048])), int(min(max(200 * math.exp(rng.randn()), 10), 20000)))
            for _ in range(count)]


def _uneven_scenes(count, seed):
    return [sr.synth_scene(1, seed, scene_index=i, width=side, height=side, n_paths=paths)
            for i, (side, paths) in enumerate(_shapes(count))]


def _rasterizer(mode, w, h):
    r = sr.ScanlineVGRasterizer(mode=sr.MODE_PIXEL if mode else sr.MODE_REFERENCE)
    r.initialize(None, w, h)
    return r


def _image(w, h):
    return torch.empty((h, w, 4), dtype=torch.uint8, device="cuda")


def _pinned(w, h):
    """Page-locked host memory for a frame (the array keeps it alive)."""
    return torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True).numpy()


def _load_rvg(name, full):
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, name + ".rvg")
        with lzma.open(os.path.join(RVG_DIR, name + ".rvg.xz"), "rb") as f, open(path, "wb") as g:
            g.write(f.read())
        return sr.load_rvg(path, full=full)


def _views(viewport, side, rng):
    """Matrices that fit the drawing to the canvas, turned and zoomed a little more from one to the next."""
    x, y, w, h = (float(v) for v in viewport)
    fit = side / max(w, h, 1.0)
    turn, zoom = rng.uniform(-0.5, 0.5), fit * math.exp(rng.uniform(-0.3, 0.7))
    out = []
    for k in range(4):
        c, s = zoom * math.cos(turn + 0.01 * k), zoom * math.sin(turn + 0.01 * k)
        cx, cy = x + w / 2, y + h / 2
        out.append(np.array([c, -s, 0, side / 2 - c * cx + s * cy,
                             s, c, 0, side / 2 - s * cx - c * cy,
                             0, 0, 1, 0, 0, 0, 0, 1], np.float32))
    return out


def _paths(n, seed):
    """Features and labels as the batch scenes' paths have them: geometric segment counts, lognormal extents,
    labels that mostly follow the control polygon's length."""
    rng = np.random.RandomState(seed % (1 << 32))
    segs = rng.geometric(1 / 12.0, n).clip(1, 256)
    r = np.exp(math.log(40.0) + rng.randn(n)).clip(1, 1024)
    bw, bh = 2 * r * rng.uniform(0.5, 1.0, n), 2 * r * rng.uniform(0.5, 1.0, n)
    length = r * np.sqrt(segs) * rng.uniform(2.0, 4.0, n)
    turn = segs * rng.uniform(0.2, 0.6, n)
    x = np.stack([np.log1p(segs), np.log1p(bw), np.log1p(bh), np.log1p(length), np.log1p(turn),
                  rng.binomial(segs, 0.6) / segs], 1)
    records = 1.3 * length + 3 * segs
    t = np.stack([np.log1p(records * np.exp(0.15 * rng.randn(n))),
                  np.log1p(0.7 * records * np.exp(0.25 * rng.randn(n)))], 1)
    return x.astype(np.float32), t.astype(np.float32)


def _sizer(x, t, seed):
    sz = sr.Sizer(seed=seed)
    sz.set_norm(sr.sizer_norm(x, t))
    return sz


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scan":
        g = torch.Generator(device="cuda").manual_seed(seed)
        d_in = torch.randint(0, 40, (case["n"],), dtype=torch.int32, device="cuda", generator=g)
        return dict(kind=kind, n=case["n"], d_in=d_in, out=torch.empty(case["n"] + 1, dtype=torch.int32, device="cuda"))
    if kind == "frame":
        r = _rasterizer(case["mode"], case["width"], case["height"])
        r.loadVG(_scene(case, seed))
        return dict(kind=kind, r=r, out=_image(case["width"], case["height"]))
    if kind == "reload":
        return dict(kind=kind, r=_rasterizer(case["mode"], case["width"], case["height"]), scene=_scene(case, seed),
                    out=_pinned(case["width"], case["height"]))
    if kind == "view":
        scene, viewport = _load_rvg(case["file"], case["full"])
        r = _rasterizer(case["mode"], case["side"], case["side"])
        r.loadVG(scene)
        return dict(kind=kind, r=r, views=_views(viewport, case["side"], np.random.RandomState(seed % (1 << 32))),
                    out=[_image(case["side"], case["side"]) for _ in range(4)])
    if kind == "aa":
        r = _rasterizer(1, case["width"], case["height"])
        r.loadVG(_scene(case, seed))
        return dict(kind=kind, r=r, samples=case["samples"], out=_pinned(case["width"], case["height"]))
    if kind == "batch":
        b = sr.SceneBatch(mode=sr.MODE_PIXEL if case["mode"] else sr.MODE_REFERENCE)
        for scene in _uneven_scenes(case["scenes"], seed):
            b.add_scene(scene)
        b.commit()
        b.render()   # exact sizing, once: the capacity that the resident batch is replayed with
        sizes = [b.size(i) for i in range(case["scenes"])]
        return dict(kind=kind, b=b, capacity=b.stats()["record_capacity"], sizes=sizes,
                    out=torch.empty(sum(w * h for w, h in sizes) * 4, dtype=torch.uint8, device="cuda"))
    if kind == "serve":
        return dict(kind=kind, scenes=_uneven_scenes(case["requests"], seed),
                    srv=sr.RenderServer(slots=2, max_batch_scenes=64, memory_budget=40e9))
    x, t = _paths(case["n"], seed)
    sz = _sizer(x, t, seed)
    if kind == "predict":
        return dict(kind=kind, sz=sz, x=torch.from_numpy(x).cuda(), n=case["n"],
                    y=torch.empty((case["n"], 2), dtype=torch.float32, device="cuda"))
    return dict(kind=kind, sz=sz, state=sz.state(), x=sr.DeviceArray.from_numpy(x), t=sr.DeviceArray.from_numpy(t),
                batch=case["batch"], epochs=case["epochs"])


def run(state):
    kind = state["kind"]
    if kind == "scan":
        sr.exclusive_scan_i32(state["d_in"].data_ptr(), state["out"].data_ptr(), state["n"])
        return state["out"]
    if kind == "frame":
        state["r"].render_device(state["out"].data_ptr())
        return state["out"]
    if kind == "reload":
        state["r"].loadVG(state["scene"])
        return state["r"].render(out=state["out"])
    if kind == "view":
        for m, out in zip(state["views"], state["out"]):
            state["r"].setMVP(m)
            state["r"].render_device(out.data_ptr())
        return state["out"]
    if kind == "aa":
        return state["r"].render_aa(state["samples"], out=state["out"])
    if kind == "batch":
        state["b"].render(capacity=state["capacity"], graph=True)
        at, get = state["out"].data_ptr(), sr.lib().sr_batch_get_image
        for i, (w, h) in enumerate(state["sizes"]):
            if get(state["b"]._h, i, at, 1, None) != 0:
                raise RuntimeError("sr_batch_get_image failed")
            at += w * h * 4
        return state["out"]
    if kind == "serve":
        tickets = [state["srv"].submit(s) for s in state["scenes"]]
        return [state["srv"].wait(t)[0] for t in tickets]
    if kind == "predict":
        if sr.lib().sr_sizer_predict(state["sz"]._h, state["x"].data_ptr(), state["n"], state["y"].data_ptr(), None):
            raise RuntimeError("sr_sizer_predict failed")
        return state["y"]
    sz = state["sz"]
    sz.load_state(state["state"])
    loss = sz.train(state["x"], state["t"], epochs=state["epochs"], batch=state["batch"], lr=LR, seed=7,
                    beta1=BETA1, beta2=BETA2, eps=EPS)
    st = sz.state()
    return dict(loss=loss, params=st["params"], adam_m=st["adam_m"], adam_v=st["adam_v"])


# ------------------------------------------------------------- work ------

def _scene_bytes(preset, paths):
    """A scene's arrays: 12 bytes a point, 12 a curve, 8 a path, at the generator's mean segments a path and points a
    segment (preset 0: 10 cubics; the mixed one: 12 segments, 60% cubic, 30% quadric, 10% line)."""
    segs, pts = (10, 4.0) if preset == 0 else (12, 3.5)
    return paths * (8 + segs * (12 + 12 * pts))


def work(case):
    kind = case["kind"]
    if kind == "scan":
        return dict(bytes=8 * case["n"], flops=0)
    if kind in ("frame", "reload"):
        return dict(bytes=_scene_bytes(case["preset"], case["paths"]) + 4 * case["width"] * case["height"], flops=0)
    if kind == "aa":
        return dict(bytes=_scene_bytes(case["preset"], case["paths"]) + 4 * case["width"] * case["height"], flops=0)
    if kind == "view":
        return dict(bytes=4 * 4 * case["side"] * case["side"], flops=0)
    if kind in ("batch", "serve"):
        n = case["scenes"] if kind == "batch" else case["requests"]
        return dict(bytes=sum(_scene_bytes(1, paths) + 4 * side * side for side, paths in _shapes(n)), flops=0)
    mac = 6 * 64 + 64 * 64 + 64 * 2
    if kind == "predict":
        return dict(bytes=32 * case["n"], flops=2 * mac * case["n"])
    # forward, and in the backward each layer's weight gradient and the upper two layers' input gradients
    return dict(bytes=32 * case["n"] * case["epochs"], flops=2 * (3 * mac - 6 * 64) * case["n"] * case["epochs"])


# ------------------------------------------------------------ 64 bits ----

def _bf16(w):
    """Nearest bfloat16 (ties to even) of float32-rounded values, as float64."""
    u = np.asarray(w, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) >> 16 << 16
    return u.astype(np.uint32).view(np.float32).astype(np.float64)


def _erf(x):
    return torch.erf(torch.from_numpy(x)).numpy()


def _unpack(p):
    """W1, b1, W2, b2, W3, b3 of a packed parameter vector; weights as the network uses them (bfloat16)."""
    o = np.cumsum([0, 384, 64, 4096, 64, 128, 2])
    w1, b1, w2, b2, w3, b3 = (p[a:b] for a, b in zip(o[:-1], o[1:]))
    return _bf16(w1).reshape(64, 6), b1, _bf16(w2).reshape(64, 64), b2, _bf16(w3).reshape(2, 64), b3


def _forward(p, norm, x):
    w1, b1, w2, b2, w3, b3 = _unpack(p)
    z = (x.astype(np.float64) - norm[:6]) * norm[6:12]
    a1 = z @ w1.T + b1
    c1 = 0.5 * (1 + _erf(a1 * math.sqrt(0.5)))
    h1 = a1 * c1
    a2 = h1 @ w2.T + b2
    c2 = 0.5 * (1 + _erf(a2 * math.sqrt(0.5)))
    h2 = a2 * c2
    return z, a1, c1, h1, a2, c2, h2, h2 @ w3.T + b3


def _gradient(p, norm, x, t):
    """Gradient of the mean squared error in standard units, and the sum of squared errors."""
    _, _, w2, _, w3, _ = _unpack(p)
    z, a1, c1, h1, a2, c2, h2, y = _forward(p, norm, x)
    e = y - (t.astype(np.float64) - norm[12:14]) / norm[14:16]
    dy = e / len(x)   # 2 / (samples * 2 outputs)
    pdf = lambda a: np.exp(-0.5 * a * a) / math.sqrt(2 * math.pi)  # noqa: E731
    d2 = (dy @ w3) * (c2 + a2 * pdf(a2))
    d1 = (d2 @ w2) * (c1 + a1 * pdf(a1))
    g = [d1.T @ z, d1.sum(0), d2.T @ h1, d2.sum(0), dy.T @ h2, dy.sum(0)]
    return np.concatenate([v.reshape(-1) for v in g]), float((e * e).sum())


def _order(n, seed):
    """The epoch's sample order: rows sorted by a splitmix64 hash of (seed, row)."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, n + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = (z ^ (z >> np.uint64(31))) >> np.uint64(32)
    return np.argsort(z, kind="stable")


def exact(case, seed):
    """The sizing network's results in 64 bits; the other cases' outputs are whole numbers."""
    if case["kind"] not in ("predict", "train"):
        return None
    x, t = _paths(case["n"], seed)
    sz = _sizer(x, t, seed)
    st = sz.state()
    sz.close()
    norm = st["norm"].astype(np.float64)
    p = st["params"].astype(np.float64)
    if case["kind"] == "predict":
        return _forward(p, norm, x)[-1] * norm[14:16] + norm[12:14]
    m, v, step = np.zeros_like(p), np.zeros_like(p), 0
    for epoch in range(case["epochs"]):
        order = _order(case["n"], (7 * 0x100000001B3 + epoch) % (1 << 64))
        loss = 0.0
        for at in range(0, case["n"], case["batch"]):
            rows = order[at:at + case["batch"]]
            g, sse = _gradient(p, norm, x[rows], t[rows])
            loss += sse
            step += 1
            m = BETA1 * m + (1 - BETA1) * g
            v = BETA2 * v + (1 - BETA2) * g * g
            p = p - LR * (m / (1 - BETA1 ** step)) / (np.sqrt(v / (1 - BETA2 ** step)) + EPS)
    return dict(loss=loss / (2 * case["n"]), params=p, adam_m=m, adam_v=v)
