"""Timed cases of the PSTD solve: what a program using this package calls.

A case is a dict of plain values: the shape of a scene (its layout is fixed by
the case, speakers, receivers and edge absorptions are drawn from the seed),
the number of time steps and the entry point:

* ``advance`` -- PSTDKernel.reset / advance / receivers / snapshot;
* ``frames``  -- PSTDKernel.run, every SaveNth-th frame and the samples
  delivered to callbacks, which keep them;
* ``noalloc`` -- pstd_solve_noalloc into caller-owned device buffers;
* ``batch``   -- BatchKernel over scenes of uneven size;
* ``serve``   -- Server: submit, tick until idle, fetch results.

``exact`` solves the same scene in 64 bits with torch alone.
"""
import ctypes
import math
import random

import numpy as np
import torch

DX = 0.2
WINDOW = 32          # window of a 70 dB patch error
SOUND, DENSITY, PML_AMP, PATCH, CFL = 340.0, 1.2, 20000.0, 70.0, 0.5
RK = (1.179799016570605e-1, 1.846469664911166e-1, 2.466236043095944e-1, 3.318395427360000e-1, 5e-1, 1.0)
SIDES = ("left", "top", "right", "bottom")
f32 = np.float32


def listed():
    return [
        # a real-time loop: a room of a few metres, stepped a handful of steps per call into device
        # buffers of an application that owns the GPU's memory
        dict(name="noalloc_73", entry="noalloc", shape="rect", nx=73, ny=73, pml=40, steps=12, rigid=0, speakers=1, receivers=4),
        # interactive use: a small open field, a few steps at a time
        dict(name="interactive_200", entry="advance", shape="rect", nx=200, ny=200, pml=50, steps=8, rigid=0, speakers=1, receivers=4),
        # the standard single-domain scene, 200 x 200 cells with absorbing edges
        dict(name="square_200", entry="advance", shape="rect", nx=200, ny=200, pml=50, steps=100, rigid=0, speakers=1, receivers=4),
        # a room of odd sizes with two hard walls and a thin absorbing layer
        dict(name="room_333x187", entry="advance", shape="rect", nx=333, ny=187, pml=37, steps=100, rigid=2, speakers=2, receivers=7),
        # a floor plan: six coupled rooms of uneven, odd sizes
        dict(name="rooms_2x3", entry="advance", shape="grid", rows=2, cols=3, nx=611, ny=405, pml=50, steps=100, rigid=1, layout=4, speakers=6, receivers=8),
        # the L-shaped scene of three coupled domains, hard and absorbing edges
        dict(name="lshape_600", entry="advance", shape="lshape", nx=600, pml=50, steps=100, rigid=3, speakers=4, receivers=16),
        # a large single domain: one transform length carries the work
        dict(name="square_1200", entry="advance", shape="rect", nx=1200, ny=1200, pml=50, steps=60, rigid=0, speakers=2, receivers=8),
        # a street canyon: very long strips one way, short ones the other
        dict(name="street_5000x90", entry="advance", shape="rect", nx=5000, ny=90, pml=50, steps=60, rigid=0, speakers=2, receivers=6),
        # an animation: every second frame of an L-shaped scene delivered to the host
        dict(name="frames_lshape_300", entry="frames", shape="lshape", nx=301, pml=50, steps=60, save=2, rigid=2, speakers=3, receivers=6),
        # a parameter study: many scenes of uneven size advanced together
        dict(name="batch_96", entry="batch", scenes=96, lo=64, hi=887, pml=50, steps=40, layout=11),
        # a service: requests of uneven size and length, batched as they fit
        dict(name="serve_24", entry="serve", scenes=24, lo=64, hi=400, pml=50, steps=60, layout=5),
        # the largest scene: 8192 x 8192 cells in 2 x 2 domains
        dict(name="large_8192", entry="advance", shape="grid", rows=2, cols=2, nx=8192, ny=8192, pml=50, steps=16, rigid=0, layout=-1, speakers=4, receivers=64),
    ]


def draw(rng):
    """One more case of the same ranges, at most half the largest one's work."""
    def size(lo, hi):
        return _fit(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    entry = rng.choice(["advance", "advance", "advance", "frames", "noalloc", "batch", "serve"])
    pml = rng.choice([33, 40, 50, 50, 57])
    if entry in ("batch", "serve"):
        n = rng.randint(3, 48 if entry == "batch" else 20)
        return dict(entry=entry, scenes=n, lo=64, hi=rng.randint(200, 887 if entry == "batch" else 400), pml=pml,
                    steps=rng.randint(20, 60), layout=rng.randint(0, 1 << 20))
    if entry == "noalloc":
        return dict(entry=entry, shape="rect", nx=size(50, 240), ny=size(50, 240), pml=pml, steps=rng.randint(3, 40),
                    rigid=rng.randint(0, 2), speakers=rng.randint(1, 2), receivers=rng.randint(1, 6))
    shape = rng.choice(["rect", "rect", "grid", "lshape"])
    c = dict(entry=entry, shape=shape, pml=pml, rigid=rng.randint(0, 2), speakers=rng.randint(1, 4), receivers=rng.randint(1, 12))
    if shape == "lshape":
        c.update(nx=_fit(size(80, 1400), twice=True))
        cells = 5 * c["nx"] ** 2
    elif shape == "rect":
        c.update(nx=size(64, 7000), ny=size(64, 2500))
        if rng.random() < 0.5:
            c["nx"], c["ny"] = c["ny"], c["nx"]
        cells = c["nx"] * c["ny"]
    else:
        rows, cols = rng.choice([(1, 2), (2, 1), (2, 2), (2, 3), (3, 2), (1, 5)])
        c.update(rows=rows, cols=cols, nx=cols * size(64, 1500), ny=rows * size(64, 1500), layout=rng.randint(0, 1 << 20))
        cells = c["nx"] * c["ny"]
    most = 120 if entry == "advance" else 80
    c["steps"] = max(4, min(most, rng.randint(most // 4, most), int(4e8 / cells)))
    if entry == "frames":
        c["steps"] = max(4, min(c["steps"], int(1e8 / cells)))
        c["save"] = rng.randint(1, 8)
    return c


# ------------------------------------------------------------------ scenes as plain numbers
def _fits(n):
    """Strips of n cells have a transform length: n plus the windows is no power of two."""
    w = WINDOW
    while w > n:
        w //= 2
    m = n + 2 * w
    return m & (m - 1) != 0


def _fit(n, twice=False):
    while not (_fits(n) and (not twice or _fits(2 * n))):
        n += 1
    return n


def _parts(total, parts, layout):
    """`total` cells in `parts` strips of uneven sizes (even ones for layout < 0)."""
    if layout < 0:
        return [total // parts] * parts
    r = random.Random(layout)
    for _ in range(10000):
        least = min(40, total // parts)
        cuts = sorted(r.randint(least, total - least) for _ in range(parts - 1))
        sizes = [b - a for a, b in zip([0] + cuts, cuts + [total])]
        if all(s >= least and _fits(s) for s in sizes):
            return sizes
    return [total // parts] * (parts - 1) + [total - (parts - 1) * (total // parts)]


def _scene(shape, pml, steps, rng, speakers, receivers, rigid=0, nx=0, ny=0, rows=1, cols=1, layout=0, save=1):
    """Rectangles (x0, y0, nx, ny, {side: absorption}) in cells, and points in cells."""
    rects = []
    if shape == "lshape":
        a = nx
        rects = [(0, 0, 2 * a, a), (2 * a, 0, a, a), (2 * a, a, a, 2 * a)]
        inner = {(0, "right"), (1, "left"), (1, "bottom"), (2, "top")}
        hard = {(0, "bottom"), (2, "left")}      # the edges that meet at the concave corner
        order = [(0, "left"), (1, "right"), (0, "top"), (2, "bottom"), (2, "right"), (1, "top")]
    else:
        ws, hs = (_parts(nx, cols, layout), _parts(ny, rows, layout + 1 if layout >= 0 else layout)) if shape == "grid" else ([nx], [ny])
        xs, ys = np.concatenate([[0], np.cumsum(ws)]), np.concatenate([[0], np.cumsum(hs)])
        inner, hard, order = set(), set(), []
        for i in range(len(hs)):
            for j in range(len(ws)):
                k = len(rects)
                rects.append((int(xs[j]), int(ys[i]), ws[j], hs[i]))
                for side, outer in (("left", j == 0), ("right", j == len(ws) - 1), ("top", i == 0), ("bottom", i == len(hs) - 1)):
                    if outer:
                        order.append((k, side))
                    else:
                        inner.add((k, side))
    hard |= set(order[:rigid])
    out = []
    for k, (x0, y0, w, h) in enumerate(rects):
        e = {}
        for s in SIDES:
            alpha = float(f32(rng.uniform(0.2, 1.0)))
            e[s] = 1.0 if (k, s) in inner else 0.0 if (k, s) in hard else alpha
        out.append((x0, y0, w, h, e))
    spk = []
    for k in range(max(speakers, len(out))):      # every domain has a source
        # receivers read the cell with the offsets exchanged, so sources stand where such a cell exists
        x0, y0, w, h, _e = out[k % len(out)]
        m = min(w, h)
        spk.append((x0 + rng.randint(5, m - 6) + 0.25, y0 + rng.randint(5, m - 6) + 0.25))
    rec = []
    reach = max(2.0, 0.4 * steps)      # cells a pulse has travelled by the last third of the run
    while len(rec) < receivers:
        x, y = spk[rng.randrange(len(spk))]
        r, t = rng.uniform(0, min(reach, 60.0)), rng.uniform(0, 2 * math.pi)
        tx, ty = math.floor(x + r * math.cos(t)), math.floor(y + r * math.sin(t))
        for x0, y0, w, h, _e in out:
            if x0 < tx < x0 + w - 1 and y0 < ty < y0 + h - 1:
                gx, gy = x0 + (ty - y0), y0 + (tx - x0)
                if x0 <= gx < x0 + w and y0 <= gy < y0 + h:
                    rec.append((gx + 0.25, gy + 0.25))
                break
    return dict(rects=out, speakers=spk, receivers=rec, pml=pml, steps=steps, save=save)


def _scenes(case, seed):
    """The scenes of a case; the layout comes from the case, everything else from the seed."""
    c = {k: v for k, v in case.items() if k not in ("name", "entry")}
    rng = random.Random(seed)
    if case["entry"] not in ("batch", "serve"):
        return [_scene(rng=rng, **c)]
    lay = random.Random(c["layout"])
    got = []
    for _ in range(c["scenes"]):
        side = math.exp(lay.uniform(math.log(c["lo"]), math.log(c["hi"])))
        aspect = math.exp(lay.uniform(math.log(0.5), math.log(2.0)) / 2)
        rows, cols = lay.choice([(1, 1), (1, 2), (2, 1), (1, 3), (2, 2), (2, 3), (3, 2)])
        nx, ny = _fit(max(40 * cols, round(side * aspect))), _fit(max(40 * rows, round(side / aspect)))
        steps = c["steps"] if case["entry"] == "batch" else max(10, round(math.exp(lay.uniform(math.log(c["steps"] / 5), math.log(c["steps"])))))
        got.append(_scene("grid", c["pml"], steps, rng, lay.randint(1, 4), lay.randint(1, 8), rigid=0, nx=nx, ny=ny,
                          rows=rows, cols=cols, layout=lay.randint(0, 1 << 30)))
    return got


def _world(cells):
    """World coordinate whose float32 quotient by dx truncates to `cells`."""
    v = f32(cells * float(f32(DX)))
    while int(f32(v / f32(DX))) < cells:
        v = np.nextafter(v, f32(np.inf))
    return float(v)


def _point(p):
    return float(f32(p[0] * float(f32(DX)))), float(f32(p[1] * float(f32(DX))))


def _configuration(s):
    from openpstd_gb300.config import DomainConf, DomainConfEdge, PSTDConfiguration
    conf = PSTDConfiguration()
    t = conf.Settings
    t.SetSoundSpeed(SOUND)
    t.SetAttenuationOfPMLCells(PML_AMP)
    t.SetDensityOfAir(DENSITY)
    t.SetPatchError(PATCH)
    t.SetFactRK(CFL)
    t.SetGridSpacing(DX)
    t.SetPMLCells(s["pml"])
    t.SetSaveNth(s["save"])
    t.SetMaxFrequency(1000.0)
    q = float(f32(SOUND) / f32(DX))
    t.SetBandWidth(3e-6 * q * q)
    t.SetSpectralInterpolation(False)
    t.SetRenderTime(float(f32((s["steps"] + 0.5) * float(t.GetTimeStep()))))
    for x0, y0, nx, ny, e in s["rects"]:
        # a domain's B is its edge at small y, T the one at large y
        conf.Domains.append(DomainConf((_world(x0), _world(y0)), (_world(nx), _world(ny)), T=DomainConfEdge(e["bottom"], False),
                                       L=DomainConfEdge(e["left"], False), B=DomainConfEdge(e["top"], False), R=DomainConfEdge(e["right"], False)))
    conf.Speakers = [(*_point(p), 0.0) for p in s["speakers"]]
    conf.Receivers = [(*_point(p), 0.0) for p in s["receivers"]]
    return conf


# ------------------------------------------------------------------ entry points
def _collector():
    from openpstd_gb300.kernel import KernelCallback

    class Collect(KernelCallback):
        def __init__(self):
            self.frames, self.samples = {}, {}

        def WriteFrame(self, frame, domain, data):
            self.frames.setdefault(domain, []).append(data)

        def WriteSample(self, start, receiver, data):
            self.samples.setdefault(receiver, []).extend(data)

    return Collect


def prepare(case, seed):
    scenes = _scenes(case, seed)
    confs = [_configuration(s) for s in scenes]
    st = dict(case=case, entry=case["entry"], confs=confs, steps=[s["steps"] for s in scenes])
    if case["entry"] in ("advance", "frames"):
        from openpstd_gb300.kernel import PSTDKernel
        k = PSTDKernel()
        k.initialize_kernel(confs[0])
        st["kernel"] = k
        st["air"] = list(range(len(scenes[0]["rects"])))
        if case["entry"] == "frames":
            st["collect"] = _collector()
    elif case["entry"] == "batch":
        from openpstd_gb300.batch import BatchKernel
        st["kernel"] = BatchKernel(confs)
        st["air"] = [len(s["rects"]) for s in scenes]
    elif case["entry"] == "serve":
        from openpstd_gb300.serving import Server
        st["server"] = Server(4 << 30, max_scenes=64)
    else:
        from openpstd_gb300 import _lib
        from openpstd_gb300.config import CConfig
        st["lib"], st["config"] = _lib, CConfig(confs[0])
        s = scenes[0]
        st["frame"] = torch.zeros(sum(r[2] * r[3] for r in s["rects"]), dtype=torch.float32, device="cuda")
        st["samples"] = torch.zeros((s["steps"], len(s["receivers"])), dtype=torch.float32, device="cuda")
    return st


def run(st):
    e, n = st["entry"], st["steps"][0]
    if e == "advance":
        k = st["kernel"]
        k.reset()
        k.advance(n)
        return {"receivers": k.receivers(), "p0": [k.snapshot(i, "p0") for i in st["air"]]}
    if e == "frames":
        k, c = st["kernel"], st["collect"]()
        k.reset()
        k.run(c)
        return {"frames": [np.stack(c.frames[d]) for d in sorted(c.frames)], "samples": np.array([c.samples[r] for r in sorted(c.samples)], dtype=np.float32)}
    if e == "batch":
        k = st["kernel"]
        k.reset()
        k.advance(n)
        return {"receivers": k.receivers(),
                "p0": np.concatenate([k.scene_snapshot(s, d, "p0").ravel() for s, m in enumerate(st["air"]) for d in range(m)])}
    if e == "serve":
        srv = st["server"]
        ids = [srv.submit(c, m, final_frame=True) for c, m in zip(st["confs"], st["steps"])]
        srv.run_until_idle()
        got = [srv.result(i) for i in ids]
        return {"receivers": np.concatenate([r.ravel() for r, _ in got]), "p0": np.concatenate([f for _, f in got])}
    lib, f, r = st["lib"], st["frame"], st["samples"]
    lib.check(lib.lib().pstd_solve_noalloc(ctypes.byref(st["config"].c), n, ctypes.c_void_p(f.data_ptr()), f.numel(),
                                           ctypes.c_void_p(r.data_ptr()), r.numel(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"frame": f, "samples": r}


# ------------------------------------------------------------------ the scene in 64 bits
class _Dom:
    def __init__(self, alpha, x0, y0, nx, ny, parent=None, edges=None):
        alpha = float(f32(alpha))
        r = math.sqrt(1.0 - alpha)
        self.alpha, self.x0, self.y0, self.nx, self.ny, self.edges = alpha, x0, y0, nx, ny, edges
        z = -((r + 1) / (r - 1)) if r != 1.0 else math.inf
        self.rigid = z > 1000
        self.rho = 1e30 if self.rigid else float(f32(DENSITY)) * z
        self.parents = [parent] if parent is not None else []
        self.pml = parent is not None
        self.corner = self.pml and parent.pml
        self.nb = {s: [] for s in SIDES}

    def span(self, side):
        return (self.y0, self.y0 + self.ny) if side in ("left", "right") else (self.x0, self.x0 + self.nx)


_OPPOSITE = {"left": "right", "right": "left", "top": "bottom", "bottom": "top"}


def _knows(a, b):
    return any(b in v for v in a.nb.values())


def _join(order, n):
    """Add a domain and link it with the domains whose edges it shares."""
    for e in order:
        if n.corner and e.corner or (n.corner and not e.pml) or (e.corner and not n.pml):
            continue
        if n.pml and e.pml and not (n.corner and e in n.parents) and not (e.corner and n in e.parents):
            if len(e.parents) != 1 or len(n.parents) != 1 or not _knows(e.parents[0], n.parents[0]) or not _knows(n.parents[0], e.parents[0]):
                continue
        if n.x0 + n.nx == e.x0:
            side = "right"
        elif n.x0 == e.x0 + e.nx:
            side = "left"
        elif n.y0 + n.ny == e.y0:
            side = "bottom"
        elif n.y0 == e.y0 + e.ny:
            side = "top"
        else:
            continue
        if (e.pml and not n.pml and n not in e.parents) or (n.pml and not e.pml and e not in n.parents):
            continue
        (a0, a1), (b0, b1) = n.span(side), e.span(side)
        if min(a1, b1) <= max(a0, b0):
            continue
        n.nb[side].append(e)
        e.nb[_OPPOSITE[side]].append(n)
    order.append(n)


def _domains(s):
    """The scene's domains with their absorbing layers, in the order they are added."""
    order, P = [], s["pml"]
    air = [_Dom(1.0, *r[:4], edges=r[4]) for r in s["rects"]]
    for d in air:
        _join(order, d)
    first, corners = [], []
    for d in air:
        for i, side in enumerate(SIDES):
            if d.nb[side]:
                continue
            alpha = d.edges[side]
            x0, y0, nx, ny = {"left": (d.x0 - P, d.y0, P, d.ny), "right": (d.x0 + d.nx, d.y0, P, d.ny),
                              "top": (d.x0, d.y0 - P, d.nx, P), "bottom": (d.x0, d.y0 + d.ny, d.nx, P)}[side]
            p = _Dom(max(alpha, 1e-5), x0, y0, nx, ny, d)
            first.append(p)
            if alpha <= 0:
                continue
            for second in (SIDES[(i + 1) % 4], SIDES[(i + 3) % 4]):
                cx, cy = {"left": (p.x0 - P, p.y0), "right": (p.x0 + p.nx, p.y0), "top": (p.x0, p.y0 - P), "bottom": (p.x0, p.y0 + p.ny)}[second]
                corners.append((_Dom(min(max(1e-5, d.edges[second]), max(1e-5, alpha)), cx, cy, P, P, p), second))
    for p in first:
        _join(order, p)
    at = {}
    for c, second in corners:
        if not c.parents[0].nb[second]:
            at.setdefault((c.x0, c.y0), []).append(c)
    for key in sorted(at):
        kept = []
        for c in at[key]:
            twin = [k for k in kept if k.parents[0].parents[0] is c.parents[0].parents[0]]
            if twin:
                twin[0].parents.append(c.parents[0])
            else:
                kept.append(c)
        for c in kept:
            _join(order, c)
    return order


def _attenuation(d, s, vel):
    """Factors along x and y of a layer (ones where it does not attenuate)."""
    has = {k: bool(v) for k, v in d.nb.items()}
    plain = {k: has[k] and not any(q.pml for q in d.nb[k]) for k in SIDES}
    if d.corner:
        both = sum(len(v) for v in d.nb.values()) == 2
        horizontal = has["left"] or has["right"]
        ax = (has["left"] if both else has["left"] or has["bottom"]) if horizontal else None
        ay = has["bottom"] if both else None if horizontal else has["left"] or has["bottom"]
    else:
        horizontal = plain["left"] or plain["right"]
        up = plain["left"] or plain["bottom"]
        ax, ay = (up, None) if horizontal else (None, up)
    P = s["pml"]
    dt = float(f32(f32(f32(CFL) * f32(DX)) / f32(SOUND)))
    rho, amp = float(f32(DENSITY)), float(f32(PML_AMP))
    i = np.arange(P + 1) / P if vel else (np.arange(P) + 0.5) / P
    prof = np.exp(-(rho if vel else 1 / rho) * amp * i ** 4 * dt)
    return [None if a is None else (prof if a else prof[::-1].copy()) for a in (ax, ay)]


def _strips(s, d, horizontal):
    """Length, window, transform length and the two neighbours of a domain's strips along x or y."""
    n = d.nx if horizontal else d.ny
    w = WINDOW
    while w > n:
        w //= 2
    L = 1
    while L < n + 2 * w:
        L *= 2
    low, high = (d.nb["left"], d.nb["right"]) if horizontal else (d.nb["bottom"], d.nb["top"])
    return n, w, L, low, high


def _solve64(s, keep=None):
    """Receivers (steps x receivers) and final p0 of every air domain, in 64 bits."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    T = dict(dtype=torch.float64, device=dev)
    doms = _domains(s)
    dx, c1 = float(f32(DX)), float(f32(SOUND))
    dt = float(f32(f32(f32(CFL) * f32(DX)) / f32(SOUND)))
    q = float(f32(SOUND) / f32(DX))
    band = float(f32(3e-6 * q * q))
    for d in doms:
        x, y = torch.arange(d.nx, **T)[None, :], torch.arange(d.ny, **T)[:, None]
        d.px, d.py, d.p0 = (torch.zeros(d.ny, d.nx, **T) for _ in range(3))
        d.vx, d.vy = torch.zeros(d.ny, d.nx + 1, **T), torch.zeros(d.ny + 1, d.nx, **T)
        for p in s["speakers"]:
            gx, gy = (f32(f32(f32(v) / f32(DX)) - f32(0.5)) for v in _point(p))
            rx, ry = float(f32(gx - f32(d.x0))) - x, float(f32(gy - f32(d.y0))) - y
            pr = torch.exp(-band * (rx * dx * rx * dx + ry * dx * ry * dx))
            a = torch.atan2(rx.expand_as(pr), ry.expand_as(pr))
            d.p0 += pr
            d.px += torch.cos(a) ** 2 * pr
            d.py += torch.sin(a) ** 2 * pr
    recs = []
    for p in s["receivers"]:
        gx, gy = (int(f32(f32(v) / f32(DX))) for v in _point(p))
        d = [d for d in doms if not d.pml and d.x0 <= gx <= d.x0 + d.nx and d.y0 <= gy <= d.y0 + d.ny][-1]
        recs.append((d, gx - d.x0, gy - d.y0))
    tables = {}

    def plan(d, horizontal):
        n, w, L, low, high = _strips(s, d, horizontal)
        if max(len(low), len(high)) > 1:
            raise ValueError("a side with several neighbours")
        if (w, L) not in tables:
            x = torch.arange(-w, w + 1, **T) / w
            win = torch.exp(-math.log(10.0) * ((int(PATCH) - 40) / 20.0 + 1) * x ** 6)
            k = torch.arange(L // 2 + 1, **T) * (math.pi / dx / (L // 2))
            fac = []
            for sg in (-0.5, 0.5):
                f = torch.exp(torch.complex(torch.zeros_like(k), sg * k * dx)) * torch.complex(torch.zeros_like(k), k)
                f[-1] = float(f[-1].real)
                fac.append(f)
            tables[w, L] = win, fac
        d1, d2 = (low[0] if low else None), (high[0] if high else None)
        return (n, w, L, d1, d2) + tables[w, L]

    live = [d for d in doms if not d.rigid]
    plans = {(d, h): plan(d, h) for d in live for h in (True, False)}

    def derive(d, h, vel):
        n, w, L, d1, d2, win, fac = plans[d, h]
        pick = (lambda q: q.vx if h else q.vy.T) if vel else (lambda q: q.p0 if h else q.p0.T)
        own, e = pick(d), 1 if vel else 0
        n += e
        buf = torch.zeros(own.shape[0], L, **T)
        buf[:, w:w + n] = own
        for q, lo in ((d1, True), (d2, False)):
            if q is None:
                continue
            z = q.rho / d.rho
            R, t = (z - 1) / (z + 1), 2 * z / (z + 1) if vel else 2 / (1 + z)
            if vel:
                R = -R
            far, a = pick(q), own
            off, base = (q.y0 - d.y0, d.ny) if h else (q.x0 - d.x0, d.nx)
            far = far[-off:base - off]
            if lo:
                buf[:, :w] = (far[:, far.shape[1] - w - e:far.shape[1] - e] * t + a[:, e:w + e].flip(1) * R) * win[:w]
            else:
                buf[:, w + n:2 * w + n] = (far[:, e:w + e] * t + a[:, n - w - e:n - e].flip(1) * R) * win[w + 1:]
        out = torch.fft.irfft(torch.fft.rfft(buf) * fac[e], n=L)[:, w:w + (n - 1 if vel else n + 1)]
        return out if h else out.T

    att = {d: [[None if a is None else torch.tensor(a, **T) for a in _attenuation(d, s, v)] for v in (False, True)] for d in doms if d.pml}
    out = []
    for step in range(s["steps"]):
        was = {d: (d.px, d.py, d.vx, d.vy) for d in live}
        for rk in RK:
            cd = dt * float(f32(rk))
            new = {}
            for d in live:
                px, py, vx, vy = was[d]
                g = d.rho * c1 * c1
                new[d] = (px - cd * g * derive(d, True, True), py - cd * g * derive(d, False, True),
                          vx - cd / d.rho * derive(d, True, False), vy - cd / d.rho * derive(d, False, False))
            for d in live:
                d.px, d.py, d.vx, d.vy = new[d]
            for d in doms:
                d.p0 = d.px + d.py
        if keep is not None:
            keep(step, [d for d in doms if not d.pml])
        for d, ((px, py), (vx, vy)) in att.items():
            d.px = d.px if px is None else d.px * px
            d.vx = d.vx if vx is None else d.vx * vx
            d.py = d.py if py is None else d.py * py[:, None]
            d.vy = d.vy if vy is None else d.vy * vy[:, None]
        out.append(torch.stack([d.p0[i, j] for d, i, j in recs]))
    return torch.stack(out).cpu().numpy(), [d.p0.cpu().numpy() for d in doms if not d.pml]


def exact(case, seed):
    scenes = _scenes(case, seed)
    doms = sum(len(_domains(s)) * s["steps"] for s in scenes)
    points = sum(_transform_points(s) * s["steps"] for s in scenes)
    if doms * 3e-3 + points * 6e-10 > 15 * (1.0 if torch.cuda.is_available() else 0.2):
        return None
    e = case["entry"]
    if e == "frames":
        kept = []

        def keep(step, air):
            if step % case["save"] == 0:
                kept.append([d.p0.cpu().numpy() for d in air])

        rec, _ = _solve64(scenes[0], keep)
        return {"frames": [np.stack([k[i].ravel() for k in kept]) for i in range(len(kept[0]))], "samples": rec[::case["save"]].T.copy()}
    got = [_solve64(s) for s in scenes]
    if e == "advance":
        return {"receivers": got[0][0], "p0": got[0][1]}
    flat = np.concatenate([p.ravel() for _, ps in got for p in ps])
    if e == "noalloc":
        return {"frame": flat, "samples": got[0][0]}
    if e == "serve":
        return {"receivers": np.concatenate([r.ravel() for r, _ in got]), "p0": flat}
    return {"receivers": np.concatenate([r for r, _ in got], axis=1), "p0": flat}


# ------------------------------------------------------------------ work of a pass
def _transform_points(s):
    """Points of all strips' transforms in one time step (forward and back counted once)."""
    total = 0
    for d in _domains(s):
        if d.rigid:
            continue
        for h in (True, False):
            _n, _w, L, _l, _h = _strips(s, d, h)
            total += 6 * 2 * L * (d.ny if h else d.nx)
    return total


def work(case):
    """Per cell and RK stage: four fields read, their stage-start values read and four written;
    per strip a real transform, a multiply and the inverse.  Outputs once."""
    moved = flops = 0
    for s in _scenes(case, 0):
        ds = _domains(s)
        moved += 288 * sum(d.nx * d.ny for d in ds if not d.rigid) * s["steps"]
        moved += 4 * (sum(r[2] * r[3] for r in s["rects"]) * (-(-s["steps"] // s["save"]) if case["entry"] == "frames" else 1) + s["steps"] * len(s["receivers"]))
        for d in ds:
            if d.rigid:
                continue
            for h in (True, False):
                _n, _w, L, _l, _h = _strips(s, d, h)
                flops += s["steps"] * 6 * 2 * (d.ny if h else d.nx) * (5 * L * math.log2(L) + 3 * L)
    return {"bytes": float(moved), "flops": float(flops)}
