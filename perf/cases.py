"""Measured cases of the stereo pipeline: what a program built on this library has it do.

A case is one call (or one batch) through the public entry points: a pyramid
level or a single-scale frame through the C API, whole frames through
StereoMatcher, batches through BatchEngine, the speckle filter on a finished
disparity map.  Images are synthetic stereo pairs made on the GPU the way
pyrsgm_gb300/synth.py makes them: value noise plus fine texture, slanted
Voronoi patches as ground truth, a forward-warped right view with occlusion
noise and sensor noise.

listed() names the cases, draw() gives others of the same ranges, prepare()
makes what the caller holds, run() is one pass, work() counts what a pass
cannot do without, and exact() restates the pipeline in plain torch (integer
costs, 64-bit confidences).
"""
import math

import torch

import pyrsgm_gb300 as pg

MAX = 32767
BT, CENSUS = 0, 1
PENALTY = {BT: (300, 2400), CENSUS: (8, 32)}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, name=None, **kw):
    c = dict(kind=kind, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one pyramid level of a small image through the C API, the call an embedding engine with its own
        # pyramid makes: the smallest work, bound by launches and latency
        _case("level", "level_census_160x96", w=160, h=96, cost=CENSUS, D=16, bs=3, adaptive=False),
        # the same entry point on a 540p refinement level with the 5x5 Birchfield-Tomasi window
        _case("level", "level_bt_960x540", w=960, h=540, cost=BT, D=16, bs=5, adaptive=True),
        # VGA frame, 64 disparities, no pyramid, through the C API: the classic SGM set-up
        _case("single", "single_bt_640x480_d64", w=640, h=480, cost=BT, D=64, adaptive=False),
        # Census frame of odd size with a label count that is no power of two, adaptive penalties
        _case("single", "single_census_641x479_d96", w=641, h=479, cost=CENSUS, D=96, adaptive=True),
        # StereoMatcher with the default parameters (Birchfield-Tomasi, 128 disparities, no pyramid) on a 720p frame
        _case("matcher", "matcher_default_1280x720", w=1280, h=720, cost=BT, D=128, levels=0, adaptive=False),
        # 720p Census with two pyramid levels: live video at moderate range
        _case("matcher", "matcher_census_1280x720_l2", w=1280, h=720, cost=CENSUS, D=128, levels=2, adaptive=True),
        # 1080p, 256 disparities, two levels, Census: the single-pair latency configuration
        _case("matcher", "matcher_census_1080p_l2", w=1920, h=1080, cost=CENSUS, D=256, levels=2, adaptive=True),
        # 1080p, 256 disparities, three levels, Birchfield-Tomasi, one pair at a time
        _case("matcher", "matcher_bt_1080p_l3", w=1920, h=1080, cost=BT, D=256, levels=3, adaptive=True),
        # a large still frame of ragged size, deepest pyramid
        _case("matcher", "matcher_bt_2879x1987_l4", w=2879, h=1987, cost=BT, D=256, levels=4, adaptive=True),
        # 32 pairs 1080p, Census and Birchfield-Tomasi in turn, replayed as a graph: offline throughput
        _case("batch", "batch_32x1080p_l3", n=32, w=1920, h=1080, D=256, levels=3, cost=-1, mix=0, graph=True),
        # pairs of mixed sizes, depths, costs and label counts run once each, as a server forms them
        _case("batch", "batch_mixed_12", n=12, w=0, h=0, D=0, levels=0, cost=-1, mix=17, graph=False),
        # speckle removal on a finished 1080p disparity map
        _case("speckle", "speckle_1080p", w=1920, h=1080, patches=60, noise=0.04),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["level", "level", "single", "single", "matcher", "matcher", "matcher", "batch", "speckle"])
    w = _log(rng, 140, 2600)
    h = max(90, min(1600, int(w * rng.uniform(0.45, 0.8))))
    cost = rng.choice([BT, CENSUS])
    adaptive = rng.random() < 0.5
    if kind == "level":
        return _case(kind, w=min(w, 1300), h=min(h, 800), cost=cost, D=16, bs=rng.choice([3, 5]), adaptive=adaptive)
    if kind == "single":
        D = 16 * rng.randint(1, 8)
        return _case(kind, w=max(min(w, 1300), 2 * D), h=min(h, 800), cost=cost, D=D, adaptive=adaptive)
    if kind == "matcher":
        levels = rng.randint(0, 4)
        D = rng.choice([64, 128, 256]) if levels else 16 * rng.randint(2, 12)
        if levels == 0:
            w, h = min(w, 1300), min(h, 800)
        return _case(kind, w=max(w, 2 * D), h=h, cost=cost, D=D, levels=levels, adaptive=adaptive)
    if kind == "batch":
        if rng.random() < 0.5:
            return _case(kind, n=rng.randint(2, 16), w=0, h=0, D=0, levels=0, cost=-1, mix=rng.randint(1, 10 ** 6),
                         graph=rng.random() < 0.5)
        D = rng.choice([64, 128, 256])
        n = max(2, min(32, int(60e6 / (w * h) * rng.random())))
        return _case(kind, n=n, w=max(w, 2 * D), h=h, D=D, levels=rng.randint(1, 4), cost=-1, mix=0,
                     graph=rng.random() < 0.7)
    return _case("speckle", w=w, h=h, patches=rng.randint(5, 200), noise=round(rng.uniform(0.0, 0.2), 3))


MIX_SIZES = [(640, 480), (960, 540), (1280, 720), (1920, 1080), (641, 481), (1237, 719)]


def _pairs(case):
    """(w, h, D, levels, cost, adaptive) of every pair of a case."""
    if case["kind"] == "batch":
        if case["mix"]:
            g = torch.Generator().manual_seed(case["mix"])

            def pick(n):
                return int(torch.randint(n, (1,), generator=g))

            out = []
            for _ in range(case["n"]):
                w, h = MIX_SIZES[pick(len(MIX_SIZES))]
                out.append((w, h, (64, 128, 256)[pick(3)], 1 + pick(4), pick(2), True))
            return out
        return [(case["w"], case["h"], case["D"], case["levels"], CENSUS if i % 2 == 0 else BT, True)
                for i in range(case["n"])]
    return [(case["w"], case["h"], case["D"], case.get("levels", 0), case["cost"], case["adaptive"])]


def _params(D, levels, cost, adaptive):
    p1, p2 = PENALTY[cost]
    return pg.Params(num_disparities=D, pyramid_levels=levels, cost_mode=cost, p1=p1, p2=p2, adaptive_p2=adaptive)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _value_noise(g, h, w, dev):
    out = torch.zeros(h, w, device=dev)
    amp, total = 1.0, 0.0
    for o in range(4):
        c = max(2, 32 >> o)
        grid = torch.rand(h // c + 2, w // c + 2, generator=g, device=dev)
        fy, fx = torch.arange(h, device=dev) / c, torch.arange(w, device=dev) / c
        y0, x0 = fy.floor().long(), fx.floor().long()
        ty, tx = fy - y0, fx - x0
        ty, tx = (ty * ty * (3 - 2 * ty))[:, None], (tx * tx * (3 - 2 * tx))[None, :]
        top = grid[y0][:, x0] + (grid[y0][:, x0 + 1] - grid[y0][:, x0]) * tx
        bot = grid[y0 + 1][:, x0] + (grid[y0 + 1][:, x0 + 1] - grid[y0 + 1][:, x0]) * tx
        out += amp * (top + (bot - top) * ty)
        total += amp
        amp *= 0.5
    return out / total * 255.0


def _truth(g, h, w, d_max, patches, dev):
    u = torch.rand(patches, 5, generator=g, device=dev)
    sy, sx = u[:, 0] * h, u[:, 1] * w
    yy = torch.arange(h, device=dev, dtype=torch.float32)[:, None]
    xx = torch.arange(w, device=dev, dtype=torch.float32)[None, :]
    best = torch.full((h, w), float("inf"), device=dev)
    d = torch.zeros(h, w, device=dev)
    for k in range(patches):
        dist = (yy - sy[k]) ** 2 + (xx - sx[k]) ** 2
        a, b = (u[k, 2] - 0.5) * 0.3 * d_max / w, (u[k, 3] - 0.5) * 0.3 * d_max / h
        plane = a * (xx - sx[k]) + b * (yy - sy[k]) + (0.1 + 0.8 * u[k, 4]) * d_max
        m = dist < best
        best = torch.where(m, dist, best)
        d = torch.where(m, plane, d)
    return d.clamp(0.0, float(d_max))


def _stereo(g, w, h, d_max, patches, dev):
    """left, right (uint8 [h, w]) and the true disparity."""
    left = (0.6 * _value_noise(g, h, w, dev) + 0.4 * 255 * torch.rand(h, w, generator=g, device=dev))
    left = left.round().clamp(0, 255)
    d = _truth(g, h, w, d_max, patches, dev)
    xx = torch.arange(w, device=dev).expand(h, w)
    xr = (xx - d).round().long()
    key = ((d * 16).round().long() << 13) | xx                    # the nearer surface wins
    key = torch.where((xr >= 0) & (xr < w), key, torch.full_like(key, -1))
    best = torch.full((h, w), -1, dtype=torch.long, device=dev)
    best.scatter_reduce_(1, xr.clamp(0, w - 1), key, "amax")
    right = 255 * torch.rand(h, w, generator=g, device=dev)
    right = torch.where(best >= 0, left.gather(1, (best & 8191).clamp(0, w - 1)), right)
    right = (right + 2.0 * torch.randn(h, w, generator=g, device=dev)).round().clamp(0, 255)
    return left.to(torch.uint8), right.to(torch.uint8), d


def _gen(seed, dev):
    return torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 11)


def _inputs(case, seed, dev):
    """The (left, right, truth) triples of a case, and the parent maps of a refinement level."""
    g = _gen(seed, dev)
    if case["kind"] == "level":
        w, h = case["w"], case["h"]
        l, r, t = _stereo(g, w, h, min(120, w // 4), 8, dev)
        ph, pw = (h + 1) // 2, (w + 1) // 2
        half = t[::2, ::2] / 2.0
        raw = ((half + 0.3 * torch.randn(ph, pw, generator=g, device=dev)) * 16).round().clamp(0, 16 * (pw - 1))
        raw = torch.where(torch.rand(ph, pw, generator=g, device=dev) < 0.05, torch.full_like(raw, -16.0), raw)
        conf = torch.rand(ph, pw, generator=g, device=dev)
        return [(l, r, t)], (raw.to(torch.int16), conf)
    out = []
    for (w, h, D, _, _, _) in _pairs(case):
        out.append(_stereo(g, w, h, min(D - 1, w // 3), 12, dev))
    return out, None


def _level_args(case):
    p1, p2 = PENALTY[case["cost"]]
    return dict(num_disparities=case["D"], max_disparity=min(255, case["w"] - 1), block_size=case["bs"], p1=p1, p2=p2,
                cost_mode=case["cost"], refine=True, adaptive_p2=case["adaptive"])


def _single_args(case):
    p1, p2 = PENALTY[case["cost"]]
    return dict(num_disparities=case["D"], p1=p1, p2=p2, cost_mode=case["cost"], adaptive_p2=case["adaptive"])


def _outputs(h, w, dev):
    return {"disp16": torch.empty((h, w), dtype=torch.int16, device=dev),
            "disp32": torch.empty((h, w), dtype=torch.float32, device=dev),
            "conf": torch.empty((h, w), dtype=torch.float32, device=dev)}


def _speckle_map(case, seed, dev):
    g = _gen(seed, dev)
    h, w = case["h"], case["w"]
    d = (_truth(g, h, w, 200.0, case["patches"], dev) * 16).round().to(torch.int16)
    u = torch.rand(h, w, generator=g, device=dev)
    d = torch.where(u < case["noise"], (torch.rand(h, w, generator=g, device=dev) * 3200).to(torch.int16), d)
    return torch.where(u > 0.93, torch.full_like(d, -16), d)


def prepare(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    if kind == "speckle":
        m = _speckle_map(case, seed, dev)
        return {"case": case, "map": m, "out": torch.empty_like(m)}
    pairs, parent = _inputs(case, seed, dev)
    if kind == "batch":
        specs = _pairs(case)
        if case["mix"]:
            out = [_outputs(s[1], s[0], dev) for s in specs]
            maps = out
        else:                                     # one size: the maps of all pairs lie together
            out = _outputs(case["n"] * case["h"], case["w"], dev)
            out = {k: v.view(case["n"], case["h"], case["w"]) for k, v in out.items()}
            maps = [{k: v[i] for k, v in out.items()} for i in range(case["n"])]
        items = [dict(left=l, right=r, params=_params(D, levels, cost, adaptive), **m)
                 for (l, r, _), m, (w, h, D, levels, cost, adaptive) in zip(pairs, maps, specs)]
        return {"case": case, "items": items, "engine": pg.BatchEngine(64 << 30), "arr": pg.BatchEngine.make_pairs(items),
                "stream": torch.cuda.Stream(), "out": out}
    l, r, _ = pairs[0]
    h, w = l.shape
    state = {"case": case, "left": l, "right": r, "out": _outputs(h, w, dev)}
    if kind == "matcher":
        state["matcher"] = pg.StereoMatcher(w, h, _params(case["D"], case["levels"], case["cost"], case["adaptive"]))
    else:
        state["ws"] = pg.Workspace()
        state["ws"].reserve(w, h, case["D"])
        state["parent"] = parent
        state["args"] = _level_args(case) if kind == "level" else _single_args(case)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "speckle":
        state["out"].copy_(state["map"])
        return pg.filter_speckles(state["out"], -16, 200, 16)
    out = state["out"]
    if kind == "batch":
        s = state["stream"]
        s.wait_stream(torch.cuda.current_stream())
        state["engine"].run_pairs(state["arr"], case["graph"], s)
        torch.cuda.current_stream().wait_stream(s)
        return out
    if kind == "matcher":
        state["matcher"].compute_into(state["left"], state["right"], out["disp16"], out["disp32"], out["conf"])
        return out
    if kind == "level":
        pd, pc = state["parent"]
        r = pg.compute_level(state["ws"], state["left"], state["right"], pd, pc, out["disp16"], out["disp32"],
                             out["conf"], **state["args"])
    else:
        r = pg.compute_single_scale(state["ws"], state["left"], state["right"], out["disp16"], out["disp32"],
                                    out["conf"], **state["args"])
    if r != 0:
        raise RuntimeError("pyrsgm: call failed")
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: images (and parent maps) in, the three maps out.  Operations: the
    matching cost, the three path recurrences (8 additions and minima per
    label), their sum and the winner, over every level's labels."""
    if case["kind"] == "speckle":
        px = case["w"] * case["h"]
        return {"bytes": 4 * px, "flops": 8 * px}
    nbytes = flops = 0.0
    for (w, h, D, levels, cost, adaptive) in _pairs(case):
        nbytes += w * h * (2 + 10)
        per = 3 * 8 + 4 + (2 if cost == CENSUS else 14)
        if case["kind"] == "matcher" or case["kind"] == "batch":
            for li in pg.level_geometry(w, h, _params(D, levels, cost, adaptive)):
                flops += li.width * li.height * li.num_labels * per
        else:
            flops += w * h * D * per
            if case["kind"] == "level":
                nbytes += (w * h) / 4 * 6
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain torch: integer costs, 64-bit confidences
# ---------------------------------------------------------------------------
def _shift(a, dy, dx):
    """a[..., clamp(y + dy), clamp(x + dx)]."""
    h, w = a.shape[-2:]
    ys = (torch.arange(h, device=a.device) + dy).clamp(0, h - 1)
    xs = (torch.arange(w, device=a.device) + dx).clamp(0, w - 1)
    return a.index_select(-2, ys).index_select(-1, xs)


def _pyrdown(a):
    h, w = a.shape[-2:]

    def reflect(i, n):
        i = i.abs()
        return torch.where(i >= n, 2 * n - 2 - i, i).clamp(min=0)

    k = (1, 4, 6, 4, 1)
    ys, xs = 2 * torch.arange((h + 1) // 2, device=a.device), 2 * torch.arange((w + 1) // 2, device=a.device)
    t = sum(k[i] * a.index_select(-2, reflect(ys + i - 2, h)) for i in range(5))
    t = sum(k[i] * t.index_select(-1, reflect(xs + i - 2, w)) for i in range(5))
    return (t + 128) >> 8


def _census(a):
    v = torch.zeros_like(a)
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            v = (v << 1) | (_shift(a, dy, dx) < a).int()
    return v


def _popcount(v):
    v = v - ((v >> 1) & 0x55555555)
    v = (v & 0x33333333) + ((v >> 2) & 0x33333333)
    v = (v + (v >> 4)) & 0x0F0F0F0F
    return ((v * 0x01010101) >> 24) & 0xFF


def _bt_features(a, cap=63):
    z = max(cap, 15) | 1
    gx = 2 * (_shift(a, 0, 1) - _shift(a, 0, -1))
    for dy in (-1, 1):
        gx = gx + _shift(a, dy, 1) - _shift(a, dy, -1)
    out = []
    for c in (gx.clamp(-z, z) + z, a):
        l, r = (c + _shift(c, 0, -1)) >> 1, (c + _shift(c, 0, 1)) >> 1
        out.append((c, torch.minimum(torch.minimum(l, r), c), torch.maximum(torch.maximum(l, r), c)))
    return out


def _bt(fl, fr):
    """Cost of matched features (value, lowest, highest) of both channels."""
    c = []
    for (u, u0, u1), (v, v0, v1) in zip(fl, fr):
        a = torch.maximum(u - v1, v0 - u).clamp(min=0)
        b = torch.maximum(v - u1, u0 - v).clamp(min=0)
        c.append(torch.minimum(a, b))
    return (c[0] + (c[1] >> 2)).clamp(max=255)


def _cost(L, R, D, cost, bs, base):
    """[h, w, D] matching costs; base None: label d is disparity d."""
    h, w = L.shape
    xs = torch.arange(w, device=L.device, dtype=torch.int32).expand(h, w)
    C = torch.empty((h, w, D), dtype=torch.int32, device=L.device)
    half = bs // 2

    def take(t, x):
        return t.gather(1, x.clamp(0, w - 1).long())

    if cost == CENSUS:
        cl, cr = _census(L), _census(R)
        for d in range(D):
            x2 = xs - d - (base if base is not None else 0)
            C[..., d] = torch.where((x2 >= 0) & (x2 < w), _popcount(cl ^ take(cr, x2)), torch.full_like(xs, 24))
        return C
    fl, fr = _bt_features(L), _bt_features(R)
    for d in range(D):
        if base is None:
            x2 = xs - d
            b = _bt(fl, [tuple(take(t, x2) for t in ch) for ch in fr])
            b = torch.where((x2 >= 0) & (x2 < w), b, torch.full_like(b, 255))
            s = sum(_shift(b, 0, dx) for dx in range(-half, half + 1)).clamp(max=MAX)
            C[..., d] = sum(_shift(s, dy, 0) for dy in range(-half, half + 1)).clamp(max=MAX)
            continue
        total = torch.zeros_like(xs)
        for dy in range(-half, half + 1):
            fry = [tuple(_shift(t, dy, 0) for t in ch) for ch in fr]
            for dx in range(-half, half + 1):
                x2 = (xs + dx).clamp(0, w - 1) - base - d
                b = _bt([tuple(_shift(t, dy, dx) for t in ch) for ch in fl],
                        [tuple(take(t, x2) for t in ch) for ch in fry])
                total = total + torch.where((x2 >= 0) & (x2 < w), b, torch.full_like(b, 255))
        C[..., d] = total.clamp(max=MAX - 1)
    return C


def _path(C, base, img, p1, p2, table, flip):
    """Path costs along dimension 1 of [k, n, D] costs (labels with C == MAX are
    invalid); base [k, n] shifts the labels from one pixel to the next."""
    if flip:
        C, img = C.flip(1), img.flip(1)
        base = base.flip(1) if base is not None else None
    k, n, D = C.shape
    out = torch.empty_like(C)
    pen = table[(img[:, 1:] - img[:, :-1]).abs().long()] if table is not None else None
    prev = out[:, 0] = C[:, 0]
    lab = torch.arange(D, device=C.device)[None, :]
    pad = torch.full((k, D + 4), MAX, dtype=C.dtype, device=C.device)
    for i in range(1, n):
        c = C[:, i]
        pad[:, 2:D + 2] = prev
        if base is None:
            s0, sm, sp = prev, pad[:, 1:D + 1], pad[:, 3:D + 3]
        else:
            at = lab + (base[:, i] - base[:, i - 1])[:, None].long() + 2
            s0 = pad.gather(1, at.clamp(0, D + 3))
            sm = pad.gather(1, (at - 1).clamp(0, D + 3))
            sp = pad.gather(1, (at + 1).clamp(0, D + 3))
        mp = prev.amin(1, keepdim=True)
        jump = mp + (pen[:, i - 1:i] if pen is not None else p2)
        best = torch.minimum(torch.minimum(s0, jump.clamp(max=MAX)), torch.minimum(sm, sp) + p1)
        v = torch.where((best >= MAX) & (mp < MAX), torch.full_like(c, MAX), (c + best - mp).clamp(max=MAX))
        v = torch.where(mp < MAX, v, c)
        prev = out[:, i] = v
    return out.flip(1) if flip else out


def _p2_table(p2, dev):
    alpha, beta, lower, upper = 3.041, 16.137, 0.601, 1.77
    ratio = lower + (1.0 + alpha - lower) * torch.exp(-torch.arange(256, dtype=torch.float64, device=dev) / beta)
    return ((p2 * ratio).clamp(max(1.0, p2 * lower), p2 * upper) + 0.5).int()


def _median(d):
    """3x3 median over the in-image neighbours (the upper one of an even count)."""
    h, w = d.shape
    p = torch.full((h + 2, w + 2), 1 << 20, dtype=d.dtype, device=d.device)
    p[1:-1, 1:-1] = d
    v = torch.stack([p[y:y + h, x:x + w] for y in range(3) for x in range(3)], -1)
    n = (v < (1 << 20)).sum(-1, keepdim=True)
    return v.sort(-1).values.gather(-1, n // 2)[..., 0]


def _frame(L, R, D, cost, bs, adaptive, maxD, pyr, parent, lr_check, median):
    """One level: disparity * 16 (int), 64-bit confidence before the output rule."""
    dev = L.device
    h, w = L.shape
    p1, p2 = PENALTY[cost]
    xs = torch.arange(w, device=dev, dtype=torch.int32).expand(h, w)
    labels = torch.arange(D, device=dev, dtype=torch.int32)
    base, known = torch.zeros_like(xs), torch.ones_like(xs, dtype=torch.bool)
    min_conf = torch.tensor(0.05, dtype=torch.float32, device=dev)
    if parent is not None:
        pd, pc = parent
        py = (torch.arange(h, device=dev) >> 1).clamp(max=pd.shape[0] - 1)
        px = (torch.arange(w, device=dev) >> 1).clamp(max=pd.shape[1] - 1)
        raw, conf = pd[py][:, px].int(), pc[py][:, px].float()
        known = (raw != -16) & (conf >= min_conf)
        center = (2 * raw + 8) >> 4
        b = center - D // 2 + (2 * raw - center * 16 >= 0).int()
        largest = xs.clamp(max=maxD) - D + 1
        base = torch.where(largest >= 0, torch.minimum(b.clamp(min=0), largest), torch.zeros_like(b))
    C = _cost(L, R, D, cost, bs, base if parent is not None else None)
    if pyr:
        real = base[..., None] + labels
        ok = known[..., None] & (real <= maxD) & (real <= xs[..., None])
        C = torch.where(ok, C, torch.full_like(C, MAX))
        count = ok.sum(-1)
    img = L
    table = _p2_table(p2, dev) if adaptive else None
    sh = base if parent is not None else None
    x0 = 0 if pyr else min(D, w)
    total = torch.zeros_like(C)
    sent = torch.zeros_like(C, dtype=torch.bool)
    for name in ("lr", "tb", "rl"):
        if name == "tb":
            v = _path(C.transpose(0, 1).contiguous(), sh.t().contiguous() if sh is not None else None,
                      img.t().contiguous(), p1, p2, table, False).transpose(0, 1)
        elif name == "lr":
            v = torch.full_like(C, 0)
            if x0 < w:
                v[:, x0:] = _path(C[:, x0:], sh, img[:, x0:], p1, p2, table, False)
        else:
            v = _path(C, sh, img, p1, p2, table, True)
        sent |= v >= MAX
        total += v
    if pyr:
        total = torch.where(sent, torch.full_like(total, MAX), total.clamp(max=MAX - 1))
    else:
        total = total.clamp(max=MAX)
    key = ((total.long() << 16) | labels).amin(-1)
    lowest, best = (key >> 16).int(), (key & 0xFFFF).int()
    near = (labels - best[..., None]).abs() <= 1
    alt = torch.where(near, torch.full_like(total, MAX), total).amin(-1)

    def at(d):
        return total.gather(-1, d.clamp(0, D - 1)[..., None].long())[..., 0]

    c0, c1, c2 = at(best - 1), at(best), at(best + 1)
    den = (c0 + c2 - 2 * c1).clamp(min=1)
    sub = torch.div((c0 - c2) * 16 + den, 2 * den, rounding_mode="trunc")
    inner = (best > 0) & (best < D - 1)
    conf = ((alt.double() - lowest.double()) / lowest.double().clamp(min=1.0)).clamp(0.0, 1.0)
    disp = base + best
    if pyr:
        good = (count >= 3) & (lowest < MAX) & (alt < MAX) & ~(alt * 90 < lowest * 100)
        good &= ~((best == 0) & (base > 0)) & ~((best == D - 1) & (base + D - 1 < xs.clamp(max=maxD)))
        good &= ~(conf.float() < min_conf)
        inner &= (c0 < MAX) & (c1 < MAX) & (c2 < MAX)
    else:
        good = (lowest < MAX // 2) & ~(alt * 90 < lowest * 100) & (xs >= x0) & (xs != w - 1)
    d16 = torch.where(good, disp * 16 + torch.where(inner, sub, torch.zeros_like(sub)), torch.full_like(disp, -16))
    conf = torch.where(good, conf, torch.zeros_like(conf))
    if lr_check:
        x2 = xs - disp
        fits = good & (x2 >= 0)
        k = torch.full((h, w + 1), 1 << 40, dtype=torch.long, device=dev)
        k.scatter_reduce_(1, torch.where(fits, x2, torch.full_like(x2, w)).long(),
                          (lowest.long() << 16) | (0xFFFF - xs).long(), "amin")
        k = k[:, :w]
        d2 = torch.where(k < (1 << 40), 0xFFFF - (k & 0xFFFF) - xs, torch.full_like(k, -1)).int()
        seen = []
        for d in (d16 >> 4, (d16 + 15) >> 4):
            r = xs - d
            inside = (r >= 0) & (r < w)
            v = d2.gather(1, r.clamp(0, w - 1).long())
            seen.append((inside & (v >= 0), (v - d).abs() <= 1))
        if pyr:
            keep = (seen[0][0] & seen[0][1]) | (seen[1][0] & seen[1][1])
        else:
            keep = ~((seen[0][0] & ~seen[0][1]) & (seen[1][0] & ~seen[1][1]))
        keep |= d16 == -16
        d16 = torch.where(keep, d16, torch.full_like(d16, -16))
        conf = torch.where(keep, conf, torch.zeros_like(conf))
    if median:
        m = _median(d16)
        conf = torch.where(m == d16, conf, torch.zeros_like(conf))
        d16 = m
    return d16, conf


def _maps(d16, conf):
    ok = d16 > 0
    z = torch.zeros_like(conf)
    return {"disp16": d16.to(torch.int16), "disp32": torch.where(ok, d16.double() / 16, z),
            "conf": torch.where(ok, conf, z)}


def exact(case, seed):
    if case["kind"] == "speckle":
        return None                               # whole numbers only
    specs = _pairs(case)
    if case["kind"] == "batch" and (not case["mix"] and case["w"] * case["n"] > 8000 or case["n"] > 12):
        return None                               # too long in plain torch
    dev = torch.device("cuda")
    pairs, parent = _inputs(case, seed, dev)
    out = []
    for (l, r, _), (w, h, D, levels, cost, adaptive) in zip(pairs, specs):
        L, R = l.int(), r.int()
        if case["kind"] == "level":
            return _maps(*_frame(L, R, D, cost, case["bs"], adaptive, min(255, w - 1), True, parent, True, False))
        if levels == 0:
            out.append(_maps(*_frame(L, R, D, cost, 5, adaptive, 0, False, None, True, True)))
            continue
        info = pg.level_geometry(w, h, _params(D, levels, cost, adaptive))
        pyr = [(L, R)]
        for _ in range(levels):
            pyr.append((_pyrdown(pyr[-1][0]), _pyrdown(pyr[-1][1])))
        up = None
        for k in range(levels, -1, -1):
            li = info[k]
            maxD = min(li.max_disparity, li.width - 1, MAX // 16)
            if k == levels:
                maxD = min(maxD, li.num_labels - 1)
            up = _frame(*pyr[k], li.num_labels, cost, li.block_size, adaptive, maxD, True, up, True, k == 0)
        out.append(_maps(*up))
    if case["kind"] != "batch":
        return out[0]
    return out if case["mix"] else {k: torch.stack([o[k] for o in out]) for k in out[0]}
