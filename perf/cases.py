"""Performance cases: the calls a user of this framework makes, over the range of sizes they are made at.

    listed()            the listed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program has in hand before the call: frames, samples, candidates, forest
    run(state)          one pass through the public entry points, and its whole outputs
    exact(case, seed)   what run() returns, in 64 bits, from plain torch (None where there is no such value)
    work(case)          bytes and operations one pass cannot do without

Scenes are seeded Voronoi RGB-D frames (uint8 colour with noise, per-cell depth planes between 0.5 and 5 m
with 10 % of the depths missing, labels with 5 % flips), as the tests and the benchmark use them, drawn on
the GPU so that preparing a case is quick. Forests are grown here on a scene's own pixels (median-free
random thresholds, the best of a few candidates by information gain), so that trees have the uneven depths
and the spatially coherent decisions of trained ones.
"""
import math

import numpy as np
import torch

import curfil_b200 as cf

DEV = "cuda"
BOX, REGION = 60, 15      # boxRadius and regionSize of every training configuration of this repository
_context = None


def context():
    global _context
    if _context is None:
        _context = cf.Context(torch.cuda.current_device())
    return _context


# ------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: one quarter-VGA/2 frame of a live stream through a small forest, labels only
        dict(name="predict_tiny", kind="predict", frames=1, width=160, height=120, trees=3, classes=8, probs=False,
             fill=False, lab=False),
        # one VGA camera frame through the full-size forest, probabilities and labels
        dict(name="predict_frame", kind="predict", frames=1, width=640, height=480, trees=10, classes=40, probs=True,
             fill=False, lab=False),
        # batched prediction of a recorded sequence: 64 VGA frames resident on the device
        dict(name="predict_batch", kind="predict", frames=64, width=640, height=480, trees=10, classes=40, probs=True,
             fill=False, lab=False),
        # a forest trained with useCIELab and useDepthFilling: raw device frames preprocessed and predicted
        dict(name="predict_lab", kind="predict", frames=4, width=640, height=480, trees=3, classes=13, probs=True,
             fill=True, lab=True),
        # frames from a host, ragged size, in one CUDA graph replay: pinned copies, integral images, labels back
        dict(name="predict_graph", kind="graph", frames=16, width=333, height=251, trees=10, classes=40),
        # a small training from raw host frames: integral images, device sampling, one tree of depth 12
        dict(name="forest_small", kind="forest", frames=16, width=320, height=240, classes=8, cells=12,
             per_image=3500, features=500, thresholds=20, depth=12, min_samples=1),
        # one tree of the full-size training: 200 VGA frames, 266 600 samples, depth 20
        dict(name="tree_full", kind="tree", frames=200, width=640, height=480, classes=40, cells=40, per_image=1333,
             features=2000, thresholds=20, depth=20, min_samples=50, flip=0),
        # the split search of a middle level with horizontal flipping on ragged frames within L2
        dict(name="level_flip", kind="level", frames=24, width=313, height=235, classes=13, cells=20, per_image=2500,
             nodes=97, features=500, thresholds=20, flip=2),
        # the split search of a root: one node of 800 000 samples
        dict(name="level_root", kind="level", frames=100, width=640, height=480, classes=40, cells=40, per_image=8000,
             nodes=1, features=4000, thresholds=32, flip=0),
        # the split search of a deep level of the batching configuration: 8 M samples over 8000 open nodes
        dict(name="level_deep", kind="level", frames=1000, width=640, height=480, classes=40, cells=40, per_image=8000,
             nodes=8000, features=4000, thresholds=32, flip=0),
        # refined prediction (forest, context means, per-pixel network) of a few frames
        dict(name="refine_predict", kind="refine", frames=4, width=640, height=480, trees=10, classes=40, hidden=64),
        # one epoch of the refinement network's training: features of every frame, minibatches, Adam
        dict(name="refine_train", kind="refine_train", frames=4, width=320, height=240, trees=3, classes=13, hidden=64,
             pixels=8000, batch=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["predict", "predict", "graph", "forest", "tree", "level", "level", "refine", "refine_train"])
    classes = rng.choice([5, 8, 13, 24, 33, 40])
    w = _log_int(rng, 160, 1280 if kind == "predict" else 640)
    h = max(96, int(w * rng.uniform(0.6, 0.8)))
    if kind in ("predict", "graph"):
        most = max(1, (64 if kind == "predict" else 16) * 640 * 480 // (w * h))
        case = dict(kind=kind, frames=_log_int(rng, 1, min(64, most)), width=w, height=h, trees=rng.randint(1, 10),
                    classes=classes)
        if kind == "predict":
            pre = rng.random() < 0.35
            case.update(probs=rng.random() < 0.6, fill=pre and rng.random() < 0.7, lab=pre)
        return case
    if kind == "refine":
        return dict(kind=kind, frames=rng.randint(1, 6), width=w, height=h, trees=rng.randint(1, 6), classes=classes,
                    hidden=rng.choice([16, 32, 48, 64]))
    if kind == "refine_train":
        return dict(kind=kind, frames=rng.randint(2, 6), width=min(w, 400), height=min(h, 300), trees=rng.randint(1, 4),
                    classes=classes, hidden=rng.choice([32, 48, 64]), pixels=rng.randint(3000, 9000), batch=2048)
    frames = _log_int(rng, 8, 200)
    thresholds = rng.choice([10, 20, 31, 32, 50])
    if kind == "forest":
        return dict(kind=kind, frames=min(frames, 24), width=min(w, 400), height=min(h, 300), classes=8, cells=12,
                    per_image=_log_int(rng, 500, 3500), features=_log_int(rng, 100, 800), thresholds=thresholds,
                    depth=rng.randint(8, 14), min_samples=rng.randint(1, 20))
    if kind == "tree":
        return dict(kind=kind, frames=frames, width=w, height=h, classes=classes, cells=40,
                    per_image=_log_int(rng, 200, 1500), features=_log_int(rng, 200, 2000), thresholds=thresholds,
                    depth=rng.randint(10, 20), min_samples=rng.randint(10, 50), flip=rng.choice([0, 0, 2]))
    return dict(kind=kind, frames=frames, width=w, height=h, classes=classes, cells=40,
                per_image=_log_int(rng, 300, 6000), nodes=_log_int(rng, 1, 4000), features=_log_int(rng, 200, 3000),
                thresholds=thresholds, flip=rng.choice([0, 0, 0, 2]))


# ------------------------------------------------------------------------------------------- scenes
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)
    return g


def scene(seed, n, w, h, cells, classes):
    """(rgb uint8 [n][h][w][3], depth int16 [n][h][w] mm, labels uint8 [n][h][w]) on the GPU."""
    g = _generator(seed)
    base_rgb = 30 + 195 * torch.rand(classes, 3, device=DEV, generator=g)
    base_depth = 900 + 3600 * torch.rand(classes, device=DEV, generator=g)
    rgb = torch.empty(n, h, w, 3, dtype=torch.uint8, device=DEV)
    depth = torch.empty(n, h, w, dtype=torch.int16, device=DEV)
    labels = torch.empty(n, h, w, dtype=torch.uint8, device=DEV)
    ys = torch.arange(h, device=DEV, dtype=torch.float32).view(1, h, 1)
    xs = torch.arange(w, device=DEV, dtype=torch.float32).view(1, 1, w)
    step = max(1, 10_000_000 // (w * h))
    for a in range(0, n, step):
        m = min(step, n - a)
        sx = torch.rand(m, cells, device=DEV, generator=g) * w
        sy = torch.rand(m, cells, device=DEV, generator=g) * h
        cls = torch.randint(0, classes, (m, cells), device=DEV, generator=g)
        if m * cells >= classes:       # every class is seen
            cls.view(-1)[:classes] = torch.arange(classes, device=DEV)
        best = torch.zeros(m, h, w, dtype=torch.int64, device=DEV)
        near = torch.full((m, h, w), 1e30, device=DEV)
        for k in range(cells):
            d = (xs - sx[:, k].view(m, 1, 1)) ** 2 + (ys - sy[:, k].view(m, 1, 1)) ** 2
            best = torch.where(d < near, k, best)
            near = torch.minimum(d, near)
        del near
        flat = best.view(m, -1)
        of = lambda t: torch.gather(t, 1, flat).view(m, h, w)  # noqa: E731
        c = of(cls)
        tint = (torch.rand(m, cells, 3, device=DEV, generator=g) - 0.5) * 30
        for ch in range(3):
            v = of(base_rgb[:, ch][cls] + tint[:, :, ch]) + 8 * torch.randn(m, h, w, device=DEV, generator=g)
            rgb[a:a + m, :, :, ch] = v.round_().clamp_(0, 255).to(torch.uint8)
        off = base_depth[cls] + (torch.rand(m, cells, device=DEV, generator=g) - 0.5) * 600
        bx = (torch.rand(m, cells, device=DEV, generator=g) - 0.5) * 4
        by = (torch.rand(m, cells, device=DEV, generator=g) - 0.5) * 4
        d = of(off - bx * sx - by * sy) + of(bx) * xs + of(by) * ys
        d = d.clamp_(500, 5000).round_()
        d = torch.where(torch.rand(m, h, w, device=DEV, generator=g) < 0.1, torch.zeros_like(d), d)
        depth[a:a + m] = d.to(torch.int16)
        other = (c + torch.randint(1, max(2, classes), (m, h, w), device=DEV, generator=g)) % classes
        labels[a:a + m] = torch.where(torch.rand(m, h, w, device=DEV, generator=g) < 0.05, other, c).to(torch.uint8)
    return rgb, depth, labels


def divided(v, by):
    """v / by, correctly rounded (torch multiplies by the reciprocal of a number)."""
    return v / torch.tensor(by, dtype=v.dtype, device=v.device)


def fill_depth(depth):
    """Missing depths from the right neighbour, the left, the upper and the lower one, in four passes."""
    d = depth.long()

    def spread(v, dim, backwards):
        n = v.shape[dim]
        at = torch.arange(n, device=DEV).view([-1 if k == dim else 1 for k in range(3)]).expand_as(v)
        if backwards:
            last = torch.where(v > 0, at, n).flip(dim).cummin(dim).values.flip(dim)
        else:
            last = torch.where(v > 0, at, -1).cummax(dim).values
        ok = (last >= 0) & (last < n)
        return torch.where(ok, torch.gather(v, dim, last.clamp(0, n - 1)), 0)

    d = spread(d, 2, True)
    d = spread(d, 2, False)
    d = spread(d, 1, False)
    return spread(d, 1, True)


def to_lab(rgb):
    """CIE L*a*b* float planes of linear RGB (BT.709 primaries, D65)."""
    r, g, b = (divided(rgb[..., k].double(), 255) for k in range(3))
    X = 0.412453 * r + 0.357580 * g + 0.180423 * b
    Y = 0.212671 * r + 0.715160 * g + 0.072169 * b
    Z = 0.019334 * r + 0.119193 * g + 0.950227 * b

    def f(t):
        return torch.where(t > 216.0 / 24389.0, t.clamp_min(1e-30).pow(1.0 / 3), t * (841.0 / 108.0) + 4.0 / 29.0)
    fx, fy, fz = f(X / 0.950456), f(Y), f(Z / 1.088754)
    return torch.stack([116 * fy - 16, 500 * (fx - fy), 200 * (fy - fz)], 1).float()


def integrals(rgb, depth, fill=False, lab=False):
    """Integral images of frames: colour float32 [n][3][h][w], depth sums and valid counts int64 [n][h][w]."""
    depth = fill_depth(depth) if fill else depth.long()
    planes = to_lab(rgb).double() if lab else rgb.permute(0, 3, 1, 2).long()
    color = planes.cumsum(3).cumsum(2).float()
    return color, depth.cumsum(2).cumsum(1), (depth > 0).long().cumsum(2).cumsum(1), depth


def response(ints, img, x, y, d, f, flip=None):
    """Two-box responses in 64 bits (NaN where a box leaves the frame or holds no depth). img, x, y, d
    (metres, float32; <= 0 invalid) and the feature rows f (dict of tensors) broadcast."""
    color, dsum, dcnt, _ = ints
    n, _, h, w = color.shape
    nan = float("nan")

    def scaled(v):
        return torch.trunc(v.float() / d).long()

    def corners(flat, base, cx, cy, bw, bh):
        def at(yy, xx):
            return flat[base + yy.clamp(0, h - 1) * w + xx.clamp(0, w - 1)]
        return at(cy + bh, cx + bw), at(cy - bh, cx + bw), at(cy - bh, cx - bw), at(cy + bh, cx - bw)

    def box(ox, oy, rx, ry, ch):
        cx, cy = x + scaled(ox), y + scaled(oy)
        bw, bh = scaled(rx).clamp_min(1), scaled(ry).clamp_min(1)
        ok = (cx - bw >= 0) & (cx + bw < w) & (cy - bh >= 0) & (cy + bh < h)
        lr, ur, ul, ll = corners(dsum.view(-1), img * (h * w), cx, cy, bw, bh)
        nlr, nur, nul, nll = corners(dcnt.view(-1), img * (h * w), cx, cy, bw, bh)
        count = nlr - nur + nul - nll
        deep = divided((lr - ur + ul - ll).double(), 1000) / count.double()
        deep = torch.where(count != 0, deep, nan)
        lr, ur, ul, ll = (v.double() for v in corners(color.view(-1), (img * 3 + ch) * (h * w), cx, cy, bw, bh))
        return torch.where(ok, torch.where(f["type"] == 0, deep, (lr - ur) + (ul - ll)), nan)

    ox1, ox2 = f["o1x"], f["o2x"]
    if flip is not None:
        ox1, ox2 = torch.where(flip, -ox1, ox1), torch.where(flip, -ox2, ox2)
    r = box(ox1, f["o1y"], f["r1x"], f["r1y"], f["ch1"]) - box(ox2, f["o2y"], f["r2x"], f["r2y"], f["ch2"])
    return torch.where(d > 0, r, nan)


ROWS = ("type", "o1x", "o1y", "o2x", "o2y", "r1x", "r1y", "r2x", "r2y", "ch1", "ch2")


def random_features(g, count):
    """int64 feature rows, half depth (type 0) and half colour (type 1)."""
    f = {}
    for k in ("o1x", "o1y", "o2x", "o2y"):
        f[k] = torch.randint(-BOX, BOX + 1, (count,), device=DEV, generator=g)
    for k in ("r1x", "r1y", "r2x", "r2y"):
        f[k] = torch.randint(1, REGION + 1, (count,), device=DEV, generator=g)
    f["type"] = (torch.arange(count, device=DEV) >= count // 2).long()
    for k in ("ch1", "ch2"):
        f[k] = torch.randint(0, 3, (count,), device=DEV, generator=g) * f["type"]
    return f


def sample_pixels(g, depth, labels, per_image):
    """Up to per_image pixels with a depth per frame: (image, x, y, depth m, label), in the order of
    training samples (image, label, 10-pixel blocks)."""
    n, h, w = depth.shape
    p = torch.randint(0, h * w, (n, per_image + per_image // 3 + 16), device=DEV, generator=g)
    d = torch.gather(depth.view(n, -1).long(), 1, p)
    lab = torch.gather(labels.view(n, -1).long(), 1, p)
    ok = (d > 0) & ((d > 0).cumsum(1) <= per_image)
    img = torch.arange(n, device=DEV).view(n, 1).expand_as(p)[ok]
    p, d, lab = p[ok], d[ok], lab[ok]
    y, x = p // w, p % w
    order = torch.argsort((img * 256 + lab) * (1 << 26) + (y // 10) * (1 << 13) + x // 10, stable=True)
    img, x, y, d, lab = (t[order] for t in (img, x, y, d, lab))
    return img, x, y, divided(d.float(), 1000), lab


def sample_rows(s, flip):
    """cf_sample rows of sampled pixels, in pinned host memory."""
    img, x, y, d, lab = s
    rows = torch.stack([x | (y << 16), img, torch.zeros_like(x), lab | (flip << 8)], 1).to(torch.int32)
    rows[:, 2] = d.contiguous().view(torch.int32)
    host = torch.empty(rows.shape, dtype=torch.int32, pin_memory=True)
    host.copy_(rows)
    torch.cuda.synchronize()
    return host.numpy().view(cf.SAMPLE_DTYPE).reshape(-1)


# ------------------------------------------------------------------------------------------- forests
def grow_tree(g, ints, s, classes, max_depth=20, least=25, candidates=12):
    """One tree grown breadth-first in torch: arrays left, feature rows, threshold, histogram."""
    img, x, y, d, lab = s
    node = torch.zeros_like(img)
    nodes = 1
    left, thr, hist, rows = [], [], [], []
    active = torch.ones(1, dtype=torch.bool, device=DEV)
    first = 0                                    # id of the level's first node
    for level in range(max_depth):
        counts = torch.bincount(node * classes + lab, minlength=nodes * classes).view(nodes, classes)
        hist.append(counts)
        total = counts.sum(1)
        split = active & (total >= least) & ((counts > 0).sum(1) > 1) & (level + 1 < max_depth)
        f = random_features(g, candidates)
        pick = torch.randperm(candidates, device=DEV, generator=g)
        f = {k: v[pick].view(1, -1) for k, v in f.items()}
        r = response(ints, img.view(-1, 1), x.view(-1, 1), y.view(-1, 1), d.view(-1, 1), f)
        # threshold of (node, candidate): the response of one of the node's samples
        start = total.cumsum(0) - total
        order = torch.argsort(node, stable=True)
        at = order[(start + (torch.rand(nodes, device=DEV, generator=g) * total).long().clamp_min(0)
                    ).clamp(0, max(0, len(order) - 1))]
        t = torch.nan_to_num(r[at], nan=0.0).float()                       # [nodes][candidates]
        right = ~(r <= t[node].double())                                    # NaN right
        key = ((node.view(-1, 1) * candidates + torch.arange(candidates, device=DEV)) * classes + lab.view(-1, 1))
        rc = torch.bincount(key[right], minlength=nodes * candidates * classes).view(nodes, candidates, classes).double()
        lc = counts.view(nodes, 1, classes) - rc

        def plogp(v):
            return torch.where(v > 0, v * v.clamp_min(1).log(), 0)
        nl, nr = lc.sum(2), rc.sum(2)
        gain = plogp(lc).sum(2) + plogp(rc).sum(2) - plogp(nl) - plogp(nr)
        gain = torch.where((nl > 0) & (nr > 0), gain, -torch.inf)
        gain = (gain * 1024).round() * candidates - torch.arange(candidates, device=DEV)   # one best, on any device
        best = gain.argmax(1)
        split &= torch.isfinite(gain.gather(1, best.view(-1, 1))[:, 0])
        rank = split.long().cumsum(0) - 1
        left.append(torch.where(split, first + nodes + 2 * rank, -1))
        thr.append(torch.where(split, t.gather(1, best.view(-1, 1))[:, 0], torch.nan))
        rows.append(torch.stack([torch.where(split, f[k].view(-1)[best], 0) for k in ROWS], 1))
        kids = int(split.sum()) * 2
        keep = split[node]
        go = right.gather(1, best[node].view(-1, 1))[:, 0]
        node = (2 * rank[node] + go.long())[keep]
        img, x, y, d, lab = (v[keep] for v in (img, x, y, d, lab))
        first += nodes
        nodes = kids
        active = torch.ones(max(nodes, 1), dtype=torch.bool, device=DEV)
        if nodes == 0:
            break
    return torch.cat(left), torch.cat(rows), torch.cat(thr).float(), torch.cat(hist)


def forest_arrays(seed, trees, classes, width, height, fill=False, lab=False):
    """Trees (arrays) and the class prior of a forest grown on frames of its own."""
    g = _generator(seed + 77)
    w, h = max(width, 200), max(height, 150)
    rgb, depth, labels = scene(seed + 1000003, 12, min(w, 640), min(h, 480), 40, classes)
    ints = integrals(rgb, depth, fill, lab)
    grown = []
    for _ in range(trees):
        s = sample_pixels(g, ints[3], labels, 8000)
        grown.append(grow_tree(g, ints, s, classes))
    return grown, torch.bincount(labels.view(-1).long(), minlength=classes)


def make_forest(grown, prior, fill=False, lab=False):
    trees = []
    for k, (left, rows, thr, hist) in enumerate(grown):
        trees.append(cf.Tree.from_arrays(k, left.cpu().numpy().astype(np.int32), rows.cpu().numpy().astype(np.int8),
                                         thr.cpu().numpy(), hist.cpu().numpy().astype(np.uint32)))
    f = cf.Forest(context(), trees, prior=prior.cpu().numpy().astype(np.uint32))
    f.set_preprocessing(fill_depth=fill, cie_lab=lab)
    return f


def forest_exact(grown, prior, ints, frame):
    """Class probabilities of one frame in 64 bits, [classes][h][w]."""
    color, dsum, dcnt, depth = ints
    h, w = depth.shape[1:]
    y, x = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")
    x, y = x.reshape(-1), y.reshape(-1)
    d = divided(depth[frame].reshape(-1).float(), 1000)
    img = torch.full_like(x, frame)
    weights = prior.double() / prior.sum().double()
    total = None
    for left, rows, thr, hist in grown:
        node = torch.zeros_like(x)
        while True:
            go = torch.nonzero(left[node] >= 0)[:, 0]
            if len(go) == 0:
                break
            at = node[go]
            f = {k: rows[at, i] for i, k in enumerate(ROWS)}
            r = response(ints, img[go], x[go], y[go], d[go], f)
            node[go] = left[at] + (~(r <= thr[at].double())).long()
        leaf = hist.double() / hist.sum(1, keepdim=True).double() * weights
        total = leaf[node] if total is None else total + leaf[node]
    return (total / total.sum(1, keepdim=True)).t().reshape(-1, h, w)


# ------------------------------------------------------------------------------------------- levels
def level_inputs(case, seed):
    """Samples of a level's open nodes, candidate features and thresholds, as the level's training has them."""
    g = _generator(seed + 5)
    n, w, h, C, M = case["frames"], case["width"], case["height"], case["classes"], case["nodes"]
    F, T = case["features"], case["thresholds"]
    rgb, depth, labels = scene(seed, n, w, h, case["cells"], C)
    s = sample_pixels(g, depth, labels, case["per_image"])
    # an open node holds a few classes; node sizes are skewed, each node's samples stay in frame order
    M = min(M, len(s[0]) // 4)
    group = (s[4] + torch.randint(0, 3, s[4].shape, device=DEV, generator=g)) % C
    per = max(1, M // C)
    u = torch.rand(s[4].shape, device=DEV, generator=g)
    node = (group * per + (u * u * per).long().clamp_max(per - 1)) % M if M > 1 else torch.zeros_like(s[4])
    order = torch.argsort(node, stable=True)
    s = tuple(v[order] for v in s)
    counts = torch.bincount(node, minlength=M)
    counts = counts[counts > 0]
    # candidates: features sorted as training sorts them, thresholds the responses of random samples
    f = random_features(g, F)
    key = (f["type"] << 30) | (f["ch1"] << 26) | (f["ch2"] << 22) | ((f["o1y"] + 127) << 14) | ((f["o1x"] + 127) << 6)
    key = torch.where(key >= 1 << 31, key - (1 << 32), key)
    order = torch.argsort(key, stable=True)
    f = {k: v[order] for k, v in f.items()}
    k = min(n, 40)
    few = torch.nonzero(s[0] < k)[:, 0]
    ints = integrals(rgb[:k], depth[:k])
    at = few[torch.randint(0, len(few), (T, F), device=DEV, generator=g)]
    r = response(ints, s[0][at], s[1][at], s[2][at], s[3][at], {q: v.view(1, -1) for q, v in f.items()})
    thr = torch.nan_to_num(r, nan=0.0).float()
    return rgb, depth, s, counts, f, thr


def level_exact(case, seed):
    """The best score of every open node, in 64 bits."""
    if case["frames"] * case["width"] * case["height"] > 40_000_000 or case["nodes"] > 200:
        return None
    rgb, depth, s, counts, f, thr = level_inputs(case, seed)
    img, x, y, d, lab = s
    M, C, T, F = len(counts), case["classes"], case["thresholds"], case["features"]
    if len(img) * F > 4_000_000_000:
        return None
    ints = integrals(rgb, depth)
    node = torch.repeat_interleave(torch.arange(M, device=DEV), counts)
    both = case["flip"] == 2
    hist = torch.bincount(node * C + lab, minlength=M * C).view(M, C).double() * (2 if both else 1)
    N = hist.sum(1)

    def plogp(v):
        return torch.where(v > 0, v * v.clamp_min(1e-300).log2(), 0)
    hc = (plogp(N) - plogp(hist).sum(1)) / N
    best = torch.zeros(M, dtype=torch.float64, device=DEV)
    none = torch.zeros(1, dtype=torch.bool, device=DEV)
    for k in range(F):
        fk = {q: v[k] for q, v in f.items()}
        t = thr[:, k].sort().values.double()
        cum = 0
        for flipped in ((False, True) if both else (False,)):
            r = response(ints, img, x, y, d, fk, ~none if flipped else none)
            b = torch.searchsorted(t, torch.nan_to_num(r, nan=torch.inf))        # thresholds below r
            cum = cum + torch.bincount((node * C + lab) * (T + 1) + b, minlength=M * C * (T + 1)).view(M, C, T + 1)
        l = cum.cumsum(2)[:, :, :T].double()
        rr = hist.view(M, C, 1) - l
        L, R = l.sum(1), rr.sum(1)
        # information gain and its normalisation by the entropies of the split and of the classes
        S = plogp(l).sum(1) + plogp(rr).sum(1) - plogp(L) - plogp(R) + (plogp(N) - plogp(hist).sum(1)).view(M, 1)
        hs = (plogp(N).view(M, 1) - plogp(L) - plogp(R)) / N.view(M, 1)
        score = 2 * (S / N.view(M, 1)).clamp(0, 1) / (hs + hc.view(M, 1))
        score = torch.where((L > 0) & (R > 0), score.clamp(0, 1), 0)
        best = torch.maximum(best, score.max(1).values)
    return dict(score=best, feature=None, threshold=None, threshold_index=None)


# ------------------------------------------------------------------------------------------- prepare
def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    ctx = context()
    n, w, h, C = case["frames"], case["width"], case["height"], case["classes"]
    st = dict(case=case, kind=kind)
    if kind in ("predict", "graph", "refine", "refine_train"):
        fill, lab = case.get("fill", False), case.get("lab", False)
        st["forest"] = make_forest(*forest_arrays(seed, case["trees"], C, w, h, fill, lab), fill, lab)
        rgb, depth, labels = scene(seed, n, w, h, 40, C)
    if kind == "graph":
        st["graph"] = cf.PredictGraph(st["forest"], n, w, h, probabilities=False)
        st["graph"].rgb[...] = _host(rgb)
        st["graph"].depth[...] = _host(depth).view(np.uint16)
        return st
    if kind in ("predict", "refine", "refine_train"):
        st["ds"] = cf.Dataset(ctx, n, w, h)
        st["labels"] = torch.empty(n, h, w, dtype=torch.uint8, device=DEV)
        st["probs"] = None
        if case.get("probs", kind == "refine"):
            st["probs"] = torch.empty(n, C, h, w, dtype=torch.float32, device=DEV)
        st["rgb"], st["depth"] = rgb, depth
        torch.cuda.synchronize()
        st["ds"].upload_raw(rgb.data_ptr(), (depth.data_ptr(), n), fill_depth=fill, cie_lab=lab)
        ctx.synchronize()
    if kind in ("refine", "refine_train"):
        st["net"] = cf.Refiner(ctx, C, hidden=case["hidden"], epochs=1, batch=case.get("batch", 4096),
                               pixels_per_image=case.get("pixels", 20000), seed=seed % 1000003 + 1)
        st["params"] = refiner_params(case, seed)
        st["net"].params(new=st["params"])
        st["truth"] = _host(labels)
    if kind in ("forest", "tree"):
        count = n * case["per_image"] * (2 if case.get("flip") == 2 else 1)
        st["tree"], st["most_nodes"] = {}, min(2 * count + 1, 8 * count // case["min_samples"] + 64)
    if kind == "forest":
        rgb, depth, labels = scene(seed, n, w, h, case["cells"], C)
        st["frames"] = _host(rgb), _host(depth).view(np.uint16), _host(labels)
        ignored = np.zeros(C, np.uint8)
        ignored[0] = 1
        st["ignored"] = ignored
        st["config"] = cf.TrainConfig(feature_count=case["features"], thresholds=case["thresholds"],
                                      samples_per_image=case["per_image"], max_depth=case["depth"],
                                      min_sample_count=case["min_samples"], box_radius=BOX, region_size=REGION,
                                      random_seed=seed % 65521, sampler=1)
    if kind == "tree":
        rgb, depth, labels = scene(seed, n, w, h, case["cells"], C)
        st["samples"] = sample_rows(sample_pixels(_generator(seed + 5), depth, labels, case["per_image"]), case["flip"])
        st["config"] = cf.TrainConfig(feature_count=case["features"], thresholds=case["thresholds"],
                                      max_depth=case["depth"], min_sample_count=case["min_samples"], box_radius=BOX,
                                      region_size=REGION)
        st["counter"] = seed % 1000003
    if kind == "level":
        rgb, depth, s, counts, f, thr = level_inputs(case, seed)
        st["samples"] = sample_rows(s, case["flip"])
        st["offsets"] = np.concatenate([[0], np.cumsum(_host(counts))]).astype(np.int64)
        st["features"] = _host(torch.stack([f[k] for k in ROWS])).astype(np.int8)
        st["thresholds"] = np.ascontiguousarray(_host(thr))
    if kind in ("tree", "level"):
        torch.cuda.synchronize()
        st["ds"] = cf.Dataset(ctx, n, w, h)
        st["ds"].upload_raw_device(rgb.data_ptr(), depth.data_ptr(), n)
        ctx.synchronize()
    return st


# ------------------------------------------------------------------------------------------- run
def run(st):
    case, kind = st["case"], st["kind"]
    n = case["frames"]
    if kind == "predict":
        ds, rgb, depth = st["ds"], st["rgb"], st["depth"]
        if case["fill"] or case["lab"]:
            # raw frames arriving on the device: preprocessing and integral images are part of the call
            ds.upload_raw(rgb.data_ptr(), (depth.data_ptr(), n), fill_depth=case["fill"], cie_lab=case["lab"])
        else:
            ds.upload_raw_device(rgb.data_ptr(), depth.data_ptr(), n)
        probs = st["probs"]
        st["forest"].predict_dataset(ds, 0, n, 0 if probs is None else probs.data_ptr(), st["labels"].data_ptr())
        return dict(labels=st["labels"]) if probs is None else dict(labels=st["labels"], probs=probs)
    if kind == "graph":
        st["graph"].run()
        return dict(labels=st["graph"].labels)
    if kind == "refine":
        st["net"].predict(st["forest"], st["ds"], 0, n, st["probs"].data_ptr(), st["labels"].data_ptr())
        return dict(labels=st["labels"], probs=st["probs"])
    if kind == "refine_train":
        net = st["net"]
        net.params(new=st["params"])
        losses = net.train(st["forest"], st["ds"], 0, n, st["truth"])
        return dict(losses=losses, params=net.params())
    if kind == "forest":
        rgb, depth, labels = st["frames"]
        trees = cf.train_forest(context(), rgb, depth, labels, case["classes"], st["config"], 1, ignored=st["ignored"])
        return [_tree(st, t) for t in trees]
    if kind == "tree":
        tree, counter = cf.train_tree(st["ds"], st["samples"], case["classes"], st["config"],
                                      seed_counter=st["counter"])
        return dict(_tree(st, tree), counter=counter)
    best = cf.evaluate_best_splits(st["ds"], st["offsets"], st["samples"], case["classes"], st["features"],
                                   st["thresholds"])
    return {k: np.ascontiguousarray(best[k]) for k in ("score", "feature", "threshold", "threshold_index")}


def _tree(st, tree):
    """A tree's node arrays, placed in arrays that hold any tree of the case."""
    a = tree.arrays()
    tree.close()
    for k, v in a.items():
        if k not in st["tree"]:
            st["tree"][k] = np.zeros((st["most_nodes"],) + v.shape[1:], v.dtype)
        st["tree"][k][:len(v)] = v
    return dict(st["tree"], nodes=len(a["left"]))


# ------------------------------------------------------------------------------------------- exact
def refiner_params(case, seed):
    """W1 [hidden][D], b1, W2 [C][hidden], b2 in one float32 array."""
    C, H = case["classes"], case["hidden"]
    D = 3 * C + 2
    r = np.random.default_rng(seed)
    a1, a2 = math.sqrt(6 / (D + H)), math.sqrt(6 / (H + C))
    return np.concatenate([r.uniform(-2 * a1, 2 * a1, H * D), r.uniform(-0.1, 0.1, H), r.uniform(-2 * a2, 2 * a2, C * H),
                           r.uniform(-0.1, 0.1, C)]).astype(np.float32)


def box_mean(p, r):
    """Means over (2r + 1)^2 boxes clipped at the border, [planes][h][w] in 64 bits."""
    h, w = p.shape[1:]
    s = torch.nn.functional.pad(p.cumsum(1).cumsum(2), (1, 0, 1, 0))
    y, x = torch.arange(h, device=DEV), torch.arange(w, device=DEV)
    y0, y1 = (y - r).clamp_min(0), (y + r + 1).clamp_max(h)
    x0, x1 = (x - r).clamp_min(0), (x + r + 1).clamp_max(w)
    box = s[:, y1][:, :, x1] - s[:, y0][:, :, x1] - s[:, y1][:, :, x0] + s[:, y0][:, :, x0]
    return box / ((y1 - y0).view(-1, 1) * (x1 - x0).view(1, -1)).double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "level":
        return level_exact(case, seed)
    if kind not in ("predict", "refine") or not case.get("probs", kind == "refine"):
        return None        # whole numbers alone, or a training that draws from the framework's own random streams
    n, w, h, C = case["frames"], case["width"], case["height"], case["classes"]
    fill, lab = case.get("fill", False), case.get("lab", False)
    grown, prior = forest_arrays(seed, case["trees"], C, w, h, fill, lab)
    rgb, depth, _ = scene(seed, n, w, h, 40, C)
    out = torch.empty(n, C, h, w, dtype=torch.float64, device=DEV)
    for i in range(n):
        ints = integrals(rgb[i:i + 1], depth[i:i + 1], fill, lab)
        out[i] = forest_exact(grown, prior, ints, 0)
        if kind == "refine":
            p = out[i].clone()
            p[p.isnan()] = 0
            d = divided(ints[3][0].double(), 1000)
            H, D = case["hidden"], 3 * C + 2
            prm = torch.from_numpy(refiner_params(case, seed)).to(DEV).double()
            W1, b1, W2, b2 = prm.split([H * D, H, C * H, C])
            X = torch.cat([p, box_mean(p, 4), box_mean(p, 16), (d / 5)[None], (d > 0).double()[None]]).reshape(D, -1)
            z = W2.view(C, H) @ (W1.view(H, D) @ X + b1[:, None]).relu() + b2[:, None]
            out[i] = z.softmax(0).view(C, h, w)
    return dict(labels=None, probs=out)


# ------------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    px = case["frames"] * case["width"] * case["height"]
    C = case["classes"]
    if kind in ("predict", "graph"):
        # raw frames in; labels and probabilities out; about 12 two-box responses of 25 operations per tree
        out = 1 + (4 * C if case.get("probs") else 0)
        return dict(bytes=px * (5 + out), flops=px * (case["trees"] * 12 * 25 + 2 * C))
    if kind == "refine":
        D, H = 3 * C + 2, case["hidden"]
        return dict(bytes=px * (20 + 4 * C + 1), flops=px * 2 * (D * H + H * C))
    if kind == "refine_train":
        D, H = 3 * C + 2, case["hidden"]
        rows = case["frames"] * case["pixels"]
        return dict(bytes=px * 21 + rows * (D + 1) * 4, flops=6 * rows * (D * H + H * C) + px * 300 * case["trees"])
    evals = case["frames"] * case["per_image"] * case["features"] * (2 if case.get("flip") == 2 else 1)
    samples = case["frames"] * case["per_image"] * 16
    if kind == "level":
        # frames and samples read once; a response and its place among the thresholds per evaluation
        return dict(bytes=px * 20 + samples, flops=evals * 25)
    levels = 8 if kind == "forest" else 10     # levels that hold about all samples
    return dict(bytes=px * 20 + samples * levels, flops=evals * 25 * levels)
