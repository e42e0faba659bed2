"""The work that the speed of this package is measured on.

A case is one forward pass, or one forward and backward pass, of a network or a layer on a batch of voxelised surfaces:
what a program that uses the package calls for every new batch.  Every pass starts from coordinates, so it builds a fresh
Metadata (site hash and rulebooks), as a program with a new batch does; weights, BatchNorm statistics and what the
package keeps for them stay from pass to pass, as they do in such a program.

`listed()` gives the named cases, `draw(rng)` one more of the same ranges.  Inputs come from generators on the GPU with the
shapes of the package's synthetic workloads (``sparseconvnet_b200/workloads.py``): indoor rooms made of box and cylinder
surfaces, 2-D strokes, superquadric surfaces, moving sphere shells, shells with plane patches.
"""
import math

import numpy as np
import torch

import sparseconvnet_b200 as scn
from sparseconvnet_b200 import workloads

CLASSES = 20
DEVICE = "cuda"


def listed():
    return [
        # The benchmark's workload: semantic segmentation of eight rooms at once, a 3-D U-Net of seven levels, batch already
        # on the GPU, fp32-class tensor-core arithmetic.  Throughput serving.
        dict(name="unet_8_rooms", kind="unet", samples=8, voxels=200000, m=32, reps=2, levels=7, residual=False,
             precision="tf32x3", coords="cuda"),
        # One room that has just been scanned, coordinates on the host as the InputLayer of the reference takes them.
        # Interactive segmentation: the same launches as the batch above on an eighth of the rows.
        dict(name="unet_1_room_host", kind="unet", samples=1, voxels=200000, m=32, reps=2, levels=7, residual=False,
             precision="tf32x3", coords="cpu"),
        # The package as it comes (fp32 is its default precision), an odd number of voxels.
        dict(name="unet_2_rooms_fp32", kind="unet", samples=2, voxels=137001, m=32, reps=2, levels=7, residual=False,
             precision="fp32", coords="cuda"),
        # Per-point segmentation of scans: several points per voxel, averaged by the InputLayer and handed back by the
        # OutputLayer; the small U-Net (16 planes per level, one block) in its residual form.
        dict(name="scan_points", kind="scan", samples=4, points=250000, m=16, reps=1, levels=7, residual=True,
             precision="tf32x3", coords="cuda"),
        # A training step's forward and backward pass on two rooms, without the optimizer: a U-Net of four levels (with more,
        # the few sites of the deepest ones decide how far the gradients of two correct programs lie apart).
        dict(name="unet_train", kind="unet_train", samples=2, voxels=200000, m=32, reps=1, levels=4, residual=False,
             precision="tf32x3", coords="cpu"),
        # A single layer on a new cloud, 3-D, 27 offsets: hash, rulebook and convolution each count.
        dict(name="layer_32_32", kind="layer", samples=1, sites=267011, size=256, nin=32, nout=32, precision="tf32x3",
             train=False, coords="cuda"),
        # A layer of an encoder on its own with its gradients, at a ragged size and other plane counts.
        dict(name="layer_64_96_train", kind="layer", samples=1, sites=131071, size=211, nin=64, nout=96, precision="tf32x3",
             train=True, coords="cuda"),
        # Handwriting classification, one character: the smallest call, all launches and host work.
        dict(name="strokes_1", kind="strokes", samples=1, precision="fp32", train=False, coords="cpu"),
        # The same network on a batch of a hundred characters.
        dict(name="strokes_100", kind="strokes", samples=100, precision="fp32", train=False, coords="cpu"),
        # ... and its training step.
        dict(name="strokes_100_train", kind="strokes", samples=100, precision="fp32", train=True, coords="cpu"),
        # Part segmentation of sixteen shapes with a pre-activated ResNet (overlapping strided layers, pooling).
        dict(name="shapes_16", kind="shapes", samples=16, precision="fp32", coords="cuda"),
        # Space-time stack: 81 offsets, 64 planes, bf16.
        dict(name="stack4d_4", kind="stack4d", samples=4, sites=373000, layers=4, precision="bf16", coords="cuda"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["unet", "unet", "unet_train", "scan", "layer", "layer", "strokes", "shapes", "stack4d"])
    coords = rng.choice(["cuda", "cpu"])
    if kind == "unet":
        m = rng.choice([16, 32, 32, 48])
        precision = rng.choice(["tf32x3", "tf32x3", "bf16", "tf32", "fp32"])
        most = {"fp32": 2, "tf32": 4}.get(precision, 8)
        samples = rng.randint(1, most if m < 48 else max(1, most // 2))
        return dict(kind=kind, samples=samples, voxels=_log_int(rng, 12000, 200000), m=m, reps=rng.choice([1, 2]),
                    levels=rng.randint(3, 7), residual=rng.random() < 0.3, precision=precision, coords=coords)
    if kind == "unet_train":
        return dict(kind=kind, samples=rng.randint(1, 2), voxels=_log_int(rng, 12000, 160000), m=rng.choice([16, 32]),
                    reps=1, levels=rng.randint(3, 4), residual=rng.random() < 0.3,
                    precision=rng.choice(["tf32x3", "tf32x3", "fp32"]), coords=coords)
    if kind == "scan":
        return dict(kind=kind, samples=rng.randint(1, 4), points=_log_int(rng, 20000, 300000), m=rng.choice([16, 32]),
                    reps=1, levels=rng.randint(4, 7), residual=rng.random() < 0.5,
                    precision=rng.choice(["tf32x3", "fp32"]), coords=coords)
    if kind == "layer":
        sites = _log_int(rng, 6000, 300000)
        return dict(kind=kind, samples=rng.randint(1, 2), sites=sites, size=256 if sites > 60000 else rng.randint(97, 256),
                    nin=rng.choice([1, 3, 16, 24, 32, 64, 96, 128]), nout=rng.choice([16, 24, 32, 64, 96, 128, 160]),
                    precision=rng.choice(["tf32x3", "bf16", "tf32", "fp32"]), train=rng.random() < 0.4, coords=coords)
    if kind == "strokes":
        return dict(kind=kind, samples=_log_int(rng, 1, 200), precision=rng.choice(["fp32", "tf32x3"]),
                    train=rng.random() < 0.4, coords=coords)
    if kind == "shapes":
        return dict(kind=kind, samples=rng.randint(1, 16), precision=rng.choice(["fp32", "tf32x3"]), coords=coords)
    return dict(kind=kind, samples=rng.randint(1, 4), sites=_log_int(rng, 40000, 373000), layers=rng.randint(1, 4),
                precision=rng.choice(["bf16", "tf32x3"]), coords=coords)


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _grid(*ranges):
    """All points of a box of integer ranges (lo, hi), hi exclusive: int64 [n, len(ranges)]."""
    axes = [torch.arange(int(a), int(b), device=DEVICE) for a, b in ranges]
    return torch.stack([g.reshape(-1) for g in torch.meshgrid(*axes, indexing="ij")], 1)


def _unique(coords, size):
    """The distinct rows of non-negative coordinates below `size`, in lexicographic order."""
    key = coords[:, 0]
    for d in range(1, coords.shape[1]):
        key = key * size + coords[:, d]
    key = torch.unique(key)
    out = []
    for _ in range(coords.shape[1]):
        out.append(key % size)
        key = key // size
    return torch.stack(out[::-1], 1)


def _box(lo, hi):
    parts = []
    for axis in range(3):
        for at in (lo[axis], hi[axis]):
            r = [(lo[d], hi[d] + 1) for d in range(3)]
            r[axis] = (at, at + 1)
            parts.append(_grid(*r))
    return torch.cat(parts)


def _cylinder(cx, cy, r, z1):
    p = _grid((cx - r - 1, cx + r + 2), (cy - r - 1, cy + r + 2))
    d = ((p[:, 0] - cx) ** 2 + (p[:, 1] - cy) ** 2).double().sqrt()
    ring, disc = p[(d - r).abs() < 0.6], p[d <= r]
    z = torch.arange(1, z1 + 1, device=DEVICE)
    side = torch.cat([ring.repeat_interleave(z.numel(), 0), z.repeat(ring.shape[0])[:, None]], 1)
    return torch.cat([side, torch.cat([disc, torch.full((disc.shape[0], 1), z1, device=DEVICE)], 1)])


def _room(rng, voxels):
    """Floor, ceiling, walls and 10 to 30 box and cylinder surfaces of an indoor scan at 2 cm, thinned to `voxels` by
    keeping whole 8^3 blocks (the last one in part); a small target makes a smaller room first."""
    s = min(1.0, max(0.3, (voxels / 200000.0) ** 0.5))
    ext = [max(60, int(rng.integers(300, 601) * s)), max(60, int(rng.integers(300, 601) * s)),
           max(50, int(rng.integers(125, 151) * s))]
    parts = [_box([0, 0, 0], [e - 1 for e in ext])]
    for _ in range(int(rng.integers(10, 31))):
        if rng.random() < 0.6:
            sz = [max(8, int(rng.integers(20, 120) * s)) for _ in range(2)] + [max(8, int(rng.integers(20, 100) * s))]
            sz = [min(v, e - 4) for v, e in zip(sz, ext)]
            lo = [int(rng.integers(1, ext[0] - sz[0] - 1)), int(rng.integers(1, ext[1] - sz[1] - 1)), 1]
            parts.append(_box(lo, [a + b for a, b in zip(lo, sz)]))
        else:
            r = max(5, int(rng.integers(8, 40) * s))
            parts.append(_cylinder(int(rng.integers(r + 2, ext[0] - r - 2)), int(rng.integers(r + 2, ext[1] - r - 2)), r,
                                   min(ext[2] - 2, max(5, int(rng.integers(20, 110) * s)))))
    c = torch.cat(parts)
    c = c[((c >= 0) & (c < torch.tensor(ext, device=DEVICE))).all(1)]
    c = _unique(c, 1024)
    b = c // 8
    h = (b[:, 0] * 73856093) ^ (b[:, 1] * 19349663) ^ (b[:, 2] * 83492791) ^ int(rng.integers(1 << 30))
    keep = torch.sort((h * 2654435761) & 0xFFFFFFFF, stable=True)[1][:voxels]
    c = c[torch.sort(keep)[0]]
    return c + torch.tensor([int(rng.integers(0, 4096 - e)) for e in ext], device=DEVICE)


def _rooms(rng, samples, voxels):
    return [_room(rng, voxels) for _ in range(samples)]


def _shell(centre, radius, size):
    lo = [max(0, int(v - radius - 1)) for v in centre]
    hi = [min(size, int(v + radius + 2)) for v in centre]
    if any(b <= a for a, b in zip(lo, hi)):
        return torch.zeros(0, 3, dtype=torch.int64, device=DEVICE)
    p = _grid(*zip(lo, hi))
    d = (p.double() - torch.tensor(centre, device=DEVICE, dtype=torch.float64)).norm(dim=1)
    return p[(d - radius).abs() < 0.5]


def _cloud(rng, sites, size):
    """Sphere shells with a patch of a plane after every fifth, as many as make `sites` voxels, cut off there."""
    c = torch.zeros(0, 3, dtype=torch.int64, device=DEVICE)
    while c.shape[0] < sites:
        parts = [c] + [_shell([float(v) for v in rng.uniform(0, size, 3)], float(rng.uniform(8, 60)), size) for _ in range(5)]
        r = [(int(o), int(o) + 80) for o in rng.integers(0, size - 80, 3)]
        axis = int(rng.integers(0, 3))
        r[axis] = (r[axis][0], r[axis][0] + 1)
        c = _unique(torch.cat(parts + [_grid(*r)]), size)
    return c[:sites]


def _strokes(rng, samples):
    """Per sample 3 to 8 polylines of 4 to 12 vertices in 64 x 64, rasterised."""
    a, b, who = [], [], []
    for s in range(samples):
        for _ in range(int(rng.integers(3, 9))):
            v = rng.integers(0, 64, (int(rng.integers(4, 13)), 2))
            a.append(v[:-1])
            b.append(v[1:])
            who.append(np.full(len(v) - 1, s))
    a, b = (torch.from_numpy(np.concatenate(x)).to(DEVICE).double() for x in (a, b))
    who = torch.from_numpy(np.concatenate(who)).to(DEVICE)
    steps = (b - a).abs().amax(1).clamp(min=1)
    t = (torch.arange(64, device=DEVICE)[None] / steps[:, None]).clamp(max=1)
    p = torch.floor(a[:, None] + t[..., None] * (b - a)[:, None] + 0.5).long()
    p = torch.cat([who[:, None, None].expand(-1, 64, 1), p], 2).reshape(-1, 3)
    p = _unique(p, 256)
    return torch.cat([p[:, 1:], p[:, :1]], 1)


def _superquadric(rng, size=127):
    """Surface voxels of a randomly rotated |x/a|^e1 + |y/b|^e2 + |z/c|^e3 = 1."""
    e, sc = rng.uniform(0.3, 3.0, 3), rng.uniform(20, 60, 3)
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    ax = torch.arange(size, device=DEVICE, dtype=torch.float32) - (size - 1) / 2.0
    g = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1) @ torch.from_numpy(q.astype(np.float32)).to(DEVICE)
    f = sum((g[..., d].abs() / float(sc[d])) ** float(e[d]) for d in range(3))
    inside = f < 1.0
    pad = torch.nn.functional.pad(inside, (1, 1, 1, 1, 1, 1))
    core = inside.clone()
    for d in range(3):
        for at in (0, 2):
            sl = [slice(1, -1)] * 3
            sl[d] = slice(at, at + size)
            core &= pad[tuple(sl)]
    return (inside & ~core).nonzero()


def _sequence(rng, sites, size=256, frames=8):
    """Sphere shells that move with constant velocity, as many as make `sites` voxels over all frames, cut off there."""
    c = torch.zeros(0, 4, dtype=torch.int64, device=DEVICE)
    while c.shape[0] < sites:
        centre, radius = rng.uniform(60, size - 60, 3), float(rng.uniform(20, 35))
        vel = rng.uniform(1, 3, 3) * rng.choice([-1.0, 1.0], 3)
        parts = [c]
        for t in range(frames):
            p = _shell([float(v) for v in centre + vel * t], radius, size)
            parts.append(torch.cat([p, torch.full((p.shape[0], 1), t, device=DEVICE)], 1))
        c = _unique(torch.cat(parts), size)
    return c[:sites]


def _colours(coords, gen):
    """Three values per voxel that vary smoothly over the surfaces, with sensor noise."""
    x = coords[:, :3].float()
    base = torch.stack([torch.sin(x @ torch.rand(3, device=DEVICE, generator=gen) * 0.1) for _ in range(3)], 1)
    return 0.7 * base + 0.3 * (torch.rand(coords.shape[0], 3, device=DEVICE, generator=gen) * 2 - 1)


def _batch(parts):
    return torch.cat([torch.cat([c, torch.full((c.shape[0], 1), s, device=DEVICE)], 1) for s, c in enumerate(parts)])


# ---- networks ---------------------------------------------------------------------------------------------------------

def _unet(case):
    planes = [case["m"] * (i + 1) for i in range(case["levels"])]
    return scn.Sequential().add(scn.SubmanifoldConvolution(3, 3, case["m"], 3, False)).add(
        scn.UNet(3, case["reps"], planes, case["residual"])).add(scn.BatchNormReLU(case["m"]))


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(DEVICE).manual_seed(int(rng.integers(1 << 40)))
    torch.manual_seed(int(rng.integers(1 << 40)))  # the layers' own initialisation
    s = {"case": case, "head": None, "out": None, "labels": None}
    train = kind == "unet_train" or case.get("train", False)

    if kind in ("unet", "unet_train"):
        coords = _batch(_rooms(rng, case["samples"], case["voxels"]))
        feats = _colours(coords, gen)
        s["input"], s["net"] = scn.InputLayer(3, 4096, mode=4), _unet(case)
        s["net"].add(scn.NetworkInNetwork(case["m"], CLASSES, True))
    elif kind == "scan":
        parts = []
        for c in _rooms(rng, case["samples"], int(case["points"] * 0.7)):
            parts.append(c[torch.randint(0, c.shape[0], (case["points"],), device=DEVICE, generator=gen)])
        coords = _batch(parts)
        feats = _colours(coords, gen)
        s["input"], s["net"], s["out"] = scn.InputLayer(3, 4096, mode=4), _unet(case), scn.OutputLayer(3)
        s["head"] = torch.nn.Linear(case["m"], CLASSES)
    elif kind == "layer":
        coords = _batch([_cloud(rng, case["sites"], case["size"]) for _ in range(case["samples"])])
        feats = torch.randn(coords.shape[0], case["nin"], device=DEVICE, generator=gen)
        s["input"] = scn.InputLayer(3, case["size"], mode=0)
        s["net"] = scn.Sequential().add(scn.SubmanifoldConvolution(3, case["nin"], case["nout"], 3, False))
        if train:
            feats.requires_grad_(True)
            s["grad"] = torch.randn(coords.shape[0], case["nout"], device=DEVICE, generator=gen)
    elif kind == "strokes":
        coords = _strokes(rng, case["samples"])
        feats = torch.rand(coords.shape[0], 1, device=DEVICE, generator=gen) * 0.5 + 0.75
        s["net"] = scn.Sequential().add(scn.SparseVggNet(2, 1, [
            ["C", 8], ["C", 8], ["MP", 3, 2], ["C", 16], ["C", 16], ["MP", 3, 2], ["C", 24], ["C", 24], ["MP", 3, 2]])).add(
            scn.SubmanifoldConvolution(2, 24, 32, 3, False)).add(scn.BatchNormReLU(32)).add(scn.SparseToDense(2, 32))
        s["input"] = scn.InputLayer(2, s["net"].input_spatial_size(torch.LongTensor([10, 10])), mode=3)
        s["head"] = torch.nn.Linear(3200, 100)
        s["labels"] = torch.randint(0, 100, (case["samples"],), device=DEVICE, generator=gen)
    elif kind == "shapes":
        coords = _batch([_superquadric(rng) for _ in range(case["samples"])])
        feats = torch.rand(coords.shape[0], 1, device=DEVICE, generator=gen) * 0.5 + 0.75
        s["input"] = scn.InputLayer(3, 127, mode=3)
        s["net"] = scn.Sequential().add(scn.SubmanifoldConvolution(3, 1, 16, 3, False)).add(scn.MaxPooling(3, 3, 2)).add(
            scn.SparseResNet(3, 16, [["b", 16, 2, 1], ["b", 32, 2, 2], ["b", 64, 2, 2], ["b", 128, 2, 2]])).add(
            scn.NetworkInNetwork(128, 50, True)).add(scn.SparseToDense(3, 50))
    else:
        coords = _batch([_sequence(rng, case["sites"]) for _ in range(case["samples"])])
        feats = torch.randn(coords.shape[0], 64, device=DEVICE, generator=gen)
        s["input"], s["net"] = scn.InputLayer(4, [256, 256, 256, 8], mode=0), scn.Sequential()
        for _ in range(case["layers"]):
            s["net"].add(scn.SubmanifoldConvolution(4, 64, 64, 3, False)).add(scn.BatchNormReLU(64))

    if kind == "unet_train":
        # one class per piece of surface, some far more frequent than others
        piece = (coords[:, :3] // 24).float() @ torch.rand(3, device=DEVICE, generator=gen)
        s["labels"] = ((piece * 3.7).frac() ** 2 * CLASSES).long()
    workloads.randomize(s["net"], seed % 1000003)
    s["net"].to(DEVICE).train(train)
    if s["head"] is not None:
        s["head"].to(DEVICE).train(train)
    if not train:
        for module in (s["net"], s["head"]):
            if module is not None:
                module.requires_grad_(False)
    s["train"], s["feats"] = train, feats
    s["coords"] = coords.contiguous() if case["coords"] == "cuda" else coords.cpu()
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------------

def _forward(s):
    x = s["net"](s["input"]([s["coords"], s["feats"]]))
    if s["out"] is not None:
        return s["head"](s["out"](x))
    if s["case"]["kind"] == "strokes":
        return s["head"](x.view(x.size(0), -1))
    return x if torch.is_tensor(x) else x.features


def _flat(tensors):
    return torch.cat([t.reshape(-1) for t in tensors])


def run(s):
    case = s["case"]
    scn.set_precision(case["precision"])
    if not s["train"]:
        with torch.no_grad():
            return _forward(s)
    # training: what a program does between two optimizer steps.  The input gradients of the convolutions run in the
    # precision of the forward pass.
    scn.set_backward_precision(case["precision"])
    modules = [m for m in (s["net"], s["head"]) if m is not None]
    for m in modules:
        m.zero_grad(set_to_none=True)
    y = _forward(s)
    if case["kind"] == "layer":
        s["feats"].grad = None
        y.backward(s["grad"])
        return [y.detach(), s["feats"].grad, s["net"][0].weight.grad]
    loss = torch.nn.functional.cross_entropy(y, s["labels"])
    loss.backward()
    # the gradient of every weight matrix on its own, those of the many short vectors and the running statistics joined
    params = [p for m in modules for p in m.parameters()]
    stats = [b for m in modules for b in m.buffers()]
    return [loss.detach()] + [p.grad for p in params if p.dim() > 1] + [_flat([p.grad for p in params if p.dim() == 1]),
                                                                         _flat(stats)]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

# Sites of a level over those of the level above it, and rules per site of a filter of size 3 (surfaces of rooms): counted
# on the generators' output.
_ROOM_RATIO = [1.0, 0.295, 0.309, 0.416, 0.403, 0.302, 0.30]
_ROOM_RULES = [8.9, 8.1, 6.4, 7.0, 10.5, 15.2, 18.0]


def _unet_work(case, sites):
    """(multiply-adds, parameters) of the U-Net on `sites` voxels."""
    m, reps, levels = case["m"], case["reps"], case["levels"]
    n, counts = float(sites), []
    for r in _ROOM_RATIO[:levels]:
        n *= r
        counts.append(n)
    macs, params = counts[0] * _ROOM_RULES[0] * 3 * m, 27.0 * 3 * m
    inner = 2 if case["residual"] else 1
    for l in range(levels):
        p, rules = m * (l + 1), counts[l] * _ROOM_RULES[l]
        blocks = [(p, p)] * reps * inner
        if l + 1 < levels:
            blocks += [(2 * p, p)] + [(p, p)] * (reps * inner - 1)
            q = m * (l + 2)
            macs += 2 * counts[l] * p * q
            params += 16 * p * q
        for a, b in blocks:
            macs += rules * a * b
            params += 27.0 * a * b
    return macs, params


def work(case):
    """Bytes: coordinates and features in, results out, parameters once (read, and their gradients written in training).
    Multiply-adds: two operations each; a backward pass takes twice the forward pass's."""
    kind, dim = case["kind"], 3
    train = kind == "unet_train" or case.get("train", False)
    if kind in ("unet", "unet_train"):
        rows = sites = case["samples"] * case["voxels"]
        macs, params = _unet_work(case, sites)
        nin, out = 3, sites * (0 if train else CLASSES)
    elif kind == "scan":
        rows = case["samples"] * case["points"]
        sites = 0.5 * rows
        macs, params = _unet_work(case, sites)
        nin, out = 3, rows * CLASSES
    elif kind == "layer":
        rows = sites = case["samples"] * case["sites"]
        nin, params = case["nin"], 27.0 * case["nin"] * case["nout"]
        macs, out = sites * 10.4 * case["nin"] * case["nout"], sites * case["nout"]
        if train:
            out += sites * (case["nin"] + case["nout"])
    elif kind == "strokes":
        dim, nin = 2, 1
        rows = sites = case["samples"] * 930.0
        macs = sites * (5 * (8 + 64) + 0.55 * 7 * (128 + 256) + 0.3 * 8 * (384 + 576) + 0.12 * 8.5 * 768) + case["samples"] * 320000.0
        params, out = 9.0 * (8 + 64 + 128 + 256 + 384 + 576 + 768) + 320000.0, (0 if train else case["samples"] * 100.0)
    elif kind == "shapes":
        nin, rows = 1, case["samples"] * 11500.0
        sites = rows
        macs, params, n = rows * 9.1 * 16, 27.0 * 16, rows * 0.5
        for i, p in enumerate([16, 32, 64, 128]):
            if i:
                n *= 0.35
                macs += 2 * n * 10 * p * p / 2
                params += 27.0 * p * p
            macs += (4 if i == 0 else 3) * n * 11 * p * p
            params += 27.0 * p * p * (4 if i == 0 else 3)
        out = case["samples"] * 50.0 * 343
    else:
        dim, nin = 4, 64
        rows = sites = case["samples"] * case["sites"]
        macs, params, out = sites * 17.4 * 64 * 64 * case["layers"], 81.0 * 64 * 64 * case["layers"], sites * 64
    passes = 3 if train else 1
    bytes_ = rows * (dim + 1) * 8 + rows * nin * 4 + params * 4 * (2 if train else 1) + out * 4
    return {"bytes": float(bytes_), "flops": 2.0 * macs * passes}


def tolerance(case):
    """Relative to the 2-norm.  fp32 sums of a few hundred products, and the split forms of the fp32-class mode (2^-17 of a
    product dropped), through up to some sixty layers; single-pass tf32 and bf16 keep 10 and 8 bits of the operands.
    In a network's backward pass an activation within rounding of zero has its whole gradient on one side of the ReLU and
    none on the other: a share of the entries as large as the forward pass's relative error, so the 2-norm of the
    difference goes with the square root of that error, and one site of a coarse level shows in single weights.  The two
    fp32-class forms of the package's own convolutions differ by up to 1.5e-2 and 0.8 in the U-Net, 7e-3 in the classifier."""
    precision, kind = case["precision"], case["kind"]
    if kind == "unet_train":
        return {"rel": 0.03, "max": 0.99}
    if kind == "strokes" and case["train"]:
        return {"rel": 0.02, "max": 0.5}
    return {"rel": {"fp32": 1e-5, "tf32x3": 5e-5, "tf32": 3e-3, "bf16": 1e-2}[precision]}
