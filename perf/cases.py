"""Performance cases: the calls a user of this package makes, over the sizes it is used at.

A case names an operation, the scene it works on (grid vertices minus one per
axis, channels, decoder, occupancy) and how many rays go through it:

  intersect  the padded traversal operators (dense or occupancy-masked)
  integrate  the feature integrator, forward and backward through autograd
  render     a field's forward without gradients, in any decoder form
  train      a training step, loss and gradients, eager or captured
  alpha      occupancy extraction: the largest rendering weight per voxel
  frame      a real-time frame of a converted model
  serve      a mixed batch of render requests over resident scenes

Scenes are synthetic and seeded: blob occupancy, Gaussian features, decoders
with the default Linear initialisation whose density layer is scaled so that
rays become opaque along the way, cameras on a sphere around the grid.
"""
import math

import torch

from diver_gb300.decoder import Decoder, pack_realtime, premultiply_features
from diver_gb300.graphs import TrainStepGraph
from diver_gb300.integrator import integrate
from diver_gb300.prune import extract_alpha_map
from diver_gb300.ray_voxel_intersection import masked_intersect, ray_voxel_intersect
from diver_gb300.realtime import RealtimeModel
from diver_gb300.renderer import DIVeRField, l2_loss
from diver_gb300.serving import GpuRenderer, Request, Residency, serve

GRID_SIZE = 2.8   # world extent of the longest grid axis
L_S = 1e-5        # weight of the sparsity term in the training loss
DEV = "cuda"


def listed():
    return [
        # The padded traversal operator on one training batch: 4096 rays
        # through the 256^3 occupancy grid.
        dict(name="intersect_train_batch", op="intersect", n="256", occ=0.6, h=64, w=64, masked=True),
        # The integrator as its own operator on 64-channel features, forward and
        # backward, for an odd number of segments of a mid-sized grid.
        dict(name="integrate_64ch", op="integrate", n="128", c=64, occ=0.6, segments=100003),
        # An interactive preview tile of the small scene in the accurate form: the
        # call is all launches and latency.
        dict(name="tile_fp32", op="render", n="64", c=32, kind="diver32", occ=0.3, h=33, w=31, form="fp32"),
        # Occupancy extraction over one 200x200 view in the reference's 4000-ray batches.
        dict(name="alpha_map_view", op="alpha", n="128", c=32, kind="diver32", occ=0.6, h=200, w=200, form="fp32"),
        # A full evaluation frame of the DIVeR32 scene with the BF16 decoder.
        dict(name="frame_bf16", op="render", n="256", c=32, kind="diver32", occ=0.6, h=800, w=800, form="bf16"),
        # A DIVeR64 view over 64-channel features with the FP16 decoder, ragged size.
        dict(name="view_diver64_fp16", op="render", n="256", c=64, kind="diver64", occ=0.6, h=399, w=401, form="fp16"),
        # An accurate-form render (split BF16) of part of a frame over the wide grid.
        dict(name="chunk_split_wide", op="render", n="320,320,160", c=32, kind="diver32", occ=0.25, h=256, w=257,
             form="bf16s"),
        # The training step at the reference's batch size, captured once and replayed.
        dict(name="train_split_graph", op="train", n="256", c=32, kind="diver32", occ=0.6, h=64, w=64, form="bf16s",
             graph=True),
        # A plain FP32 training step, eager, with an odd batch on a mid-sized grid.
        dict(name="train_fp32_odd", op="train", n="160", c=32, kind="diver32", occ=0.5, h=37, w=55, form="fp32",
             graph=False),
        # DIVeR64 training in the accurate form, eager.
        dict(name="train_diver64_split", op="train", n="192", c=64, kind="diver64", occ=0.6, h=32, w=32, form="bf16s",
             graph=False),
        # A real-time frame of a pruned scene at the reference's viewer resolution.
        dict(name="realtime_frame", op="frame", n="256", c=32, kind="diver32", occ=0.1, h=800, w=800),
        # Six requests of mixed resolution over two resident scenes.
        dict(name="serve_mixed", op="serve", n="128", c=32, kind="diver32", occ=0.4, h=400, w=400, form="bf16",
             requests=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["intersect", "integrate", "render", "render", "render", "train", "train", "train", "alpha",
                     "frame", "serve"])
    n = _log(rng, 48, 256)
    occ = round(rng.uniform(0.1, 0.6), 3)
    kind, c = rng.choice([("diver32", 32), ("diver32", 32), ("diver64", 64), ("diver64", 32)])

    def image(lo, hi):
        """h, w of an image of about lo..hi rays (log-uniform), any aspect."""
        rays = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a = math.exp(rng.uniform(-0.5, 0.5))
        return dict(h=max(1, int(math.sqrt(rays * a))), w=max(1, int(math.sqrt(rays / a))))

    grid = str(n)
    if op in ("render", "train") and rng.random() < 0.25:  # per-axis extents
        grid = "%d,%d,%d" % (n, max(32, int(n * rng.uniform(0.4, 1.0))), max(32, int(n * rng.uniform(0.4, 1.0))))
    if op == "intersect":
        return dict(op=op, n=grid, occ=occ, masked=rng.random() < 0.6, **image(64, 16384))
    if op == "integrate":
        return dict(op=op, n=grid, c=c, occ=occ, segments=_log(rng, 3000, 600000))
    if op == "render":
        form = rng.choice(["bf16", "bf16", "fp16", "fp32", "bf16s"])
        most = {"bf16": 400000, "fp16": 400000, "fp32": 40000, "bf16s": 100000}[form] // (2 if c * (kind != "diver32") else 1)
        return dict(op=op, n=grid, c=c, kind=kind, occ=occ, form=form, **image(256, most))
    if op == "train":
        form = rng.choice(["bf16s", "bf16s", "fp32", "bf16", "fp16"])
        return dict(op=op, n=grid, c=c, kind=kind, occ=occ, form=form, graph=rng.random() < 0.5,
                    **image(256, 4096 if kind == "diver32" and form != "fp32" else 1024))
    if op == "alpha":
        return dict(op=op, n=grid, c=c, kind=kind, occ=occ, form=rng.choice(["fp32", "bf16"]), **image(1000, 20000))
    if op == "frame":
        kind = rng.choice(["diver32", "diver32", "diver64"])
        return dict(op=op, n=str(rng.choice([64, 128, 192, 256])), c=32, kind=kind, occ=round(rng.uniform(0.03, 0.2), 3),
                    **image(4000, 600000))
    return dict(op=op, n=str(min(n, 160)), c=32, kind="diver32", occ=occ, form="bf16", requests=rng.randint(2, 6),
                **image(10000, 160000))


# --- scenes ---------------------------------------------------------------------

def _dims(case):
    v = [int(x) for x in case["n"].split(",")]
    return tuple(v) if len(v) == 3 else (v[0],) * 3


def _place(dims):
    vs = GRID_SIZE / max(dims)
    return tuple(-0.5 * vs * n for n in dims), vs


def _mask(dims, occ, g):
    """Occupancy [nz][ny][nx]: the `occ` share of the cells where a sum of 16 Gaussian blobs is largest."""
    lo, vs = _place(dims)
    f = torch.zeros(dims[2], dims[1], dims[0], device=DEV)
    par = torch.rand(16, 5, generator=g, device=DEV)
    for k in range(16):
        e = [torch.exp(-((lo[a] + (torch.arange(dims[a], device=DEV) + 0.5) * vs - (par[k, a] * 2 - 1) * 0.8) ** 2)
                       / (2 * (0.25 + 0.35 * par[k, 3]) ** 2)) for a in range(3)]
        f += (0.5 + par[k, 4]) * e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
    sub = f[::2, ::2, ::2].reshape(-1)
    return f > torch.kthvalue(sub, max(1, int((1 - occ) * sub.numel()))).values


def _layers(kind, c, g):
    """Decoder layers with the default Linear initialisation, the density row scaled and shifted so that about half of
    the voxels are empty (density below zero) and a ray becomes opaque within some tens of the others."""
    w, depth = (32, 2) if kind == "diver32" else (64, 1)
    sizes = [(c, w)] + [(w, w)] * (depth - 1) + [(w, w + 1), (w + 27, w), (w, 3)]
    out = []
    for i, (a, b) in enumerate(sizes):
        k = torch.rand(b, a + 1, generator=g, device=DEV) * 2 - 1
        k /= math.sqrt(a)
        if i == depth:
            h = torch.randn(4096, c, generator=g, device=DEV) * 0.1
            for m, v in out:
                h = torch.relu(h @ m.t() + v)
            sigma = h @ k[0, :a]
            k[0] *= 0.15 / sigma.std()
            k[0, a] = 0.02 - (sigma * (0.15 / sigma.std())).mean()
        out.append((k[:, :a].contiguous(), k[:, a].contiguous()))
    return out


def _scene(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    dims = _dims(case)
    s = {"dims": dims, "g": g, "mask": _mask(dims, case["occ"], g)}
    if "c" in case:
        s["voxels"] = torch.randn(dims[2] + 1, dims[1] + 1, dims[0] + 1, case["c"], generator=g, device=DEV) * 0.2
    if "kind" in case:
        s["layers"] = _layers(case["kind"], case["c"], g)
    return s


def _camera(g):
    """Camera-to-world [3, 4] (FP32, host) of a camera on the radius-4 sphere looking at the origin."""
    eye = torch.randn(3, generator=g, device=DEV).double().cpu()
    eye = eye / eye.norm() * 4.0
    back = eye / 4.0
    right = torch.linalg.cross(torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64), back)
    right = right / right.norm()
    up = torch.linalg.cross(back, right)
    return torch.stack([right, up, back, eye], 1).float()


def _directions(c2w, h, w, focal):
    """Unit directions [h * w, 3] in FP64."""
    i = torch.arange(h * w, device=DEV)
    x = (i % w).double() + 0.5
    y = (i // w).double() + 0.5
    d = torch.stack([(x - w / 2) / focal, -(y - h / 2) / focal, -torch.ones_like(x)], -1)
    d = d @ c2w[:, :3].to(DEV).double().t()
    return d / d.norm(dim=-1, keepdim=True)


def _rays(case, s):
    c2w = _camera(s["g"])
    d = _directions(c2w, case["h"], case["w"], 1.2 * max(case["h"], case["w"])).float().contiguous()
    return c2w[:, 3].to(DEV).expand(d.shape).contiguous(), d


def _batch(case, s):
    """A training batch: rays of several cameras towards points inside the grid, and target colours."""
    b = case["h"] * case["w"]
    eyes = torch.stack([_camera(s["g"])[:, 3] for _ in range(8)]).to(DEV)
    pick = torch.randint(0, 8, (b,), generator=s["g"], device=DEV)
    half = torch.tensor(s["dims"], device=DEV) / max(s["dims"]) * (0.35 * GRID_SIZE)
    at = (torch.rand(b, 3, generator=s["g"], device=DEV) * 2 - 1) * half
    o = eyes[pick].contiguous()
    d = at - o
    return o, (d / d.norm(dim=-1, keepdim=True)).contiguous(), torch.rand(b, 3, generator=s["g"], device=DEV)


def _field(case, s):
    lo, vs = _place(s["dims"])
    cubic = len(set(s["dims"])) == 1
    return DIVeRField(s["voxels"], Decoder(case["kind"], case["c"], s["layers"]), s["mask"], lo[0] if cubic else lo, vs)


def _realtime(case, s):
    """The converted model: the table of the corners of the occupied voxels and the folded decoder."""
    n = s["dims"][0]
    m = torch.nn.functional.pad(s["mask"], (1, 1, 1, 1, 1, 1))
    corner = torch.zeros(n + 1, n + 1, n + 1, dtype=torch.bool, device=DEV)
    for k in range(8):
        z, y, x = k >> 2, (k >> 1) & 1, k & 1
        corner |= m[z:z + n + 1, y:y + n + 1, x:x + n + 1]
    inds = torch.nonzero(corner.reshape(-1))[:, 0]
    dec = Decoder(case["kind"], case["c"], s["layers"])
    ser = {"f": premultiply_features(dec, s["voxels"].reshape(-1, case["c"])[inds]), "i": inds.int(),
           "m": torch.nn.functional.pad(s["mask"], (0, 1, 0, 1, 0, 1)).reshape(-1)[inds], "p": pack_realtime(dec)}
    lo, vs = _place(s["dims"])
    return RealtimeModel.from_serialized(ser, n, lo[0], vs, DEV)


def _requests(case, s):
    """(scene, camera, height, width) of each request: the case's resolution, halves and thirds of it."""
    return [(k % 2, _camera(s["g"]), max(1, case["h"] // (1 + k % 3)), max(1, case["w"] // (1 + k % 3)))
            for k in range(case["requests"])]


def _fma(a, b, c):
    """a * b + c of FP32 tensors, rounded once (the product is exact in FP64)."""
    return (a.double() * b.double() + c.double()).float()


def _walk(s, o, d):
    """The occupied voxels that the rays cross, in ray order: cell [S, 3], entry and exit points [S, 3] (FP32, voxel
    units) and ray [S].  The definition of the path's segments: a walk from grid plane to grid plane in FP32, each point
    computed from the previous one, so the points themselves carry no freedom of rounding."""
    lo, vs = _place(s["dims"])
    n = torch.tensor(s["dims"], device=DEV).float()
    p = (o - torch.tensor(lo, device=DEV)) / torch.full_like(o, vs)
    a, b = -p / d, (n - p) / d
    near, far = torch.minimum(a, b).amax(1), torch.maximum(a, b).amin(1)
    inside = ((p >= 0) & (p <= n)).all(1)
    hit = inside | (near <= far)
    p = torch.where(inside[:, None], p, torch.minimum(_fma(d, near[:, None].expand_as(d), p).clamp_min(0), n))
    ray = torch.nonzero(hit)[:, 0]
    p, d, sgn = p[ray], d[ray], d[ray].sign()
    one = torch.ones_like(p)
    found = []
    for step in range(sum(s["dims"]) + 3):
        plane = _fma(p, sgn, one).floor() * sgn
        t = (plane - p) / d
        dt = t.amin(1, keepdim=True)
        q = _fma(d, dt.expand_as(d), p)
        axis = (t == dt).int().argmax(1, keepdim=True)  # ties: x, then y, then z
        q = q.scatter(1, axis, plane.gather(1, axis))
        live = ((q >= 0) & (q <= n)).all(1)
        cell = torch.minimum((p + 1e-4).int(), (q + 1e-4).int()).long()
        c = torch.minimum(cell.clamp_min(0), n.long() - 1)
        k = torch.nonzero(live & (c == cell).all(1) & s["mask"][c[:, 2], c[:, 1], c[:, 0]])[:, 0]
        found.append((ray[k], cell[k], p[k], q[k]))
        p = q
        if step % 32 == 31:
            k = torch.nonzero(live)[:, 0]
            if not k.numel():
                break
            ray, p, d, sgn, one = ray[k], p[k], d[k], sgn[k], one[k]
        else:
            d = torch.where(live[:, None], d, torch.full_like(d, float("nan")))
    ray, cell, p0, p1 = (torch.cat(x) for x in zip(*found))
    order = torch.sort(ray, stable=True).indices
    return cell[order], p0[order], p1[order], ray[order]


def _some_segments(case, s):
    """The first case["segments"] segments of enough camera rays (again from the first where there are fewer)."""
    rays = max(16, int(case["segments"] / (0.5 * s["dims"][0] * case["occ"])) + 1)
    o, d = _rays(dict(h=max(1, rays // 64), w=64), s)
    cell, p0, p1, _ = _walk(s, o, d)
    k = torch.arange(case["segments"], device=DEV) % max(1, p0.shape[0])
    return cell[k], p0[k].contiguous(), p1[k].contiguous()


def _longest(case, s):
    """One ray along the grid's diagonal with every cell near it occupied: the padded traversal outputs are as wide
    as the longest ray, and with this one in the batch the width is the grid's for every seed."""
    n = s["dims"][0]
    k = torch.arange(n, device=DEV)
    for a in range(27):
        i = [(k + (a // 3 ** b) % 3 - 1).clamp(0, n - 1) for b in range(3)]
        s["mask"][i[0], i[1], i[2]] = True
    lo, _ = _place(s["dims"])
    d = torch.tensor([1.0, 0.99993, 1.00011], device=DEV)
    d = (d / d.norm())[None]
    return d * (lo[0] * 1.8), d


# --- the calls --------------------------------------------------------------------

def prepare(case, seed):
    s = _scene(case, seed)
    op = case["op"]
    lo, vs = _place(s["dims"])
    st = {"case": case}
    if op == "intersect":
        st["o"], st["d"] = (torch.cat(x) for x in zip(_rays(case, s), _longest(case, s)))
        st.update(lo=lo[0], vs=vs, n=s["dims"][0], mask=s["mask"])
    elif op == "integrate":
        _, st["p0"], st["p1"] = _some_segments(case, s)
        st["voxels"] = s["voxels"].requires_grad_()
        st["grad"] = torch.randn(st["p0"].shape[0], case["c"], generator=s["g"], device=DEV)
    elif op == "render":
        st["o"], st["d"] = _rays(case, s)
        st["field"] = _field(case, s)
    elif op == "train":
        st["o"], st["d"], st["target"] = _batch(case, s)
        st["field"] = _field(case, s)
        if case["graph"]:
            st["step"] = TrainStepGraph(st["field"], st["o"], st["d"], st["target"], form=case["form"], l_s=L_S)
    elif op == "alpha":
        st["rays"] = torch.cat(_rays(case, s), 1)
        st["field"] = _field(case, s)
    elif op == "frame":
        o, st["d"] = _rays(case, s)
        st["eye"] = o[0].cpu()
        st["model"] = _realtime(case, s)
    else:
        fields = [_field(case, s), _field(case, _scene(case, seed + 1))]
        st["requests"] = _requests(case, s)
        st["residency"] = Residency(60 << 30, 36 << 30)
        for k, f in enumerate(fields):
            st["residency"].register(str(k), f.voxels.numel() * 6, lambda f=f: f)
        st["renderer"] = GpuRenderer(case["form"])
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "intersect":
        args = (st["o"], st["d"], st["lo"], -st["lo"], st["n"], st["vs"])
        return masked_intersect(*args, st["mask"], 1.0) if case["masked"] else ray_voxel_intersect(*args)
    if op == "integrate":
        f = integrate(st["voxels"], st["p0"], st["p1"])
        return f.detach(), torch.autograd.grad(f, st["voxels"], st["grad"])[0]
    if op == "render":
        with torch.no_grad():
            return st["field"](st["o"], st["d"], form=case["form"])
    if op == "train":
        if case["graph"]:
            return st["step"](st["o"], st["d"], st["target"])
        f = st["field"]
        rgb, reg = f(st["o"], st["d"], form=case["form"])
        loss = l2_loss(rgb, reg, st["target"], L_S)
        return (loss.detach(), *torch.autograd.grad(loss, [f.voxels, f.params]))
    if op == "alpha":
        return extract_alpha_map(st["field"], st["rays"], batch=4000, form=case["form"])
    if op == "frame":
        return st["model"].render_frame(st["eye"], st["d"])[0]
    reqs = [Request(k, str(scene), c2w, h, w, 1.2 * max(h, w)) for k, (scene, c2w, h, w) in enumerate(st["requests"])]
    done = serve(reqs, st["residency"], st["renderer"], realtime=False)
    return [r.rgb for r in sorted(done, key=lambda r: r.rid)]


# --- what a pass cannot do without ------------------------------------------------

def work(case):
    """Bytes: inputs once and outputs once, a feature row or an occupancy byte once per voxel that any ray can meet;
    operations: the decoder's and the integral's multiply-adds per segment.  Segments per ray are estimated from the
    occupancy: a ray towards the grid crosses about 1.5 n voxels, `occ` of the blob region more often than not."""
    op, dims = case["op"], _dims(case)
    rays = 0 if op == "integrate" else case["h"] * case["w"]
    if op == "serve":
        rays = sum(max(1, case["h"] // (1 + k % 3)) * max(1, case["w"] // (1 + k % 3)) for k in range(case["requests"]))
    cells = dims[0] * dims[1] * dims[2]
    across = 0.5 * sum(dims)
    seg = rays * across * (1 if op == "intersect" and not case["masked"] else min(1.0, 1.2 * case["occ"]))
    seg = case.get("segments", seg)
    seen = min(cells * case["occ"], seg)  # voxels met at all
    if op == "intersect":
        per = (24 + 1 + 4) if case["masked"] else (12 + 1 + 4)
        return {"bytes": 24 * rays + seg * per + (seen if case["masked"] else 0), "flops": 30 * rays * across}
    c = case["c"]
    row = seen * c * 4
    if op == "integrate":
        return {"bytes": row + cells * c * 4 + seg * (24 + 8 * c), "flops": 2 * 16 * c * seg}
    w = 32 if case["kind"] == "diver32" else 64
    mlp = 2 * (c * w + (w * w if w == 32 else 0) + w * (w + 1) + w * w + 3 * w) + 16 * c
    if op == "frame":
        seg = min(seg, 24 * rays)
        seen = min(seen, seg)
        return {"bytes": 12 * rays + 12 * rays + seen * (c * 4 + 5), "flops": mlp * seg}
    half = 0.5 if case["form"] in ("bf16", "fp16") and op in ("render", "serve") else 1.0
    out = {"render": 12 * rays, "serve": 12 * rays, "alpha": 4 * cells, "train": cells * c * 4}[op]
    return {"bytes": 24 * rays + seen + row * half + out, "flops": mlp * seg * (3 if op == "train" else 1)}


# --- the same in 64 bits ----------------------------------------------------------

def _features64(rows, cell, p0, p1):
    """Integral over a segment of the trilinear interpolant of the corner rows [S, 8, C] (bit 0 = x, 1 = y, 2 = z)."""
    a, b = p0 - cell, p1 - cell
    m1 = (a + b) / 2

    def m2(i, j):
        return (a[:, i] * b[:, j] + b[:, i] * a[:, j]) / 6 + (a[:, i] * a[:, j] + b[:, i] * b[:, j]) / 3

    xy, yz, xz = m2(0, 1), m2(1, 2), m2(0, 2)
    xyz = (a + b).prod(1) / 12 + (a.prod(1) + b.prod(1)) / 6
    x, y, z = m1.unbind(1)
    w = [1 - x - y - z + xy + yz + xz - xyz, x - xy - xz + xyz, y - xy - yz + xyz, xy - xyz, z - xz - yz + xyz,
         xz - xyz, yz - xyz, xyz]
    return (torch.stack(w, 1)[:, :, None] * rows).sum(1)


def _corner_ids(cell, dims):
    k = torch.arange(8, device=DEV)
    x, y, z = (cell[:, i, None] + ((k >> i) & 1)[None] for i in range(3))
    return (z * (dims[1] + 1) + y) * (dims[0] + 1) + x


def _decode64(layers, feat, dirs):
    n1 = len(layers) - 2
    x = feat
    for i, (w, b) in enumerate(layers[:n1]):
        x = torch.nn.functional.linear(x, w, b)
        x = torch.relu(x) if i + 1 < n1 else x
    pe = [dirs]
    for k in range(4):
        pe += [torch.sin(2 ** k * math.pi * dirs), torch.cos(2 ** k * math.pi * dirs)]
    h = torch.relu(torch.nn.functional.linear(torch.cat([x[:, 1:]] + pe, 1), *layers[-2]))
    return x[:, 0], torch.sigmoid(torch.nn.functional.linear(h, *layers[-1]))


def _padded(values, ray, rays, m):
    """[S, ...] in ray order -> [rays, m, ...], zeros behind each ray's last."""
    count = torch.bincount(ray, minlength=rays)
    first = torch.cumsum(count, 0) - count
    out = values.new_zeros((rays, m) + values.shape[1:])
    out[ray, torch.arange(ray.numel(), device=DEV) - first[ray]] = values
    return out


def _chunks(s, rays):
    step = max(64, int(2e9 / sum(s["dims"]) / s["voxels"].shape[-1] / 8))
    return [(a, min(rays, a + step)) for a in range(0, rays, step)]


def _render64(s, o, d, cut=False):
    """(rgb, [(cell, weight)]) in 64 bits; cut: with the real-time path's rules (alpha below 1e-2 skipped, a ray
    stops when its transmittance is below 1e-2)."""
    layers = [(w.double(), b.double()) for w, b in s["layers"]]
    grid = s["voxels"].detach().reshape(-1, s["voxels"].shape[-1])
    rgb, met = [], []
    for a, b in _chunks(s, o.shape[0]):
        cell, p0, p1, ray = _walk(s, o[a:b], d[a:b])
        if not ray.numel():
            rgb.append(torch.ones(b - a, 3, device=DEV, dtype=torch.float64))
            continue
        feat = _features64(grid[_corner_ids(cell, s["dims"])].double(), cell, p0.double(), p1.double())
        sigma, color = _decode64(layers, feat, d[a:b].double()[ray])
        m = int(torch.bincount(ray).max())
        alpha = _padded(1 - torch.exp(-torch.relu(sigma)), ray, b - a, m)
        if cut:
            alpha = torch.where(alpha < 1e-2, torch.zeros_like(alpha), alpha)
        trans = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1 - alpha], 1), 1)
        weight = alpha * trans[:, :-1]
        if cut:
            weight = weight * (trans[:, :-1] >= 1e-2)
        left = 1 - weight.sum(1)
        rgb.append((weight[..., None] * _padded(color, ray, b - a, m)).sum(1) + left[:, None])
        count = torch.bincount(ray, minlength=b - a)
        first = torch.cumsum(count, 0) - count
        met.append((cell, weight[ray, torch.arange(ray.numel(), device=DEV) - first[ray]]))
    return torch.cat(rgb), met


def _packed(grads):
    """Decoder gradients in the packed order: each layer's W^T with rows padded to a multiple of 4, then its bias."""
    out = []
    for w, b in grads:
        pad = -w.shape[0] % 4
        out += [torch.nn.functional.pad(w.t(), (0, pad)).reshape(-1), torch.nn.functional.pad(b, (0, pad))]
    return torch.cat(out)


def _train64(s, o, d, target):
    layers = [(w.double().requires_grad_(), b.double().requires_grad_()) for w, b in s["layers"]]
    flat = [x for wb in layers for x in wb]
    grid = s["voxels"].detach().reshape(-1, s["voxels"].shape[-1])
    gv = torch.zeros(grid.shape, device=DEV, dtype=torch.float64)
    gl = [torch.zeros_like(x) for x in flat]
    rays = o.shape[0]
    parts = [(a, b, _walk(s, o[a:b], d[a:b])) for a, b in _chunks(s, rays)]
    m = max([int(torch.bincount(q[3]).max()) for _, _, q in parts if q[3].numel()] + [1])
    loss = torch.zeros((), device=DEV, dtype=torch.float64)
    for a, b, (cell, p0, p1, ray) in parts:
        ids = _corner_ids(cell, s["dims"])
        rows = grid[ids].double().requires_grad_()
        sigma, color = _decode64(layers, _features64(rows, cell, p0.double(), p1.double()), d[a:b].double()[ray])
        alpha = _padded(1 - torch.exp(-torch.relu(sigma)), ray, b - a, m)
        trans = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1 - alpha], 1), 1)[:, :-1]
        weight = alpha * trans
        rgb = (weight[..., None] * _padded(color, ray, b - a, m)).sum(1) + (1 - weight.sum(1))[:, None]
        part = ((rgb - target[a:b].double()) ** 2).sum() / (3 * rays) + L_S * torch.log(1 + sigma ** 2 / 0.5).sum() / (rays * m)
        got = torch.autograd.grad(part, [rows] + flat)
        gv.index_add_(0, ids.reshape(-1), got[0].reshape(-1, grid.shape[1]))
        for x, y in zip(gl, got[1:]):
            x += y
        loss += part.detach()
    return loss, gv.reshape(s["voxels"].shape), _packed(list(zip(gl[::2], gl[1::2])))


def exact(case, seed):
    op = case["op"]
    if op == "intersect":
        return None  # the walk's FP32 steps are the definition of its points
    s = _scene(case, seed)
    if op == "integrate":
        cell, p0, p1 = _some_segments(case, s)
        grad = torch.randn(p0.shape[0], case["c"], generator=s["g"], device=DEV)
        p0, p1 = p0.double(), p1.double()
        ids = _corner_ids(cell, s["dims"])
        grid = s["voxels"].reshape(-1, case["c"])
        out, gv = [], torch.zeros(grid.shape, device=DEV, dtype=torch.float64)
        for a in range(0, p0.shape[0], 1 << 19):
            q = slice(a, a + (1 << 19))
            rows = grid[ids[q]].double().requires_grad_()
            f = _features64(rows, cell[q], p0[q], p1[q])
            gr, = torch.autograd.grad(f, rows, grad[q].double())
            out.append(f.detach())
            gv.index_add_(0, ids[q].reshape(-1), gr.reshape(-1, case["c"]))
        return torch.cat(out), gv.reshape(s["voxels"].shape)
    if op == "train":
        return _train64(s, *_batch(case, s))
    if op == "render":
        with torch.no_grad():
            return _render64(s, *_rays(case, s))[0], None
    if op == "alpha":
        dims = s["dims"]
        out = torch.zeros(dims[0] * dims[1] * dims[2], device=DEV, dtype=torch.float64)
        with torch.no_grad():
            for cell, weight in _render64(s, *_rays(case, s))[1]:
                out.scatter_reduce_(0, (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0], weight, "amax")
        return out.reshape(dims[2], dims[1], dims[0])
    if op == "frame":
        with torch.no_grad():
            return _render64(s, *_rays(case, s), cut=True)[0]
    scenes, out = [s], []
    requests = _requests(case, s)
    scenes.append(_scene(case, seed + 1))
    with torch.no_grad():
        for scene, c2w, h, w in requests:
            d = _directions(c2w, h, w, 1.2 * max(h, w)).float()
            o = c2w[:, 3].to(DEV).expand(d.shape)
            out.append(_render64(scenes[scene], o, d)[0])
    return out
