"""The work that a program using this library has it do, as cases that can be timed.

A case is one pass through the public entry points on one synthetic scene: the voxel shell of a seeded union of spheres
and tori (what the surface of an object looks like to the decoder), in Morton order, with exactly ``n`` voxels.

kinds
  step      build_neighbors + subm_conv: the operator on a scene it has not seen (map, schedule and conv)
  resblock  conv -> LayerNorm -> GELU -> conv -> residual on a level whose cache the program keeps
  convnext  conv -> LayerNorm, Linear C -> 4C -> SiLU, Linear 4C -> C -> residual, cache kept
  layers    stacked plain convs on one large scene, cache kept
  up        the up block: subdivision maps, the children's map, conv1 into the kept children with LayerNorm and SiLU,
            conv2 with the skip
  maps      the maps alone: neighbour map, masks and the mask-sorted row order
  host      the whole operator on host buffers (copies in, map, conv, copy out)
"""
import math

import numpy as np
import torch

import trellis2_cuda_b200 as sp

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
TAPS_SHELL = 14.7        # present taps per voxel of a shell of thickness 1.5 (27 for a solid)
CHILDREN = 3.7           # kept children per voxel of such a shell
HALF = 0.75              # half the shell's thickness, in voxels


def listed():
    return [
        # the smallest calls: two small objects in one batch, a scene of a coarse level; launches and host work count
        dict(name="step_700_c64_f16", kind="step", n=700, batch=2, ci=64, co=64, dtype="f16"),
        # the 64^3 sphere-sized scene in fp32, where the tensor cores' input types would lose precision
        dict(name="step_14534_c64_f32", kind="step", n=14534, batch=1, ci=64, co=64, dtype="f32"),
        # the headline operator: mid-decoder scene, 256 channels
        dict(name="step_217821_c256_bf16", kind="step", n=217821, batch=1, ci=256, co=256, dtype="bf16"),
        # widths that are multiples of 32 and nothing more, which the operator takes as well
        dict(name="step_30011_c96_c160_bf16", kind="step", n=30011, batch=1, ci=96, co=160, dtype="bf16"),
        # residual block of the decoder stack's widest, smallest level: few rows, 1024 channels
        dict(name="resblock_3727_c1024_bf16", kind="resblock", n=3727, batch=1, ci=1024, co=1024, dtype="bf16"),
        # the decoder's ConvNeXt block at its second and at its last level (512 channels and few rows, 64 and many)
        dict(name="convnext_16725_c512_f16", kind="convnext", n=16725, batch=1, ci=512, co=512, dtype="f16"),
        dict(name="convnext_727949_c64_bf16", kind="convnext", n=727949, batch=1, ci=64, co=64, dtype="bf16"),
        # up block between the two finest levels, 512^3 -> 1024^3, 128 -> 64 channels (about 3.3 M children)
        dict(name="up_886752_c128_c64_f16", kind="up", n=886752, batch=1, ci=128, co=64, dtype="f16"),
        # up block between coarse levels
        dict(name="up_3727_c1024_c512_bf16", kind="up", n=3727, batch=1, ci=1024, co=512, dtype="bf16"),
        # the largest scene on one GPU: stacked 128-channel layers
        dict(name="layers_8597581_c128_bf16", kind="layers", n=8597581, batch=1, ci=128, co=128, dtype="bf16", layers=2),
        # the maps with the row order that goes with them, for a program that has its own schedule
        dict(name="maps_1000003", kind="maps", n=1000003, batch=1, ci=0, co=0, dtype="f16"),
        # the operator called with host buffers
        dict(name="host_217821_c256_bf16", kind="host", n=217821, batch=1, ci=256, co=256, dtype="bf16"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "resblock", "convnext", "up", "layers", "maps", "host"])
    dtype = rng.choice(["f16", "bf16"])
    batch = rng.choice([1, 1, 1, 2, 4])
    if kind == "step":
        form = rng.choice(["even", "even", "ragged", "f32"])
        if form == "f32":
            c = rng.choice([32, 64, 64, 128])
            return dict(kind=kind, n=_spread(rng, 300, 60000), batch=batch, ci=c, co=rng.choice([c, 64]), dtype="f32")
        if form == "ragged":
            return dict(kind=kind, n=_spread(rng, 300, 60000), batch=batch, ci=32 * rng.randint(1, 8), co=32 * rng.randint(1, 8), dtype=dtype)
        c, most = rng.choice([(64, 2000000), (128, 1000000), (256, 500000), (512, 100000), (1024, 20000)])
        return dict(kind=kind, n=_spread(rng, 300, most), batch=batch, ci=c, co=c, dtype=dtype)
    if kind in ("resblock", "convnext"):
        c, lo, hi = rng.choice([(1024, 1000, 15000), (512, 4000, 70000), (256, 15000, 250000), (128, 50000, 800000), (64, 200000, 3000000)])
        return dict(kind=kind, n=_spread(rng, lo, hi), batch=1, ci=c, co=c, dtype=dtype)
    if kind == "up":
        c, lo, hi = rng.choice([(1024, 1000, 15000), (512, 4000, 70000), (256, 15000, 250000), (128, 50000, 880000)])
        return dict(kind=kind, n=_spread(rng, lo, hi), batch=1, ci=c, co=c // 2, dtype=dtype)
    if kind == "layers":
        c = rng.choice([64, 128])
        return dict(kind=kind, n=_spread(rng, 1000000, 8500000), batch=1, ci=c, co=c, dtype=dtype, layers=rng.choice([1, 2]))
    if kind == "maps":
        return dict(kind=kind, n=_spread(rng, 1000, 4000000), batch=batch, ci=0, co=0, dtype=dtype)
    c = rng.choice([64, 128, 256])
    return dict(kind=kind, n=_spread(rng, 2000, 300000), batch=1, ci=c, co=c, dtype=rng.choice(["f16", "bf16", "f32"]) if c == 64 else dtype)


# ------------------------------------------------------------------------------------------ scenes
def _distance(shapes, p):
    """Signed distance of the points p (float64 [..., 3]) to the union of (kind, centre, R, r, axis) shapes."""
    out = None
    for kind, c, R, r, axis in shapes:
        d = p - torch.tensor(c, dtype=torch.float64, device=p.device)
        if kind == 0:
            v = d.square().sum(-1).sqrt() - R
        else:
            o = [i for i in range(3) if i != axis]
            q = (d[..., o[0]].square() + d[..., o[1]].square()).sqrt() - R
            v = (q.square() + d[..., axis].square()).sqrt() - r
        out = v if out is None else torch.minimum(out, v)
    return out


def _shell(shapes, res):
    """int64 [m, 3]: the voxels of a res^3 grid within HALF of the union's surface; cells of 64^3 and 8^3 are culled first."""
    g = torch.arange((res + 63) // 64, device="cuda")
    cells, size = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3), 64
    while True:
        bound = HALF + (math.sqrt(3.0) * (size - 1) / 2 + 1e-9 if size > 1 else 0.0)
        keep = torch.cat([_distance(shapes, q.double() * size + (size - 1) / 2).abs() <= bound for q in cells.split(1 << 24)])
        cells = cells[keep]
        if size == 1:
            return cells[(cells >= 0).all(1) & (cells < res).all(1)]
        size //= 8
        o = torch.arange(8, device="cuda")
        cells = (cells[:, None, :] * 8 + torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3)[None]).reshape(-1, 3)


def _morton(p):
    key = torch.zeros(p.shape[0], dtype=torch.int64, device=p.device)
    for bit in range(12):
        for axis in range(3):
            key |= ((p[:, axis] >> bit) & 1) << (3 * bit + 2 - axis)
    return key


def _object(n, seed):
    """(coords int64 [n, 3], shapes): the first n voxels, in Morton order, of a shell with hardly more than n."""
    rng = np.random.default_rng(seed)
    unit = []                                   # shapes in a unit cube, then scaled until the shell has the voxels
    for i in range(6):
        R = rng.uniform(0.10, 0.30)
        r = 0.0 if i % 2 == 0 else R * rng.uniform(0.2, 0.4)
        ext = R + r
        unit.append((i % 2, rng.uniform(ext, 1 - ext, 3), R, r, int(rng.integers(3))))
    res = math.sqrt(n / 4.0)
    for _ in range(12):
        shapes = [(k, tuple(2.5 + res * c), res * R, res * r, a) for k, c, R, r, a in unit]
        p = _shell(shapes, int(res) + 6)
        if n <= p.shape[0] <= 1.02 * n + 60:
            break
        res *= math.sqrt((1.01 * n + 20) / max(p.shape[0], 1))
    while p.shape[0] < n:
        res *= 1.01
        shapes = [(k, tuple(2.5 + res * c), res * R, res * r, a) for k, c, R, r, a in unit]
        p = _shell(shapes, int(res) + 6)
    return p[_morton(p).argsort()][:n], shapes


def _scene(n, batch, seed):
    """(coords int32 [n, 4], shapes of the first object)."""
    parts, first = [], None
    for b in range(batch):
        m = n // batch + (1 if b < n % batch else 0)
        p, shapes = _object(m, [seed, b])
        first = first or shapes
        parts.append(torch.cat([torch.full((m, 1), b, dtype=torch.int64, device="cuda"), p], 1))
    return torch.cat(parts).to(torch.int32).contiguous(), first


def _child_logits(coords, shapes):
    """fp16 [n, 8]: what the decoder's subdivision head says of each child: positive for the CHILDREN * n children nearest to
    the finer surface (those within HALF of it, give or take a few)."""
    fine = [(k, tuple(2 * v for v in c), 2 * R, 2 * r, a) for k, c, R, r, a in shapes]
    s = torch.arange(8, device="cuda")
    child = 2 * coords[:, None, 1:].long() + torch.stack([s & 1, (s >> 1) & 1, (s >> 2) & 1], 1)[None]
    logit = torch.cat([HALF - _distance(fine, q.double()).abs() for q in child.split(1 << 20)]).reshape(-1)
    kept = logit.argsort(descending=True)[: int(CHILDREN * coords.shape[0])]
    out = logit.clamp(max=-1e-3)
    out[kept] = logit[kept].clamp(min=1e-3)
    return out.to(torch.float16).reshape(-1, 8).contiguous()


def prepare(case, seed):
    n, ci, co, td, kind = case["n"], case["ci"], case["co"], DTYPES[case["dtype"]], case["kind"]
    coords, shapes = _scene(n, case["batch"], seed)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, scale=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * scale).to(td)

    def weight(rows, cin, taps=27):             # Kaiming-uniform over the fan-in, as a conv or Linear layer starts with
        a = 1.0 / math.sqrt(taps * cin)
        shape = (rows, taps, cin) if taps > 1 else (rows, cin)
        return (torch.rand(shape, generator=g, device="cuda") * (2 * a) - a).to(td)

    s = dict(case=case, coords=coords)
    if kind == "maps":
        return s
    s["x"] = randn(n, ci)
    gamma, beta = 1 + 0.1 * torch.randn(ci, generator=g, device="cuda"), 0.1 * torch.randn(ci, generator=g, device="cuda")
    s["ln"] = (gamma, beta, 1e-6)
    if kind == "up":
        s["logits"] = _child_logits(coords, shapes)
        s["w"], s["b"] = weight(8 * co, ci), randn(8 * co, scale=0.1)
        s["w2"], s["b2"] = weight(co, co), randn(co, scale=0.1)
    else:
        s["w"], s["b"] = weight(co, ci), randn(co, scale=0.1)
    if kind == "resblock":
        s["w2"], s["b2"] = weight(co, co), randn(co, scale=0.1)
    if kind == "convnext":
        s["w_in"], s["b_in"] = weight(4 * co, co, 1), randn(4 * co, scale=0.1)
        s["w_out"], s["b_out"] = weight(co, 4 * co, 1), randn(co, scale=0.1)
    if kind == "layers":
        s["ws"] = [weight(co, co) * 2 for _ in range(case["layers"])]
    if kind == "host":
        for k in ("coords", "x", "w", "b"):
            s[k] = s[k].cpu().pin_memory()
        s["out"] = torch.empty((n, co), dtype=td, pin_memory=True)
    elif kind != "step":
        s["cache"] = sp.build_neighbors(coords, want_sorted=False)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "step":
        cache = sp.build_neighbors(s["coords"], want_sorted=False)
        return {"y": sp.subm_conv(s["x"], s["w"], s["b"], cache), "nbr": cache.nbr, "gray": cache.gray}
    if kind == "maps":
        cache = sp.build_neighbors(s["coords"])
        return {"nbr": cache.nbr, "gray": cache.gray, "sorted": cache.sorted}
    if kind == "host":
        return sp.subm_conv_host(s["coords"], s["x"], s["w"], s["b"], out=s["out"])
    x, cache = s["x"], s["cache"]
    if kind == "resblock":
        h = sp.subm_conv(x, s["w"], s["b"], cache, ln=s["ln"], act="gelu")
        return sp.subm_conv(h, s["w2"], s["b2"], cache, residual=x)
    if kind == "convnext":
        h = sp.subm_conv(x, s["w"], s["b"], cache, ln=s["ln"])
        h = sp.linear(h, s["w_in"], s["b_in"], act="silu")
        return sp.linear(h, s["w_out"], s["b_out"], residual=x)
    if kind == "layers":
        for w in s["ws"]:
            x = sp.subm_conv(x, w, None, cache)
        return x
    h = sp.row_epilogue(x, ln=s["ln"], act="silu")
    level = sp.subdivide(cache, s["logits"])
    h = sp.subdiv_conv(h, s["w"], s["b"], level, ln=(None, None, 1e-6), act="silu")
    rep = s["case"]["co"] // (s["case"]["ci"] // 8)
    y = sp.subm_conv(h, s["w2"], s["b2"], level.nb, skip=(x, level.src, rep))
    return {"y": y, "coords": level.coords, "src": level.src, "nbr": level.nb.nbr, "gray": level.nb.gray}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _map64(coords):
    """int64 [n, 27]: row of each neighbour, -1 where there is none."""
    key = lambda q: ((q[..., 0] * 4100 + q[..., 1] + 1) * 4100 + q[..., 2] + 1) * 4100 + q[..., 3] + 1
    q = coords.long()
    have, order = key(q).sort()
    o = torch.tensor([-1, 0, 1], device=q.device)
    taps = torch.cat([torch.zeros(27, 1, dtype=torch.int64, device=q.device), torch.cartesian_prod(o, o, o)], 1)
    out = []
    for part in q.split(1 << 20):
        k = key(part[:, None] + taps[None])
        at = torch.searchsorted(have, k).clamp(max=have.numel() - 1)
        out.append(torch.where(have[at] == k, order[at], -1))
    return torch.cat(out)


def _conv64(x, w, b, nbr, rows=None, slot=None):
    """Rows of the map (all, or the listed ones with the weight set of their slot) times x and w in 64 bits, the bias added."""
    rows = torch.arange(nbr.shape[0], device=x.device) if rows is None else rows
    co = w.shape[0] if slot is None else w.shape[0] // 8
    y = torch.zeros((rows.numel(), co), dtype=torch.float64, device=x.device)
    for s in range(1 if slot is None else 8):
        mine = torch.arange(rows.numel(), device=x.device) if slot is None else (slot == s).nonzero()[:, 0]
        ws = w[s * co:(s + 1) * co].double()
        for at in mine.split(1 << 19):
            part = torch.zeros((at.numel(), co), dtype=torch.float64, device=x.device)
            for v in range(27):
                r = nbr[rows[at], v]
                have = (r >= 0).nonzero()[:, 0]
                part[have] += x[r[have]].double() @ ws[:, v].T
            y[at] = part if b is None else part + b[s * co:(s + 1) * co].double()
    return y


def _norm64(x, ln):
    gamma, beta, eps = ln
    y = torch.nn.functional.layer_norm(x, x.shape[-1:], eps=eps)
    return y if gamma is None else y * gamma.double() + beta.double()


def exact(case, seed):
    kind, s = case["kind"], prepare(case, seed)
    if kind == "maps":
        return None
    s = {k: v.cuda() if isinstance(v, torch.Tensor) else v for k, v in s.items()}
    x, nbr, f = s["x"], _map64(s["coords"]), torch.nn.functional
    if kind == "layers":
        y = x
        for w in s["ws"]:
            y = _conv64(y, w, None, nbr)
        return y
    if kind == "up":
        kept = (s["logits"] > 0).nonzero()
        parent, slot = kept[:, 0], kept[:, 1]
        coords = torch.cat([s["coords"][parent, :1], 2 * s["coords"][parent, 1:] + torch.stack([slot & 1, (slot >> 1) & 1, slot >> 2], 1)], 1)
        h = f.silu(_norm64(x.double(), s["ln"]))
        h = f.silu(_norm64(_conv64(h, s["w"], s["b"], nbr, parent, slot), (None, None, 1e-6)))
        cs, co = case["ci"] // 8, case["co"]
        skip = x.view(-1, 8, cs)[parent, slot].double().repeat_interleave(co // cs, 1)
        return {"y": _conv64(h, s["w2"], s["b2"], _map64(coords)) + skip, "coords": None, "src": None, "nbr": None, "gray": None}
    y = _conv64(x, s["w"], s["b"], nbr)
    if kind == "step":
        return {"y": y, "nbr": None, "gray": None}
    if kind == "host":
        return y
    if kind == "resblock":
        return _conv64(f.gelu(_norm64(y, s["ln"])), s["w2"], s["b2"], nbr) + x.double()
    y = f.silu(_norm64(y, s["ln"]) @ s["w_in"].double().T + s["b_in"].double())
    return y @ s["w_out"].double().T + s["b_out"].double() + x.double()


# ------------------------------------------------------------------------------------------ cost and precision
MAP_ROW = 27 * 4 + 4          # bytes of a row of the neighbour map and its mask


def work(case):
    n, ci, co, kind = case["n"], case["ci"], case["co"], case["kind"]
    es = 4 if case["dtype"] == "f32" else 2
    conv = 2.0 * TAPS_SHELL * n * ci * co                       # present taps only
    weights = 27 * ci * co * es
    rows = n * (ci + co) * es
    if kind == "step":
        return {"bytes": n * (16 + MAP_ROW) + rows + weights, "flops": conv}
    if kind == "maps":
        return {"bytes": n * (16 + MAP_ROW + 4), "flops": 0}
    if kind == "host":
        return {"bytes": n * 16 + rows + weights, "flops": conv}
    if kind == "resblock":                                      # x twice (input and residual), the hidden rows out and in
        return {"bytes": n * MAP_ROW + 5 * n * ci * es + 2 * weights, "flops": 2 * conv}
    if kind == "convnext":
        return {"bytes": n * MAP_ROW + n * ci * es * (1 + 2 + 2 * 4 + 2) + weights + 8 * ci * ci * es, "flops": conv + 2 * 8.0 * n * ci * ci}
    if kind == "layers":
        return {"bytes": case["layers"] * (rows + weights + n * MAP_ROW), "flops": case["layers"] * conv}
    m = int(CHILDREN * n)                                       # up: a child has its parent's taps in conv1, its own in conv2
    return {"bytes": n * (MAP_ROW + 16 + 16) + n * ci * es * 4 + m * (16 + 4 + MAP_ROW + 4 * co * es) + 8 * weights + 27 * co * co * es,
            "flops": 2.0 * TAPS_SHELL * m * (ci * co + co * co)}


def tolerance(case):
    """About four times what the path differs by from itself with the sums in 64 bits and the same roundings to the storage type in
    between (largest seen: 5.4e-7 in fp32, 7.4e-4 in bf16, 1.5e-4 in fp16, all where a LayerNorm or a sum over many taps follows)."""
    if case["kind"] == "maps":
        return "exact"
    if case["dtype"] == "f32":
        return {"rel": 3e-6}
    return {"rel": {"bf16": 3e-3, "f16": 6e-4}[case["dtype"]]}
