"""The work that users of this library have it do, as cases to be timed: isosurface
queries on compressed volumes from 64^3 to 1024 x 1024 x 1080, a sweep delivered to host
memory, a batch over several resident volumes, the codec in both directions, the render
pass, and the sort and compaction primitives.

Every case is a dict of plain values.  ``prepare`` builds what a program holds before the
call (a synthetic volume of the seed, compressed by the library's encoder, and the handle
made from it), ``run`` is one pass through the public entry points, ``work`` the bytes and
operations no implementation can do without.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "webgpu-bcmc_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "webgpu-bcmc_gb300"))

import bcmc  # noqa: E402
from bcmc import camera  # noqa: E402

# What a field is like at a mean isovalue: the share of its 4^3 blocks that a query meshes,
# vertices per voxel of the volume (both measured over the isovalues below), the vertices per
# voxel that a program makes room for, and the range the isovalues come from.
FIELDS = {
    "blobs": dict(active=0.43, verts=0.24, room=1.0, lo=0.05, hi=0.70),
    "ct": dict(active=0.39, verts=0.30, room=1.5, lo=30.0, hi=220.0),
    "spectral": dict(active=0.75, verts=1.2, room=2.5, lo=-0.5, hi=0.5),
    "ct16": dict(active=0.12, verts=0.07, room=0.6, lo=400.0, hi=3600.0),
}


def listed():
    def query(name, field, dims, rate, cache, order):
        return dict(name=name, kind="query", field=field, x=dims[0], y=dims[1], z=dims[2], rate=rate, cache=cache,
                    order=order)

    return [
        # moving the isovalue slider on a small volume held in the cache whole: latency and launches
        query("query_64", "blobs", (64, 64, 64), 8, 1.0, "random"),
        # a cropped scan with ragged edges, random isovalues, the reference's initial cache of 5 %
        query("query_ragged", "ct", (131, 98, 57), 5, 0.05, "random"),
        # the headline: a sweep of 16 isovalues over a 256^3 scan, cache of half the blocks, reset per sweep
        query("query_256", "ct", (256, 256, 256), 4, 0.5, "sweep"),
        # following a feature through a 512^3 simulation field: a random walk of the isovalue
        query("query_512", "spectral", (512, 512, 512), 2, 0.25, "walk"),
        # the largest served volume, 17.7 M blocks
        query("query_1080", "ct16", (1024, 1024, 1080), 4, 0.1, "random"),
        # a sweep whose meshes a host program keeps: every mesh into one page-locked buffer
        dict(name="host_sweep_256", kind="host", field="ct", x=256, y=256, z=256, rate=4, cache=0.5, queries=4),
        # a server's batch: queries over several resident volumes in one launch sequence
        dict(name="batch_32", kind="batch", rate=4, queries=32, scale=256),
        # compressing a scan before it is loaded
        dict(name="encode_256", kind="encode", field="ct", x=256, y=256, z=256, rate=4),
        # decompressing a simulation field whole, for a consumer of the raw voxels
        dict(name="decode_512", kind="decode", field="spectral", x=512, y=512, z=512, rate=2),
        # a frame of the scan's surface with fog, full HD
        dict(name="render_1080p", kind="render", field="ct", x=256, y=256, z=256, width=1920, height=1080, fog=True),
        # the radix sorter by itself, random 32-bit keys
        dict(name="sort_1m", kind="sort", n=1 << 20, keys="random", reverse=False),
        # scan and stream compaction of a flag buffer, as the reference's pipeline chains them
        dict(name="compact_4m", kind="compact", n=4_000_000, density=0.3),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(lo, hi):
        # a mean edge over the whole range, stretched a little along each axis, odd values included
        e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        d = [max(5, int(round(e * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3)]
        return dict(x=d[0], y=d[1], z=d[2])

    kind = rng.choice(["query"] * 5 + ["host", "batch", "encode", "decode", "render", "sort", "compact"])
    field = rng.choice(["blobs", "ct", "spectral", "ct16"])
    if kind == "query":
        d = dims(24, 96) if field == "blobs" else dims(24, 420)
        return dict(kind=kind, field=field, rate=rng.randint(1, 16), cache=rng.choice([0.05, 0.25, 0.5, 1.0]),
                    order=rng.choice(["random", "sweep", "walk"]), **d)
    if kind == "host":
        return dict(kind=kind, field=rng.choice(["ct", "spectral"]), rate=rng.randint(2, 8), cache=0.5,
                    queries=rng.randint(2, 6), **dims(40, 200))
    if kind == "batch":
        return dict(kind=kind, rate=rng.randint(2, 8), queries=log_int(2, 48), scale=log_int(96, 256))
    if kind == "encode":
        return dict(kind=kind, field=field, rate=rng.randint(1, 16), **(dims(24, 96) if field == "blobs" else dims(24, 230)))
    if kind == "decode":
        return dict(kind=kind, field=field, rate=rng.randint(1, 12), **(dims(24, 96) if field == "blobs" else dims(24, 300)))
    if kind == "render":
        w = log_int(320, 2560)
        return dict(kind=kind, field=rng.choice(["ct", "spectral"]), width=w, height=max(200, int(w * rng.uniform(0.5, 0.8))),
                    fog=rng.random() < 0.5, **dims(40, 256))
    if kind == "sort":
        return dict(kind=kind, n=log_int(100, 6_000_000), keys=rng.choice(["random", "ages", "small"]),
                    reverse=rng.random() < 0.5)
    return dict(kind=kind, n=log_int(100, 20_000_000), density=rng.choice([0.01, 0.3, 0.9]))


# ---- synthetic fields, made on the GPU from a seed ----------------------------------------
def _weights(n, lattice, spacing):
    """Cubic-smoothstep interpolation weights from lattice points to samples."""
    x = np.arange(n, dtype=np.float64) / spacing
    i = np.floor(x).astype(np.int64)
    t = x - i
    t = t * t * (3.0 - 2.0 * t)
    w = np.zeros((n, lattice), dtype=np.float32)
    w[np.arange(n), i] += (1.0 - t).astype(np.float32)
    w[np.arange(n), i + 1] += t.astype(np.float32)
    return torch.from_numpy(w).cuda()


def _value_noise(dims, rng, spacing):
    """Smooth value noise in [0, 1], two octaves, as a [z, y, x] tensor."""
    X, Y, Z = dims
    out = torch.zeros((Z, Y, X), device="cuda")
    for rel, weight in ((1.0, 1.0), (0.25, 0.35)):
        sp = spacing * rel
        g = [int(math.ceil(n / sp)) + 2 for n in (Z, Y, X)]
        f = torch.from_numpy(rng.random(g, dtype=np.float32)).cuda()
        wz, wy, wx = (_weights(n, k, sp) for n, k in zip((Z, Y, X), g))
        f = torch.einsum("yj,kji->kyi", wy, f)
        f = torch.einsum("xi,kyi->kyx", wx, f)
        for z in range(0, Z, 64):
            out[z: z + 64] += weight * torch.einsum("zk,kyx->zyx", wz[z: z + 64], f)
    out -= out.min()
    return out.div_(out.max().clamp(min=1e-12))


def _threshold(f, share):
    """The value that `share` of the 4^3 blocks lie below."""
    Z, Y, X = f.shape
    p = torch.nn.functional.pad(f[None, None], (0, -X % 4, 0, -Y % 4, 0, -Z % 4), mode="replicate")[0, 0]
    m = p.reshape(p.shape[0] // 4, 4, p.shape[1] // 4, 4, p.shape[2] // 4, 4).amax(dim=(1, 3, 5)).reshape(-1)
    return m.sort().values[min(m.numel() - 1, int(share * m.numel()))]


def _field(kind, dims, seed):
    X, Y, Z = dims
    rng = np.random.default_rng([seed, X, Y, Z])
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 30)))
    if kind == "blobs":  # Gaussian blobs, eight to each 64^3
        f = torch.zeros((Z, Y, X), device="cuda")
        z, y, x = (torch.arange(n, device="cuda", dtype=torch.float32) for n in (Z, Y, X))
        for _ in range(max(4, round(8 * X * Y * Z / 64 ** 3))):
            c, s, a = rng.uniform(0, 1, 3) * [X, Y, Z], rng.uniform(4, 12), rng.uniform(0.5, 1)
            gx, gy, gz = (torch.exp(-(v - float(m)) ** 2 / (2 * s * s)) for v, m in zip((x, y, z), c))
            f += float(a) * gz[:, None, None] * gy[None, :, None] * gx
        return f
    if kind == "spectral":  # isotropic k^-5/3 energy spectrum, random phases, in [-1, 1]
        kz, ky = (torch.fft.fftfreq(n, device="cuda") for n in (Z, Y))
        kx = torch.fft.rfftfreq(X, device="cuda")
        k2 = kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx ** 2
        k2[0, 0, 0] = math.inf
        phase = torch.rand(k2.shape, device="cuda", generator=gen) * (2 * math.pi)
        f = torch.fft.irfftn(torch.polar(k2 ** (-11 / 12), phase), s=(Z, Y, X))
        lo, hi = f.min(), f.max()
        return 2 * (f - lo) / (hi - lo).clamp(min=1e-12) - 1
    if kind == "ct":  # 35 % constant background blocks, interior 20..255 with scanner noise
        n = _value_noise(dims, rng, 24.0)
        t = _threshold(n, 0.35)
        v = 20.0 + (n - t) / (1 - t).clamp(min=1e-6) * 235.0
        v += torch.randn(v.shape, device="cuda", generator=gen) * 3.0
        return torch.where(n >= t, v.clamp_(20.0, 255.0), torch.zeros_like(v))
    n = _value_noise(dims, rng, 48.0)  # ct16: 60 % background blocks, whole values up to 4095
    t = _threshold(n, 0.60)
    v = torch.round(((n - t) / (1 - t).clamp(min=1e-6)).clamp_(0, 1) * 4095.0)
    return torch.where(n >= t, v, torch.zeros_like(v))


def _dims(case):
    return case["x"], case["y"], case["z"]


def _stream(ctx, field, rate):
    """The field's compressed stream on the device, without the encoder's padding word."""
    words = bcmc.zfp_encode(ctx, field, rate)
    torch.cuda.synchronize()
    Z, Y, X = field.shape
    return words[: -(-X // 4) * -(-Y // 4) * -(-Z // 4) * rate]


def _isovalues(case, seed):
    f = FIELDS[case["field"]]
    lo, hi = f["lo"], f["hi"]
    rng = np.random.default_rng([seed, 77])
    if case["order"] == "sweep":
        return np.linspace(lo, hi, 16) + rng.uniform(0, 0.01) * (hi - lo)
    if case["order"] == "walk":  # steps of 2 % of the range, back at either end
        v = [0.5 * (lo + hi) + rng.uniform(-0.1, 0.1) * (hi - lo)]
        for _ in range(63):
            s = 0.02 * (hi - lo) * rng.choice([-1.0, 1.0])
            v.append(v[-1] + s if lo <= v[-1] + s <= hi else v[-1] - s)
        return np.asarray(v)
    return rng.uniform(lo, hi, 64)


class _Surface:
    """A program's volume and the isovalues its user goes through."""

    def __init__(self, case, seed):
        self.ctx = bcmc.Context(0, initial_cache_fraction=case["cache"])
        self.mc = bcmc.CompressedMarchingCubes(self.ctx)
        self.mc.setCompressedVolume(_stream(self.ctx, _field(case["field"], _dims(case), seed), case["rate"]),
                                    case["rate"], _dims(case))
        torch.cuda.empty_cache()


def _mesh(vertices):
    """A program's own vertex buffer, that a mesh is kept in."""
    return torch.zeros((int(vertices) + 4096, 2), dtype=torch.int32, device="cuda")


def _keep(state, n, buffer):
    """The vertices into the program's buffer: the library's is overwritten by the next query."""
    if n > state["mesh"].shape[0]:
        state["mesh"] = _mesh(1.5 * n)
    if n:
        state["mesh"][:n].copy_(buffer.torch())
    return state["mesh"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "query":
        s = _Surface(case, seed)
        s.isos, s.at = [float(v) for v in _isovalues(case, seed)], 0
        return dict(kind=kind, surface=s, reset=case["order"] == "sweep",
                    mesh=_mesh(FIELDS[case["field"]]["room"] * math.prod(_dims(case))))
    if kind == "host":
        s = _Surface(case, seed)
        f = FIELDS[case["field"]]
        u = np.random.default_rng([seed, 78]).uniform(0, 0.01)
        isos = np.linspace(f["lo"], f["hi"], case["queries"]) + u * (f["hi"] - f["lo"])
        room = sum(s.mc.computeSurface(float(v)) for v in isos)
        s.mc.lruCache.reset()
        room = max(room, int(1.8 * f["verts"] * case["queries"] * math.prod(_dims(case)))) + 4096
        return dict(kind=kind, surface=s, isos=isos,
                    out=torch.zeros((room, 2), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32))
    if kind == "batch":
        k = case["scale"]
        volumes = [("blobs", (k // 4, k // 4, k // 4)), ("spectral", (3 * k // 8, k // 2, 5 * k // 16)),
                   ("ct", (k // 2 + 3, k // 2, k // 2 - 5)), ("ct", (k, k, k)), ("spectral", (k, k, k // 2))]
        ctx = bcmc.Context(0)
        streams = [_stream(ctx, _field(f, d, seed + i), case["rate"]).cpu().numpy() for i, (f, d) in enumerate(volumes)]
        blocks = sum(math.prod(-(-n // 4) for n in d) for _, d in volumes)
        engine = bcmc.Engine(ctx, pool_slots=blocks, max_batch=case["queries"])
        for w, (_, d) in zip(streams, volumes):
            engine.addVolume(w, case["rate"], d)
        rng = np.random.default_rng([seed, 79])
        batches = []
        for _ in range(4):
            v = rng.integers(0, len(volumes), case["queries"])
            u = rng.uniform(0, 1, case["queries"])
            f = [FIELDS[volumes[i][0]] for i in v]
            batches.append([(int(i), float(g["lo"] + t * (g["hi"] - g["lo"]))) for i, t, g in zip(v, u, f)])
        room = 0.4 * case["queries"] * sum(FIELDS[f]["room"] * math.prod(d) for f, d in volumes)
        return dict(kind=kind, engine=engine, batches=batches, at=[0], mesh=_mesh(room))
    if kind == "encode":
        return dict(kind=kind, ctx=bcmc.Context(0), field=_field(case["field"], _dims(case), seed), rate=case["rate"])
    if kind == "decode":
        ctx = bcmc.Context(0)
        words = _stream(ctx, _field(case["field"], _dims(case), seed), case["rate"])
        torch.cuda.empty_cache()
        return dict(kind=kind, ctx=ctx, words=words, blocks=words.numel() // case["rate"], rate=case["rate"])
    if kind == "render":
        s = _Surface(dict(case, rate=4, cache=0.5), seed)
        f = FIELDS[case["field"]]
        n = s.mc.computeSurface(f["lo"] + 0.53 * (f["hi"] - f["lo"]))
        mesh = s.mc.vertexBuffer.torch().clone()
        a = 0.3 * np.random.default_rng([seed, 80]).uniform(-1, 1)  # the camera orbits a little around its start
        view, eye = camera.default_view(case["width"], case["height"], eye=(math.sin(a), 0.1, math.cos(a)))
        return dict(kind=kind, ctx=s.ctx, mesh=mesh, n=n, dims=_dims(case), view=view, eye=eye, width=case["width"],
                    height=case["height"], fog=case["fog"])
    rng = np.random.default_rng([seed, 81])
    if kind == "sort":
        n = case["n"]
        if case["keys"] == "random":
            keys = rng.integers(0, 1 << 32, n, dtype=np.uint32)
        elif case["keys"] == "ages":  # cache-slot ages: small counts, or 100000 plus one
            keys = (rng.integers(0, 60, n) + np.where(rng.random(n) < 0.5, 100000, 0)).astype(np.uint32)
        else:
            keys = rng.integers(0, 1 << 16, n, dtype=np.uint32)
        aligned = bcmc.RadixSorter.getAlignedSize(n)
        k, v = (torch.zeros(aligned, dtype=torch.int32, device="cuda") for _ in range(2))
        src = torch.from_numpy(keys.view(np.int32)).cuda()
        return dict(kind=kind, sorter=bcmc.RadixSorter(bcmc.Context(0)), src=src, keys=k, values=v, n=n,
                    ids=torch.arange(n, dtype=torch.int32, device="cuda"), reverse=case["reverse"])
    n = case["n"]
    pipeline = bcmc.ExclusiveScanPipeline(bcmc.Context(0))
    aligned = pipeline.getAlignedSize(n)
    flags = torch.zeros(aligned, dtype=torch.int32, device="cuda")
    flags[:n] = torch.from_numpy((rng.random(n) < case["density"]).astype(np.int32)).cuda()
    offsets = torch.zeros_like(flags)
    return dict(kind=kind, scanner=pipeline.prepareGPUInput(offsets, aligned), compact=bcmc.StreamCompact(pipeline),
                flags=flags, offsets=offsets, out=torch.zeros_like(flags), n=n)


def run(state):
    kind = state["kind"]
    if kind == "query":
        s = state["surface"]
        if s.at == len(s.isos):
            s.at = 0
            if state["reset"]:
                s.mc.lruCache.reset()
        n = s.mc.computeSurface(s.isos[s.at])
        s.at += 1
        return {"n": n, "vertices": _keep(state, n, s.mc.vertexBuffer)}
    if kind == "host":
        counts = state["surface"].mc.computeSurfacesToHost(state["isos"], state["out"])
        return {"counts": counts, "vertices": state["out"].view(np.int32)}
    if kind == "batch":
        e = state["engine"]
        res = e.run(state["batches"][state["at"][0] % len(state["batches"])])
        state["at"][0] += 1
        return {"offsets": res["vertex_offset"].astype(np.int64), "counts": res["num_vertices"].astype(np.int64),
                "active": res["num_active_blocks"].astype(np.int64), "vertices": _keep(state, int(res["num_vertices"].sum()), e.vertexBuffer)}
    if kind == "encode":
        return bcmc.zfp_encode(state["ctx"], state["field"], state["rate"])
    if kind == "decode":
        return bcmc.zfp_decode_volume(state["ctx"], state["words"], state["blocks"], state["rate"])
    if kind == "render":
        rgba, depth, triangle = bcmc.render(state["ctx"], state["mesh"], state["n"], state["dims"], state["view"],
                                            state["eye"], state["width"], state["height"], fog=state["fog"])
        return {"rgba": rgba, "depth": depth, "triangle": triangle}
    if kind == "sort":
        n = state["n"]
        state["keys"][:n].copy_(state["src"])  # the sort works in place: new keys for each pass
        state["values"][:n].copy_(state["ids"])
        state["sorter"].sort(state["keys"], state["values"], n, state["reverse"])
        return {"keys": state["keys"], "values": state["values"]}
    state["offsets"].copy_(state["flags"])
    total = state["scanner"].scan(state["n"])
    state["compact"].compactActiveIDs(state["n"], state["flags"], state["offsets"], state["out"])
    return {"total": total, "offsets": state["offsets"], "ids": state["out"]}


def _query_work(field, dims):
    """A cached query: each block's value range and the active blocks' voxels read, the vertices written and kept."""
    blocks = math.prod(-(-n // 4) for n in dims)
    f = FIELDS[field]
    verts = f["verts"] * math.prod(dims)
    # a vertex: two values compared, an interpolation and a packing; a voxel of an active block: one test
    return blocks * (8 + f["active"] * 256) + 24 * verts, 12 * verts + 64 * f["active"] * blocks


def work(case):
    kind = case["kind"]
    if kind in ("query", "host"):
        q = case.get("queries", 1)
        b, f = _query_work(case["field"], _dims(case))
        return {"bytes": q * b, "flops": q * f}
    if kind == "batch":
        k, share = case["scale"], case["queries"] / 5
        parts = [_query_work(f, d) for f, d in (
            ("blobs", (k // 4,) * 3), ("spectral", (3 * k // 8, k // 2, 5 * k // 16)), ("ct", (k // 2,) * 3),
            ("ct", (k, k, k)), ("spectral", (k, k, k // 2)))]
        return {"bytes": share * sum(p[0] for p in parts), "flops": share * sum(p[1] for p in parts)}
    if kind in ("encode", "decode"):
        voxels = 64 * math.prod(-(-n // 4) for n in _dims(case))
        # the lifting steps along three axes, about eleven operations to four values each, and a scale
        return {"bytes": voxels * (4 + case["rate"] / 8), "flops": voxels * 10}
    if kind == "render":
        verts = FIELDS[case["field"]]["verts"] * math.prod(_dims(case))
        pixels = case["width"] * case["height"]
        return {"bytes": 8 * verts + 24 * pixels, "flops": 40 * verts + 120 * pixels}
    if kind == "sort":
        return {"bytes": 16 * case["n"] + 16 * case["n"], "flops": 0}  # the pairs in and out, and the copies before
    return {"bytes": case["n"] * (4 + 4 + 4 * case["density"]) + 8 * case["n"], "flops": case["n"]}


# ---- what the passes give, in 64 bits -------------------------------------------------------
# the order of a block's coefficients in the stream (part of the zfp format), x + 4 * (y + 4 * z)
_ORDER = [0, 1, 4, 16, 20, 17, 5, 2, 8, 32, 21, 6, 18, 24, 9, 33, 36, 3, 12, 48, 22, 25, 37, 40, 34, 10, 7, 19, 28, 13,
          49, 52, 41, 38, 26, 23, 29, 53, 11, 35, 44, 14, 50, 56, 42, 27, 39, 45, 30, 54, 57, 60, 51, 15, 43, 46, 58,
          61, 55, 31, 62, 59, 47, 63]


def _decode64(words, blocks, rate):
    """The fixed-rate stream's values in 64 bits: the embedded code read one bit per step for every block at once."""
    dev = words.device
    base = torch.arange(blocks, device=dev) * rate
    end = 64 * rate

    def bit(pos):
        return (words[base + torch.div(pos.clamp(max=end - 1), 64, rounding_mode="floor")] >> (pos % 64)) & 1

    head = words[base]
    some = (head & 1).bool()
    emax = ((head >> 1) & 255) - 127
    u = torch.zeros((blocks, 64), dtype=torch.int64, device=dev)
    pos = torch.full((blocks,), 9, device=dev)
    n, i, m = (torch.zeros_like(pos) for _ in range(3))
    k = torch.full_like(pos, 31)
    raw, run_ = torch.zeros_like(some), torch.zeros_like(some)  # reading raw bits, a run; else a group test
    live = some.clone()
    for _ in range(end - 9):
        b = bit(pos).bool()
        pos = pos + live
        left = end - pos
        # raw bits of the coefficients already significant
        at_raw = live & raw
        # a run of zeros up to the next significant coefficient
        zero = live & run_ & ~b
        n2 = n + zero.long()
        group = live & ~raw & ~run_
        opened = group & b & (n2 < 63) & (left > 0)
        hit = (live & run_ & (b | (n2 == 63) | (left == 0))) | (group & b & ~opened)
        idx = torch.where(at_raw, i, n2.clamp(max=63))
        val = ((at_raw & b) | hit).long() << k.clamp(min=0)
        u.scatter_add_(1, idx[:, None], val[:, None])
        n = n2 + hit.long()
        i = i + at_raw.long()
        raw = at_raw & (i < m)
        run_ = (run_ & live & ~hit) | opened
        # the plane goes on with a group test after a hit or the last raw bit, unless all are significant
        plane_end = (group & ~b) | ((hit | (at_raw & ~raw)) & (n >= 64))
        k = k - plane_end.long()
        m = torch.where(plane_end, torch.minimum(n, left), m)
        i = torch.where(plane_end, torch.zeros_like(i), i)
        raw = raw | (plane_end & (m > 0))
        live = live & (left > 0) & (k >= 0)
    del raw, run_, i, m, n
    v = torch.zeros_like(u)
    v[:, torch.tensor(_ORDER, device=dev)] = (u ^ 0xAAAAAAAA) - 0xAAAAAAAA
    v = v.reshape(blocks, 4, 4, 4)
    for axis in (1, 2, 3):  # the inverse lift along z, y, x
        x, y, z, w = v.unbind(axis)
        y = y + (w >> 1)
        w = w - (y >> 1)
        y = y + w
        w = 2 * w - y
        z = z + x
        x = 2 * x - z
        y = y + z
        z = 2 * z - y
        w = w + x
        x = 2 * x - w
        v = torch.stack((x, y, z, w), axis)
    out = torch.ldexp(v.reshape(blocks, 64).double(), (emax - 30).double()[:, None])
    return torch.where(some[:, None], out, torch.zeros_like(out)).reshape(-1)


def exact(case, seed):
    if case["kind"] != "decode":
        # whole values, or (the render pass) colours and depths behind the choice of a nearest triangle
        return None
    s = prepare(case, seed)
    return _decode64(s["words"], s["blocks"], s["rate"])
