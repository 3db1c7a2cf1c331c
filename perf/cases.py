"""The renders that this framework is used for, as measurable cases: single
frames through `euc_render` (from a thumbnail to a two-pass 1080p frame),
blended frames, lines, batches (plain and recorded), host buffers through the
`Pipeline` API, the serving loop and texture ingest.

`listed()` gives the fixed cases, `draw(rng)` more of the same ranges,
`prepare` / `run` one pass, `work` what a pass cannot do without, and `exact`
the depth targets by a 64-bit rasteriser of its own.
"""
import ctypes as C
import functools
import math
from dataclasses import replace

import numpy as np
import torch

from euc_gb300 import abi, capi, pipeline, scenes, serve
from euc_gb300 import frames as fr

FMTS = {"rgba8": abi.FMT_RGBA8, "bgra8": abi.FMT_BGRA8, "rgb8": abi.FMT_RGB8, "rgba32f": abi.FMT_RGBA32F}
SOURCES = {"rgba8": (abi.SRC_RGBA8, 4), "bgra8": (abi.SRC_BGRA8, 4), "rgb8": (abi.SRC_RGB8, 3),
           "luma8": (abi.SRC_LUMA8, 1), "luma_alpha8": (abi.SRC_LUMA_ALPHA8, 2), "r32f": (abi.SRC_R32F, 4)}
TESTS = {"less": (abi.TEST_LESS, 1), "less_pass": (abi.TEST_LESS, 0), "none": (abi.TEST_NONE, 0)}
READBACK = ("color", "depth")


def listed():
    return [
        # a thumbnail or icon: the smallest call, all launch latency
        {"name": "sphere_160", "kind": "sphere", "w": 160, "h": 120, "lon": 16, "lat": 8, "fmt": "rgb8", "aa": 0},
        # the small plain scene of the benchmark: one 640x480 Gouraud frame a call
        {"name": "sphere_vga", "kind": "sphere", "w": 640, "h": 480, "lon": 64, "lat": 32, "fmt": "rgb8", "aa": 0},
        # the wireframe example's pipeline: a mesh drawn as lines, no depth target
        {"name": "wire_vga", "kind": "wire", "w": 640, "h": 480, "lon": 64, "lat": 32, "fmt": "bgra8", "aa": 0},
        # the drop-in call: `Pipeline.render` on the caller's host buffers, cleared by the host for each frame
        {"name": "host_vga", "kind": "host", "w": 640, "h": 480, "lon": 64, "lat": 32, "fmt": "rgba8", "aa": 0},
        # translucent triangles blended src-over in submission order (particles, glass)
        {"name": "alpha_540p", "kind": "soup", "w": 960, "h": 540, "tris": 8000, "area_hi": 3000.0, "blend": "alpha",
         "test": "less", "fmt": "rgba8", "aa": 0},
        # the benchmark's fill-rate scene: heavy overdraw of triangles of every size
        {"name": "soup_1080p", "kind": "soup", "w": 1920, "h": 1080, "tris": 200000, "area_hi": 1e4,
         "blend": "replace", "test": "less", "fmt": "rgba8", "aa": 0},
        # the benchmark's two-pass scene: shadow map, then textured Phong with MSAA over a dense mesh
        {"name": "knot_1080p", "kind": "knot", "w": 1920, "h": 1080, "shadow": 2048, "tubular": 1250, "radial": 200,
         "tex": 1024, "aa": 1},
        # uneven scenes drawn by one `euc_render_batch` call, as a renderer of changing scene sets makes it
        {"name": "batch_48", "kind": "batch", "scenes": 48, "tri_hi": 100000, "form": "call"},
        # the benchmark's headline: 256 uneven scenes recorded once and replayed
        {"name": "batch_256_graph", "kind": "batch", "scenes": 256, "tri_hi": 100000, "form": "graph"},
        # a stream of small frames (thumbnails of one mesh, views of one object) recorded and replayed
        {"name": "spheres_256_graph", "kind": "spheres", "frames": 256, "w": 640, "h": 480, "lon": 64, "lat": 32},
        # a burst of requests at the serving loop: resident meshes and textures, two passes, images read back
        {"name": "serve_192", "kind": "serve", "requests": 192, "meshes": 24, "textures": 8, "tex": 512},
        # a decoded RGB image turned into a texture on the device
        {"name": "ingest_2k", "kind": "ingest", "w": 2048, "h": 2048, "src": "rgb8"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sphere", "sphere", "wire", "lines", "host", "soup", "soup", "alpha", "alpha", "knot", "batch",
                       "batch", "spheres", "serve", "ingest"))
    w = _log(rng, 120, 1920)
    h = max(64, min(1080, int(w * rng.uniform(0.5, 1.0))))
    lon = _log(rng, 8, 128)
    mesh = {"lon": lon, "lat": max(4, lon // 2 + rng.randint(-2, 2))}
    fmt = rng.choice(sorted(FMTS))
    aa = rng.choice((0, 0, 1, 2))
    if kind in ("sphere", "wire"):
        return {"kind": kind, "w": w, "h": h, **mesh, "fmt": fmt if kind == "sphere" else "bgra8", "aa": aa}
    if kind == "host":
        return {"kind": kind, "w": min(w, 1280), "h": min(h, 720), **mesh, "fmt": rng.choice(("rgba8", "bgra8", "rgb8")),
                "aa": aa}
    if kind == "lines":
        return {"kind": kind, "w": w, "h": h, "lines": _log(rng, 50, 20000), "len_hi": rng.uniform(20.0, 500.0), "aa": aa}
    if kind == "soup":
        return {"kind": "soup", "w": w, "h": h, "tris": _log(rng, 300, 150000), "area_hi": float(_log(rng, 50, 8000)),
                "blend": "replace", "test": rng.choice(sorted(TESTS)), "fmt": fmt, "aa": min(aa, 1)}
    if kind == "alpha":  # 1 to 12 layers of triangles on average
        area_hi = float(_log(rng, 100, 5000))
        layers = math.exp(rng.uniform(0.0, math.log(12.0)))
        tris = int(min(60000, max(50, layers * w * h * 1.44 / (area_hi / math.log(area_hi)))))
        return {"kind": "soup", "w": w, "h": h, "tris": tris, "area_hi": area_hi, "blend": "alpha",
                "test": rng.choice(sorted(TESTS)), "fmt": fmt, "aa": min(aa, 1)}
    if kind == "knot":
        radial = _log(rng, 12, 200)
        return {"kind": kind, "w": w, "h": h, "shadow": rng.choice((256, 512, 1024, 2048)), "tubular": radial * 6 + 1,
                "radial": radial, "tex": rng.choice((64, 256, 1024)), "aa": rng.choice((0, 1, 1, 2))}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 2, 160), "tri_hi": _log(rng, 1000, 100000),
                "form": rng.choice(("call", "graph"))}
    if kind == "spheres":
        return {"kind": kind, "frames": _log(rng, 2, 200), "w": min(w, 800), "h": min(h, 600), **mesh}
    if kind == "serve":
        return {"kind": kind, "requests": _log(rng, 8, 192), "meshes": _log(rng, 4, 24), "textures": 4,
                "tex": rng.choice((64, 256, 512))}
    return {"kind": "ingest", "w": _log(rng, 600, 4000), "h": _log(rng, 600, 4000), "src": rng.choice(sorted(SOURCES))}


# ---------------------------------------------------------------------------
# The frames of a case
# ---------------------------------------------------------------------------
def _recolor(frame, fmt):
    """The frame with a colour target of another format."""
    t = frame.target("color")
    frame.targets[frame.targets.index(t)] = scenes.TargetSpec("color", t.width, t.height, FMTS[fmt], 0)
    return frame


# The scenes of a batch and the requests of a burst keep their meshes, sizes and
# options from seed to seed, so that every seed's outputs have the same layout;
# the cameras and textures are the seed's.
@functools.lru_cache(maxsize=2)
def _batch_base(n, tri_hi):
    return scenes.batch_frames(seed=n, n=n, tri_hi=tri_hi)


def _batch_frames(n, tri_hi, seed):
    rng = np.random.default_rng(seed)
    out = []
    for f in _batch_base(n, tri_hi):
        p = f.passes[0]
        u = type(p.uniforms).from_buffer_copy(p.uniforms)
        u.model = scenes.f32mat(scenes.quat_rotation(rng))
        s = p.samplers[0]
        tex = np.roll(s.source, rng.integers(0, s.source.shape[0], 2), axis=(0, 1))
        out.append(replace(f, passes=[replace(p, uniforms=u, samplers=[replace(s, source=tex)])]))
    return out


@functools.lru_cache(maxsize=2)
def _serve_base(requests, meshes, textures, tex):
    assets = scenes.serve_assets(seed=requests, nmeshes=meshes, ntextures=textures, tex_size=tex)
    rng = np.random.default_rng(requests)
    return [scenes.serve_frame(assets, rng) for _ in range(requests)]


def _serve_frames(c, seed):
    rng = np.random.default_rng(seed)
    out = []
    for f in _serve_base(c["requests"], c["meshes"], c["textures"], c["tex"]):
        shadow, color = f.passes
        model = scenes.quat_rotation(rng)
        su = type(shadow.uniforms).from_buffer_copy(shadow.uniforms)
        pu = type(color.uniforms).from_buffer_copy(color.uniforms)
        su.mvp = scenes.f32mat(np.array(list(pu.light_vp), dtype=np.float64).reshape(4, 4) @ model)
        pu.model = scenes.f32mat(model)
        out.append(replace(f, passes=[replace(shadow, uniforms=su), replace(color, uniforms=pu)]))
    return out


def _frames(c, seed):
    kind = c["kind"]
    if kind in ("sphere", "host"):
        f = scenes.sphere_frame(seed=seed, width=c["w"], height=c["h"], lon=c["lon"], lat=c["lat"])
        f.passes[0].desc.aa_level = c["aa"]
        return [_recolor(f, c["fmt"])]
    if kind == "wire":
        return [scenes.wireframe_frame(seed=seed, width=c["w"], height=c["h"], lon=c["lon"], lat=c["lat"],
                                       fmt=FMTS[c["fmt"]], aa_level=c["aa"])]
    if kind == "lines":
        return [scenes.lines_frame(seed=seed, width=c["w"], height=c["h"], nlines=c["lines"], len_hi=c["len_hi"],
                                   aa_level=c["aa"])]
    if kind == "soup":
        f = scenes.soup_frame(seed=seed, width=c["w"], height=c["h"], ntris=c["tris"], area_hi=c["area_hi"],
                              alpha=c["blend"] == "alpha")
        d = f.passes[0].desc
        d.depth_test, d.depth_write = TESTS[c["test"]]
        d.aa_level = c["aa"]
        return [_recolor(f, c["fmt"])]
    if kind == "knot":
        return [scenes.knot_frame(seed=seed, width=c["w"], height=c["h"], shadow_size=c["shadow"],
                                  tubular=c["tubular"], radial=c["radial"], tex_size=c["tex"], aa_level=c["aa"])]
    if kind == "batch":
        return _batch_frames(c["scenes"], c["tri_hi"], seed)
    if kind == "spheres":
        return [scenes.sphere_frame(seed=seed * 1000 + k, width=c["w"], height=c["h"], lon=c["lon"], lat=c["lat"])
                for k in range(c["frames"])]
    return _serve_frames(c, seed)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _context():
    """The context that a program keeps for its plain calls."""
    return capi.Context(0)


class _Calls:
    """Frames rendered pass by pass with `euc_render`, their arguments ready."""

    def __init__(self, c, seed):
        self.batch = fr.DeviceBatch(_frames(c, seed))
        self.ctx = _context()
        self.stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        lib = capi.lib()
        self.render = lib.euc_render
        self.args = [(self.ctx.handle, C.byref(s.desc), s.uniforms, s.uniforms_size, C.byref(s.layout), s.vertices,
                      s.nverts, s.indices, s.nindices, C.byref(s.pixel), C.byref(s.depth), self.stream)
                     for arr in self.batch.scene_arrays() for s in arr]

    def run(self):
        self.batch.clear()
        for a in self.args:
            capi.check(self.render(*a), "euc_render")
        return _targets(self.batch)


class _Batch:
    """All frames in one `euc_render_batch` call a pass, or their recorded graph."""

    def __init__(self, c, seed):
        self.batch = fr.DeviceBatch(_frames(c, seed))
        # a recorded batch belongs to the scratch of its context: each keeps its own
        self.ctx = capi.Context(0) if c.get("form", "graph") == "graph" else _context()
        self.graph = fr.BatchGraph(self.ctx, self.batch) if c.get("form", "graph") == "graph" else None

    def run(self):
        if self.graph is not None:
            self.graph.launch()
        else:
            fr.render_batch(self.ctx, self.batch)
        return _targets(self.batch)


def _targets(batch):
    """Every target of the batch: bytes as they are, f32 colours as floats."""
    out = {}
    if any("depth" in f.targets for f in batch.frames):
        out["depth"] = batch.depth
    t = batch.frames[0].targets.get("color")
    out["color"] = t if t is not None and t.dtype == torch.float32 else batch.color
    return out


class _HostPipeline(pipeline.Pipeline):
    """The Gouraud mesh as a `Pipeline` implementation of a program."""

    SHADER = abi.SHADER_GOURAUD

    def __init__(self, frame):
        self.p = frame.passes[0]

    def depth_mode(self):
        return pipeline.DepthMode.LESS_WRITE

    def aa_mode(self):
        return pipeline.AaMode(self.p.desc.aa_level)

    def uniforms(self):
        return self.p.uniforms

    def vertex_layout(self):
        return self.p.layout


class _Host:
    def __init__(self, c, seed):
        f = _frames(c, seed)[0]
        t = f.target("color")
        self.pipe = _HostPipeline(f)
        self.verts = pipeline.IndexedVertices(f.passes[0].indices, f.passes[0].vertices)
        self.color = pipeline.Buffer2d.fill([t.width, t.height], 0, fmt=t.fmt)
        self.depth = pipeline.Buffer2d.fill([t.width, t.height], 1.0)
        self.ctx = _context()

    def run(self):
        self.color.data.fill(0)
        self.depth.data.fill(1.0)
        self.pipe.render(self.verts, self.color, self.depth, ctx=self.ctx)
        return {"color": self.color.data, "depth": self.depth.data}


class _Serve:
    def __init__(self, c, seed):
        frames = _frames(c, seed)
        self.server = serve.Server(0, framebuffer_budget=1 << 30, max_batch=64, slots=3)
        res = serve.Resident(self.server)
        sizes = [(serve.out_bytes(f, READBACK) + 63) // 64 * 64 for f in frames]
        self.out = torch.zeros(sum(sizes), dtype=torch.uint8).pin_memory()
        reqs, self.keep, at = [], [res], 0
        for k, (f, n) in enumerate(zip(frames, sizes)):
            r, kp = serve.request_for(f, res, READBACK, tag=k, out=self.out.data_ptr() + at, out_size=n)
            reqs.append(r)
            self.keep.append(kp)
            at += n
        self.reqs = (abi.ServerRequest * len(reqs))(*reqs)

    def run(self):
        n = len(self.reqs)
        _, accepted = self.server.submit(self.reqs)
        if accepted != n:
            raise RuntimeError("the server took %d of %d requests" % (accepted, n))
        capi.check(self.server.drain(), "drain")
        done = 0
        while done < n:
            comp = self.server.poll(n - done, wait_ms=1000)
            if not len(comp) or comp["status"].any():
                raise RuntimeError("a request failed or is missing")
            done += len(comp)
        return {"images": self.out}


class _Ingest:
    def __init__(self, c, seed):
        self.fmt, bpp = SOURCES[c["src"]]
        self.w, self.h = c["w"], c["h"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        if self.fmt == abi.SRC_R32F:
            self.src = torch.rand((self.h, self.w), generator=g, device="cuda")
        else:
            self.src = torch.randint(0, 256, (self.h, self.w, bpp), generator=g, device="cuda", dtype=torch.uint8)
        self.pitch = self.w * bpp
        self.dst = torch.empty((self.h, self.w), dtype=torch.int32, device="cuda")
        self.ctx = _context()
        self.stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        self.ingest = capi.lib().euc_texture_ingest

    def run(self):
        capi.check(self.ingest(self.ctx.handle, self.src.data_ptr(), self.w, self.h, self.pitch, self.fmt,
                               self.dst.data_ptr(), self.w * 4, self.stream), "euc_texture_ingest")
        return {"texels": self.dst}


def prepare(case, seed):
    kind = case["kind"]
    make = {"batch": _Batch, "spheres": _Batch, "host": _Host, "serve": _Serve, "ingest": _Ingest}.get(kind, _Calls)
    return make(case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------
# The least a pass must do
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _work(items):
    c = dict(items)
    if c["kind"] == "ingest":
        n = c["w"] * c["h"]
        return float(n * (SOURCES[c["src"]][1] + 4)), float(n)
    nbytes = flops = 0.0
    for f in _frames(c, 1):
        nbytes += f.algorithmic_bytes()
        for p in f.passes:
            # the clip transform of a vertex, the setup of a triangle
            flops += 28.0 * p.nverts + 120.0 * p.ntris
        if c["kind"] == "soup":  # the z of every fragment: the on-screen share of the triangles' mean area
            flops += 14.0 * c["tris"] * c["area_hi"] / math.log(c["area_hi"]) * 0.69
        for t in f.targets:
            nbytes += t.width * t.height * t.bpp  # the clears
            flops += 20.0 * t.width * t.height    # one visible fragment a pixel
            if c["kind"] == "serve" and t.name in READBACK:
                nbytes += t.width * t.height * t.bpp
    return nbytes, flops


def work(case):
    b, f = _work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The depth targets in 64 bits
# ---------------------------------------------------------------------------
_POSITION = {abi.SHADER_VCOLOR: 4}


def _mat(m):
    return torch.tensor(list(m), dtype=torch.float64, device="cuda").reshape(4, 4)


def _clip_positions(p):
    """Clip-space vertices of a pass, from its packed f32 inputs, in 64 bits."""
    n = _POSITION.get(p.desc.shader, 3)
    raw = np.ascontiguousarray(p.vertices).reshape(p.nverts, p.layout.stride)
    raw = np.ascontiguousarray(raw[:, p.layout.position:p.layout.position + 4 * n]).view(np.float32)
    v = torch.from_numpy(raw.astype(np.float64)).cuda()
    if n == 3:
        v = torch.cat([v, torch.ones_like(v[:, :1])], 1)
    u = p.uniforms
    if p.desc.shader == abi.SHADER_PHONG:
        return v @ (_mat(u.proj) @ _mat(u.view) @ _mat(u.model)).T
    return v @ _mat(u.mvp).T


def _depth_of(p, depth, budget):
    """Rasterises the triangles of a pass into `depth` (a 64-bit tensor, Less
    with write); the pixel-triangle pairs that it may still look at."""
    h, w = depth.shape
    v = _clip_positions(p)
    idx = torch.from_numpy(p.indices.astype(np.int64)).cuda()
    ndc = v[:, :3] / v[:, 3:]
    tri = ndc[idx[:len(idx) // 3 * 3]].reshape(-1, 3, 3)
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cross = e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]
    keep = cross != 0
    if p.desc.cull != abi.CULL_NONE:
        keep &= cross * (1.0 if p.desc.cull == abi.CULL_BACK else -1.0) >= 0
    tri = tri[keep]
    sx, sy, z = w * (tri[..., 0] * 0.5 + 0.5), h * (tri[..., 1] * -0.5 + 0.5), tri[..., 2]
    x0, x1 = sx.amin(1).clamp(0, w).floor().long(), (sx.amax(1) + 1).clamp(0, w).floor().long()
    y0, y1 = sy.amin(1).clamp(0, h).floor().long(), (sy.amax(1) + 1).clamp(0, h).floor().long()
    n = (x1 - x0).clamp(min=0) * (y1 - y0).clamp(min=0)
    ends = n.cumsum(0)
    total = int(ends[-1]) if len(ends) else 0
    if total > budget:
        return None
    area = (sx[:, 1] - sx[:, 0]) * (sy[:, 2] - sy[:, 0]) - (sy[:, 1] - sy[:, 0]) * (sx[:, 2] - sx[:, 0])
    flat = depth.view(-1)
    step = 1 << 24
    for a in range(0, total, step):
        k = torch.arange(a, min(a + step, total), device="cuda")
        t = torch.searchsorted(ends, k, right=True)
        k = k - (ends[t] - n[t])
        wide = (x1 - x0)[t]
        px, py = x0[t] + k % wide, y0[t] + k // wide
        b = []
        for i, j in ((1, 2), (2, 0)):
            b.append(((sx[t, j] - sx[t, i]) * (py - sy[t, i]) - (sy[t, j] - sy[t, i]) * (px - sx[t, i])) / area[t])
        b.append(1.0 - b[0] - b[1])
        zz = z[t, 0] * b[0] + z[t, 1] * b[1] + z[t, 2] * b[2]
        hit = (b[0] >= 0) & (b[1] >= 0) & (b[2] >= 0)
        if p.desc.z_clip:
            hit &= (zz >= p.desc.z_clip_min) & (zz <= p.desc.z_clip_max)
        flat.scatter_reduce_(0, (py * w + px)[hit], zz[hit], "amin")
    return budget - total


def exact(case, seed):
    if case["kind"] in ("wire", "lines", "serve", "ingest"):
        return None  # lines have no area to compare; the others return bytes
    if case.get("test", "less") != "less":
        return None
    budget, got = 3 << 30, []
    for f in _frames(case, seed):
        made = {}
        for p in f.passes:
            t = f.target(p.depth)
            d = torch.full((t.height, t.width), float(np.float32(t.clear)), dtype=torch.float64, device="cuda")
            budget = _depth_of(p, d, budget)
            if budget is None:
                return None
            made[p.depth] = d
        got += [made[t.name].reshape(-1) for t in f.targets if t.fmt == abi.FMT_R32F]
    depth = torch.cat(got)
    if case["kind"] == "host":
        depth = depth.reshape(case["h"], case["w"])
    return {"color": None, "depth": depth}
