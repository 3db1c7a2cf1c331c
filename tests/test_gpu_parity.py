"""GPU pipeline vs the CPU oracle on the same seeded inputs.

Bar: depth bit-exact, per-pass candidate-fragment counts exact, colour exact
for shaders without transcendental functions and within +-1 LSB per 8-bit
channel for the Phong shader (its lighting uses the hardware reciprocal square
root and power; texel and shadow-map coordinates stay exact); on an f32 colour
target Phong within a relative 1e-5, the others bit-exact.
"""
import ctypes as C

import numpy as np
import pytest

from euc_gb300 import abi, scenes
from frameutil import assert_same_inputs, assert_targets_match, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def _sphere(seed=3, **kw):
    return lambda: scenes.sphere_frame(seed=seed, **kw)


def _mod(make, **desc):
    def wrapped():
        f = make()
        for p in f.passes:
            for k, v in desc.items():
                setattr(p.desc, k, v)
        return f
    return wrapped


def _soup(seed=1, w=320, h=180, n=4000, hi=3000.0, alpha=False, **desc):
    return _mod(lambda: scenes.soup_frame(seed=seed, width=w, height=h, ntris=n, area_hi=hi, alpha=alpha), **desc)


def _fmt(make, fmt):
    def wrapped():
        f = make()
        t = f.target("color")
        f.targets[f.targets.index(t)] = scenes.TargetSpec("color", t.width, t.height, fmt, 0x80402010)
        return f
    return wrapped


def _f32(make, clear=(0.25, 0.5, 0.75, 1.0)):
    """The colour target as four floats a pixel (Buffer2d<[f32; 4]>)."""
    def wrapped():
        f = make()
        t = f.target("color")
        f.targets[f.targets.index(t)] = scenes.TargetSpec("color", t.width, t.height, abi.FMT_RGBA32F, clear)
        return f
    return wrapped


def _clear(make, name, value):
    def wrapped():
        f = make()
        f.target(name).clear = value
        return f
    return wrapped


def _perspective_soup(seed=7, zclip=True):
    """Soup with w != 1 and z outside the clip range (per-fragment z clip)."""
    def make():
        f = scenes.soup_frame(seed=seed, width=257, height=131, ntris=3000, area_hi=4000.0)
        p = f.passes[0]
        rng = np.random.default_rng(seed + 100)
        vb = p.vertices.reshape(p.nverts, 20).copy()
        pos = vb[:, :16].copy().view(np.float32).reshape(-1, 4)
        w = rng.uniform(0.5, 2.0, len(pos)).astype(np.float32)
        pos[:, 0] *= w
        pos[:, 1] *= w
        pos[:, 2] = rng.uniform(-0.3, 1.3, len(pos)).astype(np.float32) * w
        pos[:, 3] = w
        vb[:, :16] = pos.view(np.uint8).reshape(-1, 16)
        p.vertices = vb.reshape(-1)
        if not zclip:
            p.desc.z_clip = 0
        return f
    return make


def _knot(aa, seed=2, w=320, h=180, shadow=256):
    return lambda: scenes.knot_frame(seed=seed, width=w, height=h, shadow_size=shadow, tubular=180, radial=20,
                                     tex_size=64, aa_level=aa)


def _textured(filt, wrap, seed=4, w=200, h=150):
    def make():
        rng = np.random.default_rng(seed)
        pos, nrm, uv, idx = scenes.uv_sphere(20, 10)
        uv = uv * 3.0 - 1.0  # exercise the wrap modes outside [0, 1]
        buf, stride, offs = scenes.pack_vertices(pos, uv)
        model = scenes.translation(0, 0, 2.6) @ scenes.quat_rotation(rng)
        proj = scenes.perspective_lh_zo(1.0, w / h, 0.1, 50.0)
        u = abi.TexturedUniforms()
        u.mvp = scenes.f32mat(proj @ model)
        tex = rng.integers(0, 256, (13, 17, 4), dtype=np.uint8)
        p = scenes.PassSpec(scenes.make_desc(abi.SHADER_TEXTURED), scenes.layout(stride, position=offs[0], uv=offs[1]),
                            buf, len(pos), idx, u, [scenes.SamplerSpec("tex", tex, filt, wrap, 1.0)],
                            pixel="color", depth="depth")
        return scenes.FrameSpec("tex", [scenes.TargetSpec("color", w, h, abi.FMT_BGRA8, 0x20406080),
                                        scenes.TargetSpec("depth", w, h, abi.FMT_R32F, 1.0)], [p])
    return make


def _flat(seed=6):
    def make():
        f = scenes.sphere_frame(seed=seed, width=160, height=120, lon=16, lat=8)
        p = f.passes[0]
        u = abi.FlatUniforms()
        u.mvp = p.uniforms.mvp
        u.color = (C.c_float * 4)(0.25, 0.5, 0.75, 1.0)
        p.uniforms = u
        p.desc.shader = abi.SHADER_FLAT
        return f
    return make


def _unindexed():
    def make():
        f = scenes.soup_frame(seed=9, width=150, height=100, ntris=500, area_hi=800.0)
        p = f.passes[0]
        nv = p.nverts
        vb = p.vertices.reshape(nv, 20)[p.indices].reshape(-1)  # un-permute
        p.vertices = np.ascontiguousarray(vb)
        p.indices = None
        return f
    return make


def _ragged(nverts, prims=abi.PRIM_TRIANGLE_LIST, indexed=False):
    """A stream of `nverts` vertices: empty, or shorter than one primitive."""
    def make():
        rng = np.random.default_rng(nverts)
        clip = np.concatenate([rng.uniform(-0.9, 0.9, (nverts, 2)), rng.uniform(0.1, 0.9, (nverts, 1)),
                               np.ones((nverts, 1))], axis=1)
        col = np.full((nverts, 4), 200, dtype=np.uint8)
        idx = np.arange(nverts, dtype=np.uint32)[::-1].copy() if indexed else None
        return scenes.clip_triangles_frame(clip, col, 32, 24, indices=idx, primitives=prims)
    return make


def _lines(seed=31, prims=abi.PRIM_LINE_LIST, **kw):
    return lambda: scenes.lines_frame(seed=seed, prims=prims, **kw)


CASES = {
    "sphere640x480": (_sphere(seed=3), 0),
    "sphere_small_odd": (_sphere(seed=5, width=97, height=61, lon=24, lat=12), 0),
    "sphere_cull_none": (_mod(_sphere(seed=8), cull=abi.CULL_NONE), 0),
    "sphere_cull_front_yup": (_mod(_sphere(seed=8), cull=abi.CULL_FRONT, y_axis=abi.Y_UP), 0),
    "sphere_bands_seq": (_mod(_sphere(seed=11), band_rows=abi.BANDS_SEQ), 0),
    "sphere_bands_7": (_mod(_sphere(seed=11), band_rows=7), 0),
    "sphere_par_small_fallback": (_sphere(seed=12, width=64, height=64, lon=16, lat=8), 0),
    "sphere_par_empty": (_mod(_sphere(seed=12, width=64, height=64, lon=16, lat=8), flags=abi.FLAG_PAR_EMPTY), 0),
    "soup_less": (_soup(), 0),
    "soup_greater": (_clear(_soup(seed=2, depth_test=abi.TEST_GREATER), "depth", 0.0), 0),
    "soup_equal_write": (_clear(_soup(seed=3, depth_test=abi.TEST_EQUAL), "depth", 0.5), 0),
    "soup_none_write": (_soup(seed=4, depth_test=abi.TEST_NONE), 0),
    "soup_less_pass": (_soup(seed=5, depth_write=0), 0),
    "soup_depth_only": (_soup(seed=6, pixel_write=0), 0),
    "soup_color_only": (_soup(seed=13, depth_test=abi.TEST_NONE, depth_write=0), 0),
    "soup_perspective_zclip": (_perspective_soup(7, True), 0),
    "soup_perspective_noclip": (_perspective_soup(8, False), 0),
    "soup_large_tris": (_soup(seed=14, w=640, h=360, n=300, hi=150000.0), 0),
    "knot_aa0": (_knot(0), 1),
    "knot_aa1": (_knot(1), 1),
    "knot_aa2": (_knot(2, seed=3), 1),
    "knot_aa3": (_knot(3, seed=4, w=333, h=211), 1),
    "tex_linear_tile": (_textured(abi.FILTER_LINEAR, abi.WRAP_TILE), 0),
    "tex_linear_clamp": (_textured(abi.FILTER_LINEAR, abi.WRAP_CLAMP), 0),
    "tex_linear_mirror": (_textured(abi.FILTER_LINEAR, abi.WRAP_MIRROR), 0),
    "tex_linear_none": (_textured(abi.FILTER_LINEAR, abi.WRAP_NONE), 0),
    "tex_nearest_tile": (_textured(abi.FILTER_NEAREST, abi.WRAP_TILE), 0),
    "tex_nearest_clamp": (_textured(abi.FILTER_NEAREST, abi.WRAP_CLAMP), 0),
    "tex_nearest_mirror": (_textured(abi.FILTER_NEAREST, abi.WRAP_MIRROR), 0),
    "tex_nearest_none": (_textured(abi.FILTER_NEAREST, abi.WRAP_NONE), 0),
    "flat": (_flat(), 0),
    "f32_sphere": (_f32(_sphere(seed=3)), 0),
    "f32_flat": (_f32(_flat()), 0),
    "f32_tex_linear_tile": (_f32(_textured(abi.FILTER_LINEAR, abi.WRAP_TILE)), 0),
    "f32_soup_less": (_f32(_soup(seed=2)), 0),
    "f32_alpha_soup": (_f32(_soup(seed=21, alpha=True)), 0),
    "f32_alpha_soup_msaa1": (_f32(_soup(seed=24, alpha=True, aa_level=1)), 0),
    "f32_knot_aa1": (_f32(_knot(1)), 1),
    "unindexed": (_unindexed(), 0),
    # order-dependent blend: per-pixel fragment lists replayed in order
    "alpha_soup_less": (_soup(seed=21, alpha=True), 0),
    "alpha_soup_less_pass": (_soup(seed=22, alpha=True, depth_write=0), 0),
    "alpha_soup_no_depth": (_soup(seed=23, alpha=True, depth_test=abi.TEST_NONE, depth_write=0), 0),
    "alpha_soup_msaa1": (_soup(seed=24, alpha=True, aa_level=1), 0),
    "alpha_soup_msaa2_bands": (_soup(seed=25, w=333, h=177, alpha=True, aa_level=2, band_rows=11), 0),
    "alpha_soup_rgb8": (_fmt(_soup(seed=26, alpha=True), abi.FMT_RGB8), 0),
    "alpha_soup_bgra8": (_fmt(_soup(seed=27, alpha=True), abi.FMT_BGRA8), 0),
    # replace blends forced through the ordered path must give the same bytes
    # empty and ragged streams: nothing is drawn (primitives.rs collect_primitive)
    "empty_stream": (_ragged(0), 0),
    "empty_indexed": (_ragged(0, indexed=True), 0),
    "two_vertices": (_ragged(2), 0),
    "five_vertices_indexed": (_ragged(5, indexed=True), 0),
    "one_vertex_lines": (_ragged(1, prims=abi.PRIM_LINE_LIST), 0),
    "five_vertices_line_tris": (_ragged(5, prims=abi.PRIM_LINE_TRIANGLE_LIST), 0),
    # lines (lines.rs) and the wireframe example's LineTriangleList pipeline
    "lines_less": (_lines(), 0),
    "lines_tri_list": (_lines(seed=32, prims=abi.PRIM_LINE_TRIANGLE_LIST, nlines=2000), 0),
    "lines_perspective_zclip": (_lines(seed=33, perspective=True), 0),
    "lines_perspective_noclip": (_lines(seed=34, perspective=True, z_clip=None, depth_test=abi.TEST_NONE), 0),
    "lines_equal_pass": (_clear(_lines(seed=35, depth_test=abi.TEST_EQUAL, depth_write=0), "depth", 0.5), 0),
    "lines_msaa1_bands": (_lines(seed=36, width=333, height=177, aa_level=1, band_rows=9), 0),
    "lines_msaa2": (_lines(seed=37, aa_level=2), 0),
    "lines_long_offscreen": (_lines(seed=38, nlines=300, len_lo=500.0, len_hi=5000.0, extent=2.0), 0),
    "lines_alpha": (_lines(seed=39, alpha=True), 0),
    "lines_ordered": (_lines(seed=40, flags=abi.FLAG_ORDERED), 0),
    "wireframe_bgra8": (lambda: scenes.wireframe_frame(seed=41), 0),
    "wireframe_msaa1_rgba8": (lambda: scenes.wireframe_frame(seed=42, fmt=abi.FMT_RGBA8, aa_level=1), 0),
    # built-in geometry stages (Pipeline::geometry)
    "geom_sphere_subdivide": (_mod(_sphere(seed=43), geometry=abi.GEOM_SUBDIVIDE), 0),
    "geom_soup_shrink": (_soup(seed=44, geometry=abi.GEOM_SHRINK, geometry_param=0.6), 0),
    "geom_soup_duplicate": (_soup(seed=45, geometry=abi.GEOM_DUPLICATE, geometry_param=0.05), 0),
    "geom_soup_discard": (_soup(seed=46, geometry=abi.GEOM_DISCARD, geometry_param=0.5), 0),
    "geom_knot_subdivide_aa1": (_mod(_knot(1, seed=47), geometry=abi.GEOM_SUBDIVIDE), 1),
    "geom_tex_shrink": (_mod(_textured(abi.FILTER_LINEAR, abi.WRAP_TILE, seed=48), geometry=abi.GEOM_SHRINK,
                             geometry_param=0.8), 0),
    "geom_alpha_duplicate": (_soup(seed=49, alpha=True, geometry=abi.GEOM_DUPLICATE, geometry_param=-0.03), 0),
    "ordered_sphere": (_mod(_sphere(seed=3), flags=abi.FLAG_ORDERED), 0),
    "ordered_soup_less": (_soup(seed=1, flags=abi.FLAG_ORDERED), 0),
    "ordered_soup_equal": (_clear(_soup(seed=3, depth_test=abi.TEST_EQUAL, flags=abi.FLAG_ORDERED), "depth", 0.5), 0),
    "ordered_soup_greater": (_clear(_soup(seed=2, depth_test=abi.TEST_GREATER, flags=abi.FLAG_ORDERED), "depth", 0.0), 0),
    "ordered_knot_aa1": (_mod(_knot(1), flags=abi.FLAG_ORDERED), 1),
    "ordered_tex_linear_mirror": (_mod(_textured(abi.FILTER_LINEAR, abi.WRAP_MIRROR), flags=abi.FLAG_ORDERED), 0),
}


_ORACLE = {}


def _oracle(name):
    """The oracle's targets and statistics of case `name`, computed once."""
    if name not in _ORACLE:
        _ORACLE[name] = run_oracle(CASES[name][0]())
    return _ORACLE[name]


@pytest.fixture(scope="module")
def strip_ctx():
    """A context that sends every scene the shared-memory strips can take to
    them, whatever its overdraw (the default routes only overdrawn scenes)."""
    from euc_gb300 import capi
    ctx = capi.Context(0)
    ctx.set_tuning(strip_path=2)
    yield ctx
    ctx.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_gpu_matches_oracle(name, gpu_ctx):
    make, tol = CASES[name]
    assert_same_inputs(make(), make())
    ref, ref_stats = _oracle(name)
    got, got_stats = run_gpu(gpu_ctx, make())
    assert [s[0] for s in got_stats] == [s[0] for s in ref_stats]
    assert [s[1] for s in got_stats] == [s[1] for s in ref_stats], "candidate fragment counts"
    assert [s[2] for s in got_stats] == [s[2] for s in ref_stats], "culled primitive counts"
    assert_targets_match(make(), ref, got, color_tol=tol)


@pytest.mark.parametrize("name", sorted(CASES))
def test_gpu_matches_oracle_on_the_strips(name, strip_ctx):
    make, tol = CASES[name]
    ref, ref_stats = _oracle(name)
    got, got_stats = run_gpu(strip_ctx, make())
    assert [s[0] for s in got_stats] == [s[0] for s in ref_stats]
    assert [s[1] for s in got_stats] == [s[1] for s in ref_stats], "candidate fragment counts"
    assert [s[2] for s in got_stats] == [s[2] for s in ref_stats], "culled primitive counts"
    assert_targets_match(make(), ref, got, color_tol=tol)


@pytest.mark.parametrize("strips", [False, True])
def test_index_out_of_bounds_draws_nothing(gpu_ctx, strip_ctx, strips):
    ctx = strip_ctx if strips else gpu_ctx
    def make():
        f = scenes.sphere_frame(seed=1, width=120, height=90, lon=12, lat=6)
        f.passes[0].indices = f.passes[0].indices.copy()
        f.passes[0].indices[-1] = f.passes[0].nverts  # one past the end: index.rs:53 panics
        return f
    ref, ref_stats = run_oracle(make())
    got, got_stats = run_gpu(ctx, make())
    assert ref_stats[0][0] == abi.ERR_INDEX_OOB
    assert got_stats[0][0] == abi.ERR_INDEX_OOB
    clean = make().alloc_host_targets()
    for k in clean:
        assert np.array_equal(got[k], clean[k])


def _layers(n, w=37, h=19, seed=60, **desc):
    """n full-target triangles over each other with random depths, in a
    shuffled order, blended src-over: every pixel's list has n fragments."""
    def make():
        rng = np.random.default_rng(seed + n)
        tri = np.array([[-1.5, -1.5], [4.0, -1.5], [-1.5, 4.0]], dtype=np.float32)
        clip = np.zeros((n, 3, 4), dtype=np.float32)
        clip[:, :, :2] = tri
        clip[:, :, 2] = rng.uniform(0.05, 0.95, (n, 1))
        clip[:, :, 3] = 1.0
        col = rng.integers(0, 256, (n * 3, 4), dtype=np.uint8)
        kw = dict(blend=abi.BLEND_ALPHA)
        kw.update(desc)
        return scenes.clip_triangles_frame(clip.reshape(-1, 4), col, w, h, **kw)
    return make


@pytest.mark.parametrize("test,write", [(abi.TEST_LESS, 1), (abi.TEST_NONE, 0), (abi.TEST_GREATER, 0)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 41])
def test_ordered_lists_at_the_window_edges(gpu_ctx, n, test, write):
    """Lists of one window, exactly full, one over and several windows, and a
    fragment buffer that has to grow (more than four fragments a pixel)."""
    make = _layers(n, depth_test=test, depth_write=write, depth_clear=0.5 if test == abi.TEST_GREATER else 1.0)
    ref, ref_stats = run_oracle(make())
    got, got_stats = run_gpu(gpu_ctx, make())
    assert [s[1] for s in got_stats] == [s[1] for s in ref_stats]
    assert_targets_match(make(), ref, got)
    from euc_gb300 import capi
    fresh = capi.Context(0)  # its buffer starts at four fragments a pixel
    try:
        got, _ = run_gpu(fresh, make())
    finally:
        fresh.close()
    assert_targets_match(make(), ref, got)


@pytest.mark.parametrize("clear", [1.0, 0.0, -0.0, float("inf"), float("nan")])
@pytest.mark.parametrize("z", [0.0, -0.0, 1.0, 0.5])
def test_depths_at_the_edges_of_the_positive_class(gpu_ctx, strip_ctx, z, clear):
    """Triangles whose vertex depths are at or above +0 take a shorter key:
    zeros of both signs, the clip limits, and targets that hold infinity or a
    NaN, on both raster paths; one triangle's w is tiny (weights near the f32
    limit), one mixes the zeros."""
    def make():
        rng = np.random.default_rng(71)
        clip = np.zeros((9, 3, 4), dtype=np.float32)
        clip[:, :, :2] = rng.uniform(-1.3, 1.3, (9, 3, 2))
        clip[:, :, 2] = np.float32(z)
        clip[1:4, :, 2] = rng.uniform(0.0, 1.0, (3, 3))
        clip[4, 1, 2] = -0.0
        clip[5, 2, 2] = 0.0
        clip[:, :, 3] = 1.0
        clip[6] *= np.float32(1e-30)
        clip[7] *= np.float32(1e30)
        col = rng.integers(0, 256, (27, 4), dtype=np.uint8)
        return scenes.clip_triangles_frame(clip.reshape(-1, 4), col, 61, 43, depth_clear=clear)
    ref, ref_stats = run_oracle(make())
    for ctx in (gpu_ctx, strip_ctx):
        got, got_stats = run_gpu(ctx, make())
        assert [s[1] for s in got_stats] == [s[1] for s in ref_stats]
        a, b = ref["depth"].view(np.uint32), got["depth"].view(np.uint32)
        assert np.array_equal(a, b)
        assert np.array_equal(ref["color"], got["color"])


@pytest.mark.parametrize("prims", [abi.PRIM_TRIANGLE_LIST, abi.PRIM_LINE_LIST])
@pytest.mark.parametrize("n,w,h", [(1, 70, 33), (31, 64, 32), (33, 64, 33), (257, 97, 61), (1023, 1, 50), (4000, 255, 9),
                                   (32768, 160, 90), (32769, 160, 90), (300, 1024, 1024), (300, 1024, 1025)])
def test_frames_at_the_edges_of_the_small_scene_path(prims, n, w, h):
    """Primitive groups, setup blocks and both limits of the three-launch path
    (32768 primitives, 2^20 pixels), one scene more than fits included; three
    calls: plain, recorded, replayed with other inputs."""
    from euc_gb300 import capi
    ctx = capi.Context(0)
    try:
        for seed in (80, 81, 82):
            if prims == abi.PRIM_LINE_LIST:
                make = lambda: scenes.lines_frame(seed=seed, width=w, height=h, nlines=n, len_hi=40.0)
            else:
                make = lambda: scenes.soup_frame(seed=seed, width=w, height=h, ntris=n, area_hi=60.0)
            ref, ref_stats = run_oracle(make())
            got, got_stats = run_gpu(ctx, make())
            assert got_stats == ref_stats
            assert_targets_match(make(), ref, got)
        bad = make()
        bad.passes[0].indices = bad.passes[0].indices.copy()
        bad.passes[0].indices[-1] = bad.passes[0].nverts
        got, got_stats = run_gpu(ctx, bad)
        assert got_stats[0][0] == abi.ERR_INDEX_OOB
        clean = bad.alloc_host_targets()
        assert all(np.array_equal(got[k], clean[k]) for k in clean)
    finally:
        ctx.close()


@pytest.mark.parametrize("n,area", [(40, 30000.0), (700, 3000.0), (9000, 900.0), (60000, 120.0)])
def test_strip_units_of_every_size(strip_ctx, n, area):
    """Few entries (units of kStripUnitMin) to many (full units): the unit
    size follows from the launch's entry count."""
    make = _soup(seed=90, w=300, h=200, n=n, hi=area)
    ref, ref_stats = run_oracle(make())
    got, got_stats = run_gpu(strip_ctx, make())
    assert got_stats == ref_stats
    assert_targets_match(make(), ref, got)


@pytest.mark.parametrize("fmt", [abi.FMT_RGBA8, abi.FMT_RGB8])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 7), (32, 8), (33, 9), (127, 3), (128, 16), (129, 17), (255, 5), (256, 8), (257, 9),
                                 (700, 1)])
def test_row_segments_at_their_edges(gpu_ctx, strip_ctx, w, h, fmt):
    """Targets covered whole, at the edges of the 128- and 256-pixel row
    segments of the resolve and the key seeds; the batch's kernels (strip_ctx
    keeps off the small-scene path) and the frame's."""
    def make():
        f = _layers(5, w=w, h=h, blend=abi.BLEND_REPLACE, pixel_fmt=fmt)()
        return f
    ref, ref_stats = run_oracle(make())
    for ctx in (gpu_ctx, strip_ctx):
        got, got_stats = run_gpu(ctx, make())
        assert got_stats == ref_stats
        assert_targets_match(make(), ref, got)


@pytest.mark.parametrize("w,h", [(1, 1), (33, 7), (64, 4), (257, 5), (190, 101)])
@pytest.mark.parametrize("kind", ["soup", "perspective", "phong", "lines"])
def test_ordered_frames_on_both_paths(gpu_ctx, strip_ctx, kind, w, h):
    """src-over scenes through the small-scene path and through the batch's
    kernels (strip_ctx keeps off the former): rows at the edges of 32 lanes
    and of the pixel scan's blocks, rectangles smaller than the target, runs
    of uneven lists whose fragments the warp shades together, rows with and
    without the guard tests, and a shader of every record size."""
    if kind == "soup":
        make = _soup(seed=95, w=w, h=h, n=700, hi=0.2 * w * h + 20.0, alpha=True)
    elif kind == "lines":
        make = lambda: scenes.lines_frame(seed=95, width=w, height=h, nlines=300, len_hi=40.0)
    elif kind == "phong":
        make = _knot(0, w=w, h=h, shadow=64)
    else:
        make = _sphere(width=w, height=h)
    base = make
    def make():
        f = base()
        f.passes[-1].desc.blend = abi.BLEND_ALPHA
        return f
    ref, ref_stats = run_oracle(make())
    for ctx in (gpu_ctx, strip_ctx):
        got, got_stats = run_gpu(ctx, make())
        assert [s[:2] for s in got_stats] == [s[:2] for s in ref_stats]
        # a Phong byte may be one step off, and so may the blend's rounding of it
        assert_targets_match(make(), ref, got, 2 if kind == "phong" else 0)


@pytest.mark.parametrize("order,pad,shift", [("pnu", 0, 0), ("pnu", 1, 0), ("pnu", 4, 0), ("pnu", 0, 4), ("pnu", 4, 8),
                                             ("pun", 0, 0), ("npu", 0, 0), ("pn", 0, 0), ("pn", 2, 0)])
def test_phong_vertices_of_every_layout(gpu_ctx, strip_ctx, order, pad, shift):
    """Packed vertices on 16-byte boundaries take two loads: the same values
    with padding between them, on other boundaries, in another order and
    without texture coordinates give the oracle's image, and the layouts that
    hold the same attributes the packed one's bytes."""
    import torch
    from euc_gb300 import frames
    base = _knot(0, w=97, h=61, shadow=64)()
    spec = base.passes[-1]
    words = np.frombuffer(spec.vertices.tobytes(), dtype=np.float32).reshape(-1, 8)
    attrs = {"p": words[:, 0:3], "n": words[:, 3:6], "u": words[:, 6:8]}

    def images(order, pad, shift):
        cols, at, offs = [], 0, {"u": -1}
        for c in order:
            offs[c] = 4 * at
            cols.append(attrs[c])
            at += attrs[c].shape[1]
        cols.append(np.full((len(words), pad), 7.0, dtype=np.float32))
        f = _knot(0, w=97, h=61, shadow=64)()
        p = f.passes[-1]
        p.vertices = np.ascontiguousarray(np.concatenate(cols, axis=1)).view(np.uint8).reshape(-1)
        p.layout = scenes.layout(4 * (at + pad), position=offs["p"], normal=offs["n"], uv=offs["u"])
        ref, _ = run_oracle(f)
        got = []
        for ctx in (gpu_ctx, strip_ctx):
            df = frames.DeviceFrame(f, "cuda:0")
            df.clear()
            for k, q in enumerate(f.passes):
                desc, uni, keep = df.bound_pass(k)
                v, i, _ = df.passes[k]
                if q is p:
                    v = torch.cat([torch.zeros(shift, dtype=torch.uint8, device=v.device), v])
                px = frames.tensor_target(df.targets[q.pixel] if q.pixel else None,
                                          f.target(q.pixel).fmt if q.pixel else abi.FMT_NONE)
                dp = frames.tensor_target(df.targets[q.depth] if q.depth else None, abi.FMT_R32F)
                assert ctx.render(desc.desc, uni, desc.layout, v.data_ptr() + (shift if q is p else 0), q.nverts,
                                  i.data_ptr(), i.numel(), px, dp, frames._stream_ptr(None)) == abi.OK
                torch.cuda.synchronize()
                del keep
            got.append(df.to_host())
            assert_targets_match(f, ref, got[-1], 1)
        return got

    got = images(order, pad, shift)
    if "u" in order:
        for a, b in zip(got, images("pnu", 0, 0)):
            for name in a:
                assert np.array_equal(a[name].view(np.uint8), b[name].view(np.uint8)), name


@pytest.mark.parametrize("layers", [3, 41])
@pytest.mark.parametrize("blended_first", [False, True])
def test_a_batch_draws_its_blended_scenes_over_its_opaque_ones(layers, blended_first):
    """An opaque and a src-over scene on the same targets and two more on
    targets of their own, in one batch call: the blended scene lands on the
    opaque image whatever the order in the call, with lists that fit the first
    fragment buffer and with lists it has to grow for."""
    import torch
    from euc_gb300 import capi, frames

    def make():
        opaque, blended = _soup(seed=61, w=37, h=19, n=60, hi=150.0)(), _layers(layers)()
        shared = scenes.FrameSpec("shared", opaque.targets, [opaque.passes[0], blended.passes[0]])
        return [shared, _soup(seed=62, w=37, h=19, n=200, hi=90.0)(), _layers(layers, seed=63)()]
    ctx = capi.Context(0)
    try:
        dfs = [frames.DeviceFrame(f, "cuda:0") for f in make()]
        arr, keep = [], []
        for df in dfs:
            df.clear()
            for k in range(len(df.frame.passes)):
                s, kp = df.scene(k)
                arr.append(s)
                keep.append(kp)
        assert ctx.render_batch(arr[::-1] if blended_first else arr, frames._stream_ptr(None)) == abi.OK
        assert ctx.sync(frames._stream_ptr(None)) == abi.OK
        candidates = ctx.stats(frames._stream_ptr(None)).candidates
        total = 0
        for f, df in zip(make(), dfs):
            ref, ref_stats = run_oracle(f)
            total += sum(s[1] for s in ref_stats)
            assert_targets_match(f, ref, df.to_host())
        assert candidates == total
    finally:
        ctx.close()


def test_the_fragment_buffer_is_sized_by_the_blended_scenes(gpu_ctx):
    """A 64x64 blended scene beside large opaque ones takes list space for its
    own pixels, not for the batch's (8.4 M: 268 MB at four fragments each)."""
    import torch
    from euc_gb300 import capi, frames
    opaque = [scenes.soup_frame(seed=k, width=512, height=512, ntris=50, area_hi=500.0) for k in range(32)]
    last = [scenes.soup_frame(seed=9, width=64, height=64, ntris=50, area_hi=500.0, alpha=a) for a in (False, True)]
    batches = [frames.DeviceBatch(opaque + [f]) for f in last]
    ctx = capi.Context(0)
    try:
        frames.render_batch(ctx, batches[0])  # the scratch of every scene, but for the lists
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        frames.render_batch(ctx, batches[1])
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] < 32 << 20
        got = batches[1].frames[-1].to_host()
        ref, _ = run_oracle(last[1])
        assert_targets_match(last[1], ref, got)
    finally:
        ctx.close()


@pytest.mark.parametrize("parts", ["KO", "KkOo", "KkOoL", "KLL", "OoL", "EO", "KE", "KeL", "eK"])
def test_batches_of_ordered_and_other_scenes(parts):
    """Each raster launch of a mixed batch takes the items of its own scenes:
    opaque ones (K, k), blended triangles (O, o) and lines (L), and scenes none
    of whose primitives has a row (E opaque, e blended), in one call on a fresh
    context, twice (the second with the buffers of the first)."""
    from euc_gb300 import capi, frames
    off = np.tile(np.array([5.0, 5.0, 0.5, 1.0], dtype=np.float32), (300, 1))
    kinds = {
        "K": lambda: scenes.soup_frame(seed=1, width=200, height=120, ntris=3000, area_hi=300.0),
        "k": lambda: scenes.lines_frame(seed=2, width=97, height=61, nlines=300, len_hi=60.0),
        "O": lambda: scenes.soup_frame(seed=3, width=150, height=90, ntris=700, area_hi=900.0, alpha=True),
        "o": lambda: scenes.soup_frame(seed=4, width=33, height=17, ntris=257, area_hi=300.0, alpha=True),
        "L": lambda: scenes.lines_frame(seed=5, width=128, height=65, nlines=2000, len_hi=90.0, alpha=True),
        "E": lambda: scenes.clip_triangles_frame(off, np.zeros((300, 4), np.uint8), 64, 64),
        "e": lambda: scenes.clip_triangles_frame(off, np.zeros((300, 4), np.uint8), 64, 64, blend=abi.BLEND_ALPHA),
    }
    ctx = capi.Context(0)
    try:
        for _ in range(2):
            made = [kinds[c]() for c in parts]
            dfs = [frames.DeviceFrame(f, "cuda:0") for f in made]
            frames.render_batch(ctx, dfs)
            assert ctx.sync(frames._stream_ptr(None)) == abi.OK
            candidates, total = ctx.stats(frames._stream_ptr(None)).candidates, 0
            for f, df in zip(made, dfs):
                ref, ref_stats = run_oracle(f)
                total += ref_stats[0][1]
                assert_targets_match(f, ref, df.to_host())
            assert candidates == total
    finally:
        ctx.close()


@pytest.mark.parametrize("w,h", [(1, 700), (3, 401), (4, 64), (5, 333), (8, 33), (9, 100), (16, 257), (17, 65), (63, 40),
                                 (64, 33), (65, 33), (127, 20), (128, 9), (129, 9)])
@pytest.mark.parametrize("test,write", [(abi.TEST_LESS, 1), (abi.TEST_NONE, 0)])
def test_narrow_targets(gpu_ctx, strip_ctx, w, h, test, write):
    """Covered rectangles at the edges of the lanes that a row of the key seeds
    (eight pixels a lane) and of the resolve (four) takes, at the target's left
    edge and off it, on both raster paths."""
    def make(k):
        f = _layers(4, w=w + 5 * k, h=h, blend=abi.BLEND_REPLACE, depth_test=test, depth_write=write)()
        if k:  # the last w columns of the target only
            clip = np.zeros((6, 4), dtype=np.float32)
            x0 = 2.0 * 5 / (w + 5) - 1.0
            clip[:, :2] = [(x0, -1), (1, -1), (x0, 1), (1, -1), (1, 1), (x0, 1)]
            clip[:, 2:] = [0.25, 1.0]
            f = scenes.clip_triangles_frame(clip, np.arange(24, dtype=np.uint8).reshape(6, 4), w + 5, h,
                                            depth_test=test, depth_write=write)
        return f
    for k in (0, 1):
        ref, ref_stats = run_oracle(make(k))
        for ctx in (gpu_ctx, strip_ctx):
            got, got_stats = run_gpu(ctx, make(k))
            assert got_stats == ref_stats
            assert_targets_match(make(k), ref, got)


@pytest.mark.parametrize("w,h,n,area", [(300, 200, 9000, 4000.0), (300, 200, 32768, 1500.0), (33, 700, 9001, 5000.0),
                                        (1100, 60, 8192, 9000.0), (130, 97, 20000, 6000.0)])
@pytest.mark.parametrize("desc", [dict(), dict(depth_test=abi.TEST_GREATER), dict(depth_test=abi.TEST_NONE, depth_write=0),
                                  dict(depth_test=abi.TEST_LESS, depth_write=0), dict(aa_level=1, band_rows=11)])
def test_overdrawn_small_scenes(gpu_ctx, w, h, n, area, desc):
    """Small scenes with enough fragments for the strips: several strips and
    ranges of primitives (the last one short), units packed in one and in
    several goes, both kinds of keys, bands; and one with a bad index, which
    draws nothing."""
    def make(bad=False):
        rng = np.random.default_rng(n)
        clip = scenes.soup_triangles(rng, n, w, h, 0.9 * area, area, extent=0.8)
        clip[:, 2] = rng.uniform(-0.1, 1.1, n * 3)
        idx = rng.permutation(n * 3).astype(np.uint32)
        if bad:
            idx[-1] = n * 3
        return scenes.clip_triangles_frame(clip, rng.integers(0, 256, (n * 3, 4), dtype=np.uint8), w, h, indices=idx,
                                           depth_clear=0.5 if desc else 1.0, **desc)
    ref, ref_stats = run_oracle(make(), threads=8)
    for _ in range(3):  # plain, recorded, replayed
        got, got_stats = run_gpu(gpu_ctx, make())
        assert got_stats == ref_stats
        assert_targets_match(make(), ref, got)
    if not desc:
        got, got_stats = run_gpu(gpu_ctx, make(bad=True))
        assert got_stats[0][0] == abi.ERR_INDEX_OOB and got_stats[0][1] == 0
        clean = make().alloc_host_targets()
        assert all(np.array_equal(got[k], clean[k]) for k in clean)


@pytest.mark.parametrize("n", [32, 33, 1024, 1025, 1500])
def test_batches_of_many_tiny_scenes(n):
    """Scene lookups by the whole warp, up to their third level (more than 1024
    scenes): every scene's image is the oracle's."""
    from euc_gb300 import capi, frames
    made = [scenes.soup_frame(seed=k, width=7 + k % 5, height=6 + k % 3, ntris=1 + k % 4, area_hi=40.0) for k in range(n)]
    batch = frames.DeviceBatch(made)
    ctx = capi.Context(0)
    try:
        frames.render_batch(ctx, batch)
        assert ctx.sync(frames._stream_ptr(None)) == abi.OK
        candidates, total = ctx.stats(frames._stream_ptr(None)).candidates, 0
        for f, df in zip(made, batch.frames):
            ref, ref_stats = run_oracle(f)
            total += ref_stats[0][1]
            assert_targets_match(f, ref, df.to_host())
        assert candidates == total
    finally:
        ctx.close()
