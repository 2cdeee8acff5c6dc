"""The queue tracer's brick -> voxel walk (csrc/dda_walk.cuh).  Ray
batches run it directly and are held to the CPU oracle; frames are held to the
per-thread nested loops (the path-trace megakernel, itself held to the CPU
oracle by the parity tests): the same frame through both, at the grid sizes
where the walk's packed words change shape -- one brick, grids whose side is no
power of two, and a grid of more than 128^3 bricks, which takes the tracer's
wide form -- and from cameras that start outside the world, on voxel edges and
that look along an axis.  Images and counters must be equal bit for bit.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(vrt):
    c = vrt.Context(0)
    yield c
    c.close()


def _world(vrt, ctx, n):
    """Boxes of voxels over an empty grid (built by edits, so that the largest grid needs no host world)."""
    sc = vrt.Scene(ctx, np.zeros(n ** 3, np.uint32), n)
    rng = np.random.default_rng(n)
    sc.edit_box(0, 0, 0, n - 1, max(n // 16 - 1, 0), n - 1, 0x0080A0C0)          # floor
    for _ in range(40):
        lo = rng.integers(0, n, 3)
        hi = np.minimum(lo + rng.integers(0, max(n // 8, 2), 3), n - 1)
        sc.edit_box(*map(int, lo), *map(int, hi), int(rng.integers(1, 1 << 32)))
    return sc


@pytest.mark.parametrize("n", [8, 24, 104, 1024, 1032])
def test_walk_matches_nested_loops(vrt, ctx, n):
    W, H = 96, 61
    sc = _world(vrt, ctx, n)
    ext = n / 16.0
    poses = [vrt.CameraPose((ext * 0.5, ext * 0.6, ext * 0.4), 0.3, -0.2),       # inside
             vrt.CameraPose((-0.7 * ext, ext * 1.5, -0.4 * ext), 0.8, -0.5),     # outside, looking in
             vrt.CameraPose((ext * 0.5, ext * 0.5, ext * 0.25), 0.0, 0.0),       # on a voxel edge, along +z
             vrt.CameraPose((ext * 0.5, ext, ext * 0.5), 0.0, -math.pi / 2)]     # on the top face, straight down
    wave = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True)
    mega = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True, path_kernel="megakernel")
    for k, pose in enumerate(poses):
        u = vrt.make_uniforms(pose, None, vrt.Lighting(), 11 + k, 3, 0, W, H)
        for s in (wave, mega):
            s.set_timing(True)
            s.frame(u)
        a, b = wave.stats(), mega.stats()
        assert (a.rays, a.dda_outer, a.dda_inner, a.voxel_reads) == (b.rays, b.dda_outer, b.dda_inner, b.voxel_reads)
        assert np.array_equal(wave.radiance_f32().view(np.uint32), mega.radiance_f32().view(np.uint32))
        assert np.array_equal(wave.gbuffer().view(np.uint32), mega.gbuffer().view(np.uint32))
    for o in (wave, mega, sc):
        o.close()


# The primary rays start in 8 x 4 tiles: sizes below, at and past a tile's side, alone and as the views of a batch.
@pytest.mark.parametrize("W,H", [(1, 1), (7, 3), (8, 4), (9, 5), (33, 2), (3, 33), (131, 67)])
def test_primary_order_covers_the_image(vrt, ctx, W, H):
    vox, spawn = vrt.generate_scene(vrt.VRT_SCENE_FULL, 64, 3)
    sc = vrt.Scene(ctx, vox, 64)
    mega = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True, path_kernel="megakernel")
    wave = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True)
    views = [vrt.Session(ctx, sc, W + k, H, keep_radiance_f32=True, path_kernel="batch_only") for k in (0, 1, 0)]
    batch = vrt.Batch(ctx, views)
    u = [vrt.make_uniforms(vrt.camera_spline(spawn, 2), None, vrt.Lighting(), 5, 2, 0, W + k, H) for k in (0, 1, 0)]
    mega.frame(u[0])
    wave.frame(u[0])
    batch.frame(u)
    want = (mega.radiance_f32().tobytes(), mega.gbuffer().tobytes())
    for s in (wave, views[0], views[2]):
        assert (s.radiance_f32().tobytes(), s.gbuffer().tobytes()) == want
    batch.close()
    for o in (mega, wave, *views, sc):
        o.close()


def _odd_rays(n, ext, seed):
    """Random rays, and the forms a walk can trip over: zero, tiny, huge, infinite and NaN components,
    origins on voxel and brick edges, far away or not finite, bounds of every size."""
    r = np.random.default_rng(seed)
    o = (r.random((n, 3)) * ext).astype(np.float32)
    d = r.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    t = np.where(r.random(n) < 0.6, 1e4, r.random(n) * ext).astype(np.float32)
    form, ax = r.integers(0, 16, n), r.integers(0, 3, n)
    rows = np.arange(n)

    def put(a, k, v):
        m = form == k
        a[rows[m], ax[m]] = v
    put(d, 0, 0.0)
    put(d, 1, -0.0)
    put(d, 2, 1e-9)
    put(d, 3, 1e30)
    put(d, 4, np.inf)
    put(d, 5, np.nan)
    put(o, 6, np.nan)
    put(o, 7, np.inf)
    o[form == 8] = np.floor(o[form == 8] * 16) / 16
    o[form == 9] = np.floor(o[form == 9] * 2) / 2
    d[form == 10] = np.sign(d[form == 10]) / np.float32(math.sqrt(3))
    o[form == 11] = o[form == 11] * 3 - ext
    o[form == 12] += np.float32(3e5)
    d[form == 13] = np.eye(3, dtype=np.float32)[ax[form == 13]]
    t[form == 14] = np.float32(np.nan)
    t[form == 15] = np.float32(-1.0)
    return o, d, t


@pytest.mark.parametrize("grid", [8, 104, 256])
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 13_999, 14_001, 140_001, 600_001, 1_100_003])
def test_ray_batch_matches_oracle(vrt, orc, ctx, grid, n):
    vox, _ = vrt.generate_scene(vrt.VRT_SCENE_RANDOM, grid, 3)
    b, m = orc.build_bricks(vox, grid)
    sc = vrt.Scene(ctx, vox, grid)
    o, d, t = _odd_rays(n, grid / 16.0, grid + n)
    got, want = sc.trace_rays(o, d, t), orc.trace(vox, b, m, grid, o, d, t)
    for f in ("t", "n"):            # as bits, any NaN equal to any other
        x, y = got[f], want[f]
        assert np.array_equal(np.isnan(x), np.isnan(y))
        assert np.array_equal(x.view(np.uint32)[~np.isnan(x)], y.view(np.uint32)[~np.isnan(y)])
    for f in ("mat", "voxel", "face", "steps", "bytes"):
        assert np.array_equal(got[f], want[f]), f
    sc.close()


# pixel counts on both sides of the lines at which the remaining paths of a
# frame move to one thread each, by default and at every wave, and below the
# line at which a path has two lanes there
@pytest.mark.parametrize("W,H,bounces", [(1, 1, 2), (64, 41, 3), (223, 213, 4), (401, 297, 2), (401, 303, 3), (611, 331, 2), (611, 331, 3), (811, 501, 4),
                                         (1201, 801, 5)])
def test_tail_waves_leave_the_image(vrt, ctx, W, H, bounces):
    vox, spawn = vrt.generate_scene(vrt.VRT_SCENE_VOXELRT, 128, 7)
    sc = vrt.Scene(ctx, vox, 128)
    u = vrt.make_uniforms(vrt.camera_spline(spawn, 3), None, vrt.Lighting(), 9, bounces, 0, W, H)
    want = None
    for tail in (0, -1, 1, bounces + 1):
        s = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True)
        s.set_tuning(tail_wave=tail)
        s.set_timing(True)
        s.frame(u)
        st = s.stats()
        got = (s.radiance_f32().tobytes(), s.ldr().tobytes(), st.rays, st.dda_outer, st.dda_inner, st.voxel_reads)
        want = want or got
        assert got == want, f"tail wave {tail}"
        s.close()
    sc.close()


# The kernels of a frame overlap the launch of the next one; a session with
# timing on has an event between its passes, which orders them fully.
@pytest.mark.parametrize("preset", ["base", "ours"])
@pytest.mark.parametrize("W,H", [(33, 17), (401, 297), (1283, 721)])
def test_overlapped_frames_match_ordered_frames(vrt, ctx, W, H, preset):
    vox, spawn = vrt.generate_scene(vrt.VRT_SCENE_FULL, 64, 7)
    sc = vrt.Scene(ctx, vox, 64)
    lights = int(sc.build_lights().count) if preset != "base" else 0
    us = [vrt.make_uniforms(vrt.camera_spline(spawn, f), vrt.camera_spline(spawn, max(f - 1, 0)), vrt.Lighting(), f,
                            2, 3, W, H, preset=preset, light_count=lights) for f in range(12)]
    got = []
    for ordered in (True, False):
        s = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True)
        s.set_timing(ordered)
        for u in us:
            s.frame(u)
            if ordered:
                ctx.synchronize()
        got.append((s.radiance_f32().tobytes(), s.ldr().tobytes()))
        s.close()
    assert got[0] == got[1]
    sc.close()


def test_stored_albedo_is_the_material_byte():
    """rgba8unorm of sqrt(albedo) gives back each colour byte, in binary32 as the shader forms it."""
    s = np.float32(1.0) / np.float32(255.0)
    a = np.arange(256, dtype=np.float32) * s
    q = np.clip(np.sqrt(a * a), np.float32(0.0), np.float32(1.0))
    np.testing.assert_array_equal(np.floor(q * np.float32(255.0) + np.float32(0.5)).astype(np.int64), np.arange(256))


# Directions whose components lie below the bound of the reciprocals (1e-8), two or three at a time, from up to a
# world outside and without a bound on t: the point on the ray then lags far behind the walk's cell.
@pytest.mark.parametrize("grid", [16, 64])
def test_short_directions_match_oracle(vrt, orc, ctx, grid):
    n, ext = 1_500_000, grid / 16.0
    r = np.random.default_rng(grid)
    vox, _ = vrt.generate_scene(vrt.VRT_SCENE_RANDOM, grid, 3)
    b, m = orc.build_bricks(vox, grid)
    sc = vrt.Scene(ctx, vox, grid)
    o = (r.random((n, 3)) * 3 * ext - ext).astype(np.float32)
    d = (np.exp(r.uniform(np.log(1e-10), np.log(1e-8), (n, 3))) * r.choice([-1.0, 1.0], (n, 3))).astype(np.float32)
    long = np.flatnonzero(r.random(n) < 0.3)
    d[long, r.integers(0, 3, len(long))] = np.exp(r.uniform(np.log(1e-8), np.log(1e-6), len(long))).astype(np.float32)
    t = np.full(n, 1e30, np.float32)
    got, want = sc.trace_rays(o, d, t), orc.trace(vox, b, m, grid, o, d, t)
    for f in ("t", "n"):
        assert np.array_equal(got[f].view(np.uint32), want[f].view(np.uint32)), f
    for f in ("mat", "voxel", "face", "steps", "bytes"):
        assert np.array_equal(got[f], want[f]), f
    sc.close()


def test_host_entry_survives_device_pointers(vrt, ctx):
    """vrt_trace_rays takes host arrays; device pointers get the runtime's answer at every batch size, and host arrays
    are answered as before afterwards."""
    import ctypes as C

    import torch
    vox, _ = vrt.generate_scene(vrt.VRT_SCENE_RANDOM, 64, 3)
    sc = vrt.Scene(ctx, vox, 64)
    o, d, t = _odd_rays(64, 4.0, 5)
    want = sc.trace_rays(o, d, t).tobytes()
    dev = torch.zeros(20_000 * 12, dtype=torch.float32, device="cuda")
    host = np.zeros(20_000 * 12, np.float32)
    torch.cuda.synchronize()
    p, q = C.c_void_p(dev.data_ptr()), C.c_void_p(host.ctypes.data)
    for args in ((p, q, q, q), (q, p, q, q), (q, q, p, q), (q, q, q, p)):
        few, many = (vrt.lib.vrt_trace_rays(sc.h, *args[:3], n, args[3]) for n in (64, 20_000))
        assert few == many
    assert sc.trace_rays(o, d, t).tobytes() == want
    sc.close()


def test_ray_batches_of_several_threads(vrt, ctx):
    """Threads that query one world at once, with batches of the sizes that go through the context's pinned memory:
    each gets its own rays' hits."""
    import threading
    vox, _ = vrt.generate_scene(vrt.VRT_SCENE_RANDOM, 64, 3)
    sc = vrt.Scene(ctx, vox, 64)
    rays = [_odd_rays(n, 4.0, n) for n in (1, 64, 700, 5000, 16_384, 16_385)]
    want = [sc.trace_rays(*r).tobytes() for r in rays]
    wrong = []

    def work(k):
        for _ in range(60):
            if sc.trace_rays(*rays[k]).tobytes() != want[k]:
                wrong.append(k)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(rays))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    sc.close()


def test_trace_blocks_count_256_threads(vrt, ctx):
    """A tuning's tracer blocks are counted as blocks of 256 threads: one per SM already holds a warp for each of
    8 rays per SM, so that twice as many change nothing (a warp that holds two rays walks fewer lane slots)."""
    import torch
    W, H = 8, torch.cuda.get_device_properties(0).multi_processor_count
    vox, spawn = vrt.generate_scene(vrt.VRT_SCENE_FULL, 64, 3)
    sc = vrt.Scene(ctx, vox, 64)
    u = vrt.make_uniforms(vrt.camera_spline(spawn, 2), None, vrt.Lighting(), 5, 0, 0, W, H)
    slots = []
    for blocks in (1, 2):
        s = vrt.Session(ctx, sc, W, H)
        s.set_tuning(trace_blocks_per_sm=blocks, tail_wave=0)
        s.frame(u)
        slots.append(s.stats().trace_step_slots)
        s.close()
    assert slots[0] == slots[1] > 0
    sc.close()


# Lane step slots are counted wherever a path's rays are walked: no more iterations than slots, at every tail wave.
@pytest.mark.parametrize("W,H,bounces", [(64, 41, 3), (401, 297, 2), (611, 331, 3)])
def test_step_slots_cover_the_tail(vrt, ctx, W, H, bounces):
    vox, spawn = vrt.generate_scene(vrt.VRT_SCENE_VOXELRT, 128, 7)
    sc = vrt.Scene(ctx, vox, 128)
    u = vrt.make_uniforms(vrt.camera_spline(spawn, 3), None, vrt.Lighting(), 9, bounces, 0, W, H)
    for tail in (0, -1, 1, 2):
        s = vrt.Session(ctx, sc, W, H)
        s.set_tuning(tail_wave=tail)
        s.frame(u)
        st = s.stats()
        steps = st.dda_outer + st.dda_inner
        assert steps <= st.trace_step_slots <= 32 * 5 * steps, f"tail wave {tail}"
        s.close()
    sc.close()


# Batches on both sides of the lines between the walk and the nested loops, which depend on the world's size.
@pytest.mark.parametrize("grid,n", [(32, 6_999), (32, 7_001), (32, 1_600_000), (32, 1_600_001), (64, 1_000_000), (64, 1_000_001),
                                    (80, 320_000), (80, 320_001), (128, 0), (128, 1)])
def test_ray_batch_lines_match_oracle(vrt, orc, ctx, grid, n):
    import torch
    if n < 2:     # at one wave of blocks, and past it
        n += 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    vox, _ = vrt.generate_scene(vrt.VRT_SCENE_RANDOM, grid, 3)
    b, m = orc.build_bricks(vox, grid)
    sc = vrt.Scene(ctx, vox, grid)
    o, d, t = _odd_rays(n, grid / 16.0, grid + n)
    got, want = sc.trace_rays(o, d, t), orc.trace(vox, b, m, grid, o, d, t)
    for f in ("t", "n"):            # as bits, any NaN equal to any other
        x, y = got[f], want[f]
        assert np.array_equal(np.isnan(x), np.isnan(y))
        assert np.array_equal(x.view(np.uint32)[~np.isnan(x)], y.view(np.uint32)[~np.isnan(y)])
    for f in ("mat", "voxel", "face", "steps", "bytes"):
        assert np.array_equal(got[f], want[f]), f
    sc.close()


@pytest.mark.parametrize("variant", range(9))
def test_tracer_variants_leave_the_image(vrt, ctx, variant):
    """Every shape of the tracer that a tuning can name, for a session and for a batch, against the megakernel."""
    W, H = 160, 90
    vox, spawn = vrt.generate_scene(vrt.VRT_SCENE_FULL, 128, 2)
    sc = vrt.Scene(ctx, vox, 128)
    u = vrt.make_uniforms(vrt.camera_spline(spawn, 4), None, vrt.Lighting(), 9, 4, 0, W, H)
    mega = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True, path_kernel="megakernel")
    wave = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True)
    view = vrt.Session(ctx, sc, W, H, keep_radiance_f32=True, path_kernel="batch_only")
    batch = vrt.Batch(ctx, [view])
    for t in (wave, batch):
        t.set_tuning(trace_variant=variant, tail_wave=0)
    mega.frame(u)
    wave.frame(u)
    batch.frame([u])
    a = mega.stats()
    for s, st in ((wave, wave.stats()), (view, batch.stats())):
        assert s.radiance_f32().tobytes() == mega.radiance_f32().tobytes()
        assert (st.rays, st.dda_outer, st.dda_inner, st.voxel_reads) == (a.rays, a.dda_outer, a.dda_inner, a.voxel_reads)
    batch.close()
    for o in (mega, wave, view, sc):
        o.close()


@pytest.mark.parametrize("n", [8, 24, 104])
def test_edits_keep_the_bitmap(vrt, ctx, n):
    """A world after boxes of voxels were set and cleared, bricks at its edges among them, answers rays as a world
    uploaded with those voxels does, and as one uploaded with its bricks and masks."""
    r = np.random.default_rng(n)
    sc = vrt.Scene(ctx, np.zeros(n ** 3, np.uint32), n)
    o, d, t = _odd_rays(4000, n / 16.0, n)
    for k in range(24):
        lo = r.integers(0, n, 3)
        hi = np.minimum(lo + r.integers(0, 20, 3), n - 1)
        if k % 6 == 5:                       # whole bricks, the world's first or last
            lo = np.zeros(3, int) if k % 12 == 5 else np.full(3, n - 8)
            hi = lo + 7
        sc.edit_box(*map(int, lo), *map(int, hi), 0 if k % 3 == 2 else int(r.integers(1, 1 << 32)))
        if k % 4 == 3:
            v, b, m = sc.read()
            want = sc.trace_rays(o, d, t).tobytes()
            for other in (vrt.Scene(ctx, v, n), vrt.Scene(ctx, v, n, b, m)):
                assert other.trace_rays(o, d, t).tobytes() == want
                other.close()
    sc.close()
