"""Launches that do not fill the GPU take their own forms; they give what the full ones give."""
import numpy as np
import pytest

from sharpray_gb300 import Renderer, _abi, synth
from tests.golden.make_golden import seeded_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["c1", "features"])
def traced(request, gpu_ctx, oracle_mod):
    d = synth.config_c1(32, 24, 1) if request.param == "c1" else synth.config_features(32, 24, 1)
    rays = seeded_rays(103000, seed=31)
    g = d.instantiate(gpu_ctx)
    g.build()
    return g, rays, oracle_mod.instantiate(d).trace(rays)


# one query, around a warp, around one per warp of a full launch, the last size that is dealt out over
# the warps (24 per warp of 152 x 7 blocks of 4) and the first that is not
@pytest.mark.parametrize("n", [1, 2, 31, 33, 4255, 4257, 102143, 102144, 102145, 103000])
def test_few_ray_queries_bit_exact(traced, n):
    g, rays, want = traced
    got = g.trace(rays[:n])
    for k in ("object", "triangle"):
        assert np.array_equal(got[k], want[k][:n]), k
    for k in ("dist", "uv"):
        assert np.array_equal(got[k].view(np.uint32), want[k][:n].view(np.uint32)), k


# around the origin and where a float's steps are as large as the gaps between the surfaces; objects of
# a like size and from a hundredth to a hundred times as large
@pytest.mark.parametrize("far", [0.0, 1e2, 1e4])
@pytest.mark.parametrize("spread", [1.0, 1e2])
def test_nested_objects_bit_exact(gpu_ctx, oracle_mod, far, spread):
    """A ray that has a hit looks for nearer ones only: in meshes one inside the other, copies that
    coincide or nearly do, and larger ones around them, the hits stay the ones of a full search."""
    rng = np.random.default_rng(int(far) + int(spread))
    d = synth.config_c1(8, 8, 1)
    mat = d.objects[0].material
    d.objects = []
    for i in range(24):
        size = np.exp(rng.uniform(-1.0, 1.0) * np.log(spread)) * rng.uniform(0.9, 1.1, 3)
        gap = (0.0, 1e-6, 1e-3, 0.3)[i % 4]
        at = (far + gap * rng.normal(), -far + gap * rng.normal(), gap * rng.normal())
        for copy in range(1 + (i % 3 == 0)):
            d.objects.append(synth.ObjectDesc(f"o{i}_{copy}", synth.Transform(at, scale=tuple(float(v) for v in size)), mat,
                                              ("mesh", 0)))
    to = np.array([far, -far, 0.0]) + rng.normal(size=(4000, 3))
    pos = to + 3.0 * rng.normal(size=to.shape) * np.exp(rng.uniform(-1.0, 1.0, (len(to), 1)) * np.log(spread))
    way = to - pos
    rays = np.concatenate([pos, way / np.linalg.norm(way, axis=1, keepdims=True)], axis=1).astype(np.float32)
    g = d.instantiate(gpu_ctx)
    g.build()
    want = oracle_mod.instantiate(d).trace(rays)
    assert 0 <= want["object"].max() and len(np.unique(want["object"])) > 4
    for mode in (_abi.SR_RENDER_AUTO, _abi.SR_RENDER_MEGAKERNEL):
        g.set_render_mode(mode)
        got = g.trace(rays)
        for k in ("object", "triangle"):
            assert np.array_equal(got[k], want[k]), k
        for k in ("dist", "uv"):
            assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k


def panes(count, width, height):
    """The feature scene with `count` panes of glass above it, which the shadow rays cross one by one."""
    d = synth.config_features(width, height, 3)
    for i in range(count):
        y = 1.9 + 0.1 * i
        d.objects.append(synth.ObjectDesc(f"pane{i}", synth.Transform(),
                                          {"albedo": (0.9, 0.8, 0.95), "roughness": 0.1, "transparency": 0.7, "ior": 1.2},
                                          ("box", (-6.0, y, -6.0), (6.0, y + 0.02, 6.0))))
    return d


def planes(scene, d):
    r = Renderer(scene, d.view, *d.render_args())
    return {k: getattr(r, k) for k in ("radiance", "radiance_fog", "normals", "uv", "depth", "samples", "variance")}


def same(a, b):
    for k in a:
        assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k


# no pane (the feature scene's own glass), one, and more than the attenuation lets through; a single
# warp's pixels, a ragged image
@pytest.mark.parametrize("count,width,height", [(0, 8, 4), (1, 17, 9), (12, 33, 21)])
def test_shadow_rays_through_glass(gpu_ctx, count, width, height):
    """Shadow rays traced hit by hit in the traversal loop give the one-thread-per-pixel image."""
    d = panes(count, width, height)
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_render_mode(_abi.SR_RENDER_MEGAKERNEL)
    want = planes(g, d)
    for mode in (_abi.SR_RENDER_WAVEFRONT, _abi.SR_RENDER_WAVEFRONT_GRAPH, _abi.SR_RENDER_AUTO):
        g.set_render_mode(mode)
        for threads in (128, 64, 256):
            g.set_tuning(trace_block_threads=threads)
            same(planes(g, d), want)


# thin and thick fog (scatters behind every surface, between and in front of them), around the origin and
# where a float's steps are coarse
@pytest.mark.parametrize("density", [1e-3, 0.2, 20.0])
@pytest.mark.parametrize("far", [0.0, 3e3])
def test_hits_behind_scatters(gpu_ctx, density, far):
    """Rays that look for hits up to their scatter in fog only give the full search's image."""
    d = synth.config_c2(41, 29, 5, rings=40, rock_rings=12, env=(64, 32))
    move = lambda t: synth.Transform(tuple(p + far for p in t.pos), t.rot, t.scale)
    for o in d.objects:
        o.transform = move(o.transform)
    d.view = synth.View(move(d.view.trans), d.view.fov, d.view.near)
    d.fog = synth.Fog(density, (0.8, 0.75, 0.6), 0.6, 1e-4)
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_render_mode(_abi.SR_RENDER_MEGAKERNEL)
    want = planes(g, d)
    for mode in (_abi.SR_RENDER_WAVEFRONT, _abi.SR_RENDER_WAVEFRONT_GRAPH, _abi.SR_RENDER_AUTO):
        g.set_render_mode(mode)
        same(planes(g, d), want)


def features(w, h):
    return synth.config_features(w, h)


def mesh(w, h):
    return synth.config_c1(w, h)


def fog(w, h):
    return synth.config_c2(w, h, rings=40, rock_rings=12, env=(64, 32))


# one pixel, one 8x4 tile, ragged tiles, fewer tiles than SMs and more; no bounce, one sample, the
# adaptive stop; fewer slots than pixels; another random-number stream; the largest images that the path
# kernel takes on 152 SMs (2,048 pixels each, half of it for the general kernels) and the next larger
@pytest.mark.parametrize("make,w,h,spp,min_spp,bounces,slots,seed", [
    (mesh, 1, 1, 1, 1, 0, 0, 0), (mesh, 8, 4, 5, 5, 4, 0, 0), (fog, 9, 5, 3, 3, 8, 0, 3),
    (features, 31, 33, 6, 2, 6, 0, 0), (features, 97, 61, 4, 1, 5, 0, 9), (fog, 193, 107, 3, 1, 8, 0, 0),
    (fog, 160, 96, 2, 2, 6, 1000, 5), (features, 40, 40, 3, 3, 3, 32, 0), (mesh, 300, 200, 2, 2, 0, 0, 0),
    (fog, 608, 512, 1, 1, 8, 0, 0), (fog, 616, 512, 1, 1, 8, 0, 0),
    (features, 304, 512, 2, 1, 4, 0, 0), (features, 312, 512, 2, 1, 4, 0, 0)])
def test_path_kernel_matches_bounce_loop(gpu_ctx, make, w, h, spp, min_spp, bounces, slots, seed):
    d = make(w, h)
    d.spp, d.min_samples, d.bounces, d.variance_threshold = spp, min_spp, bounces, 0.1
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_seed(seed)
    g.set_tuning(max_slots=slots)
    g.set_render_mode(_abi.SR_RENDER_WAVEFRONT_GRAPH)
    want = planes(g, d)
    g.set_render_mode(_abi.SR_RENDER_AUTO)
    for _ in range(2):
        same(planes(g, d), want)


# shares of one SM that hold every pixel, and that do not (the first scene's pixels are then claimed as
# slots come free); a scene of its own render mode, which takes the whole batch to the graph
@pytest.mark.parametrize("sizes,spps,mode", [([(40, 24), (33, 21)], [3, 2], 0), ([(160, 96), (256, 192)], [1, 24], 0),
                                             ([(64, 48), (24, 8), (17, 5)], [2, 1, 4], 3)])
def test_small_batches_match_single_renders(gpu_ctx, sizes, spps, mode):
    torch = pytest.importorskip("torch")
    from sharpray_gb300 import render_batch, render_params
    from sharpray_gb300.autograd import current_stream_handle, device_aovs
    descs, scenes, want = [], [], []
    for (w, h), spp, make in zip(sizes, spps, (mesh, fog, features)):
        d = make(w, h)
        d.spp = d.min_samples = spp
        g = d.instantiate(gpu_ctx)
        g.build()
        g.set_render_mode(_abi.SR_RENDER_WAVEFRONT_GRAPH)
        want.append(planes(g, d))
        g.set_render_mode(_abi.SR_RENDER_AUTO)
        descs.append(d)
        scenes.append(g)
    scenes[-1].set_render_mode(mode)
    outs = [device_aovs(d.width, d.height) for d in descs]
    for _ in range(2):
        for bufs, _a in outs:
            for t in bufs.values():
                t.zero_()
        render_batch(scenes, [d.view for d in descs], [render_params(*d.render_args()) for d in descs],
                     [a for _b, a in outs], stream=current_stream_handle())
        torch.cuda.synchronize()
        for (bufs, _a), ref in zip(outs, want):
            same({k: v.cpu().numpy() for k, v in bufs.items()}, {k: v.reshape(-1) for k, v in ref.items()})


# what the bounce loop hands over: everything after two bounces (divisor 1, at most what the path kernel
# holds), a half, the last few paths; with shadow rays pending, with slots that claim more pixels
@pytest.mark.parametrize("make,w,h,slots", [(fog, 123, 77, 0), (features, 61, 45, 0), (fog, 96, 80, 1500), (mesh, 9, 3, 0)])
@pytest.mark.parametrize("divisor", [1, 2, 64])
def test_hand_over_to_path_kernel(gpu_ctx, make, w, h, slots, divisor):
    d = make(w, h)
    d.spp, d.min_samples, d.variance_threshold = 5, 2, 0.1
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_render_mode(_abi.SR_RENDER_MEGAKERNEL)
    want = planes(g, d)
    for mode in (_abi.SR_RENDER_WAVEFRONT, _abi.SR_RENDER_WAVEFRONT_GRAPH):
        g.set_render_mode(mode)
        g.set_tuning(tail_divisor=divisor, max_slots=slots)
        same(planes(g, d), want)


# the last size of the 384-thread blocks on 152 SMs (768 slots each) and the first of the 512-thread ones
@pytest.mark.parametrize("make,w,h", [(mesh, 304, 384), (mesh, 312, 384), (fog, 304, 384), (fog, 304, 388),
                                      (features, 304, 384), (features, 304, 388)])
def test_path_kernel_block_sizes(gpu_ctx, make, w, h):
    test_path_kernel_matches_bounce_loop(gpu_ctx, make, w, h, 2, 1, 4, 0, 1)


@pytest.mark.parametrize("w,h,mode,paths", [(96, 64, _abi.SR_RENDER_AUTO, True), (616, 512, _abi.SR_RENDER_AUTO, False),
                                            (96, 64, _abi.SR_RENDER_WAVEFRONT_GRAPH, False)])
def test_autotuner_times_the_form_that_runs(gpu_ctx, w, h, mode, paths):
    from sharpray_gb300 import render_params
    d = mesh(w, h)
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_render_mode(mode)
    chosen = g.autotune(d.view, render_params(*d.render_args()), trial_spp=2)
    info = g.render_info()  # of the last trial
    assert (info["bounce_iterations"] == 0) == paths
    if paths:  # no other dimension is one of the path kernel's
        assert (chosen["trace_block_threads"], chosen["trace_blocks_per_sm"], chosen["fog_shade_blocks_per_sm"],
                chosen["tail_divisor"]) == (128, 0, 0, 8)
    planes(g, d)
    assert (g.render_info()["bounce_iterations"] == 0) == paths


def test_launches_of_counting_renders(gpu_ctx):
    """A graph render that counts work runs every bounce itself: it has one launch less than its bounces and
    loop bodies tell of a render that hands over to the path kernel."""
    d = mesh(96, 64)
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_render_mode(_abi.SR_RENDER_WAVEFRONT_GRAPH)
    planes(g, d)
    plain = g.render_info()
    k, n = plain["bounce_iterations"], plain["kernel_launches"]
    per_bounce, rest = divmod(n - 2 - k // 2, k)  # one launch at the start, one at the end, a condition per two bounces
    assert rest == 0
    g.set_counting(True)
    planes(g, d)
    counted = g.render_info()
    k = counted["bounce_iterations"]
    assert counted["kernel_launches"] == 1 + per_bounce * k + k // 2


# hand-overs of more than 768 paths a block on 152 SMs, which the 512-thread form takes, up to all that its
# blocks hold (2,048 slots; half of it for the general kernels, with glass, and one tile row more)
@pytest.mark.parametrize("make,w,h", [(fog, 616, 512), (mesh, 640, 512), (features, 312, 512), (features, 304, 512)])
@pytest.mark.parametrize("divisor", [1, 2])
def test_large_hand_overs(gpu_ctx, make, w, h, divisor):
    d = make(w, h)
    d.spp, d.min_samples, d.variance_threshold = 3, 1, 0.1
    g = d.instantiate(gpu_ctx)
    g.build()
    g.set_render_mode(_abi.SR_RENDER_MEGAKERNEL)
    want = planes(g, d)
    for mode in (_abi.SR_RENDER_WAVEFRONT, _abi.SR_RENDER_WAVEFRONT_GRAPH):
        g.set_render_mode(mode)
        g.set_tuning(tail_divisor=divisor)
        same(planes(g, d), want)
