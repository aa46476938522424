"""Rays in the plane of large triangles.  The intersection's determinant is then mostly rounding, and the
distance it gives can lie far before the triangle's box: such a hit is found by a search that goes on to
that box and by no other, so a search may not end at a distance that only its answer is compared with."""
import numpy as np
import pytest

from sharpray_gb300 import Renderer, _abi, synth

pytestmark = pytest.mark.gpu


def strip(length, quads, frame, offset):
    """A strip of quads in the plane of the first two axes of `frame`."""
    x = np.linspace(0.0, length, quads + 1)
    w = length / quads
    corners = []
    for a, b in zip(x[:-1], x[1:]):
        p = [(a, -w), (b, -w), (b, w), (a, w)]
        corners += [[p[0], p[1], p[2]], [p[0], p[2], p[3]]]
    t = np.array(corners)
    pos = t[..., :1] * frame[0] + t[..., 1:] * frame[1] + offset
    return synth.MeshDesc(pos.astype(np.float32), np.zeros(pos.shape[:2] + (2,), np.float32))


def strip_scene(seed, length):
    """A strip in a plane of some orientation, and a point of that plane before it."""
    rng = np.random.default_rng(seed)
    frame, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    offset = rng.uniform(-2.0, 2.0, 3)
    d = synth.config_c1(64, 48, 4)
    d.meshes = [strip(length, 8, frame, offset)]
    d.objects = [synth.ObjectDesc("strip", synth.Transform(), d.objects[0].material, ("mesh", 0))]
    return d, rng, frame, offset


@pytest.mark.parametrize("length,density", [(8.0, 0.2), (80.0, 0.02), (80.0, 0.2)])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_grazing_hits_in_fog(gpu_ctx, length, density, seed):
    """A camera in the plane, its rays so close together that all of them graze: those that scatter in fog
    before the strip's boxes see the hits of a full search, as the one-thread-per-pixel render does."""
    d, _, frame, offset = strip_scene(seed, length)
    cam, to = (tuple(float(v) for v in x * frame[0] + offset) for x in (-20.0, length))
    d.view = synth.View(synth.Transform(cam, synth.look_rotation(cam, to)), 1e-6, 1e-3)
    d.fog = synth.Fog(density, (0.8, 0.75, 0.6), 0.6, 1e-4)
    g = d.instantiate(gpu_ctx)
    g.build()
    want = None
    for mode in (_abi.SR_RENDER_MEGAKERNEL, _abi.SR_RENDER_WAVEFRONT, _abi.SR_RENDER_WAVEFRONT_GRAPH, _abi.SR_RENDER_AUTO):
        g.set_render_mode(mode)
        r = Renderer(g, d.view, *d.render_args())
        got = {k: getattr(r, k) for k in ("radiance", "radiance_fog", "normals", "uv", "depth", "samples", "variance")}
        want = want or got
        assert 0 < np.isfinite(want["depth"]).sum()
        for k in want:
            assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k


def wall(at, frame, offset):
    """A quad across the strip's way, and a sliver before the strip that makes its box start first."""
    c = [(-2.0, -2.0), (2.0, -2.0), (2.0, 2.0), (-2.0, 2.0)]
    q = np.array([at * frame[0] + y * frame[1] + z * frame[2] for y, z in c])
    s = np.array([-15.0 * frame[0] + y * frame[1] + z * frame[2] for y, z in ((3.0, 0.5), (3.1, 0.5), (3.0, 0.6))])
    pos = np.stack([q[[0, 1, 2]], q[[0, 2, 3]], s]) + offset
    return synth.MeshDesc(pos.astype(np.float32), np.zeros((3, 3, 2), np.float32))


@pytest.mark.parametrize("length", [8.0, 80.0, 800.0])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_grazing_hits_behind_a_wall(gpu_ctx, oracle_mod, length, seed):
    """Rays that already have a hit, on a wall, find the strip's hits before it as the oracle does."""
    d, rng, frame, offset = strip_scene(seed, length)
    d.meshes.append(wall(0.3 * length, frame, offset))
    d.objects.append(synth.ObjectDesc("wall", synth.Transform(), d.objects[0].material, ("mesh", 1)))
    n = 20000
    o = -20.0 * frame[0] + rng.uniform(-0.5, 0.5, (n, 1)) * frame[1] + offset
    way = length * frame[0] + rng.uniform(-1.0, 1.0, (n, 1)) * frame[1] + offset - o
    rays = np.concatenate([o, way / np.linalg.norm(way, axis=1, keepdims=True)], axis=1).astype(np.float32)
    g = d.instantiate(gpu_ctx)
    g.build()
    want = oracle_mod.instantiate(d).trace(rays)
    assert (want["object"] == 0).sum() > 1000 < (want["object"] == 1).sum()
    for mode in (_abi.SR_RENDER_AUTO, _abi.SR_RENDER_MEGAKERNEL):
        g.set_render_mode(mode)
        got = g.trace(rays)
        for k in ("object", "triangle"):
            assert np.array_equal(got[k], want[k]), k
        for k in ("dist", "uv"):
            assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
