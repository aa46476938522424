"""Failure detection without a GPU fault: the loop caps of SrTuning.

A render whose bounce loop, or a trace whose traversal, runs past its cap ends early.  The kernel
sets the device error word (2 = loop cap) and returns; the call returns SR_ERR_DEVICE with a
message naming the loop cap; and the context stays usable, so the next render with the default
caps gives the same image as before.  The caps are lowered here far below what the scene needs,
so that they run out on purpose; nothing traps, faults or waits without a bound.  (The reference
has no such guard: Renderer.Tick waits without a timeout, renderer.cs:98-105.)
"""
import numpy as np
import pytest

from sharpray_gb300 import Renderer, SharpRayError, _abi, synth
from tests.golden.make_golden import seeded_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(gpu_ctx):
    d = synth.config_c1(32, 24, 4)
    g = d.instantiate(gpu_ctx)
    g.build()
    return d, g


def render(d, g):
    return Renderer(g, d.view, *d.render_args())


@pytest.mark.parametrize("mode", [_abi.SR_RENDER_WAVEFRONT_GRAPH, _abi.SR_RENDER_WAVEFRONT])
def test_bounce_loop_cap_reports_and_recovers(scene, mode):
    d, g = scene
    g.set_render_mode(mode)
    try:
        before = render(d, g)
        g.set_tuning(max_bounce_iterations=2)  # 4 spp x 5 segments need ~25 bounces
        with pytest.raises(SharpRayError) as e:
            render(d, g)
        assert e.value.code == _abi.SR_ERR_DEVICE
        assert "loop cap" in str(e.value)
        g.set_tuning()
        after = render(d, g)
    finally:
        g.set_tuning()
        g.set_render_mode(_abi.SR_RENDER_AUTO)
    for plane in ("radiance", "radiance_fog", "samples", "depth"):
        assert np.array_equal(getattr(before, plane).view(np.uint32), getattr(after, plane).view(np.uint32)), plane


def test_traversal_cap_in_trace_and_render(scene, oracle_mod):
    d, g = scene
    rays = seeded_rays(4096, seed=21)
    want = oracle_mod.instantiate(d).trace(rays)
    try:
        g.set_tuning(max_traversal_steps=3)  # fewer actions than any hit needs
        with pytest.raises(SharpRayError) as e:
            g.trace(rays)
        assert e.value.code == _abi.SR_ERR_DEVICE and "loop cap" in str(e.value)
        with pytest.raises(SharpRayError) as e:
            render(d, g)
        assert e.value.code == _abi.SR_ERR_DEVICE
        g.set_tuning()
        got = g.trace(rays)
    finally:
        g.set_tuning()
    assert np.array_equal(got["object"], want["object"]) and np.array_equal(got["triangle"], want["triangle"])


# a cap that stops the loop with more live paths than it hands over, which the path kernel then leaves
# alone: a launch of its 384-thread form (tail_paths up to 768 a block) and one of its 512-thread form, the
# general kernels, an adjoint replay's loop, a batch's graph
@pytest.mark.parametrize("make,w,h,divisor", [(synth.config_c1, 1024, 768, 0), (synth.config_c1, 1024, 768, 1),
                                              (synth.config_c1, 1920, 1080, 32), (synth.config_features, 1024, 768, 0),
                                              (synth.config_c1, 64, 48, 0)])
def test_bounce_loop_cap_of_large_images(gpu_ctx, make, w, h, divisor):
    torch = pytest.importorskip("torch")
    from sharpray_gb300 import render_batch, render_params
    from sharpray_gb300.autograd import current_stream_handle, device_aovs
    d = make(w, h, 4)
    d.min_samples = 4  # no pixel is done after two bounces
    g = d.instantiate(gpu_ctx)
    g.build()
    bufs, aovs = device_aovs(w, h)
    for mode in (_abi.SR_RENDER_WAVEFRONT_GRAPH, _abi.SR_RENDER_AUTO):
        g.set_render_mode(mode)
        g.set_tuning(tail_divisor=divisor)
        before = render(d, g)
        g.set_tuning(tail_divisor=divisor, max_bounce_iterations=2)
        with pytest.raises(SharpRayError) as e:
            render(d, g)
        assert e.value.code == _abi.SR_ERR_DEVICE and "loop cap" in str(e.value)
        render_batch([g], [d.view], [render_params(*d.render_args())], [aovs], current_stream_handle())
        torch.cuda.synchronize()
        with pytest.raises(SharpRayError) as e:  # the batch's error word, read by the next synchronous call
            g.trace(seeded_rays(8, seed=1))
        assert "loop cap" in str(e.value)
        g.set_tuning(tail_divisor=divisor)
        after = render(d, g)
        for plane in ("radiance", "radiance_fog", "samples", "depth"):
            assert np.array_equal(getattr(before, plane).view(np.uint32), getattr(after, plane).view(np.uint32)), plane
