"""The persistent kernel's takeover of a staged engine's last paths, and its
share of the dispatches: the same bits whichever kernels render, around the
sizes where the route changes (2^18 and 2^19 samples), from pools that recycle,
with suspended marches, on another stream right after, and in batches."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt(built):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: -m gpu tests need a GPU")
    from pathtracer_gb300 import Batch, Context, Scene, cie_analytic, native

    return {"Batch": Batch, "Context": Context, "Scene": Scene, "cie": cie_analytic(), "native": native}


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


def _mega(rt, scene, push, W, H):
    with rt["Context"](0) as ctx:
        ctx.set_engine(rt["native"].PT_ENGINE_MEGAKERNEL)
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        ctx.dispatch(push)
        ctx.wait()
        return ctx.read_accum()


@pytest.mark.parametrize("name", ["feature_mix", "menger_terrain", "mandelbulb_plane", "cornell_box_full"])
@pytest.mark.parametrize("W,H,spf", [(1, 1, 1), (33, 7, 1), (256, 128, 8), (257, 128, 8), (512, 256, 4), (512, 257, 4)])
def test_dispatch_routes_equal_the_megakernel(rt, name, W, H, spf):
    scene = rt["Scene"].load(os.path.join(SCENES, name + ".json"))
    push = scene.push_constants(W, H, spf, spf, spf, 7)
    want = _mega(rt, scene, push, W, H)
    with rt["Context"](0) as ctx:
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        ctx.dispatch(push)
        ctx.wait()
        assert _same(ctx.read_accum(), want)
        ctx.set_march_budget(64)  # a staged knob: the staged engine renders all of it
        ctx.dispatch(push)
        ctx.wait()
        assert _same(ctx.read_accum(), want)


def test_dispatch_after_a_stream_change(rt):
    """Dispatches return with work queued: the next one, on another stream and
    of another scene, follows it."""
    import torch

    a = rt["Scene"].load(os.path.join(SCENES, "cornell_box.json"))
    b = rt["Scene"].load(os.path.join(SCENES, "feature_mix.json"))
    W, H, spf = 320, 200, 12
    pa, pb = a.push_constants(W, H, spf, spf, spf, 8), b.push_constants(W, H, spf, spf, spf, 6)
    want = _mega(rt, b, pb, W, H)
    streams = [torch.cuda.Stream() for _ in range(2)]
    with rt["Context"](0) as ctx:
        ctx.bind(a, rt["cie"])
        ctx.resize_accum(W, H)
        for k in range(4):
            ctx.set_stream(streams[k % 2].cuda_stream)
            ctx.bind(a, rt["cie"])
            ctx.dispatch(pa)
            ctx.set_stream(streams[(k + 1) % 2].cuda_stream)
            ctx.bind(b, rt["cie"])
            ctx.dispatch(pb)
            got = ctx.read_accum()
            assert _same(got, want)
        ctx.set_stream(None)


@pytest.mark.parametrize("name,W,H,spf,depth", [("mandelbulb_plane", 200, 150, 9, 6), ("menger_terrain", 160, 90, 12, 12),
                                                ("feature_mix", 211, 97, 10, 6)])
def test_batch_finish_equals_the_megakernel(rt, name, W, H, spf, depth):
    """pt_batch_run ends staged passes with the takeover: a pool that recycles,
    two targets, two passes each, FP64 sums beside."""
    scene = rt["Scene"].load(os.path.join(SCENES, name + ".json"))
    pushes = [scene.push_constants(W, H, k * spf, k * spf, spf, depth) for k in (1, 2)]
    with rt["Context"](0) as ctx:
        ctx.set_engine(rt["native"].PT_ENGINE_MEGAKERNEL)
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        for p in pushes:
            ctx.dispatch(p)
        ctx.wait()
        want = ctx.read_accum()
    with rt["Batch"](0, pool_slots=1 << 15, max_passes=16) as b:
        sid = b.add_scene(scene.pack_ubo(rt["cie"]), scene.sdf_plugins())
        b.set_scene_ext(sid, scene.ext_or_none())
        tids = [b.add_target(W, H) for _ in range(2)]
        for _ in range(2):  # a second round reuses the emptied pool
            for p in pushes:
                for t in tids:
                    b.add_pass(sid, t, p)
            b.run()
            for t in tids:
                assert _same(b.read_target(t), want)
