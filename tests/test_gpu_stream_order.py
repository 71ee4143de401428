"""pt_set_stream: what a context has queued on its old stream comes before what
it queues on the new one.  The old stream is held back by a kernel that spins
for a fixed number of cycles, so that work left behind would run last."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu

HOLD = 300_000_000  # cycles: about 0.15 s


@pytest.fixture(scope="module")
def rt(built):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: -m gpu tests need a GPU")
    from pathtracer_gb300 import Context, Scene, cie_analytic, native

    return {"torch": torch, "Context": Context, "Scene": Scene, "cie": cie_analytic(), "native": native}


def _case(rt, name, spf=2):
    scene = rt["Scene"].load(os.path.join(SCENES, name + ".json"))
    W, H = 96, 64
    push = scene.push_constants(W, H, spf, spf, spf, 4)
    with rt["Context"](0) as ctx:
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        ctx.dispatch(push)
        ctx.wait()
        return scene, W, H, push, ctx.read_accum()


def _hold(rt, stream):
    with rt["torch"].cuda.stream(stream):
        rt["torch"].cuda._sleep(HOLD)


def _read_last(rt, ctx):
    """The accumulator once every stream is idle."""
    rt["torch"].cuda.synchronize()
    return ctx.read_accum().view(np.uint32)


@pytest.mark.parametrize("engine", [0, 1])  # plain, default
@pytest.mark.parametrize("name", ["cornell_box", "mandelbulb12_plane"])  # the latter's SDF is compiled at run time
def test_zeroed_accumulator_then_dispatch(rt, name, engine):
    scene, W, H, push, want = _case(rt, name)
    a, b = rt["torch"].cuda.Stream(), rt["torch"].cuda.Stream()
    with rt["Context"](0) as ctx:
        ctx.set_engine(engine)
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        ctx.dispatch(push)  # compiled and loaded, buffers there
        ctx.wait()
        ctx.set_stream(a.cuda_stream)
        _hold(rt, a)
        ctx.resize_accum(W, H)
        ctx.set_stream(b.cuda_stream)
        ctx.dispatch(push)
        assert np.array_equal(_read_last(rt, ctx), want.view(np.uint32))
        ctx.set_stream(None)


@pytest.mark.parametrize("name", ["cornell_box", "mandelbulb12_plane"])
def test_plain_dispatch_then_another(rt, name):
    """The second dispatch, on a zeroed accumulator, follows the first."""
    scene, W, H, push, want = _case(rt, name)
    a, b = rt["torch"].cuda.Stream(), rt["torch"].cuda.Stream()
    with rt["Context"](0) as ctx:
        ctx.set_engine(rt["native"].PT_ENGINE_MEGAKERNEL)
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        ctx.dispatch(push)
        ctx.wait()
        ctx.set_stream(a.cuda_stream)
        _hold(rt, a)
        ctx.dispatch(push)
        ctx.set_stream(b.cuda_stream)
        ctx.resize_accum(W, H)
        ctx.dispatch(push)
        assert np.array_equal(_read_last(rt, ctx), want.view(np.uint32))
        ctx.set_stream(None)


@pytest.mark.parametrize("budget", [None, 64])  # the persistent kernel; the staged ones
def test_scene_change_then_dispatch(rt, budget):
    """The plug-ins change on the old stream, the dispatch follows on the new."""
    scene, W, H, push, want = _case(rt, "mandelbulb_plane")
    plugins = scene.sdf_plugins()
    other = rt["Scene"].load(os.path.join(SCENES, "menger_terrain.json")).sdf_plugins()
    a, b = rt["torch"].cuda.Stream(), rt["torch"].cuda.Stream()
    with rt["Context"](0) as ctx:
        if budget:
            ctx.set_march_budget(budget)
        ctx.bind(scene, rt["cie"])
        ctx.set_sdf_plugins(other[: len(plugins)])
        ctx.resize_accum(W, H)
        ctx.dispatch(push)
        ctx.resize_accum(W, H)
        ctx.wait()
        ctx.set_stream(a.cuda_stream)
        _hold(rt, a)
        ctx.set_sdf_plugins(plugins)
        ctx.set_stream(b.cuda_stream)
        ctx.dispatch(push)
        assert np.array_equal(_read_last(rt, ctx), want.view(np.uint32))
        ctx.set_stream(None)
