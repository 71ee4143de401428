"""The default engine's dispatch in a stream capture: refused, whichever of its
kernels would run and whether or not its buffers exist already, with the
capture left valid; a graph of the plain engine captured beside it replays
to the same image after a larger dispatch has replaced those buffers."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("name,staged", [("cornell_box", False), ("cornell_box", True), ("feature_mix", False),
                                         ("mandelbulb12_plane", True)])
def test_default_engine_is_refused_in_a_capture(built, name, staged, warm):
    import torch

    from pathtracer_gb300 import Context, Scene, cie_analytic, native
    from pathtracer_gb300.renderer import PathTracerError

    W, H = 96, 64
    scene = Scene.load(os.path.join(SCENES, name + ".json"))
    push = scene.push_constants(W, H, 2, 2, 2, 4)
    with Context(0) as ctx:
        ctx.bind(scene, cie_analytic())
        ctx.resize_accum(W, H)
        if staged:
            ctx.set_march_budget(64)
        # one of each engine: modules compiled and loaded, buffers there when warm
        ctx.set_engine(native.PT_ENGINE_MEGAKERNEL)
        ctx.dispatch(push)
        ctx.wait()
        want = ctx.read_accum()
        ctx.set_engine(native.PT_ENGINE_WAVEFRONT)
        if warm:
            ctx.dispatch(push)
            ctx.wait()
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            with pytest.raises(PathTracerError):
                ctx.dispatch(push)
            ctx.set_engine(native.PT_ENGINE_MEGAKERNEL)
            ctx.dispatch(push)
        ctx.set_engine(native.PT_ENGINE_WAVEFRONT)
        ctx.resize_accum(W, H)
        ctx.dispatch(scene.push_constants(W, H, 16, 16, 16, 4))  # a larger dispatch
        ctx.resize_accum(W, H)  # the same size: zeroed in place
        ctx.wait()  # the graph replays on another stream
        graph.replay()
        torch.cuda.synchronize()
        got = ctx.read_accum()
        ctx.set_stream(None)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
