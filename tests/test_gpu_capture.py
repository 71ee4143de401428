"""The plain engine's dispatch inside a stream capture: the stream set before
or within it, after a dispatch that is still queued on the context's own."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("set_inside", [False, True])
def test_captured_dispatch_replays(built, set_inside):
    import torch

    from pathtracer_gb300 import Context, Scene, cie_analytic, native

    W, H = 96, 64
    scene = Scene.load(os.path.join(SCENES, "cornell_box.json"))
    push = scene.push_constants(W, H, 2, 2, 2, 6)
    images = []
    for captured in (False, True):
        with Context(0) as ctx:
            ctx.bind(scene, cie_analytic())
            ctx.resize_accum(W, H)
            ctx.dispatch(push)  # the engine's own kernels, queued when the stream changes
            if not captured:
                ctx.wait()
            ctx.set_engine(native.PT_ENGINE_MEGAKERNEL)
            stream = torch.cuda.Stream()
            if captured:
                graph = torch.cuda.CUDAGraph()
                if not set_inside:
                    ctx.set_stream(stream.cuda_stream)
                with torch.cuda.graph(graph, stream=stream):
                    if set_inside:
                        ctx.set_stream(stream.cuda_stream)
                    ctx.dispatch(push)
                    if set_inside:
                        ctx.set_stream(None)
                graph.replay()
                torch.cuda.synchronize()
                ctx.set_stream(None)
                graph.replay()
                torch.cuda.synchronize()
            else:
                ctx.dispatch(push)
                ctx.dispatch(push)
                ctx.wait()
            images.append(ctx.read_accum())
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
