"""The plain engine's variant for small frames: frames on both sides of where
it ends (228 blocks of 16x8 pixels, 608 for spheres and planes), of one pixel, of ragged blocks and of
many blocks one way, for every class of scene without SDFs; the same bits as the
default engine's."""
import json
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["spheres", "cornell_box", "cornell_box_full", "feature_mix"])
def test_small_frames_equal_the_default_engine(built, name):
    from pathtracer_gb300 import Context, Scene, cie_analytic, native

    if name == "spheres":
        scene = Scene.generate(native.PT_GEN_SPHERES, 1)[0]
    else:
        with open(os.path.join(SCENES, name + ".json")) as f:
            d = json.load(f)
        d.pop("sdf", None)
        scene = Scene.parse(json.dumps(d))
    with Context(0) as ctx:
        ctx.bind(scene, cie_analytic())
        for W, H in ((1, 1), (17, 9), (192, 152), (192, 153), (1, 1824), (1, 1825), (3648, 8), (3649, 8), (512, 152), (513, 152)):
            push = scene.push_constants(W, H, 2, 2, 2, 5)
            images = []
            for engine in (native.PT_ENGINE_MEGAKERNEL, native.PT_ENGINE_WAVEFRONT):
                ctx.set_engine(engine)
                ctx.resize_accum(W, H)
                ctx.dispatch(push)
                ctx.wait()
                images.append(ctx.read_accum().view(np.uint32))
            assert np.array_equal(*images), (W, H)
