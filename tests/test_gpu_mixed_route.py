"""Scenes without SDFs that mix cyclides with boxes or lenses, on both sides of
the size where the default engine hands them to its staged kernels (3 * 2^19
samples): the same bits as the plain engine's."""
import json
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drop", [[], ["box"], ["lens"], ["cyclide"]])
def test_mixed_scenes_equal_the_plain_engine(built, drop):
    from pathtracer_gb300 import Context, Scene, cie_analytic, native

    with open(os.path.join(SCENES, "feature_mix.json")) as f:
        d = json.load(f)
    for k in ["sdf"] + drop:
        d.pop(k)
    scene = Scene.parse(json.dumps(d))
    with Context(0) as ctx:
        ctx.bind(scene, cie_analytic())
        for W, H, spp in ((1024, 512, 3), (1024, 513, 3)):
            push = scene.push_constants(W, H, spp, spp, spp, 5)
            images = []
            for engine in (native.PT_ENGINE_MEGAKERNEL, native.PT_ENGINE_WAVEFRONT):
                ctx.set_engine(engine)
                ctx.resize_accum(W, H)
                ctx.dispatch(push)
                ctx.wait()
                images.append(ctx.read_accum().view(np.uint32))
            assert np.array_equal(*images), (W, H)
