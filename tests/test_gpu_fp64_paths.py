"""The FP64 renderer's path kernel against its megakernel (which renders traced
dispatches): the same sums bit for bit.  Sizes: one sample; fewer than a warp's
share; odd; more than one block an SM (2^18 samples); two launches (2^21
samples), the second of them small.  Scenes with every primitive class,
mirrors and dielectrics, SDFs, sky; scratch that grows and is reused."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (1, 1, 77), (37, 3, 5), (256, 256, 4), (725, 724, 4)]


@pytest.mark.parametrize("name", ["cornell_box_full", "feature_mix", "spheres"])
def test_sums_equal_the_megakernel(built, name):
    import torch

    from pathtracer_gb300 import Context, Scene, cie_analytic, native

    if name == "spheres":
        scene, _ = Scene.generate(native.PT_GEN_SPHERES_FULL, 11)
    else:
        scene = Scene.load(os.path.join(SCENES, name + ".json"))
    with Context(0) as ctx:
        ctx.bind(scene, cie_analytic())
        for W, H, spp in SIZES if name != "feature_mix" else SIZES[:3]:
            push = scene.push_constants(W, H, 3 * spp, 3 * spp, spp, 7)
            sums = torch.full((2, H, W, 4), 0.5, dtype=torch.float64, device="cuda")  # added to what is there
            nev = torch.zeros(W * H * spp, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            ctx.render_fp64(push, sums[0].data_ptr())
            ctx.set_trace(0, nev.data_ptr(), 0, 0)
            ctx.render_fp64(push, sums[1].data_ptr())
            ctx.set_trace(0, 0, 0, 0)
            ctx.wait()
            got, want = sums.cpu().numpy().view(np.uint64)
            assert np.array_equal(got, want), (W, H, spp)
