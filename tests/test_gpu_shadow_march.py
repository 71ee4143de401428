"""Shadow rays that march no further than their answer needs: no march when
the analytic hit decides, no normal or material, the SDF's sign at the origin
kept for the bounce ray.  Against the oracle per path, on scenes with one and
several SDFs and with light lists that name no object (index -1: an SDF hit or
a miss reaches "the light"; an index past the objects: nothing does)."""
import os

import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt(built):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: -m gpu tests need a GPU")
    from pathtracer_gb300 import Context, Scene, cie_analytic, native

    return {"Context": Context, "Scene": Scene, "cie": cie_analytic(), "native": native}


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("light", [None, -1.0, 190.0])
@pytest.mark.parametrize("name,depth", [("feature_mix", 5), ("menger_terrain", 5), ("mandelbulb_plane", 4)])
def test_shadow_rays_match_oracle(rt, name, depth, light, engine):
    from oracle import compare

    scene = rt["Scene"].load(os.path.join(SCENES, name + ".json"))
    ubo = scene.pack_ubo(rt["cie"])
    if light is not None:
        off, n = rt["native"].UBO_OFFSETS["lightIDs"]
        ubo[off:off + n] = light
    W, H, spf = 48, 36, 4
    push = scene.push_constants(W, H, spf, spf, spf, depth)
    acc_o, tr_o = compare.run_oracle(ubo, push, compare.plugins_for(scene), trace_depth=depth)
    with rt["Context"](0) as ctx:
        ctx.set_engine(engine)
        ctx.set_march_budget(5)  # suspended and resumed shadow marches too
        ctx.set_sdfs(scene.sdf_sources())
        ctx.upload_scene(ubo)
        ctx.resize_accum(W, H)
        acc_g, tr_g = compare.run_gpu(ctx, push, trace_depth=depth)
    rep = compare.compare(acc_o, tr_o, acc_g, tr_g, spf)
    assert compare.passes(rep) and rep["path_match"] == 1.0, rep
