"""The shipped SDF plug-ins' kernels where their forms change: terrain beyond
the range of the fast sine reduction, against the oracle per path."""
import json
import os

import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt(built):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: -m gpu tests need a GPU")
    from pathtracer_gb300 import Context, Scene, cie_analytic

    return {"Context": Context, "Scene": Scene, "cie": cie_analytic()}


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("x,z", [(65520.0, 0.0), (-70000.0, 66000.0), (0.0, 9.0e6)])
def test_terrain_far_out_matches_oracle(rt, x, z, engine):
    """The camera near and past |x| = 65536, where the terrain's 22 sines take
    their general form, over terrain whose box reaches there."""
    from oracle import compare

    with open(os.path.join(SCENES, "menger_terrain.json")) as f:
        d = json.load(f)
    terrain = [s for s in d["sdf"] if s["builtin"] == "terrain"][0]
    terrain["boundingSize"] = [4.0e7, 12.0, 4.0e7]
    for pos in d["camera"]["position"] + [s["position"] for s in d["sphere"]]:
        pos[0] += x
        pos[2] += z
    scene = rt["Scene"].parse(json.dumps(d))
    W, H, spf, depth = 40, 30, 2, 4
    push = scene.push_constants(W, H, spf, spf, spf, depth)
    acc_o, tr_o = compare.run_oracle(scene.pack_ubo(rt["cie"]), push, compare.plugins_for(scene), trace_depth=depth)
    with rt["Context"](0) as ctx:
        ctx.set_engine(engine)
        ctx.bind(scene, rt["cie"])
        ctx.resize_accum(W, H)
        acc_g, tr_g = compare.run_gpu(ctx, push, trace_depth=depth)
    rep = compare.compare(acc_o, tr_o, acc_g, tr_g, spf)
    assert compare.passes(rep) and rep["path_match"] == 1.0, rep
