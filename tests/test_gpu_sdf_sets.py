"""Scenes with several SDFs, whose rays carry different sets of them: copies of
one SDF apart, touching and in a row, SDFs of several kinds whose boxes meet,
more than a walked group holds, and a mixture; against the oracle per path and
by every route, the rays crossing from one group of boxes into the next."""
import json
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
    from pathtracer_gb300 import Batch, Context, Scene, cie_analytic

    return {"Batch": Batch, "Context": Context, "Scene": Scene, "cie": cie_analytic()}


def _row(names, gap, size):
    n = len(names)
    return [{"position": [gap * (k % 4 - 1.5), 1.2, -gap * (k // 4)], "boundingSize": [size] * 3, "builtin": names[k]}
            for k in range(n)]


TERRAIN = {"position": [0.0, -5.2, 0.0], "boundingSize": [60.0, 12.0, 60.0], "builtin": "terrain"}
SETS = {
    "copies apart": _row(["menger"] * 5, 2.6, 2.2),
    "copies touching": _row(["menger"] * 6, 2.0, 2.2),
    "kinds apart": _row(["menger", "blob", "mandelbulb"], 3.2, 2.4),
    "kinds meeting": _row(["menger", "blob", "mandelbulb"], 1.1, 2.4) + [TERRAIN],
    "copies on terrain": _row(["menger"] * 4, 2.4, 2.2) + [TERRAIN],
    "many": _row(["menger", "blob"] * 6, 1.3, 2.2),
}


@pytest.mark.parametrize("name", SETS)
def test_sets_match_oracle(rt, name):
    from oracle import compare

    with open(os.path.join(SCENES, "menger_terrain.json")) as f:
        d = json.load(f)
    d["sdf"] = SETS[name]
    scene = rt["Scene"].parse(json.dumps(d))
    W, H, spf, depth = 48, 32, 2, 6
    ubo = scene.pack_ubo(rt["cie"])
    push = scene.push_constants(W, H, spf, spf, spf, depth)
    acc_o, tr_o = compare.run_oracle(ubo, push, compare.plugins_for(scene), trace_depth=depth)
    images = []
    for engine in (0, 1):
        with rt["Context"](0) as ctx:
            ctx.set_engine(engine)
            ctx.bind(scene, rt["cie"])
            ctx.resize_accum(W, H)
            acc_g, tr_g = compare.run_gpu(ctx, push, trace_depth=depth)  # the default engine: its staged kernels
            rep = compare.compare(acc_o, tr_o, acc_g, tr_g, spf)
            assert compare.passes(rep) and rep["path_match"] == 1.0, (engine, rep)
            images.append(acc_g)
            ctx.resize_accum(W, H)
            ctx.set_trace(0, 0, 0, 0)
            ctx.dispatch(push)  # the default engine: the persistent kernel
            images.append(ctx.read_accum())
            ctx.set_march_budget(5)  # suspended marches
            ctx.resize_accum(W, H)
            ctx.dispatch(push)
            images.append(ctx.read_accum())
    with rt["Batch"](0, pool_slots=1 << 12, max_passes=4) as b:
        sid = b.add_scene(ubo, scene.sdf_plugins())
        tid = b.add_target(W, H)
        b.add_pass(sid, tid, push)
        b.run()
        images.append(b.read_target(tid))
    for im in images:
        np.testing.assert_array_equal(im[..., :3], images[0][..., :3])


def test_many_snippets_equal_on_both_engines(rt):
    """Ten compiled snippets in boxes that meet, one of them a copy's text: the
    staged march walks them together; both engines give the same bits."""
    with open(os.path.join(SCENES, "menger_terrain.json")) as f:
        d = json.load(f)
    text = ("float sdf(vec3 p){ vec3 q = abs(p) - vec3(0.%d); return length(max(q, 0.0)) + min(max(q.x, max(q.y, q.z)), 0.0)"
            " - 0.05; }\nfloat sdfmaterial(vec3 p){ return 2.0; }")
    d["sdf"] = [{"position": [0.6 * (k % 5 - 2), 1.2, 0.6 * (k // 5)], "boundingSize": [1.6] * 3,
                 "glsl": text % (30 + min(k, 8))} for k in range(10)]
    scene = rt["Scene"].parse(json.dumps(d))
    W, H = 64, 40
    push = scene.push_constants(W, H, 3, 3, 3, 6)
    images = []
    for engine in (0, 1):
        with rt["Context"](0) as ctx:
            ctx.set_engine(engine)
            ctx.bind(scene, rt["cie"])
            ctx.resize_accum(W, H)
            ctx.dispatch(push)
            images.append(ctx.read_accum().view(np.uint32))
    assert np.array_equal(*images)
