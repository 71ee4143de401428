"""The sphere loop's two passes (intersect_spheres) against the oracle per
path: counts around the threshold and the 32-sphere chunks, spheres inside one
another, very small, far from the origin, and behind the camera."""
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
    from pathtracer_gb300 import Batch, Context, Scene, cie_analytic, native

    return {"Batch": Batch, "Context": Context, "Scene": Scene, "cie": cie_analytic(), "native": native}


def _scene(rt, n, shift):
    rng = np.random.default_rng(100 + n)
    with open(os.path.join(SCENES, "feature_mix.json")) as f:
        d = json.load(f)
    pos = np.array(d["camera"]["position"][0])
    spheres = []
    for i in range(n):
        p = rng.uniform(-3, 3, 3) + [0, 1.5, 0]
        r = float(np.exp(rng.uniform(np.log(0.004), np.log(1.2))))
        if i % 7 == 3 and spheres:  # inside the one before
            p, r = np.array(spheres[-1]["position"]), 0.5 * spheres[-1]["radius"]
        spheres.append({"position": [float(x) for x in p], "radius": r, "materialID": 1 + i % 3,
                        "lightID": 1 if i % 9 == 4 else 0})
    spheres[-1] = {"position": [float(x) for x in pos + [0, 2.5, 0]], "radius": 1.0, "materialID": 1, "lightID": 2}
    d["sphere"] = spheres
    for k in ("box", "lens", "cyclide", "sdf"):
        d.pop(k, None)
    for s in d["sphere"] + d["plane"]:
        s["position"] = [float(np.float32(x + shift)) for x in s["position"]]
    d["camera"]["position"][0] = [float(x + shift) for x in pos]
    return rt["Scene"].parse(json.dumps(d))


@pytest.mark.parametrize("n,shift", [(3, 0.0), (4, 0.0), (5, 0.0), (31, 0.0), (32, 0.0), (33, 0.0), (64, 0.0), (65, 0.0),
                                     (120, 0.0), (33, 400.0)])
def test_sphere_counts_match_oracle(rt, n, shift):
    """Both engines and the batch's persistent kernel."""
    from oracle import compare

    scene = _scene(rt, n, shift)
    ubo = scene.pack_ubo(rt["cie"])
    W, H, spf, depth = 40, 30, 3, 6
    push = scene.push_constants(W, H, spf, spf, spf, depth)
    acc_o, tr_o = compare.run_oracle(ubo, push, [], trace_depth=depth)
    for engine in (0, 1):
        with rt["Context"](0) as ctx:
            ctx.set_engine(engine)
            ctx.bind(scene, rt["cie"])
            ctx.resize_accum(W, H)
            acc_g, tr_g = compare.run_gpu(ctx, push, trace_depth=depth)
            rep = compare.compare(acc_o, tr_o, acc_g, tr_g, spf)
            assert compare.passes(rep) and rep["path_match"] == 1.0, (engine, rep)
            ctx.resize_accum(W, H)
            ctx.set_trace(0, 0, 0, 0)
            ctx.dispatch(push)
            np.testing.assert_array_equal(ctx.read_accum()[..., :3], acc_o[..., :3])
    with rt["Batch"](0, pool_slots=1 << 12, max_passes=4) as b:
        b.set_route(rt["native"].PT_BATCH_ROUTE_PERSISTENT)
        sid = b.add_scene(ubo, [])
        tid = b.add_target(W, H)
        b.add_pass(sid, tid, push)
        b.run()
        np.testing.assert_array_equal(b.read_target(tid)[..., :3], acc_o[..., :3])
