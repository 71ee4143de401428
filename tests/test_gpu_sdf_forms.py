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


def test_device_export_bytes_match_host(rt):
    """A large image with values on both sides of every byte's border, zeros,
    negatives, infinities and NaN, through every tonemap."""
    import numpy as np
    import torch

    from pathtracer_gb300 import export_rgb8, native

    rng = np.random.default_rng(5)
    W, H = 1031, 517
    acc = np.ones((H, W, 4), np.float32)
    acc[..., :3] = np.exp(rng.uniform(-9.0, 3.0, (H, W, 1))) * rng.uniform(0.5, 1.5, (H, W, 3))
    acc.reshape(-1, 4)[::11, :3] *= -1.0
    acc.reshape(-1, 4)[5::997, 0] = np.nan
    acc.reshape(-1, 4)[6::997, 1] = np.inf
    acc.reshape(-1, 4)[7::997, :3] = 0.0
    d_acc, d_rgb = torch.from_numpy(acc).cuda(), torch.zeros(H * W * 3, dtype=torch.uint8, device="cuda")
    for tm in range(4):
        assert native.cuda().pt_export_rgb8_device(d_acc.data_ptr(), W, H, tm, d_rgb.data_ptr(), None) == native.PT_OK
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            assert np.array_equal(d_rgb.cpu().numpy().reshape(H, W, 3), export_rgb8(acc, tm)), tm
