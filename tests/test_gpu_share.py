"""The persistent kernel at launches of every share a warp's path slots are
chosen by (kernel/pt_share.h): around one and two warps' worth, around the size
of its arrays and between, in a context without SDFs, in one with built-in
SDFs, and in batches, one launch within a pass and one across passes.  The
same bits as the megakernel's."""
import json
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu

SHARES = (31, 32, 33, 64, 65, 72, 79, 80, 81)
WARPS = 4  # of a block


@pytest.fixture(scope="module")
def rt(built):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: -m gpu tests need a GPU")
    from pathtracer_gb300 import Batch, Context, Scene, cie_analytic, native

    return {"Batch": Batch, "Context": Context, "Scene": Scene, "cie": cie_analytic(), "native": native,
            "sms": torch.cuda.get_device_properties(0).multi_processor_count}


def _scene(rt, name):
    if name == "spheres":
        return rt["Scene"].generate(rt["native"].PT_GEN_SPHERES, 1)[0]
    with open(os.path.join(SCENES, name.split("-")[0] + ".json")) as f:
        d = json.load(f)
    if name.endswith("-analytic"):
        d.pop("sdf", None)
    return rt["Scene"].parse(json.dumps(d))


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("blocks", [4, 5])  # what the kernel's variants fit on an SM
@pytest.mark.parametrize("name", ["spheres", "cornell_box", "feature_mix-analytic", "feature_mix", "menger_terrain"])
def test_context_shares_equal_the_megakernel(rt, name, blocks):
    scene = _scene(rt, name)
    W = rt["sms"] * blocks
    with rt["Context"](0) as ctx:
        ctx.bind(scene, rt["cie"])
        for share in SHARES:
            H = WARPS * share
            push = scene.push_constants(W, H, 1, 1, 1, 4)
            got = []
            for engine in (rt["native"].PT_ENGINE_WAVEFRONT, rt["native"].PT_ENGINE_MEGAKERNEL):
                ctx.set_engine(engine)
                ctx.resize_accum(W, H)
                ctx.dispatch(push)
                ctx.wait()
                got.append(ctx.read_accum())
            assert _same(*got), share


@pytest.mark.parametrize("checks", [False, True])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("blocks", [4, 5])
def test_batch_shares_equal_the_megakernel(rt, passes, blocks, checks):
    scenes = [_scene(rt, "spheres"), _scene(rt, "feature_mix-analytic")][:passes]
    W = rt["sms"] * blocks
    for share in SHARES if not checks else (65, 79):
        H = WARPS * share
        if passes == 2:
            H //= 2
        got = []
        with rt["Batch"](0, pool_slots=4096, max_passes=8) as b:
            b.set_device_checks(checks)
            tids = []
            for s in scenes:
                sid = b.add_scene(s.pack_ubo(rt["cie"]), s.sdf_plugins())
                b.set_scene_ext(sid, s.ext_or_none())
                tids.append(b.add_target(W, H))
                b.add_pass(sid, tids[-1], s.push_constants(W, H, 1, 1, 1, 4))
            b.run()
            got = [b.read_target(t) for t in tids]
        for s, g in zip(scenes, got):
            with rt["Context"](0) as ctx:
                ctx.set_engine(rt["native"].PT_ENGINE_MEGAKERNEL)
                ctx.bind(s, rt["cie"])
                ctx.resize_accum(W, H)
                ctx.dispatch(s.push_constants(W, H, 1, 1, 1, 4))
                ctx.wait()
                assert _same(ctx.read_accum(), g), share
