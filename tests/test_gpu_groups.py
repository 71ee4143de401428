"""A batch of scenes whose SDFs run different code (march groups): every job's
image is the same bits as alone on the megakernel, with one group, a few, and
more scenes than groups; pools that recycle and suspended marches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt(built):
    import torch

    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: -m gpu tests need a GPU")
    from pathtracer_gb300 import Batch, Context, Scene, cie_analytic, native

    return {"Batch": Batch, "Context": Context, "Scene": Scene, "cie": cie_analytic(), "native": native}


@pytest.mark.parametrize("kind,count,checks", [("shipped", 1, False), ("shipped", 6, False), ("varied", 5, True),
                                               ("varied", 19, False)])
def test_grouped_batch_equals_each_job_alone(rt, kind, count, checks):
    native = rt["native"]
    k = native.PT_GEN_SDF if kind == "shipped" else native.PT_GEN_SDF_VARIED
    jobs = []
    for s in range(count):
        scene, _ = rt["Scene"].generate(k, s)
        W, H, spf = 40 + 3 * (s % 5), 30 + s % 3, 3 + s % 4
        jobs.append((scene, W, H, [scene.push_constants(W, H, n * spf, n * spf, spf, 6) for n in (1, 2)]))
    with rt["Batch"](0, pool_slots=4096, max_passes=64) as b:
        b.set_march_budget(7)
        b.set_device_checks(checks)
        ids = []
        for scene, W, H, _ in jobs:
            sid = b.add_scene_sources(scene.pack_ubo(rt["cie"]), scene.sdf_sources())
            b.set_scene_ext(sid, scene.ext_or_none())
            ids.append((sid, b.add_target(W, H)))
        for n in range(2):
            for (sid, tid), (_, _, _, pushes) in zip(ids, jobs):
                b.add_pass(sid, tid, pushes[n])
        b.run()
        got = [b.read_target(t) for _, t in ids]
    with rt["Context"](0) as ctx:
        ctx.set_engine(native.PT_ENGINE_MEGAKERNEL)
        for i in sorted({0, 1, 2, 3, count // 2, count - 2, count - 1} & set(range(count))):
            scene, W, H, pushes = jobs[i]
            ctx.bind(scene, rt["cie"])
            ctx.resize_accum(W, H)
            for p in pushes:
                ctx.dispatch(p)
            ctx.wait()
            assert np.array_equal(ctx.read_accum().view(np.uint32), got[i].view(np.uint32)), i
