"""March groups follow the live scenes: an iteration sorts its queue only while
scenes with different SDF code are live, however many came and went; the
images are the megakernel's bits throughout."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu

W, H, SPF = 72, 48, 3


def test_released_scenes_leave_their_group(built):
    from pathtracer_gb300 import Batch, Context, Scene, cie_analytic, native

    cie = cie_analytic()
    names = ["mandelbulb_plane", "menger_terrain", "feature_mix"]
    scenes = [Scene.load(os.path.join(SCENES, n + ".json")) for n in names]
    push = [s.push_constants(W, H, SPF, SPF, SPF, 5) for s in scenes]
    want = []
    with Context(0) as ctx:
        ctx.set_engine(native.PT_ENGINE_MEGAKERNEL)
        for s, p in zip(scenes, push):
            ctx.bind(s, cie)
            ctx.resize_accum(W, H)
            ctx.dispatch(p)
            ctx.wait()
            want.append(ctx.read_accum())

    with Batch(0, pool_slots=4096, max_passes=16) as b:
        def add(k):
            sid = b.add_scene(scenes[k].pack_ubo(cie), scenes[k].sdf_plugins())
            b.set_scene_ext(sid, scenes[k].ext_or_none())
            return sid

        def render(ids):
            """Kernels of one iteration; the images of the scenes ids[k] -> k are checked."""
            tids = {sid: b.add_target(W, H) for sid in ids}
            for sid, k in ids.items():
                b.add_pass(sid, tids[sid], push[k])
            before = b.stats()["kernel_launches"]
            assert b.step(1) == []
            launched = b.stats()["kernel_launches"] - before
            b.run()
            for sid, k in ids.items():
                assert np.array_equal(b.read_target(tids[sid]).view(np.uint32), want[k].view(np.uint32)), names[k]
            return launched

        first = add(0)
        one = render({first: 0})
        for turn in range(20):  # more scenes than groups
            k = 1 + turn % 2
            second = add(k)
            assert render({first: 0, second: k}) == one + 2
            b.release_scene(second)
            if turn % 5 == 0:
                assert render({first: 0}) == one
        third = [add(0), add(0)]  # the same code: one group
        assert render({first: 0, third[0]: 0, third[1]: 0}) == one
        b.release_scene(first)
        assert render({third[0]: 0}) == one
