"""Batches asked for more path slots than a queue entry can name (2^28): they
use that many, and their images are the same bits as with a small pool.  New
samples take the highest slots first, so the largest slots are used."""
import os

import numpy as np
import pytest

from conftest import SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [(1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 28) + (1 << 20)])
def test_batch_with_the_largest_pool(built, slots):
    import torch

    from pathtracer_gb300 import Batch, Scene, cie_analytic

    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB for a pool of 2^28 slots")
    W, H, spf = 128, 96, 4
    scene = Scene.load(os.path.join(SCENES, "feature_mix.json"))
    images = []
    for n in (4096, slots):
        with Batch(0, pool_slots=n, max_passes=8) as b:
            b.set_march_budget(5)  # suspended marches
            sid = b.add_scene(scene.pack_ubo(cie_analytic()), scene.sdf_plugins())
            b.set_scene_ext(sid, scene.ext_or_none())
            tid = b.add_target(W, H)
            b.add_pass(sid, tid, scene.push_constants(W, H, spf, spf, spf, 6))
            for _ in range(12):  # iterations of the staged kernels alone
                b.step(1)
            b.run()
            images.append(b.read_target(tid))
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
