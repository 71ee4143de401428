"""The work users have this renderer do, as measurable cases.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (scene, context, batch or server, all on the GPU), `run` makes one
pass through the public entry points and returns whole images.  Everything is
made from the seed: the camera of a scene file is moved by it, generated jobs
are drawn from it, an image to export is filled from it.

Kinds of work:
  frame      one dispatch on a context, the reference host's DrawFrame
  offscreen  the whole offscreen call: bind, dispatches, read-back
  batch      a few scenes and targets rendered as one batch, passes in order
  serve      a burst of requests through the server until every image is done
  fp64       the double-precision reference renderer
  export     the accumulator through the tonemap to 8-bit RGB on the host
"""
import json
import os

import numpy as np
import torch

from pathtracer_gb300 import SCENES_DIR, Batch, Context, Scene, Server, cie_analytic, native, render_offscreen

# FP32 operations of one path sample per scene, from the event counts of the
# CPU restatement (pathtracer_gb300/workmodel.py); the sphere jobs' average
# scene has 34 spheres.
FLOPS = {"cornell_box": 3200, "cornell_box_full": 3200, "feature_mix": 3200, "mandelbulb_plane": 9300,
         "mandelbulb12_plane": 16700, "mandelbulb12_plane_full": 9000, "menger_terrain": 24000,
         "menger_terrain_full": 20000, "spheres": 4000, "sdf_varied": 12000}

COMPILED = ("mandelbulb12_plane", "mandelbulb12_plane_full", "menger_terrain_full")  # SDF text compiled on load


def listed():
    return [
        # an interactive viewport: one sample per pixel per frame, latency counts
        {"name": "frame_cornell_256x1", "kind": "frame", "scene": "cornell_box", "w": 256, "h": 256, "spp": 1,
         "depth": 8, "plain": False},
        # a viewport of odd size on a scene with every primitive class and three shipped SDFs
        {"name": "frame_features_641x2", "kind": "frame", "scene": "feature_mix", "w": 641, "h": 359, "spp": 2,
         "depth": 6, "plain": False},
        # the small still: the Cornell box from host data to host image
        {"name": "offscreen_cornell_256x16", "kind": "offscreen", "scene": "cornell_box", "w": 256, "h": 256,
         "spp": 16, "depth": 8},
        # the benchmark's still: the 12-iteration mandelbulb, scene GLSL compiled at run time
        {"name": "still_bulb12_1024x64", "kind": "frame", "scene": "mandelbulb12_plane", "w": 1024, "h": 1024,
         "spp": 64, "depth": 6, "plain": False},
        # a mid-sized still of the shipped mandelbulb snippet, ragged size
        {"name": "still_bulb_777x16", "kind": "frame", "scene": "mandelbulb_plane", "w": 777, "h": 431, "spp": 16,
         "depth": 6, "plain": False},
        # one 16-sample pass of progressive refinement at full HD: menger sponge on the sine terrain
        {"name": "progressive_menger_1080x16", "kind": "batch", "scene": "menger_terrain", "w": 1920, "h": 1080,
         "spp": 16, "passes": 1, "depth": 12, "jobs": 1},
        # two passes of the same composition in its full form: fBm terrain as GLSL, dispersive glass, sky
        {"name": "progressive_menger_full_963x8", "kind": "batch", "scene": "menger_terrain_full", "w": 963, "h": 541,
         "spp": 8, "passes": 2, "depth": 12, "jobs": 1},
        # a render-farm batch: generated sphere jobs of mixed resolution with mirrors and dielectrics
        {"name": "batch_spheres_16jobs", "kind": "batch", "scene": "spheres", "w": 0, "h": 0, "spp": 24, "passes": 1,
         "depth": 8, "jobs": 16},
        # the plain drop-in kernel on one generated sphere scene
        {"name": "plain_spheres_1024x16", "kind": "frame", "scene": "spheres", "w": 1024, "h": 1024, "spp": 16,
         "depth": 8, "plain": True},
        # a served burst: sphere jobs and generated SDF jobs, 8-sample passes, error targets against references
        {"name": "serve_burst_8jobs", "kind": "serve", "scene": "spheres", "w": 512, "h": 512, "spp": 32, "passes": 4,
         "depth": 8, "jobs": 8},
        # a double-precision reference image, as error targets are measured against
        {"name": "fp64_cornell_full_128x4", "kind": "fp64", "scene": "cornell_box_full", "w": 128, "h": 128, "spp": 4,
         "depth": 8},
        # saving a finished render: tonemap on the device, bytes on the host
        {"name": "export_2560x1440", "kind": "export", "w": 2560, "h": 1440},
    ]


def _log(rng, lo, hi):
    """A whole number, uniform in its logarithm."""
    return int(round(float(lo) * (float(hi) / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "offscreen", "batch", "batch", "serve", "fp64", "export"])
    if kind == "export":
        return {"kind": kind, "w": _log(rng, 160, 2560), "h": _log(rng, 120, 1440)}
    if kind == "fp64":
        return {"kind": kind, "scene": rng.choice(["cornell_box_full", "cornell_box"]), "w": _log(rng, 32, 128),
                "h": _log(rng, 32, 128), "spp": rng.randint(1, 4), "depth": rng.randint(4, 8)}
    if kind == "offscreen":
        return {"kind": kind, "scene": rng.choice(["cornell_box", "feature_mix", "mandelbulb_plane"]),
                "w": _log(rng, 64, 512), "h": _log(rng, 64, 512), "spp": _log(rng, 1, 32), "depth": rng.randint(4, 8)}
    if kind == "serve":
        return {"kind": kind, "scene": "spheres", "w": _log(rng, 128, 512), "h": _log(rng, 128, 512),
                "spp": 8 * rng.randint(1, 4), "passes": 4, "depth": 8, "jobs": rng.randint(2, 8)}
    if kind == "batch":
        scene = rng.choice(["spheres", "menger_terrain", "mandelbulb_plane"])
        if scene == "spheres":
            return {"kind": kind, "scene": scene, "w": 0, "h": 0, "spp": _log(rng, 4, 24), "passes": rng.randint(1, 2),
                    "depth": 8, "jobs": rng.randint(2, 12)}
        return {"kind": kind, "scene": scene, "w": _log(rng, 160, 1920), "h": _log(rng, 90, 1080),
                "spp": _log(rng, 2, 16), "passes": 1, "depth": rng.randint(4, 12), "jobs": 1}
    scene = rng.choice(["cornell_box", "cornell_box_full", "feature_mix", "mandelbulb_plane", "mandelbulb12_plane",
                        "menger_terrain", "spheres"])
    return {"kind": kind, "scene": scene, "w": _log(rng, 64, 1024), "h": _log(rng, 64, 1024), "spp": _log(rng, 1, 32),
            "depth": rng.randint(4, 8), "plain": scene in ("cornell_box", "spheres") and rng.random() < 0.5}


class _DeviceImage:
    """A float4 image that a context or batch owns, as torch sees device memory; keeps its owner alive."""

    def __init__(self, owner, ptr, w, h):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (h, w, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _image(owner, ptr, w, h):
    return torch.as_tensor(_DeviceImage(owner, ptr, w, h), device="cuda")


def _scene(name, rng, seed):
    """The scene of a case and its camera's move: scene files by name, generated jobs from the seed."""
    if name == "spheres":
        scene, _ = Scene.generate(native.PT_GEN_SPHERES_FULL, seed)
    elif name == "sdf_varied":
        scene, _ = Scene.generate(native.PT_GEN_SDF_VARIED, seed)
    else:
        scene = Scene.load(os.path.join(SCENES_DIR, name + ".json"))
    return scene, (rng.uniform(-1.5, 1.5), rng.uniform(-0.75, 0.75))


def _push(scene, move, w, h, k, spp, depth):
    """Push constants of pass k (1-based) of spp samples, the camera turned by `move` degrees."""
    push = scene.push_constants(w, h, k * spp, k * spp, spp, depth)
    push.cameraAngle[0] += move[0]
    push.cameraAngle[1] += move[1]
    return push


def _job_size(case, j):
    """Width, height and samples of a batch's job j: mixed squares and sample counts where the case fixes no size."""
    if case["w"]:
        return case["w"], case["h"], case["spp"]
    side = (512, 128, 1024, 256)[j % 4]
    return side, side, max(4, case["spp"] * (4 - j % 3) // 4)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 20])
    cie = cie_analytic()
    kind = case["kind"]
    w, h = case.get("w"), case.get("h")
    if kind == "export":
        ctx = Context(0)
        ctx.resize_accum(w, h)
        img = rng.standard_normal((h, w, 4), dtype=np.float32)
        np.exp(img, out=img)  # a linear image spans a few stops
        ctx.write_accum(img * np.float32(0.3))
        return {"ctx": ctx}
    if kind == "frame":
        scene, move = _scene(case["scene"], rng, seed)
        ctx = Context(0)
        ctx.set_engine(native.PT_ENGINE_MEGAKERNEL if case["plain"] else native.PT_ENGINE_WAVEFRONT)
        ctx.bind(scene, cie)
        ctx.resize_accum(w, h)
        if case["scene"] in COMPILED:  # the compile on loading a scene, as the reference does it
            ctx.dispatch(_push(scene, move, w, h, 1, 1, case["depth"]))
        return {"ctx": ctx, "push": _push(scene, move, w, h, 1, case["spp"], case["depth"]),
                "out": _image(ctx, ctx.accum_device_ptr(), w, h)}
    if kind == "offscreen":
        scene, move = _scene(case["scene"], rng, seed)
        # the camera's move, in the scene itself: this call makes its own push constants
        d = json.loads(scene.to_json())
        d["camera"]["angle"][0][0] += move[0]
        d["camera"]["angle"][0][1] += move[1]
        return {"ctx": Context(0), "scene": Scene.parse(json.dumps(d)), "cie": cie, "case": case}
    if kind == "fp64":
        scene, move = _scene(case["scene"], rng, seed)
        ctx = Context(0)
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        ctx.bind(scene, cie)
        return {"ctx": ctx, "stream": stream, "push": _push(scene, move, w, h, 1, case["spp"], case["depth"]),
                "sums": torch.zeros((h, w, 4), dtype=torch.float64, device="cuda")}
    if kind == "batch":
        b = Batch(0, pool_slots=1 << 22)
        jobs = []
        for j in range(case["jobs"]):
            job_seed = 1000 * seed + j
            scene, move = _scene(case["scene"], rng, job_seed)
            jw, jh, spp = _job_size(case, j)
            sid = b.add_scene_sources(scene.pack_ubo(cie), scene.sdf_sources())
            b.set_scene_ext(sid, scene.ext_or_none())
            tid = b.add_target(jw, jh)
            pushes = [_push(scene, move, jw, jh, k + 1, spp, case["depth"]) for k in range(case["passes"])]
            jobs.append((sid, tid, pushes, _image(b, b.target_device_ptr(tid), jw, jh)))
        b.step(0)  # compiles what the scenes' texts need
        return {"batch": b, "jobs": jobs}
    # serve: one scene in four holds a generated SDF; half the jobs ask for an error target
    srv = Server(0, keep_images=True)
    jobs = []
    for j in range(case["jobs"]):
        scene, move = _scene("sdf_varied" if j % 4 == 3 else "spheres", rng, 1000 * seed + j)
        srv.add_scene_sources(j, scene.pack_ubo(cie), scene.sdf_sources())
        srv.set_scene_ext(j, scene.ext_or_none())
        push = _push(scene, move, w, h, 1, 8, case["depth"])
        target = 0.0
        if j % 2 == 0:
            srv.render_reference(j, push, 64)
            target = 0.12
        jobs.append(Server.job(j, push, case["spp"], target))
    return {"server": srv, "jobs": jobs}


def run(state):
    if "jobs" in state and "batch" in state:
        b = state["batch"]
        for k in range(max(len(p) for _, _, p, _ in state["jobs"])):
            for sid, tid, pushes, _ in state["jobs"]:
                if k < len(pushes):
                    b.add_pass(sid, tid, pushes[k])
        b.run()
        return [image for _, _, _, image in state["jobs"]]
    if "server" in state:
        srv = state["server"]
        ids = [srv.submit(j) for j in state["jobs"]]
        done = {r.job_id: r for r in srv.drain()}
        out = {"images": [srv.read_image(i) for i in ids], "spp": [done[i].spp for i in ids],
               "rmse": [float(done[i].rmse) for i in ids]}
        for i in ids:
            srv.release(i)
        return out
    if "sums" in state:
        with torch.cuda.stream(state["stream"]):
            state["sums"].zero_()
        state["ctx"].render_fp64(state["push"], state["sums"].data_ptr())
        return state["sums"]
    if "scene" in state:
        c = state["case"]
        image, _ = render_offscreen(state["ctx"], state["scene"], state["cie"], c["w"], c["h"], c["spp"], c["spp"],
                                    c["depth"])
        return image
    if "push" in state:
        state["ctx"].dispatch(state["push"])
        return state["out"]
    return state["ctx"].read_rgb8(3)


def work(case):
    """Each image written once (export: read as floats, written as bytes), each sample's path arithmetic."""
    if case["kind"] == "export":
        return {"bytes": 19.0 * case["w"] * case["h"], "flops": 60.0 * case["w"] * case["h"]}
    jobs = case.get("jobs", 1)
    if case["kind"] == "batch":
        sizes = [_job_size(case, j) for j in range(jobs)]
        pixels = sum(w * h for w, h, _ in sizes)
        samples = sum(w * h * spp for w, h, spp in sizes) * case["passes"]
    else:
        pixels = jobs * case["w"] * case["h"]
        samples = pixels * case["spp"]
    per = FLOPS[case["scene"]]
    if case["kind"] == "serve":
        per = 0.75 * FLOPS["spheres"] + 0.25 * FLOPS["sdf_varied"]
    return {"bytes": pixels * (32.0 if case["kind"] == "fp64" else 16.0), "flops": samples * per}


def exact(case, seed):
    # A Monte Carlo image has no value in 64 bits that a float run could be held to: the last bit of one
    # rounding moves whole paths (the renderer's own double-precision form is one of the cases).  The
    # exported bytes are whole numbers.
    return None
