"""A context's scratch memory: set up in the order of the stream whose kernels
use it, and counted for a batch's group as it is allocated."""
import os
import re

import numpy as np
import pytest

from rtrace_b200 import workloads

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rtrace_b200", "csrc")


def _function(name):
    src = open(os.path.join(CSRC, "render.cu")).read()
    body = src[src.index("rt_status %s(" % name):]
    return body[:body.index("\n}\n")]


def test_the_scratch_is_set_up_on_the_contexts_stream():
    # the context's stream does not wait for the legacy stream, so what is
    # set up there is not ordered before the frame's kernels
    body = _function("ensure_scratch")
    calls = re.findall(r"cudaMem(?:set|cpy)\w*\(.*?\)\);", body, re.S)
    assert len(calls) >= 2
    assert all("Async(" in c and "ctx->stream" in c for c in calls), calls


# a frame whose deep levels share one launch, on contexts whose scratch is
# new, then grown, while the legacy stream is busy
@pytest.mark.gpu
def test_first_frames_beside_a_busy_legacy_stream(gpu_ctx, tmp_path):
    import torch
    import rtrace_b200 as rt
    path = workloads.write_scene(str(tmp_path), "s.json", workloads.sphere_grid_scene())
    want = {}
    for w, h in ((64, 48), (160, 120)):
        want[w] = rt.Renderer(w, h).render(rt.Scene.from_json_file(path, gpu_ctx))
    a = torch.rand((4096, 4096), device="cuda")
    for _ in range(4):
        ctx = rt.Context(gpu_ctx.device)
        scene = rt.Scene.from_json_file(path, ctx)
        for w, h in ((64, 48), (160, 120)):
            for _ in range(10):
                a = torch.tanh(a @ a)
            assert np.array_equal(rt.Renderer(w, h).render(scene), want[w])
        scene.close()
    torch.cuda.synchronize()


# a budget for four frames of a group holds four: per primary ray and level 36
# bytes, 241 more (queues, hits, records, outline), 32 per light and 57 per
# disk light; per pixel 80
@pytest.mark.gpu
@pytest.mark.parametrize("disk,point", [(0, 1), (2, 0), (3, 1)])
def test_a_group_holds_the_frames_its_budget_pays_for(gpu_ctx, tmp_path, disk, point):
    import rtrace_b200 as rt
    s = workloads.sphere_grid_scene()
    light = {"position": [3, -3, 5], "color": "#FFFFFF", "intensity": 0.3}
    s["lights"] = [dict(light, diameter=0.5) for _ in range(disk)] + [dict(light) for _ in range(point)]
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", s), gpu_ctx)
    jobs = []
    for k in range(6):
        r = rt.Renderer(200, 150)
        r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
        r.max_depth = 2
        jobs.append(rt.Job(scene, r))
    frame = 200 * 150 * (2 * 36 + 241 + 32 * (disk + point) + 57 * disk + 80)
    saved = rt.batch_tuning(gpu_ctx)
    try:
        for frames in (2, 4, 5):
            rt.batch_tuning(gpu_ctx, fuse_pixels=1 << 20, fuse_bytes=int((frames + 0.1) * frame))
            rt.render_batch(jobs, lanes=2, ctx=gpu_ctx)
            assert sum(j.renderer.last_stats.graph != 0 for j in jobs) == frames
    finally:
        rt.batch_tuning(gpu_ctx, lanes=saved["lanes"], fuse_pixels=saved["fuse_pixels"],
                        fuse_bytes=saved["fuse_bytes"], blocks_per_sm=saved["blocks_per_sm"])
    scene.close()


# a frame that no device holds gives back what the scratch held before it
@pytest.mark.gpu
def test_a_context_is_usable_after_a_frame_that_does_not_fit(tmp_path):
    import torch
    import rtrace_b200 as rt
    from rtrace_b200 import _capi, denoiser
    ctx = rt.Context(0)
    ctx.load_denoiser(denoiser.pack(denoiser.random_layers(7)))
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", workloads.sphere_grid_scene()), ctx)
    feat = torch.rand((1, 40, 60, 16), device="cuda").half()
    torch.cuda.synchronize()

    def net():
        vis = torch.zeros((1, 2, 40, 60), device="cuda")
        torch.cuda.synchronize()
        L = _capi.lib()
        assert L.rt_denoiser_run(ctx.handle, feat.data_ptr(), 1, 40, 60, vis.data_ptr(), None, None) == 0, \
            L.rt_last_error(ctx.handle)
        return vis
    image, vis = rt.Renderer(64, 48).render(scene), net()
    huge = rt.Renderer(30000, 30000)  # 1.8 billion rays: 900 GB
    huge.anti_aliasing_mode, huge.samples = rt.AntiAliasingMode.Stochastic, 2
    for _ in range(2):
        with pytest.raises(rt.DeviceError, match="memory"):
            huge.render(scene, device_ptr=feat.data_ptr())  # fails before anything is written
        assert torch.equal(net(), vis)
    assert np.array_equal(rt.Renderer(64, 48).render(scene), image)
    scene.close()


# pinned host memory of a group's frames: their results, a kilobyte each, and no
# image buffer that no frame of a group uses
@pytest.mark.gpu
def test_a_group_of_many_frames_pins_little_host_memory(tmp_path):
    import rtrace_b200 as rt

    def pinned_mb():
        return next(int(line.split()[1]) for line in open("/proc/self/status") if line.startswith("RssShmem")) / 1024
    ctx = rt.Context(0)
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", workloads.sphere_grid_scene()), ctx)
    jobs = []
    for _ in range(128):
        r = rt.Renderer(16, 12)
        r.max_depth = 2
        jobs.append(rt.Job(scene, r))
    want = jobs[0].renderer.render(scene)
    rt.batch_tuning(ctx, fuse_pixels=1 << 20)
    before = pinned_mb()
    images, _ = rt.render_batch(jobs, lanes=1, ctx=ctx)
    assert pinned_mb() - before < 32
    assert all(j.renderer.last_stats.graph != 0 for j in jobs) and all(np.array_equal(i, want) for i in images)
    scene.close()
