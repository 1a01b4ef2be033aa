"""A context's scratch memory: set up in the order of the stream whose kernels
use it."""
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
