"""What light cones may cost: cones along a surface give up."""
import json

import numpy as np
import pytest

from rtrace_b200 import workloads


def _count(gpu_ctx, path, w, h, dsamp):
    import rtrace_b200 as rt
    from rtrace_b200 import _capi
    scene = rt.Scene.from_json_file(path, gpu_ctx)
    r = rt.Renderer(w, h)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    r.disk_samples = dsamp
    r.flags = _capi.RT_FLAG_COUNT_WORK
    r.render(scene)
    scene.close()
    return r.last_stats


@pytest.mark.gpu
def test_cones_along_a_surface_give_up(gpu_ctx, tmp_path):
    with open(workloads.make_noisy_icosphere(str(tmp_path), level=5, seed=7)) as f:
        scene = json.load(f)
    scene["lights"][0]["diameter"] = 10.0
    scene["camera"]["fov"] = 0.5
    rng = np.random.default_rng(0)
    most = 0.0
    for k in range(60):  # a few pixels around points of the side that the camera sees
        p = rng.normal(size=3) + [0.8, -1.0, 0.5]
        scene["camera"]["target"] = [round(float(v), 4) for v in p / np.linalg.norm(p)]
        st = _count(gpu_ctx, workloads.write_scene(str(tmp_path), "view%d.json" % k, scene), 4, 4, 1)
        if st.shadow_rays:
            most = max(most, st.work["shadow_nodes"] / st.shadow_rays)
    # one ray a light: its cone visits 64 nodes at most, and the ray itself no
    # more than that at 15 levels of four boxes
    assert 0 < most <= 128
