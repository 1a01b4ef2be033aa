"""Levels with many walked pairs, which have a kernel of their own and fewer
lanes a pair the more there are: the frame is that of its row bands, which are
too small for either."""
import json

import numpy as np
import pytest

from rtrace_b200 import workloads


# samples per pixel, lights, rays a light; 16, 8, 2 and 1 lanes a pair
@pytest.mark.gpu
@pytest.mark.parametrize("spp,lights,rays", [(1, 1, 16), (1, 2, 16), (1, 1, 64), (1, 1, 1), (1, 1, 5), (4, 1, 16), (4, 2, 16)])
def test_frame_is_that_of_its_bands(gpu_ctx, tmp_path, spp, lights, rays):
    import rtrace_b200 as rt
    with open(workloads.make_noisy_icosphere(str(tmp_path), level=4, seed=7, outline=False)) as f:
        scene = json.load(f)
    first = dict(scene["lights"][0], diameter=16.0)  # every point lies within its radius: each ray walks
    scene["lights"] = [first, dict(first, position=[-3.0, -2.0, 4.0], intensity=0.4)][:lights]
    sc = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "walks.json", scene), gpu_ctx)
    w, h = 1200, 900
    r = rt.Renderer(w, h)
    r.anti_aliasing_mode = rt.AntiAliasingMode.Stochastic if spp > 1 else rt.AntiAliasingMode.NoJitter
    r.samples = spp
    r.disk_samples = rays
    r.max_depth = 2
    whole = r.render(sc)
    assert r.last_stats.hits * lights >= 1 << 18
    step = (1 << 18) // (w * spp * lights)
    bands = [r.render_rows(sc, y, min(h, y + step)) for y in range(0, h, step)]
    sc.close()
    assert np.array_equal(whole, np.concatenate(bands))
