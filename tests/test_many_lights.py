"""Hits of many lights, a thread for each of a hit's lights where hits are few:
work by level and images against the oracle around the rule's line."""

import numpy as np
import pytest

from rtrace_b200 import workloads


def _scene(lights, disks):
    s = workloads.ring_spheres_scene(seed=1, n_rings=3, per_ring=15)
    rng = np.random.default_rng(lights)
    s["lights"] = []
    for k in range(lights):
        p = [round(float(v), 4) for v in rng.uniform([-6, -6, 4], [6, 6, 8])]
        light = {"position": p, "color": "#FFFFFF", "intensity": round(1.5 / lights, 4)}
        if k % 2 < disks:
            light["diameter"] = [0.8, 0.8, 1.4][k % 3]
        s["lights"].append(light)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("lights", [4, 5, 9])
@pytest.mark.parametrize("disks", [0, 1])
def test_many_lights_match_the_oracle(gpu_ctx, tmp_path, lights, disks):
    import rtrace_b200 as rt
    from tests import oracle_lib
    path = workloads.write_scene(str(tmp_path), "lights.json", _scene(lights, disks))
    scene = rt.Scene.from_json_file(path, gpu_ctx)
    r = rt.Renderer(96, 54)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    got, st = r.render(scene), r.last_stats
    scene.close()
    want, cnt = oracle_lib.render(path=path, width=96, height=54, aa="no-jitter", counts=True)
    assert np.array_equal(got, want)
    assert (st.primary_rays, st.reflection_rays, st.shadow_rays) == (int(cnt[0]), int(cnt[1]), int(cnt[2]))


@pytest.mark.gpu
@pytest.mark.parametrize("lights", [5, 12])
@pytest.mark.parametrize("disks", [0, 1])
def test_frames_on_both_sides_of_the_line_are_the_same(gpu_ctx, tmp_path, lights, disks):
    """A frame of more than 2^22 pairs, whose level 0 takes a thread per hit and
    whose other levels one per light, against its bands, which split all."""
    import rtrace_b200 as rt
    path = workloads.write_scene(str(tmp_path), "lights.json", _scene(lights, disks))
    scene = rt.Scene.from_json_file(path, gpu_ctx)
    r = rt.Renderer(1280, 720)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    r.max_depth = 6
    whole = r.render(scene)
    assert 1280 * 720 * lights > 1 << 22 and r.last_stats.hits > 1 << 16
    bands = [r.render_rows(scene, y, min(720, y + 48)) for y in range(0, 720, 48)]  # 61,440 pixels each
    scene.close()
    assert np.array_equal(whole, np.concatenate(bands))
