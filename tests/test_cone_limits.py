"""What light cones may cost: cones along a surface give up, and cubes off the
cone leave its rays unwalked.  Cubes of every kind of transform, byte for byte
against the oracle."""
import json

import numpy as np
import pytest

from rtrace_b200 import workloads

MAT = workloads._mat


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


def _cubes(rng, n, scale):
    out = []
    for _ in range(n):
        c = [round(float(v), 4) for v in rng.uniform([-4, -4, 0], [4, 4, 2.5])]
        m = {"kind": "cube", "center": c, "size": [round(float(v), 3) for v in rng.uniform(0.2, 0.8, 3)],
             "material": MAT("#60A0C0", reflectivity=0.2)}
        if scale:
            m["transform"] = ["scale(%s)" % scale, "rotate(%d, %d, %d)" % tuple(rng.integers(-80, 80, 3))]
        out.append(m)
    return out


def _scene(objects, diameter):
    return {
        "camera": {"kind": "perspective", "position": [1, -9, 6], "target": [0, 0, 0.5], "up": [0, 0, 1], "fov": 50,
                   "width": 16, "height": 9},
        "objects": objects + [{"kind": "plane", "point": [0, 0, -0.5], "normal": [0, 0, 1], "material": MAT("#B0B0B0")}],
        "lights": [{"position": [-3, -2, 6], "color": "#FFF0E0", "intensity": 0.8, "diameter": diameter},
                   {"position": [1, 1, 3.2], "color": "#E0F0FF", "intensity": 0.5, "diameter": 0.6}],
        "scene_settings": {"ambient_illumination": {"color": "#FFFFFF", "intensity": 0.1},
                           "background_color": "#101820"},
    }


@pytest.mark.gpu
def test_cubes_off_the_cone_leave_rays_unwalked(gpu_ctx, tmp_path):
    rng = np.random.default_rng(3)
    objs = []
    for c in _cubes(rng, 20, "1, 1, 1"):  # spheres between cubes: no run of them, each ray that walks tests all
        p = [round(float(v), 4) for v in rng.uniform([-4, -4, 0], [4, 4, 2.5])]
        objs += [c, {"kind": "sphere", "center": p, "radius": 0.2, "material": MAT("#C04040")}]
    st = _count(gpu_ctx, workloads.write_scene(str(tmp_path), "cubes.json", _scene(objs, 1.0)), 161, 93, 16)
    # 20 spheres: each cone tests them once, and fewer than half of the rays
    pairs = st.shadow_rays / 16
    assert 0 < st.work["shadow_spheres"] < 20 * (pairs + st.shadow_rays / 2)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", ["", "1, 1, 1", "3, 0.5, 1", "0.1, 0.1, 0.1", "8, 8, 8", "1, 1, 0.00001", "-2, 1, 1",
                                   "0, 1, 1"])
@pytest.mark.parametrize("diameter", [0.3, 3.0])
def test_transformed_cubes_match_the_oracle(gpu_ctx, tmp_path, scale, diameter):
    import rtrace_b200 as rt
    from tests import oracle_lib
    rng = np.random.default_rng(len(scale) + int(diameter))
    objs = _cubes(rng, 9, scale)
    objs[0]["size"] = [0.0, 0.5, 0.5]
    path = workloads.write_scene(str(tmp_path), "cubes.json", _scene(objs, diameter))
    scene = rt.Scene.from_json_file(path, gpu_ctx)
    r = rt.Renderer(97, 61)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    got = r.render(scene)
    scene.close()
    want = oracle_lib.render(path=path, width=97, height=61, aa="no-jitter")
    assert np.array_equal(got, want), int((got != want).any(2).sum())
