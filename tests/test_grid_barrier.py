"""The barrier between the stages of the queue levels that share one launch:
it waits for as long as the stage makes progress, and gives up, with an
error and a usable context, when nothing moves."""
import numpy as np
import pytest

from rtrace_b200 import workloads

MAT = workloads._mat


def _scene():
    """Two facing mirrors, so that every level has all of its rays, and 1,000
    cubes that every shadow ray tests one by one: too flat for the light cones
    to leave them out."""
    objs = [{"kind": "plane", "point": [0, 0, z], "normal": [0, 0, n], "material": MAT("#909090", reflectivity=0.6)}
            for z, n in ((-1, 1), (1, -1))]
    for k in range(1000):
        objs.append({"kind": "cube", "center": [-50 - k % 10, k // 100, (k // 10) % 10 * 0.1], "size": [0.05, 0.05, 0.05],
                     "transform": ["scale(1, 1, 0.0000001)"], "material": MAT("#4040C0")})
    return {"camera": {"kind": "perspective", "position": [0, -8, 0], "target": [0, 0, 0.3], "up": [0, 0, 1], "fov": 50,
                       "width": 16, "height": 9},
            "objects": objs,
            "lights": [{"position": [-2, 1, 0.2], "color": "#FFFFFF", "intensity": 0.8, "diameter": 0.5},
                       {"position": [2, 1, -0.2], "color": "#FFF0E0", "intensity": 0.5, "diameter": 0.4}],
            "scene_settings": {"ambient_illumination": {"color": "#FFFFFF", "intensity": 0.1},
                               "background_color": "#101820"}}


def _limit(ctx, ns):
    from rtrace_b200 import _capi
    assert _capi.lib().rt_debug_set_barrier_limit(ctx.handle, ns) == 0


@pytest.mark.gpu
def test_waits_end_with_the_work_not_with_the_time(tmp_path):
    import rtrace_b200 as rt
    from rtrace_b200 import _capi
    ctx = rt.Context(0)
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", _scene()), ctx)
    r = rt.Renderer(16, 12)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    r.max_depth, r.disk_samples = 4, 4096
    r.flags = _capi.RT_FLAG_STAGE_TIMES  # every stage in its own launch
    want = r.render(scene)
    r.flags = 0
    # 384 lights of a level keep a sixth of the launch's warps at work on 128
    # rounds of samples each; the others wait all that time
    limit_ms = 1.0
    _limit(ctx, int(limit_ms * 1e6))
    for flags in (0, _capi.RT_FLAG_CUDA_GRAPH, _capi.RT_FLAG_CUDA_GRAPH):
        r.flags = flags
        assert np.array_equal(r.render(scene), want)
    assert r.last_stats.device_ms > 4 * 3 * limit_ms
    scene.close()


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_an_error(tmp_path):
    import rtrace_b200 as rt
    ctx = rt.Context(0)
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", _scene()), ctx)
    r = rt.Renderer(64, 48)
    r.max_depth = 5
    want = r.render(scene)
    for _ in range(3):
        _limit(ctx, 1)
        with pytest.raises(rt.RtraceError, match="grid barrier"):
            r.render(scene)
        _limit(ctx, 0)
        assert np.array_equal(r.render(scene), want)
    scene.close()


# contexts on threads of their own, whose launches each want the whole device
@pytest.mark.gpu
def test_contexts_on_threads_share_the_device(tmp_path):
    import threading
    import rtrace_b200 as rt
    s = _scene()
    s["objects"] = s["objects"][:40]
    path = workloads.write_scene(str(tmp_path), "s.json", s)
    r = rt.Renderer(160, 120)
    r.max_depth = 6
    want = r.render(rt.Scene.from_json_file(path, rt.Context(0)))
    right = []

    def work():
        ctx = rt.Context(0)
        scene = rt.Scene.from_json_file(path, ctx)
        mine = rt.Renderer(160, 120)
        mine.max_depth = 6
        for _ in range(25):
            right.append(np.array_equal(mine.render(scene), want))
        scene.close()
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(right) == 100 and all(right)
