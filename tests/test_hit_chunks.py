"""Frames whose hits are shaded in chunks, and scenes of more lights than the
lit ones are paired for."""
import numpy as np
import pytest

from rtrace_b200 import workloads

from .test_light_cones import _compare, _scene


def _chunk(ctx, pairs):
    from rtrace_b200 import _capi
    assert _capi.lib().rt_debug_set_chunk_pairs(ctx.handle, pairs) == 0


# chunks of one hit (three lights), of a part of a block, of whole blocks with
# and without a remainder
@pytest.mark.gpu
@pytest.mark.parametrize("pairs", [1, 3 * 100, 3 * 128, 3 * 1000, 3 * 4000])
def test_chunks_match_one_pass(tmp_path, pairs):
    import rtrace_b200 as rt
    from rtrace_b200 import _capi
    ctx = rt.Context(0)
    w, h = (16, 9) if pairs == 1 else (97, 55)
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", _scene(str(tmp_path), 1.0)), ctx)
    for aa, samples in ((rt.AntiAliasingMode.NoJitter, 1), (rt.AntiAliasingMode.Stochastic, 2), (rt.AntiAliasingMode.Quincunx, 1)):
        r = rt.Renderer(w, h)
        r.anti_aliasing_mode, r.samples, r.max_depth, r.disk_samples = aa, samples, 4, 6
        want, st = r.render(scene), r.last_stats
        _chunk(ctx, pairs)
        for flags in (0, _capi.RT_FLAG_CUDA_GRAPH, _capi.RT_FLAG_CUDA_GRAPH, _capi.RT_FLAG_COUNT_WORK):
            r.flags = flags
            assert np.array_equal(r.render(scene), want), (aa, flags)
            assert r.last_stats.kernel_launches > st.kernel_launches
            assert (r.last_stats.hits, r.last_stats.shadow_rays) == (st.hits, st.shadow_rays)
        _chunk(ctx, 0)
    scene.close()


# hits of a scene without lights, whose records are held all the same
@pytest.mark.gpu
def test_chunks_without_lights(tmp_path):
    import rtrace_b200 as rt
    ctx = rt.Context(0)
    s = _scene(str(tmp_path), 1.0)
    s["lights"] = []
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", s), ctx)
    r = rt.Renderer(97, 55)
    r.max_depth = 3
    want, st = r.render(scene), r.last_stats
    _chunk(ctx, 1000)
    assert np.array_equal(r.render(scene), want)
    assert r.last_stats.kernel_launches > st.kernel_launches
    scene.close()


# the visibility of a chunked level 0
@pytest.mark.gpu
def test_chunked_shadow_aov(tmp_path):
    import torch
    import rtrace_b200 as rt
    ctx = rt.Context(0)
    scene = rt.Scene.from_json_file(workloads.write_scene(str(tmp_path), "s.json", _scene(str(tmp_path), 1.0)), ctx)
    r = rt.Renderer(97, 55)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    got = []
    for pairs in (0, 3 * 700):
        _chunk(ctx, pairs)
        vis = torch.zeros((1, 2, 55, 97), device="cuda")
        feat = torch.zeros((1, 55, 97, 16), dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        img = r.render_shadow_aov(scene, vis.data_ptr(), feat.data_ptr())
        hit = feat[..., 0] == 1  # the planes are written where a ray hit
        got.append((img, vis[hit.unsqueeze(1).expand_as(vis)], feat))
    assert np.array_equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][2], got[1][2])
    scene.close()


# 32 lights are paired from a mask, more are queued one by one; few hits take
# a thread per light, many one per hit
@pytest.mark.gpu
@pytest.mark.parametrize("lights", [31, 32, 33, 70])
@pytest.mark.parametrize("w,h", [(24, 14), (120, 70)])
def test_many_lights_match_the_oracle(gpu_ctx, oracle, tmp_path, lights, w, h):
    s = _scene(str(tmp_path), 1.0, scene=5)
    s["lights"] = []
    for k in range(lights):
        light = {"position": [round(5 * float(np.cos(k)), 4), round(5 * float(np.sin(k)), 4), 4.0 + k % 5], "color": "#FFFFFF",
                 "intensity": round(1.5 / lights, 5)}
        if k % 4:
            light["diameter"] = (1.0, 1.0, 0.6)[k % 3]
        s["lights"].append(light)
    _compare(gpu_ctx, workloads.write_scene(str(tmp_path), "s.json", s), w, h, 2)
