"""The shadow rays a learned render reports: its point lights' once, also for
hits whose disk lights fall back to the plain path."""
import pytest

from rtrace_b200 import denoiser, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("threshold", [1e-30, 0.0, -1.0])  # all fall back, some, none
@pytest.mark.parametrize("points", [0, 1, 2])
def test_shadow_rays_of_a_learned_render(gpu_ctx, points, threshold):
    import json
    import rtrace_b200 as rt
    sc = workloads.ring_spheres_scene(seed=5, n_rings=2, per_ring=6)
    disks = len(sc["lights"])
    assert disks == 2
    sc["lights"] += [{"position": [2.0, -3.0 + k, 7.0], "color": "#FFE0C0", "intensity": 0.4} for k in range(points)]
    scene = rt.Scene.from_json_str(json.dumps(sc), gpu_ctx)
    gpu_ctx.load_denoiser(denoiser.pack_net(denoiser.random_net(11, threshold=0.5)))
    r = rt.Renderer(120, 64)
    r.anti_aliasing_mode = rt.AntiAliasingMode.NoJitter
    r.max_depth = 1
    r.learned_shadows, r.learned_rays, r.fallback_samples, r.confidence_threshold = True, 1, 5, threshold
    r.render(scene)
    st = r.last_stats
    assert st.hits > 0 and (st.fallback_lights > 0) == (threshold >= 0)
    assert st.shadow_rays == st.hits * (points + disks) + st.fallback_lights * 5
    scene.close()
