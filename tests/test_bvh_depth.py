"""The depth of the surface-area trees: a walk keeps a sibling per level, leaf
or not, and its stack is finite, so primitives that shrink towards a point
must not make one level each."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rtrace_b200", "csrc")
LEVELS, STACK = 60, 64

HARNESS = """
#include "bvh_build.hpp"
#include <vector>
// levels of nodes, and each primitive's count in the leaves
extern "C" int levels(int n, const double* mn, const double* mx, double pad, int* seen) {
  std::vector<rtb::BvhNode> nodes;
  std::vector<int32_t> order;
  rtb::build_bvh_sah({mn, mn + 3 * n}, {mx, mx + 3 * n}, 4, pad, &nodes, &order);
  struct At { int node, depth; };
  std::vector<At> st{{0, 1}};
  int deepest = 0;
  while (!st.empty()) {
    const At a = st.back();
    st.pop_back();
    if (a.depth > deepest) deepest = a.depth;
    const rtb::BvhNode& nd = nodes[a.node];
    const int idx[2] = {nd.lidx, nd.ridx}, cnt[2] = {nd.lcnt, nd.rcnt};
    for (int c = 0; c < 2; c++) {
      if (cnt[c] == 0) st.push_back({idx[c], a.depth + 1});
      if (cnt[c] > 4) return -1;
      const double *lo = c ? nd.rmin : nd.lmin, *hi = c ? nd.rmax : nd.lmax;
      for (int j = 0; j < cnt[c]; j++) {
        const int p = order[idx[c] + j];
        seen[p]++;
        for (int k = 0; k < 3; k++)
          if (mn[3 * p + k] < lo[k] || mx[3 * p + k] > hi[k]) return -2;
      }
    }
  }
  return deepest;
}
"""


@pytest.fixture(scope="module")
def levels(tmp_path_factory):
    d = tmp_path_factory.mktemp("bvh")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", str(d / "h.so"),
                    str(d / "h.cpp"), os.path.join(CSRC, "bvh_build.cpp")], check=True)
    L = ctypes.CDLL(str(d / "h.so"))

    def f(tris):
        v = tris.reshape(-1, 3, 3)
        mn, mx = np.ascontiguousarray(v.min(1)), np.ascontiguousarray(v.max(1))
        seen = np.zeros(len(v), np.int32)
        n = L.levels(len(v), mn.ctypes.data_as(ctypes.c_void_p), mx.ctypes.data_as(ctypes.c_void_p),
                     ctypes.c_double(1e-7 * (1.0 + np.abs(v).max())), seen.ctypes.data_as(ctypes.c_void_p))
        assert (seen == 1).all()
        return n
    return f


def comb(n, copies=1):
    """Triangles across the x axis at 2^-k, of that size, `copies` of each:
    walked from -x, the smaller ones come first at every level."""
    s = 2.0 ** -np.arange(n)
    t = np.stack([np.stack([s, -s, -s], 1), np.stack([1.5 * s, s, -s], 1), np.stack([1.25 * s, 0 * s, s], 1)], 1)
    return np.ascontiguousarray(np.repeat(t, copies, 0).reshape(-1, 9))


@pytest.mark.parametrize("n,copies", [(1, 1), (5, 1), (30, 1), (240, 1), (400, 1), (1000, 1), (1000, 5), (300, 40)])
def test_shrinking_triangles_keep_to_the_levels(levels, n, copies):
    assert 0 < levels(comb(n, copies)) <= LEVELS < STACK


@pytest.mark.parametrize("n", [1, 4, 5, 100, 20000])
def test_ordinary_triangles(levels, n):
    rng = np.random.default_rng(n)
    got = levels(rng.random((n, 1, 3)) * 10 + rng.normal(0, 0.1, (n, 3, 3)))
    assert 0 < got <= 1 + 3 * max(1, int(np.ceil(np.log2(n))))


@pytest.mark.gpu
def test_a_comb_of_triangles_is_walked(gpu_ctx):
    import tempfile
    import rtrace_b200 as rt
    from rtrace_b200 import _capi, workloads
    L = _capi.lib()
    v = comb(1000)
    nodes, idx = rt.kd_build(v)
    with tempfile.TemporaryDirectory() as d:
        cube = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32)
        workloads.write_binary_stl(os.path.join(d, "m.stl"), cube, np.array([[0, 1, 2]]))
        mat = workloads._mat("#60A0A0")
        path = workloads.write_scene(d, "s.json", {
            "camera": {"kind": "perspective", "position": [-4, 0.1, 0.1], "target": [0, 0, 0], "up": [0, 0, 1], "fov": 30,
                       "width": 16, "height": 9},
            "objects": [{"kind": "mesh", "filename": "m.stl", "material": mat},
                        {"kind": "plane", "point": [3, 0, 0], "normal": [-1, 0, 0], "material": mat}],
            "lights": [{"position": [-6, 1, 1], "color": "#FFFFFF", "intensity": 1.0, "diameter": 0.5}],
            "scene_settings": {"ambient_illumination": {"color": "#FFFFFF", "intensity": 0.1},
                               "background_color": "#000000"}})
        host = rt.HostScene.from_json_file(path)
    md = L.rt_host_scene_desc(host.handle).contents.meshes[0]
    old = {f: getattr(md, f) for f in ("vertices", "n_triangles", "nodes", "n_nodes", "tri_index", "n_tri_index")}
    md.vertices, md.n_triangles = v.ctypes.data, len(v)
    md.nodes, md.n_nodes = nodes.ctypes.data, len(nodes)
    md.tri_index, md.n_tri_index = idx.ctypes.data, len(idx)
    for k in range(3):
        md.bounds_min[k], md.bounds_max[k] = v.reshape(-1, 3)[:, k].min(), v.reshape(-1, 3)[:, k].max()
    scene = rt.Scene.upload(host, gpu_ctx)
    for f, x in old.items():
        setattr(md, f, x)
    # rays along the axis, close enough to it to meet the boxes of all levels
    rng = np.random.default_rng(3)
    rays = np.zeros((256, 6))
    rays[:, 0], rays[:, 3] = -1.0, 1.0
    rays[:, 1:3] = rng.uniform(-1, 1, (256, 2)) * 10.0 ** -rng.uniform(1, 12, (256, 1))
    want = np.zeros((len(rays), 8))
    for mode in (1, 0, 2):
        out = np.zeros((len(rays), 8))
        st = L.rt_debug_mesh_hit(gpu_ctx.handle, scene._handle, 0, 1 | (mode << 1), rays.ctypes.data, len(rays), 0.001,
                                 float("inf"), out.ctypes.data)
        assert st == 0, L.rt_last_error(gpu_ctx.handle)
        if mode == 1:
            want = out
            assert want[:, 0].all()
        elif mode == 0:
            assert np.array_equal(out, want)
        else:
            assert np.array_equal(out[:, 0], want[:, 0])
    img = rt.Renderer(64, 36).render(scene)
    assert img.any()
    scene.close()
    host.close()
