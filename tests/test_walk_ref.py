"""A walk's references to BVH children (walk_ref, dmath.cuh): leaves are told
from nodes and read back whole up to the largest mesh an upload accepts."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rtrace_b200", "csrc")
MAX_PRIMS = 1 << 29


@pytest.fixture(scope="module")
def ref(tmp_path_factory):
    from rtrace_b200.build import _nvcc
    d = tmp_path_factory.mktemp("walk_ref")
    (d / "r.cu").write_text(
        '#include "dmath.cuh"\nextern "C" {\nint ref(int i, int c) { return rtb::walk_ref(i, c); }\n'
        "int first(int r) { return rtb::leaf_first(r); }\nint count(int r) { return rtb::leaf_count(r); }\n"
        "int done() { return RTB_WALK_DONE; }\nint leaf() { return RTB_LEAF; }\nint most() { return RTB_MAX_PRIMS; }\n}\n")
    subprocess.run([_nvcc(), "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-I", CSRC,
                    "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(d / "r.so"), str(d / "r.cu")], check=True)
    return ctypes.CDLL(str(d / "r.so"))


@pytest.mark.parametrize("idx", [0, 1, 15, (1 << 25) - 1, (1 << 27) - 1, 1 << 27, (1 << 28) + 5, MAX_PRIMS - 4, MAX_PRIMS - 1])
def test_leaves_and_nodes_read_back(ref, idx):
    assert ref.leaf() == 4 and ref.most() == MAX_PRIMS
    for cnt in range(1, ref.leaf() + 1):
        r = ref.ref(idx, cnt)
        assert r < 0 and ref.first(r) == idx and ref.count(r) == cnt
    assert ref.ref(idx, 0) == idx != ref.done()


@pytest.mark.gpu
def test_larger_meshes_are_refused(gpu_ctx):
    from rtrace_b200 import _capi
    v = (ctypes.c_double * 9)()
    d = _capi.rt_mesh_desc()
    d.vertices, d.n_triangles = ctypes.addressof(v), MAX_PRIMS + 1
    mask = ctypes.c_uint32()
    L = _capi.lib()
    assert L.rt_debug_mesh_prep(gpu_ctx.handle, ctypes.byref(d), ctypes.byref(mask)) != 0
    assert b"2^29" in L.rt_last_error(gpu_ctx.handle)
