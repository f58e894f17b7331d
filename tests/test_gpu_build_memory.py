"""The builder's work buffers (230 bytes per box) above 256 MB go back when the call ends, also when it ends
in an error: a leaf of over 127 boxes at the depth cap (an infinite box), and a scene without lights."""
import ctypes as C

import numpy as np
import pytest

from barnacle_gb300 import BarnacleError, Context, capi

pytestmark = pytest.mark.gpu
N = 3_000_000  # 690 MB of work buffers


def free_bytes():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info(0)[0]


def test_a_refused_tree_keeps_no_large_buffers():
    with Context(0) as c:
        rng = np.random.default_rng(1)
        lo = rng.uniform(-50, 50, (N, 3)).astype(np.float32)
        b = np.concatenate([lo, lo + np.float32(0.1)], 1)
        b[N // 2, 3] = np.inf
        c.bvh_build(np.ascontiguousarray(b[:300][b[:300, 3] < 1e9]))
        before = free_bytes()
        with pytest.raises(BarnacleError, match="127"):
            c.bvh_build(b)
        assert before - free_bytes() < 300 << 20


def test_a_refused_scene_keeps_no_large_buffers():
    with Context(0) as c:
        rng = np.random.default_rng(2)
        v = rng.uniform(-50, 50, (N, 3)).astype(np.float32)
        idx = np.stack([np.arange(N), (np.arange(N) + 1) % N, (np.arange(N) + 2) % N], 1).astype(np.int32)
        mesh = capi.bn_mesh_desc(v.ctypes.data_as(C.POINTER(C.c_float)), idx.ctypes.data_as(C.POINTER(C.c_int32)), None, N, N)
        prim = capi.bn_primitive_desc(capi.BN_PRIM_MESH, 0, 0.0)
        mat = capi.bn_material_desc(capi.BN_MAT_LAMBERTIAN)
        inst = capi.bn_instance_desc(0, 0, -1)
        inst.object_to_world[:] = inst.world_to_object[:] = np.eye(4, dtype=np.float32).reshape(16)
        s = capi.bn_scene_desc()
        s.primitives, s.n_primitives = C.pointer(prim), 1
        s.meshes, s.n_meshes = C.pointer(mesh), 1
        s.instances, s.n_instances = C.pointer(inst), 1
        s.materials, s.n_materials = C.pointer(mat), 1
        before = free_bytes()
        with pytest.raises(BarnacleError, match="No light"):
            c.upload(C.pointer(s))
        # what stays is the scene's own: 48 + 4 bytes a triangle, 0.8 nodes of 32, records of 128 for a third
        # of the nodes
        assert before - free_bytes() < (N * 52 + N * 26 + N * 40) + (300 << 20)
