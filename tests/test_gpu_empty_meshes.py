"""Meshes without triangles and empty leaves: a wide walk has no code for them, so they must not be
entered.  The instance's matrix is dense and positive, which makes its world box [-inf, -inf] (other
matrices make it NaN, which no ray passes): a ray with negative directions and no end passes it."""
import ctypes as C

import numpy as np
import pytest

from barnacle_gb300 import Bundle, capi, mat4_invert

pytestmark = pytest.mark.gpu
DENSE = np.array([[2, 1, 1, 0], [1, 2, 1, 0], [1, 1, 2, 0], [0, 0, 0, 1]], np.float32)


def with_empty(b, keep):
    """The bundle's scene with the instances `keep` of its own and one of an empty mesh."""
    s = capi.bn_scene_desc()
    C.memmove(C.byref(s), b.scene, C.sizeof(s))
    meshes = (capi.bn_mesh_desc * (s.n_meshes + 1))(*[s.meshes[i] for i in range(s.n_meshes)], capi.bn_mesh_desc())
    prims = (capi.bn_primitive_desc * (s.n_primitives + 1))(*[s.primitives[i] for i in range(s.n_primitives)],
                                                            capi.bn_primitive_desc(capi.BN_PRIM_MESH, s.n_meshes, 0.0))
    empty = capi.bn_instance_desc(s.n_primitives, 0, -1)
    empty.object_to_world[:] = DENSE.reshape(16)
    empty.world_to_object[:] = mat4_invert(DENSE)
    inst = [s.instances[i] for i in keep]
    insts = (capi.bn_instance_desc * (len(inst) + 1))(*inst, empty)
    s.meshes, s.primitives, s.instances = meshes, prims, insts
    s.n_meshes, s.n_primitives, s.n_instances = s.n_meshes + 1, s.n_primitives + 1, len(inst) + 1
    return s, (meshes, prims, insts)


def rays():
    rng = np.random.default_rng(1)
    r = np.zeros(6000, capi.RAY_DTYPE)
    r["origin"] = rng.uniform(0.05, 0.95, (6000, 3))
    d = rng.normal(size=(6000, 3))
    d[:3000] = -np.abs(d[:3000])
    r["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r["t_max"] = np.inf
    return r


@pytest.mark.parametrize("keep", [[7], [7, 0, 1], list(range(8))])  # a TLAS of one leaf, and a chain of empty ones
@pytest.mark.parametrize("builder", [capi.BN_BUILDER_HOST, capi.BN_BUILDER_DEVICE])
def test_an_empty_mesh_is_never_entered(ctx, keep, builder):
    b = Bundle.generate("cornell", 1)
    q = rays()
    s, _arrays = with_empty(b, keep)
    s.bvh_builder = builder
    got = {}
    for width in (capi.BN_BVH_BINARY, capi.BN_BVH_WIDE):
        s.bvh_width = width
        ctx.upload(C.pointer(s))
        order = ctx.instance_order(s.n_instances)
        for flags in (0, capi.BN_TRACE_WATERTIGHT, capi.BN_TRACE_ANY, capi.BN_TRACE_COUNT):
            for n in (64, 6000):  # persistent lanes, a thread per ray
                h = ctx.trace(q[:n], flags)
                assert not (order[h["instance"][h["instance"] >= 0]] == len(keep)).any()
                got.setdefault((flags, n), []).append(h.tobytes())
        r, v = b.render, b.views[0]
        v.width, v.height, r.spp = 40, 30, 2
        for mode in (capi.BN_MODE_MEGAKERNEL, capi.BN_MODE_WAVEFRONT):
            r.mode = mode
            got.setdefault(("film", mode), []).append(np.round(ctx.render(r, [v])[0], 4).tobytes())
    for key, (binary, wide) in got.items():
        assert binary == wide, key
