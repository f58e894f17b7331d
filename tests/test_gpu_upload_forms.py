"""Scenes whose BLASes are built and kept on the GPU against the same scenes prepared on the host: hit
records, visit counts and renders are the same bytes (triangle order, wide records, pdfs and light
tables included)."""
import numpy as np
import pytest

from barnacle_gb300 import BarnacleError, Bundle, capi

pytestmark = pytest.mark.gpu


def rays(n, lo, hi, seed=3):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, capi.RAY_DTYPE)
    r["origin"] = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    r["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True).astype(np.float32)
    r["t_max"] = np.inf
    return r


def state(ctx, b, builder, width):
    s = b.scene.contents
    s.bvh_builder, s.bvh_width = builder, width
    ctx.upload(b)
    box = ([-60, 0, -60], [60, 25, 60]) if s.n_instances > 100 else ([0.05] * 3, [0.95] * 3)
    q = rays(5000, *box)
    ctx.reset_stats()
    out = [ctx.instance_order(s.n_instances).tobytes(), ctx.trace(q).tobytes(), ctx.trace(q, capi.BN_TRACE_COUNT).tobytes()]
    st = ctx.stats()
    out += [st.nodes_visited, st.tris_tested, st.instances_visited]
    r = b.render
    r.mode, r.spp = capi.BN_MODE_MEGAKERNEL, 2
    v = b.views[0]
    v.width, v.height = 61, 47
    out.append(ctx.render(r, [v])[0].tobytes())
    return out


@pytest.mark.parametrize("name", ["cornell", "cornell-objects", "materials", "instances"])
@pytest.mark.parametrize("width", [capi.BN_BVH_AUTO, capi.BN_BVH_BINARY, capi.BN_BVH_WIDE])
def test_device_scene_equals_host_scene(ctx, name, width):
    b = Bundle.generate(name, 2)
    host = state(ctx, b, capi.BN_BUILDER_HOST, width)
    assert state(ctx, b, capi.BN_BUILDER_DEVICE, width) == host
    assert state(ctx, b, capi.BN_BUILDER_AUTO, width) == host
    assert state(ctx, b, capi.BN_BUILDER_HOST, width) == host  # after the larger buffers


def test_large_emitter_and_bad_values(ctx):
    """A mesh built on the GPU that emits (its triangles come back for the light table), one whose
    vertices hold a NaN (the host builder's tree), and an index out of range."""
    b = Bundle.generate("cornell-objects", 2)
    s = b.scene.contents
    big = next(i for i in range(s.n_instances) if s.meshes[s.primitives[s.instances[i].primitive].mesh].n_triangles > 50000)
    s.instances[big].light = 0
    host = state(ctx, b, capi.BN_BUILDER_HOST, capi.BN_BVH_AUTO)
    assert state(ctx, b, capi.BN_BUILDER_DEVICE, capi.BN_BVH_AUTO) == host
    s.instances[big].light = -1
    mesh = s.meshes[s.primitives[s.instances[big].primitive].mesh]
    kept = mesh.vertices[mesh.indices[0] * 3]
    mesh.vertices[mesh.indices[0] * 3] = float("nan")
    try:
        host = state(ctx, b, capi.BN_BUILDER_HOST, capi.BN_BVH_BINARY)
    except BarnacleError:
        with pytest.raises(BarnacleError):
            state(ctx, b, capi.BN_BUILDER_DEVICE, capi.BN_BVH_BINARY)
    else:
        assert state(ctx, b, capi.BN_BUILDER_DEVICE, capi.BN_BVH_BINARY) == host
    mesh.vertices[mesh.indices[0] * 3] = kept
    index = mesh.indices[5]
    for bad in (-1, mesh.n_vertices):
        mesh.indices[5] = bad
        with pytest.raises(BarnacleError):
            ctx.upload(b)
    mesh.indices[5] = index
    assert state(ctx, b, capi.BN_BUILDER_AUTO, capi.BN_BVH_AUTO)
