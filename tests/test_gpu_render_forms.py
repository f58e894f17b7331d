"""The forms a megakernel-mode render takes (the path machine, the plain loop for short renders of
simple scenes, the wavefront's queues with sums in this mode's order) give one image, bit for bit:
the counting render, which always runs the plain loop in the reference's order, is the measure."""
import ctypes as C

import numpy as np
import pytest

from barnacle_gb300 import Bundle, capi

pytestmark = pytest.mark.gpu


def both(ctx, b, views, spp, flags=0, **desc):
    r = b.render
    r.mode, r.spp, r.flags, r.frame_id = capi.BN_MODE_MEGAKERNEL, spp, flags, 3
    for k, x in desc.items():
        setattr(r, k, x)
    got = ctx.render(r, views)
    r.flags = flags | capi.BN_RENDER_COUNT
    want = ctx.render(r, views)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.view(np.uint32), w.view(np.uint32))
    return got


# 1 path, one path per lane and fewer lanes than a warp, the plain loop's band and its ends, the
# wavefront's first size and one whose paths end inside a chunk (spp not a multiple of spc)
@pytest.mark.parametrize("name", ["cornell", "cornell-objects", "materials"])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (33, 31, 1), (128, 64, 1), (91, 90, 1), (256, 256, 2), (257, 255, 3),
                                     (256, 256, 16), (241, 239, 19)])
def test_forms_give_one_image(ctx, name, w, h, spp):
    b = Bundle.generate(name, 1)
    ctx.upload(b)
    v = b.views[0]
    v.width, v.height = w, h
    img = both(ctx, b, [v], spp)[0]
    assert np.isfinite(img).mean() > 0.99


@pytest.mark.parametrize("flags", [0, capi.BN_RENDER_WATERTIGHT, capi.BN_RENDER_CULL_SHADOW])
@pytest.mark.parametrize("spp", [1, 9])
def test_forms_give_one_image_of_many_views(ctx, flags, spp):
    b = Bundle.generate("instances", 1)
    ctx.upload(b)
    views = b.views[:5]
    for k, v in enumerate(views):  # 105,800 and 952,200 paths below, 1,057,300 paths with the last size
        v.width, v.height = 230 - 7 * k, 100 + 9 * k
    if spp == 9:
        views[4].width = 292
    both(ctx, b, views, spp, flags)


@pytest.mark.parametrize("width,bvh", [(64, capi.BN_BVH_WIDE), (400, capi.BN_BVH_BINARY)])
def test_forms_agree_on_depths_and_walks(ctx, width, bvh):
    b = Bundle.generate("cornell-objects", 1)
    b.scene.contents.bvh_width = bvh
    ctx.upload(b)
    v = b.views[0]
    v.width, v.height = width, 263
    for depth, rr in ((0, 0), (1, 0), (2, 1), (5, 0)):
        both(ctx, b, [v], 10, max_depth=depth, rr_depth=rr)


@pytest.mark.parametrize("name", ["cornell", "materials"])
@pytest.mark.parametrize("w,h,spp", [(4369, 6, 30), (512, 512, 3), (617, 425, 3)])
def test_forms_agree_at_the_queues_line(ctx, name, w, h, spp):
    """786,420, 786,432 and 786,675 paths: the last on the path machine, the first in the queues."""
    b = Bundle.generate(name, 1)
    ctx.upload(b)
    v = b.views[0]
    v.width, v.height = w, h
    both(ctx, b, [v], spp)


def test_wavefront_limits_leave_megakernel_renders_alone(ctx):
    """bn_set_limits' iteration cap is the wavefront mode's; the stack cap is every walk's."""
    b = Bundle.generate("cornell", 1)
    ctx.upload(b)
    try:
        assert ctx.lib.bn_set_limits(ctx._h, 0, 3) == capi.BN_OK
        both(ctx, b, b.views, 17)
        assert ctx.lib.bn_set_limits(ctx._h, 1, 0) == capi.BN_OK
        r = b.render
        r.spp = 17
        out = np.zeros(256 * 256 * 3, np.float32)
        assert ctx.lib.bn_render(ctx._h, C.byref(r), b.views_array(), 1, capi.ptr(out)) == capi.BN_ERR_DEVICE
    finally:
        ctx.lib.bn_set_limits(ctx._h, 0, 0)
