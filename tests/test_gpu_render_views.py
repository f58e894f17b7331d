"""Megakernel-mode renders of several views with several samples per pixel on both sides of 786,432 paths,
where the path machine hands over to the wavefront's queues: one image, that of the counting plain loop."""
import numpy as np
import pytest

from barnacle_gb300 import Bundle, capi

pytestmark = pytest.mark.gpu
QUEUE_PATHS = 3 << 18


@pytest.mark.parametrize("flags", [0, capi.BN_RENDER_WATERTIGHT, capi.BN_RENDER_CULL_SHADOW])
@pytest.mark.parametrize("spp,queues", [(2, False), (6, False), (7, True)])
def test_many_views_give_one_image_in_every_form(ctx, flags, spp, queues):
    b = Bundle.generate("instances", 1)
    ctx.upload(b)
    views = b.views[:5]
    for k, v in enumerate(views):
        v.width, v.height = 230 - 7 * k, 100 + 9 * k
    paths = sum(v.width * v.height for v in views) * spp
    assert (paths >= QUEUE_PATHS) == queues and paths > 200_000
    r = b.render
    r.mode, r.spp, r.flags, r.frame_id = capi.BN_MODE_MEGAKERNEL, spp, flags, 3
    got = [g.copy() for g in ctx.render(r, views)]
    r.flags = flags | capi.BN_RENDER_COUNT
    for g, w in zip(got, ctx.render(r, views)):
        np.testing.assert_array_equal(g.view(np.uint32), w.view(np.uint32))
