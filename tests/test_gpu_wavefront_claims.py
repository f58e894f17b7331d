"""The last claims of a wavefront render: path counts at and beside whole rows (32), whole claims (128) and
whole pools, in pools that are filled several times, with other warps claiming at the same moment.  Every
path must be run once: the image is the megakernel mode's, and so is the count."""
import numpy as np
import pytest

from barnacle_gb300 import Bundle, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, capi.BN_RENDER_NO_GRAPH])
@pytest.mark.parametrize("paths,pool", [(1025, 1024), (1055, 1024), (1057, 1024), (1151, 1024), (1153, 1024), (4095, 1024),
                                        (4097, 1024), (100003, 1024), (100003, 33333), (99999, 50000)])
def test_every_path_is_claimed_once(ctx, paths, pool, flags):
    b = Bundle.generate("cornell", 1)
    ctx.upload(b)
    v, r = b.views[0], b.render
    v.width, v.height = paths, 1
    r.spp, r.mode = 1, capi.BN_MODE_MEGAKERNEL
    want = ctx.render(r, [v])[0].copy()
    r.mode, r.queue_capacity, r.flags = capi.BN_MODE_WAVEFRONT, pool, flags
    ctx.reset_stats()
    got = ctx.render(r, [v])[0]
    assert ctx.stats().paths == paths
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))  # one path per pixel: no sums
