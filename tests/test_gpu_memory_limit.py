"""Renders and gradients whose path state does not fit (bn_set_memory_limit): the same results from fewer
slots or from the one kernel, or BN_ERR_OUT_OF_MEMORY where the caller chose the slots; and the calls
after them, of the sizes that fitted before, have their memory again."""
import numpy as np
import pytest

from barnacle_gb300 import Bundle, Context, capi
from barnacle_gb300.capi import BarnacleError
from barnacle_gb300.inverse import MaterialProblem

pytestmark = pytest.mark.gpu
SLOT, PATH = 240, 16  # bytes


@pytest.fixture
def c():
    with Context(0) as ctx:
        yield ctx


def limit(c, n):
    assert c.lib.bn_set_memory_limit(c._h, n) == capi.BN_OK, c.error()


def render(c, b, mode, size, spp, slots=0):
    r, v = b.render, b.views[0]
    r.mode, r.spp, r.queue_capacity = mode, spp, slots
    v.width, v.height = size
    return c.render(r, [v])[0].copy()


def test_megakernel_mode_falls_back_to_one_kernel_and_recovers(c):
    b = Bundle.generate("cornell-objects", 1)
    c.upload(b)
    small, large = ((1024, 513), 2), ((1024, 1025), 2)
    want = [render(c, b, capi.BN_MODE_MEGAKERNEL, *s) for s in (small, large)]
    for n in (1, (1024 * 513 * 2) * (SLOT + PATH), 0):
        limit(c, n)  # neither fits, the small one does, both do
        for s, w in [(small, want[0]), (large, want[1]), (small, want[0])]:
            np.testing.assert_array_equal(render(c, b, capi.BN_MODE_MEGAKERNEL, *s).view(np.uint32), w.view(np.uint32))


def test_wavefront_mode_halves_its_slots_and_recovers(c):
    b = Bundle.generate("cornell", 1)
    c.upload(b)
    size, spp = (1024, 1024), 4  # 4 M paths
    want = render(c, b, capi.BN_MODE_MEGAKERNEL, size, spp)
    for slots in (1 << 20, 1 << 21):
        limit(c, slots * SLOT)
        render(c, b, capi.BN_MODE_WAVEFRONT, (1024, slots // 4096), spp)  # holds exactly the slots halved to
        np.testing.assert_allclose(render(c, b, capi.BN_MODE_WAVEFRONT, size, spp), want, rtol=2e-5, atol=1e-6)
    limit(c, 1000 * SLOT)
    for slots in (0, 4096):
        with pytest.raises(BarnacleError) as e:
            render(c, b, capi.BN_MODE_WAVEFRONT, size, spp, slots)
        assert e.value.code == capi.BN_ERR_OUT_OF_MEMORY
    limit(c, 0)
    for slots in (4096 * 16, 0):
        np.testing.assert_allclose(render(c, b, capi.BN_MODE_WAVEFRONT, size, spp, slots), want, rtol=2e-5, atol=1e-6)


def test_pssmlt_chains_without_memory_report_it(c):
    b = Bundle.generate("pssmlt", 1)
    c.upload(b)
    r, v = b.render, b.views[0]
    v.width = v.height = 64
    r.mode, r.spp, r.n_bootstrap, r.n_chains = capi.BN_MODE_WAVEFRONT, 2, 4096, 2048
    limit(c, 2047 * SLOT)
    with pytest.raises(BarnacleError) as e:
        c.render(r, [v])
    assert e.value.code == capi.BN_ERR_OUT_OF_MEMORY
    limit(c, 2048 * SLOT)
    c.reset_stats()
    c.render(r, [v])
    accepted = c.stats().accepted
    r.mode = capi.BN_MODE_MEGAKERNEL
    c.reset_stats()
    c.render(r, [v])
    assert c.stats().accepted == accepted > 0


def test_adjoint_paths_fall_back_to_one_kernel_and_recover(c):
    """Images bit for bit; gradients are the same FP32 sums added in FP64 in another order: at most 2^20
    additions, each off by 2^-53 of terms that may be 2^8 times their sum."""
    pb = MaterialProblem(c, Bundle.generate("materials", 1), width=256, height=256, spp=16)
    theta = pb.random_params(5)
    target = np.zeros((256, 256, 3), np.float32)
    img = pb.render(theta, frame=4).copy()
    loss, g = pb.loss_and_grad(theta, target, frame=4)
    for n in (1, 0):
        limit(c, n)
        np.testing.assert_array_equal(pb.render(theta, frame=4).view(np.uint32), img.view(np.uint32))
        loss2, g2 = pb.loss_and_grad(theta, target, frame=4)
        assert abs(loss2 - loss) <= 1e-12 * loss
        assert np.abs(g2 - g).max() <= 2.0 ** (20 - 53 + 8) * np.abs(g).max()
