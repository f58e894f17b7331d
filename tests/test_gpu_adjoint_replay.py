"""The adjoint from recorded vertices against the one that traces its paths again.

Sampling at the parameters that are rendered, given as sampling_params, takes the two-material route
(trace, replay by tracing); the same call without them takes the patched scene's route (path machine
below 1 M paths, wavefront queues from there on, replay from records).  The images are the same floats.
The gradients are the same terms in FP32 sums of at most 32 of them, each off by at most 32 eps of the
terms' magnitudes (2e-6), added in FP64: 1e-5 of the largest entry of the kind bounds the difference."""
import numpy as np
import pytest

from barnacle_gb300 import Bundle, capi
from barnacle_gb300.inverse import MaterialProblem

pytestmark = pytest.mark.gpu


def same_gradients(g, ref):
    g, ref = g.reshape(-1, 6), ref.reshape(-1, 6)
    for kind in (slice(0, 3), slice(3, 4), slice(4, 5), slice(5, 6)):
        assert np.abs(g[:, kind] - ref[:, kind]).max() <= 1e-5 * np.abs(ref[:, kind]).max()


@pytest.mark.parametrize("bvh", [capi.BN_BVH_WIDE, capi.BN_BVH_BINARY])
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 8), (33, 7, 1, 1), (64, 48, 5, 8), (257, 255, 16, 3), (256, 256, 16, 8)])
def test_replay_equals_traced_adjoint(ctx, bvh, w, h, spp, depth):
    b = Bundle.generate("materials", 1)
    b.scene.contents.bvh_width = bvh
    pb = MaterialProblem(ctx, b, width=w, height=h, spp=spp, max_depth=depth)
    rng = np.random.default_rng(w)
    theta = pb.random_params(5)
    img = pb.render(theta, frame=4)
    ref = pb.render(theta, frame=4, sampling_params=theta)
    np.testing.assert_array_equal(img.view(np.uint32), ref.view(np.uint32))
    target = rng.uniform(0, 1, img.shape).astype(np.float32)
    loss, g = pb.loss_and_grad(theta, target, frame=4)
    loss_ref, g_ref = pb.loss_and_grad(theta, target, frame=4, sampling_params=theta)
    assert np.isfinite(g_ref).all()
    assert abs(loss - loss_ref) <= 1e-12 * abs(loss_ref)
    same_gradients(g, g_ref)


def test_zero_scale_and_non_finite_parameters_keep_their_derivatives(ctx):
    """A light scaled to zero still has a derivative, and a NaN parameter gives what it gave: both
    are left to the two-material route."""
    b = Bundle.generate("materials", 1)
    pb = MaterialProblem(ctx, b, width=48, height=48, spp=4)
    theta = pb.random_params(5)
    theta.reshape(-1, 6)[pb.emissive_base, 5] = 0.0
    target = np.zeros((48, 48, 3), np.float32)
    _, g = pb.loss_and_grad(theta, target, frame=4)
    _, ref = pb.loss_and_grad(theta, target, frame=4, sampling_params=theta)
    assert ref.reshape(-1, 6)[pb.emissive_base, 5] != 0
    same_gradients(g, ref)
    theta.reshape(-1, 6)[0, 0] = np.nan
    a, b2 = pb.render(theta, frame=4), pb.render(theta, frame=4, sampling_params=theta)
    np.testing.assert_array_equal(a, b2)
