"""Where the replayed adjoint's terms meet: a vertex's light-sample and BSDF-sample terms are added in FP64,
as the two-material form's atomics add them.  One path of two vertices in different material slots: the
first one's row is the sum of two FP32 numbers, which mostly is no FP32 number; added in FP32 it always
would be."""
import numpy as np
import pytest

from barnacle_gb300 import Bundle
from barnacle_gb300.inverse import MaterialProblem

pytestmark = pytest.mark.gpu


def test_terms_of_one_vertex_are_added_in_64_bits(ctx):
    pb = MaterialProblem(ctx, Bundle.generate("materials", 1), width=1, height=1, spp=1, max_depth=2)
    theta = pb.random_params(5)
    target = np.zeros((1, 1, 3), np.float32)
    paths = wide = 0
    for frame in range(400):
        _, g = pb.loss_and_grad(theta, target, frame=frame)
        _, ref = pb.loss_and_grad(theta, target, frame=frame, sampling_params=theta)
        assert np.abs(g - ref).max() <= 1e-5 * max(np.abs(ref).max(), 1e-30)
        rows = g.reshape(-1, 6)[: pb.emissive_base, :5]
        rows = rows[(rows != 0).any(1)]
        if len(rows) == 2:
            paths += 1
            wide += (rows != rows.astype(np.float32)).any()
    assert paths >= 5 and wide >= paths // 2
