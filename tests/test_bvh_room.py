"""A tree that does not fit the caller's 2 n nodes (boxes without a finite extent make a chain of up to 129)
is refused, and nothing is written past them: the host builder, and the device call's host route for NaN."""
import ctypes as C

import numpy as np
import pytest

from barnacle_gb300 import BarnacleError, bvh_build, capi
from barnacle_gb300.capi import ptr


def boxes(n, bad):
    rng = np.random.default_rng(n)
    c = rng.normal(size=(n, 3))
    b = np.concatenate([c - 0.1, c + 0.1], 1).astype(np.float32)
    if bad in ("inf", "inf and nan"):
        b[n // 2, 3] = np.inf
    if bad in ("nan", "inf and nan"):
        b[1, 0] = np.nan
    if bad == "-inf to inf":
        b[n // 2, 0], b[n // 2, 3] = -np.inf, np.inf
    return b


def build(call, b):
    n = len(b)
    nodes = np.full(400 * 32, 0xA5, np.uint8)  # room for any chain, so that an overrun is seen and not suffered
    perm, count = np.zeros(n, np.int32), C.c_int32(-7)
    rc = call(ptr(b), n, ptr(nodes), C.byref(count), ptr(perm))
    assert (nodes[2 * n * 32:] == 0xA5).all()
    assert rc == (capi.BN_ERR_UNSUPPORTED if count.value < 0 else capi.BN_OK) and count.value <= 2 * n
    return rc, nodes[: max(count.value, 0) * 32].tobytes()


@pytest.mark.parametrize("bad", ["inf", "nan", "inf and nan", "-inf to inf"])
@pytest.mark.parametrize("n", [5, 10, 64, 65, 100])
def test_host_builder_stays_within_two_n_nodes(n, bad):
    b = boxes(n, bad)
    rc, _ = build(capi.load_library().bn_bvh_build, b)
    if rc:
        with pytest.raises(BarnacleError):
            bvh_build(b)
    else:
        assert len(bvh_build(b)[0]) <= 2 * n


@pytest.mark.gpu
@pytest.mark.parametrize("bad", ["inf", "nan", "inf and nan", "-inf to inf"])
@pytest.mark.parametrize("n", [5, 10, 64, 65, 100])
def test_device_call_stays_within_two_n_nodes(ctx, n, bad):
    b = boxes(n, bad)
    host = build(ctx.lib.bn_bvh_build, b)
    assert build(lambda *a: ctx.lib.bn_bvh_build_device(ctx._h, *a), b) == host
