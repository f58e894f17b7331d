"""Ray queries in their forms (rays spread over warps, a thread per ray, persistent lanes) against the
counting query, which always walks a thread per ray in the reference's order: the same records."""
import numpy as np
import pytest

from barnacle_gb300 import Bundle, capi

pytestmark = pytest.mark.gpu


def rays(n, scene, seed):
    rng = np.random.default_rng(seed)
    lo, hi = ([-60, 0.1, -60], [60, 22, 60]) if scene == "instances" else ([0.05] * 3, [0.95] * 3)
    r = np.zeros(n, capi.RAY_DTYPE)
    r["origin"] = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[::7, 0] = 0  # on box planes and along them
    d /= np.sqrt((d ** 2).sum(1, dtype=np.float32))[:, None]
    r["direction"] = d
    r["t_max"] = np.where(rng.random(n) < 0.5, np.inf, rng.uniform(0, 30, n))
    return r


# ends of the three forms, one ray, sizes that fill no warp and that pass the pinned result buffer
@pytest.mark.parametrize("scene", ["cornell", "cornell-objects", "instances"])
@pytest.mark.parametrize("n", [1, 3, 31, 64, 1487, 1489, 4096, 4097, 50001, 196607, 196608, 400003])
def test_forms_give_the_same_records(ctx, scene, n):
    b = Bundle.generate(scene, 1)
    ctx.upload(b)
    q = rays(n, scene, n)
    for flags in (0, capi.BN_TRACE_WATERTIGHT, capi.BN_TRACE_ANY, capi.BN_TRACE_ANY | capi.BN_TRACE_WATERTIGHT):
        got = ctx.trace(q, flags)
        want = ctx.trace(q, flags | capi.BN_TRACE_COUNT)
        assert got.tobytes() == want.tobytes()
