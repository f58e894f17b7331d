"""Calls that ask for more than any GPU has (859 GB of draws): the call says so, and the context goes on."""
import ctypes as C

import numpy as np
import pytest

from barnacle_gb300 import Bundle, Context, capi
from barnacle_gb300.capi import ptr

pytestmark = pytest.mark.gpu


def ask_too_much(c):
    seeds = np.zeros((100, 3), np.uint32)
    out = np.zeros(1, np.float32)  # never written: the device memory is refused first
    assert c.lib.bn_sampler_stream(c._h, ptr(seeds), 100, 2**31 - 1, ptr(out)) == capi.BN_ERR_OUT_OF_MEMORY


def test_the_next_call_does_not_report_it_again():
    with Context(0) as c:
        b = Bundle.generate("cornell", 1)
        c.upload(b)
        rays = np.zeros(64, capi.RAY_DTYPE)
        rays["origin"], rays["direction"], rays["t_max"] = 0.5, [0.6, 0.0, 0.8], np.inf
        want = c.trace(rays).tobytes()
        ask_too_much(c)
        assert c.trace(rays).tobytes() == want
        b.render.spp = 2
        want = c.render(b.render, b.views)[0].copy()
        ask_too_much(c)
        np.testing.assert_array_equal(c.render(b.render, b.views)[0], want)


def test_the_path_state_makes_room_for_other_buffers():
    """What a render of 4 M paths leaves (1 GB) goes when another buffer finds no memory, and comes back."""
    torch = pytest.importorskip("torch")
    with Context(0) as c:
        b = Bundle.generate("cornell", 1)
        c.upload(b)
        want = c.render(b.render, b.views)[0].copy()
        held = torch.cuda.mem_get_info(0)[0]
        ask_too_much(c)
        assert torch.cuda.mem_get_info(0)[0] - held >= 0.9 * (256 * 256 * 64 * 256)
        np.testing.assert_array_equal(c.render(b.render, b.views)[0], want)
