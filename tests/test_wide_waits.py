"""The many-row projection's converter warps store into tensor memory with instructions that take whole warps, so every wait ahead
of them has one outcome in all lanes. What a wait does at its limit cannot be reached in a test without starving a kernel; the
source is held to the warp-wide waits instead, and the hand-over is run many times over."""
import os
import re

import numpy as np
import pytest

import quant_fixtures as qf

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "splash_b200", "csrc")


def test_converter_warps_wait_as_warps():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "sb_linear_wide.cu")).read())
    role = re.search(r"else if \(warp < kWideDequantWarps\) \{(.*?)\n  \} else \{", text, re.S).group(1)
    assert "tmem_st16" in role
    waits = re.findall(r"\b(\w*wait\w*|\w*spin\w*)\(", role)
    assert {w for w in waits if w not in ("pdl_wait", "tmem_wait_st")} == {"wide_warp_wait", "wide_warp_spin"}
    for helper in ("wide_warp_wait", "wide_warp_spin"):
        body = re.search(helper + r"\([^)]*\) \{(.*?)\}\n", text, re.S).group(1)
        assert "__shfl_sync(0xffffffffu" in body or "__all_sync(0xffffffffu" in body


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,n,k,rows", [(0, 384, 17408, 128), (0, 256, 256, 17), (4, 256, 8192, 33), (4, 512, 4096, 160)])
def test_hand_over_repeats_itself(fmt, n, k, rows):
    """Up to 68 super-blocks a converter warp, one, two passes: the same bits every time, and no wait at its limit."""
    from test_linear_gpu import run_linear
    from test_linear_wide_gpu import image_of, run_image
    from splash_b200 import lib
    lib.init(0)
    W, X = qf.realistic(fmt, n, k, seed=k), qf.activations(rows, k, seed=rows)
    image = image_of(lib, fmt, W, n, k) if fmt else None
    call = lambda: run_image(lib, fmt, image, n, k, X, rows, out_f32=True) if fmt else run_linear(lib, fmt, W, n, k, X, rows, out_f32=True)
    first = call()
    for _ in range(20):
        assert np.array_equal(call(), first)
    assert lib.device_status() == 0
