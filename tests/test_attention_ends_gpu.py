"""The attention kernels' ends (Q into tensor memory, the splits' partials and their merge) where their runs of rows end: every
count of fused rows around 4, 8, 16, 32 and the most, few and many splits, on both kernels. Against the fp64 oracle."""
import numpy as np
import pytest

import oracle_lib as ol
from test_ops_gpu import _setup, attention_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("q_heads,kv_heads,rows,committed,D", [
    (2, 2, 1, 0, 128), (2, 2, 4, 40, 256), (2, 2, 5, 700, 128), (8, 2, 2, 3000, 256), (6, 2, 3, 500, 128), (8, 2, 4, 130, 256),
    (2, 1, 16, 5000, 128), (3, 1, 11, 1000, 256), (8, 1, 13, 20000, 128), (24, 4, 16, 9000, 256), (8, 1, 16, 60, 256),
])
def test_fused_rows_and_splits(kernel, q_heads, kv_heads, rows, committed, D):
    lib, l, o = _setup()
    r = attention_case(lib, l, o, q_heads=q_heads, kv_heads=kv_heads, D=D, page_tokens=64, scale_f16=True, committed=committed, rows=rows, gated=True,
                       seed=rows * 7 + committed, kernel=kernel)
    got, want = ol.bf2f(r["got"]).astype(np.float64), r["want64"]
    # P is rounded to half (2^-11) before P V, the result to bf16 (2^-9, twice with the gate); the rest is fp32
    assert np.abs(got - want).max() <= (2 * 2.0 ** -8 + 2.0 ** -10) * np.abs(want).max()
    assert np.linalg.norm(got - want) <= 2.0 ** -7 * np.linalg.norm(want)
