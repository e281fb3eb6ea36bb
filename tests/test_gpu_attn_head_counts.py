"""Sparse attention of many rows with few heads: the score tile is as tall as the heads (16, 32 or 64 of them), and rows
shorter than a tile is wide keep the small one.  Bit for bit against the kernels that know no tiles, as in
test_gpu_tile_edges.py, on both sides of each line of that choice."""
import numpy as np
import pytest

import cases
from _gpu import bits
from test_gpu_tile_edges import D, PAD, attn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("s,h,idxw", [(64, 8, 256), (64, 8, 257), (65, 16, 258), (80, 3, 321), (32, 17, 257), (33, 32, 300), (16, 33, 400),
                                      (400, 8, 32), (400, 8, 33), (330, 32, 9), (148, 5, 31), (149, 5, 31)])
def test_few_heads_many_rows(s, h, idxw, bf16):
    c = cases.sparse_attn_case(100 * s + idxw, s, h, D, 40, 90, idxw, "holes")
    q, ka, kb = c["q"], c["kv_a"], c["kv_b"]
    q[1, :, 7] = np.float32(1.0009765625 + 2.0 ** -20)   # one row whose products are not exact in f32
    got = attn(c, q, ka, kb, s, h, D, idxw, bf16)
    wide = lambda a: np.concatenate([a, np.zeros(a.shape[:-1] + (PAD - D,), np.float32)], -1)   # noqa: E731
    want = attn(c, wide(q), wide(ka), wide(kb), s, h, PAD, idxw, bf16)[:, :, :D]
    assert np.array_equal(bits(got), bits(want))
