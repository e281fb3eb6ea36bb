"""The f32 linears of 32 tokens per CTA with tiles of 32 and of 64 output rows (csrc/linear.cu, seq64_pays): products and
sums rounded one by one, k ascending."""
import numpy as np
import pytest

from _gpu import P, bits, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,O", [(32, 136, 4736), (32, 136, 4737), (32, 64, 9472), (31, 64, 9504), (320, 72, 1000), (505, 72, 1001)])
def test_both_tile_heights_are_the_sequential_sum(M, K, O):
    rng = np.random.default_rng(M + O)
    w, x = rng.standard_normal((O, K)).astype(np.float32), rng.standard_normal((M, K)).astype(np.float32)
    want = np.zeros((M, O), np.float32)
    for k in range(K):
        want += x[:, k, None] * w[None, :, k]
    got = np.empty((M, O), np.float32)
    assert lib().apus_cuda_f32_linear(P(w), P(x), P(got), M, K, O, 0) == 0, lib().apus_cuda_last_error()
    lib().apus_cuda_forget(P(w))
    assert np.array_equal(bits(got), bits(want))
