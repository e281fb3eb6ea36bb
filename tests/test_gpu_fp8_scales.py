"""apus_cuda_fp8_gemm takes the caller's f32 activation scales, which need not be powers of two: a product
dot * scale is then not exact, and the fold of c/fp8.h:136 rounds it before it is added.  From 64 rows on the
128-row kernel folds with one fused instruction where that cannot show; a row's bits must not depend on how many
rows come with it.  Compared bit for bit with the same rows in calls of 32."""
import numpy as np
import pytest

from _gpu import bits, cuda_qgemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,O,K", [(64, 256, 512), (129, 128, 1024), (300, 384, 384)])
@pytest.mark.parametrize("scales", ["all", "one_row", "one_block", "odd_ulp", "negative", "zero"])
def test_caller_scales_that_are_no_powers_of_two(M, O, K, scales):
    rng = np.random.default_rng(M + K)
    code = lambda *s: rng.integers(0, 127, s).astype(np.uint8) | (rng.integers(0, 2, s).astype(np.uint8) << 7)   # noqa: E731
    codes, acodes = code(O, K), code(M, K)
    ws = rng.integers(119, 122, (O // 128, K // 128)).astype(np.uint8)
    asc = np.exp2(rng.integers(-12, 3, (M, K // 128))).astype(np.float32)
    if scales == "all":
        asc = rng.uniform(0.01, 3.0, asc.shape).astype(np.float32)
    elif scales == "one_row":
        asc[M - 1] = np.float32(0.3)
    elif scales == "one_block":
        asc[:, 1] = rng.uniform(0.01, 3.0, M).astype(np.float32)
    elif scales == "odd_ulp":                    # the two neighbours of a power of two
        asc[::2] = np.nextafter(asc[::2], np.float32(0))
        asc[1::2] = np.nextafter(asc[1::2], np.float32(np.inf))
    elif scales == "negative":
        asc[::3] *= -1
    else:
        asc[::3] = 0.0
    got = cuda_qgemm(8, codes, ws, acodes, asc, O)
    want = np.concatenate([cuda_qgemm(8, codes, ws, acodes[i:i + 32], asc[i:i + 32], O) for i in range(0, M, 32)])
    assert np.array_equal(bits(got), bits(want))
