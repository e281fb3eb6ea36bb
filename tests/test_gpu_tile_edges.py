"""The tiled kernels at the edges of their tiles and on both sides of their dispatch rules, bit for bit against a
kernel of this library that knows no tiles."""
import numpy as np
import pytest

from _gpu import bits, cuda_moe, cuda_qgemm, lib
from _oracle import P
from apus_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,O,K", [(64, 128, 128), (65, 256, 384), (127, 128, 1024), (129, 384, 256), (260, 4096, 640),
                                   (1200, 2048, 512)])
@pytest.mark.parametrize("scales", ["usual", "extreme"])
def test_fp8_wide_rows_equal_narrow_rows(M, O, K, scales):
    rng = np.random.default_rng(M + K)
    code = lambda *s: rng.integers(0, 127, s).astype(np.uint8) | (rng.integers(0, 2, s).astype(np.uint8) << 7)   # noqa: E731
    codes, acodes = code(O, K), code(M, K)
    ws = rng.integers(119, 122, (O // 128, K // 128)).astype(np.uint8)
    asc = np.exp2(rng.integers(-12, 3, (M, K // 128))).astype(np.float32)
    if scales == "extreme":                      # scale products outside the window of the one-rounding fold
        ws.flat[:: 2] = 0
        ws.flat[1:: 5] = 20
        asc[:: 3] = np.float32(2.0 ** -22)
    got = cuda_qgemm(8, codes, ws, acodes, asc, O)
    want = np.concatenate([cuda_qgemm(8, codes, ws, acodes[i:i + 32], asc[i:i + 32], O) for i in range(0, M, 32)])
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("T", [33, 513, 2100])
def test_grouping_of_many_routings(T):
    """n = T * topk routings: a few per warp, several steps per warp, more than 4,096 in all."""
    W = synth.MoeWeights(seed=5, E=9, topk=2)
    x = synth.activations(np.random.default_rng(T), T, W.dim)
    whole = cuda_moe(W, x)
    for lo in (0, T // 2, T - 7):
        part = cuda_moe(W, x[lo:lo + 7])
        assert np.array_equal(whole["idx"][lo:lo + 7], part["idx"])
        assert np.array_equal(bits(whole["out"][lo:lo + 7]), bits(part["out"]))


@pytest.mark.parametrize("n,k", [(1, 1), (31, 31), (33, 7), (1024, 512), (2049, 512), (4097, 2048), (5000, 1), (16383, 1025), (16384, 512),
                                 (65537, 512), (70001, 2048), (262144, 512), (262147, 40)])
@pytest.mark.parametrize("values", ["normal", "coarse", "one", "ends"])
def test_topk_selection(n, k, values):
    """Every layout of the selection (keys in registers or read again, one CTA or a cluster): order by (score
    descending, index ascending), with ties at the boundary, one value everywhere, infinities and both zeros."""
    rng = np.random.default_rng(n + k)
    rows = 3
    sc = rng.standard_normal((rows, n)).astype(np.float32)
    if values == "coarse":
        sc = synth.bf16_round(sc)
        sc[1] = np.round(sc[1])
    elif values == "one":
        sc[:] = np.float32(-0.25)
        sc[1, n // 2] = 3.0
    elif values == "ends":
        sc[:, rng.integers(0, n, 3)] = np.inf
        sc[:, rng.integers(0, n, 3)] = -np.inf
        sc[1] = np.where(rng.random(n) < 0.5, np.float32(0.0), np.float32(-0.0))
        sc[2] = np.finfo(np.float32).min
    idx = np.empty((rows, k), np.int32)
    assert lib().apus_cuda_topk_stable(P(sc), n, k, P(idx), rows) == 0, lib().apus_cuda_last_error()
    want = np.argsort(-(sc + np.float32(0)).astype(np.float64), axis=1, kind="stable")[:, :k]
    assert np.array_equal(idx, want)
