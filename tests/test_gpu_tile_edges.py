"""The tiled kernels at the edges of their tiles and on both sides of their dispatch rules, bit for bit against a
kernel of this library that knows no tiles: sparse attention against the one-thread-per-score kernels (a head size
that the tiles do not take: 512 values and 8 zeros, which change no sum), the 128-row FP8 GEMM against the 32-row
one, the grouping of routings against a call per piece."""
import numpy as np
import pytest

import cases
from _gpu import bits, cuda_moe, cuda_qgemm, lib
from _oracle import P
from apus_b200 import synth

pytestmark = pytest.mark.gpu
D, PAD = 512, 520


def attn(c, q, ka, kb, s, h, d, idxw, bf16):
    if not bf16:
        o = np.empty((s, h, d), np.float32)
        assert lib().apus_cuda_sparse_attn(P(q), P(c["sink"]), h, d, P(c["idx"]), idxw, s, D ** -0.5, P(ka), len(ka), P(kb), len(kb),
                                           P(o)) == 0, lib().apus_cuda_last_error()
        return o
    import torch
    lib()
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()   # noqa: E731
    # a query pointer that is only 4-byte aligned is a legal one
    qd = torch.empty(q.size + 1, device="cuda")[1:]
    qd.copy_(t(q).reshape(-1))
    sink, idx, a, b = t(c["sink"]), t(c["idx"]), t(synth.bf16_bits(ka).view(np.int16)), t(synth.bf16_bits(kb).view(np.int16))
    o = torch.empty(s * h * d + 1, device="cuda")[1:]
    assert lib().apus_cuda_sparse_attn_dev(qd.data_ptr(), sink.data_ptr(), h, d, idx.data_ptr(), idxw, s, D ** -0.5, a.data_ptr(),
                                           len(ka), b.data_ptr(), len(kb), o.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream) == 0, lib().apus_cuda_last_error()
    torch.cuda.synchronize()
    return o.cpu().numpy().reshape(s, h, d)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("values", ["bf16", "f32", "tiny", "sharp"])
@pytest.mark.parametrize("s,h,idxw", [(1, 64, 1), (1, 64, 9), (2, 3, 129), (5, 64, 640), (7, 64, 911), (13, 64, 33), (32, 64, 130),
                                      (33, 64, 257), (48, 20, 640), (2, 64, 1537)])
def test_attention_tiles(s, h, idxw, values, bf16):
    c = cases.sparse_attn_case(1000 * s + idxw, s, h, D, 40, 90, idxw, "holes" if s > 1 else "full")
    rng = np.random.default_rng(idxw)
    q, ka, kb = c["q"], c["kv_a"], c["kv_b"]
    if values == "f32":                          # products that are not exact in f32
        q = (q * np.float32(1.0009765625 + 2.0 ** -20)).astype(np.float32)
    elif values == "tiny":                       # products below the normal range, in a few chunks of a few rows
        q[:, :, 40:60] = synth.bf16_round((rng.standard_normal((s, h, 20)) * 2.0 ** -75).astype(np.float32))
        ka[3, 40:60] = synth.bf16_round((rng.standard_normal(20) * 2.0 ** -70).astype(np.float32))
    elif values == "sharp":                      # probabilities from 1 down to far below 2^-60
        q = synth.bf16_round(q * np.float32(40.0))
    got = attn(c, q, ka, kb, s, h, D, idxw, bf16)
    wide = lambda a: np.concatenate([a, np.zeros(a.shape[:-1] + (PAD - D,), np.float32)], -1)   # noqa: E731
    want = attn(c, wide(q), wide(ka), wide(kb), s, h, PAD, idxw, bf16)[:, :, :D]
    assert np.array_equal(bits(got), bits(want))


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


@pytest.mark.parametrize("M,K,O", [(1, 8, 1), (1, 4096, 256), (2, 136, 33), (5, 264, 31), (8, 128, 1024), (17, 24, 5), (33, 520, 64),
                                   (40, 392, 4400), (300, 256, 96), (700, 136, 1000)])
def test_f32_linear_is_the_sequential_sum(M, K, O):
    """Every layout of the f32 linears (one chain per lane, four tokens per lane, two rows per lane; short K tiles,
    ragged rows and tokens): products and sums rounded one by one, k ascending."""
    rng = np.random.default_rng(M + O)
    w = rng.standard_normal((O, K)).astype(np.float32)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[0, ::3] = -0.0
    want = np.zeros((M, O), np.float32)
    for k in range(K):
        want += x[:, k, None] * w[None, :, k]
    got = np.empty((M, O), np.float32)
    assert lib().apus_cuda_f32_linear(P(w), P(x), P(got), M, K, O, 0) == 0, lib().apus_cuda_last_error()
    lib().apus_cuda_forget(P(w))
    assert np.array_equal(bits(got), bits(want))
