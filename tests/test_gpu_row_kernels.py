"""The row kernels of long prompts at the sizes where they take over from those of few rows, bit for bit against the
same rows in calls that stay below: mHC (one CTA per row from 512 rows on, maps eight rows per CTA from 256 on), the
activation quantisation (four groups per warp from 37,888 groups on), also with gathered rows and a row count that is
only known on the device."""
import numpy as np
import pytest

import cases
from _gpu import P, bits, cuda_act_quant, lib
from _oracle import ora_act_quant
from apus_b200 import check, synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def order(request):
    L = lib()
    old = L.apus_cuda_set_tree_ops(-1)
    L.apus_cuda_set_tree_ops(L.apus_cuda_set_tree_ops(-2) if request.param == "default" else request.param)
    yield
    L.apus_cuda_set_tree_ops(old)


def hc_pre(c, lo, hi, d, n, normed):
    rows = hi - lo
    x = np.ascontiguousarray(c["x4"][lo:hi])
    y, yn = np.zeros((rows, d), np.float32), np.zeros((rows, d), np.float32)
    po, co = np.empty((rows, n), np.float32), np.empty((rows, n, n), np.float32)
    check(lib().apus_cuda_hc_pre(P(x), d, n, P(c["fn"]), P(c["scale"]), P(c["base"]), 1e-6, 1e-6, 20, P(c["norm_w"]) if normed else None,
                                 1e-6, P(y), P(yn), P(po), P(co), rows))
    yh = np.empty((rows, d), np.float32)
    check(lib().apus_cuda_hc_head(P(x), d, n, P(c["hfn"]), 0.8, P(c["hbase"]), 1e-6, 1e-6, P(yh), rows))
    return y, yn, po, co, yh


@pytest.mark.parametrize("order", [0, "default", 511], indirect=True)
@pytest.mark.parametrize("rows,d,normed", [(16, 256, True), (17, 256, True), (64, 256, True), (255, 256, True), (256, 256, True),
                                           (261, 320, True), (511, 512, True), (512, 256, True), (513, 1280, True), (700, 4096, True),
                                           (530, 192, False), (11, 4096, True), (12, 4096, True)])
def test_mhc_rows_do_not_depend_on_their_number(rows, d, normed, order):
    n = 4
    c = cases.mhc_case(rows + d, rows, d)
    whole = hc_pre(c, 0, rows, d, n, normed)
    for lo in range(0, rows, 7 if rows < 100 else 97):
        hi = min(rows, lo + (7 if rows < 100 else 97))
        for got, part in zip(whole, hc_pre(c, lo, hi, d, n, normed)):
            assert np.array_equal(bits(got[lo:hi]), bits(part))
    for k in ("fn", "hfn"):
        lib().apus_cuda_forget(P(c[k]))


@pytest.mark.parametrize("M,K", [(37887, 128), (37888, 128), (37889, 128), (37891, 128), (9473, 512), (12630, 384), (1185, 4096)])
def test_quantised_rows_do_not_depend_on_their_number(M, K):
    rng = np.random.default_rng(M)
    x = synth.activations(rng, M, K, std=3.0)
    x[M // 2] = 0.0
    codes, scales = cuda_act_quant(x)
    want_c, want_s = ora_act_quant(x)
    assert np.array_equal(codes, want_c) and np.array_equal(bits(scales), bits(want_s))


@pytest.mark.parametrize("n_rout", [9472, 9475])
def test_gathered_rows_of_many_routings(n_rout):
    """The experts of a shard quantise the rows of the routings that are theirs, in sorted order: rows through a map, and
    fewer of them than the launch was sized for."""
    import torch
    E, topk, dim = 5, 2, 512
    W = synth.MoeWeights(seed=9, E=E, topk=topk, dim=dim, inter=dim)
    w = W.moew()
    import ctypes as C
    m = lib().apus_cuda_moe_create(C.byref(w), 1, 4)
    assert m, lib().apus_cuda_last_error()
    rng = np.random.default_rng(n_rout)
    T = 700
    x = torch.from_numpy(synth.activations(rng, T, dim)).cuda()
    row = torch.from_numpy(rng.integers(0, T, n_rout).astype(np.int32)).cuda()
    eid = torch.from_numpy(rng.integers(0, E, n_rout).astype(np.int32)).cuda()
    st = torch.cuda.current_stream().cuda_stream

    def run(lo, hi):
        eo = torch.zeros(hi - lo, dim, device="cuda")
        check(lib().apus_cuda_moe_experts_dev(m, x.data_ptr(), T, row[lo:hi].contiguous().data_ptr(), eid[lo:hi].contiguous().data_ptr(),
                                              hi - lo, eo.data_ptr(), st))
        torch.cuda.synchronize()
        return eo.cpu().numpy()
    try:
        whole = run(0, n_rout)
        for lo in range(0, n_rout, 1500):
            hi = min(n_rout, lo + 1500)
            assert np.array_equal(bits(whole[lo:hi]), bits(run(lo, hi)))
        assert np.abs(whole).max() > 0
    finally:
        lib().apus_cuda_moe_destroy(m)
