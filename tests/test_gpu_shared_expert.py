"""The shared expert on both sides of the line where gate and up go through the 128-row kernel one after the other (the
up projection then waits in the output rows): the same bits as calls of few rows, also into an output that is only
4-byte aligned and with an output row shorter than a hidden one, where the paired kernel is kept."""
import ctypes as C

import numpy as np
import pytest

from _gpu import lib
from apus_b200 import check, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,inter,rows", [(2048, 2048, 288), (2048, 2048, 289), (512, 512, 1184), (512, 512, 1187), (512, 1024, 600)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows_do_not_depend_on_their_number(dim, inter, rows, shift):
    import torch
    W = synth.MoeWeights(seed=3, E=2, topk=1, dim=dim, inter=inter)
    w = W.moew()
    m = lib().apus_cuda_moe_create(C.byref(w), 0, 2)
    assert m, lib().apus_cuda_last_error()
    x = torch.from_numpy(synth.activations(np.random.default_rng(rows), rows, dim)).cuda()
    st = torch.cuda.current_stream().cuda_stream

    def run(part):
        out = torch.full((part.shape[0] * dim + shift,), float("nan"), device="cuda")[shift:]
        check(lib().apus_cuda_moe_shared_dev(m, part.data_ptr(), part.shape[0], out.data_ptr(), st))
        torch.cuda.synchronize()
        return out.cpu().numpy().reshape(-1, dim).view(np.uint32)
    try:
        whole = run(x)
        for lo in range(0, rows, 60):
            assert np.array_equal(whole[lo:lo + 60], run(x[lo:lo + 60].contiguous()))
    finally:
        lib().apus_cuda_moe_destroy(m)
