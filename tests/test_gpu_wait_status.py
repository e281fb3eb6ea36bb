"""A bounded wait that ran out leaves outputs unwritten, so every entry point that returns finished results has to say
so.  The code is planted by the host in the word the kernels would record it in (nothing waits in vain on the GPU):
the call must fail and name it, leave the word clear, and the next call succeed."""
import ctypes as C

import numpy as np
import pytest

import cases
from _gpu import P, lib
from apus_b200 import capi, synth

pytestmark = pytest.mark.gpu


def plant(code):
    import torch
    f = lib()._ZN4apus9wait_wordEv                       # int *apus::wait_word()
    f.restype, f.argtypes = C.c_void_p, []

    class Word:
        __cuda_array_interface__ = dict(data=(f(), False), shape=(1,), typestr="<i4", version=3)
    torch.as_tensor(Word(), device="cuda").fill_(code)
    torch.cuda.synchronize()


def f32_linear(M):
    rng = np.random.default_rng(M)
    w, x, o = (rng.standard_normal(s).astype(np.float32) for s in ((40, 256), (M, 256), (M, 40)))
    rc = lib().apus_cuda_f32_linear(P(w), P(x), P(o), M, 256, 40, 0)
    lib().apus_cuda_forget(P(w))
    return rc


def sparse_attn():
    c = cases.sparse_attn_case(3, 2, 4, 128, 16, 40, 24, "holes")
    o = np.empty((2, 4, 128), np.float32)
    return lib().apus_cuda_sparse_attn(P(c["q"]), P(c["sink"]), 4, 128, P(c["idx"]), 24, 2, 128 ** -0.5, P(c["kv_a"]), 16, P(c["kv_b"]), 40,
                                       P(o))


def moe(router_only, dim=512):
    W = synth.MoeWeights(seed=5, E=8, topk=2, dim=dim, inter=dim)
    x = synth.activations(np.random.default_rng(4), 3, W.dim)
    w, o = W.moew(), np.empty((3, W.dim), np.float32)
    sp, b = np.empty((3, 8), np.float32), np.empty((3, 8), np.float32)
    rc = lib().apus_cuda_router_score(C.byref(w), P(x), 3, P(sp), P(b)) if router_only else \
        lib().apus_cuda_moe_forward(C.byref(w), P(x), None, 3, P(o), None)
    lib().apus_cuda_forget(P(W.gate_w))
    return rc


def fp8(M):
    rng = np.random.default_rng(M)
    codes, scales = synth.fp8_weight(rng, 128, 256)
    x, o = synth.activations(rng, M, 256), np.empty((M, 128), np.float32)
    w = capi.qw(codes, scales, 128, 256)
    rc = lib().apus_cuda_fp8_linear(C.byref(w), P(x), P(o), M, 256, 128)
    lib().apus_cuda_forget(P(codes))
    return rc


def fp8_expert():
    rng = np.random.default_rng(8)
    w = [synth.fp8_weight(rng, 128, 128) for _ in range(3)]
    q = [capi.qw(*a, 128, 128) for a in w]
    x, o = synth.activations(rng, 3, 128), np.empty((3, 128), np.float32)
    rc = lib().apus_cuda_expert(*(C.byref(a) for a in q), 1, 0.0, P(x), 3, 128, 128, P(o))
    for a in w:
        lib().apus_cuda_forget(P(a[0]))
    return rc


CALLS = {"f32_linear_1": lambda: f32_linear(1), "f32_linear_5": lambda: f32_linear(5), "sparse_attn": sparse_attn,
         "router_score": lambda: moe(True), "moe_forward": lambda: moe(False), "moe_forward_mma_sync": lambda: moe(False, 128),
         "fp8_linear": lambda: fp8(3), "fp8_expert": fp8_expert}


@pytest.mark.parametrize("name", list(CALLS))
def test_a_wait_that_ran_out_is_reported(name):
    L = lib()
    plant(42)
    try:
        assert CALLS[name]() != 0
        assert b"code 42" in L.apus_cuda_last_error()
    finally:
        left = L.apus_cuda_kernel_status(1)
    assert left == 0
    assert CALLS[name]() == 0, L.apus_cuda_last_error()
