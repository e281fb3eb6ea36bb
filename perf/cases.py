"""What a user of this framework has it do, as measurable cases.

A case is one call (or the few calls that belong together) through the C ABI of
include/apus_b200.h on inputs a program has in hand: quantised linears, one
MXFP4 expert, a MoE sublayer, a sparse-attention decode step, and the token loop
of a model -- decode steps, the verify batch of speculative decoding, a prompt.
Sizes are those of DeepSeek-V4-Flash as in flash.py and of the benchmark's
configurations, spread over the ranges a serving program meets.

The token-loop cases run the model cut after eight of its 43 layers (two
sliding-window, three compressed-sparse, three heavily-compressed; hash routing
in the first three) with the true vocabulary and head, so that a state is about
30 GB and several of them fit the card.
"""
import ctypes as C
import math

import torch

import apus_b200
from apus_b200 import capi
from apus_b200.flash import FlashConfig, RandomFlashModel, prompt_ids

MODEL_LAYERS = 8
HEADS, HEAD_DIM, WINDOW, TOPK = 64, 512, 128, 512
# the FP8 projections of a layer, [O, K]: q down / q up / kv / o up / shared expert up and down / a square one
FP8_SHAPES = ((1024, 4096), (32768, 1024), (512, 4096), (4096, 8192), (2048, 4096), (4096, 2048), (4096, 4096))


def listed():
    return [
        # one projection for one token: launches and latency
        {"name": "fp8_linear_m1", "kind": "fp8", "M": 1, "O": 4096, "K": 4096},
        # the same projection over a long prompt: the tensor cores
        {"name": "fp8_linear_m4096", "kind": "fp8", "M": 4096, "O": 4096, "K": 4096},
        # a MoE sublayer at a decode batch (most experts touched by one token or two) ...
        {"name": "moe_t32", "kind": "moe", "T": 32, "hash": False},
        # ... and over a prompt (every expert touched by a dozen)
        {"name": "moe_t512", "kind": "moe", "T": 512, "hash": False},
        # one query against a million tokens of context: the selection over 262,144 scores
        {"name": "attn_csa_1m_b1", "kind": "attn", "form": "csa", "ctx": 1 << 20, "B": 1},
        # a decode batch at an everyday context
        {"name": "attn_csa_8k_b32", "kind": "attn", "form": "csa", "ctx": 8192, "B": 32},
        # a heavily compressed layer attends every entry it has; odd batch, ragged context
        {"name": "attn_hca_100k_b7", "kind": "attn", "form": "hca", "ctx": 100003, "B": 7},
        # the token loop for one user
        {"name": "decode_b1", "kind": "decode", "B": 1, "ctx": 512, "temp": 0.0},
        # the token loop of a full batch
        {"name": "decode_b32", "kind": "decode", "B": 32, "ctx": 512, "temp": 0.0},
        # a handful of users who sample (the serve loop's default), further into their conversations
        {"name": "decode_b5_sampled", "kind": "decode", "B": 5, "ctx": 1501, "temp": 0.8},
        # speculative decoding: one pass over the held token and five drafts, mid-stream
        {"name": "verify_s6", "kind": "verify", "B": 1, "s": 6, "ctx": 1001},
        # the prompts of eight users in one call
        {"name": "prefill_b8_s512", "kind": "prefill", "B": 8, "s": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("fp8", "expert", "moe", "attn", "decode", "decode", "verify", "prefill"))
    if kind == "fp8":
        O, K = rng.choice(FP8_SHAPES)
        return {"kind": "fp8", "M": _log(rng, 1, 4096), "O": O, "K": K}
    if kind == "expert":                      # one routed expert for the tokens a step sends it
        return {"kind": "expert", "T": _log(rng, 1, 96)}
    if kind == "moe":
        return {"kind": "moe", "T": _log(rng, 1, 1024), "hash": rng.random() < 0.25}
    if kind == "attn":
        return {"kind": "attn", "form": rng.choice(("csa", "hca")), "ctx": _log(rng, 1500, 1 << 20), "B": _log(rng, 1, 32)}
    if kind == "decode":
        B = _log(rng, 1, 32)
        return {"kind": "decode", "B": B, "ctx": _log(rng, 24, min(4096, 16384 // B)), "temp": rng.choice((0.0, 0.0, 0.8))}
    if kind == "verify":
        return {"kind": "verify", "B": 1, "s": rng.randint(2, 8), "ctx": _log(rng, 24, 4096)}
    B = _log(rng, 1, 16)
    return {"kind": "prefill", "B": B, "s": _log(rng, 17, min(1500, 4096 // B))}


# ---- what a program has in hand before the call --------------------------------------------------
class _Handle:
    """A library object that goes when the state goes; keeps alive the device memory it points into."""

    def __init__(self, p, free, keep=()):
        if not p:
            raise RuntimeError(apus_b200.lib().apus_cuda_last_error().decode())
        self.p, self.free, self.keep = p, free, keep

    def __del__(self):
        self.free(self.p)


def _ok(rc):
    apus_b200.check(rc)


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _gen(seed):
    return torch.Generator(device=_dev()).manual_seed(seed)


def _rows(g, *shape):
    """Activations: N(0, 1) BF16 values carried as f32, the form every sublayer hands on."""
    return torch.randn(*shape, generator=g, device=_dev()).bfloat16().float()


def prepare(case, seed):
    L = apus_b200.lib()
    err = C.create_string_buffer(512)
    if L.apus_cuda_enable(err, 512):
        raise RuntimeError(err.value.decode())
    return {"fp8": _prep_fp8, "expert": _prep_expert, "moe": _prep_moe, "attn": _prep_attn, "decode": _prep_model,
            "verify": _prep_model, "prefill": _prep_model}[case["kind"]](L, case, seed)


def _prep_fp8(L, c, seed):
    g, O, K = _gen(seed), c["O"], c["K"]
    codes = (torch.randn(O, K, generator=g, device=_dev()) * 2.56).to(torch.float8_e4m3fn).view(torch.uint8)
    scales = torch.randint(119, 122, ((O + 127) // 128, K // 128), generator=g, device=_dev(), dtype=torch.uint8)
    torch.cuda.synchronize()
    h = _Handle(L.apus_cuda_fp8_upload(capi.qw(codes, scales, O, K)), L.apus_cuda_fp8_free, (codes, scales))
    return {"kind": "fp8", "M": c["M"], "w": h, "x": _rows(g, c["M"], K), "out": torch.empty(c["M"], O, device=_dev())}


def _prep_expert(L, c, seed):
    g, dim, inter = _gen(seed), 4096, 2048

    def up(O, K):
        codes = torch.randint(0, 256, (O, K // 2), generator=g, device=_dev(), dtype=torch.uint8)
        scales = torch.randint(120, 127, (O, K // 32), generator=g, device=_dev(), dtype=torch.uint8)
        torch.cuda.synchronize()
        return _Handle(L.apus_cuda_fp4_upload(capi.qw(codes, scales, O, K)), L.apus_cuda_fp4_free, (codes, scales))
    return {"kind": "expert", "T": c["T"], "w1": up(inter, dim), "w2": up(dim, inter), "w3": up(inter, dim),
            "x": _rows(g, c["T"], dim), "out": torch.empty(c["T"], dim, device=_dev())}


def _prep_moe(L, c, seed):
    cfg = FlashConfig(n_layers=4, vocab=4096)
    W = RandomFlashModel(cfg, seed, _dev(), max_pos=16, layer_ids=[0 if c["hash"] else 3])
    mw = W.desc.layers[0].mw
    h = _Handle(L.apus_cuda_moe_create(C.byref(mw), 0, cfg.n_experts), L.apus_cuda_moe_destroy, (W,))
    ids = None
    if c["hash"]:
        _ok(L.apus_cuda_moe_set_hash_table(h.p, mw.tid2eid, cfg.vocab))
        ids = torch.randint(0, cfg.vocab, (c["T"],), generator=_gen(seed), device=_dev(), dtype=torch.int64)
    return {"kind": "moe", "T": c["T"], "moe": h, "x": _rows(_gen(seed + 1), c["T"], cfg.dim), "ids": ids,
            "out": torch.empty(c["T"], cfg.dim, device=_dev())}


def _prep_attn(L, c, seed):
    g, B = _gen(seed), c["B"]
    nb = c["ctx"] // (4 if c["form"] == "csa" else 128)
    bf = lambda *s: torch.randn(*s, generator=g, device=_dev(), dtype=torch.bfloat16)  # noqa: E731
    k = min(TOPK, nb) if c["form"] == "csa" else nb
    s = {"kind": "attn", "B": B, "nb": nb, "k": k, "q": _rows(g, B, HEADS, HEAD_DIM),
         "sink": torch.randn(HEADS, generator=g, device=_dev()) * 0.5, "ring": bf(B, WINDOW, HEAD_DIM),
         "cache": bf(B, nb, HEAD_DIM), "idx": torch.empty(B, WINDOW + k, dtype=torch.int32, device=_dev()),
         "o": torch.empty(B, HEADS, HEAD_DIM, device=_dev())}
    s["idx"][:, :WINDOW] = torch.arange(WINDOW, dtype=torch.int32, device=_dev())
    if c["form"] == "csa":
        s["scores"] = torch.randn(B, nb, generator=g, device=_dev())
        s["topk"] = torch.empty(B, k, dtype=torch.int32, device=_dev())
    else:
        s["idx"][:, WINDOW:] = WINDOW + torch.arange(nb, dtype=torch.int32, device=_dev())
    return s


def _prep_model(L, c, seed):
    cfg, B = FlashConfig(n_layers=MODEL_LAYERS), c["B"]
    ctx, steps = c.get("ctx", 0), c.get("s", 4)
    W = RandomFlashModel(cfg, seed, _dev(), max_pos=ctx + steps + 16)
    m = _Handle(L.apus_cuda_model_create(C.byref(W.desc), B, ctx + steps + 16), L.apus_cuda_model_destroy, (W,))
    ids = prompt_ids(seed, 0, B, ctx + steps, cfg.vocab)
    rows = steps if c["kind"] == "verify" else 1
    s = {"kind": c["kind"], "B": B, "s": steps, "model": m, "ids": ids[:, ctx:].copy(),
         "logits": torch.empty(B, rows, cfg.vocab, pin_memory=True),
         "next": torch.empty(B if c["kind"] != "decode" else steps * B, rows, dtype=torch.int32, pin_memory=True)}
    if c.get("temp", 0.0) > 0:
        _ok(L.apus_cuda_model_set_sampling(m.p, c["temp"], 0.95, seed))
    if ctx:                                    # the sequences so far, and the point a pass returns to
        before = ids[:, :ctx].copy()
        _ok(L.apus_cuda_model_forward(m.p, before.ctypes.data, ctx, None, None))
        s["snap"] = _Handle(L.apus_cuda_model_snapshot(m.p, None), L.apus_cuda_snap_free, (m,))
    if c["kind"] == "decode":
        s["cols"] = [ids[:, ctx + t].copy() for t in range(steps)]
    return s


# ---- one pass -------------------------------------------------------------------------------------
def run(s):
    L, k = apus_b200.lib(), s["kind"]
    if k == "fp8":
        _ok(L.apus_cuda_fp8_linear_dev(s["w"].p, s["x"].data_ptr(), s["out"].data_ptr(), s["M"], _stream()))
        return s["out"]
    if k == "expert":
        _ok(L.apus_cuda_expert_fp4_dev(s["w1"].p, s["w2"].p, s["w3"].p, 10.0, s["x"].data_ptr(), s["T"], s["out"].data_ptr(),
                                       _stream()))
        return s["out"]
    if k == "moe":
        _ok(L.apus_cuda_moe_forward_dev(s["moe"].p, s["x"].data_ptr(), capi.ptr(s["ids"]), s["T"], s["out"].data_ptr(), _stream()))
        return s["out"]
    if k == "attn":
        if "scores" in s:                     # selection, then the index row: window entries first, the chosen ones after them
            _ok(L.apus_cuda_topk_stable_dev(s["scores"].data_ptr(), s["nb"], s["k"], s["topk"].data_ptr(), s["B"], _stream()))
            torch.add(s["topk"], WINDOW, out=s["idx"][:, WINDOW:])
        _ok(L.apus_cuda_sparse_attn_batch_dev(s["q"].data_ptr(), s["sink"].data_ptr(), HEADS, HEAD_DIM, s["idx"].data_ptr(),
                                              WINDOW + s["k"], s["B"], HEAD_DIM ** -0.5, s["ring"].data_ptr(), WINDOW, WINDOW,
                                              s["cache"].data_ptr(), s["nb"], s["nb"], s["o"].data_ptr(), _stream()))
        return {"o": s["o"], "idx": s["idx"]}
    m, logits, nxt = s["model"].p, s["logits"], s["next"]
    if k == "decode":                         # four steps, each with the ids of its position from the host and its picks back
        _ok(L.apus_cuda_model_restore(m, s["snap"].p))
        for t in range(s["s"]):
            _ok(L.apus_cuda_model_forward(m, s["cols"][t].ctypes.data, 1, logits.data_ptr() if t == s["s"] - 1 else None,
                                          nxt.data_ptr() + 4 * t * s["B"]))
    elif k == "verify":                       # all positions' logits and picks in one pass
        _ok(L.apus_cuda_model_restore(m, s["snap"].p))
        _ok(L.apus_cuda_model_forward_all(m, s["ids"].ctypes.data, s["s"], logits.data_ptr(), nxt.data_ptr()))
    else:
        _ok(L.apus_cuda_model_reset(m))
        _ok(L.apus_cuda_model_forward(m, s["ids"].ctypes.data, s["s"], logits.data_ptr(), nxt.data_ptr()))
    return {"logits": logits, "next": nxt}


# ---- what a pass cannot do without -----------------------------------------------------------------
def _touched(T, E=256, k=6):
    """Distinct experts T tokens reach on average."""
    return E * (1.0 - (1.0 - k / E) ** T)


def _moe_work(T):
    exp_b, exp_w, sh_w, gate_w = 3 * 2048 * 4096 * 17 // 32, 3 * 2048 * 4096, 3 * 2048 * 4096, 256 * 4096
    return (_touched(T) * exp_b + sh_w + gate_w * 4 + T * 4096 * 8, 2.0 * T * (6 * exp_w + sh_w + gate_w))


def _attn_work(B, h, d, rows, esz):
    return B * (rows * d * esz + h * d * 8), 4.0 * B * h * rows * d


def work(case):
    k = case["kind"]
    if k == "fp8":
        M, O, K = case["M"], case["O"], case["K"]
        return {"bytes": O * K + O * K // 16384 + 4 * M * (K + O), "flops": 2.0 * M * O * K}
    if k == "expert":
        return {"bytes": 3 * 2048 * 4096 * 17 // 32 + 8 * case["T"] * 4096, "flops": 6.0 * case["T"] * 2048 * 4096}
    if k == "moe":
        b, f = _moe_work(case["T"])
        return {"bytes": b, "flops": f}
    if k == "attn":
        nb, csa = case["ctx"] // (4 if case["form"] == "csa" else 128), case["form"] == "csa"
        sel = min(TOPK, nb) if csa else nb
        b, f = _attn_work(case["B"], HEADS, HEAD_DIM, WINDOW + sel, 2)
        return {"bytes": b + case["B"] * (4 * nb if csa else 0), "flops": f}
    # token loop: the projections, the routed and the shared experts, the attention over what is selected, the head
    cfg = FlashConfig(n_layers=MODEL_LAYERS)
    B, s = case["B"], case.get("s", 4)
    passes, T = (s, B) if k == "decode" else (1, B * s)
    heads = passes * (B if k != "verify" else T)           # rows whose logits are computed
    tot_b, tot_f = 0.0, 0.0
    for ratio in cfg.layer_kinds():
        fp8 = 4096 * 1024 + 32768 * 1024 + 512 * 4096 + 4096 * 8192
        dense = 8 * 1024 * 4096 * 2 + 2 * 24 * 16384 * 4   # o-projection (BF16), the two mHC maps (f32)
        mac = fp8 + 8 * 1024 * 4096 + 2 * 24 * 16384
        if ratio:
            cd = 1024 if ratio == 4 else 512
            dense += 2 * cd * 4096 * 4
            mac += 2 * cd * 4096
        if ratio == 4:
            fp8 += 8192 * 1024
            dense += (2 * 256 + 64) * 4096 * 4
            mac += 8192 * 1024 + (2 * 256 + 64) * 4096
        mb, mf = _moe_work(T)
        pos = case.get("ctx", 0) + (s if k != "prefill" else s // 2)
        rows = min(WINDOW, pos) + (0 if not ratio else min(TOPK if ratio == 4 else 1 << 30, pos // ratio))
        ab, af = _attn_work(T, HEADS, HEAD_DIM, rows, 4)
        if k == "prefill":                                 # the rows of a prompt share one cache
            ab = B * s * HEAD_DIM * 4 + T * HEADS * HEAD_DIM * 8
        tot_b += fp8 + dense + mb + ab
        tot_f += 2.0 * T * mac + mf + af
    return {"bytes": passes * tot_b + (passes if k == "decode" else 1) * cfg.vocab * 4096 * 2 + 4 * heads * cfg.vocab,
            "flops": passes * tot_f + 2.0 * heads * cfg.vocab * 4096}


def tolerance(case):
    """Every sum is f32 over exact products; outputs are rounded to BF16, so another order of a sum moves a few of
    them by one BF16 step (2^-8 to 2^-7 of the value).  The figures are four times the distance from the same
    arithmetic with its sums in 64 bits."""
    k = case["kind"]
    if k == "fp8":
        return {"rel": 6e-5, "max": 0.03}
    if k in ("expert", "moe"):                # the SwiGLU outputs are quantised again: a step there can move an E4M3 code
        return {"rel": 5e-4, "max": 0.03}
    if k == "attn":
        return {"rel": 8e-4, "max": 0.03}
    # Layer after layer of quantised activations multiply the least difference (one BF16 step in one embedding value
    # ends far away in the logits after a few layers), so hidden states are the same bits in every correct run; only the
    # head's own f32 sums, which nothing quantises, have room.
    return {"rel": 1e-5, "max": 4e-4, "differ": 0.0}
