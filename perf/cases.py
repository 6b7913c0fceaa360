"""The work that users of this library have it do, as cases that can be timed and compared: which calls, at which sizes, from
which inputs.  listed() names the ones that are looked at first; draw() gives more of the same ranges.

Kinds of case:
  moe      one SEED4P4 expert layer for T rows that are on the device (Moe.forward_dev): decode rows, a batch of sequences, a prompt
  step     the same layer from pinned host memory to pinned host memory (Moe.forward_pinned), as an engine steps a batch
  experts3 one expert layer of the P = 3 format at decode, through the entry points an engine calls for it
  mv       a dense seed projection for 1..8 rows (kc_mv)
  mm       a dense seed projection for the rows of a prompt (kc_mm)
  head     the affine int4 LM head for 1..8 rows and the greedy tokens (kc_mv with MF_Q4, kc_argmax)
  attn     decode attention over a BF16 or 8-bit KV cache, rows of different lengths (kc_attn)
  decoder  a whole decode step of a small MoE decoder (Decoder.step)

Weights are uniform random streams (a seed stream of real weights looks the same to the kernels), activations N(0, 1) rounded
to bf16, router logits N(0, 1), as in bench.py."""
import ctypes as C
import math

import numpy as np
import torch

from nanoseedlm_b200 import decoder as dec
from nanoseedlm_b200 import lib as L
from nanoseedlm_b200 import moe
from nanoseedlm_b200.kernels import stream_table

SPLITS = 32      # attention splits the decoder asks for


def listed():
    return [
        # a dense 2048 x 4096 projection for one token: the smallest call, a few microseconds
        {"name": "mv_2048x4096_1", "kind": "mv", "p": 4, "R": 2048, "K": 4096, "T": 1},
        # one token through an expert layer: single-stream decode
        {"name": "moe_128x8_1", "kind": "moe", "d": 2048, "ff": 512, "E": 128, "k": 8, "T": 1},
        # eight rows (multi-token-prediction verify) from host memory to host memory, one step in flight
        {"name": "step_128x8_8", "kind": "step", "d": 2048, "ff": 512, "E": 128, "k": 8, "T": 8},
        # a layer whose widths are not powers of two, and a batch that is not one either
        {"name": "moe_60x4_5_wide1536", "kind": "moe", "d": 1536, "ff": 704, "E": 60, "k": 4, "T": 5},
        # eight rows of a layer stored in the 3-coefficient format
        {"name": "experts3_128x8_8", "kind": "experts3", "d": 2048, "ff": 512, "E": 128, "k": 8, "T": 8},
        # continuous batching: 64 sequences, one token each, over 512 experts
        {"name": "moe_512x10_64", "kind": "moe", "d": 2048, "ff": 512, "E": 512, "k": 10, "T": 64},
        # a prompt chunk of ordinary size
        {"name": "moe_128x8_512", "kind": "moe", "d": 2048, "ff": 512, "E": 128, "k": 8, "T": 512},
        # a long prompt in one call: the largest work
        {"name": "moe_128x8_4096", "kind": "moe", "d": 2048, "ff": 512, "E": 128, "k": 8, "T": 4096},
        # a dense projection of a prompt of odd length
        {"name": "mm_2048x2048_777", "kind": "mm", "p": 4, "R": 2048, "K": 2048, "T": 777},
        # the LM head and the greedy tokens for eight rows
        {"name": "head_151936x2048_8", "kind": "head", "R": 151936, "K": 2048, "T": 8},
        # attention of a batch of sequences of different lengths over the 8-bit cache
        {"name": "attn_q8_24x5000", "kind": "attn", "q8": True, "n_kv": 2, "group": 8, "T": 24, "ctx": 5000, "gate": False},
        # a decode step at batch 32 (three layers of the benchmark's decoder, whose other 45 are the same)
        {"name": "decoder_3_layers_32", "kind": "decoder", "layers": 3, "E": 512, "k": 10, "T": 32, "ctx": 4096, "vocab": 151936, "dense_bf16": True},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of step in [lo, hi], its logarithm uniform."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(["moe", "moe", "moe", "step", "experts3", "mv", "mm", "head", "attn", "decoder"])
    if kind in ("moe", "step", "experts3"):
        if rng.random() < 0.5:
            d, ff = rng.choice([1024, 2048]), rng.choice([256, 512, 1024])
        else:
            d, ff = _log(rng, 768, 3072, 64), _log(rng, 256, 1024, 64)
        E = _log(rng, 16, 512)
        while E * d * ff > 512 * 2048 * 512:
            E = E // 2
        k = rng.randint(2, 10)
        T = _log(rng, 1, 4096) if kind == "moe" else rng.randint(1, 16) if kind == "step" else rng.randint(1, 8)
        while T > 1 and (T * k * d * ff > 4096 * 8 * 2048 * 512 or T > 1024 and E * d * ff > 128 * 2048 * 512):
            T = T * 2 // 3
        return {"kind": kind, "d": d, "ff": ff, "E": E, "k": k, "T": T}
    if kind == "mv":
        return {"kind": "mv", "p": rng.choice([4, 4, 3]), "R": _log(rng, 256, 8192, 2), "K": rng.choice([512, 1024, 2048, 4096, _log(rng, 512, 6144, 64), _log(rng, 512, 4096, 8)]),
                "T": rng.randint(1, 8)}
    if kind == "mm":
        return {"kind": "mm", "p": rng.choice([4, 4, 3]), "R": _log(rng, 256, 8192), "K": _log(rng, 512, 4096, 64), "T": _log(rng, 9, 2048)}
    if kind == "head":
        return {"kind": "head", "R": _log(rng, 16000, 151936), "K": rng.choice([1024, 2048, 4096, _log(rng, 768, 4096, 64)]), "T": rng.randint(1, 8)}
    if kind == "attn":
        T, n_kv = _log(rng, 1, 64), rng.choice([1, 2, 4, 8])
        return {"kind": "attn", "q8": rng.random() < 0.5, "n_kv": n_kv, "group": rng.randint(1, 16), "T": T,
                "ctx": _log(rng, 64, min(32768, 2000000 // (T * n_kv))), "gate": rng.random() < 0.3}
    return {"kind": "decoder", "layers": rng.randint(1, 3), "E": _log(rng, 32, 512), "k": rng.randint(2, 10), "T": _log(rng, 1, 32), "ctx": _log(rng, 256, 4096),
            "vocab": _log(rng, 16000, 151936), "dense_bf16": rng.random() < 0.6}


class _State:
    """What a user's program holds between calls."""

    def __init__(self, kind):
        self.kind = kind


class _Owner:
    """Owns one of the library's handles: closed when nothing refers to it or to a view of its buffers any more."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        torch.cuda.synchronize()
        self.handle.close()


def _bf16(shape, gen, scale=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(torch.bfloat16).float()


def _ptr(t):
    return C.c_void_p(t.data_ptr() if t is not None else 0)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _bits(n, hi, gen, dtype):
    return torch.randint(0, hi, (n,), generator=gen, device="cuda", dtype=torch.int32).to(dtype)


class _Stack3:
    """E matrices of R x K in the P = 3 format: seeds, nibble words and the device table of their slices."""

    def __init__(self, E, R, K, gen, eb=-22):
        nb = R * K // 8
        self.seeds = (_bits(E * nb, 65535, gen, torch.int32) + 1).to(torch.int16).view(E, nb)
        self.nibs = _bits(E * nb, 65536, gen, torch.int16).view(E, nb)
        arr = (L.WSlice * E)()
        for e in range(E):
            arr[e].p[0], arr[e].p[1], arr[e].eb = self.seeds.data_ptr() + 2 * nb * e, self.nibs.data_ptr() + 2 * nb * e, eb
        self.first = arr[0]
        self.table = torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).cuda()


class _View:
    """A float32 buffer of a handle as something torch (device memory) or numpy (pinned memory) can look at; it keeps the handle."""

    def __init__(self, owner, ptr, shape, device):
        self.owner = owner
        setattr(self, "__cuda_array_interface__" if device else "__array_interface__",
                {"data": (int(ptr), False), "shape": shape, "typestr": "<f4", "version": 2 if device else 3})


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = _State(kind)
    st.lib, st.case, st.G = L.load(), case, stream_table()
    if kind in ("moe", "step"):
        d, E, T = case["d"], case["E"], case["T"]
        layer = moe.DeviceLayer.random_on_device(d, case["ff"], E, gen)
        st.owner = _Owner(moe.Moe(layer, case["k"], T))
        st.handle = st.owner.handle
        st.x, st.logits, st.out = _bf16((T, d), gen), torch.randn((T, E), generator=gen, device="cuda"), torch.zeros((T, d), device="cuda")
        if kind == "step":
            st.handle.hx[:] = st.x.cpu().numpy()
            st.handle.hlogits[:] = st.logits.cpu().numpy()
            st.result = np.asarray(_View(st.owner, st.lib.nsl_moe_host_out(st.handle.h), (T, d), False))
    elif kind == "experts3":
        d, ff, E, k, T = (case[n] for n in ("d", "ff", "E", "k", "T"))
        st.gate, st.up, st.down = _Stack3(E, ff, d, gen), _Stack3(E, ff, d, gen), _Stack3(E, d, ff, gen)
        st.x, st.logits = _bf16((T, d), gen), torch.randn((T, E), generator=gen, device="cuda")
        st.ind, st.wt = torch.zeros((T, k), dtype=torch.int32, device="cuda"), torch.zeros((T, k), device="cuda")
        st.A, st.D, st.out = (torch.zeros(s, device="cuda") for s in ((T * k, ff), (T * k, d), (T, d)))
    elif kind in ("mv", "mm"):
        R, K, T = case["R"], case["K"], case["T"]
        if case["p"] == 3:
            st.fmt, st.keep = L.MF_SEED4, _Stack3(1, R, K, gen)
            st.w = st.keep.first
        else:
            st.fmt, st.keep = L.MF_SEED4P4, moe.ExpertStack.random_on_device(1, R, K, gen)
            st.w = L.WSlice()
            st.w.p[0], st.w.p[1], st.w.p[3], st.w.eb = st.keep.seeds.data_ptr(), st.keep.coefs.data_ptr(), st.keep.codes.data_ptr(), -22
        st.x, st.y = _bf16((T, K), gen), torch.zeros((T, R), device="cuda")
    elif kind == "head":
        R, K, T = case["R"], case["K"], case["T"]
        st.codes = torch.randint(-2 ** 31, 2 ** 31 - 1, (R, K // 8), generator=gen, device="cuda", dtype=torch.int32)
        st.scales = (torch.rand((R, K // 64), generator=gen, device="cuda") * 0.02 + 0.001).to(torch.bfloat16)
        st.biases = (torch.rand((R, K // 64), generator=gen, device="cuda") * -0.2).to(torch.bfloat16)
        # a row of activations leans towards the weights of the token that follows, so that one logit stands out as in a trained model
        tok = torch.randint(0, R, (T,), generator=gen, device="cuda")
        q = (st.codes[tok].unsqueeze(-1) >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)) & 15
        w = q.reshape(T, K).float() * st.scales[tok].float().repeat_interleave(64, 1) + st.biases[tok].float().repeat_interleave(64, 1)
        st.x = (torch.randn((T, K), generator=gen, device="cuda") + 16.0 * w / w.norm(dim=1, keepdim=True)).to(torch.bfloat16).float()
        st.w = L.WSlice()
        st.w.p[0], st.w.p[1], st.w.p[2] = st.codes.data_ptr(), st.scales.data_ptr(), st.biases.data_ptr()
        st.y, st.tokens = torch.zeros((T, R), device="cuda"), torch.zeros(T, dtype=torch.int32, device="cuda")
    elif kind == "attn":
        T, n_kv, ctx, nh = case["T"], case["n_kv"], case["ctx"], case["n_kv"] * case["group"]
        lens = (torch.rand(T, generator=gen, device="cuda") * 0.5 + 0.5).mul(ctx).int().clamp(min=1).tolist()
        rows = T * ctx
        if case["q8"]:
            st.kv = [torch.randint(-127, 128, (rows, n_kv, 128), generator=gen, device="cuda", dtype=torch.int32).to(torch.int8) for _ in range(2)]
            st.kv += [torch.rand((rows, n_kv), generator=gen, device="cuda") * 0.02 + 0.005 for _ in range(2)]
        else:
            st.kv = [torch.randn((rows, n_kv, 128), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2)]
        st.view = L.KvView()
        st.view.a.k, st.view.a.v = st.kv[0].data_ptr(), st.kv[1].data_ptr()
        if case["q8"]:
            st.view.a.ks, st.view.a.vs = st.kv[2].data_ptr(), st.kv[3].data_ptr()
        st.view.nv, st.view.fmt = rows, int(case["q8"])
        st.args = L.AttnArgs(nh, n_kv, 128, SPLITS, 1.0 / math.sqrt(128.0))
        st.ri = dec.row_info([n - 1 for n in lens], [t * ctx for t in range(T)])
        st.q, st.o = _bf16((T, nh, 128), gen), torch.zeros((T, nh, 128), device="cuda")
        st.g = _bf16((T, nh, 128), gen) if case["gate"] else None
        st.part = torch.zeros(T * nh * SPLITS * 130, device="cuda")
    else:
        T, ctx = case["T"], case["ctx"]
        cfg = dec.make_cfg(case["layers"], 2048, 16, 2, case["E"], case["k"], 512, 512, case["vocab"], T, ctx, dense_bf16=int(case["dense_bf16"]))
        st.owner = _Owner(dec.random_decoder(cfg, seed=seed))
        st.handle = st.owner.handle
        n = T * ctx * 2 * 128
        for l in range(case["layers"]):
            k, v = (torch.randn(n, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
            torch.cuda.synchronize()
            st.handle.fill_cache(l, k, v)
        st.ids = torch.randint(0, case["vocab"], (T,), generator=gen, device="cuda", dtype=torch.int32)
        pos = torch.randint(ctx * 3 // 4, ctx, (T,), generator=gen, device="cuda").tolist()
        st.ri, st.next = dec.row_info(pos, [t * ctx for t in range(T)]), torch.zeros(T, dtype=torch.int32, device="cuda")
        h = C.c_void_p(st.handle.h)
        st.hidden = torch.as_tensor(_View(st.owner, st.lib.nsl_decoder_hidden(h), (T, 2048), True), device="cuda")
        st.lm = torch.as_tensor(_View(st.owner, st.lib.nsl_decoder_logits(h), (T, case["vocab"]), True), device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    c, lib = st.case, st.lib
    if st.kind == "moe":
        st.handle.forward_dev(st.x, st.logits, st.out)
        return st.out
    if st.kind == "step":
        st.handle.forward_pinned(c["T"])
        return st.result
    if st.kind == "experts3":
        d, ff, E, k, T = (c[n] for n in ("d", "ff", "E", "k", "T"))
        s = _stream()
        lib.nsl_route(s, E, k, _ptr(st.logits), E, _ptr(st.ind), _ptr(st.wt), T)
        lib.kc_mv_gu(s, L.MF_SEED4, _ptr(st.gate.table), _ptr(st.up.table), d, ff, _ptr(st.x), d, _ptr(st.A), ff, _ptr(st.ind), T * k, k, _ptr(st.G))
        lib.kc_mv_sel(s, L.MF_SEED4, _ptr(st.down.table), ff, d, _ptr(st.A), ff, _ptr(st.D), d, _ptr(st.ind), T * k, 1, _ptr(st.G))
        lib.kq4_moe_combine(s, d, k, _ptr(st.D), _ptr(st.wt), None, None, 0, _ptr(st.out), T)
        return {"out": st.out, "ind": st.ind, "wt": st.wt}
    if st.kind in ("mv", "mm"):
        fn = lib.kc_mv if st.kind == "mv" else lib.kc_mm
        fn(_stream(), st.fmt, st.w, c["K"], c["R"], _ptr(st.x), c["K"], _ptr(st.y), c["R"], c["T"], 0, _ptr(st.G))
        return st.y
    if st.kind == "head":
        s = _stream()
        lib.kc_mv(s, L.MF_Q4, st.w, c["K"], c["R"], _ptr(st.x), c["K"], _ptr(st.y), c["R"], c["T"], 0, None)
        lib.kc_argmax(s, _ptr(st.y), _ptr(st.tokens), c["R"], c["T"])
        return {"logits": st.y, "tokens": st.tokens}
    if st.kind == "attn":
        lib.kc_attn(_stream(), st.args, _ptr(st.q), st.view, _ptr(st.ri), _ptr(st.part), _ptr(st.g), _ptr(st.o), c["T"])
        return st.o
    # the tokens are the logits' arg-max, where a tie between two bf16 logits may fall either way: the logits are what is compared
    st.handle.step(st.ids, st.ri, c["T"], st.next)
    return {"hidden": st.hidden, "logits": st.lm}


def _distinct(E, k, T):
    """Expected number of experts that T rows of top-k routing touch."""
    return E * (1.0 - (1.0 - k / E) ** T)


def work(case):
    kind = case["kind"]
    T = case["T"]
    if kind in ("moe", "step", "experts3"):
        d, ff, E, k = case["d"], case["ff"], case["E"], case["k"]
        per_weight = 0.5 if kind == "experts3" else 0.5625
        return {"bytes": 3 * d * ff * per_weight * _distinct(E, k, T) + 4 * T * (2 * d + E), "flops": 2.0 * 3 * d * ff * T * k}
    if kind in ("mv", "mm"):
        R, K = case["R"], case["K"]
        return {"bytes": R * K * (0.5 if case["p"] == 3 else 0.5625) + 4 * T * (R + K), "flops": 2.0 * R * K * T}
    if kind == "head":
        R, K = case["R"], case["K"]
        return {"bytes": R * K * 0.5625 + 4 * T * (R + K), "flops": 2.0 * R * K * T}
    if kind == "attn":
        n_kv, nh, ctx = case["n_kv"], case["n_kv"] * case["group"], 0.75 * case["ctx"]
        return {"bytes": T * ctx * n_kv * 2 * (132 if case["q8"] else 256) + 8 * T * nh * 128, "flops": 4.0 * T * ctx * nh * 128}
    d, E, k, layers, vocab = 2048, case["E"], case["k"], case["layers"], case["vocab"]
    dense = 2 * 2048 * d + 2 * 256 * d + (E + 1) * d + 3 * 512 * d
    expert, ctx = 3 * d * 512, 0.875 * case["ctx"]
    per_layer = dense * (2 if case["dense_bf16"] else 0.5625) + expert * 0.5625 * _distinct(E, k, T) + T * ctx * 2 * 512
    return {"bytes": layers * per_layer + vocab * d * 0.5625 + 4 * T * (vocab + 2 * d),
            "flops": 2.0 * T * (layers * (dense + expert * k + 2 * ctx * 2048) + vocab * d)}


def tolerance(case):
    # bf16 rounding points on the way (activations after SwiGLU, every projection's result): another summation order moves
    # some of them by one bf16 unit
    if case["kind"] == "decoder":      # ... and the layers pass them on
        return {"rel": 1e-2, "max": 0.5}
    return {"rel": 5e-3, "max": 0.2}
