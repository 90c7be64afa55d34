"""The work that users of this package have it do, as measurable cases.

A case names a kind of call sequence and its sizes; ``prepare`` makes what a program holds before it calls (weights on the
GPU, inputs, argument dicts, for token-by-token decoding a recorded launch sequence), ``run`` makes the calls.

  gemm    one multiply with quantised or fp16 weights: a projection of a text encoder, a language model or a transformer
  mlp     the gated MLP block of a language model: row statistics, RMS-normed gate/up multiply with SwiGLU or GeGLU, down
          multiply added into the fp32 residual stream (up to 32 tokens: recorded once and replayed, as a decoding loop does)
  dit     the attention half of a diffusion transformer's block: LayerNorm statistics, modulated QKV projection with QK-norm,
          RoPE and head split, then the attention over those heads
  attn    attention by itself: a causal prefill with grouped heads, or a few new tokens over a key/value cache
  conv2d  a convolution of an image decoder: GroupNorm statistics, GroupNorm + SiLU + 3x3 convolution (strided or 2x upsampling
          without the norm as well)
  conv3   a 3x3x3 convolution over a video latent, whole or in chunks of frames, with or without the fused PixelNorm
"""
import math

import numpy as np
import torch

import p0pc0rn_kernels_b200 as P

ENC = {"q4": "q4g32a.t64", "q8": "q8g64s.t64", "f16": "f16"}
_context = None


def _gpu():
    """one context for the process, as a program has it"""
    global _context
    if _context is None:
        _context = P.createGpu()
    return _context


# ------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one projection of a text encoder over a short prompt: the smallest call, all latency
        {"name": "proj_q4_m64_1024", "kind": "gemm", "enc": "q4", "M": 64, "N": 1024, "K": 1024, "epi": "f16"},
        # a language model's MLP block, one token (single-user decoding), a small batch, and a prompt
        {"name": "mlp_q4_m1", "kind": "mlp", "enc": "q4", "M": 1, "hidden": 4096, "ffn": 14336, "act": "silu"},
        {"name": "mlp_q4_m16", "kind": "mlp", "enc": "q4", "M": 16, "hidden": 4096, "ffn": 14336, "act": "silu"},
        {"name": "mlp_q4_m512", "kind": "mlp", "enc": "q4", "M": 512, "hidden": 4096, "ffn": 14336, "act": "silu"},
        # a very wide projection for one token: nothing but the stream of weights
        {"name": "proj_q4_m1_16384", "kind": "gemm", "enc": "q4", "M": 1, "N": 16384, "K": 16384, "epi": "f16"},
        # a medium, ragged prompt through 8-bit weights: between the weight stream and the tensor cores
        {"name": "proj_q8_m130", "kind": "gemm", "enc": "q8", "M": 130, "N": 14336, "K": 4096, "epi": "f16"},
        # the largest multiply of the sweep: all tensor cores
        {"name": "proj_q4_m8192_16384", "kind": "gemm", "enc": "q4", "M": 8192, "N": 16384, "K": 16384, "epi": "f16"},
        # a 1280 x 720 image's 3600 tokens through the attention half of a transformer block
        {"name": "dit_q8_3600", "kind": "dit", "enc": "q8", "L": 3600, "heads": 24},
        # a causal prefill of ragged length with grouped key/value heads
        {"name": "attn_causal_1000", "kind": "attn", "Hq": 32, "Hkv": 8, "Lq": 1000, "Lk": 1000, "mode": 1, "nvalid": 1000},
        # one new token over a cache that is partly filled
        {"name": "attn_decode_4000", "kind": "attn", "Hq": 32, "Hkv": 8, "Lq": 1, "Lk": 4096, "mode": 2, "nvalid": 4000},
        # a residual block's convolution in an image decoder
        {"name": "conv2d_gn_128", "kind": "conv2d", "enc": "f16", "H": 128, "W": 128, "Ci": 512, "N": 512, "stride": 1, "gn": True, "up2": False},
        # a video latent of 13 frames, whole
        {"name": "conv3_clip_13", "kind": "conv3", "enc": "f16", "T": 13, "H": 92, "W": 160, "Ci": 128, "N": 128, "chunk": 0, "pn": False},
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, int(round(v / step)) * step)


def _draw(rng):
    kind = rng.choice(["gemm"] * 4 + ["mlp"] * 3 + ["attn"] * 2 + ["dit", "conv2d", "conv3"])
    if kind == "gemm":
        return {"kind": kind, "enc": rng.choice(["q4", "q4", "q8", "f16"]), "M": _log(rng, 1, 8192), "N": _log(rng, 512, 16384, 8), "K": _log(rng, 512, 16384, 64),
                "epi": rng.choice(["f16", "f16", "bias", "f32"])}
    if kind == "mlp":
        hidden = _log(rng, 1024, 8192, 128)
        return {"kind": kind, "enc": rng.choice(["q4", "q8"]), "M": _log(rng, 1, 2048), "hidden": hidden, "ffn": int(hidden * rng.uniform(2.5, 4.0) / 128) * 128,
                "act": rng.choice(["silu", "silu", "gelu"])}
    if kind == "attn":
        hkv = rng.choice([2, 4, 8, 16]); hq = hkv * rng.choice([1, 2, 4])
        if rng.random() < 0.5:
            lk = _log(rng, 128, 16384); return {"kind": kind, "Hq": hq, "Hkv": hkv, "Lq": _log(rng, 1, 64), "Lk": lk, "mode": 2, "nvalid": max(1, int(lk * rng.uniform(0.3, 1.0)))}
        l = _log(rng, 128, 8192); mode = rng.choice([0, 1, 2])
        return {"kind": kind, "Hq": hq, "Hkv": hkv, "Lq": l, "Lk": l, "mode": mode, "nvalid": l if mode < 2 else max(1, int(l * rng.uniform(0.5, 1.0)))}
    if kind == "dit":
        return {"kind": kind, "enc": rng.choice(["q4", "q8"]), "L": _log(rng, 128, 5000), "heads": rng.randrange(8, 33)}
    w = rng.randrange(16, 209); w = w if rng.random() < 0.5 else (w + 7) // 8 * 8       # a latent's width is often, not always, a multiple of 8
    ci, n = rng.choice([64, 128, 256, 512]), rng.choice([64, 128, 256, 512])
    if kind == "conv2d":
        form = rng.choice(["plain", "gn", "gn", "up2", "stride"])
        return {"kind": kind, "enc": rng.choice(["f16", "f16", "q8"]), "H": rng.randrange(8, 129) * 2, "W": w // 2 * 2, "Ci": ci, "N": n, "stride": 2 if form == "stride" else 1,
                "gn": form == "gn", "up2": form == "up2"}
    return {"kind": kind, "enc": rng.choice(["f16", "f16", "q8"]), "T": rng.randrange(1, 17), "H": rng.randrange(8, 121), "W": w, "Ci": ci, "N": n,
            "chunk": rng.choice([0, 0, 4]), "pn": rng.random() < 0.25}


def draw(rng):
    """a case of the same kinds over the whole range of sizes, at most as much work as the largest listed one"""
    while True:
        c = _draw(rng)
        if work(c)["flops"] <= (1e12 if c["kind"].startswith("conv") else 4.3e12):
            return c


# ------------------------------------------------------------------------------------------------------------- the inputs
def _pack_q4(w):
    """fp32 [rows][K] on the GPU -> q4g32a.t64 bytes (per row and 32 columns: fp16 minimum and scale, 4-bit codes)"""
    rows, k = w.shape
    v = w.view(rows // 64, 64, k // 32, 32).permute(0, 2, 1, 3)                          # tile, group, row, column
    mn = v.amin(3, keepdim=True).half().float()
    s = ((v.amax(3, keepdim=True) - mn) / 15.0).half().float()
    s = torch.where(s == 0, torch.ones_like(s), s)
    q = ((v - mn) / s).round_().clamp_(0, 15).to(torch.uint8)
    codes = q[..., 0::2] | (q[..., 1::2] << 4)
    sm = torch.cat([s.half(), mn.half()], 3).contiguous().view(torch.uint8)             # scale | min << 16
    return torch.cat([codes.reshape(rows // 64, k // 32, 1024), sm.reshape(rows // 64, k // 32, 256)], 2).reshape(-1)


def _pack_q8(w):
    """fp32 [rows][K] on the GPU -> q8g64s.t64 bytes (per row and 64 columns: an fp16 scale, 8-bit codes)"""
    rows, k = w.shape
    v = w.view(rows // 64, 64, k // 64, 64).permute(0, 2, 1, 3)
    s = (v.abs().amax(3, keepdim=True) / 127.0).half().float()
    s = torch.where(s == 0, torch.ones_like(s), s)
    q = (v / s).round_().clamp_(-128, 127).to(torch.int8).view(torch.uint8)
    return torch.cat([q.reshape(rows // 64, k // 64, 4096), s.half().contiguous().view(torch.uint8).reshape(rows // 64, k // 64, 128)], 2).reshape(-1)


class _State:
    """what a program keeps between calls: device memory, the argument dicts of its calls, perhaps their recording"""

    def __init__(self, seed):
        self.gpu = _gpu(); self.gen = torch.Generator(device="cuda"); self.gen.manual_seed(seed)
        self.tensors, self.buffers, self.calls, self.outputs, self.graph = [], [], [], [], None

    def randn(self, *shape, std=1.0, mean=0.0):
        return torch.empty(shape, device="cuda", dtype=torch.float32).normal_(mean, std, generator=self.gen)

    def buf(self, t):
        self.tensors.append(t)
        b = self.gpu.wrap(t.data_ptr(), t.numel() * t.element_size())
        self.buffers.append(b)
        return b

    def weight(self, enc, rows, cols, std=0.02):
        """a weight for gemm's `w`: N(0, std), quantised; quantised encodings hold whole tiles of 64 rows"""
        if enc != "f16": rows = -(-rows // 64) * 64
        parts = []
        for r0 in range(0, rows, 4096):
            w = self.randn(min(4096, rows - r0), cols, std=std)
            parts.append(w.half().view(torch.uint8).reshape(-1) if enc == "f16" else _pack_q4(w) if enc == "q4" else _pack_q8(w))
        b = self.buf(torch.cat(parts))
        return {"enc": ENC[enc], "buf": b, "off": 0, "bytes": b.size, "rows": rows, "cols": cols}

    def out(self, *shape, dtype=torch.float16):
        t = torch.zeros(shape, device="cuda", dtype=dtype)
        self.outputs.append(t)
        return self.buf(t)

    def call(self, op, args):
        self.calls.append((op, args))

    def go(self):
        for op, args in self.calls: op(self.gpu, args)

    def __del__(self):
        self.gpu.done()
        if self.graph is not None: self.graph.free()
        for b in self.buffers: self.gpu.free(b)


def _gemm_state(s, c):
    M, N, K = c["M"], c["N"], c["K"]
    a = {"w": s.weight(c["enc"], N, K), "x": {"buf": s.buf(s.randn(M, K).half())}, "M": M, "N": N, "K": K, "epi": c["epi"]}
    a["y"] = {"buf": s.out(M, N, dtype=torch.float32 if c["epi"] == "f32" else torch.float16)}
    if c["epi"] == "bias": a["ev"] = {"buf": s.buf(s.randn(N, std=0.1))}
    s.call(P.gemm, a)


def _mlp_state(s, c):
    M, D, F = c["M"], c["hidden"], c["ffn"]
    x = s.randn(M, D); xb = s.buf(x); st = s.buf(torch.zeros(M, 2, device="cuda"))
    gamma = s.buf(s.randn(D, std=0.1, mean=1.0))
    h = s.out(M, F)
    s.outputs.append(x)
    s.call(P.rowstats, {"x": {"buf": xb}, "rows": M, "cols": D, "mode": "rms", "eps": 1e-6, "st": {"buf": st}})
    s.call(P.gemm, {"w": s.weight(c["enc"], 2 * F, D), "x": {"buf": xb, "mode": "rms"}, "y": {"buf": h, "ld": F}, "M": M, "N": 2 * F, "K": D, "wr0": 0, "wr1": F,
                    "epi": "swiglu", "act": c["act"], "stats": {"buf": st}, "pv": {"buf": gamma}})
    s.call(P.gemm, {"w": s.weight(c["enc"], D, F), "x": {"buf": h}, "y": {"buf": xb}, "M": M, "N": D, "K": F, "epi": "resadd"})
    if M <= 32:
        keep = x.clone()
        torch.cuda.synchronize()
        s.go(); s.graph = s.gpu.record(s.go)          # (the first pass sizes the library's scratch memory)
        s.gpu.done(); x.copy_(keep)


def _dit_state(s, c):
    L, H = c["L"], c["heads"]; D = 128 * H
    x = s.buf(s.randn(L, D)); st = s.buf(torch.zeros(L, 2, device="cuda"))
    mod = s.buf(s.randn(2, D, std=0.5).half().float())
    norm = s.buf(s.randn(256, std=0.1, mean=1.0))
    ang = torch.rand(L, 64, device="cuda", generator=s.gen) * (2 * math.pi)
    rope = s.buf(torch.stack([torch.cos(ang), torch.sin(ang)], -1).contiguous())
    qkv = s.out(3, H, L, 128)
    n = H * L * 256
    s.call(P.rowstats, {"x": {"buf": x}, "rows": L, "cols": D, "mode": "ln", "eps": 1e-6, "st": {"buf": st}})
    s.call(P.gemm, {"w": s.weight(c["enc"], 3 * D, D), "x": {"buf": x, "mode": "lnmod"}, "y": {"buf": qkv}, "M": L, "N": 3 * D, "K": D, "epi": "heads", "stats": {"buf": st},
                    "pv": {"buf": mod, "off": 0, "stride": D}, "ev": {"buf": norm}, "heads": {"Ltot": L, "Hq": H, "Hkv": H, "rowOff": 0, "eps": 1e-6, "rope": {"buf": rope}}})
    s.call(P.attention, {"q": {"buf": qkv}, "k": {"buf": qkv, "off": n}, "v": {"buf": qkv, "off": 2 * n}, "o": {"buf": s.out(L, D)}, "Hq": H, "Hkv": H, "Lq": L, "Lk": L, "mode": 0})


def _attn_state(s, c):
    q = s.buf(s.randn(c["Hq"], c["Lq"], 128).half()); k = s.buf(s.randn(c["Hkv"], c["Lk"], 128).half()); v = s.buf(s.randn(c["Hkv"], c["Lk"], 128).half())
    s.call(P.attention, {"q": {"buf": q}, "k": {"buf": k}, "v": {"buf": v}, "o": {"buf": s.out(c["Lq"], c["Hq"] * 128)}, "Hq": c["Hq"], "Hkv": c["Hkv"], "Lq": c["Lq"], "Lk": c["Lk"],
                         "mode": c["mode"], "nvalid": c["nvalid"]})


def _conv2d_shape(c):
    return (2 * c["H"], 2 * c["W"]) if c["up2"] else (c["H"] // c["stride"], c["W"] // c["stride"])


def _conv2d_state(s, c):
    H, W, Ci, N = c["H"], c["W"], c["Ci"], c["N"]; Ho, Wo = _conv2d_shape(c)
    x = s.buf(s.randn(H, W, Ci).half()); bias = s.buf(s.randn(N, std=0.1))
    a = {"w": s.weight(c["enc"], N, 9 * Ci, std=0.03), "x": {"buf": x}, "y": {"buf": s.out(Ho, Wo, N)}, "M": Ho * Wo, "N": N, "K": 9 * Ci, "epi": "bias", "ev": {"buf": bias},
         "conv": {"kind": "conv", "Hi": H, "Wi": W, "Ci": Ci, "Ho": Ho, "Wo": Wo, "stride": c["stride"], "padT": 1, "padL": 1, "ks": 3, "gn": c["gn"], "up2": c["up2"]}}
    if c["gn"]:
        part = s.buf(torch.zeros(P.gnPartBytes(H * W), device="cuda", dtype=torch.uint8))
        gb = s.buf(torch.cat([s.randn(Ci, std=0.2, mean=1.0), s.randn(Ci, std=0.3)])); ab = s.buf(torch.zeros(2 * Ci, device="cuda"))
        s.call(P.groupnormStats, {"x": {"buf": x}, "pix": H * W, "C": Ci, "part": part, "gb": {"buf": gb, "gOff": 0, "bOff": 4 * Ci}, "ab": {"buf": ab, "off": 0}, "eps": 1e-6})
        a["pv"] = {"buf": ab, "off": 0, "stride": Ci}
    s.call(P.gemm, a)


def _conv3_state(s, c):
    T, H, W, Ci, N = c["T"], c["H"], c["W"], c["Ci"], c["N"]
    x = s.buf(s.randn(T, H, W, Ci).half()); y = s.out(T, H, W, N); bias = s.buf(s.randn(N, std=0.1)); w = s.weight(c["enc"], N, 27 * Ci, std=0.03)
    st = s.buf(torch.zeros(T * H * W, device="cuda")) if c["pn"] else None
    if c["pn"]: s.call(P.pixstats, {"x": {"buf": x}, "V": T * H * W, "C": Ci, "eps": 1e-6, "r": {"buf": st}, "ro": 0})
    step = c["chunk"] if c["chunk"] and not c["pn"] else T
    for t0 in range(0, T, step):
        nf = min(step, T - t0); first = max(0, t0 - 1)                       # the chunk's clip begins one frame before its first output frame
        a = {"w": w, "x": {"buf": x, "off": first * H * W * Ci * 2}, "y": {"buf": y, "off": t0 * H * W * N * 2}, "M": nf * H * W, "N": N, "K": 27 * Ci, "epi": "bias", "ev": {"buf": bias},
             "conv": {"kind": "conv3", "Hi": H, "Wi": W, "Ci": Ci, "Ho": H, "Wo": W, "stride": T, "padT": t0, "padL": first, "ks": 1, "pn": c["pn"]}}
        if c["pn"]: a["stats"] = {"buf": st}
        s.call(P.gemm, a)


def prepare(case, seed):
    s = _State(seed)
    {"gemm": _gemm_state, "mlp": _mlp_state, "dit": _dit_state, "attn": _attn_state, "conv2d": _conv2d_state, "conv3": _conv3_state}[case["kind"]](s, case)
    torch.cuda.synchronize()                          # the inputs were made on torch's stream, the library has its own
    return s


def run(state):
    if state.graph is not None: state.graph.launch()
    else: state.go()
    return state.outputs


# ------------------------------------------------------------------------------------------------------------- the accounting
def _wbytes(enc, rows, cols):
    return rows * cols * {"q4": 0.625, "q8": 1.03125, "f16": 2.0}[enc]


def _attn_work(hq, hkv, lq, lk, mode, nvalid):
    n = np.minimum(nvalid, lk) if mode else lk
    seen = float(np.minimum(np.arange(1, lq + 1), n).sum()) if mode == 1 else float(lq) * float(n)      # (query, visible key) pairs
    return {"bytes": 256.0 * (2 * hq * lq + 2 * hkv * float(n)), "flops": 4.0 * 128 * hq * seen}


def work(case):
    c = case; kind = c["kind"]
    if kind == "gemm":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": _wbytes(c["enc"], N, K) + 2.0 * M * K + (4.0 if c["epi"] == "f32" else 2.0) * M * N, "flops": 2.0 * M * N * K}
    if kind == "mlp":
        M, D, F = c["M"], c["hidden"], c["ffn"]
        return {"bytes": 3 * _wbytes(c["enc"], D, F) + 8.0 * M * D + 2.0 * M * F, "flops": 6.0 * M * D * F}
    if kind == "dit":
        L, D = c["L"], 128 * c["heads"]; at = _attn_work(c["heads"], c["heads"], L, L, 0, L)
        return {"bytes": _wbytes(c["enc"], 3 * D, D) + 4.0 * L * D + 512.0 * L + 6.0 * L * D + 2.0 * L * D, "flops": 6.0 * L * D * D + at["flops"]}
    if kind == "attn":
        return _attn_work(c["Hq"], c["Hkv"], c["Lq"], c["Lk"], c["mode"], c["nvalid"])
    if kind == "conv2d":
        Ho, Wo = _conv2d_shape(c); K = 9 * c["Ci"]
        return {"bytes": 2.0 * c["H"] * c["W"] * c["Ci"] + _wbytes(c["enc"], c["N"], K) + 2.0 * Ho * Wo * c["N"], "flops": 2.0 * Ho * Wo * c["N"] * K}
    V, K = c["T"] * c["H"] * c["W"], 27 * c["Ci"]
    return {"bytes": 2.0 * V * c["Ci"] + _wbytes(c["enc"], c["N"], K) + 2.0 * V * c["N"], "flops": 2.0 * V * c["N"] * K}


def tolerance(case):
    """About four times what two kernels of this package that are both correct differ by (weights rounded to fp16 or used as codes
    and scales, sums in another order, probabilities in fp16): one multiply 3e-4 in the 2-norm and 1e-3 at most, two passes of the
    MLP block 7e-4 and 7e-3, attention 3.7e-4 and 4.4e-3, a convolution 5e-5 and 1e-3 (single values flip to the next fp16)"""
    return {"gemm": {"rel": 1.2e-3, "max": 5e-3}, "mlp": {"rel": 2.8e-3, "max": 2.8e-2}, "dit": {"rel": 1.5e-3, "max": 1.8e-2},
            "attn": {"rel": 1.5e-3, "max": 1.8e-2}, "conv2d": {"rel": 3e-4, "max": 5e-3}, "conv3": {"rel": 3e-4, "max": 5e-3}}[case["kind"]]
