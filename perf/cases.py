"""What a program built on this library has it do, as measurable cases: decode steps, output heads, prompt projections,
feed-forward blocks and mixture-of-experts blocks, each through the package's public calls.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) weights, activations and buffers on the GPU, made from the seed
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    tolerance(case)     how far another correct implementation may be

Every kind of case is a dict with "kind" and its sizes:

    decode  one dense transformer layer's projections for 1..8 token rows (no attention: its output is stood in for by the
            query columns): norm, Q | K | V, O, norm, gate | up, SwiGLU, down.  "down" is the type of the down projection:
            mixed files keep it in Q6_K.  "post_norm": the residual additions carry a norm of their own.
    head    the output head over the vocabulary for 1..8 rows, with a logit soft-cap where "cap" is set
    gemm    one projection of a prompt chunk: quantise T rows, multiply
    ffn     the feed-forward block of a prompt chunk: norm, gate | up with the SwiGLU product, down added to the residual
    moe     a mixture-of-experts block from the router's logits to the residual
"""
import math

import torch

import arcinferzero_b200 as izb

Q4_0, Q8_0, Q4_K, Q5_K, Q6_K, IQ4_XS = izb.Q4_0, izb.Q8_0, izb.Q4_K, izb.Q5_K, izb.Q6_K, izb.IQ4_XS
FILE_BYTES = {Q4_0: 144, Q8_0: 272, Q4_K: 144, Q5_K: 176, Q6_K: 210, IQ4_XS: 136}  # of 256 weights
EPS = 1e-6
MOST_OPS = 2.0 * 8192 * 17408 * 5120      # of a drawn case: the largest listed projection's
MOST_WEIGHT_BYTES = 700e6                 # of a drawn case (the largest listed head holds 826e6)


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a small dense model answering one request: eight short calls in a row
        {"name": "decode_small_q8", "kind": "decode", "T": 1, "E": 1024, "KV": 512, "F": 3072, "type": Q8_0, "down": Q8_0, "post_norm": False},
        # a large dense model answering one request: the weights of a layer stream once
        {"name": "decode_q4k", "kind": "decode", "T": 1, "E": 5120, "KV": 1024, "F": 17408, "type": Q4_K, "down": Q4_K, "post_norm": False},
        # five requests decoded together, mixed file (down projection in Q6_K), residual additions with their own norm
        {"name": "decode_batch5_mixed", "kind": "decode", "T": 5, "E": 4096, "KV": 1024, "F": 12288, "type": Q4_K, "down": Q6_K, "post_norm": True},
        # the output head of a Q8_0 file, one token
        {"name": "head_q8", "kind": "head", "T": 1, "N": 151936, "K": 5120, "type": Q8_0, "cap": 0.0},
        # the output head of a mixed file, three requests, soft-capped logits
        {"name": "head_q6k_batch3", "kind": "head", "T": 3, "N": 151936, "K": 5120, "type": Q6_K, "cap": 30.0},
        # a short question: one projection over few rows
        {"name": "prompt37_q4k", "kind": "gemm", "T": 37, "N": 5120, "K": 5120, "type": Q4_K},
        # one projection over an ordinary prompt chunk
        {"name": "prompt512_q8", "kind": "gemm", "T": 512, "N": 4096, "K": 4096, "type": Q8_0},
        # the down projection of a mixed file over a prompt
        {"name": "prompt300_q6k_down", "kind": "gemm", "T": 300, "N": 5120, "K": 17408, "type": Q6_K},
        # a long prompt's widest projection
        {"name": "prompt8192_q4k", "kind": "gemm", "T": 8192, "N": 17408, "K": 5120, "type": Q4_K},
        # a feed-forward block over a prompt of ragged length
        {"name": "ffn1000_q4k", "kind": "ffn", "T": 1000, "E": 5120, "F": 17408, "type": Q4_K, "down": Q4_K},
        # an expert block over a long prompt: tiles of 128 slots
        {"name": "moe4096_q4k", "kind": "moe", "T": 4096, "E": 2048, "F": 768, "NE": 128, "NU": 8, "type": Q4_K},
        # the same block for four requests decoded together: most experts see one token
        {"name": "moe4_q4k", "kind": "moe", "T": 4, "E": 2048, "F": 768, "NE": 128, "NU": 8, "type": Q4_K},
    ]


def _log(rng, lo, hi, unit=1):
    """A multiple of `unit` in [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / unit)) * unit))


def _rows_of(rng, lo, hi):
    """Token rows: any number, odd ones among them."""
    return _log(rng, lo, hi)


def _cols(rng, lo, hi):
    """Output columns: mostly whole multiples of 128 as in model files, sometimes the multiples of 16 that the split of a matrix
    over several devices leaves."""
    return _log(rng, lo, hi, 128 if rng.random() < 0.7 else 16)


def draw(rng):
    kind = rng.choices(["decode", "head", "gemm", "ffn", "moe"], [30, 12, 30, 10, 18])[0]
    while True:
        if kind == "decode":
            E = _log(rng, 512, 8192, 256)
            c = {"kind": kind, "T": rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8]), "E": E, "KV": rng.choice([256, 512, 1024]), "F": _log(rng, 2 * E, min(4 * E, 20480), 256),
                 "type": rng.choice([Q4_K, Q4_K, Q8_0]), "down": Q4_K, "post_norm": rng.random() < 0.3}
            c["down"] = rng.choice([Q6_K, c["type"]]) if c["type"] == Q4_K else c["type"]
        elif kind == "head":
            c = {"kind": kind, "T": rng.randint(1, 8), "N": _log(rng, 16000, 152000, 8), "K": _log(rng, 1024, 8192, 256), "type": rng.choice([Q8_0, Q6_K, Q4_K]),
                 "cap": rng.choice([0.0, 30.0])}
        elif kind == "gemm":
            c = {"kind": kind, "T": _rows_of(rng, 9, 8192), "N": _cols(rng, 256, 17408), "K": _log(rng, 512, 17408, 256),
                 "type": rng.choices([Q4_K, Q8_0, Q6_K, Q5_K, Q4_0, IQ4_XS], [40, 20, 20, 8, 6, 6])[0]}
        elif kind == "ffn":
            E = _log(rng, 1024, 5120, 256)
            c = {"kind": kind, "T": _rows_of(rng, 9, 4096), "E": E, "F": _log(rng, 2 * E, 17408, 256), "type": rng.choice([Q4_K, Q8_0]), "down": Q4_K}
            c["down"] = c["type"]
        else:
            NE = rng.choice([8, 16, 32, 64, 128])
            c = {"kind": kind, "T": _rows_of(rng, 1, 4096), "E": _log(rng, 1024, 4096, 256), "F": _log(rng, 512, 2048, 256), "NE": NE,
                 "NU": rng.randint(1, min(8, NE // 4)), "type": rng.choice([Q4_K, Q4_K, Q8_0])}
        if work(c)["flops"] <= MOST_OPS and _weight_bytes(c, c.get("NE")) <= MOST_WEIGHT_BYTES:
            return c


def _moe_tile(c):
    """Slots per tile, as a caller picks them: the per-tile kernels while an expert sees few tokens, else the grouped GEMM."""
    return 128 if c["T"] * c["NU"] >= 16 * c["NE"] else 8


# ------------------------------------------------------------------------------------------------ inputs
def _gguf_rows(qt, n, K, gen):
    """n rows of K weights in the file's block form, zero-mean, root-mean-square about 1 / sqrt(K); every quant and sub-scale uniform
    over its range.  Made on the GPU, handed over as host bytes."""
    nsb = K // 256
    R = n * nsb

    def f16(shape, lo, hi, scale):
        v = torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo
        return (v * scale).half().view(torch.uint8)

    b = torch.randint(0, 256, (R, FILE_BYTES[qt]), dtype=torch.uint8, generator=gen, device="cuda")
    s = 1.0 / math.sqrt(K)
    if qt in (Q4_K, Q5_K):  # fp16 d, dmin | 6-bit scales and mins | quants: d * sc * q - dmin * mn
        mean_q, rms = (7.5, 1.77) if qt == Q4_K else (15.5, 3.6)
        b[:, 0:2] = f16((R, 1), 0.0, 0.01, s / rms)
        b[:, 2:4] = f16((R, 1), 0.0, 0.01, mean_q * s / rms)
    elif qt == Q6_K:        # low nibbles | upper bits | 16 int8 scales | fp16 d
        b[:, 208:210] = f16((R, 1), 0.5, 1.5, s / 1400.0)
    elif qt == IQ4_XS:      # fp16 d | scale bits | codebook indices
        b[:, 0:2] = f16((R, 1), 0.5, 1.5, s / 1300.0)
    else:                   # Q8_0 / Q4_0: eight blocks of fp16 d | quants
        v = b.view(R, 8, -1)
        v[:, :, 0:2] = f16((R, 8, 1), 0.5, 1.5, s / (76.0 if qt == Q8_0 else 4.8))
    return b.view(n, -1).cpu().numpy()


def _randn(shape, gen, scale=1.0):
    return torch.randn(shape, generator=gen, device="cuda") * scale


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    c, st = case, {"case": dict(case)}

    def weight(qt, n, K, n_mats=1):
        return izb.Weight(qt, _gguf_rows(qt, n * n_mats, K, gen), n, K, n_mats=n_mats)

    def norm(K):
        return 1.0 + _randn((K,), gen, 0.1)

    def zeros(*shape):
        return torch.zeros(shape, dtype=torch.float32, device="cuda")

    T, Mp = c["T"], izb.pad_rows(c["T"])
    if c["kind"] == "decode":
        E, KV, F = c["E"], c["KV"], c["F"]
        st.update(qkv=weight(c["type"], E + 2 * KV, E), o=weight(c["type"], E, E), gu=weight(c["type"], 2 * F, E), down=weight(c["down"], E, F),
                  n1=norm(E), n2=norm(E), x=_randn((T, E), gen), b_qkv=zeros(Mp, E + 2 * KV), b_gu=zeros(Mp, 2 * F))
        if c["post_norm"]:
            st.update(p1=norm(E), p2=norm(E), n3=norm(E), b_o=zeros(T, E), b_d=zeros(T, E))
    elif c["kind"] == "head":
        x = _randn((T, c["K"]), gen)
        aq, asc, _ = izb.quantize_act(x)  # (the last norm's output, already quantised by the layer before)
        st.update(w=weight(c["type"], c["N"], c["K"]), aq=aq, asc=asc, logits=zeros(T, c["N"]))
    elif c["kind"] == "gemm":
        N, K = c["N"], c["K"]
        st.update(w=weight(c["type"], N, K), x=_randn((T, K), gen), out=zeros(Mp, N),
                  q=(torch.empty((Mp, K), dtype=torch.int8, device="cuda"), torch.empty((K // 32, Mp), dtype=torch.float32, device="cuda")))
    elif c["kind"] == "ffn":
        E, F = c["E"], c["F"]
        x = zeros(Mp, E)
        x[:T] = _randn((T, E), gen)
        st.update(gu=izb.gateup_weight(c["type"], _gguf_rows(c["type"], F, E, gen), _gguf_rows(c["type"], F, E, gen), F, E), down=weight(c["down"], E, F),
                  n=norm(E), x=x, h=zeros(Mp, F),
                  q=(torch.empty((Mp, F), dtype=torch.int8, device="cuda"), torch.empty((F // 32, Mp), dtype=torch.float32, device="cuda")))
    else:
        E, F, NE, qt = c["E"], c["F"], c["NE"], c["type"]
        if _moe_tile(c) == 128:
            st.update(wg=izb.gateup_weight(qt, _gguf_rows(qt, NE * F, E, gen), _gguf_rows(qt, NE * F, E, gen), F, E, n_mats=NE), wu=None)
        else:
            st.update(wg=weight(qt, F, E, NE), wu=weight(qt, F, E, NE))
        # (some experts are more popular than others)
        st.update(wd=weight(qt, E, F, NE), x=_randn((T, E), gen), n=norm(E), logits=_randn((T, NE), gen) + _randn((NE,), gen, 0.5))
    return st


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    c = st["case"]
    return {"decode": _run_decode, "head": _run_head, "gemm": _run_gemm, "ffn": _run_ffn, "moe": _run_moe}[c["kind"]](st, c)


def _run_decode(st, c):
    # The residual stream x is updated in place and runs on from pass to pass, as it does from layer to layer.
    T, E, F, x, qkv, gu = c["T"], c["E"], c["F"], st["x"], st["b_qkv"], st["b_gu"]
    aq, asc, _ = izb.rmsnorm_quant(x, st["n1"], EPS)
    izb.matmul(st["qkv"], aq, asc, T, out=qkv)
    aq, asc, _ = izb.quantize_act(qkv[:T, :E])
    if c["post_norm"]:
        izb.matmul(st["o"], aq, asc, T, out=st["b_o"])
        aq, asc = izb.add_norm_quant(x, st["b_o"], st["p1"], EPS, w2=st["n2"])
    else:
        izb.matmul(st["o"], aq, asc, T, out=x, acc=1)
        aq, asc, _ = izb.rmsnorm_quant(x, st["n2"], EPS)
    izb.matmul(st["gu"], aq, asc, T, out=gu)
    aq, asc, _ = izb.swiglu_quant(gu[:T], F)
    if c["post_norm"]:
        izb.matmul(st["down"], aq, asc, T, out=st["b_d"])
        izb.add_norm_quant(x, st["b_d"], st["p2"], EPS, w2=st["n3"])
    else:
        izb.matmul(st["down"], aq, asc, T, out=x, acc=1)
    return {"x": x, "qkv": qkv[:T], "gu": gu[:T]}


def _run_head(st, c):
    out = izb.matmul(st["w"], st["aq"], st["asc"], c["T"], out=st["logits"])
    if c["cap"]:
        izb.softcap_rows(out, c["T"], c["N"], c["cap"])
    return out


def _run_gemm(st, c):
    out, aq, _ = izb.quant_matmul(st["w"], st["x"], c["T"], out=st["out"], qout=st["q"])
    return {"out": out[:c["T"]], "aq": aq[:c["T"]]}


def _run_ffn(st, c):
    T, x, h = c["T"], st["x"], st["h"]
    aq, asc, _ = izb.rmsnorm_quant(x[:T], st["n"], EPS)
    izb.matmul(st["gu"], aq, asc, T, out=h, acc=3)
    izb.quant_matmul(st["down"], h[:T], T, out=x, acc=1, qout=st["q"])
    return {"x": x[:T], "h": h[:T]}


def _run_moe(st, c):
    T, NU, TM, x = c["T"], c["NU"], _moe_tile(c), st["x"]
    S = T * NU
    aq, asc, _ = izb.rmsnorm_quant(x, st["n"], EPS)
    ids, wts, counts = izb.moe_route(st["logits"], NU)
    _, tiles, max_tiles, stok, swt, inv = izb.moe_sort(ids, wts, counts, TM)
    h = izb.moe_gateup(st["wg"], st["wu"], aq, asc, tiles, max_tiles, TM, stok, S)
    hq, hsc, _ = izb.quantize_act(h)
    y = izb.moe_down(st["wd"], hq, hsc, tiles, max_tiles, TM, swt, S)
    izb.moe_combine(x, y, inv, NU)
    return {"x": x, "ids": ids, "wts": wts}


# ------------------------------------------------------------------------------------------------ what a pass needs
def _weight_bytes(c, experts=None):
    """Bytes of the weights in the file's form; of a mixture of experts, `experts` of them (default: as many as a pass is expected
    to reach when every token picks NU of NE at random)."""
    def wb(qt, n, K):
        return float(n) * K / 256 * FILE_BYTES[qt]
    if c["kind"] == "decode":
        E, KV, F, qt = c["E"], c["KV"], c["F"], c["type"]
        return wb(qt, 2 * E + 2 * KV + 2 * F, E) + wb(c["down"], E, F)
    if c["kind"] in ("head", "gemm"):
        return wb(c["type"], c["N"], c["K"])
    if c["kind"] == "ffn":
        return wb(c["type"], 2 * c["F"], c["E"]) + wb(c["down"], c["E"], c["F"])
    if experts is None:
        experts = c["NE"] * (1.0 - (1.0 - c["NU"] / c["NE"]) ** c["T"])
    return experts * (wb(c["type"], 2 * c["F"], c["E"]) + wb(c["type"], c["E"], c["F"]))


def work(case):
    c, T = case, case["T"]
    w = _weight_bytes(c)
    if c["kind"] == "decode":
        E, KV, F = c["E"], c["KV"], c["F"]
        # residual in and out, Q | K | V and gate | up out
        return {"bytes": w + 4.0 * T * (2 * E + E + 2 * KV + 2 * F), "flops": 2.0 * T * (E * (2 * E + 2 * KV) + 3.0 * E * F)}
    if c["kind"] == "head":
        return {"bytes": w + T * (1.125 * c["K"] + 4.0 * c["N"]), "flops": 2.0 * T * c["N"] * c["K"]}
    if c["kind"] == "gemm":
        return {"bytes": w + T * (4.0 * c["K"] + 1.125 * c["K"] + 4.0 * c["N"]), "flops": 2.0 * T * c["N"] * c["K"]}
    if c["kind"] == "ffn":
        return {"bytes": w + 4.0 * T * (2 * c["E"] + c["F"]), "flops": 6.0 * T * c["E"] * c["F"]}
    return {"bytes": w + 4.0 * T * (2 * c["E"] + c["NE"]), "flops": 6.0 * T * c["NU"] * c["E"] * c["F"]}


def tolerance(case):
    # One product: exact integer block sums, added up in f32.
    if case["kind"] in ("gemm", "head"):
        return {"rel": 1e-5}
    # Several products with their results requantised to int8 in between: f32 sums in another order (about 3e-7) move a few of
    # 1e5 values across a rounding boundary of the quantiser, and each of those changes by one step of its block's 127.
    return {"rel": 2e-4}
