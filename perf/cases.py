"""What a user of this framework has it do, as cases that can be timed and compared.

Every case is one pass through the public entry points on seeded synthetic layers (any bit pattern is a valid trellis
stream and any 16-bit value a valid E8 index): single linears of both storage formats from one token to a long prompt,
a stack of decoder layers replayed from a CUDA graph, and one mixture-of-experts layer.  `exact` restates the
arithmetic in 64 bits with plain torch.
"""
import os

import numpy as np
import torch

import glq_b200
from glq_b200 import ops
from glq_b200.linear import GLQLinear
from glq_b200.plan import block_decompose

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


# ------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one attention projection of a small decoder, one token, called from Python: a decode step without graphs
        dict(name="trellis_1tok_2048x2048", kind="trellis", m=2048, n=2048, k1=4, k2=0, tokens=1, dtype="bf16"),
        # the module of a loaded model (nn.Module forward, power-of-two padded E8 layer), four sequences decoding
        dict(name="module_e8_4tok_2000x1536", kind="module", m=2000, n=1536, stages=2, tokens=4, dtype="fp16"),
        # the whole call: four decoder layers, one token, each projection reading the previous one's output, replayed
        # from a CUDA graph as a serving loop does (attention stands aside: its input is passed through)
        dict(name="layers_trellis_1tok", kind="layers", layers=4, hidden=2048, inter=11008, kv=512, k1=4, dtype="bf16"),
        # the widest projection of a larger decoder in E8 storage, one token: above the size of one L2-resident table
        dict(name="e8_1tok_14336x4096", kind="e8", m=14336, n=4096, stages=2, tokens=1, dtype="bf16"),
        # a batch of sixteen sequences decoding through a wide-input projection
        dict(name="e8_16tok_4096x14336", kind="e8", m=4096, n=14336, stages=2, tokens=16, dtype="bf16"),
        # two-stage trellis (6 bits per weight), an odd batch that is larger than one tile of sequences
        dict(name="trellis42_27tok_11008x2048", kind="trellis", m=11008, n=2048, k1=4, k2=2, tokens=27, dtype="fp16"),
        # a short ragged prompt through a wide-input projection
        dict(name="trellis_333tok_2048x11008", kind="trellis", m=2048, n=11008, k1=4, k2=0, tokens=333, dtype="fp16"),
        # a long prompt through the gate projection
        dict(name="trellis_2048tok_11008x2048", kind="trellis", m=11008, n=2048, k1=4, k2=0, tokens=2048, dtype="bf16"),
        # a long prompt through E8 storage, two stages
        dict(name="e8_2048tok_14336x4096", kind="e8", m=14336, n=4096, stages=2, tokens=2048, dtype="bf16"),
        # three stages, a ragged prompt, the widest input any configuration has
        dict(name="e8_700tok_5376x21504", kind="e8", m=5376, n=21504, stages=3, tokens=700, dtype="bf16"),
        # a mixture-of-experts layer: a batch of decoding sequences, and a long prompt
        dict(name="moe_256tok", kind="moe", experts=128, topk=8, hidden=2048, inter=768, k1=4, tokens=256, dtype="bf16"),
        dict(name="moe_4096tok", kind="moe", experts=128, topk=8, hidden=2048, inter=768, k1=4, tokens=4096, dtype="bf16"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    def width(step, lo=512, hi=21504):
        return max(step, log_int(lo, hi) // step * step)

    kind = rng.choice(["trellis", "trellis", "e8", "e8", "module", "layers", "moe"])
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    if kind in ("trellis", "e8", "module"):
        while True:
            tokens = rng.choice([1, 1, 2, 3, 8, log_int(1, 64), log_int(9, 64), log_int(65, 2048), log_int(129, 2048), 2048])
            if kind == "module":
                tokens = min(tokens, 64)
                m, n = log_int(256, 4096) // 8 * 8, log_int(256, 4096) // 8 * 8
            elif rng.random() < 0.5:
                m, n = rng.choice([(2048, 2048), (512, 2048), (11008, 2048), (2048, 11008), (4096, 4096), (1024, 4096),
                                   (14336, 4096), (4096, 14336), (5376, 4096), (4096, 5376)])
            else:
                step = 32 if kind == "trellis" else 64
                m, n = width(step), width(step)
            if 512 * 512 <= m * n <= 64_000_000 and tokens * m * n <= 2048 * 14336 * 4096:
                break
        if kind == "trellis":
            k1, k2 = rng.choice([(2, 0), (3, 0), (4, 0), (4, 0), (4, 2), (4, 4)])
            return dict(kind=kind, m=m, n=n, k1=k1, k2=k2, tokens=tokens, dtype=dtype)
        return dict(kind=kind, m=m, n=n, stages=rng.choice([1, 2, 2, 3]), tokens=tokens, dtype=dtype)
    if kind == "layers":
        hidden = 32 * rng.randint(32, 96)
        return dict(kind=kind, layers=rng.randint(1, 4), hidden=hidden, inter=32 * rng.randint(96, 344),
                    kv=32 * rng.randint(8, hidden // 64), k1=rng.choice([3, 4]), dtype=rng.choice(["bf16", "fp16"]))
    return dict(kind=kind, experts=rng.choice([32, 64, 128]), topk=rng.choice([2, 4, 8]), hidden=rng.choice([1024, 2048]),
                inter=rng.choice([512, 768]), k1=rng.choice([3, 4]), tokens=log_int(16, 4096), dtype=rng.choice(["bf16", "fp16"]))


# ------------------------------------------------------------------------------------------------------------------
# inputs: seeded streams, indices, signs and scales; activations N(0, 1)
# ------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _i16(g, *shape):
    return torch.randint(-32768, 32768, shape, generator=g, device="cuda", dtype=torch.int32).to(torch.int16)


def _signs(g, *shape):
    return (torch.randint(0, 2, shape, generator=g, device="cuda", dtype=torch.int32) * 2 - 1).to(torch.float16)


def _scale(g):
    return float((0.5 + torch.rand((), generator=g, device="cuda").item()) * 0.02)


def _randn(g, shape, dtype):
    return torch.randn(shape, generator=g, device="cuda").to(DTYPES[dtype])


_NIBBLES = None


def _codebook():
    """The (65536, 8) E8 shell codebook the package ships, as fp16."""
    global _NIBBLES
    if _NIBBLES is None:
        _NIBBLES = np.load(os.path.join(os.path.dirname(glq_b200.__file__), "data", "e8_shell_packed.npy")).view(np.uint32)
    nib = (_NIBBLES[:, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15
    return torch.from_numpy(nib.astype(np.float32) * 0.5 - 3.0).to("cuda", torch.float16)


def _trellis_layer(g, m, n, bits):
    return dict(m=m, n=n, codes=[_i16(g, (m // 16) * (n // 16), 16 * k) for k in bits], bits=bits, inv=0.21,
                su=_signs(g, m), sv=_signs(g, n), wscale=_scale(g))


def _e8_layer(g, m, n, stages):
    return dict(m=m, n=n, codes=[_i16(g, m, n // 8) for _ in range(stages)], inv=[0.1 ** (s + 1) for s in range(stages - 1)],
                su=_signs(g, m), sv=_signs(g, n), wscale=_scale(g))


def _stack(case, g):
    out = []
    h, i, kv, bits = case["hidden"], case["inter"], case["kv"], [case["k1"]]
    for _ in range(case["layers"]):
        d = dict(q=_trellis_layer(g, h, h, bits), k=_trellis_layer(g, kv, h, bits), v=_trellis_layer(g, kv, h, bits),
                 o=_trellis_layer(g, h, h, bits), gate=_trellis_layer(g, i, h, bits), up=_trellis_layer(g, i, h, bits),
                 down=_trellis_layer(g, h, i, bits))
        d["k"]["sv"] = d["v"]["sv"] = d["q"]["sv"]          # parts of a merged projection share their input signs
        d["up"]["sv"] = d["gate"]["sv"]
        d["norm1"], d["norm2"] = (1 + 0.1 * torch.randn(2, h, generator=g, device="cuda")).to(DTYPES[case["dtype"]])
        out.append(d)
    return out


def _experts(case, g):
    E, H, I, K = case["experts"], case["hidden"], case["inter"], case["k1"]
    return dict(w13=_i16(g, E, (2 * I // 16) * (H // 16), 16 * K), w2=_i16(g, E, (H // 16) * (I // 16), 16 * K),
                su13=_signs(g, E, 2 * I), sv13=_signs(g, H), su2=_signs(g, E, H), sv2=_signs(g, I),
                ws13=(0.5 + torch.rand(E, generator=g, device="cuda")) * 0.02,
                ws2=(0.5 + torch.rand(E, generator=g, device="cuda")) * 0.02)


def _inputs(case, seed):
    """(weights, activations) of a case: the same for prepare and exact."""
    g = _gen(seed)
    if case["kind"] == "trellis":
        w = _trellis_layer(g, case["m"], case["n"], [case["k1"]] + ([case["k2"]] if case["k2"] else []))
        return w, _randn(g, (case["tokens"], case["n"]), case["dtype"])
    if case["kind"] == "e8":
        return _e8_layer(g, case["m"], case["n"], case["stages"]), _randn(g, (case["tokens"], case["n"]), case["dtype"])
    if case["kind"] == "module":
        up2 = lambda v: 1 << (v - 1).bit_length()
        return (_e8_layer(g, up2(case["m"]), up2(case["n"]), case["stages"]),
                _randn(g, (case["tokens"], case["n"]), case["dtype"]))
    if case["kind"] == "layers":
        return _stack(case, g), _randn(g, (1, case["hidden"]), case["dtype"])
    w = _experts(case, g)
    x = _randn(g, (case["tokens"], case["hidden"]), case["dtype"])
    probs = torch.softmax(torch.randn(case["tokens"], case["experts"], generator=g, device="cuda"), -1)
    weights, ids = torch.topk(probs, case["topk"], dim=-1)
    return w, (x, ids, (weights / weights.sum(-1, keepdim=True)).float().contiguous())


def _forward_stack(stack, x):
    """One token through the stack: norm + q/k/v, o + residual, norm + gate/up, activation + down + residual."""
    h = x.clone()
    qkvs = []
    lin = lambda L, a, **kw: ops.fused_linear_trellis_3inst(a, L["sv"], L["su"], L["codes"][0], None, None, None, None,
                                                           L["wscale"], L["n"], L["m"], L["n"], L["m"], **kw)
    part = lambda L: (L["su"], L["codes"][0], None, L["wscale"], 0.0, L["m"])
    for d in stack:
        qkv = ops.fused_linear_trellis_3inst_shards(h, d["q"]["sv"], [part(d[p]) for p in ("q", "k", "v")],
                                                    in_norm_weight=d["norm1"])
        lin(d["o"], qkv[:, :d["q"]["m"]], accumulate_into=h)
        gu = ops.fused_linear_trellis_3inst_shards(h, d["gate"]["sv"], [part(d[p]) for p in ("gate", "up")],
                                                   in_norm_weight=d["norm2"])
        lin(d["down"], gu, gated_act=0, accumulate_into=h)
        qkvs.append(qkv)
    return [h] + qkvs


def prepare(case, seed):
    w, x = _inputs(case, seed)
    state = dict(case=case, w=w, x=x)
    if case["kind"] in ("trellis", "e8"):
        # the block lists as the reference's callers hold them: host tensors made at load time
        state["bn"], state["bm"] = torch.tensor(block_decompose(w["n"])), torch.tensor(block_decompose(w["m"]))
    if case["kind"] == "e8":
        cb, tail = _codebook(), []
        for s in range(1, 4):
            tail += [w["codes"][s], cb, w["inv"][s - 1]] if s < case["stages"] else [None, None, 0.0]
        state["cb"], state["tail"] = cb, tail
    elif case["kind"] == "module":
        mod = GLQLinear(case["n"], case["m"])
        sd = {"SU": w["su"], "SV": w["sv"], "Wscale": torch.tensor(w["wscale"])}
        for s, q in enumerate(w["codes"]):
            sd["Qidxs" + (str(s + 1) if s else "")] = q
        for s, v in enumerate(w["inv"]):
            sd["inv_resid_scale" + (str(s + 1) if s else "")] = torch.tensor(v)
        mod.load_state_dict(sd, strict=False)
        mod.to("cuda")
        cb = _codebook()
        mod.set_codebook(cb, cb)
        state["module"] = mod
    elif case["kind"] == "layers":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _forward_stack(w, x)
            _forward_stack(w, x)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["out"] = _forward_stack(w, x)
        state["graph"] = graph
    elif case["kind"] == "moe":
        bl = lambda v: torch.tensor(block_decompose(v))
        H, I = case["hidden"], case["inter"]
        state["blocks"] = (bl(H), bl(2 * I), None, None, bl(I), bl(H), None, None)
        state["none"] = torch.zeros(case["experts"], 1, 1, dtype=torch.int16, device="cuda")
    return state


def run(state):
    case, w, x = state["case"], state["w"], state["x"]
    kind = case["kind"]
    if kind == "trellis":
        if case["k2"]:
            return ops.fused_linear_trellis_3inst_rvq2(x, w["sv"], w["su"], w["codes"][0], w["codes"][1], state["bn"], state["bm"],
                                                       None, None, w["wscale"], w["inv"], w["n"], w["m"], w["n"], w["m"])
        return ops.fused_linear_trellis_3inst(x, w["sv"], w["su"], w["codes"][0], state["bn"], state["bm"], None, None,
                                              w["wscale"], w["n"], w["m"], w["n"], w["m"])
    if kind == "e8":
        return ops.fused_linear_block_diag(x, w["sv"], w["su"], w["codes"][0], state["cb"], w["wscale"], w["n"], w["m"], w["n"],
                                           w["m"], state["bn"], state["bm"], None, None, *state["tail"])
    if kind == "module":
        return state["module"](x)
    if kind == "layers":
        state["graph"].replay()
        return state["out"]
    xs, ids, weights = x
    H, I = case["hidden"], case["inter"]
    return ops.fused_moe_trellis_3inst(xs, ids, weights, w["w13"], state["none"], w["su13"], w["sv13"], w["ws13"], w["ws13"],
                                       w["w2"], state["none"], w["su2"], w["sv2"], w["ws2"], w["ws2"], H, I, 2 * I, H, 2 * I, I, H,
                                       *state["blocks"], 1)


# ------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
def work(case):
    es = 4 if case["dtype"] == "fp32" else 2
    linear = lambda m, n, bpw, t: dict(bytes=m * n * bpw / 8 + t * (m + n) * es + 2 * (m + n), flops=2 * t * m * n)
    kind = case["kind"]
    if kind == "trellis":
        return linear(case["m"], case["n"], case["k1"] + case["k2"], case["tokens"])
    if kind == "e8":
        d = linear(case["m"], case["n"], 2 * case["stages"], case["tokens"])
        return dict(bytes=d["bytes"] + 65536 * 4, flops=d["flops"])
    if kind == "module":
        up2 = lambda v: 1 << (v - 1).bit_length()
        d = linear(up2(case["m"]), up2(case["n"]), 2 * case["stages"], 0)
        return dict(bytes=d["bytes"] + 65536 * 4 + case["tokens"] * (case["m"] + case["n"]) * es,
                    flops=2 * case["tokens"] * up2(case["m"]) * up2(case["n"]))
    if kind == "layers":
        h, i, kv = case["hidden"], case["inter"], case["kv"]
        parts = [linear(h + 2 * kv, h, case["k1"], 1), linear(h, h, case["k1"], 1), linear(2 * i, h, case["k1"], 1),
                 linear(h, i, case["k1"], 1)]
        return {k: case["layers"] * sum(p[k] for p in parts) for k in ("bytes", "flops")}
    H, I, E, T, J = case["hidden"], case["inter"], case["experts"], case["tokens"], case["topk"]
    used = E * (1 - (1 - J / E) ** T)                         # experts that some token is routed to
    return dict(bytes=used * 3 * H * I * case["k1"] / 8 + 2 * T * H * es + T * J * 12, flops=2 * T * J * 3 * H * I)


def tolerance(case):
    # Four times the error against `exact` (measured: bf16 1.7e-3, fp16 2.9e-4, fp32 1.9e-4; experts 1.8e-3 / 6e-4;
    # the last of four layers 8.6e-3): rotated activations are fp16 and sums fp32, a 16-bit result adds its rounding.
    if case["kind"] == "layers":
        return {"rel": 0.03}
    if case["kind"] == "moe":
        return {"rel": 7e-3 if case["dtype"] == "bf16" else 2.5e-3}
    return {"rel": {"bf16": 7e-3, "fp16": 1.2e-3, "fp32": 8e-4}[case["dtype"]]}


# ------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------------------------
def _fht(x, blocks):
    """Orthonormal block-diagonal Walsh-Hadamard transform of the last axis."""
    out, off = [], 0
    for b in blocks:
        v = x[..., off:off + b].reshape(-1, b)
        h = 1
        while h < b:
            v = v.reshape(-1, b // (2 * h), 2, h)
            v = torch.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]), 2).reshape(-1, b)
            h *= 2
        out.append((v / b ** 0.5).reshape(*x.shape[:-1], b))
        off += b
    return torch.cat(out, -1)


_LUT = None


def _lut():
    """Value of each of the 65,536 trellis states: a multiply-add hash whose halves are read as fp16 and added in fp16."""
    global _LUT
    if _LUT is None:
        s = np.arange(65536, dtype=np.uint64)
        r = ((((s * 89226354 + 64248484) & 0xFFFFFFFF) & 0x8FFF8FFF) ^ 0x3B603B60).astype(np.uint32)
        hi, lo = (r >> 16).astype(np.uint16).view(np.float16), (r & 0xFFFF).astype(np.uint16).view(np.float16)
        _LUT = torch.from_numpy((hi + lo).astype(np.float64)).cuda()
    return _LUT


def _trellis_weights(packed, m, n, k):
    """(m, n) weights of one packed stage.  Groups of 32 x 32 hold, per lane and 16 x 16 tile, k bytes of the tile's
    cyclic bit stream; weight j of a lane is the state at bit k * j of the lane's bytes."""
    by = packed.reshape(-1).view(torch.uint8).reshape(m // 32, n // 32, 32, 2, 2, k).to(torch.int64)
    c = sum(by[..., i] << (8 * i) for i in range(k))
    cn, cn2 = torch.roll(c, -1, 2), torch.roll(c, -2, 2)
    if k == 1:
        win, bits = (c << 16) | (cn << 8) | cn2, 24
    else:
        win, bits = (c << (8 * k)) | cn, 16 * k
    W = torch.empty(m // 32, 2, 2, 8, n // 32, 2, 2, 4, 2, dtype=torch.float64, device=c.device)   # R mi a g C ni c t e
    for j in range(8):
        v = _lut()[(win >> (bits - 16 - k * j)) & 0xFFFF].reshape(m // 32, n // 32, 8, 4, 2, 2)         # R C g t ni mi
        W[:, :, (j >> 1) & 1, :, :, :, (j >> 2) & 1, :, j & 1] = v.permute(0, 5, 2, 1, 4, 3)
    return W.reshape(m, n)


def _trellis_dense(L):
    W = _trellis_weights(L["codes"][0], L["m"], L["n"], L["bits"][0])
    if len(L["codes"]) > 1:
        W += L["inv"] * _trellis_weights(L["codes"][1], L["m"], L["n"], L["bits"][1])
    return W


def _rotated(x, W, L, blocks_n, blocks_m):
    return L["su"].double() * _fht(L["wscale"] * (_fht(x * L["sv"].double(), blocks_n) @ W.t()), blocks_m)


def _trellis_linear(x, L):
    return _rotated(x, _trellis_dense(L), L, block_decompose_64(L["n"]), block_decompose_64(L["m"]))


def block_decompose_64(n):
    return [1 << b for b in range(n.bit_length() - 1, -1, -1) if n >> b & 1]


def exact(case, seed):
    w, x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "trellis":
        return _trellis_linear(x.double(), w)
    if kind in ("e8", "module"):
        cb = _codebook().double()
        W = torch.zeros(w["m"], w["n"], dtype=torch.float64, device="cuda")
        for s, q in enumerate(w["codes"]):
            W += (w["inv"][s - 1] if s else 1.0) * cb[q.long() & 0xFFFF].reshape(w["m"], w["n"])
        if kind == "e8":
            return _rotated(x.double(), W, w, block_decompose_64(w["n"]), block_decompose_64(w["m"]))
        padded = torch.nn.functional.pad(x.double(), (0, w["n"] - case["n"]))
        return _rotated(padded, W, w, [w["n"]], [w["m"]])[:, :case["m"]]
    if kind == "layers":
        norm = lambda v, g: v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-6) * g.double()
        h, qkvs = x.double(), []
        for d in w:
            a = norm(h, d["norm1"])
            qkv = torch.cat([_trellis_linear(a, d[p]) for p in ("q", "k", "v")], -1)
            h = h + _trellis_linear(qkv[:, :case["hidden"]], d["o"])
            a = norm(h, d["norm2"])
            h = h + _trellis_linear(torch.nn.functional.silu(_trellis_linear(a, d["gate"])) * _trellis_linear(a, d["up"]), d["down"])
            qkvs.append(qkv)
        return [h] + qkvs
    xs, ids, weights = x
    H, I = case["hidden"], case["inter"]
    y = torch.zeros(case["tokens"], H, dtype=torch.float64, device="cuda")
    for e in range(case["experts"]):
        tok, j = torch.nonzero(ids == e, as_tuple=True)
        if not tok.numel():
            continue
        L13 = dict(m=2 * I, n=H, codes=[w["w13"][e]], bits=[case["k1"]], su=w["su13"][e], sv=w["sv13"], wscale=w["ws13"][e].double())
        L2 = dict(m=H, n=I, codes=[w["w2"][e]], bits=[case["k1"]], su=w["su2"][e], sv=w["sv2"], wscale=w["ws2"][e].double())
        gu = _trellis_linear(xs[tok].double(), L13)
        a = torch.nn.functional.gelu(gu[:, :I], approximate="tanh") * gu[:, I:]
        y.index_add_(0, tok, weights[tok, j].double()[:, None] * _trellis_linear(a, L2))
    return y
