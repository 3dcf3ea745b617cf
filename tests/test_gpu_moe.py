"""MoE grouped expert matmul on the GPU against the CPU oracle (per-expert decode + dense loop)."""
import numpy as np
import pytest
import torch

from oracle import glq_oracle as O

pytestmark = pytest.mark.gpu


def cuda(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t.to(dtype) if dtype is not None else t


def _make(rng, E, hidden, inter, K, K2=0):
    w13_out = 2 * inter
    def packed(m, n, k):
        return rng.integers(0, 65536, size=(E, (m // 16) * (n // 16), 16 * k), dtype=np.uint16).view(np.int16)
    sg = lambda *s: (rng.integers(0, 2, size=s) * 2 - 1).astype(np.float16)
    d = dict(w13=packed(w13_out, hidden, K), w2=packed(hidden, inter, K),
             w13_2=packed(w13_out, hidden, K2) if K2 else None, w2_2=packed(hidden, inter, K2) if K2 else None,
             su13=sg(E, w13_out), sv13=sg(hidden), su2=sg(E, hidden), sv2=sg(inter),
             ws13=(rng.uniform(0.5, 1.5, size=E) * 0.03).astype(np.float32),
             ws2=(rng.uniform(0.5, 1.5, size=E) * 0.03).astype(np.float32),
             inv13=np.full(E, 0.2, np.float32), inv2=np.full(E, 0.15, np.float32))
    return d, w13_out


def _oracle(d, x, ids, w, E, hidden, inter, w13_out, K, K2, act):
    W13, W2 = {}, {}
    def dec(p, p2, inv, e, m, n):
        if K2:
            return O.trellis_decode_layer_nstage([p[e], p2[e]], [K, K2], [1.0, float(inv[e])], m, n)
        return O.trellis_decode_layer(p[e], m, n, K).astype(np.float32)
    def f13(e, xb):
        if e not in W13:
            W13[e] = dec(d["w13"], d["w13_2"], d["inv13"], e, w13_out, hidden)
        y = O.linear_forward(xb, W13[e], d["su13"][e], d["sv13"], float(d["ws13"][e]))
        return y.astype(np.float16).astype(np.float32)
    def f2(e, hb):
        if e not in W2:
            W2[e] = dec(d["w2"], d["w2_2"], d["inv2"], e, hidden, inter)
        hb = hb.astype(np.float16).astype(np.float32)
        return O.linear_forward(hb, W2[e], d["su2"][e], d["sv2"], float(d["ws2"][e])).astype(np.float16).astype(np.float32)
    return O.moe_forward(x, ids, w, f13, f2, inter, act)


def _run(ops, d, x_t, ids_t, w_t, E, hidden, inter, w13_out, K2, act_code):
    sentinel = torch.zeros(E, 1, 1, dtype=torch.int16, device="cuda")
    bl = lambda n: torch.tensor(O.block_decompose(n))
    return ops.fused_moe_trellis_3inst(
        x_t, ids_t, w_t,
        cuda(d["w13"]), cuda(d["w13_2"]) if K2 else sentinel, cuda(d["su13"]), cuda(d["sv13"]), cuda(d["ws13"]), cuda(d["inv13"]),
        cuda(d["w2"]), cuda(d["w2_2"]) if K2 else sentinel, cuda(d["su2"]), cuda(d["sv2"]), cuda(d["ws2"]), cuda(d["inv2"]),
        hidden, inter, w13_out, hidden, w13_out, inter, hidden,
        bl(hidden), bl(w13_out), None, None, bl(inter), bl(hidden), None, None, act_code)


@pytest.mark.parametrize("K,K2", [(4, 0), (2, 0), (4, 2)])
@pytest.mark.parametrize("T,act", [(1, 1), (7, 0), (40, 1), (40, 2)])
def test_moe_vs_oracle(K, K2, T, act):
    from glq_b200 import ops
    E, hidden, inter, k = 8, 256, 96, 2
    rng = np.random.default_rng(K * 100 + K2 * 10 + T + act)
    d, w13_out = _make(rng, E, hidden, inter, K, K2)
    x = rng.standard_normal((T, hidden)).astype(np.float32)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = rng.random((T, k)).astype(np.float32)
    w /= w.sum(1, keepdims=True)
    x_t = cuda(x, torch.float16)
    y = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, K2, act)
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, K, K2, O.ACT_CODES[act])
    err = np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err <= 5e-3, err      # two chained layers with fp16 hand-offs (the reference's own gate is rtol=atol=2e-2)
    y2 = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, K2, act)
    assert torch.equal(y, y2)


def test_moe_skewed_routing_and_int32_ids():
    """Everything routed to two experts (many decode passes for one expert, empty experts elsewhere)."""
    from glq_b200 import ops
    E, hidden, inter, k, T = 16, 128, 64, 2, 70
    rng = np.random.default_rng(3)
    d, w13_out = _make(rng, E, hidden, inter, 4)
    x = rng.standard_normal((T, hidden)).astype(np.float32)
    ids = np.tile(np.array([[3, 11]], dtype=np.int64), (T, 1))
    w = rng.random((T, k)).astype(np.float32)
    x_t = cuda(x, torch.bfloat16)
    y = _run(ops, d, x_t, cuda(ids.astype(np.int32)), cuda(w), E, hidden, inter, w13_out, 0, 1)
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, 4, 0, "gelu_tanh")
    err = np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err <= 5e-3 + 2.0 ** -8, err


def test_moe_expert_roll_invariance():
    """Renaming the experts (rolling the stacked weights and the ids together) changes nothing."""
    from glq_b200 import ops
    E, hidden, inter, k, T = 8, 128, 64, 2, 9
    rng = np.random.default_rng(5)
    d, w13_out = _make(rng, E, hidden, inter, 4)
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = cuda(rng.random((T, k)).astype(np.float32))
    y = _run(ops, d, x_t, cuda(ids), w, E, hidden, inter, w13_out, 0, 0)
    d2 = {kk: (np.roll(v, 3, axis=0) if isinstance(v, np.ndarray) and v.shape[:1] == (E,) else v) for kk, v in d.items()}
    y2 = _run(ops, d2, x_t, cuda((ids + 3) % E), w, E, hidden, inter, w13_out, 0, 0)
    assert torch.equal(y, y2)


@pytest.mark.parametrize("K,K2", [(4, 0), (3, 0), (4, 2)])
@pytest.mark.parametrize("T,skew", [(200, False), (333, True)])
def test_moe_tensor_core_form(K, K2, T, skew, monkeypatch):
    """Many routed tokens per expert: both matmuls run on the tcgen05 GEMM kernel over a device-built work
    list.  Checked against the oracle, for determinism, and against the streaming form of the same step."""
    from glq_b200 import ops
    E, hidden, inter, k = 8, 256, 128, 2
    rng = np.random.default_rng(7000 + K * 100 + K2 * 10 + T)
    d, w13_out = _make(rng, E, hidden, inter, K, K2)
    x = rng.standard_normal((T, hidden)).astype(np.float32)
    if skew:      # two hot experts take most routings, one expert gets none
        p = np.array([0.45, 0.35, 0.05, 0.05, 0.04, 0.03, 0.03, 0.0])
        ids = np.stack([rng.choice(E, size=k, replace=False, p=p) for _ in range(T)]).astype(np.int64)
    else:
        ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = rng.random((T, k)).astype(np.float32)
    w /= w.sum(1, keepdims=True)
    x_t = cuda(x, torch.float16)
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, K, K2, O.ACT_CODES[1])
    outs = {}
    for form, min_avg in (("gemm", "1"), ("stream", "1000000")):
        monkeypatch.setenv("GLQB_MOE_GEMM_MIN_AVG", min_avg)
        ops.clear_caches()
        y = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, K2, 1)
        y2 = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, K2, 1)
        assert torch.equal(y, y2), form
        err = np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max()
        assert err <= 5e-3, (form, err)
        outs[form] = y.float()
    ops.clear_caches()
    # same math, different summation order (and one fp16 rounding of the folded second stage)
    rel = (outs["gemm"] - outs["stream"]).abs().max() / outs["stream"].abs().max()
    assert rel <= 4e-3, rel


def test_moe_zero_tokens_and_unrouted_tokens():
    """No tokens: empty result.  Routings with id -1 (what expert parallelism leaves for other ranks' experts)
    are skipped; a token whose routings are all skipped gets zeros."""
    from glq_b200 import ops
    E, hidden, inter, k = 8, 256, 96, 2
    rng = np.random.default_rng(4242)
    d, w13_out = _make(rng, E, hidden, inter, 4, 0)
    x0 = torch.zeros(0, hidden, dtype=torch.float16, device="cuda")
    y0 = _run(ops, d, x0, torch.zeros(0, k, dtype=torch.int64, device="cuda"),
              torch.zeros(0, k, dtype=torch.float32, device="cuda"), E, hidden, inter, w13_out, 0, 1)
    assert y0.shape == (0, hidden)
    T = 6
    x = rng.standard_normal((T, hidden)).astype(np.float32)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = rng.random((T, k)).astype(np.float32)
    x_t = cuda(x, torch.float16)
    full = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, 1).float()
    masked = ids.copy()
    masked[2, :] = -1                      # token 2: nothing routed here
    masked[4, 1] = -1                      # token 4: only its first routing
    y = _run(ops, d, x_t, cuda(masked), cuda(w), E, hidden, inter, w13_out, 0, 1).float()
    assert torch.count_nonzero(y[2]) == 0
    keep = [0, 1, 3, 5]
    assert torch.equal(y[keep], full[keep])
    only_first = ids.copy(); only_first[:, 1] = -1
    y_first = _run(ops, d, x_t, cuda(only_first), cuda(w), E, hidden, inter, w13_out, 0, 1).float()
    assert torch.equal(y[4], y_first[4])


def test_moe_large_step_uses_split_grouping():
    """More than 8192 routings: counting and placement run as many-CTA kernels around the table-building CTA."""
    from glq_b200 import ops
    E, hidden, inter, k, T = 8, 256, 128, 2, 4200
    rng = np.random.default_rng(9001)
    d, w13_out = _make(rng, E, hidden, inter, 4, 0)
    x = rng.standard_normal((T, hidden)).astype(np.float32)
    p = np.array([0.3, 0.25, 0.15, 0.1, 0.08, 0.07, 0.05, 0.0])
    ids = np.stack([rng.choice(E, size=k, replace=False, p=p) for _ in range(T)]).astype(np.int64)
    ids[17, 0] = -1                                   # a skipped routing in the middle
    w = rng.random((T, k)).astype(np.float32)
    w /= w.sum(1, keepdims=True)
    x_t = cuda(x, torch.float16)
    ops.clear_caches()
    y = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, 1)
    y2 = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, 1)
    assert torch.equal(y, y2)
    keep = ids >= 0
    ref = _oracle(d, x_t.float().cpu().numpy(), np.where(keep, ids, 7), np.where(keep, w, 0.0).astype(np.float32),
                  E, hidden, inter, w13_out, 4, 0, O.ACT_CODES[1])
    err = np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err <= 5e-3, err
    ops.clear_caches()


# sizes whose rows need more shared memory than the three-CTAs-per-SM budget (many short blocks: 8160, 8128, 4064), blocks
# of several 1024-value chunks on either side (8192, 4096, 3136 = 2048 + 1024 + 64, 1056), with routings in several passes
@pytest.mark.parametrize("form", ["1", "1000000"], ids=["gemm", "stream"])
@pytest.mark.parametrize("hidden,inter", [(8160, 64), (8128, 64), (8192, 64), (128, 4064), (128, 4096), (256, 3136), (4096, 1056)])
def test_moe_block_lists(hidden, inter, form, monkeypatch):
    from glq_b200 import ops
    monkeypatch.setenv("GLQB_MOE_GEMM_MIN_AVG", form)       # (sizes that are not multiples of 64 stream either way)
    E, k, T = 3, 2, 5
    rng = np.random.default_rng(hidden + inter)
    d, w13_out = _make(rng, E, hidden, inter, 2)
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = rng.random((T, k)).astype(np.float32)
    ops.clear_caches()
    y = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, 1)
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, 2, 0, O.ACT_CODES[1])
    err = np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max()
    ops.clear_caches()
    assert err <= 5e-3, err      # as above: two chained layers with fp16 hand-offs


@pytest.mark.parametrize("T", [13, 40, 255])
def test_moe_two_stages_keep_a_sum_per_stage(T, monkeypatch):
    """Below 64 routed tokens per expert two-stage experts run the streaming kernels, whose weights are exact and whose
    stages are summed in fp32 each (the GEMM multiplies fp16(w1 + s * w2)): the same bits as with that form forced."""
    from glq_b200 import ops
    E, hidden, inter, k = 8, 256, 128, 2
    rng = np.random.default_rng(8000 + T)
    d, w13_out = _make(rng, E, hidden, inter, 4, 2)
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = rng.random((T, k)).astype(np.float32)
    w /= w.sum(1, keepdims=True)
    outs = []
    for forced in (None, "1000000"):
        monkeypatch.delenv("GLQB_MOE_GEMM_MIN_AVG", raising=False)
        if forced:
            monkeypatch.setenv("GLQB_MOE_GEMM_MIN_AVG", forced)
        ops.clear_caches()
        outs.append(_run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 2, 1))
    ops.clear_caches()
    assert torch.equal(outs[0], outs[1])
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, 4, 2, O.ACT_CODES[1])
    assert np.abs(outs[0].float().cpu().numpy() - ref).max() <= 5e-3 * np.abs(ref).max()


def test_moe_even_tiles():
    """Routed tokens per expert at the edges of the token tiles of the tensor-core form: none, one, one step of 16 and one
    more, one whole tile of 192 and one more (two even tiles of 112 and 81), three tiles."""
    from glq_b200 import ops
    counts = [0, 1, 16, 17, 192, 193, 385, 0]
    E, hidden, inter, T = len(counts), 128, 64, sum(counts)
    rng = np.random.default_rng(77)
    d, w13_out = _make(rng, E, hidden, inter, 4)
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int64)[:, None]
    w = rng.random((T, 1)).astype(np.float32)
    ops.clear_caches()
    y = _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, 1)
    assert torch.equal(y, _run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, 1))
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, 4, 0, O.ACT_CODES[1])
    ops.clear_caches()
    assert np.abs(y.float().cpu().numpy() - ref).max() <= 5e-3 * np.abs(ref).max()


# routings around the share of a grouping CTA (256), of many CTAs (32 x 256), and past the one-launch form (65536), experts
# of about one and two token tiles (160 and 320): a token's
# result does not depend on the tokens around it.  inter 736 = 512 + 128 + 64 + 32: blocks of fewer values than a warp's chunk.
@pytest.mark.parametrize("T", [127, 128, 129, 640, 1281, 4096, 4097, 32767, 32768])
def test_moe_grouping_sizes(T, monkeypatch):
    from glq_b200 import ops
    monkeypatch.setenv("GLQB_MOE_GEMM_MIN_AVG", "0")
    E, hidden, inter, k = 8, 128, 736 if T < 5000 else 64, 2
    rng = np.random.default_rng(T)
    d, w13_out = _make(rng, E, hidden, inter, 4, 0)
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = np.argsort(rng.random((T, E)), axis=1)[:, :k].astype(np.int64)
    w = cuda(rng.random((T, k)).astype(np.float32))
    run = lambda a, b: _run(ops, d, x_t[a:b].contiguous(), cuda(ids[a:b]), w[a:b].contiguous(), E, hidden, inter, w13_out, 0, 1)
    ops.clear_caches()
    y = run(0, T)
    cut = T // 2 + 3
    assert torch.equal(y, torch.cat([run(0, cut), run(cut, T)]))
    ops.clear_caches()


@pytest.mark.parametrize("T", [5, 200])
def test_moe_plans_differ_by_every_argument(T):
    """Steps on the same packed weights with other signs, scales, second-stage scales or blocks give what fresh plans give."""
    from glq_b200 import ops
    E, hidden, inter, k = 8, 256, 128, 2
    rng = np.random.default_rng(T)
    d, w13_out = _make(rng, E, hidden, inter, 4, 2)
    o, _ = _make(rng, E, hidden, inter, 4, 2)
    d, o = ({key: cuda(v) for key, v in t.items()} for t in (d, o))
    x = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = cuda(np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64))
    w = cuda(rng.random((T, k)).astype(np.float32))
    bl = [O.block_decompose(v) for v in (hidden, w13_out, inter, hidden)]

    def call(t, b):
        return ops.fused_moe_trellis_3inst(x, ids, w, t["w13"], t["w13_2"], t["su13"], t["sv13"], t["ws13"], t["inv13"], t["w2"], t["w2_2"],
                                           t["su2"], t["sv2"], t["ws2"], t["inv2"], hidden, inter, w13_out, hidden, w13_out, inter, hidden,
                                           b[0], b[1], None, None, b[2], b[3], None, None, 0)
    o["ws13"], o["ws2"], o["inv13"], o["inv2"] = 2 * d["ws13"], 2 * d["ws2"], 2 * d["inv13"], 2 * d["inv2"]
    variants = [(d, bl)] + [(dict(d, **{key: o[key]}), bl) for key in ("w13_2", "su13", "sv13", "ws13", "inv13", "w2_2", "su2", "sv2", "ws2", "inv2")]
    variants += [(d, bl[:i] + [[bl[i][0] // 2] * 2] + bl[i + 1:]) for i in range(4)]
    ops.clear_caches()
    got = [call(*v) for v in variants]
    for v, y in zip(variants, got):
        ops.clear_caches()
        assert torch.equal(call(*v), y)
    assert not any(torch.equal(got[0], y) for y in got[1:])
    ops.clear_caches()


@pytest.mark.parametrize("E,hidden,inter,k,T,act", [(8, 256, 736, 2, 37, 1), (8, 256, 192, 3, 200, 0), (4, 128, 96, 2, 9, 4)])
def test_moe_between_the_matmuls_by_warps_and_by_ctas(E, hidden, inter, k, T, act, monkeypatch):
    """The two kernels between the matmuls give the oracle's result and each other's bits, over blocks of 32 to 1024 values, an odd
    number of slots, gated and plain activations, in the streaming and in the tensor-core form."""
    from glq_b200 import ops
    rng = np.random.default_rng(E + hidden + inter + T)
    d, w13_out = _make(rng, E, hidden, inter, 4, 0)
    if act > 2:
        w13_out = inter
        d["w13"], d["su13"] = d["w13"][:, :(w13_out // 16) * (hidden // 16)].copy(), d["su13"][:, :w13_out].copy()
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)
    w = rng.random((T, k)).astype(np.float32)
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, 4, 0, O.ACT_CODES[act])
    got = []
    for least in ("1", "1000000"):
        monkeypatch.setenv("GLQB_MOE_MID_WARP_MIN", least)
        ops.clear_caches()
        got.append(_run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, 0, act))
        assert np.abs(got[-1].float().cpu().numpy() - ref).max() <= 5e-3 * np.abs(ref).max()
    assert torch.equal(*got)
    ops.clear_caches()


@pytest.mark.parametrize("K2", [0, 2])
def test_moe_pairs_of_token_tiles(K2, monkeypatch):
    """Routed tokens per expert at the edges of tiles of 160 and of the pairs of tiles that an item takes.  inter 704 is eleven
    chunks of 64 columns (an odd number: the last pair of chunks is half) and blocks of 512, 128 and 64.  With two stages the
    GEMM multiplies fp16 sums of weights and the streaming form does not: other bits show which one ran."""
    from glq_b200 import ops
    counts = [0, 1, 16, 17, 159, 160, 161, 319, 320, 321, 480, 481, 640, 641]
    E, hidden, inter, T = len(counts), 128, 704, sum(counts)
    assert hidden % 64 == 0 and inter % 64 == 0              # else there is no tensor-core form
    rng = np.random.default_rng(78)
    d, w13_out = _make(rng, E, hidden, inter, 4, K2)
    x_t = cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16)
    ids = rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int64)[:, None]
    w = rng.random((T, 1)).astype(np.float32)
    got = []
    for least in ("0", "1000000"):
        monkeypatch.setenv("GLQB_MOE_GEMM_MIN_AVG", least)
        ops.clear_caches()
        got.append(_run(ops, d, x_t, cuda(ids), cuda(w), E, hidden, inter, w13_out, K2, 1))
    ops.clear_caches()
    ref = _oracle(d, x_t.float().cpu().numpy(), ids, w, E, hidden, inter, w13_out, 4, K2, O.ACT_CODES[1])
    for y in got:
        assert np.abs(y.float().cpu().numpy() - ref).max() <= 5e-3 * np.abs(ref).max()
    if K2:
        assert not torch.equal(*got)


@pytest.mark.parametrize("T", [6, 150])
def test_moe_steps_on_two_streams(T):
    """Steps of one layer that may overlap, in the streaming and the tensor-core form, then alone again."""
    from glq_b200 import ops
    E, hidden, inter, k = 8, 256, 128, 2
    rng = np.random.default_rng(T)
    d, w13_out = _make(rng, E, hidden, inter, 4)
    d = {key: cuda(v) if v is not None else None for key, v in d.items()}
    none, bl = torch.zeros(E, 1, 1, dtype=torch.int16, device="cuda"), [O.block_decompose(v) for v in (hidden, w13_out, inter, hidden)]
    steps = []
    for _ in range(2):
        steps.append((cuda(rng.standard_normal((T, hidden)).astype(np.float32), torch.float16),
                      cuda(np.stack([rng.permutation(E)[:k] for _ in range(T)]).astype(np.int64)), cuda(rng.random((T, k)).astype(np.float32))))
    call = lambda x, ids, w: ops.fused_moe_trellis_3inst(
        x, ids, w, d["w13"], none, d["su13"], d["sv13"], d["ws13"], d["inv13"], d["w2"], none, d["su2"], d["sv2"], d["ws2"], d["inv2"],
        hidden, inter, w13_out, hidden, w13_out, inter, hidden, bl[0], bl[1], None, None, bl[2], bl[3], None, None, 0)
    ops.clear_caches()
    refs = [call(*s) for s in steps]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in steps], [[], []]
    for _ in range(20):
        for i, s in enumerate(steps):
            with torch.cuda.stream(streams[i]):
                got[i].append(call(*s))
    torch.cuda.synchronize()
    ops.check_device_status()
    assert all(torch.equal(y, ref) for ys, ref in zip(got, refs) for y in ys)
    assert all(torch.equal(call(*s), ref) for s, ref in zip(steps, refs))
    ops.clear_caches()
