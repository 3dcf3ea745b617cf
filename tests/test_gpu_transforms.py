"""The Hadamard transforms at the edges of their tiles: every block length from 1 to 32768 (8192 is one tile), ragged token
counts, padded and cut-off columns, rows that are not aligned for vector accesses, every activation type."""
import numpy as np
import pytest
import torch

from glq_b200 import ops

pytestmark = pytest.mark.gpu


def fht64(v, blocks):
    out, off = np.empty_like(v), 0
    for b in blocks:
        a, h = v[:, off:off + b].copy(), 1
        while h < b:
            a = a.reshape(len(v), b // (2 * h), 2, h)
            a = np.stack((a[:, :, 0] + a[:, :, 1], a[:, :, 0] - a[:, :, 1]), 2).reshape(len(v), b)
            h *= 2
        out[:, off:off + b] = a / np.sqrt(b)
        off += b
    return out


BLOCKS = [[1], [2], [4], [8, 4, 2, 1], [16], [32, 2], [64, 32, 8], [128], [256, 64], [1024, 512], [2048, 32], [4096], [8192, 256],
          [16384, 1024], [32768]]
ROUND = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("blocks", BLOCKS, ids=str)
def test_transform_blocks(blocks, dtype):
    g = torch.Generator(device="cuda").manual_seed(sum(blocks))
    total = sum(blocks)
    for tokens, cut, shift in ((1, 0, 0), (3, min(3, total - 1), 1), (67, 0, 3)):
        feat = total - cut
        signs = (torch.randint(0, 2, (total,), generator=g, device="cuda") * 2 - 1).half()
        # rows of feat + shift values: with shift != 0 they are not aligned for vector loads
        x = torch.randn(tokens, feat + shift, generator=g, device="cuda").to(dtype)[:, shift:]
        out = torch.full((tokens, total), float("nan"), device="cuda")
        ops.input_rht_blocks(x, signs, out, feat, total, blocks)
        xp = np.zeros((tokens, total))
        xp[:, :feat] = x.double().cpu().numpy()
        ref = fht64(xp * signs.double().cpu().numpy(), blocks)
        # at most 15 additions per value, each rounding to 2^-24 of a partial sum that stays below max |ref| * 16
        assert np.abs(out.double().cpu().numpy() - ref).max() <= 15 * 16 * 2.0 ** -24 * max(1.0, np.abs(ref).max())
        y = torch.full((tokens, feat + shift), float("nan"), dtype=dtype, device="cuda")
        ops.output_rht_blocks(out, signs, y[:, shift:], feat, total, blocks)
        ref = (fht64(out.double().cpu().numpy(), blocks) * signs.double().cpu().numpy())[:, :feat]
        err = np.abs(y[:, shift:].double().cpu().numpy() - ref)
        assert (err <= ROUND[dtype] * np.abs(ref) + 15 * 16 * 2.0 ** -24 * max(1.0, np.abs(ref).max())).all()


@pytest.mark.parametrize("tokens", [1, 5, 9, 33, 65, 200])
@pytest.mark.parametrize("shape", [(96, 160), (1312, 2080), (8224, 64), (64, 16416)], ids=str)
def test_linear_is_the_transforms_around_the_matrix(shape, tokens):
    """Whole linears whose block lists mix short, tile-sized and longer-than-tile blocks, through the streaming kernels'
    and the tensor-core path's activation layouts."""
    from glq_b200 import synth
    from glq_b200.plan import block_decompose
    m, n = shape
    g = torch.Generator(device="cuda").manual_seed(m + n + tokens)
    x = torch.randn(tokens, n, generator=g, device="cuda").half()
    L = synth.trellis_layer("t", m, n, [4], g, "cuda")
    W = ops.glq_decompress_trellis_3inst_cuda(L.codes[0], m, n).double().cpu().numpy()
    y = ops.fused_linear_trellis_3inst(x, L.sv, L.su, L.codes[0], None, None, None, None, L.wscale, n, m, n, m,
                                       out_dtype=torch.float32)
    _check(x, W, L, y, block_decompose(n), block_decompose(m))
    if n % 64 == 0 or tokens <= 64:
        table = synth.load_e8_table("cuda")
        E = synth.e8_layer("e", m, n, 2, table, g, "cuda")
        spec = E.spec(batch=ops.token_bucket(tokens), x_dtype=x.dtype, y_dtype=torch.float32)
        from glq_b200.plan import Plan
        plan = Plan([spec])
        xb = x.new_zeros((spec.batch, n))
        xb[:tokens] = x
        yb = torch.empty(spec.batch, m, device="cuda")
        plan.run(xb, yb)
        nib = (table.cpu().numpy().view(np.uint32)[:, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15
        cb = nib.astype(np.float64) * 0.5 - 3.0
        W = sum(s * cb[q.cpu().numpy().view(np.uint16)].reshape(m, n) for q, s in zip(E.codes, [1.0] + list(E.stage_scale)))
        _check(x, W, E, yb[:tokens], block_decompose(n), block_decompose(m))
        plan.close()


def _check(x, W, L, y, bn, bm):
    xr = fht64(x.double().cpu().numpy() * L.sv.double().cpu().numpy(), bn)
    ref = fht64((xr @ W.T) * L.wscale, bm) * L.su.double().cpu().numpy()
    # the rotated activations (and, above 64 tokens, two-stage weights) are fp16: 2e-3 of the largest output
    assert np.abs(y.double().cpu().numpy() - ref).max() <= 2e-3 * np.abs(ref).max()


def test_output_transform_beyond_32_bit_offsets():
    """131073 rows of 32768 sums: the last row starts 2^32 elements in.  Only its sums are written and only its result is
    looked at (six of the columns, so that the general body runs)."""
    tokens, m, out = 131073, 32768, 6
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 17 GiB")
    g = torch.Generator(device="cuda").manual_seed(5)
    src = torch.empty(tokens, m, device="cuda")
    src[0] = 1.0
    src[-1] = torch.randn(m, generator=g, device="cuda")
    signs = (torch.randint(0, 2, (m,), generator=g, device="cuda") * 2 - 1).half()
    y = torch.empty(tokens, out, device="cuda")
    ops.output_rht_blocks(src, signs, y, out, m, [8192] * 4)
    ref = (fht64(src[-1:].double().cpu().numpy(), [8192] * 4) * signs.double().cpu().numpy())[:, :out]
    err = np.abs(y[-1:].double().cpu().numpy() - ref).max()
    del src
    torch.cuda.empty_cache()
    assert err <= 13 * 16 * 2.0 ** -24 * max(1.0, np.abs(ref).max())      # as in test_transform_blocks, 13 stages


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("tokens", [1, 8, 9])
def test_wide_inputs_of_decode_steps(tokens, shift):
    """Input blocks of 8192 and 4096 values in front of the single-launch kernel (up to 8 tokens) and of the streaming ones
    (9), rows aligned for vector loads and not, both formats' activation layouts."""
    from glq_b200 import synth
    from glq_b200.plan import Plan, block_decompose
    m, n = 64, 12352                                        # 8192 + 4096 + 64
    g = torch.Generator(device="cuda").manual_seed(tokens + shift)
    x = torch.randn(tokens, n + shift, generator=g, device="cuda").half()[:, shift:]
    L = synth.trellis_layer("t", m, n, [4], g, "cuda")
    W = ops.glq_decompress_trellis_3inst_cuda(L.codes[0], m, n).double().cpu().numpy()
    y = ops.fused_linear_trellis_3inst(x, L.sv, L.su, L.codes[0], None, None, None, None, L.wscale, n, m, n, m,
                                       out_dtype=torch.float32)
    _check(x, W, L, y, block_decompose(n), block_decompose(m))
    table = synth.load_e8_table("cuda")
    E = synth.e8_layer("e", m, n, 1, table, g, "cuda")
    plan = Plan([E.spec(batch=tokens, x_dtype=x.dtype, y_dtype=torch.float32, x_stride=x.stride(0))])
    yb = torch.empty(tokens, m, device="cuda")
    plan.run(x, yb)
    plan.close()
    nib = (table.cpu().numpy().view(np.uint32)[:, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15
    W = (nib.astype(np.float64) * 0.5 - 3.0)[E.codes[0].cpu().numpy().view(np.uint16)].reshape(m, n)
    _check(x, W, E, yb, block_decompose(n), block_decompose(m))


@pytest.mark.parametrize("tokens", [1, 8, 9, 64])
@pytest.mark.parametrize("shape", [(16352, 64), (16416, 64), (64, 16352), (64, 16416)], ids=str)
def test_decode_steps_every_block_length(shape, tokens):
    """16352 has one block of every length from 32 to 8192, 16416 one that two tiles share: the transforms of decode calls,
    plain, behind a norm and behind an activation, with rows that are not aligned and results added to a residual."""
    from glq_b200 import synth
    from glq_b200.plan import block_decompose
    m, n = shape
    g = torch.Generator(device="cuda").manual_seed(m + tokens)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w = randn(tokens, 2 * n + 1)[:, 1:], 1 + 0.2 * randn(n)
    gate, up = x[:, :n].double(), x[:, n:].double()
    # (fp32 inputs: nothing is rounded between the steps)
    steps = [(x[:, :n], gate, {}),
             (x[:, :n], gate * torch.rsqrt(gate.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double(), dict(in_norm_weight=w, in_norm_eps=1e-5)),
             (x, torch.nn.functional.silu(gate) * up, dict(gated_act=0))]
    table = synth.load_e8_table("cuda")
    nib = (table.cpu().numpy().view(np.uint32)[:, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15
    cb = nib.astype(np.float64) * 0.5 - 3.0
    T = synth.trellis_layer("t", m, n, [4], g, "cuda")
    E = synth.e8_layer("e", m, n, 1, table, g, "cuda")
    half = torch.from_numpy(cb).to("cuda", torch.float16)
    none = (None, None, 0.0)
    forms = [(T, ops.glq_decompress_trellis_3inst_cuda(T.codes[0], m, n).double().cpu().numpy(),
              lambda a, **kw: ops.fused_linear_trellis_3inst(a, T.sv, T.su, T.codes[0], None, None, None, None, T.wscale,
                                                             n, m, n, m, **kw)),
             (E, cb[E.codes[0].cpu().numpy().view(np.uint16)].reshape(m, n),
              lambda a, **kw: ops.fused_linear_block_diag(a, E.sv, E.su, E.codes[0], half, E.wscale, n, m, n, m, block_decompose(n),
                                                          block_decompose(m), None, None, *none * 3, **kw))]
    for L, W, call in forms:
        for a, seen, kw in steps:
            _check(seen, W, L, call(a, **kw), block_decompose(n), block_decompose(m))
            h0 = randn(tokens, m)
            h = h0.clone()
            call(a, accumulate_into=h, **kw)
            _check(seen, W, L, h.double() - h0.double(), block_decompose(n), block_decompose(m))


@pytest.mark.parametrize("kind", ["trellis", "e8"])
@pytest.mark.parametrize("m", [64, 16352, 16416])
def test_few_tiles_and_many_give_the_same_bits(m, kind):
    """A layer alone takes the output transform with 1024 threads per tile (at most a tile per SM), four of it in one plan the
    general one: every block length from 32 to 8192 (16352) and one that two tiles share (16416)."""
    from glq_b200 import synth
    from glq_b200.plan import Plan
    n, tokens = 32 if kind == "trellis" else 64, 16          # one column group: one partial sum per row, whatever the plan
    copies = 4 if m > 64 else 160
    g = torch.Generator(device="cuda").manual_seed(m)
    L = synth.trellis_layer("t", m, n, [4], g, "cuda") if kind == "trellis" else synth.e8_layer("e", m, n, 1, synth.load_e8_table("cuda"), g, "cuda")
    x = torch.randn(tokens, n, generator=g, device="cuda").half()
    got = []
    for k in (1, copies):
        plan = Plan([L.spec(batch=tokens, x_dtype=x.dtype, y_dtype=torch.float32, y_stride=k * m, y_offset=i * m) for i in range(k)])
        y = torch.empty(tokens, k, m, device="cuda")
        plan.run(x, y)
        plan.close()
        got.append(y)
    assert torch.equal(got[1], got[0].expand(tokens, copies, m))


@pytest.mark.parametrize("n,copies,step", [(224, 50, "norm"), (2016, 25, "gate")])
def test_few_and_many_input_tiles_give_the_same_bits(n, copies, step):
    """The same for the input transform behind a norm or an activation: two layers of different inputs, or many.  (A row of up to
    256 values is a value per thread in both forms of the norm, so that its sum has one order.)"""
    from glq_b200 import synth
    from glq_b200.plan import Plan
    m = 32
    g = torch.Generator(device="cuda").manual_seed(n)
    L = synth.trellis_layer("t", m, n, [4], g, "cuda")
    x = torch.randn(2 * n, generator=g, device="cuda").half()
    steps = dict(in_norm_weight=1 + 0.2 * torch.randn(n, generator=g, device="cuda"), in_norm_eps=1e-5) if step == "norm" else dict(in_gated_act=0)
    got = []
    for k in (2, copies):
        plan = Plan([L.spec(batch=1, x_dtype=x.dtype, y_dtype=torch.float32, x_stride=2 * n, x_offset=2 * n * i, y_offset=i * m, **steps)
                     for i in range(k)])
        y = torch.empty(k, m, device="cuda")
        plan.run(x.repeat(k), y)
        plan.close()
        got.append(y)
    assert torch.equal(got[1], got[0][:1].expand(copies, m))


@pytest.mark.parametrize("tokens", [1, 8, 9])
@pytest.mark.parametrize("bn,bm", [([64], [32, 16]), ([64], [16, 16]), ([64, 8], [64, 16, 8, 2]), ([16, 32, 16], [16, 32, 8, 8])], ids=str)
def test_blocks_shorter_than_a_warp(bn, bm, tokens):
    """Output and input blocks of less than 32 values, which the transforms inside the single-launch kernel cannot take."""
    from glq_b200 import synth
    m, n = sum(bm), sum(bn)
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn(tokens, n, generator=g, device="cuda")
    table = synth.load_e8_table("cuda")
    nib = (table.cpu().numpy().view(np.uint32)[:, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15
    cb = nib.astype(np.float64) * 0.5 - 3.0
    E = synth.e8_layer("e", m, n, 1, table, g, "cuda")
    y = ops.fused_linear_block_diag(x, E.sv, E.su, E.codes[0], torch.from_numpy(cb).to("cuda", torch.float16), E.wscale, n, m, n, m, bn, bm, None, None)
    _check(x, cb[E.codes[0].cpu().numpy().view(np.uint16)].reshape(m, n), E, y, bn, bm)
    if m % 32 == 0 and n % 32 == 0:
        L = synth.trellis_layer("t", m, n, [4], g, "cuda")
        y = ops.fused_linear_trellis_3inst(x, L.sv, L.su, L.codes[0], bn, bm, None, None, L.wscale, n, m, n, m)
        _check(x, ops.glq_decompress_trellis_3inst_cuda(L.codes[0], m, n).double().cpu().numpy(), L, y, bn, bm)


@pytest.mark.parametrize("kind", ["trellis", "e8"])
def test_one_cta_completes_many_output_blocks(kind):
    """Seven layers of sixteen output blocks of 32 rows (one strip, E8: two) beside one of 12288 strips (E8: 22528): a CTA takes
    some 41 (76 or more) strips in a row, and with them more than 32 blocks."""
    from glq_b200 import synth
    from glq_b200.plan import Plan
    n, m, big = 64, 512, (12 if kind == "trellis" else 11) * 32768
    g = torch.Generator(device="cuda").manual_seed(big)
    table = synth.load_e8_table("cuda")
    layer = lambda k: synth.trellis_layer("t", k, n, [4], g, "cuda") if kind == "trellis" else synth.e8_layer("e", k, n, 1, table, g, "cuda")
    layers = [layer(m) for _ in range(7)]
    for L in layers[1:]:
        L.sv = layers[0].sv
    L = layer(big)
    L.sv = layers[0].sv
    x = torch.randn(1, n, generator=g, device="cuda")

    def spec(L, off):
        s = L.spec(batch=1, x_dtype=x.dtype, y_dtype=torch.float32, y_offset=off)
        s.blocks_m = [32] * 16 if L.m == m else [32768] * (big // 32768)
        return s
    plan = Plan([spec(a, i * m) for i, a in enumerate(layers)] + [spec(L, 7 * m)])
    y = torch.full((7 * m + big,), -7.0, device="cuda")
    plan.run(x, y)
    plan.close()
    for i, a in enumerate(layers):
        alone = torch.empty(m, device="cuda")
        plan = Plan([spec(a, 0)])
        plan.run(x, alone)
        plan.close()
        assert torch.equal(y[i * m:(i + 1) * m], alone)


@pytest.mark.parametrize("normed", [False, True])
@pytest.mark.parametrize("tokens", [1, 3, 8])
@pytest.mark.parametrize("feat", [303, 700, 1361, 2050, 3640, 3643])
def test_padded_inputs_of_decode_steps(feat, tokens, normed):
    """Layers padded to 512, 1024, 2048 and 4096 columns, whose inputs end inside a thread's values and inside a group of four."""
    from glq_b200 import synth
    n, m = 1 << (feat - 1).bit_length(), 64
    g = torch.Generator(device="cuda").manual_seed(feat + tokens)
    E = synth.e8_layer("e", m, n, 1, synth.load_e8_table("cuda"), g, "cuda")
    nib = (synth.load_e8_table("cuda").cpu().numpy().view(np.uint32)[:, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15
    cb = nib.astype(np.float64) * 0.5 - 3.0
    W = cb[E.codes[0].cpu().numpy().view(np.uint16)].reshape(m, n)
    x = torch.randn(tokens, 3648, generator=g, device="cuda")[:, :feat]
    w = 1 + 0.2 * torch.randn(feat, generator=g, device="cuda")
    steps = dict(in_norm_weight=w, in_norm_eps=1e-5) if normed else {}
    y = ops.fused_linear(x, E.sv, E.su, E.codes[0], torch.from_numpy(cb).to("cuda", torch.float16), E.wscale, feat, m, n, m, 0, 0, **steps)
    seen = x.double()
    if normed:
        seen = seen * torch.rsqrt(seen.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    _check(torch.nn.functional.pad(seen, (0, n - feat)), W, E, y, [n], [m])


def test_plan_output_beyond_32_bit_offsets():
    """32769 tokens of a layer of 131072 rows: the last token's partial sums start 2^32 elements in (rows of the result are
    not aligned, so the general body runs).  Against the same token alone."""
    from glq_b200 import synth
    from glq_b200.plan import Plan
    tokens, m, n = 32769, 131072, 32
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 27 GiB")
    g = torch.Generator(device="cuda").manual_seed(9)
    L = synth.trellis_layer("t", m, n, [4], g, "cuda")
    x = torch.zeros(tokens, n, device="cuda", dtype=torch.float16)
    x[0] = 1.0
    x[-1] = torch.randn(n, generator=g, device="cuda").half()
    spec = L.spec(batch=tokens, x_dtype=x.dtype, y_dtype=torch.float16, y_stride=m + 1)
    spec.blocks_m = [32768] * 4
    plan = Plan([spec])
    y = torch.empty(tokens * (m + 1), device="cuda", dtype=torch.float16)
    plan.run(x, y)
    last = y[(tokens - 1) * (m + 1):(tokens - 1) * (m + 1) + m].float()
    plan.check_status()
    plan.close()
    del plan, y
    torch.cuda.empty_cache()
    spec = L.spec(batch=1, x_dtype=x.dtype, y_dtype=torch.float32)
    spec.blocks_m = [32768] * 4
    plan = Plan([spec])
    one = torch.empty(1, m, device="cuda")
    plan.run(x[-1:].contiguous(), one)
    plan.close()
    # the result's fp16 rounding, and fp32 sums in another order
    assert (last - one[0]).abs().max() <= (2.0 ** -11 + 1e-4) * one.abs().max()
