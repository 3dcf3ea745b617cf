"""The decode-once forms of the prefill path against the fused one: the same fp16 weights, so the same bits."""
import pytest
import torch

from glq_b200 import synth
from glq_b200.plan import Plan

pytestmark = pytest.mark.gpu


def run(layer, x, monkeypatch, env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    y = torch.full((x.shape[0], layer.m), float("nan"), device="cuda")
    plan = Plan([layer.spec(batch=x.shape[0], x_dtype=x.dtype, y_dtype=torch.float32)])
    plan.run(x, y)
    plan.check_status()
    n = plan.launches
    plan.close()
    return y, n


# rows that end inside a 128-row tile and a 32-row slice, columns that end inside a 64-column chunk
@pytest.mark.parametrize("bits", [[1], [2], [3], [4], [4, 1], [4, 2], [4, 3], [4, 4]], ids=str)
@pytest.mark.parametrize("shape", [(32, 32), (160, 96), (256, 64), (416, 1056)], ids=str)
def test_trellis_tiles_equal_fused(shape, bits, monkeypatch):
    m, n = shape
    g = torch.Generator(device="cuda").manual_seed(m + n + sum(bits))
    L = synth.trellis_layer("t", m, n, bits, g, "cuda")
    x = torch.randn(300, n, generator=g, device="cuda").half()
    a, na = run(L, x, monkeypatch, {"GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS": "1"})
    b, nb = run(L, x, monkeypatch, {"GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS": "1e30"})
    assert na == nb + 1
    assert torch.equal(a, b)


# index rows that are not 16-byte aligned, a last group of fewer than four chunks, a last chunk of fewer than eight
@pytest.mark.parametrize("stages", [1, 2, 3, 4])
@pytest.mark.parametrize("shape", [(24, 8), (136, 264), (256, 1024), (400, 1096)], ids=str)
def test_e8_tiles_equal_fused(shape, stages, monkeypatch):
    m, n = shape
    g = torch.Generator(device="cuda").manual_seed(m + n + stages)
    L = synth.e8_layer("e", m, n, stages, synth.load_e8_table("cuda"), g, "cuda")
    x = torch.randn(300, n, generator=g, device="cuda").half()
    fused, _ = run(L, x, monkeypatch, {"GLQB_E8_TWO_PHASE_MIN_TOKENS": "100000"})
    for resident in ("0", str(1 << 40)):
        tiles, _ = run(L, x, monkeypatch, {"GLQB_E8_TWO_PHASE_MIN_TOKENS": "65", "GLQB_E8_SMEM_MIN_BYTES": resident})
        assert torch.equal(tiles, fused)


# every token tile of the two forms: below, at and just above a step of 16, one 128-token tile, the first of 256, the
# first even split (193 tokens are two tiles of 112), with several chunks of 64 columns
@pytest.mark.parametrize("bits", [[4], [4, 2]], ids=str)
@pytest.mark.parametrize("tokens", [65, 72, 100, 112, 113, 128, 129, 192, 193])
def test_trellis_tiles_equal_fused_token_counts(tokens, bits, monkeypatch):
    m, n = 160, 1056
    g = torch.Generator(device="cuda").manual_seed(tokens)
    L = synth.trellis_layer("t", m, n, bits, g, "cuda")
    x = torch.randn(tokens, n, generator=g, device="cuda").half()
    a, _ = run(L, x, monkeypatch, {"GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS": "1"})
    b, _ = run(L, x, monkeypatch, {"GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS": "1e30"})
    assert torch.equal(a, b)


# two-stage layers with 256-token tiles decoded into shared memory: one tile, its edge, the first sizes of two and three
@pytest.mark.parametrize("bits", [[4, 1], [4, 2], [4, 3], [4, 4]], ids=str)
@pytest.mark.parametrize("shape", [(32, 32), (160, 1056), (416, 96)], ids=str)
def test_two_stage_256_token_tiles(shape, bits, monkeypatch):
    m, n = shape
    g = torch.Generator(device="cuda").manual_seed(m + n + sum(bits))
    L = synth.trellis_layer("t", m, n, bits, g, "cuda")
    for tokens in (193, 256, 385, 577):
        x = torch.randn(tokens, n, generator=g, device="cuda").half()
        a, _ = run(L, x, monkeypatch, {"GLQB_TRELLIS_256_MIN_WEIGHTS": "1"})
        b, _ = run(L, x, monkeypatch, {"GLQB_TRELLIS_256_MIN_WEIGHTS": str(1 << 60)})
        assert torch.equal(a, b)


# fewer tokens than the plan was built for: edges of the 16-row steps, of the token tiles (192, 256) and of the two schedules
# of a plan; rows past the tokens are neither read (NaN) nor written.  The same products in fp32, split over K in another
# order: n 2^-24 = 6e-5 of a row's absolute sum, about sqrt(n) of which is its largest value (2e-6), with a margin of ten.
@pytest.mark.parametrize("kind", ["trellis", "two stages", "tiles", "e8", "e8 fused"])
@pytest.mark.parametrize("bucket,tokens", [(16, 9), (32, 27), (64, 57), (128, 65), (128, 113), (256, 129), (256, 192), (256, 193),
                                           (512, 257), (512, 384), (512, 385), (512, 20)])
def test_run_of_fewer_tokens(kind, bucket, tokens, monkeypatch):
    m, n = 160, 1056
    monkeypatch.setenv("GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS", "1" if kind == "tiles" else "1e30")
    monkeypatch.setenv("GLQB_E8_TWO_PHASE_MIN_TOKENS", "65" if kind == "e8" else "100000")
    if kind == "two stages" and bucket == 64:
        pytest.skip("two stages take 32 tokens per pass")
    g = torch.Generator(device="cuda").manual_seed(bucket + tokens)
    if kind.startswith("e8"):
        L = synth.e8_layer("e", m, n, 2, synth.load_e8_table("cuda"), g, "cuda")
    else:
        L = synth.trellis_layer("t", m, n, [4, 2] if kind == "two stages" else [4], g, "cuda")
    x = torch.randn(bucket, n, generator=g, device="cuda").half()
    plan = Plan([L.spec(batch=bucket, x_dtype=x.dtype, y_dtype=torch.float32)])
    full = torch.empty(bucket, m, device="cuda")
    plan.run(x, full)
    x[tokens:] = float("nan")
    y = torch.full((bucket, m), -7.0, device="cuda")
    plan.run(x, y, tokens=tokens)
    plan.check_status()
    plan.close()
    assert (y[tokens:] == -7.0).all()
    assert (y[:tokens] - full[:tokens]).abs().max() <= 2e-5 * full.abs().max()


# two token tiles per item: two whole tiles, an odd last tile, a second tile that the tokens of the run cut short or away, the
# schedule for one tile fewer, columns that end inside a pair of chunks.  352 columns are one K range in both forms and so the same
# bits; 1056 may be split, see above.
@pytest.mark.parametrize("bits", [[4], [2], [4, 2]], ids=str)
@pytest.mark.parametrize("n", [352, 1056])
@pytest.mark.parametrize("bucket,tokens", [(256, 193), (256, 256), (512, 512), (512, 500), (512, 385), (512, 300), (768, 768), (768, 600),
                                           (768, 577), (768, 390), (1024, 1000), (1024, 20)])
def test_pairs_of_token_tiles(bits, n, bucket, tokens, monkeypatch):
    m = 160
    monkeypatch.setenv("GLQB_TRELLIS_TWO_PHASE_MIN_FLOPS", "1e30")
    g = torch.Generator(device="cuda").manual_seed(n + tokens)
    L = synth.trellis_layer("t", m, n, bits, g, "cuda")
    x = torch.randn(bucket, n, generator=g, device="cuda").half()
    x[tokens:] = float("nan")
    got = []
    for pairs in ("0", "1"):
        monkeypatch.setenv("GLQB_GEMM_PAIRS", pairs)
        plan = Plan([L.spec(batch=bucket, x_dtype=x.dtype, y_dtype=torch.float32)])
        y = torch.full((bucket, m), -7.0, device="cuda")
        plan.run(x, y, tokens=tokens)
        plan.check_status()
        plan.close()
        assert (y[tokens:] == -7.0).all()
        got.append(y[:tokens])
    if n == 352:
        assert torch.equal(*got)
    assert (got[0] - got[1]).abs().max() <= 2e-5 * got[0].abs().max()


# a shape for which the costs choose pairs: all tokens, and a ragged number of them
@pytest.mark.parametrize("tokens", [1024, 1000])
def test_pairs_of_token_tiles_by_cost(tokens, monkeypatch):
    from glq_b200 import ops
    m, n = 11008, 2048
    g = torch.Generator(device="cuda").manual_seed(tokens)
    L = synth.trellis_layer("t", m, n, [4], g, "cuda")
    x = torch.randn(tokens, n, generator=g, device="cuda").half()
    H = torch.ones(1, 1, dtype=torch.float64, device="cuda")
    had = {}
    for k in range(14):
        had[1 << k] = H
        H = torch.cat([torch.cat([H, H], 1), torch.cat([H, -H], 1)])
    turn = lambda v, blocks: torch.cat([p @ had[b] / b ** 0.5 for p, b in zip(v.split(blocks, 1), blocks)], 1)
    W = ops.glq_decompress_trellis_3inst_cuda(L.codes[0], m, n).double()
    ref = turn(turn(x.double() * L.sv.double(), [2048]) @ W.T * L.wscale, [8192, 2048, 512, 256]) * L.su.double()
    ops.clear_caches()
    y = ops.fused_linear_trellis_3inst(x, L.sv, L.su, L.codes[0], None, None, None, None, L.wscale, n, m, n, m, out_dtype=torch.float32)
    # the rotated activations are fp16: 2e-3 of the largest output, as for every linear
    assert (y.double() - ref).abs().max() <= 2e-3 * ref.abs().max()
    ops.clear_caches()
