"""Launches that start before the one in front of them has ended (programmatic dependent launch): calls of every form, one right
behind the other on one stream and in one workspace, give what they give alone, and what ordinary launches give."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

# (format, rows, columns, stages or bits, tokens): single-launch, streaming (E8: table in global and in shared memory), the GEMM that
# decodes, tiles decoded ahead (trellis; E8 with the table in global and in shared memory), output blocks of 8192 and 16384 rows
CALLS = [("trellis", 544, 1024, [4], 1), ("e8", 544, 1024, 2, 3), ("trellis", 2048, 2048, [4, 2], 27), ("e8", 512, 2048, 2, 16),
         ("e8", 4096, 4096, 2, 9), ("trellis", 1056, 2048, [4], 130), ("trellis", 1056, 2048, [3], 700), ("trellis", 2048, 4096, [4], 4096),
         ("e8", 1024, 2048, 2, 100), ("e8", 1024, 2048, 2, 300), ("e8", 8192, 8192, 3, 200), ("trellis", 8192, 512, [4], 5),
         ("e8", 16384, 256, 1, 20)]


def calls():
    from glq_b200 import ops, synth
    g = torch.Generator(device="cuda").manual_seed(1)
    table = synth.load_e8_table("cuda")
    bits = (table.view(-1, 1) >> (4 * torch.arange(8, device="cuda", dtype=torch.int32))) & 15
    book = (bits.float() * 0.5 - 3.0).half()
    out = []
    for kind, m, n, form, tokens in CALLS:
        x = torch.randn(tokens, n, generator=g, device="cuda").half()
        if kind == "trellis":
            L = synth.trellis_layer("t", m, n, form, g, "cuda")
            if len(form) == 2:
                out.append(lambda L=L, x=x, m=m, n=n: ops.fused_linear_trellis_3inst_rvq2(x, L.sv, L.su, *L.codes, None, None, None, None, L.wscale, 0.2,
                                                                                         n, m, n, m))
            else:
                out.append(lambda L=L, x=x, m=m, n=n: ops.fused_linear_trellis_3inst(x, L.sv, L.su, L.codes[0], None, None, None, None, L.wscale,
                                                                                    n, m, n, m))
        else:
            L = synth.e8_layer("e", m, n, form, table, g, "cuda")
            tail = sum(((q, book, 0.1 ** (s + 1)) for s, q in enumerate(L.codes[1:])), ())
            out.append(lambda L=L, x=x, m=m, n=n, tail=tail: ops.fused_linear_block_diag(x, L.sv, L.su, L.codes[0], book, L.wscale, n, m, n, m, None,
                                                                                        None, None, None, *tail))
    E, hidden, inter = 8, 256, 192
    i16 = lambda *s: torch.randint(-32768, 32768, s, generator=g, device="cuda", dtype=torch.int32).to(torch.int16)
    signs = lambda *s: (torch.randint(0, 2, s, generator=g, device="cuda") * 2 - 1).half()
    w13, w2, none = i16(E, 2 * inter // 16 * (hidden // 16), 64), i16(E, hidden // 16 * (inter // 16), 64), torch.zeros(E, 1, 1, dtype=torch.int16, device="cuda")
    su13, sv13, su2, sv2, ws, inv = signs(E, 2 * inter), signs(hidden), signs(E, hidden), signs(inter), torch.full((E,), 0.02, device="cuda"), torch.zeros(E, device="cuda")
    for tokens in (5, 200):
        x = torch.randn(tokens, hidden, generator=g, device="cuda").half()
        ids, w = torch.rand(tokens, E, generator=g, device="cuda").topk(2).indices, torch.rand(tokens, 2, generator=g, device="cuda")
        out.append(lambda x=x, ids=ids, w=w: ops.fused_moe_trellis_3inst(x, ids, w, w13, none, su13, sv13, ws, inv, w2, none, su2, sv2, ws, inv, hidden,
                                                                         inter, 2 * inter, hidden, 2 * inter, inter, hidden, None, None, None, None,
                                                                         None, None, None, None, 0))
    return out


def alone():
    out = []
    for call in calls():
        out.append(call())
        torch.cuda.synchronize()
    return out


def test_calls_behind_one_another():
    from glq_b200 import ops
    refs = alone()
    todo = calls()
    order = [(i * step) % len(todo) for step in (1, 2, 4, 7) for i in range(len(todo))]      # (15 calls: every order is a permutation)
    for _ in range(3):
        got = [(i, todo[i]()) for i in order]
        torch.cuda.synchronize()
        ops.check_device_status()
        for i, y in got:
            assert torch.equal(y, refs[i]), CALLS[i] if i < len(CALLS) else "experts"


def test_ordinary_launches_give_the_same(tmp_path):
    """GLQB_PDL is read once per process: a process without chained launches computes the same calls."""
    code = "import torch, test_gpu_chains as t; torch.save(t.alone(), %r)" % str(tmp_path / "y.pt")
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, GLQB_PDL="0", PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)
    for y, ref in zip(torch.load(tmp_path / "y.pt"), alone()):
        assert torch.equal(y, ref)
