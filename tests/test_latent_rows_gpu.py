"""Latent attention with 64 rows a block against the kernel with 16: the same sums in the same order, so the same bits.

Sequences that
share a block, tiles that do not fill the last one, windows that begin and end inside a page, heads that do not fill a tile, ranks and rotated parts
with an odd number of k-steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,rank,rot,window", [(16, 512, 64, 1 << 30), (8, 256, 32, 100), (20, 256, 16, 64), (3, 256, 0, 200),
                                               (16, 512, 48, 70), (16, 256, 64, 1 << 30)])
def test_same_bits(H, rank, rot, window):
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(rank + rot)
    tq = lib.latent_attention_tile_tokens(H)
    before, new = [0, 61, 200, 0, 130], [450 * tq, 3, 270 * tq + 1, 1, 66 * tq]      # at least 786 tiles
    bf = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    I = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    per_seq = [(a + b + 63) // 64 for a, b in zip(before, new)]
    max_pages, nt, q_head = max(per_seq), sum(new), 16 + rot
    perm = torch.randperm(sum(per_seq) + 2, generator=g).tolist()
    table = torch.zeros(len(new), max_pages, dtype=torch.int32)
    for b, n in enumerate(per_seq):
        table[b, :n] = torch.tensor([perm.pop() for _ in range(n)])
    cache, qa, q, gate = bf(sum(per_seq) + 2, 64, rank + rot), bf(nt, H, rank), bf(nt, H * q_head), bf(nt, H)
    angle = torch.rand(4096, max(rot // 2, 1), generator=g)
    cos, sin, sinks, table = angle.cos().cuda(), angle.sin().cuda(), torch.randn(H, generator=g).cuda(), table.cuda()
    seq, t0, nq, pos, at = [], [], [], [], 0
    for b, n in enumerate(new):
        for off in range(0, n, tq):
            seq.append(b), t0.append(at + off), nq.append(min(tq, n - off))
        pos += range(before[b], before[b] + n)
        at += n
    seq, t0, nq, pos = I(seq), I(t0), I(nq), I(pos)

    def run(name, step):
        out = torch.full((nt, H, rank), 7.0, dtype=torch.bfloat16, device="cuda")
        partial, splits = ((), ()) if name == "rows" else ((0,), (1,))
        for i in range(0, len(t0), step):
            n = min(step, len(t0) - i)
            assert lib.try_call(f"tb_latent_attention_{name}_bf16", lib.ptr(qa), lib.ptr(q), lib.ptr(out), *partial, lib.ptr(cache),
                                lib.ptr(seq[i:]), lib.ptr(t0[i:]), lib.ptr(nq[i:]), lib.ptr(pos), lib.ptr(table), lib.ptr(cos),
                                lib.ptr(sin), n, nt, max_pages, H * q_head, q_head, H, rank, rot, rot, window, *splits,
                                (16 + rot) ** -0.5, lib.ptr(sinks), lib.ptr(gate), H)
        torch.cuda.synchronize()
        return out

    want = run("mma", len(t0))
    assert bool(torch.isfinite(want).all()) and float(want.abs().mean()) > 1e-3
    for step in (len(t0), len(t0) - 1, len(t0) - 3, 5):
        assert torch.equal(run("rows", step), want)
