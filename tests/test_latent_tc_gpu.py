"""The tcgen05 latent attention against the mma.sync kernel with 16 rows a block: the same sums in the same order, so the same bits.

Tiles of 128 rows that no sequence fills, windows that begin and end inside a page, heads that do not divide 128, one and two
blocks a tile, rotated parts of 0, 32 and 64 entries of which not all turn."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _latents(H, rank, rot, rdims, window, pitch):
    """The sequences' caches and queries, and a function that runs a kernel over them."""
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(rank + rot + H)
    tile = lib.latent_tc_tile_tokens(H, rank, rot)
    assert tile == 128 // H
    before, new = [0, 61, 200, 0, 130, 64], [300, 3, tile + 1, 1, tile, 5 * tile - 1]
    bf = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    I = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    per_seq = [(a + b + 63) // 64 for a, b in zip(before, new)]
    max_pages, nt, q_head = max(per_seq), sum(new), pitch + rot
    perm = torch.randperm(sum(per_seq) + 2, generator=g).tolist()
    table = torch.zeros(len(new), max_pages, dtype=torch.int32)
    for b, n in enumerate(per_seq):
        table[b, :n] = torch.tensor([perm.pop() for _ in range(n)])
    cache, qa, q, gate = bf(sum(per_seq) + 2, 64, rank + rot), bf(nt, H, rank), bf(nt, H * q_head), bf(nt, H)
    qa *= 0.3
    angle = torch.rand(4096, max(rdims // 2, 1), generator=g) * 6
    cos, sin, sinks, table = angle.cos().cuda(), angle.sin().cuda(), torch.randn(H, generator=g).cuda(), table.cuda()
    pos = I([p for b, n in zip(before, new) for p in range(b, b + n)])

    def tiles(size):
        seq, t0, nq, at = [], [], [], 0
        for b, n in enumerate(new):
            for off in range(0, n, size):
                seq.append(b), t0.append(at + off), nq.append(min(size, n - off))
            at += n
        return I(seq), I(t0), I(nq), len(seq)

    def run(name, size, extra, pages=(), sink=None, gates=None):
        out = torch.full((nt, H, rank), 7.0, dtype=torch.bfloat16, device="cuda")
        seq, t0, nq, n = tiles(size)
        lib.call(f"tb_latent_attention_{name}_bf16", lib.ptr(qa), lib.ptr(q), lib.ptr(out), *extra, lib.ptr(cache), lib.ptr(seq),
                 lib.ptr(t0), lib.ptr(nq), lib.ptr(pos), lib.ptr(table), lib.ptr(cos), lib.ptr(sin), n, nt, max_pages, H * q_head,
                 q_head, H, rank, rot, rdims, *pages, window, *((1,) if extra else ()), q_head ** -0.5, lib.ptr(sink),
                 lib.ptr(gates), H)
        assert lib.gemm_tc_status() == 0
        return out

    return SimpleNamespace(run=run, tile=tile, cache=cache, table=table, before=before, new=new, sinks=sinks, gate=gate,
                           mma_tile=lib.latent_attention_tile_tokens(H))


@pytest.mark.parametrize("H,rank,rot,rdims,window,pitch", [
    (16, 512, 64, 64, 1 << 30, 16), (8, 256, 32, 32, 100, 16), (20, 256, 64, 32, 64, 16), (3, 256, 0, 0, 200, 16),
    (16, 512, 64, 20, 70, 12), (128, 512, 32, 16, 300, 16), (1, 256, 64, 64, 1, 16), (5, 512, 0, 0, 65, 3)])
def test_same_bits(H, rank, rot, rdims, window, pitch):
    c = _latents(H, rank, rot, rdims, window, pitch)
    for sink, gates in ((None, None), (c.sinks, c.gate)):
        want = c.run("mma", c.mma_tile, (0,), (), sink, gates)
        assert bool(torch.isfinite(want).all()) and float(want.abs().mean()) > 1e-3
        assert torch.equal(c.run("tc", c.tile, (), (c.cache.shape[0],), sink, gates), want)


@pytest.mark.parametrize("H,rank,rot,rdims,window,pitch", [
    (16, 512, 64, 64, 1 << 30, 16), (8, 256, 32, 32, 100, 16), (3, 256, 0, 0, 70, 16), (1, 256, 64, 64, 1 << 30, 16)])
def test_what_is_no_number_stays_with_the_rows_that_see_it(H, rank, rot, rdims, window, pitch):
    """Entries that are infinite or NaN: the rows that do not see their tokens keep their bits, the others have no number there."""
    c = _latents(H, rank, rot, rdims, window, pitch)
    good = c.run("tc", c.tile, (), (c.cache.shape[0],))
    # (sequence, key, column, value): one in the middle of a page, at a page's border, of three tokens, behind a sequence's end
    bad = [(0, 250, 3, float("nan")), (0, 128, rank - 1, float("inf")), (1, 62, 0, float("-inf")), (0, 310, 70, float("nan")),
           (5, 64 + 3 * c.tile, 200, float("inf")), (2, 200, 5, float("nan"))]
    for b, key, col, value in bad:
        c.cache[int(c.table[b, key // 64]), key % 64, col] = value
    got, want, at = c.run("tc", c.tile, (), (c.cache.shape[0],)), good.clone(), 0
    for b, n in enumerate(c.new):
        p = torch.arange(c.before[b], c.before[b] + n, device="cuda")
        for _, key, col, value in (e for e in bad if e[0] == b):
            see = (key <= p) & (p - key < window)
            assert not bool(torch.isfinite(got[at:at + n][see][:, :, col]).any())
            want[at:at + n][see] = got[at:at + n][see]
        at += n
    same = (got == want) | (got.isnan() & want.isnan())
    assert bool(same.all())
