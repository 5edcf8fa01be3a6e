"""The windowed form of the tcgen05 prompt attention at the edges of tiles, pages, windows and chunks, against float64.

Tolerance of the first: the weights are rounded to bfloat16 (2^-9 of each, against a sum of unrounded ones) and so is the result:
2^-8 of the largest |value|.  The products and exponentials in 32 bits add some 1e-6; 1e-3 covers the gate's and the
cap's approximate divisions as well."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BEFORE, NEW = [0, 61, 200, 0, 130, 64], [300, 3, 129, 1, 128, 257]


def _batch(g, extra_pages=2):
    """Shuffled pages and the step's arrays of the sequences (BEFORE, NEW), tiles of 128 tokens."""
    I = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    per_seq = [(a + b + 63) // 64 for a, b in zip(BEFORE, NEW)]
    perm = torch.randperm(sum(per_seq) + extra_pages, generator=g).tolist()
    pages = [[perm.pop() for _ in range(n)] for n in per_seq]
    table = torch.zeros(len(NEW), max(per_seq), dtype=torch.int32)
    seq, t0, nq, pos, at = [], [], [], [], 0
    for b, n in enumerate(NEW):
        table[b, :per_seq[b]] = torch.tensor(pages[b])
        for off in range(0, n, 128):
            seq.append(b), t0.append(at + off), nq.append(min(128, n - off))
        pos += range(BEFORE[b], BEFORE[b] + n)
        at += n
    return dict(n_pages=sum(per_seq) + extra_pages, pages=pages, table=table.cuda(), max_pages=max(per_seq), seq=I(seq), t0=I(t0),
                nq=I(nq), pos=I(pos), nt=at, tiles=len(seq))


def _attend(q, k, v, scale, visible, cap=0.0, sinks=None):
    """q [n, H, dk], k [m, H, dk], v [m, H, dv] float64; visible [n, m]."""
    s = torch.einsum("nhd,mhd->hnm", q, k) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    s = s.masked_fill(~visible, float("-inf"))
    if sinks is not None:
        s = torch.cat([s, sinks.double()[:, None, None].expand(-1, s.shape[1], 1)], dim=2)
        v = torch.cat([v, v.new_zeros(1, *v.shape[1:])])
    return torch.einsum("hnm,mhd->nhd", torch.softmax(s, dim=2), v)


@pytest.mark.parametrize("nh,nkvh,dh,window,keep,chunk,cap,more", [
    (8, 2, 128, 100, 4, 0, 30.0, "gate"), (4, 4, 64, 64, 0, 0, 0.0, "sinks"), (6, 2, 64, 65, 70, 0, 5.0, "heads"),
    (5, 1, 128, 1 << 30, 0, 96, 0.0, "gate"), (2, 2, 128, 1, 1, 0, 50.0, ""), (4, 2, 64, 130, 3, 64, 20.0, "sinks")])
def test_windowed_form(nh, nkvh, dh, window, keep, chunk, cap, more):
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(nh + dh + keep)
    c = _batch(g)
    bf = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    nt = c["nt"]
    kc, vc, z = bf(c["n_pages"], nkvh, 64, dh), bf(c["n_pages"], nkvh, 64, dh), bf(nt, 2 * nh * dh + 16)
    gate, per_head, mult, ldo, sinks = None, 0, 1.0, nh * dh, None
    if more == "gate":
        gate = z[:, nh * dh:]
    elif more == "heads":
        gate, per_head, mult, ldo = bf(nt, nh), 1, 0.7, nh * dh + 24
    elif more == "sinks":
        sinks = torch.randn(nh, generator=g).cuda() * 2
    out = torch.full((nt, ldo), 7.0, dtype=torch.bfloat16, device="cuda")
    scale = 3.0 * dh ** -0.5
    lib.call("tb_attention_tc_window_bf16", lib.ptr(z), lib.ptr(out), lib.ptr(kc), lib.ptr(vc), lib.ptr(gate), lib.ptr(c["seq"]),
             lib.ptr(c["t0"]), lib.ptr(c["nq"]), lib.ptr(c["pos"]), lib.ptr(c["table"]), c["tiles"], nt, c["max_pages"], z.stride(0),
             0 if gate is None else gate.stride(0), nh, nkvh, dh, c["n_pages"], window, keep, scale, cap, chunk, lib.ptr(sinks),
             per_head, mult, ldo)
    assert lib.gemm_tc_status() == 0
    assert bool((out[:, nh * dh:] == 7.0).all())
    at = 0
    for b, n in enumerate(NEW):
        p, m = c["pos"][at:at + n].long(), BEFORE[b] + n
        at_pages = torch.tensor(c["pages"][b], device="cuda")
        k, v = (t[at_pages].transpose(1, 2).reshape(-1, nkvh, dh)[:m].double().repeat_interleave(nh // nkvh, dim=1) for t in (kc, vc))
        j = torch.arange(m, device="cuda")
        see = (j[None] <= p[:, None]) & ((p[:, None] - j[None] < window) | (j[None] < keep))
        if chunk:
            see &= p[:, None] // chunk == j[None] // chunk
        want = _attend(z[at:at + n, :nh * dh].reshape(n, nh, dh).double(), k, v, scale, see, cap=cap, sinks=sinks) * mult
        if gate is not None:
            want = want * torch.sigmoid(gate[at:at + n, :nh * (1 if per_head else dh)].reshape(n, nh, -1).double())
        err = float((out[at:at + n, :nh * dh].reshape(n, nh, dh).double() - want).abs().max())
        assert err <= 2.0 ** -8 * float(vc.abs().max()) + 1e-3, (b, err)
        at += n


@pytest.mark.parametrize("nh,nkvh,dh,window,keep,chunk,cap,more", [
    (8, 2, 128, 100, 4, 0, 30.0, "gate"), (4, 4, 64, 64, 0, 0, 0.0, "sinks"), (6, 2, 64, 65, 70, 0, 5.0, "heads"),
    (5, 1, 128, 1 << 30, 0, 96, 0.0, "gate"), (4, 2, 128, 1 << 30, 0, 0, 0.0, ""), (16, 1, 64, 200, 3, 0, 20.0, "")])
def test_bits_of_the_mma_form(nh, nkvh, dh, window, keep, chunk, cap, more):
    """The mma.sync kernel without slices: the same weights (against the row's true maximum) and sums in the same order, so the same
    bits, whichever of the two a step takes."""
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(nh + dh + window % 1000)
    c = _batch(g)
    bf = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    nt, mma = c["nt"], lib.attention_window_mma_tile_tokens(nh, nkvh)
    kc, vc, z = bf(c["n_pages"], nkvh, 64, dh), bf(c["n_pages"], nkvh, 64, dh), bf(nt, 2 * nh * dh)
    z[:, :nh * dh] *= 2
    gate, per_head, mult = (z[:, nh * dh:], 0, 1.0) if more == "gate" else (bf(nt, nh), 1, 0.7) if more == "heads" else (None, 0, 1.0)
    sinks = torch.randn(nh, generator=g).cuda() * 2 if more == "sinks" else None
    I = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    seq, t0, nq, at = [], [], [], 0
    for b, n in enumerate(NEW):
        for off in range(0, n, mma):
            seq.append(b), t0.append(at + off), nq.append(min(mma, n - off))
        at += n
    seq, t0, nq = I(seq), I(t0), I(nq)
    got, want = (torch.empty(nt, nh * dh, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    data = lambda out: (lib.ptr(z), lib.ptr(out), lib.ptr(kc), lib.ptr(vc), lib.ptr(gate))
    rows = (nt, c["max_pages"], z.stride(0), 0 if gate is None else gate.stride(0), nh, nkvh)
    rule = (window, keep, dh ** -0.5, cap, chunk, lib.ptr(sinks))
    lib.call("tb_attention_tc_window_bf16", *data(got), lib.ptr(c["seq"]), lib.ptr(c["t0"]), lib.ptr(c["nq"]), lib.ptr(c["pos"]),
             lib.ptr(c["table"]), c["tiles"], *rows, dh, c["n_pages"], *rule, per_head, mult, nh * dh)
    lib.call("tb_attention_window_mma_heads_bf16", *data(want), lib.ptr(seq), lib.ptr(t0), lib.ptr(nq), lib.ptr(c["pos"]),
             lib.ptr(c["table"]), 0, len(seq), *rows, dh, dh, 1, *rule, 0, 0, per_head, mult, nh * dh)
    assert lib.gemm_tc_status() == 0 and bool(torch.isfinite(want).all())
    assert torch.equal(got, want)


@pytest.mark.parametrize("nh,nkvh,dh,window,keep,chunk,cap", [
    (4, 2, 128, 100, 4, 0, 30.0), (4, 4, 64, 64, 0, 0, 0.0), (6, 2, 64, 1 << 30, 0, 96, 0.0), (3, 1, 128, 1 << 30, 0, 0, 20.0)])
def test_what_is_no_number_stays_with_the_rows_that_see_it(nh, nkvh, dh, window, keep, chunk, cap):
    """Values that are infinite or NaN at places before, in and behind the tiles (one of them in a page's rows that no sequence has
    reached): the rows that do not see them keep their bits, the others too but in the columns of those values."""
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(7 * nh + dh)
    c = _batch(g)
    bf = lambda *shape: torch.randn(*shape, generator=g).bfloat16().cuda()
    nt = c["nt"]
    kc, vc, z = bf(c["n_pages"], nkvh, 64, dh), bf(c["n_pages"], nkvh, 64, dh), bf(nt, nh * dh)

    def run():
        out = torch.empty((nt, nh, dh), dtype=torch.bfloat16, device="cuda")
        lib.call("tb_attention_tc_window_bf16", lib.ptr(z), lib.ptr(out), lib.ptr(kc), lib.ptr(vc), 0, lib.ptr(c["seq"]),
                 lib.ptr(c["t0"]), lib.ptr(c["nq"]), lib.ptr(c["pos"]), lib.ptr(c["table"]), c["tiles"], nt, c["max_pages"], nh * dh,
                 0, nh, nkvh, dh, c["n_pages"], window, keep, dh ** -0.5, cap, chunk, 0, 0, 1.0, nh * dh)
        assert lib.gemm_tc_status() == 0
        return out

    good = run()
    assert bool(torch.isfinite(good).all())
    # (sequence, key, key head, column, value); the last is behind its sequence's end
    bad = [(0, 250, 0, 3, float("nan")), (0, 0, nkvh - 1, dh - 1, float("inf")), (0, 130, 0, 40, float("-inf")), (2, 190, 0, 0, float("inf")),
           (2, 328, nkvh - 1, 17, float("nan")), (4, 131, 0, 33, float("nan")), (5, 320, 0, dh // 2, float("inf")),
           (1, 62, 0, 9, float("nan")), (0, 310, 0, 9, float("nan"))]
    for b, key, head, col, value in bad:
        vc[c["pages"][b][key // 64], head, key % 64, col] = value
    got, want, at = run(), good.clone(), 0
    for b, n in enumerate(NEW):
        p = torch.arange(BEFORE[b], BEFORE[b] + n, device="cuda")
        for _, key, head, col, value in (e for e in bad if e[0] == b):
            see = (key <= p) & ((p - key < window) | (key < keep))
            if chunk:
                see &= p // chunk == key // chunk
            heads = range(head * (nh // nkvh), (head + 1) * (nh // nkvh))
            for h in heads:
                hit = got[at:at + n, h, col][see]
                assert not bool(torch.isfinite(hit).any()), (b, key, h)
                want[at:at + n, h, col][see] = hit
        at += n
    same = (got == want) | (got.isnan() & want.isnan())
    assert bool(same.all())
