"""The delta rule 16 tokens at a time against the recurrence in 64 bits: sequences around a chunk's edges, one in two
steps, heads that share a key, one decay per head, and decays from 1 down to 0.

The bound: results are sums of at most (tokens + dim) float terms whose sizes the values bound (unit keys, beta <= 1,
decays <= 1), so 1e-5 of the largest value, as for the token-by-token kernel; bfloat16 inputs are exact here."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plain(x, conv, a, beta, G, H, dim, vdim):
    """x [n, C] inputs, a [n, H, dim] decays, beta [n, H], float64 -> (o [n, H, vdim], S [H, dim, vdim])."""
    n, C = x.shape
    xp = torch.cat([torch.zeros(3, C, dtype=x.dtype), x])
    y = sum(conv[:, j] * xp[j:j + n] for j in range(4))
    y = y * torch.sigmoid(y)
    unit = lambda t: t / (t.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    q = unit(y[:, :G * dim].view(n, G, dim)).repeat_interleave(H // G, 1) * dim ** -0.5
    k = unit(y[:, G * dim:2 * G * dim].view(n, G, dim)).repeat_interleave(H // G, 1)
    v = y[:, 2 * G * dim:].view(n, H, vdim)
    S = torch.zeros(H, dim, vdim, dtype=x.dtype)
    out = []
    for t in range(n):
        S = a[t][:, :, None] * S
        u = beta[t][:, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], S))
        S = S + k[t][:, :, None] * u[:, None]
        out.append(torch.einsum("hd,hdv->hv", q[t], S))
    return torch.stack(out), S


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("dim", [64, 128])
def test_what_is_no_number_stays_behind_its_token(dim, bad):
    """One value channel of one token is no number: the outputs of the tokens before it, those of its own chunk among them, and
    of the other channels keep their bits, as token by token."""
    from transformer_b200.csrc import lib
    gen = torch.Generator().manual_seed(dim)
    n, H, vdim, at, channel = 50, 2, 32, 21, 5
    C = 2 * H * dim + H * vdim
    x, a, bz = torch.randn(n, C, generator=gen), torch.randn(n, H * dim, generator=gen).cuda(), torch.randn(n, H, generator=gen).cuda()
    conv, bias, A_log = torch.randn(C, 4, generator=gen).cuda(), torch.randn(H * dim, generator=gen).cuda(), torch.rand(H, generator=gen).cuda()
    starts, slots = torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()
    chunks, outs = n // 16 + 1, []
    for value in (0.5, bad):
        z = x.clone()
        z[at, 2 * H * dim + channel] = value
        z, state = z.cuda(), torch.zeros(1, lib.delta_state_size(H, H, dim, vdim, 4)).cuda()
        rec = torch.empty(H, chunks, lib.delta_chunk_record_size(dim, vdim, 4)).cuda()
        o = torch.full((n, H, vdim), 7.0, device="cuda")
        where = (lib.ptr(starts), lib.ptr(slots), n, 1, H, H, dim, vdim, 4, chunks)
        lib.call("tb_delta_chunk_f32", lib.ptr(z), C, lib.ptr(conv), lib.ptr(state), lib.ptr(a), lib.ptr(bias), lib.ptr(A_log), lib.ptr(bz),
                 lib.ptr(rec), *where, H * dim, H, 0)
        lib.call("tb_delta_chunk_scan", lib.ptr(rec), lib.ptr(state), lib.ptr(o), *where)
        outs.append(o.cpu())
    good, got = outs
    assert bool(torch.isfinite(good).all()) and not bool(torch.isfinite(got[at:, 0, channel]).any())
    got[at:, 0, channel] = good[at:, 0, channel]
    assert torch.equal(good, got)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("G,H,dim,vdim,per_head,steep", [(2, 4, 64, 48, False, 0.0), (1, 1, 128, 128, True, 0.0),
                                                         (2, 2, 128, 16, False, 6.0), (1, 2, 64, 256, False, -12.0)])
def test_chunks(dtype, G, H, dim, vdim, per_head, steep):
    from transformer_b200.csrc import lib
    gen = torch.Generator().manual_seed(dim + vdim)
    lens, later = [1, 16, 17, 50, 3, 32], [40, 1, 15, 33, 16, 2]        # two steps of the same sequences
    B, C, sfx = len(lens), 2 * G * dim + H * vdim, "f32" if dtype == torch.float32 else "bf16"
    size, n_a = lib.delta_state_size(G, H, dim, vdim, 4), H if per_head else H * dim
    state = torch.randn(B + 1, size, generator=gen)
    slots = torch.tensor([3, 1, 0, 5, 2, 6], dtype=torch.int32)
    state[slots.long()] = 0.0
    untouched = state[4].clone()
    state, slots = state.cuda(), slots.cuda()
    x = [torch.randn(m + n, C, generator=gen).to(dtype) for m, n in zip(lens, later)]
    pre = [torch.randn(m + n, n_a, generator=gen) * 3 + steep for m, n in zip(lens, later)]
    bz = [torch.randn(m + n, H, generator=gen) * 2 for m, n in zip(lens, later)]
    for i in (1, 3):                                    # a sequence whose tokens are all alike: keys repeat
        x[i][:] = x[i][0]
    conv, A_log = torch.randn(C, 4, generator=gen) * 0.6, torch.rand(H, generator=gen) * 3 - 2.5
    bias = torch.randn(n_a, generator=gen) - 1
    d_conv, d_A, d_bias = conv.cuda(), A_log.cuda(), bias.cuda()
    per = lib.delta_chunk_record_size(dim, vdim, 4)
    got = [[] for _ in lens]
    for first, ns in ((0, lens), (1, later)):
        pick = lambda rows: torch.cat([r[m:] if first else r[:m] for r, m in zip(rows, lens)])
        z = torch.zeros(sum(ns), C + 6, dtype=dtype)
        z[:, :C] = pick(x)
        z, a, b = z.cuda(), pick(pre).cuda(), pick(bz).cuda()
        starts = torch.tensor([0] + ns).cumsum(0).to(torch.int32).cuda()
        chunks = sum(ns) // 16 + B
        rec = torch.full((H, chunks, per), float("nan"), device="cuda")
        o = torch.full((sum(ns), H, vdim), float("nan"), device="cuda")
        where = (lib.ptr(starts), lib.ptr(slots), sum(ns), B, G, H, dim, vdim, 4, chunks)
        lib.call("tb_delta_chunk_" + sfx, lib.ptr(z), C + 6, lib.ptr(d_conv), lib.ptr(state), lib.ptr(a), lib.ptr(d_bias),
                 lib.ptr(d_A), lib.ptr(b), lib.ptr(rec), *where, n_a, H, int(per_head))
        lib.call("tb_delta_chunk_scan", lib.ptr(rec), lib.ptr(state), lib.ptr(o), *where)
        torch.cuda.synchronize()
        for i, part in enumerate(o.cpu().split(ns)):
            got[i].append(part)
    assert not lib.library().tb_gemm_tc_status()
    assert torch.equal(state[4].cpu(), untouched)
    for i in range(B):
        rate = torch.exp(A_log.double())[None, :, None]
        decay = torch.exp(-rate * torch.nn.functional.softplus(pre[i].double() + bias.double()).view(len(x[i]), H, -1))
        want, S = _plain(x[i].double(), conv.double(), decay.expand(-1, -1, dim), torch.sigmoid(bz[i].double()), G, H, dim, vdim)
        scale = float(want.abs().max()) + 1.0
        assert float((torch.cat(got[i]).double() - want).abs().max()) <= 1e-5 * scale
        row = state[int(slots[i])].cpu().double()
        assert float((row[:H * dim * vdim].view(H, dim, vdim) - S).abs().max()) <= 1e-5 * (float(S.abs().max()) + 1.0)
        assert torch.equal(row[H * dim * vdim:].view(3, C), x[i][-3:].double())


@pytest.mark.parametrize("H,vdim,copies", [(4, 128, 5), (3, 32, 25), (3, 48, 17), (1, 256, 9), (1, 256, 10)])
def test_scan_of_many_columns(H, vdim, copies):
    """Many columns, with 16 and, where they come in 32s, with 32 of them a block, which give the same bits: lengths around a chunk's
    edges and an empty sequence.  The bound is that of `test_chunks`."""
    from transformer_b200.csrc import lib
    gen, dim = torch.Generator().manual_seed(vdim + copies), 128
    lens = [(1, 15, 0, 16, 33, 50, 17)[i % 7] for i in range(copies)]
    B, nt, C = copies, sum(lens), 2 * H * dim + H * vdim
    x, a, bz = torch.randn(nt, C, generator=gen), torch.randn(nt, H * dim, generator=gen) * 3, torch.randn(nt, H, generator=gen) * 2
    conv, bias, A_log = torch.randn(C, 4, generator=gen) * 0.6, torch.randn(H * dim, generator=gen) - 1, torch.rand(H, generator=gen) * 3 - 2.5
    state, slots = torch.zeros(B, lib.delta_state_size(H, H, dim, vdim, 4)).cuda(), torch.arange(B).flip(0).int().cuda()
    d = [t.cuda() for t in (x, conv, a, bias, A_log, bz, torch.tensor([0] + lens).cumsum(0).int())]
    chunks = nt // 16 + B
    rec = torch.full((H, chunks, lib.delta_chunk_record_size(dim, vdim, 4)), float("nan"), device="cuda")
    o = torch.full((nt, H, vdim), float("nan"), device="cuda")
    where = (lib.ptr(d[6]), lib.ptr(slots), nt, B, H, H, dim, vdim, 4, chunks)
    lib.call("tb_delta_chunk_f32", lib.ptr(d[0]), C, lib.ptr(d[1]), lib.ptr(state), *(lib.ptr(t) for t in d[2:6]), lib.ptr(rec), *where,
             H * dim, H, 0)
    before, wide = state.clone(), vdim % 32 == 0
    assert lib.try_call("tb_delta_chunk_scan_wide", lib.ptr(rec), lib.ptr(before), lib.ptr(o), *where) is wide
    first = o.clone()
    lib.call("tb_delta_chunk_scan", lib.ptr(rec), lib.ptr(state), lib.ptr(o), *where)
    if wide:
        assert torch.equal(o, first) and torch.equal(state, before)
    got = o.cpu().double().split(lens)
    assert not lib.library().tb_gemm_tc_status()
    for i, (xi, ai, bi) in enumerate(zip(x.split(lens), a.split(lens), bz.split(lens))):
        if not lens[i]:
            continue
        decay = torch.exp(-torch.exp(A_log.double())[None, :, None] *
                          torch.nn.functional.softplus(ai.double() + bias.double()).view(lens[i], H, dim))
        want, S = _plain(xi.double(), conv.double(), decay, torch.sigmoid(bi.double()), H, H, dim, vdim)
        assert float((got[i] - want).abs().max()) <= 1e-5 * (float(want.abs().max()) + 1.0)
        row = state[B - 1 - i].cpu().double()[:H * dim * vdim].view(H, dim, vdim)
        assert float((row - S).abs().max()) <= 1e-5 * (float(S.abs().max()) + 1.0)
