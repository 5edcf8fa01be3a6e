"""Forms that a decode step takes by its size, against each other: they differ in what is in flight, not in the order of a sum,
so the same rows have the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).bfloat16().cuda()


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("K", [8, 256, 264, 512, 520, 1024, 2040, 2056, 2816, 3072, 3080])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_narrow_products_have_the_bits_of_wide_ones(M, K, kind):
    """Few blocks and up to 8 rows: 4 to 16 k-steps of a thread's weights in flight by K (for K up to 1,024, a pair's up to 512, and from
    2,056 to 3,072 all of them).  The same columns of a wider product are computed a few steps at a time."""
    from transformer_b200.parts.linear import gemm_skinny
    N, wide = 520, 5200
    x, w = _bf(M, K, seed=1), _bf((2 if kind == 2 else 1) * wide, K, seed=2) * K ** -0.5
    narrow = torch.cat([w[:N], w[wide:wide + N]]) if kind == 2 else w[:N]
    out = [torch.full((M, n), 7.0, device="cuda", dtype=torch.float32 if kind == 1 else torch.bfloat16) for n in (N, wide)]
    assert gemm_skinny(x, narrow.contiguous(), out[0], out_kind=kind) and gemm_skinny(x, w, out[1], out_kind=kind)
    assert torch.equal(out[0], out[1][:, :N])
    want = x.double() @ w[:N].double().T
    if kind == 2:
        want = torch.nn.functional.silu(want) * (x.double() @ w[wide:wide + N].double().T)
    assert float((out[0].double() - want).norm() / want.norm()) < 5e-3


@pytest.mark.parametrize("K,kind", [(688, 0), (2048, 0), (4096, 2), (24, 2)])
@pytest.mark.parametrize("groups", [[3], [5, 5], [7, 0, 7, 15], [15, 15, 15, 15], [2, 99, -1, 2], [0, 1, 2, 3, 4, 5, 6, 7]])
def test_products_by_row_have_the_bits_of_products_by_group(K, kind, groups):
    """At most a quarter as many rows as groups: a block column per row.  More rows (those of a group that no row asked for): per group.
    Rows that name no group are left alone by both."""
    from transformer_b200.parts.linear import gemm_skinny
    G, N, M, more = 64, 72, len(groups), 17
    w = _bf(G, (2 if kind == 2 else 1) * N, K, seed=3) * K ** -0.5
    x = _bf(M + more, K, seed=4)
    spare = next(g for g in range(G) if g not in groups)
    ids = torch.tensor(groups + [spare] * more, dtype=torch.int32, device="cuda")
    out = [torch.full((n, N), 7.0, device="cuda", dtype=torch.bfloat16) for n in (M, M + more)]
    for o in out:
        n = o.shape[0]
        assert gemm_skinny(x[:n], w, o, groups=G, out_kind=kind, max_group_rows=8, row_group=ids[:n])
    assert torch.equal(out[0], out[1][:M])
    for m, g in enumerate(groups):
        if not 0 <= g < G:
            assert bool((out[0][m] == 7.0).all())
            continue
        z = x[m].double() @ w[g].double().T
        want = torch.nn.functional.silu(z[:N]) * z[N:] if kind == 2 else z
        assert float((out[0][m].double() - want).norm() / want.norm()) < 5e-3


@pytest.mark.parametrize("d,E,k", [(4096, 16, 4), (4096, 5, 2), (2048, 40, 3), (1000, 16, 4), (8192, 12, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_that_routes_with_and_without_the_staged_matrix(d, E, k, dtype):
    """Up to 16 rows the first 16 rows of the router's matrix are staged in shared memory where they fit (not float32 4,096 x 16
    and the 8,192s: both calls then read it alike), from 17 rows on its first part is read into registers; more rows than
    SMs, the form with the short loop: the same bits."""
    from transformer_b200.csrc import lib
    rows, sfx = 160, "f32" if dtype == torch.float32 else "bf16"
    g = torch.Generator().manual_seed(d + E)
    x, delta = torch.randn(rows, d, generator=g), torch.randn(rows, d, generator=g).to(dtype).cuda()
    w, wr = torch.rand(d, generator=g).cuda() + 0.5, torch.randn(E, d, generator=g).to(dtype).cuda()
    got = []
    for n in (16, 17, 160):
        xs = x[:n].cuda()
        y = torch.empty(n, d, dtype=dtype, device="cuda")
        idx, p = torch.empty(n, k, dtype=torch.int32, device="cuda"), torch.empty(n, k, device="cuda")
        assert lib.try_call("tb_add_rmsnorm_router_" + sfx, lib.ptr(xs), lib.ptr(delta), 0, 0, 0, 0, 0, lib.ptr(w), 1e-5, lib.ptr(y),
                            lib.ptr(wr), lib.ptr(idx), lib.ptr(p), n, d, E, k)
        got.append((xs[:16], y[:16], idx[:16], p[:16]))
    assert all(torch.equal(a, b) and torch.equal(a, c) for a, b, c in zip(*got))
    v = x[:16].double() + delta[:16].cpu().double()
    yn = (v / (v.pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * w.cpu().double())
    # float: sums of 8,192 terms; bfloat16: half a unit in the last place of values up to 16
    assert float((got[0][1].cpu().double() - yn).abs().max()) < (1e-5 if dtype == torch.float32 else 2.0 ** -5)
    y64, w64, ids = got[0][1].cpu().double(), wr.cpu().double(), got[0][2].cpu().long()
    logits = y64 @ w64.T
    top = torch.topk(logits, k, dim=1)
    # the experts: in range, no one twice, and each place's logit as large as that of the 64-bit choice, within the error of two float sums
    # of d products: d 2^-24 sum |y w| each
    assert bool(((ids >= 0) & (ids < E)).all()) and all(len(set(row.tolist())) == k for row in ids)
    bound = 2 * d * 2.0 ** -24 * (y64.abs() @ w64.abs().T).max(dim=1, keepdim=True).values
    assert bool(((logits.gather(1, ids) - top.values).abs() <= bound).all())
    # 8,192 products of order one summed in float: |error of a logit| < 8,192 * 2^-24 * 8
    assert float((got[0][3].cpu().double() - torch.softmax(top.values, 1)).abs().max()) < 4e-3


@pytest.mark.parametrize("vdim", [32, 96, 128, 256])
@pytest.mark.parametrize("silu", [0, 1])
def test_head_norm_and_gate(vdim, silu):
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(vdim)
    nt, H, eps = 9, 3, 1e-6
    o, w = torch.randn(nt, H, vdim, generator=g), torch.rand(H * vdim, generator=g)
    gate = torch.randn(nt, H * vdim + 8, generator=g).bfloat16()
    y = torch.full((nt, H * vdim), 7.0, dtype=torch.bfloat16, device="cuda")
    d = [t.cuda() for t in (o, gate, w)]
    lib.call("tb_mlstm_out_bf16", lib.ptr(d[0]), lib.ptr(d[1]), H * vdim + 8, lib.ptr(d[2]), lib.ptr(y), nt, H, vdim, eps, silu, H * vdim)
    z = gate[:, :H * vdim].double().view(nt, H, vdim)
    want = o.double() / (o.double().pow(2).mean(2, keepdim=True) + eps).sqrt() * w.double().view(H, vdim) * torch.sigmoid(z) * (z if silu else 1)
    # one rounding to bfloat16: half a unit in the last place, 2^-8 of the value at most, and 2^-19 for the float sums and the gate
    assert bool(((y.cpu().double().view(nt, H, vdim) - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -19) + 1e-30).all())
