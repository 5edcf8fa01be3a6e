"""The 32-bit products at the edges of their kernels: passes of 4, 8 and 16 rows, four and eight warps on K, tiles of
64 x 64 with remainders, groups that are empty or hold a remainder, gathered rows, rows the 16-byte kernels refuse, and rows
below 512 entries, which the general kernel takes.

The bound is that of any order of summation in float: |error| <= (K + 8) 2^-24 sum |a b| for a product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).cuda()


def _product(a, w):
    """(a w^T in 64 bits, bound of a float product's error)."""
    a, w = a.double(), w.double()
    return a @ w.T, (a.shape[1] + 8) * 2.0 ** -24 * (a.abs() @ w.abs().T)


@pytest.mark.parametrize("M,N,K", [(1, 8, 4), (3, 1536, 1024), (4, 130, 516), (5, 67, 260), (8, 1, 2048), (9, 33, 124),
                                   (16, 100, 1028), (17, 64, 36), (63, 65, 32), (64, 64, 96), (130, 200, 100), (254, 129, 520),
                                   (3, 20, 1022), (70, 40, 33), (1, 8, 256), (4, 130, 260), (9, 33, 380),
                                   (17, 64, 292), (63, 65, 288), (64, 64, 352), (130, 200, 356), (254, 129, 260),
                                   (1, 8, 512), (5, 67, 516), (9, 33, 636), (17, 64, 548), (63, 65, 512), (64, 64, 608),
                                   (130, 200, 612)])
@pytest.mark.parametrize("kind", [0, 3])
def test_dense(M, N, K, kind):
    from transformer_b200.parts.linear import gemm_simt
    a, w = _rand((M, K), 1), _rand((N, K), 2)
    out = torch.full((M, N + 3), 7.0, device="cuda")
    gemm_simt(a, w, out[:, :N], out_kind=kind)
    want, bound = _product(a, w)
    if kind == 3:
        bound = (2 * want.clamp(min=0) + bound) * bound + 2.0 ** -23 * want ** 2
        want = want.clamp(min=0) ** 2
    assert bool(((out[:, :N].double() - want).abs() <= bound).all())
    assert bool((out[:, N:] == 7.0).all()), "nothing past the last column is written"


@pytest.mark.parametrize("sizes", [[0] * 39 + [640], [300] + [0] * 39, [257, 0, 1, 256] + [0] * 50 + [255, 12],
                                   [65, 129, 0, 64] + [1] * 76, [130] + [0] * 99, [16] * 40])
def test_crowded_groups_are_dealt_to_several_blocks(sizes):
    """Few rows a group on average (the weights' kernel) and one group with many: slices of 16 passes of 4, 8 or 16 rows, found
    by 32 groups at a time."""
    from transformer_b200.parts.linear import gemm_simt
    G, M, N, K = len(sizes), sum(sizes), 37, 516
    assert 16 * 4 < M <= 16 * G
    x, w = _rand((M, K), 8), _rand((G, N, K), 9) * K ** -0.5
    offsets = torch.tensor([0] + sizes).cumsum(0).to(torch.int32).cuda()
    out = torch.full((M, N), 7.0, device="cuda")
    gemm_simt(x, w, out, group_offsets=offsets, groups=G)
    at = 0
    for g, n in enumerate(sizes):
        if n:
            want, bound = _product(x[at:at + n], w[g])
            assert bool(((out[at:at + n].double() - want).abs() <= bound).all())
        at += n


@pytest.mark.parametrize("M,N,K", [(3, 40, 1024), (17, 70, 512), (45, 33, 516), (48, 64, 64), (49, 65, 520)])
@pytest.mark.parametrize("kind", [0, 2])
def test_groups_without_offsets_take_the_first_matrix(M, N, K, kind):
    """Up to and above 16 rows a group, where another kernel takes over: every block that writes a place has matrix 0."""
    from transformer_b200.parts.linear import gemm_simt
    a, w = _rand((M, K), 6), _rand((3, N if kind == 0 else 2 * N, K), 7) * K ** -0.5
    out, one = torch.full((M, N), 7.0, device="cuda"), torch.full((M, N), 7.0, device="cuda")
    for _ in range(20):
        gemm_simt(a, w, out, groups=3, out_kind=kind)
        gemm_simt(a, w[0], one, out_kind=kind)
        assert torch.equal(out, one)
    if kind == 0:
        want, bound = _product(a, w[0])
        assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("sizes,N,K", [([1, 0, 2], 512, 1024), ([0, 3, 0, 5, 1], 44, 300), ([40, 0, 3, 1], 33, 260),
                                       ([100, 64, 0, 65, 1], 70, 36), ([6, 6, 6, 6], 24, 22),
                                       ([100, 64, 0, 65, 1], 70, 292), ([0, 3, 0, 5, 1], 44, 256),
                                       ([100, 64, 0, 65, 1], 70, 548), ([0, 3, 0, 5, 1], 44, 512), ([40, 0, 3, 1], 33, 516)])
@pytest.mark.parametrize("glu", [None, (1.702, 7.0)])
def test_grouped_pair_of_gathered_rows(sizes, N, K, glu):
    from transformer_b200.parts.linear import gemm_simt
    G, M = len(sizes), sum(sizes)
    x, w = _rand((M + 5, K), 3), _rand((G, 2 * N, K), 4) * K ** -0.5
    rows = torch.randperm(M + 5, generator=torch.Generator().manual_seed(5))[:M].to(torch.int32).cuda()
    offsets = torch.tensor([0] + sizes).cumsum(0).to(torch.int32).cuda()
    out = torch.full((M, N), 7.0, device="cuda")
    gemm_simt(x, w, out, a_rows=rows, group_offsets=offsets, groups=G, out_kind=2, glu=glu)
    at = 0
    for g, n in enumerate(sizes):
        z, bound = _product(x[rows[at:at + n].long()], w[g])
        zg, zu, bg, bu = z[:, :N], z[:, N:], bound[:, :N], bound[:, N:]
        if glu is None:
            f, u = zg * torch.sigmoid(zg), zu
            slope = 1.1             # the largest of silu's
        else:
            zg = zg.clamp(max=glu[1])
            f, u = zg * torch.sigmoid(glu[0] * zg), zu.clamp(-glu[1], glu[1]) + 1.0
            slope = 1.1             # that of z sigmoid(alpha z) does not depend on alpha
        limit = slope * bg * (u.abs() + bu) + f.abs() * bu + 2.0 ** -20 * (f * u).abs() + 1e-7
        assert bool(((out[at:at + n].double() - f * u).abs() <= limit).all())
        at += n
