"""Products by pairs of blocks on the tensor cores, at sizes around the rule that chooses them: the bits of the same product made in pieces
of at most 128 rows (which single blocks take: a tcgen05 product adds along K in one order), and a few columns against 64 bits.
Which form a product takes is asked of the rule itself, so a case says where it lies.

The bound of the second: float sums of K products of bfloat16 values, error at most K 2^-24 of the sum of their absolute values,
and one rounding to bfloat16 (2^-9 of the value), through the pair's silu(g) u (slope at most 1.1) at most doubled.  With biases both
products are rounded to bfloat16 before these are added: 2^-9 of either product, times the other factor, doubled likewise."""
import pytest
import torch

SMS = 148       # of the GPU that the rule was measured on


def _takes_pairs(rows, N, K, kind, sms=SMS):
    from transformer_b200.csrc import lib
    return bool(lib.library().tb_gemm_tc_takes_pairs(sum(rows), N, K, len(rows), int(len(rows) > 1), min(kind, 2), sms))


def _call(a, w, out, offsets, N, kind, bias=None):
    from transformer_b200.csrc import lib
    M, K = a.shape
    if bias is not None:
        lib.call("tb_gemm_tc_bias_glu_bf16", lib.ptr(a), lib.ptr(w), lib.ptr(bias), lib.ptr(out), K, K, out.shape[1], M, N, K, out.shape[1] - N)
    else:
        lib.call("tb_gemm_tc_bf16", lib.ptr(a), lib.ptr(w), lib.ptr(out), lib.ptr(offsets) if offsets is not None else 0, K, K, out.shape[1],
                 M, N, K, w.shape[0], kind)


@pytest.mark.parametrize("rows,N,K,kind,pairs", [
    ([3000], 2048, 128, 0, False), ([3000], 2048, 504, 0, False), ([3000], 2048, 512, 0, True), ([128], 32000, 2048, 1, False), ([129], 32000, 2048, 1, True),
    ([200], 5632, 4096, 2, False), ([128] * 16, 688, 4096, 2, False), ([129] * 16, 688, 4096, 2, True), ([512] * 16, 688, 4096, 2, False),
    ([640] * 16, 688, 4096, 2, True), ([512] * 8, 14336, 4096, 2, True), ([512] * 8, 4096, 14336, 0, False), ([511] * 16, 4096, 688, 0, False),
    ([512] * 16, 4096, 688, 0, True)])
def test_sides_of_the_line(rows, N, K, kind, pairs):
    assert _takes_pairs(rows, N, K, kind) is pairs


@pytest.mark.gpu
@pytest.mark.parametrize("rows,N,K,kind,pairs", [
    ([1300], 2000, 1032, 2, True), ([1299], 2008, 1024, 3, True), ([385], 20000, 1032, 1, True), ([1025], 4104, 2048, 0, True),
    ([300], 5632, 1024, 2, False), ([512], 18944, 1024, 1, True), ([3000], 2048, 504, 0, False), ([3000], 2048, 520, 0, True),
    ([0, 257, 1, 700, 256, 255, 511, 3, 129, 900, 0, 40, 513, 300, 128, 600], 688, 1024, 2, False),
    ([384, 0, 500, 257, 1, 768, 129, 600, 450, 300, 420, 512, 380, 700, 390, 353], 688, 1032, 2, True),
    ([0, 257, 1, 1500, 256, 755, 511, 3, 129, 2100, 0, 740, 513, 1300, 828, 1400], 688, 1024, 2, True),
    ([700, 0, 640, 1, 900, 129, 257, 1030], 1408, 1032, 2, True),
    ([600, 1, 2047, 300, 1000, 260, 512, 0], 2056, 520, 0, True), ([600, 0, 700, 500], 4096, 688, 0, False)])
def test_pairs(rows, N, K, kind, pairs):
    from transformer_b200.csrc import lib
    if torch.cuda.get_device_properties(0).multi_processor_count == SMS:
        assert _takes_pairs(rows, N, K, kind, 0) is pairs
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    M, G, dual = sum(rows), len(rows), kind >= 2
    a = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    w = (torch.randn(G, 2 * N if dual else N, K, device="cuda", generator=gen) * K ** -0.5).bfloat16()
    bias = torch.randn(2 * N, device="cuda", generator=gen) if kind == 3 else None
    ldc = N + (8 if bias is not None else 0)
    new = lambda m: torch.full((m, ldc), float("nan"), dtype=torch.float32 if kind == 1 else torch.bfloat16, device="cuda")
    starts = torch.tensor([0] + rows, dtype=torch.int32).cumsum(0).int()
    whole, pieces = new(M), new(M)
    _call(a, w, whole, starts.cuda() if G > 1 else None, N, kind, bias)
    for g in range(G):
        for r in range(int(starts[g]), int(starts[g + 1]), 128):
            end = min(r + 128, int(starts[g + 1]))
            _call(a[r:end], w[g:g + 1], pieces[r:end], None, N, kind, bias)
    assert not lib.library().tb_gemm_tc_status()
    assert bool(torch.isfinite(whole).all()) and torch.equal(whole, pieces)
    cols = torch.tensor([0, 1, N // 2, N - 1], device="cuda")
    for g in range(G):
        x, got = a[starts[g]:starts[g + 1]].double(), whole[starts[g]:starts[g + 1]][:, cols].double()
        if not len(x):
            continue
        of = lambda first: (x @ w[g, first + cols].double().T, x.abs() @ w[g, first + cols].double().abs().T)
        want, size = of(0)
        rounded = 0.0
        if dual:
            g0, (u0, up_size) = want, of(N)
            up = u0
            if bias is not None:
                want, up = g0 + bias[cols].double(), u0 + bias[N + cols].double()
                rounded = (g0 * up).abs() + (u0 * want).abs()
            size, want = size * (up.abs() + up_size * K * 2.0 ** -24) + up_size * want.abs(), want * torch.sigmoid(want) * up
        bound = 2 * size * K * 2.0 ** -24 + (want.abs() + rounded) * 2.0 ** -8 + 1e-6
        assert bool(((got - want).abs() <= bound).all())
