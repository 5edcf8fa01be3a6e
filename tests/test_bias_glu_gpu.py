"""The (gate, up) pair with biases in the products' epilogues against the product stored in bfloat16 and a pass over it: the same
bits, a one and zeros behind the results, and nothing further."""
import pytest
import torch



@pytest.mark.parametrize("M,n,K,pays", [
    (1, 2816, 1024, True), (8, 5632, 2048, True), (16, 2816, 2048, True), (16, 5632, 2048, False), (1, 11008, 4096, False),
    (17, 2816, 1024, False), (100, 5632, 2048, False), (512, 5632, 2048, False), (1000, 11008, 4096, False), (1200, 2816, 4096, False),
    (2048, 2816, 1024, False), (1500, 5632, 2048, True), (2048, 5632, 1024, True), (4096, 2816, 1024, True)])
def test_sides_of_the_line(M, n, K, pays):
    from transformer_b200.parts.linear import bias_glu_pays
    assert bias_glu_pays(M, n, K) is pays


@pytest.mark.gpu
@pytest.mark.parametrize("M", [17, 100, 131, 700, 2048])
@pytest.mark.parametrize("n,K", [(2816, 1024), (5632, 2048)])
def test_bits_of_the_library_product_and_the_pass(M, n, K):
    """At the sizes of models: whichever of the two a step takes, its results do not change."""
    from transformer_b200.csrc import lib
    from transformer_b200.parts.linear import bias_glu_matmul
    g = torch.Generator().manual_seed(M + n)
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), (torch.randn(2 * n, K, generator=g) * 2 * K ** -0.5).bfloat16().cuda()
    bias = torch.randn(2 * n, generator=g).cuda()
    h, want = (torch.empty(M, n + 8, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert bias_glu_matmul(x, w, bias, h)
    gu = torch.mm(x, w.t())
    lib.call("tb_bias_glu_bf16", lib.ptr(gu), lib.ptr(bias), lib.ptr(want), M, n, n + 8)
    assert lib.gemm_tc_status() == 0
    assert torch.equal(h, want)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 7, 9, 16, 17, 128, 129, 700])
@pytest.mark.parametrize("n,K", [(8, 64), (40, 512), (128, 2048), (136, 72), (688, 2056)])
def test_pair_with_biases(M, n, K):
    from transformer_b200.csrc import lib
    from transformer_b200.parts.linear import bias_glu_matmul
    g = torch.Generator().manual_seed(M + n + K)
    x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), (torch.randn(2 * n, K, generator=g) * 2 * K ** -0.5).bfloat16().cuda()
    bias = torch.randn(2 * n, generator=g).cuda()
    for wide in (n, n + 8):
        h = torch.full((M + 1, wide), 7.0, dtype=torch.bfloat16, device="cuda")
        assert bias_glu_matmul(x, w, bias, h[:M])
        assert lib.gemm_tc_status() == 0
        gu, want = torch.empty(M, 2 * n, dtype=torch.bfloat16, device="cuda"), torch.empty(M, wide, dtype=torch.bfloat16, device="cuda")
        if M <= 16:
            lib.call("tb_gemm_skinny_bf16", lib.ptr(x), 0, lib.ptr(w), lib.ptr(gu), 0, 0, K, K, 2 * n, M, 2 * n, K, 1, 0, 0, 0, 1, 1)
        else:
            lib.call("tb_gemm_tc_bf16", lib.ptr(x), lib.ptr(w), lib.ptr(gu), 0, K, K, 2 * n, M, 2 * n, K, 1, 0)
        lib.call("tb_bias_glu_bf16", lib.ptr(gu), lib.ptr(bias), lib.ptr(want), M, n, wide)
        assert torch.equal(h[:M], want) and bool((h[M] == 7.0).all())
        gate, up = (gu.double()[:, :n] + bias[:n]), gu.double()[:, n:] + bias[n:]
        exact = gate / (1 + torch.exp(-gate)) * up
        # one rounding of the result, a few roundings in 32 bits before it
        assert float(((h[:M, :n].double() - exact).abs() - 2.0 ** -8 * exact.abs()).max()) <= 1e-5
