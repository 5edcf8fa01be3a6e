"""The (gate, up) pair with biases in the products' epilogues against the product stored in bfloat16 and a pass over it: the same
bits, a one and zeros behind the results, and nothing further."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
