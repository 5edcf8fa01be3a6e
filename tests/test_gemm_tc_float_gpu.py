"""The tcgen05 product with float results: whole lines through shared memory against row-by-row stores (a pitch that is no
multiple of four takes those): the same sums, so the same bits, and nothing written outside the product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 33, 128, 300])
@pytest.mark.parametrize("N,K", [(4, 64), (36, 72), (252, 200), (260, 64), (1000, 136), (300, 1000)])
def test_lines_have_the_bits_of_rows(M, N, K):
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    outs = []
    for pitch in (N, N + 4, N + 1):
        out = torch.full((M + 1, pitch), 7.0, device="cuda")
        assert lib.try_call("tb_gemm_tc_bf16", lib.ptr(a), lib.ptr(w), lib.ptr(out), 0, K, K, pitch, M, N, K, 1, 1)
        assert lib.gemm_tc_status() == 0
        assert bool((out[:, N:] == 7.0).all()) and bool((out[M] == 7.0).all())
        outs.append(out[:M, :N])
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[2])
    want = a.double() @ w.double().T
    # sums of K products in 32 bits
    assert float(((outs[0].double() - want).abs() - K * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)).max()) <= 0
