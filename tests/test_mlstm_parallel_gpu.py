"""The matrix memory with the chunks of a sequence side by side against the kernel that walks them: the same sums in the same
order, so the same bits, outputs and state, over two steps of sequences around a chunk's edges; all chunks at once, and in
portions that end inside and between sequences."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,dim,vdim", [(8, 128, 256), (4, 128, 256), (3, 64, 32), (2, 8, 160), (1, 256, 96), (2, 136, 128)])
@pytest.mark.parametrize("portion", [99, 1, 3])
def test_same_bits(H, dim, vdim, portion):
    from transformer_b200.csrc import lib
    gen = torch.Generator().manual_seed(dim + vdim)
    B, ld = 5, (2 * H * dim + H * vdim + 7) // 8 * 8 + 8
    per = lib.mlstm_parallel_size(H, dim, vdim, ld)
    assert per > 0
    slots = torch.tensor([4, 0, 5, 2, 1], dtype=torch.int32).cuda()
    start = torch.randn(6, H, lib.mlstm_state_size(dim, vdim), generator=gen).cuda()
    cols = (vdim + 31) // 32
    n_m = start[:, :, dim * vdim:].view(6, H, cols, dim + 1)
    n_m[:] = n_m[:, :, :1].clone()              # every block of columns keeps the same n and m
    states = [start.clone(), start.clone()]
    bias = torch.randn(2 * H, generator=gen).cuda()
    for lens in ([1, 64, 65, 200, 37], [130, 0, 63, 1, 128]):
        nt, chunks = sum(lens), sum(lens) // 64 + B
        z = torch.randn(nt, ld, generator=gen).bfloat16().cuda()
        gates = (torch.randn(nt, 2 * H, generator=gen) * 4).cuda()
        starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
        outs = [torch.full((nt, H * vdim), 7.0, device="cuda") for _ in range(2)]
        here = min(portion, chunks)
        work = torch.full((H, here, per), float("nan"), device="cuda")
        gate_work = torch.full((H, chunks, lib.mlstm_parallel_gates()), float("nan"), device="cuda")
        head = lambda i: (lib.ptr(z), lib.ptr(gates), lib.ptr(bias), lib.ptr(states[i]), lib.ptr(outs[i]))
        lib.call("tb_mlstm_chunk_bf16", *head(0), lib.ptr(starts), lib.ptr(slots), B, ld, H, dim, vdim, 15.0, dim ** -0.5)
        lib.call("tb_mlstm_parallel_bf16", *head(1), lib.ptr(work), lib.ptr(gate_work), lib.ptr(starts), lib.ptr(slots), nt, B,
                 ld, H, dim, vdim, chunks, here, 15.0, dim ** -0.5)
        torch.cuda.synchronize()
        assert bool(torch.isfinite(outs[0]).all()) and torch.equal(outs[0], outs[1])
        assert torch.equal(states[0], states[1])


def test_scratch_of_a_long_step_is_bounded(monkeypatch):
    """A step whose chunks need more than PARALLEL_BYTES of states takes that much scratch and no more, with the same logits."""
    import transformer_b200 as tb
    from transformer_b200.parts import mlstm
    from salepel_tiny import WIDE
    prompt = [(7 * i * i + i) % 120 for i in range(700)]
    logits, sizes = [], []
    for most in (mlstm.PARALLEL_BYTES, 1):
        monkeypatch.setattr(mlstm, "PARALLEL_BYTES", most)
        engine = tb.random_model(WIDE, seed=3, dtype="bfloat16", max_tokens=1024, max_slots=2)
        logits.append(engine.step([engine.open()], [prompt], want=[list(range(0, 700, 50))]).clone())
        sizes.append(engine.workspace._bufs[("mlstm.work", torch.float32)].numel())
    assert torch.equal(*logits) and sizes[0] >= 11 * sizes[1]
