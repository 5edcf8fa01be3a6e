"""Sampling with a small top_k, where the candidates are collected and sorted: ties at the edge, more ties than candidates,
rows that do not start on 16 bytes, rows of minus infinity, and the largest top_k, against the rules in 64 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kept(row, t, k, p):
    """ids (ascending) and probabilities of what the rules keep."""
    z = (row.float() * np.float32(1.0 / np.float32(t))).double().numpy()
    order = np.lexsort((np.arange(len(z)), -z))[:k]
    w = np.exp(z[order] - z[order[0]])
    if p < 1.0:
        order = order[:int(np.searchsorted(np.cumsum(w), p * w.sum()) + 1)]
    ids = np.sort(order)
    w = np.exp(z[ids] - z.max())
    return ids, np.cumsum(w) / w.sum()


@pytest.mark.parametrize("kind,V,k", [("plain", 32000, 40), ("plain", 32001, 256), ("plain", 300, 299), ("plain", 1025, 2),
                                      ("ties", 32000, 40), ("ties", 3001, 256), ("flat", 32000, 40), ("sparse", 32000, 40)])
@pytest.mark.parametrize("p", [0.9, 1.0])
def test_against_the_rules(kind, V, k, p):
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(V + k)
    rows, t = 4, 0.8
    x = torch.randn(rows, V, generator=g) * 3
    if kind == "ties":                  # the edge of top_k lies among equal values
        x = torch.minimum(x, x.sort(dim=1, descending=True).values[:, k // 2:k // 2 + 1])
    if kind == "flat":                  # more equal values than candidates
        x = torch.where(torch.arange(V) % 7 == 3, torch.full_like(x, 2.0), x.clamp(max=1.9))
    if kind == "sparse":                # fewer finite values than top_k
        x = torch.where(torch.arange(V) % 2000 == 5, x, torch.full_like(x, -float("inf")))
    d = x.cuda()
    idx, val = torch.empty(rows, dtype=torch.int32, device="cuda"), torch.empty(rows, device="cuda")
    for u in (0.0, 0.13, 0.5, 0.77, 0.999999):
        uu = torch.full((rows,), u, device="cuda")
        lib.call("tb_sample", lib.ptr(d), d.stride(0), lib.ptr(uu), rows, V, t, k, p, lib.ptr(idx), lib.ptr(val))
        for r, (i, v) in enumerate(zip(idx.tolist(), val.tolist())):
            ids, cum = _kept(x[r], t, k, p)
            at = int(np.searchsorted(ids, i))
            assert at < len(ids) and ids[at] == i and v == float(x[r, i])
            # float sums of at most 256 terms: 256 * 2^-24 of the mass at either edge
            assert (cum[at - 1] if at else 0.0) - 2e-5 <= u <= cum[at] + 2e-5


@pytest.mark.parametrize("nt", [1, 3, 4, 5, 6, 7, 40])
@pytest.mark.parametrize("nh,nkvh,dh", [(4, 1, 128), (5, 1, 64), (2, 2, 16), (6, 2, 32), (4, 2, 64)])
def test_decode_attention_in_32_bits(nt, nh, nkvh, dh):
    """Few heads (up to 8, 16 or 24 by the size of a group) take a block each with 512 threads, more the one-, two- and four-head
    forms: all against 64 bits.  Scores of unit
    normal values over sqrt(dh): 1e-5 covers the float sums of 700 keys."""
    from transformer_b200.csrc import lib
    g = torch.Generator().manual_seed(nt + dh)
    lens = [[1, 64, 700, 65, 200, 63][i % 6] for i in range(nt)]
    pages = [(n + 63) // 64 for n in lens]
    table, at = torch.zeros(nt, max(pages), dtype=torch.int32), 0
    perm = torch.randperm(sum(pages), generator=g)
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    k, v = (torch.randn(sum(pages), nkvh, 64, dh, generator=g) for _ in range(2))
    q = torch.randn(nt, nh * dh, generator=g)
    splits = max(1, min(32, 1184 // (nt * nkvh * ((nh // nkvh + 3) // 4))))
    out, part = torch.empty(nt, nh * dh, device="cuda"), torch.empty(nt, nh, splits, dh + 2, device="cuda")
    I = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    d = [t.cuda() for t in (q, k, v, table)]
    seq, pos = I(list(range(nt))), I([n - 1 for n in lens])
    lib.call("tb_attention_decode_f32", lib.ptr(d[0]), lib.ptr(out), lib.ptr(d[1]), lib.ptr(d[2]), lib.ptr(seq), lib.ptr(pos),
             lib.ptr(d[3]), lib.ptr(part), nt, max(pages), nh * dh, nh, nkvh, dh, splits, dh ** -0.5)
    got = out.cpu().double().view(nt, nh, dh)
    for b, n in enumerate(lens):
        rows = lambda x: x[table[b, :pages[b]].long()].permute(1, 0, 2, 3).reshape(nkvh, -1, dh)[:, :n].double().repeat_interleave(nh // nkvh, 0)
        s = torch.softmax(torch.einsum("hd,hnd->hn", q[b].double().view(nh, dh), rows(k)) * dh ** -0.5, -1)
        assert float((got[b] - torch.einsum("hn,hnd->hd", s, rows(v))).abs().max()) < 1e-5
