"""Which kernel a prompt takes: the rules on the host, without a GPU, at both sides of what was measured."""
from types import SimpleNamespace

import pytest

from transformer_b200.parts.attention import window_tcgen05_pays
from transformer_b200.parts.channel_delta import wide_scan_pays
from transformer_b200.parts.latent_attention import tc_pays


def _step(lens, before):
    """What the rules look at of a step's context."""
    tiles = lambda size: SimpleNamespace(count=sum(-(-n // size) for n in lens))
    return SimpleNamespace(plans={}, nt=sum(lens), B=len(lens), h_lens=lens, h_pos0=before, tiles=tiles, engine=SimpleNamespace(sm_count=148))


@pytest.mark.parametrize("lens,H,dim,vdim,pays", [
    ([700] * 3, 16, 128, 128, True), ([600] * 4, 16, 128, 128, True), ([1024] * 8, 16, 128, 128, True), ([700] * 5, 8, 128, 128, True),
    ([1000, 900, 400, 300], 16, 128, 128, True), ([2000, 1500, 1200, 800, 600, 400, 300, 300], 16, 128, 128, True),
    ([2048], 16, 128, 128, False), ([1500] * 2, 16, 128, 128, False), ([2048], 32, 128, 128, False), ([600, 1000, 400], 16, 128, 128, False),
    ([1800, 200, 200, 200], 16, 128, 128, False), ([1024] * 8, 16, 64, 64, False), ([1024] * 8, 16, 128, 48, False)])
def test_delta_scan(lens, H, dim, vdim, pays):
    assert wide_scan_pays(lens, H, dim, vdim, 148) is pays


@pytest.mark.parametrize("heads,lens,before,pays", [
    (16, [2039], [0], True), (16, [300] * 4, [0] * 4, True), (16, [100] * 16, [0] * 16, True), (16, [16] * 40, [1000] * 40, True),
    (16, [6] * 200, [0] * 200, True), (8, [6] * 200, [0] * 200, True), (16, [2] * 420, [2000] * 420, False), (8, [2] * 420, [300] * 420, False)])
def test_latent_attention(heads, lens, before, pays):
    ctx, m = _step(lens, before), SimpleNamespace(tc_tile=128 // heads)
    assert tc_pays(ctx, m) is pays and tc_pays(ctx, m) is pays


@pytest.mark.parametrize("nh,nkvh,dh,lens,before,window,chunk,pays", [
    (16, 4, 128, [2048], [0], 2048, 0, True), (16, 4, 128, [600] * 2, [0] * 2, 2048, 0, True), (16, 4, 128, [300], [0], 2048, 0, True),
    (16, 4, 128, [400] * 4, [1500] * 4, 2048, 0, True), (16, 16, 128, [2048], [0], 64, 0, True), (64, 1, 128, [512], [4000], 2048, 0, True),
    (8, 8, 64, [600] * 2, [0] * 2, 2048, 0, True), (2, 1, 128, [2048], [0], 2048, 0, False), (4, 4, 128, [512], [512], 2048, 0, False),
    (16, 4, 128, [300] * 4, [0] * 4, 64, 0, False), (16, 4, 128, [300] * 4, [0] * 4, 2048, 64, False), (64, 1, 128, [300] * 4, [0] * 4, 2048, 0, False),
    (8, 1, 64, [600] * 2, [0] * 2, 64, 0, False), (16, 4, 128, [129] * 8, [0] * 8, 2048, 0, False), (16, 4, 64, [512], [4000], 2048, 0, False)])
def test_windowed_attention(nh, nkvh, dh, lens, before, window, chunk, pays):
    ctx, m = _step(lens, before), SimpleNamespace(tc_tile=128, nh=nh, nkvh=nkvh, dh=dh, chunk=chunk)
    assert window_tcgen05_pays(ctx, m, window) is pays and window_tcgen05_pays(ctx, m, window) is pays
