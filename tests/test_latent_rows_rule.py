"""Which latent-attention kernel a step takes: the rule on the host, without a GPU."""
import random

import pytest

from transformer_b200.parts.latent_attention import keys_seen, rows_pay

NONE = 1 << 30


def test_keys_seen_counts_them():
    rng = random.Random(1)
    for _ in range(500):
        n, before, window = rng.randint(1, 60), rng.randint(0, 80), rng.choice([1, 7, 64, 65, NONE])
        assert keys_seen(n, before, window) == sum(min(window, p + 1) for p in range(before, before + n))


# (heads, rank, sequences, new tokens, cached, window): both sides of the measured steps
@pytest.mark.parametrize("heads,rank,batch,n,before,window,pays", [
    (16, 512, 1, 2039, 0, 2048, True), (16, 512, 4, 300, 0, NONE, True), (16, 512, 8, 128, 500, NONE, True),
    (32, 512, 16, 16, 1000, NONE, True), (16, 512, 1, 4096, 0, 256, True), (8, 256, 1, 2039, 0, NONE, True),
    (16, 512, 16, 100, 0, NONE, False), (16, 512, 200, 6, 0, NONE, False), (16, 512, 400, 2, 500, NONE, False),
    (16, 512, 420, 1, 2000, NONE, False), (32, 512, 8, 200, 0, NONE, False), (16, 512, 1, 300, 0, NONE, False),
    (8, 256, 8, 200, 0, NONE, False), (8, 256, 1, 4096, 0, 512, False), (8, 256, 1, 2039, 0, 1024, False),
    (16, 256, 30, 30, 500, NONE, False), (8, 256, 1000, 1, 500, NONE, False), (16, 128, 1, 4096, 0, NONE, False)])
def test_sides_of_the_line(heads, rank, batch, n, before, window, pays):
    tile = 16 // min(heads, 16)
    blocks = batch * -(-n // tile) * -(-heads // 16)
    assert rows_pay([n] * batch, [before] * batch, window, tile, rank, blocks) is pays


def test_a_long_prompt_among_decoding_sequences():
    """What the step's tokens see together decides: few or short others do not turn it, many with long contexts do."""
    step = lambda others, cached: rows_pay([2000] + [1] * others, [0] + [cached] * others, NONE, 1, 512, 2000 + others)
    assert step(9, 1000) and step(100, 500) and not step(600, 4000)
