"""Chains of greedy steps in the one-kernel decode (csrc/decode_grid.cu) when the number of streams changes between them: which
group of rows a stream belongs to depends on how many there are, so what one call left behind must mean nothing to the next."""
import random

import numpy as np
import pytest

from ferrum_gpu_b200 import CudaLlama, QKind
from ferrum_gpu_b200.hostmodel import LlamaConfig, random_llama, random_tokens

pytestmark = pytest.mark.gpu

CFG = LlamaConfig(vocab=1000, ctx=64, dim=256, heads=4, kv_heads=2, head_dim=64, layers=2, hidden=256, rope_dim=64)


def drawn(seed, calls):
    rng = random.Random(seed)
    return [(rng.randint(1, 24), rng.randint(1, 16)) for _ in range(calls)]


# (streams, steps) of every call. Tags advance by three (layers + 1) a step: in the first two the second call waits for a tag
# that the first one left at the rows of another group; among the drawn ones three calls do.
@pytest.mark.parametrize("calls", [[(8, 3), (10, 3)], [(16, 3), (17, 3)], [(8, 3), (9, 4), (20, 3), (17, 5)], drawn(14, 60)],
                         ids=["8_10", "16_17", "8_9_20_17", "drawn"])
def test_chains_of_changing_widths_are_their_steps(dev, calls):
    m = random_llama(CFG, seed=9, std=0.2)
    g = CudaLlama(dev, m, QKind.Q8_0, max_streams=24)
    ref = CudaLlama(dev, m, QKind.Q8_0, max_streams=24)
    for i, (streams, steps) in enumerate(calls):
        first = random_tokens(100 + i, streams, CFG.vocab)
        for s in range(streams):
            g.reset(s)
            ref.reset(s)
        slots = list(range(streams))
        before = dev.launch_count()
        got = g.decode_greedy(first, steps, streams=slots)
        assert dev.launch_count() - before == min(steps, 2), "the one-kernel route"
        tok = first
        for step in range(steps):
            tok, _ = ref.feed_batch(tok, streams=slots)
            assert np.array_equal(tok, got[step]), (i, streams, step)
        # the caches that both left behind
        _, a = g.feed_batch(tok, streams=slots, want_logits=True)
        _, b = ref.feed_batch(tok, streams=slots, want_logits=True)
        assert np.array_equal(a, b), (i, streams)
    g.close()
    ref.close()


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
def test_a_chain_where_most_ctas_have_attention_and_nothing_after_it(dev, kind):
    """48 heads of one or three streams are 48 or 144 attention items, and everything behind them 65 tiles of a few
    CTAs: the others go from a step's last item straight to the next step's plan, which lies where their copies' was."""
    cfg = LlamaConfig(vocab=16, ctx=320, dim=256, heads=48, kv_heads=48, head_dim=64, layers=1, hidden=256, rope_dim=64)
    m = random_llama(cfg, seed=3, std=0.3)
    g = CudaLlama(dev, m, kind, max_streams=3)
    ref = CudaLlama(dev, m, kind, max_streams=3)
    for streams in (1, 3):
        slots = list(range(streams))
        first = random_tokens(5, streams, cfg.vocab)
        for s in slots:
            g.reset(s)
            ref.reset(s)
        got = g.decode_greedy(first, 240, streams=slots)
        tok = first
        for step in range(240):
            tok, _ = ref.feed_batch(tok, streams=slots)
            assert np.array_equal(tok, got[step]), (streams, step)
        _, a = g.feed_batch(tok, streams=slots, want_logits=True)
        _, b = ref.feed_batch(tok, streams=slots, want_logits=True)
        assert np.array_equal(a, b)
    g.close()
    ref.close()


# heads, K/V heads, streams, tokens before the chain, its steps, a few of the launches it may take
@pytest.mark.parametrize("heads, kv_heads, streams, prompt, steps", [
    (4, 2, 1, 250, 20),    # past the 256 positions beyond which the attention is split
    (4, 2, 3, 310, 140),   # a split more every 64 positions
    (12, 12, 8, 1760, 120), # from one kernel to launches
    (12, 4, 12, 250, 20),
], ids=["split", "splits", "to_launches", "groups"])
def test_a_chain_is_its_single_steps_bit_for_bit(dev, heads, kv_heads, streams, prompt, steps):
    """How a step runs and how its attention is cut depends on its positions; a chain changes where its single steps would."""
    cfg = LlamaConfig(vocab=500, ctx=2000, dim=256 * (heads // 4), heads=heads, kv_heads=kv_heads, head_dim=64, layers=2,
                      hidden=3072 if heads == 12 else 512, rope_dim=64)
    m = random_llama(cfg, seed=2, std=0.05)
    g = CudaLlama(dev, m, QKind.Q4_0, max_streams=streams)
    ids = random_tokens(8, prompt, cfg.vocab)
    first = random_tokens(9, streams, cfg.vocab)
    slots = list(range(streams))

    def start():
        for s in slots:
            g.reset(s)
            for at in range(0, prompt - 3 * s, 1000):
                g.prefill(ids[at:min(at + 1000, prompt - 3 * s)], stream=s)

    start()
    before = dev.launch_count()
    chain = g.decode_greedy(first, steps, streams=slots)
    launches = dev.launch_count() - before
    _, after = g.feed_batch(chain[-1], streams=slots, want_logits=True)
    start()
    tok, single = first, set()
    for step in range(steps):
        before = dev.launch_count()
        tok, _ = g.feed_batch(tok, streams=slots)
        single.add(dev.launch_count() - before)
        assert np.array_equal(tok, chain[step]), step
    # (the caches, down to the last bit of what the chain's attention gave the layer above)
    assert np.array_equal(g.feed_batch(tok, streams=slots, want_logits=True)[1], after)
    if (heads, kv_heads) == (12, 12):
        assert min(single) == 1 < max(single), "some steps as one kernel, some as launches"
    elif streams <= 8:
        assert single == {1} and launches <= 2 + steps // 64 + 1
    g.close()
