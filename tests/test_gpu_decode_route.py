"""Which way a decode step takes, one kernel or launches (decode_grid_takes in csrc/decode_grid.cu), and that it makes no difference
beyond rounding."""
import numpy as np
import pytest

from ferrum_gpu_b200 import CudaLlama, QKind
from ferrum_gpu_b200.hostmodel import LlamaConfig, random_llama, random_tokens

pytestmark = pytest.mark.gpu


# 12 heads of their own make 96 items of 8 rows, one for two thirds of the CTAs, whatever the length: one kernel up to some 1500
# positions (measured 45 and 48 us a layer at 1000, 66 and 59 at 2000); heads in groups are split and stay longer
@pytest.mark.parametrize("kv_heads, streams, positions, one", [
    (12, 8, 100, True), (12, 8, 1000, True), (12, 8, 3000, False), (12, 1, 3000, True), (12, 3, 3000, True), (4, 8, 3000, True)])
def test_long_caches_of_many_heads_go_as_launches(dev, kv_heads, streams, positions, one):
    cfg = LlamaConfig(vocab=256, ctx=4096, dim=768, heads=12, kv_heads=kv_heads, head_dim=64, layers=2, hidden=3072, rope_dim=64)
    g = CudaLlama(dev, random_llama(cfg, seed=3, std=0.03), QKind.Q4_0, max_streams=8)
    ids = random_tokens(5, positions, cfg.vocab)
    slots = list(range(streams))
    for s in slots:
        for at in range(0, positions, 1000):
            g.prefill(ids[at:at + 1000], stream=s)
    tok = random_tokens(6, streams, cfg.vocab)
    before = dev.launch_count()
    _, rows = g.feed_batch(tok, streams=slots, want_logits=True)
    assert (dev.launch_count() - before == 1) == one
    if streams > 1:  # a stream by itself always goes as one kernel
        g.reset(0)
        for at in range(0, positions, 1000):
            g.prefill(ids[at:at + 1000], stream=0)
        alone = g.feed(int(tok[0]), stream=0)
        # both are f32-class: each within the library's 1e-5 of exact arithmetic
        assert np.max(np.abs(rows[0] - alone) / np.maximum(np.abs(alone), 1.0)) < 2e-5
    g.close()
