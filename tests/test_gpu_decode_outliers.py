"""One row of the one-kernel decode (csrc/decode_grid.cu) where a product's input has elements far larger than their neighbours, with
weights of zero behind them: x travels as two fp16 terms at its 32-block's magnitude, which must not cost the neighbours their
bits."""
import numpy as np
import pytest

from ferrum_gpu_b200 import CudaGpt2, CudaLlama, QKind
from ferrum_gpu_b200.hostmodel import Gpt2Config, LlamaConfig, random_gpt2, random_llama, random_tokens
from oracle import oracle as orc
from tests import helpers
from tests.test_gpu_decode_grid import bounds, np_gpt2_forward

pytestmark = pytest.mark.gpu


# up to 2^24 most blocks fit the terms; beyond, blocks go as they are; at 2^100 their scale would leave the normal floats
@pytest.mark.parametrize("e", [0, 16, 24, 30, 40, 100])
@pytest.mark.parametrize("name, kind", [("gpt2", QKind.Q8_0), ("gpt2", QKind.Q4_0), ("llama", QKind.Q8_0)])
def test_small_elements_beside_large_ones_keep_their_bits(dev, name, kind, e):
    ids = random_tokens(3, 70, 256)
    big = np.float32(2.0 ** e)
    if name == "gpt2":  # units of the hidden layer that are always on and go nowhere
        dim = 384 if kind == QKind.Q8_0 else 256
        cfg = Gpt2Config(vocab=256, ctx=80, dim=dim, heads=dim // 64, layers=2, hidden=4 * dim)
        m = random_gpt2(cfg, seed=5, std=0.05, bias_std=0.05, gain_jitter=0.1)
        for b in m.blocks:
            for j in (3, 40, 41, 4 * dim - 1):
                b.b1[j] = big
                b.w2.reshape(cfg.hidden, dim)[j] = 0.0
        ref, forward = orc.dequantised_gpt2(m, int(kind), snap_embedding=False), np_gpt2_forward
        g = CudaGpt2(dev, m, kind)
    else:  # channels of v that are a constant, and whose rows of wo are zero
        cfg = LlamaConfig(vocab=256, ctx=80, dim=384, heads=6, kv_heads=2, head_dim=64, layers=2, hidden=512, rope_dim=64)
        m = random_llama(cfg, seed=5, biases=True, std=0.05, gain_jitter=0.1)
        for b in m.blocks:
            for j in (5, 64 + 33):
                b.bv[j] = big
                for h in range(3):
                    b.wo.reshape(cfg.q_dim, cfg.dim)[(j // 64 * 3 + h) * 64 + j % 64] = 0.0
        ref, forward = orc.dequantised_llama(m, int(kind), snap_embedding=False), helpers.np_llama_forward
        g = CudaLlama(dev, m, kind)
    want = forward(ref, ids, np.float64)
    tol = bounds(want, forward(ref, ids, np.float32))
    for n, t in enumerate(ids):
        before = dev.launch_count()
        got = g.feed(int(t))
        assert dev.launch_count() - before == 1
        assert orc.max_rel_err(got, want[n]) < tol[n], n
    g.close()

