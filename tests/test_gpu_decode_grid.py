"""The decode step of one to 64 streams as one persistent kernel (csrc/decode_grid.cu), at the sizes where it can go wrong:
positions around the 64-position cache tiles and the limit beyond which a row's positions are split over CTAs (256), inputs
wider than a ring slot (1024 bytes of a weight row), a 256-element part that is half empty, heads whose last tile is ragged,
more head tiles per CTA than go between two barriers (9600 rows), query groups of one, three and eight heads, rows of
different lengths in one to eight groups."""
import numpy as np
import pytest

from ferrum_gpu_b200 import CudaGpt2, CudaLlama, QKind
from ferrum_gpu_b200 import _ffi
from ferrum_gpu_b200.hostmodel import Gpt2Config, LlamaConfig, random_gpt2, random_llama, random_tokens
from oracle import oracle as orc
from tests import helpers

pytestmark = pytest.mark.gpu

# Against exact (f64) arithmetic over the dequantised weights: the reference's own bound of a whole forward pass
# (ferrum_wgpu/src/tolerance.rs:L11), or 2.5 times what numpy's f32 forward pass of the same model (blocked sums) is off at
# that position where the model amplifies rounding beyond it: 0.8e-5 to 2.2e-5 for the wide one (the oracle's serial sums:
# 1.0e-5 to 3.6e-5).
def bounds(exact, f32):
    return [max(1e-5, 2.5 * orc.max_rel_err(b, a)) for a, b in zip(exact, f32)]


LENGTHS = [1, 330, 64, 257, 65, 63, 2, 256]  # tokens before and including the one the step is fed


def np_gpt2_forward(m, ids, f):
    """GPT-2's logits at every position in precision `f`."""
    c = m.cfg
    d, n, hd = c.dim, len(ids), c.dim // c.heads
    x = m.tok.reshape(c.vocab, d)[ids].astype(f) + m.pos.reshape(c.ctx, d)[:n]

    def norm(x, g, b):
        x = x - x.mean(axis=1, keepdims=True)
        return (x / np.sqrt((x * x).mean(axis=1, keepdims=True) + f(1e-5)) * g + b).astype(f)

    for b in m.blocks:
        h = norm(x, b.ln1_g, b.ln1_b)
        q, k, v = (h @ w.reshape(d, d).astype(f) + bias for w, bias in ((b.wq, b.bq), (b.wk, b.bk), (b.wv, b.bv)))
        out = np.empty((n, d), dtype=f)
        for e in range(0, d, hd):
            s = q[:, e:e + hd] @ k[:, e:e + hd].T / f(np.sqrt(hd))
            s = np.where(np.tril(np.ones((n, n), dtype=bool)), s, -np.inf)
            p = np.exp(s - s.max(axis=1, keepdims=True))
            out[:, e:e + hd] = p / p.sum(axis=1, keepdims=True) @ v[:, e:e + hd]
        x = x + out @ b.wo.reshape(d, d).astype(f) + b.bo
        h = norm(x, b.ln2_g, b.ln2_b) @ b.w1.reshape(d, c.hidden).astype(f) + b.b1
        h = f(0.5) * h * (1 + np.tanh(f(np.float32(0.7978846)) * (h + f(np.float32(0.044715)) * h * h * h)))
        x = x + h @ b.w2.reshape(c.hidden, d).astype(f) + b.b2
    return norm(x, m.lnf_g, m.lnf_b) @ m.head.reshape(d, c.vocab).astype(f)


def models(kind):
    base = dict(ctx=352, head_dim=64, layers=2)
    odd = 384 if kind == QKind.Q8_0 else 512  # (Q4_0: whole 256s)
    return {
        "group2": (LlamaConfig(vocab=1000, dim=256, heads=4, kv_heads=2, hidden=odd, rope_dim=64, **base), False),
        "group3": (LlamaConfig(vocab=9600, dim=odd, heads=12, kv_heads=4, hidden=512, rope_dim=64, rope_type=_ffi.FC_ROPE_NEOX, **base), True),
        # rows of several ring slots, a rotation of half the channels
        "group8_wide": (LlamaConfig(vocab=600, dim=1280, heads=8, kv_heads=1, hidden=2304, rope_dim=32, rope_type=_ffi.FC_ROPE_NEOX,
                                    **base), True),
        "gpt2": (Gpt2Config(vocab=300, ctx=352, dim=768, heads=12, layers=2, hidden=3072), True),
    }


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("name", ["group2", "group3", "group8_wide", "gpt2"])
def test_one_kernel_steps_match_exact_arithmetic_at_every_width(dev, name, kind):
    cfg, biased = models(kind)[name]
    ids = random_tokens(3, max(LENGTHS), cfg.vocab)
    if name == "gpt2":
        m = random_gpt2(cfg, seed=5, std=0.05, bias_std=0.05, gain_jitter=0.1)
        ref, forward = orc.dequantised_gpt2(m, int(kind), snap_embedding=False), np_gpt2_forward
        g = CudaGpt2(dev, m, kind, max_streams=64)
    else:
        m = random_llama(cfg, seed=5, biases=biased, std=0.05, gain_jitter=0.1)
        ref, forward = orc.dequantised_llama(m, int(kind), snap_embedding=False), helpers.np_llama_forward
        g = CudaLlama(dev, m, kind, max_streams=64)
    want = forward(ref, ids, np.float64)
    tol = bounds(want, forward(ref, ids, np.float32))
    for streams in (1, 2, 3, 5, 8, 9, 20, 64):
        for first in ((0, 1, 2, 3, 6) if streams == 1 else (0,)):
            lengths = (LENGTHS * 8)[first:first + streams]
            slots = list(range(streams))[::-1]  # (row i is not stream i)
            for n, s in zip(lengths, slots):
                g.reset(s)
                if n > 1:
                    g.prefill(ids[:n - 1], stream=s)
            before = dev.launch_count()
            picks, rows = g.feed_batch([int(ids[n - 1]) for n in lengths], streams=slots, want_logits=True)
            # (many rows of wide matrices go as launches, which have to fit in with what this kernel leaves behind and finds)
            assert dev.launch_count() - before == 1 or streams == 64
            for n, row, pick in zip(lengths, rows, picks):
                assert orc.max_rel_err(row, want[n - 1]) < tol[n - 1], (streams, n)
                assert pick == orc.argmax(row)
            # the cache the step left behind serves the next one, and a chain of steps is those steps
            fed = [g.feed_batch(picks, streams=slots)[0]]
            for n, s in zip(lengths, slots):
                g.reset(s)
                g.prefill(ids[:n], stream=s)
            chain = g.decode_greedy(picks, 4, streams=slots)
            assert np.array_equal(chain[0], fed[0])
            for n, s in zip(lengths, slots):
                g.reset(s)
                g.prefill(ids[:n], stream=s)
            tok = picks
            for step in range(4):
                tok, _ = g.feed_batch(tok, streams=slots)
                assert np.array_equal(tok, chain[step]), (streams, step)
    g.close()


def test_a_step_reports_a_wait_that_gave_up_and_the_next_one_works(dev):
    """A status raised by an earlier kernel ends every wait of the step at once: it returns an error, the position stays, and
    the step after it is as if nothing had been."""
    cfg, _ = models(QKind.Q8_0)["group2"]
    m = random_llama(cfg, seed=7, std=0.05)
    g = CudaLlama(dev, m, QKind.Q8_0)
    want = g.feed(3)
    g.reset()
    _ffi.load().fc_debug_raise_status(dev.handle, 1)
    with pytest.raises(Exception, match="gave up"):
        g.feed(3)
    assert g.pos() == 0
    assert np.array_equal(g.feed(3), want)
    g.close()


@pytest.mark.parametrize("streams", [1, 3])
def test_a_chain_over_two_launches_is_the_chain_in_pieces(dev, streams):
    """A chain runs in the kernel for up to 256 steps; 300 of them against pieces of 1, 100 and 199, from other launches."""
    cfg, _ = models(QKind.Q8_0)["group2"]
    m = random_llama(cfg, seed=9, std=0.2)
    g = CudaLlama(dev, m, QKind.Q8_0, max_streams=streams)
    first = random_tokens(1, streams, cfg.vocab)
    before = dev.launch_count()
    whole = g.decode_greedy(first, 300)
    assert dev.launch_count() - before == 3
    for s in range(streams):
        g.reset(s)
    tok, parts = first, []
    for n in (1, 100, 199):
        parts.append(g.decode_greedy(tok, n))
        tok = parts[-1][-1]
    assert np.array_equal(np.concatenate(parts), whole)
    assert all(g.pos(s) == 300 for s in range(streams))
    g.close()
