"""Steps of the one-kernel decode (csrc/decode_grid.cu) whose waits give up: the status word is up before the step starts, so every
wait ends at once and whatever it waited for (plans, ring slots, tokens) is not there. The step reports it, touches nothing
outside its buffers, and the next one is as if nothing had been. No kernel has to time out for it."""
import numpy as np
import pytest

from ferrum_gpu_b200 import CudaGpt2, CudaLlama, QKind
from ferrum_gpu_b200 import _ffi
from ferrum_gpu_b200.hostmodel import Gpt2Config, LlamaConfig, random_gpt2, random_llama, random_tokens

pytestmark = pytest.mark.gpu

MODELS = {
    # slots of several sizes, rows of several slots; heads in groups; every row's positions in several parts
    "wide": LlamaConfig(vocab=600, ctx=352, dim=1280, heads=8, kv_heads=1, head_dim=64, layers=2, hidden=2304, rope_dim=64),
    "gpt2": Gpt2Config(vocab=300, ctx=352, dim=768, heads=12, layers=2, hidden=3072),
    # few tiles, many attention items
    "heads": LlamaConfig(vocab=16, ctx=352, dim=256, heads=48, kv_heads=48, head_dim=64, layers=1, hidden=256, rope_dim=64),
}


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_steps_that_give_up_report_it_and_leave_the_model_as_it_was(dev, name, kind):
    cfg = MODELS[name]
    gpt2 = isinstance(cfg, Gpt2Config)
    m = random_gpt2(cfg, seed=5, std=0.05) if gpt2 else random_llama(cfg, seed=5, std=0.05)
    g = (CudaGpt2 if gpt2 else CudaLlama)(dev, m, kind, max_streams=20)
    prompt = random_tokens(3, 300, cfg.vocab)
    lib = _ffi.load()
    for streams in (1, 2, 4, 8, 20):
        slots = list(range(streams))
        for s in slots:
            g.reset(s)
            g.prefill(prompt[:300 - s], stream=s)
        first = random_tokens(7, streams, cfg.vocab)
        before = dev.launch_count()
        g.feed_batch(first, streams=slots)
        if dev.launch_count() - before > 1:
            assert streams == 20  # (decided by an estimate: as launches, which do not look at the word)
            continue
        for s in slots:
            g.reset(s)
            g.prefill(prompt[:300 - s], stream=s)
        for call in (lambda: g.feed_batch(first, streams=slots), lambda: g.decode_greedy(first, 1, streams=slots)):
            lib.fc_debug_raise_status(dev.handle, 1)
            before = dev.launch_count()
            try:
                with pytest.raises(Exception, match="gave up"):
                    call()
                assert dev.launch_count() - before == 1
            finally:
                dev.check(lib.fc_debug_raise_status(dev.handle, 0))
            assert [g.pos(s) for s in slots] == [300 - s for s in slots]
        got = g.decode_greedy(first, 6, streams=slots)
        _, after = g.feed_batch(got[-1], streams=slots, want_logits=True)
        for s in slots:
            g.reset(s)
            g.prefill(prompt[:300 - s], stream=s)
        assert np.array_equal(g.decode_greedy(first, 6, streams=slots), got)
        assert np.array_equal(g.feed_batch(got[-1], streams=slots, want_logits=True)[1], after)
    g.close()
