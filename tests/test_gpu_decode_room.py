"""The one-kernel decode's own buffers (csrc/decode_grid.cu), which lie outside the model's plan, when the device has no room left."""
import numpy as np
import pytest

from ferrum_gpu_b200 import CudaLlama, QKind, upload_quantised
from ferrum_gpu_b200 import _ffi
from ferrum_gpu_b200.hostmodel import LlamaConfig, random_llama, random_tokens

pytestmark = pytest.mark.gpu

# 64 streams of these widths have 13 MB of tagged words
CFG = LlamaConfig(vocab=64, ctx=512, dim=3072, heads=48, kv_heads=48, head_dim=64, layers=1, hidden=3072, rope_dim=64)
LEFT = 8 << 20


def launches_of_a_step(dev, g):
    before = dev.launch_count()
    g.feed(3)
    return dev.launch_count() - before


def fill_the_device():
    import torch
    torch.cuda.empty_cache()
    hogs = [torch.empty(torch.cuda.mem_get_info()[0] - LEFT, dtype=torch.uint8, device="cuda")]
    assert torch.cuda.mem_get_info()[0] <= LEFT
    return hogs


def test_the_set_up_takes_what_the_scratch_pool_holds(dev):
    import torch
    lib = _ffi.load()
    g = CudaLlama(dev, random_llama(CFG, seed=1, std=0.02), QKind.Q8_0, max_streams=64)
    m, k, n = 6000, 8192, 1024
    qw = upload_quantised(dev, QKind.Q8_0, np.zeros(k * n, dtype=np.float32), k, n)
    x, y = torch.randn(m, k, device="cuda"), torch.empty(m, n, device="cuda")
    torch.cuda.synchronize()
    dev.check(lib.fc_qmatmul_dev(qw.handle, x.data_ptr(), m, y.data_ptr(), 0))  # (leaves 197 MB of terms in the pool)
    dev.sync()
    qw.close()
    del x, y
    hogs = fill_the_device()
    try:
        assert launches_of_a_step(dev, g) == 1
    finally:
        del hogs
        torch.cuda.empty_cache()
        g.close()


def test_without_room_steps_are_launches_until_there_is_some(dev):
    import torch
    # the launches' kernels are on the device before it is full: the same with an input wider than the one kernel takes
    wide = LlamaConfig(vocab=64, ctx=64, dim=3328, heads=48, kv_heads=48, head_dim=64, layers=1, hidden=3328, rope_dim=64)
    warm = CudaLlama(dev, random_llama(wide, seed=1, std=0.02), QKind.Q8_0, max_streams=64)
    for _ in range(4):
        assert launches_of_a_step(dev, warm) > 1
    warm.close()
    m = random_llama(CFG, seed=2, std=0.02)
    g = CudaLlama(dev, m, QKind.Q8_0, max_streams=64)
    ref = CudaLlama(dev, m, QKind.Q8_0, max_streams=64)
    ids = random_tokens(4, 4, CFG.vocab)
    want = [ref.feed(int(t)) for t in ids]
    ref.close()
    dev.check(_ffi.load().fc_device_sync(dev.handle))
    hogs = fill_the_device()
    try:
        free = torch.cuda.mem_get_info()[0]
        for t, w in zip(ids, want):
            before = dev.launch_count()
            got = g.feed(int(t))
            assert dev.launch_count() - before > 1
            assert np.abs(got - w).max() <= 1e-5 * max(1.0, np.abs(w).max())
        assert free - torch.cuda.mem_get_info()[0] < 4 << 20  # (a graph of the launches; nothing of the kernel that does not run)
    finally:
        del hogs
        torch.cuda.empty_cache()
    assert 1 in [launches_of_a_step(dev, g) for _ in range(100)]
    assert launches_of_a_step(dev, g) == 1
    g.close()
