"""The small GPT-2-style configuration (6 layers, 384 wide) decoded by one stream, by the kernel that its format has: Q8_0 by the
persistent kernel over all SMs (csrc/decode_grid.cu), Q4_0, whose packed rows of 384 are not whole 128-byte lines, by the
thread-block cluster (csrc/decode_cluster.cu)."""
import pytest

from ferrum_gpu_b200 import CudaGpt2, QKind
from ferrum_gpu_b200.hostmodel import config_c1, random_gpt2, random_tokens
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, kernel", [(QKind.Q8_0, "decode_grid"), (QKind.Q4_0, "decode_cluster")])
def test_the_small_configuration_matches_the_oracle_on_either_kernel(dev, kind, kernel):
    cfg = config_c1()
    m = random_gpt2(cfg, seed=11)
    ref = orc.dequantised_gpt2(m, int(kind), snap_embedding=False)
    oracle = orc.OracleGpt2(ref)
    g = CudaGpt2(dev, m, kind)
    dev.profile(True)
    try:
        for t in random_tokens(4, 16, cfg.vocab).tolist():
            lo = oracle.feed(t)
            assert orc.max_rel_err(g.feed(t), lo) < 1e-5
        names = dev.profile_report()
        assert set(names) == {kernel}, names
    finally:
        dev.profile(False)
    want = []
    tok = first = orc.argmax(lo)
    for _ in range(100):
        lo = oracle.feed(tok)
        tok = orc.argmax(lo)
        want.append(tok)
    before = dev.launch_count()
    assert g.decode_greedy([first], 100)[:, 0].tolist() == want
    assert dev.launch_count() - before == 2
    assert orc.max_rel_err(g.feed(tok), oracle.feed(tok)) < 1e-5
    g.close()
