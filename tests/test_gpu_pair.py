"""The products of many rows on CTA pairs and the decode products at widths that are not whole 128s, at the sizes where
they can go wrong: tile edges, K tails, one column, splits of K; and the tiled exact attention. References are float64.

Bounds of the exact class: the two fp16 terms leave 2^-22 of each factor and the dropped cross term 2^-22 of the
product, f32 sums of 128 k (rounded toward zero, one unit of 2^-23 per 16 k) are added in f32: below 16 x 2^-23 = 2e-6
of sum |x w| whatever the width."""
import numpy as np
import pytest

from ferrum_gpu_b200 import CudaGpt2, CudaLlama, Mode, QKind, _ffi, linear_q, upload_quantised, upload_qweight
from ferrum_gpu_b200.hostmodel import Gpt2Config, LlamaConfig, random_gpt2, random_llama, random_tokens
from oracle import oracle as orc
from tests import helpers

pytestmark = pytest.mark.gpu

EXACT = 2e-6  # of sum |x w|


def _problem(dev, kind, m, k, n, seed=1, mag=1.0):
    rng = np.random.default_rng(seed)
    qw = upload_quantised(dev, kind, (rng.standard_normal(k * n) * 0.02).astype(np.float32), k, n)
    x = (rng.standard_normal((m, k)) * mag).astype(np.float32)
    w = qw.dequantised().reshape(n, k).astype(np.float64)
    return qw, x, x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("m,k,n", [(65, 32, 1), (65, 64, 255), (127, 96, 256), (128, 4096, 257), (129, 160, 40), (192, 800, 1000),
                                   (300, 2080, 513), (70, 1024, 9000), (1500, 128, 300), (600, 96, 3000), (300, 32, 20000)])
@pytest.mark.parametrize("mag", [1.0, 1e-30, 1e30])
def test_exact_products_of_many_rows(dev, kind, m, k, n, mag):
    qw, x, want, scale = _problem(dev, kind, m, k, n, mag=mag)
    got = linear_q(dev, x, qw, m).reshape(m, n)
    assert np.all(np.abs(got - want) <= EXACT * scale), (kind, m, k, n, np.max(np.abs(got - want) / scale))
    assert np.array_equal(got, linear_q(dev, x, qw, m).reshape(m, n)), "repeated runs are bit-identical"
    qw.close()


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("m,k", [(100, 256), (80, 2048)])
def test_rows_with_infinities_and_nans_and_zero_rows(dev, kind, m, k):
    n = 300
    qw, x, _, _ = _problem(dev, kind, m, k, n)
    clean = linear_q(dev, x, qw, m).reshape(m, n)
    x[3, 5], x[7, k - 1], x[11, 0], x[20], x[30, 1] = np.inf, -np.inf, np.nan, 0.0, 3e38
    w = qw.dequantised().reshape(n, k).astype(np.float64)
    got = linear_q(dev, x, qw, m).reshape(m, n)
    bad = [3, 7, 11]
    with np.errstate(invalid="ignore", over="ignore"):
        want = (x.astype(np.float64)[bad][:, None, :] * w[None]).sum(-1)
    for i, r in enumerate(bad):
        assert np.array_equal(np.isnan(got[r]), np.isnan(want[i])) and np.array_equal(got[r][~np.isnan(want[i])], want[i][~np.isnan(want[i])])
    assert np.all(got[20] == 0)
    # 3e38 among values about 1: an f32 chain rounds k times at most; where its weight is zero the others count in full
    big = x[30].astype(np.float64)
    assert np.all(np.abs(got[30] - big @ w.T) <= k * 2.0 ** -24 * (np.abs(big) @ np.abs(w).T)) and np.any(w[:, 1] == 0)
    others = [r for r in range(m) if r not in bad + [20, 30]]
    assert np.array_equal(got[others], clean[others]), "other rows do not change"
    qw.close()


def _spread_rows(spread, m, k):
    """Rows whose magnitudes are far apart."""
    rng = np.random.default_rng(9)
    x = rng.standard_normal((m, k))
    if spread == "ramp":
        x *= 2.0 ** (-60 * np.arange(k) / k)
    elif spread == "lognormal":
        x *= np.exp(4 * rng.standard_normal((m, k)))
    elif spread == "one small":
        x[:, 3] *= 2.0 ** -45
    else:  # two large elements, whose weights are zero in half of the outputs
        x[:, 7], x[:, k - 2] = 2.0 ** spread, -2.0 ** (spread - 1)
    return x.astype(np.float32)


def _spread_check(dev, kind, m, k, n, spread):
    w = np.random.default_rng(4).standard_normal((k, n)).astype(np.float32) * 0.02
    w[7, ::2] = w[k - 2, ::2] = 0.0
    qw = upload_quantised(dev, kind, w.reshape(-1), k, n)
    w = qw.dequantised().reshape(n, k).astype(np.float64)
    x = _spread_rows(spread, m, k)
    want, scale = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    got = linear_q(dev, x, qw, m).reshape(m, n)
    # the terms hold elements down to 2^-28 of the largest; beyond, the f32 chain: k roundings at most
    bound = k * 2.0 ** -24 if not isinstance(spread, str) and spread > 26 else EXACT
    assert np.all(np.abs(got - want) <= bound * scale), (kind, m, k, n, spread, np.max(np.abs(got - want) / scale))
    qw.close()


SPREADS = [8, 20, 26, 34, 60, 127, "ramp", "lognormal", "one small"]


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("m,k,n", [(100, 512, 300), (300, 96, 3000), (200, 2080, 513)])
@pytest.mark.parametrize("spread", SPREADS)
def test_exact_products_of_many_rows_keep_small_elements_beside_large_ones(dev, kind, m, k, n, spread):
    _spread_check(dev, kind, m, k, n, spread)


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0, QKind.F16, QKind.FP8_E4M3, QKind.MXFP4])
@pytest.mark.parametrize("m,k,n", [(2, 160, 5), (3, 224, 64), (8, 4064, 130), (5, 1056, 3000), (9, 160, 70), (16, 288, 65), (33, 2080, 300),
                                   (64, 1120, 1000), (40, 4064, 20)])
@pytest.mark.parametrize("mag", [1.0, 1e-20, 1e20, 1e-35, 1e36])
def test_decode_products_at_ragged_widths(dev, kind, m, k, n, mag):
    qw, x, want, scale = _problem(dev, kind, m, k, n, mag=mag)
    got = linear_q(dev, x, qw, m).reshape(m, n)
    # (at 1e-35 block sums come near the smallest normal number: 2^-149 for each of their roundings and splits)
    assert np.all(np.abs(got - want) <= EXACT * scale + (k // 32 + 16) * 2.0 ** -149), (kind, m, k, n, np.max(np.abs(got - want) / scale))
    qw.close()


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0, QKind.F16, QKind.FP8_E4M3, QKind.MXFP4])
@pytest.mark.parametrize("m,k,n", [(2, 160, 70), (5, 1056, 3000), (8, 4064, 130), (9, 160, 70), (40, 1056, 300), (64, 2080, 1000)])
@pytest.mark.parametrize("spread", SPREADS)
def test_decode_products_at_ragged_widths_keep_small_elements_beside_large_ones(dev, kind, m, k, n, spread):
    _spread_check(dev, kind, m, k, n, spread)


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("m,k,n", [(5, 160, 70), (7, 4064, 600), (12, 160, 70), (50, 2080, 300), (100, 2080, 300)])
def test_infinities_and_nans_go_where_an_f32_chain_puts_them(dev, kind, m, k, n):
    rng = np.random.default_rng(2)
    clean = upload_quantised(dev, kind, (rng.standard_normal(k * n) * 0.02).astype(np.float32), k, n)
    raw = clean.blocks().reshape(n, k // 32, -1)
    raw[3, 1, :2] = np.array([np.inf], dtype=np.float16).view(np.uint8)
    raw[5, 2, :2] = np.array([np.nan], dtype=np.float16).view(np.uint8)
    clean.close()
    qw = upload_qweight(dev, kind, raw.reshape(-1), k, n)
    w = qw.dequantised().reshape(n, k).astype(np.float64)
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[0, 5], x[1, k - 1], x[2, 40] = np.inf, np.nan, -np.inf
    x[3] = 0.0
    got = linear_q(dev, x, qw, m).reshape(m, n)
    with np.errstate(invalid="ignore"):
        want = np.stack([(row.astype(np.float64)[None] * w).sum(-1) for row in x])
        scale = np.abs(x).astype(np.float64) @ np.nan_to_num(np.abs(w), posinf=0.0).T
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert inf.any() and np.array_equal(got[inf], want[inf])
    ok = np.isfinite(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= EXACT * scale[ok])
    qw.close()


@pytest.mark.parametrize("kind", [QKind.Q8_0, QKind.Q4_0])
@pytest.mark.parametrize("m,k,n", [(1024, 64, 256), (1025, 192, 257), (1300, 768, 1000), (2049, 128, 8)])
def test_tensor_products_of_many_rows(dev, kind, m, k, n):
    """fp16 operands, one rounding each (2^-11), products exact, f32 sums: 2^-10 of sum |x w| bounds them."""
    qw, x, want, scale = _problem(dev, kind, m, k, n)
    got = linear_q(dev, x, qw, m, Mode.TENSOR_F16).reshape(m, n)
    assert np.all(np.abs(got - want) <= 2.0 ** -10 * scale), (kind, m, k, n, np.max(np.abs(got - want) / scale))
    # the rows that a smaller call has too: the same operands through the kernel that decodes the weights itself
    few = linear_q(dev, x[:200], qw, 200, Mode.TENSOR_F16).reshape(200, n)
    assert np.all(np.abs(got[:200] - few) <= 1e-5 * scale[:200] + 1e-30)
    qw.close()


@pytest.mark.parametrize("arch", ["llama", "gpt2"])
@pytest.mark.parametrize("t", [31, 32, 64, 65, 130, 200])
def test_exact_prefill_and_scoring_match_the_oracle(dev, arch, t):
    if arch == "llama":
        cfg = LlamaConfig(vocab=300, ctx=256, dim=128, heads=4, kv_heads=2, head_dim=64, layers=2, hidden=160, rope_dim=64)
        m = random_llama(cfg, seed=3, std=0.05)
        oracle = orc.OracleLlama(orc.dequantised_llama(m, int(QKind.Q8_0), snap_embedding=False), threads=4)
        g = CudaLlama(dev, m, QKind.Q8_0)
    else:
        cfg = Gpt2Config(vocab=300, ctx=256, dim=128, heads=2, layers=2, hidden=160)
        m = random_gpt2(cfg, seed=3, std=0.05)
        oracle = orc.OracleGpt2(orc.dequantised_gpt2(m, int(QKind.Q8_0), snap_embedding=False), threads=4)
        g = CudaGpt2(dev, m, QKind.Q8_0)
    ids = random_tokens(t, t, cfg.vocab)
    whole = g.prefill(ids)
    g.reset(0)
    head = max(1, t - 40)
    g.prefill(ids[:head])
    assert orc.max_rel_err(g.prefill(ids[head:]), whole) < 2e-5, "a prompt in two passes"
    lp, _, _ = g.score_batch(np.stack([ids, ids[::-1]]), Mode.EXACT_F32)
    for s, seq in enumerate([ids, np.ascontiguousarray(ids[::-1])]):
        want, _ = oracle.score(seq)
        assert np.max(np.abs(lp[s] - want)) < 5e-5
    g.close()


@pytest.mark.parametrize("poison", [np.inf, np.nan])
def test_a_later_row_with_infinities_does_not_reach_earlier_rows(dev, poison):
    """Causality at the bit level: a token whose embedding overflows changes nothing before its position, also inside the
    same tile of the tiled attention."""
    cfg = LlamaConfig(vocab=64, ctx=128, dim=128, heads=2, kv_heads=1, head_dim=64, layers=1, hidden=128, rope_dim=64)
    m = random_llama(cfg, seed=7, std=0.05)
    tok = np.asarray(m.tok, dtype=np.float32).reshape(cfg.vocab, cfg.dim).copy()
    tok[63, 0] = poison
    m.tok = tok.reshape(np.asarray(m.tok).shape)
    g = CudaLlama(dev, m, QKind.Q8_0)
    ids = (np.arange(100) % 60).astype(np.int32)
    clean = g.forward_all(ids)
    ids[70] = 63
    got = g.forward_all(ids)
    assert np.array_equal(got[:70], clean[:70]) and np.all(np.isnan(got[70]))
    g.close()


def test_exact_scoring_in_unequal_passes(dev):
    """A call in two passes whose shorter one would, cut for itself, take more workspace than the longer one reserved."""
    lib = _ffi.load()
    cfg = LlamaConfig(vocab=1000, ctx=64, dim=128, heads=2, kv_heads=1, head_dim=64, layers=2, hidden=768, rope_dim=64)
    if dev.props()[0] == 148:  # (`down` is the only matrix here that is not left to the tiled kernel)
        need = [lib.fc_debug_pair_bytes(148, 768, 128, seqs * 60, 0, 2**64 - 1) for seqs in (11, 10)]
        assert need[0] < need[1]
    g = CudaLlama(dev, random_llama(cfg, seed=3, std=0.05), QKind.Q8_0)
    ids = np.stack([random_tokens(i, 61, cfg.vocab) for i in range(21)])
    whole = g.score_batch(ids, Mode.EXACT_F32)
    dev.check(lib.fc_debug_score_pass_bytes(g._h, 15 << 20))  # 16 KB a row: 21 x 60 rows are passes of 11 and 10 sequences
    parts = g.score_batch(ids, Mode.EXACT_F32)
    assert np.max(np.abs(parts[0] - whole[0])) < 2e-5 and np.mean(parts[1] != whole[1]) < 0.002
    again = g.score_batch(ids, Mode.EXACT_F32)
    assert np.array_equal(again[0], parts[0])
    g.close()


@pytest.mark.parametrize("eager_rows", [0, 100, 3000])
@pytest.mark.parametrize("mode,m,k", [(Mode.EXACT_F32, 2000, 512), (Mode.EXACT_F32, 40, 512), (Mode.EXACT_F32, 5, 480), (Mode.TENSOR_F16, 2000, 512)])
def test_products_captured_into_a_graph(dev, mode, m, k, eager_rows):
    """A captured call works in memory of its own, whatever earlier calls of the same weight had, and replays read the
    operands of the moment while eager work of this and other weights goes on between them."""
    import torch
    lib = _ffi.load()
    n = 1024
    rng = np.random.default_rng(5)
    qw = upload_quantised(dev, QKind.Q8_0, (rng.standard_normal(k * n) * 0.02).astype(np.float32), k, n)
    w = torch.from_numpy(qw.dequantised().reshape(n, k)).cuda().double()
    x, y = torch.randn(max(m, eager_rows), k, device="cuda"), torch.zeros(max(m, eager_rows), n, device="cuda")
    call = lambda rows: dev.check(lib.fc_qmatmul_dev(qw.handle, x.data_ptr(), rows, y.data_ptr(), int(mode)))
    call(70)  # (the kernels' one-time settings)
    if eager_rows:
        call(eager_rows)
    dev.sync()
    other = upload_quantised(dev, QKind.Q8_0, (rng.standard_normal(k * n) * 0.02).astype(np.float32), k, n)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(dev.stream())):
        call(m)
    bound = EXACT if mode == Mode.EXACT_F32 else 2.0 ** -10
    for seed in range(2):
        x.copy_(torch.randn(x.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)))
        torch.cuda.synchronize()
        dev.check(lib.fc_qmatmul_dev(other.handle, x.data_ptr(), m, y.data_ptr(), int(mode)))
        call(m)
        dev.sync()
        y.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        dev.sync()
        xd = x[:m].double()
        assert bool(((y[:m].double() - xd @ w.T).abs() <= bound * (xd.abs() @ w.abs().T)).all())
        assert not bool(y[m:].any())
    del graph
    qw.close()
    other.close()


@pytest.mark.parametrize("mode", [Mode.EXACT_F32, Mode.TENSOR_F16])
def test_weights_share_their_scratch(dev, mode):
    """Products of many weights leave no workspace behind with each."""
    import torch
    lib = _ffi.load()
    m, k, n = 1500, 2048, 4096
    w = (np.random.default_rng(1).standard_normal(k * n) * 0.02).astype(np.float32)
    weights = [upload_quantised(dev, QKind.Q8_0, w, k, n) for _ in range(24)]
    x, y = torch.randn(m, k, device="cuda"), torch.empty(m, n, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    want = None
    for qw in weights:
        dev.check(lib.fc_qmatmul_dev(qw.handle, x.data_ptr(), m, y.data_ptr(), int(mode)))
        dev.sync()
        want = y.clone() if want is None else want
        assert torch.equal(y, want)
    assert free - torch.cuda.mem_get_info()[0] < 256 << 20  # one workspace is 28..46 MB
    for qw in weights:
        qw.close()


def test_cached_scratch_makes_room_for_weights(dev):
    """What products left in the device handle's pool goes back when a weight finds no room beside it."""
    import torch
    lib = _ffi.load()
    m, k, n = 6000, 8192, 1024
    zeros = np.zeros(k * n, dtype=np.float32)
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    qw = upload_quantised(dev, QKind.Q8_0, zeros, k, n)
    x, y = torch.randn(m, k, device="cuda"), torch.empty(m, n, device="cuda")
    torch.cuda.synchronize()
    dev.check(lib.fc_qmatmul_dev(qw.handle, x.data_ptr(), m, y.data_ptr(), 0))
    dev.sync()
    qw.close()
    del x, y
    torch.cuda.empty_cache()
    cached = before - torch.cuda.mem_get_info()[0]
    assert cached > 128 << 20, "the pool holds on to the workspace (197 MB of terms)"
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 80 << 20
        big = upload_quantised(dev, QKind.Q8_0, np.zeros(4096 * 4096, dtype=np.float32), 4096, 4096)  # 18 MB and 67 of staging
        big.close()
    finally:
        del hog
        torch.cuda.empty_cache()


def test_hidden_states_at_any_float_address(dev):
    """The exact head takes hidden states where they lie, also rows that its fp16 terms do not hold."""
    import torch
    cfg = LlamaConfig(vocab=1000, ctx=64, dim=256, heads=4, kv_heads=2, head_dim=64, layers=1, hidden=256, rope_dim=64)
    g = CudaLlama(dev, random_llama(cfg, seed=3, std=0.05), QKind.Q8_0)
    rows = 200
    h = torch.randn(rows, cfg.dim, device="cuda")
    h[7, 3], h[9, 0], h[11] = 1e30, float("inf"), h[11] * 2.0 ** (-60 * torch.arange(cfg.dim, device="cuda") / cfg.dim)
    moved = torch.empty(rows * cfg.dim + 1, device="cuda")
    moved[1:] = h.reshape(-1)
    targets = torch.arange(rows, device="cuda", dtype=torch.int32)
    out = torch.zeros(2, rows, 4, device="cuda")
    torch.cuda.synchronize()
    g.head_partial_dev(h.data_ptr(), targets.data_ptr(), rows, Mode.EXACT_F32, out[0].data_ptr())
    g.head_partial_dev(moved.data_ptr() + 4, targets.data_ptr(), rows, Mode.EXACT_F32, out[1].data_ptr())
    dev.sync()
    a, b = out.cpu().numpy()
    assert np.array_equal(a, b, equal_nan=True) and np.all(np.isfinite(np.delete(a, 9, axis=0)))
    g.close()
