"""The workspace of the exact products of many rows: a pass reserves it once, for its largest run of rows, and shorter
runs have to stay inside. Pure arithmetic of the built library, no device."""
import pytest

from ferrum_gpu_b200 import _ffi

NO_LIMIT = 2**64 - 1
SMS = 148
# (dim, q + 2 kv width, hidden, vocab)
WIDTHS = [(128, 256, 768, 1000), (768, 1280, 2048, 32000), (1024, 1280, 2816, 151936), (2048, 3072, 8192, 128256), (2048, 6144, 8192, 49152),
          (1536, 2048, 8960, 151936), (4096, 12288, 11008, 32000), (768, 2304, 3072, 50257)]


@pytest.fixture(scope="module")
def pair():
    lib = _ffi.load()
    return lambda k, n, m, limit=NO_LIMIT, sms=SMS, gelu=0: lib.fc_debug_pair_bytes(sms, k, n, m, gelu, limit)


def _matrices(d, qkv, hid, vocab):
    return [(d, qkv), (d, d), (d, 2 * hid), (hid, d), (d, vocab)]


def test_fewer_rows_may_ask_for_more(pair):
    """Why a row count is no measure of a workspace: 1413 rows are cut into more splits of K than 1884."""
    assert pair(8192, 2048, 1413) > pair(8192, 2048, 1884)


@pytest.mark.parametrize("widths", WIDTHS)
def test_no_run_of_rows_leaves_what_a_pass_reserved(pair, widths):
    mats = _matrices(*widths)
    for most in list(range(65, 3000, 97)) + [660, 1884, 2656, 5544, 11560, 20000]:
        reserved = max(pair(k, n, most) for k, n in mats)
        for rows in {65, most // 7, most // 3, most // 2, 3 * most // 4, most - most // 10, most - 1}:
            if rows <= 64:
                continue
            for k, n in mats:
                need = pair(k, n, rows, reserved)
                assert 0 < need <= reserved, (widths, most, rows, k, n)


def test_sums_are_reserved_where_they_are_written(pair):
    """One split of K and no activation: the result goes straight to y, and the workspace is the terms and scales."""
    k, n, m = 4096, 11008, 4096
    terms, kib = 2 * m * k * 2 + 2 * 4096 * k * 2, 1024  # x, and 64 MB of weight rows at once
    assert terms < pair(k, n, m) < terms + 64 * kib
    assert pair(k, n, m, gelu=1) >= terms + m * 4096 * 4


@pytest.mark.parametrize("sms", [148, 132, 60, 2])
def test_a_cut_fits_its_limit_or_there_is_none(pair, sms):
    k, n, m = 8192, 2048, 300
    best = pair(k, n, m, sms=sms)
    lo, hi = 0, best  # the smallest workspace with which some cut works
    while lo + 1 < hi:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if pair(k, n, m, mid, sms) else (mid, hi)
    assert pair(k, n, m, hi, sms) == hi and pair(k, n, m, 0, sms) == 0
    for limit in range(hi, best + (1 << 20), 1 << 19):
        assert hi <= pair(k, n, m, limit, sms) <= limit
    assert pair(k, n, m, best, sms) == best
    assert sms != 148 or hi < best, "a smaller workspace means fewer splits"
