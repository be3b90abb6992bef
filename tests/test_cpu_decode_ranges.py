"""How the decode attention hands out ranges of long contexts, on the CPU: the arithmetic that the kernel runs."""
import ctypes

import pytest

SMS = 148


def ranges(lens, n_kv, splits, window=0, chunk=0, keep_first=0):
    from llm_b200.csrc import ops
    given, got = (ctypes.c_int * len(lens))(*lens), (ctypes.c_int * len(lens))()
    total = ops.load_tensor().llmk_decode_attention_ranges(given, len(lens), n_kv, window, chunk, keep_first, splits, SMS, got)
    assert total == sum(got) * n_kv
    return list(got)


def places(lens, n_kv, longest=0):
    from llm_b200.csrc import ops
    return ops.decode_places(len(lens), n_kv, longest or max(lens), SMS)


@pytest.mark.parametrize("n_kv", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("entries", [1, 3, 8, 10, 20, 36])
@pytest.mark.parametrize("keys", [2049, 3000, 8000, 8192, 32768])
def test_equal_requests_run_in_one_wave(entries, keys, n_kv):
    """About as many ranges each as two CTAs an SM hold at once (lengths are tried in steps of 2 % or of half a tile), and never more."""
    from llm_b200.csrc import ops
    lens = [keys] * entries
    got = ranges(lens, n_kv, places(lens, n_kv))
    fair = ops.decode_splits(entries, n_kv, keys, SMS)
    assert len(set(got)) == 1
    if entries * n_kv <= 2 * SMS:
        assert entries * n_kv * got[0] <= 2 * SMS
    assert 1.08 * got[0] >= min(fair, keys // 256)


def test_a_long_request_among_short_ones_gets_more():
    assert ranges([6000] + [400] * 7, 8, 16) == [16] + [2] * 7
    got = ranges([20000] + [500] * 31, 8, 4)
    assert got[0] == 4 and set(got[1:]) == {1}
    # many short requests free their places soon: the long one is cut as finely as its share of the keys asks for
    got = ranges([20000] + [100] * 36, 8, 64)
    assert got[0] >= 20 and set(got[1:]) == {1}
    # entries without keys, or of a negative length, have a place in which zeros are written
    got = ranges([0, 8192, -5, 8192], 8, 64)
    assert got[0] == got[2] == 1 and got[1] == got[3] in (17, 18)


def test_only_the_keys_that_are_seen_count():
    """A chunk's, a window's and the kept first ones: lengths far beyond them change nothing."""
    long_chunks = [100000 + 137 * i for i in range(8)]
    seen = [(n - 1) % 8192 + 1 for n in long_chunks]
    got = ranges(long_chunks, 8, 16, chunk=8192)
    assert got == ranges(seen, 8, 16) and sum(got) > 16
    assert ranges([50000, 60000, 900], 4, 32, window=4096) == ranges([4096, 4096, 900], 4, 32)
    assert ranges([50000, 60000, 900], 4, 32, window=4096, keep_first=512) == ranges([4608, 4608, 900], 4, 32)
    assert ranges([50000, 4200], 4, 32, window=4096, keep_first=512) == ranges([4608, 4200], 4, 32)
