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
    """As many ranges each as two CTAs an SM hold at once, and never more."""
    from llm_b200.csrc import ops
    lens = [keys] * entries
    got = ranges(lens, n_kv, places(lens, n_kv))
    assert got == [ops.decode_splits(entries, n_kv, keys, SMS)] * entries
    if entries * n_kv <= 2 * SMS:                     # (shares rounded to the nearest took a second wave here)
        assert sum(got) * n_kv <= 2 * SMS


@pytest.mark.parametrize("seed", range(20))
def test_the_grid_holds_all_ranges(seed):
    """A launch has room for two CTAs an SM, and one for each request: no mix of lengths needs more."""
    import random
    rng = random.Random(seed)
    for n_kv in (1, 3, 8, 148, 296):
        lens = [int(2 ** rng.uniform(0, 20)) for _ in range(rng.randrange(1, 400))]
        got = ranges(lens, n_kv, 64)
        at_once = 2 * SMS // n_kv
        assert min(got) >= 1 and sum(got) <= at_once + sum(1 for n in lens if n * at_once < sum(lens))
        assert all(r <= max(1, -(-n // 256)) for r, n in zip(got, lens))


def test_a_long_request_among_short_ones_gets_more():
    assert ranges([6000] + [400] * 7, 8, 16) == [16] + [1] * 7
    got = ranges([20000] + [500] * 31, 8, 4)
    assert got[0] == 4 and set(got[1:]) == {1}
    assert ranges([20000] + [100] * 36, 8, 64) == [31] + [1] * 36
    # entries without keys, or of a negative length, have a place in which zeros are written
    assert ranges([0, 8192, -5, 8192], 8, 64) == [1, 18, 1, 18]


def test_only_the_keys_that_are_seen_count():
    """A chunk's, a window's and the kept first ones: lengths far beyond them change nothing."""
    long_chunks = [100000 + 137 * i for i in range(8)]
    seen = [(n - 1) % 8192 + 1 for n in long_chunks]
    got = ranges(long_chunks, 8, 16, chunk=8192)
    assert got == ranges(seen, 8, 16) and sum(got) > 16
    assert ranges([50000, 60000, 900], 4, 32, window=4096) == ranges([4096, 4096, 900], 4, 32)
    assert ranges([50000, 60000, 900], 4, 32, window=4096, keep_first=512) == ranges([4608, 4608, 900], 4, 32)
    assert ranges([50000, 4200], 4, 32, window=4096, keep_first=512) == ranges([4608, 4200], 4, 32)
