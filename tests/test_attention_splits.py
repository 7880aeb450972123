"""The default split count of the sparse attention decode against measured times."""
import pytest

from umdk_b200.ops.attention import default_splits

# (sequences, keys of each): {splits with keys: us} of the kernel and the merge on 148 SMs, back to back in a CUDA graph
MEASURED = {
    (1, 144): {1: 13.5, 2: 17.1, 3: 16.1},
    (1, 240): {1: 16.2, 2: 18.7, 3: 17.5, 5: 16.4},
    (1, 288): {1: 17.5, 2: 18.6, 3: 17.5, 6: 16.2},
    (1, 500): {1: 24.7, 2: 22.9, 3: 20.3, 4: 18.8, 6: 17.5, 11: 16.9},
    (1, 1000): {1: 39.0, 2: 29.8, 3: 24.5, 4: 23.0, 5: 21.6, 6: 20.6, 7: 19.0, 11: 18.2, 21: 17.7},
    (1, 2048): {1: 70.4, 2: 45.4, 3: 35.8, 4: 30.1, 5: 27.5, 6: 26.0, 7: 24.7, 8: 23.4, 9: 22.3, 11: 21.1, 15: 19.8, 22: 19.0, 43: 19.9},
    (1, 4000): {2: 74.2, 3: 54.5, 4: 44.5, 5: 39.0, 6: 34.6, 7: 31.9, 8: 30.5, 9: 29.5, 10: 28.1, 11: 26.7, 12: 25.4, 14: 24.2, 17: 23.2, 21: 21.9, 28: 21.0, 42: 21.3},
    (2, 384): {1: 20.5, 2: 20.4, 3: 19.0, 4: 17.6, 8: 16.7},
    (4, 336): {1: 19.1, 2: 20.5, 3: 19.2, 4: 18.1, 7: 17.1},
    (4, 1000): {1: 39.4, 2: 30.3, 3: 25.0, 4: 23.7, 5: 22.5, 6: 21.2, 7: 20.0, 11: 19.2, 21: 31.9},
    (4, 2048): {1: 70.9, 2: 46.2, 3: 36.4, 4: 30.9, 5: 28.2, 6: 26.8, 7: 25.8, 8: 24.4, 9: 23.3, 11: 22.3, 15: 21.3, 22: 34.8},
    (8, 240): {1: 16.5, 2: 19.5, 3: 18.4, 5: 17.9},
    (8, 500): {1: 25.2, 2: 23.6, 3: 21.5, 4: 20.2, 6: 19.6, 11: 32.0},
    (8, 1000): {1: 39.5, 2: 30.8, 3: 25.8, 4: 24.5, 5: 23.5, 6: 22.6, 7: 21.4, 11: 34.6},
    (8, 2048): {1: 71.0, 2: 46.8, 3: 37.4, 4: 31.9, 5: 29.2, 6: 28.2, 7: 27.2, 8: 26.0, 9: 25.0, 11: 40.3},
    (8, 4000): {2: 76.3, 3: 56.3, 4: 46.7, 5: 41.1, 6: 37.6, 7: 34.6, 8: 33.7, 9: 32.9, 10: 47.4, 11: 52.3, 12: 49.9},
    (16, 288): {1: 18.2, 2: 21.4, 3: 20.5},
    (16, 500): {1: 25.3, 2: 25.7, 3: 23.5, 4: 22.8},
    (16, 2048): {1: 72.0, 2: 49.4, 3: 39.6, 4: 34.8, 5: 53.3},
    (23, 240): {1: 16.8, 2: 22.8, 3: 22.1},
    (23, 500): {1: 25.4, 2: 27.3, 3: 25.3, 4: 38.5},
    (23, 1000): {1: 40.0, 2: 34.6, 3: 29.8, 4: 45.1},
    (23, 2048): {1: 72.8, 2: 51.0, 3: 41.9, 4: 63.1},
    (23, 4000): {2: 81.1, 3: 63.3, 4: 95.0},
}


@pytest.mark.parametrize("batch,topk", list(MEASURED))
def test_default_is_the_fastest_measured_count(batch, topk):
    times = {n: us for n, us in MEASURED[batch, topk].items() if n <= 24}
    n = default_splits(batch, topk, 148)
    assert times[n] <= 1.03 * min(times.values()), (n, times)


def test_no_split_without_keys():
    for batch in (1, 2, 3, 5, 8, 17, 23, 37, 64, 75, 200):
        for topk in list(range(1, 400)) + [480, 481, 1000, 2047, 2048, 2064, 2065, 4096, 10000, 200000]:
            least = -(-topk // 2064)   # what one CTA pair resolves
            n = default_splits(batch, topk, 148, least)
            per = -(-(-(-topk // n)) // 48) * 48   # keys per split, as the kernel rounds them
            assert least <= n <= max(least, 24, 1) and (n - 1) * per < topk <= n * per and per <= 2064
            assert n <= max(1, least, 148 // (2 * batch))


@pytest.mark.parametrize("topk", [1, 48, 2063, 2064, 2065, 4128, 4129, 100000])
def test_keys_of_a_split_are_those_that_the_kernel_takes(topk):
    from umdk_b200 import _native
    from umdk_b200.ops.attention import MAX_KEYS
    assert _native.cam().umdk_sparse_mla_min_splits(topk) == -(-topk // MAX_KEYS)


# the same of the kernel whose chunks take 0.9 us
MEASURED_SETS = {
    (1, 213): {1: 12.2, 2: 14.1, 3: 13.5, 5: 12.6},
    (1, 2048): {1: 46.8, 22: 14.8},
    (8, 2048): {1: 47.6, 9: 19.8},
    (23, 500): {1: 17.6, 2: 20.4, 3: 19.8},
    (23, 1000): {1: 28.4, 3: 24.3},
    (29, 692): {1: 21.6, 2: 24.6},
    (36, 1000): {1: 28.2, 2: 31.2},
}


@pytest.mark.parametrize("batch,topk", list(MEASURED_SETS))
def test_default_is_the_fastest_count_of_the_present_kernel(batch, topk):
    times = MEASURED_SETS[batch, topk]
    assert times[default_splits(batch, topk, 148)] <= 1.03 * min(times.values())
