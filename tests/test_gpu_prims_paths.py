"""The feedback primitives at the sizes and key distributions where a call
changes its path: one CTA or a chain of launches, full and partial tiles,
digit passes that every key shares, the first pass's unordered ranking, the
straight and the partitioned bitmap, aligned and unaligned arrays.  Integers:
compared exactly with numpy."""
import numpy as np
import pytest

import rayt_gb300 as R
from tests.golden.common import NO_HIT, feedback_words

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()


def _wide(rng, n):
    return rng.integers(-2**31, 2**31, n, dtype=np.int64).astype(np.int32)


KEYS = {
    "wide": _wide,
    "narrow": lambda rng, n: rng.integers(-100, 101, n).astype(np.int32),
    "blocks": lambda rng, n: rng.integers(0, 1 << 24, n).astype(np.int32),
    "equal": lambda rng, n: np.full(n, -7, np.int32),
    "one_digit": lambda rng, n: (0x12003400 + (rng.integers(0, 256, n) << 16)).astype(np.int32),
    "two_digits": lambda rng, n: (rng.integers(0, 256, n) * 0x01000100 - 2**31).astype(np.int64).astype(np.int32),
    "skewed": lambda rng, n: np.where(rng.random(n) < 0.9, np.int32(5), _wide(rng, n)).astype(np.int32),
    "count_limit": lambda rng, n: (rng.integers(0, 1 << 14, n) - 2**31).astype(np.int64).astype(np.int32),
    "over_count_limit": lambda rng, n: np.where(np.arange(n) == 1, np.int32(16384 - 77),
                                                rng.integers(-77, 16384 - 77, n)).astype(np.int32),
    "by_lane_limit": lambda rng, n: (2**31 - 1 - rng.integers(0, 512, n)).astype(np.int32),
    "over_by_lane": lambda rng, n: rng.integers(-256, 257, n).astype(np.int32),
    "sorted": lambda rng, n: np.sort(_wide(rng, n)),
}


@pytest.mark.parametrize("n", [2, 33, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 8195, 16384, 16385, 24578, 100003])
@pytest.mark.parametrize("keys", sorted(KEYS))
@pytest.mark.parametrize("offset", [0, 1])
def test_sort_paths(built, n, keys, offset):
    a = KEYS[keys](np.random.default_rng(n), n)
    x = _dev(np.concatenate([np.full(offset, 9, np.int32), a, np.full(5, 9, np.int32)]))
    R.GPUSort(x[offset:], n)
    got = x.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + n], np.sort(a))
    assert np.all(got[:offset] == 9) and np.all(got[offset + n:] == 9)


def _digits(rng, n, *pick):
    """Keys of four digits: a number draws the digit as the numbers before it drew
    theirs, so every digit is spread evenly but the keys are not."""
    d = [rng.integers(0, 256, n) for _ in range(4)]
    return (sum(d[p] << (24 - 8 * k) for k, p in enumerate(pick)) - 2**31).astype(np.int32)


SPLIT_KEYS = {
    "wide": _wide,
    "blocks": KEYS["blocks"],
    "odd_range": lambda rng, n: rng.integers(-77, 3 << 22, n).astype(np.int32),
    "over_count_limit": KEYS["over_count_limit"],
    "sorted": KEYS["sorted"],
    "overfull": lambda rng, n: _digits(rng, n, 0, 0, 1, 2),
    "repeats": lambda rng, n: _digits(rng, n, 0, 1, 0, 1),
}


# one region for each resident CTA at most, whole turns of regions, partial and
# several tiles; the digits of "overfull" and "repeats" look even, but a region
# gets more keys than it holds, and bins get repeats by the dozen
@pytest.mark.parametrize("n", [8193, 155648, 155649, 622593, 1 << 20, 2000003, 4669441, 5000003, 1 << 23])
@pytest.mark.parametrize("keys", sorted(SPLIT_KEYS))
@pytest.mark.parametrize("offset", [0, 3])
def test_sort_split(built, n, keys, offset):
    a = SPLIT_KEYS[keys](np.random.default_rng(n), n)
    x = _dev(np.concatenate([np.full(offset, 9, np.int32), a, np.full(5, 9, np.int32)]))
    R.GPUSort(x[offset:], n)
    got = x.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + n], np.sort(a))
    assert np.all(got[:offset] == 9) and np.all(got[offset + n:] == 9)


@pytest.mark.parametrize("n", [1, 3, 127, 128, 1023, 8191, 8192, 8193, 16384, 16387, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_scan_paths(built, n, offset):
    a = _wide(np.random.default_rng(n), n)
    x = _dev(np.concatenate([np.full(offset, 9, np.int32), a, np.full(5, 9, np.int32)]))
    R.GPUScan(x[offset:], n)
    got = x.cpu().numpy()
    ref = np.cumsum(a.astype(np.int64)).astype(np.uint64).astype(np.uint32).view(np.int32)
    np.testing.assert_array_equal(got[offset:offset + n], ref)
    assert np.all(got[:offset] == 9) and np.all(got[offset + n:] == 9)


def _check_unique(words, nib, offset=0):
    import torch
    w = _dev(np.concatenate([np.zeros(offset, np.int32), words]))[offset:]
    out = torch.full((words.size + 3,), 9, dtype=torch.int32, device="cuda")
    cnt = R.feedback_unique(w, words.size, nib, out)
    conv = words.astype(np.int64)
    hit = (conv > 0) & (conv != NO_HIT)
    if nib > 0:
        conv[hit] = ((((conv[hit] >> 1) - 1) // nib + 1) << 1) | (conv[hit] & 1)
    ref = np.unique(conv).astype(np.int32)
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[:cnt], ref)
    assert np.all(got[words.size:] == 9)
    np.testing.assert_array_equal(w.cpu().numpy(), words)


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 12289, 65536, 262145])
@pytest.mark.parametrize("kind", ["feedback", "all_no_hit", "wide", "extremes", "no_no_hit", "dense"])
def test_unique_paths(built, n, kind):
    rng = np.random.default_rng(n)
    nib = 512 if kind in ("feedback", "no_no_hit") else 0
    if kind == "feedback":
        words = feedback_words(n, n)
    elif kind == "all_no_hit":
        words = np.full(n, NO_HIT, np.int32)
    elif kind == "wide":
        words = _wide(rng, n)
        words[rng.random(n) < 0.3] = NO_HIT
    elif kind == "extremes":
        words = rng.choice(np.array([-2**31, 2**31 - 2, NO_HIT, -1, 0, 1], np.int64), n).astype(np.int32)
    elif kind == "no_no_hit":
        words = feedback_words(n, n, no_hit=False, id_bits=12)
    else:  # every value of a range: full bitmap words
        words = (np.arange(n) - n // 2).astype(np.int32)
        rng.shuffle(words)
    _check_unique(words, nib, offset=n % 2)


@pytest.mark.parametrize("case", ["direct_limit", "over_limit", "few_keys", "more_keys", "small_bitmap", "partition", "partition_one_bucket", "wide_over_direct"])
def test_unique_large_paths(built, case):
    """The largest inputs that go straight into the bitmap (2^21 words), kept
    keys around 2^18 and a wide bitmap, the partitioned bitmap on even and
    skewed ranges, the radix passes."""
    rng = np.random.default_rng(11)
    if case == "direct_limit":
        words = (rng.permutation((1 << 21) + 64)[:1 << 21] - 5000).astype(np.int32)
    elif case == "over_limit":
        words = (rng.permutation((1 << 21) + 64)[:1 << 21] - 5000).astype(np.int32)
        words = np.concatenate([words, np.full(9, NO_HIT, np.int32)])
    elif case in ("few_keys", "more_keys"):
        words = np.full((1 << 21) + 4097, NO_HIT, np.int32)
        m = (1 << 18) + (case == "more_keys")
        words[rng.permutation(words.size)[:m]] = rng.permutation(1 << 25)[:m]
    elif case == "small_bitmap":  # 2^20 values, each several times
        words = rng.integers(-1000, (1 << 20) - 1000, (1 << 22) + 5).astype(np.int32)
    elif case == "partition":
        words = rng.permutation((1 << 22) + 4097).astype(np.int32)
    elif case == "partition_one_bucket":
        words = np.concatenate([rng.permutation(3 << 20), [(1 << 26) - 1, NO_HIT]]).astype(np.int32)
    else:
        words = _wide(rng, (1 << 22) + 3)
    _check_unique(words, 0)


@pytest.mark.parametrize("n", [8193, 70001, 1 << 19, (1 << 21) - 3, (1 << 21) + 1])
@pytest.mark.parametrize("bits", [15, 20, 21, 22, 25, 26])
@pytest.mark.parametrize("kept", [0.03, 0.9])
def test_unique_bitmap_slices(built, n, bits, kept):
    """Bitmaps of one slice, of several (few keys and many), wider than 32 bits
    per input word, of the widest range that has one, and one value wider."""
    rng = np.random.default_rng(n + bits)
    for span in {15: [31 << 15], 20: [1 << 20, (1 << 20) + 1], 26: [1 << 26, (1 << 26) + 1]}.get(bits, [1 << bits]):
        words = np.full(n, NO_HIT, np.int32)
        at = rng.permutation(n)[:max(2, int(n * kept))]
        keys = np.where(rng.random(at.size) < 0.5, rng.integers(0, span, at.size), rng.integers(0, 1 + span // 64, at.size))
        keys[:2] = 0, span - 1
        words[at] = (keys - span // 3).astype(np.int32)
        _check_unique(words, 0, offset=n % 2)


# a round is 16384 elements per SM (152): one, two and three rounds and the
# element after them, and rounds enough that every buffer and slot is used again
@pytest.mark.parametrize("n", [2490368, 2490369, 4980736, 4980739, 7471104, 7471107, 17432581, 40000003])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_scan_rounds(built, n, offset):
    a = _wide(np.random.default_rng(n), n)
    x = _dev(np.concatenate([np.full(offset, 9, np.int32), a, np.full(5, 9, np.int32)]))
    R.GPUScan(x[offset:], n)
    got = x.cpu().numpy()
    ref = np.cumsum(a.astype(np.int64)).astype(np.uint64).astype(np.uint32).view(np.int32)
    np.testing.assert_array_equal(got[offset:offset + n], ref)
    assert np.all(got[:offset] == 9) and np.all(got[offset + n:] == 9)


# the split's largest size (15 turns of 304 regions of 15360 keys) and the
# smallest that takes the digit passes, or the counting in them, at once
@pytest.mark.parametrize("n,keys,offset", [(70041600, "wide", 0), (70041600, "narrow", 0), (70041601, "wide", 0),
                                           (70041601, "narrow", 0), (70041601, "count_limit", 3),
                                           (70041601, "over_count_limit", 0), (70041601, "one_digit", 1),
                                           (70041601, "equal", 0)])
def test_sort_beyond_the_split(built, n, keys, offset):
    a = KEYS[keys](np.random.default_rng(n), n)
    x = _dev(np.concatenate([np.full(offset, 9, np.int32), a, np.full(5, 9, np.int32)]))
    R.GPUSort(x[offset:], n)
    got = x.cpu().numpy()
    a.sort()
    np.testing.assert_array_equal(got[offset:offset + n], a)
    assert np.all(got[:offset] == 9) and np.all(got[offset + n:] == 9)


@pytest.mark.parametrize("n", [8193, 40000, (1 << 21) + 5, 7000001])
@pytest.mark.parametrize("span", [199, 1 << 22, 1 << 30])
def test_unique_full_and_sparse_stretches(built, n, span):
    """Stretches of 512 words of which all, most, some or none are kept follow
    one another, so a warp's region of kept words meets every fill before a
    stretch that is kept whole."""
    rng = np.random.default_rng(n + span)
    share = rng.choice([0.0, 0.02, 0.1, 0.24, 0.9, 1.0, 1.0], n // 512 + 1).repeat(512)[:n]
    words = np.where(rng.random(n) < share, rng.integers(-span, span, n), NO_HIT).astype(np.int32)
    _check_unique(words, 0, offset=n % 2)
