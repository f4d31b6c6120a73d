"""The further compile-time and TMA lengths the build instantiates
(ct_more_sizes.h, tma_more_sizes.h), beside those of test_length_tables.py."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "k-wave_b200"))

import build  # noqa: E402  (k-wave_b200/build.py)


def _smooth(n, primes):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


def test_more_lengths_are_the_seven_smooth_ones_from_40_to_1024():
    more = build._lengths("ct_more_sizes.h")
    assert sorted(set(more) | set(build.ct_sizes())) == [n for n in range(40, 1025) if _smooth(n, (2, 3, 5, 7))]
    assert not set(more) & set(build.ct_sizes()) and len(more) == len(set(more))


def test_every_compile_time_length_has_tma_kernels_and_equal_segments():
    tma = build.tma_sizes() + build._lengths("tma_more_sizes.h") + build._lengths("ct_more_sizes.h")
    assert sorted(tma) == sorted(build.ct_sizes() + build._lengths("ct_more_sizes.h"))
    for n in tma:  # the fewest segments of at most 256 points that divide n (make_spec_map)
        s = -(-n // 256)
        while n % s:
            s += 1
        assert n // s <= 256 and s <= 256
