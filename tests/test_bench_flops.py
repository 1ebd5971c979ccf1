"""bench.py's count of the I3 kernel's flops: the middle node of an odd number of
radial nodes runs alone and costs less than a pair."""
import math

import bench


def test_flops_per_angle():
    N = 32
    P2, F = 4 * N * N, 5.0 * 4 * N * N * math.log2(4 * N * N)
    pair = 38 * F + 16 * 24 * P2 + 56 * N * N
    assert bench.i3_flops_per_angle(N, 16) == 8 * pair
    middle = bench.i3_flops_per_angle(N, 9) - 4 * pair
    assert middle == 35 * F + 16 * 16 * P2 + 24 * N * N < pair
