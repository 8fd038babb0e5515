"""How many CTAs share a key block of the dK/dV kernel, and when the dQ kernel runs beside it, by what was measured."""
import ctypes

import pytest

import hipkittens_b200 as hk

# clusters of 2 to 8 dK/dV CTAs that a GPU of 148 SMs holds
HELD = [74, 45, 33, 27, 22, 18, 16]


def deal(B, N, H, H_KV, D, causal, NK=None):
    """CTAs per key block, CTAs of the dQ kernel (negative: behind the dK/dV kernel)."""
    held, ctas = (ctypes.c_int * 9)(0, 0, *HELD), ctypes.c_int()
    split = hk.capi().hk_selftest_bwd_dealing(B, N, NK or N, H, H_KV, D, int(causal), 148, held, ctypes.byref(ctas))
    return split, ctas.value


# us per backward, alone / shared
@pytest.mark.parametrize("shape,split", [
    ((1, 1024, 8, 1, 128, True), 8),    # 108 / 33
    ((1, 4096, 8, 1, 128, False), 4),   # 488 / 214
    ((1, 8192, 8, 1, 128, True), 3),    # 936 / 423
    ((1, 2048, 8, 1, 64, True), 8),     # 164 / 38
    ((2, 384, 8, 2, 128, True), 4),     # 28 / 21
    ((2, 1024, 16, 4, 128, False), 2),  # 87 / 71
    # not shared, so that a batch element's gradients are the same bits in a batch of any size: 131 / 81, 149 / 101, 163 / 126
    ((1, 2048, 16, 4, 128, True), 1), ((1, 2944, 16, 4, 64, True), 1), ((2, 2048, 16, 4, 128, True), 1),
    # nothing to gain: 204 / 220, 825 / 844, more than two blocks per SM
    ((2, 2048, 16, 4, 128, False), 1), ((1, 4096, 32, 4, 128, False), 1), ((16, 2048, 64, 8, 128, False), 1),
])
def test_key_blocks_are_shared_where_they_are_few(native_built, shape, split):
    assert deal(*shape)[0] == split


def test_no_cluster_that_the_gpu_does_not_hold(native_built):
    held, ctas = (ctypes.c_int * 9)(0, 0, 74, 45, 33), ctypes.c_int()
    for n, want in ((8, 4), (3, 3), (2, 1), (0, 1)):  # causal calls take no pairs
        sizes = (ctypes.c_int * 9)(*[held[i] if i <= n else 0 for i in range(9)])
        assert hk.capi().hk_selftest_bwd_dealing(1, 1024, 1024, 8, 1, 128, 1, 148, sizes, ctypes.byref(ctas)) == want


# us per backward in a loop: behind / beside
@pytest.mark.parametrize("shape", [
    (4, 940, 16, 8, 64, False),     # 89.4 / 104.8
    (3, 1405, 16, 4, 64, False),    # 115.8 / 132.5
    (6, 1129, 16, 4, 64, False),    # 164.4 / 188.2
    (7, 1152, 12, 4, 64, False),    # 140.6 / 160.6
    (4, 295, 64, 8, 64, False),     # 67.9 / 80.5
    (2, 2048, 16, 4, 64, False),    # 156 / 172
    (3, 423, 64, 8, 128, False),    # 108.0 / 116.0
    (2, 1280, 64, 8, 128, True),    # 233.4 / 259.2
    (2, 2347, 16, 4, 128, True),    # 196.1 / 214.0
    (9, 640, 32, 4, 64, True),      # 112.6 / 121.9
    (3, 2073, 16, 4, 64, True),     # 150.6 / 162.2
    (10, 256, 32, 4, 64, True),     # 49.4 / 54.7
    (5, 1408, 8, 2, 64, False),     # 101 / 118
    (8, 2176, 4, 4, 64, False),     # 166 / 182: the fourth round is 0.7 full
    (9, 2857, 8, 4, 64, True),      # 348.4 / 356.5, in pairs
])
def test_dq_waits_where_it_would_hold_up_the_key_blocks(native_built, shape):
    split, ctas = deal(*shape)
    assert split == 1 and ctas < 0


# ... and the calls that dQ beside dK/dV makes faster
@pytest.mark.parametrize("shape,split,ctas", [
    ((1, 512, 8, 8, 128, False), 1, 32),      # 23.6 / 15.3
    ((4, 1024, 12, 12, 64, False), 1, 148),   # 85 / 70
    ((9, 1100, 8, 8, 128, False), 1, 148),    # 180 / 167: the fifth round is 0.4 full
    ((5, 4218, 4, 1, 64, True), 1, 148),      # 254 / 241
    ((6, 567, 4, 4, 128, True), 1, 120),      # 29.3 / 23.8
    ((1, 2560, 8, 8, 64, True), 1, 148),      # 56.4 / 42.7
    ((1, 1024, 8, 1, 128, True), 8, 64),
    ((5, 512, 32, 8, 128, False), 1, 136),    # one by one: 108 behind, 78 on the SMs of the second round
])
def test_dq_fills_the_gaps(native_built, shape, split, ctas):
    assert deal(*shape) == (split, ctas)


def test_edges(native_built):
    assert deal(0, 1, 1, 1, 64, False)[0] < 0 and deal(1, 1, 3, 2, 64, False)[0] < 0 and deal(1, 1, 1, 1, 96, False)[0] < 0
    for B in (1, 2, 3, 5, 8, 16, 40, 200):
        for n in (1, 128, 129, 700, 3000):
            for h, hkv in ((1, 1), (8, 8), (8, 2), (24, 3), (64, 8)):
                for causal in (False, True):
                    split, ctas = deal(B, n, h, hkv, 128, causal)
                    items = B * h * ((n + 127) // 128)
                    assert 1 <= split <= 8 and 0 < abs(ctas) <= min(148, items)
                    blocks = B * hkv * ((n + 127) // 128)
                    assert split == 1 or blocks <= 2 * 148
