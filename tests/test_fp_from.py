"""Where a call's projections fetch their corners (the rule stt_fp and
stt_fp_correction follow), for calls whose forms were timed: a copy of the volume is
made only where it pays, and near an axis FP32 volumes that stay in the L2 are
projected by loads.  No GPU needed."""
import ctypes as C

import pytest

LOADS, OWN, ANY = 0, 1, 2


@pytest.fixture(scope="module")
def rule():
    from spacetimetomography_b200 import build

    build.build_libstt()
    from spacetimetomography_b200._lib import lib

    f = lib.stt_internal_fp_from
    f.argtypes = [C.c_longlong, C.c_float, C.c_int, C.c_int, C.POINTER(C.c_int), C.c_longlong]
    f.restype = C.c_int

    def of(n, det, degrees, esize=4):
        views = (C.c_int * 18)()
        for d in degrees:  # angles of the rotation about y: along z from 0 to 45 and 135 to 225
            d = d % 180
            along_x = 45 < d < 135
            off = abs(d - 90) if along_x else min(d, 180 - d)
            views[9 * along_x + min(int(off // 5), 8)] += 1
        own = n * n * esize % 32 == 0  # (slices the texture unit can step over)
        return f(n**3, 2.0 * n / det * 0.6, esize, own, views, det * det * len(degrees))

    return of


@pytest.mark.parametrize("n,det,degrees,want", [
    (255, 512, [0], LOADS),            # 106 us, with a mirror 144
    (255, 256, [10], OWN),             # 52 / 74 with a mirror; 256^3 from its own texture 42
    (255, 512, [20], OWN),             # 125 / 147
    (255, 512, [18] * 8, LOADS),       # 772 / 884; 256^3 from its own texture 720
    (256, 512, [18] * 8, ANY),
    (129, 512, [12] * 3, LOADS),       # 147 / 171
    (65, 32, [0] * 24, OWN),           # 19 / 22
    (255, 512, [30], ANY),             # 163 / 147
    (255, 512, [40], ANY),             # 202 / 148
    (255, 512, [90], ANY),             # 178 / 141: loads copy the volume too
    (255, 128, [0], OWN),              # 48 / 50
    (187, 128, [0], ANY),              # 37 / 27
    (187, 192, [0], OWN),              # 37 / 39
    (301, 256, [0], ANY),              # 112 / 98: past the L2
    (301, 64, [0] * 24, LOADS),        # 92 / 196: few rows, far apart
    (301, 64, [0], OWN),               # 56 / 69
    (256, 64, [0] * 24, LOADS),        # 75 / 117
    (256, 512, [0] * 8, LOADS),        # 730 / 852
    (256, 512, [90] * 8, LOADS),       # 765 / 827
    (256, 512, [90], ANY),             # 176 / 116
    (256, 256, [0] * 3, ANY),          # 111 / 103
    (256, 512, [0] * 3, LOADS),        # 293 / 329
    (255, 128, [18] * 8, OWN),         # 103 / 141
    (192, 512, [90] * 3, LOADS),       # 222 / 239
    (320, 512, [0] * 8, ANY),          # 1211 / 1090
    (128, 256, [10] * 3, ANY),         # 55 / 53 (loads / own texture)
    (187, 128, [18] * 8, ANY),         # 92 / 77
    (187, 256, [23], ANY),             # 58 / 43
    (256, 512, [20] * 8, ANY),         # 782 / 720
    (256, 512, [0, 36, 72, 108, 144, 180, 216, 252], ANY),
])
def test_fp32_calls(rule, n, det, degrees, want):
    assert rule(n, det, degrees) == want


@pytest.mark.parametrize("n,det,degrees,want", [
    (301, 256, [0], OWN),              # 60 / 74
    (301, 128, [0] * 8, OWN),          # 89 / 120
    (301, 128, [0], ANY),              # 64 / 53
    (203, 64, [0] * 24, OWN),          # 59 / 71
    (187, 64, [12] * 8, ANY),          # 46 / 38
    (65, 64, [0] * 8, OWN),            # 17 / 22
    (65, 256, [0] * 8, ANY),           # 70 / 61
    (301, 512, [0], ANY),              # 128 / 137, three views 329 / 298
    (255, 512, [0], ANY),              # 110 / 100
    (301, 256, [30], ANY),             # 109 / 80
    (187, 333, [0] * 15, ANY),
])
def test_bf16_calls(rule, n, det, degrees, want):
    assert rule(n, det, degrees, esize=2) == want


def test_a_ring_uses_textures_whatever_its_size(rule):
    ring = [137.508 * k + 17 for k in range(36)]
    for n in (64, 129, 192, 255, 301, 361):
        for det in (64, 128, 256, 512):
            for esize in (4, 2):
                assert rule(n, det, ring, esize) == ANY
