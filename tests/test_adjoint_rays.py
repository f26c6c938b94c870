"""How many neighbouring rows' rays a thread of the exact adjoint marches, for launches
whose forms were timed: merging takes several times the rays where most of them may
carry a zero residual and be skipped.  No GPU needed."""
import ctypes as C

import pytest


@pytest.fixture(scope="module")
def rays():
    from spacetimetomography_b200 import build

    build.build_libstt()
    from spacetimetomography_b200._lib import lib

    f = lib.stt_internal_adjoint_rays
    f.argtypes = [C.c_int] * 3 + [C.c_float, C.c_int, C.c_int]
    f.restype = C.c_int
    return f


@pytest.mark.parametrize("W,H,n,pitch,views,want", [
    (512, 512, 256, 0.6, 1, 1),      # 214 us with one ray a thread, 287 with four (an ellipse of 20 % is live)
    (512, 512, 256, 0.6, 2, 2),      # 338 / 281 with two / 344 with four; in spots 254 / 283 / 363
    (512, 512, 256, 0.6, 4, 2),      # 782 / 639 / 610; in spots 465 / 432 / 557
    (512, 512, 256, 0.6, 12, 4),     # 2082 / 1491 / 1298
    (256, 256, 128, 0.6, 1, 1),      # 43 / 78
    (256, 256, 128, 0.6, 2, 1),      # 57 / 86
    (256, 240, 192, 0.9, 2, 1),      # 63 / 109
    (256, 240, 192, 0.9, 4, 1),      # 234 / 190; in spots 115 / 141
    (132, 106, 83, 0.9, 11, 2),      # of an object's shadow 101 / 95
    (121, 153, 108, 1.0, 1, 1),      # of shadows: 47 / 77
    (184, 187, 176, 1.0, 6, 1),      # 136 / 185
    (256, 256, 160, 0.75, 4, 2),     # 187 / 163
    (256, 256, 160, 0.75, 2, 1),     # 64 / 105
    (256, 240, 192, 0.9, 12, 2),     # 444 / 424; of an object's shadow 407 / 399
    (256, 240, 192, 0.9, 24, 2),     # 732 / 619
    (341, 341, 256, 0.9, 1, 1),      # 92 / 154
    (341, 341, 256, 0.9, 12, 2),     # 1026 / 905
    (128, 128, 128, 1.2, 128, 1),
])
def test_of_residuals_with_empty_surroundings(rays, W, H, n, pitch, views, want):
    assert rays(W, H, n, pitch, views, 0) == want


@pytest.mark.parametrize("W,H,n,pitch,views,want", [
    (512, 512, 256, 0.6, 1, 4),      # 453 / 356 / 338
    (256, 256, 128, 0.6, 1, 1),      # 80 / 90
    (256, 240, 192, 0.9, 1, 1),      # 86 / 106
    (256, 240, 192, 0.9, 2, 2),      # 174 / 139
    (341, 341, 256, 0.9, 1, 2),      # 229 / 195
    (128, 128, 128, 1.2, 128, 1),
])
def test_of_dense_residuals(rays, W, H, n, pitch, views, want):
    assert rays(W, H, n, pitch, views, 1) == want
