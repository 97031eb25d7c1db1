"""The rule that cuts a GEMM into whole tiles and split ones, checked on the CPU over the shapes it can meet."""
import ctypes
import random

import pytest

from pippy_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib.available(), reason="the CUDA library is not built")


def test_plan_covers_every_tile_and_fits_the_workspace():
    fn = _lib.lib().pb_gemm_plan
    plan = (ctypes.c_int * 4)()
    rng = random.Random(0)
    split = 0
    for _ in range(4000):
        M, N, K = (max(1, int(2 ** rng.uniform(0, 16))) for _ in range(3))
        sms = rng.choice([2, 3, 100, 140, 147, 148])
        fn(M, N, K, sms, 1, plan)
        variant, whole, splits, items = plan
        ctas, bn = (2 if variant == 2 else 1), (128 if variant == 3 else 256)
        assert variant in (1, 2, 3) and (variant != 2 or M > 128)
        tiles = -(-M // (128 * ctas)) * -(-N // bn)
        if splits == 1:
            assert items == 0 and whole == tiles
            continue
        split += 1
        units, kb = sms // ctas, -(-K // 64)
        assert whole % units == 0 and whole < tiles and items == (tiles - whole) * splits <= units
        assert items * ctas <= 148 and (tiles - whole) * 4 * ctas <= 1024  # partials and counters of the workspace
        ranges = [(kb * i // splits, kb * (i + 1) // splits) for i in range(splits)]
        assert ranges[0][0] == 0 and ranges[-1][1] == kb and all(lo < hi for lo, hi in ranges)
        fn(M, N, K, sms, 0, plan)
        assert plan[2] == 1 and plan[3] == 0
    assert split > 200
