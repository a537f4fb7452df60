"""bench.py counts the products of a table MSM by the library's own rule for
the affine rounds (csrc/msm.cuh)."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _constants():
    text = open(os.path.join(ROOT, "liblightzk_b200", "csrc", "msm.cuh")).read()
    low, fill = re.search(r"kAffMinEntries = 1u << (\d+), kAffFillTable = (\d+)", text).groups()
    return 1 << int(low), int(fill), int(re.search(r"kAffMaxRounds = (\d+);", text).group(1))


def test_rounds_of_the_product_count():
    import bench
    low, fill, top = _constants()

    def rounds(entries, buckets):          # affine_rounds of msm.cuh
        r = 0
        if entries < low:
            return 0
        while r < top and entries >= (buckets << (r + 1)) * fill:
            r += 1
        return r

    for points in (1, 100, 4369, 4370, 10000, 30000, 66000, 131072, 1000003, 1 << 20, 1 << 22):
        for c in (2, 8, 10, 13, 15, 16, 17, 20):
            w = -(-255 // c)
            rest = points * w / (1 << rounds(points * w, 1 << (c - 1)))
            want = (points * w - rest) * bench.FP_MUL_PER_G1_AFFINE + rest * bench.FP_MUL_PER_G1_MADD
            assert bench.g1_products(points, c, w) == want, (points, c)
