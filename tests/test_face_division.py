"""Division by multiplication of the fused face kernel's flat indexes
(FaceDiv, ard_face.cuh): i / d = umulhi(i + 1, floor((2^32 - 1) / d)) is exact for
0 <= i and (i + 1) d <= 2^32, checked at the multiples of d, where it can fail,
and far above every index that a layer of the largest extents gives."""
import numpy as np


def test_face_division_is_exact():
    for d in list(range(1, 2049)) + [4093, 8191, 65535, 65536]:
        m = np.uint64(0xFFFFFFFF // d)
        last = 2 ** 32 // d - 1                    # the largest i of the range
        q = np.unique(np.concatenate([np.arange(0, min(last // d, 400) + 1),
                                      np.linspace(0, last // d, 64).astype(np.int64)]))
        i = np.concatenate([q * d, q * d + d - 1, [last]])
        i = i[(i >= 0) & (i <= last)].astype(np.uint64)
        got = ((i + np.uint64(1)) * m) >> np.uint64(32)
        assert np.array_equal(got, i // np.uint64(d)), d
