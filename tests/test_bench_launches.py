"""The launches the bench counts for one shallow-water gradient whose reverse sweep runs by segments."""

import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


def test_swm_segment_launches():
    # boundary rules, one call or six stages a step forward; per step six stages again, the stage
    # cotangents and six pairs of adjoint and scatter; per segment zeroed sums and their write-out
    def count(forward, steps, segments):
        return 1 + forward + steps * (6 + 1 + 12) + 2 * segments + 1

    assert bench.swm_segment_launches("cluster", 360, 30) == count(12, 360, 12) == 6878
    assert bench.swm_segment_launches("stages", 360, 30) == count(360 * 6, 360, 12)
    assert bench.swm_segment_launches("cluster", 31, 30) == count(2, 31, 2)
    assert bench.swm_segment_launches("stages", 1, 30) == count(6, 1, 1)
