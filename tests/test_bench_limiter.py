"""bench.py names as limiter what the histogram kernel of the layout issues, and gives a share only of a rate measured for it."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize('mode', ['fp32', 'exact'])
def test_limiter_of_the_layouts(mode):
    sys.path.insert(0, ROOT)
    import bench
    sparse, dense = bench.hist_limiter(mode, True, 1e11), bench.hist_limiter(mode, False, 1e11)
    assert sparse['limiter_frac'] is None and sparse['pair_peak_per_s'] is None and '64-bit' in sparse['limiter']
    assert 0 < dense['limiter_frac'] < 1 and ('4' if mode == 'fp32' else '2') in dense['limiter']
    assert set(sparse) == set(dense) and bench.hist_limiter(mode, False, None)['limiter_frac'] is None
