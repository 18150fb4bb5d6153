"""Loops over stored values (tgbm::each_step, thundergbm_b200/csrc/tgbm_steps.h) up to the largest position, which a step from the
last value leaves.  No GPU is involved: 2^31 values are not loaded for this."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_position_is_met_once(tmp_path):
    exe = tmp_path / 'steps_check'
    subprocess.check_call(['g++', '-O1', '-std=c++17', os.path.join(ROOT, 'tests', 'cpp', 'steps_check.cpp'), '-o', str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, check=True).stdout
    got = {l.split()[0]: [int(v) for v in l.split()[1:]] for l in out.strip().splitlines()}
    sizes = dict(few=7, none=0, many=100_000, last_warp=70, last_value=1, last_grid=1000)
    assert got == {k: [n, n * (n - 1) // 2, max(n - 1, 0)] for k, n in sizes.items()}


def test_kernels_step_through_values_that_way():
    """None of the kernels that step through stored values counts their positions with a sign."""
    csrc = os.path.join(ROOT, 'thundergbm_b200', 'csrc')
    for name in ('tgbm_kernels.cuh', 'tgbm_level.cuh', 'tgbm_hist_f32.cuh'):
        text = open(os.path.join(csrc, name)).read()
        for start in ('row_ptr[r]', 'j0 + lane', 'c.bin_ptr[span.x]', '(int)run'):
            assert f'for (int j = {start}' not in text and f'for (int e = {start}' not in text and f'for (int e0 = {start}' not in text, (name, start)
            assert f'for (int i = {start} + 1 + lane' not in text and f'for (int j0 = {start}; j0 < j1; j0 +=' not in text, (name, start)
