"""The standing host threads (tgbm::WorkerPool, thundergbm_b200/csrc/tgbm_workers.h) where threads cannot be started, and
after a fork.  No GPU is involved."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tasks_run_with_however_many_threads(tmp_path):
    exe = tmp_path / 'workers_check'
    subprocess.check_call(['g++', '-O1', '-std=c++17', '-pthread', os.path.join(ROOT, 'tests', 'cpp', 'workers_check.cpp'), '-o', str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120, check=True).stdout
    got = {l.split()[0]: [int(v) for v in l.split()[1:]] for l in out.strip().splitlines()}
    assert got == {'all': [36 * 50, 4], 'some': [36 * 150, 2], 'one': [36 * 150, 1], 'none': [36 * 150, 0], 'empty': [0, 0]}
