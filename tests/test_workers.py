"""The standing host threads (tgbm::WorkerPool, thundergbm_b200/csrc/tgbm_workers.h) where threads cannot be started, and
after a fork.  No GPU is involved."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tasks_run_with_however_many_threads(tmp_path):
    exe = tmp_path / 'workers_check'
    subprocess.check_call(['g++', '-O1', '-std=c++17', '-pthread', os.path.join(ROOT, 'tests', 'cpp', 'workers_check.cpp'), '-o', str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120, check=True).stdout
    got = {l.split()[0]: [int(v) for v in l.split()[1:]] for l in out.strip().splitlines()}
    assert got == {'all': [36 * 50, 4], 'some': [36 * 150, 2], 'one': [36 * 150, 1], 'none': [36 * 150, 0], 'empty': [0, 0]}


def test_a_forked_process_has_threads_of_its_own():
    """Labels of a classification are looked through by the standing threads before anything asks for a GPU.  (A process made
    by fork() cannot use the GPU of its parent; it must say so, not wait for threads that it does not have.)"""
    code = '''
import os, signal
import numpy as np
from thundergbm_b200.booster import Booster
from thundergbm_b200.synth import CsrData
n = 300_000
d = CsrData(n, 1, np.arange(n + 1, dtype=np.int32), np.zeros(n, np.int32), np.ones(n, np.float32), (np.arange(n) % 2).astype(np.float32))
def attempt():
    try:
        Booster(d, objective='binary:logistic', num_class=2, n_trees=1, depth=1).close()
    except RuntimeError as e:
        print(e)
attempt()
pid = os.fork()
if pid == 0:
    signal.alarm(30)
    attempt()
    os._exit(0)
_, status = os.waitpid(pid, 0)
assert status == 0, status
'''
    r = subprocess.run([sys.executable, '-c', code], cwd=ROOT, capture_output=True, text=True, timeout=120, env={**os.environ, 'CUDA_VISIBLE_DEVICES': ''})
    assert r.returncode == 0, r.stderr[-2000:]
