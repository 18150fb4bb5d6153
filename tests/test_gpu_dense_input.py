"""A NumPy matrix through fit() / predict() (dense_train_scikit, dense_predict_scikit: its CSR is made on the GPU) gives what
the same matrix gives as the CSR scipy makes of it, and every prediction kernel gives the oracle's scores."""
import numpy as np
import pytest
import scipy.sparse as sp

from common import NODE_DTYPE
from thundergbm_b200 import synth

pytestmark = pytest.mark.gpu


def _matrix(n, f, zeros, dtype, seed=0):
    r = np.random.default_rng(seed)
    x = r.standard_normal((n, f)).astype(dtype)
    if zeros:
        x[r.random((n, f)) < zeros] = 0
        if n > 3 and f > 2:
            x[:, f - 1] = 0       # trailing column without a value
            x[2] = 0              # row without a value
            x[1, 0] = np.nan      # a NaN is stored
            x[0, 1] = -0.0
    return x


@pytest.mark.parametrize('n,f,zeros,dtype', [(1, 1, 0, np.float32), (33, 5, 0.5, np.float64), (257, 33, 0.3, np.float32),
                                             (1000, 28, 0, np.float32), (1000, 28, 0, np.float64), (2049, 97, 0.9, np.float32),
                                             (5000, 300, 0.2, np.float64)])
@pytest.mark.parametrize('objective', ['reg:linear', 'multi:softprob'])
def test_matrix_equals_its_csr(gpu, monkeypatch, n, f, zeros, dtype, objective):
    from thundergbm_b200.thundergbm import TGBMModel
    if objective == 'multi:softprob' and n < 100:
        pytest.skip('needs three classes')
    monkeypatch.setenv('TGBM_HIST_MODE', 'exact')
    x = _matrix(n, f, zeros, dtype)
    y = np.arange(n) % 3 if objective == 'multi:softprob' else np.nan_to_num(x[:, 0]) + np.arange(n) % 5
    got = []
    for form in (x, sp.csr_matrix(x), np.asfortranarray(x)):
        m = TGBMModel(depth=4, n_trees=5, learning_rate=0.5, verbose=0, objective=objective, tree_method='hist').fit(form, y)
        got.append((m.get_trees(), m.predict(form), m.predict(form[:max(1, n // 3)]), m.group_label))
    for trees, all_rows, some_rows, labels in got[1:]:
        for a, b in zip(got[0][0], trees):
            assert all(np.array_equal(a[k], b[k]) for k in a)
        assert np.array_equal(got[0][1], all_rows) and np.array_equal(got[0][2], some_rows)
        assert got[0][3] == labels
    assert len(got[0][3]) == len(set(np.float32(y).tolist()))


def _random_trees(rounds, k, depth, f, rng, cuts=200):
    n = (1 << (depth + 1)) - 1
    t = np.zeros((rounds, k, n), NODE_DTYPE)
    i = np.arange(n)
    t['lch_index'], t['rch_index'] = 2 * i + 1, 2 * i + 2
    t['is_leaf'] = (i >= n // 2) | ((i > 0) & (rng.random((rounds, k, n)) < 0.1))
    t['is_valid'] = 1
    t['split_feature_id'] = rng.integers(0, f, (rounds, k, n))
    grid = rng.standard_normal((f, cuts)).astype(np.float32)
    t['split_value'] = grid[t['split_feature_id'], rng.integers(0, cuts, (rounds, k, n))]
    t['default_right'] = rng.integers(0, 2, (rounds, k, n))
    t['base_weight'] = rng.standard_normal((rounds, k, n)).astype(np.float32)
    return t


@pytest.mark.parametrize('n,f,rounds,k,depth', [(1, 28, 100, 1, 6), (31, 28, 3, 1, 1), (600, 96, 40, 7, 8), (9001, 97, 9, 3, 5), (40_000, 31, 60, 1, 7),
                                                (700, 1200, 5, 1, 6), (200_000, 28, 300, 1, 8), (3, 20_000, 12, 2, 9)])
@pytest.mark.parametrize('full', [True, False])
def test_every_walk_equals_the_oracle(gpu, orc, n, f, rounds, k, depth, full):
    from thundergbm_b200.booster import predict_raw
    rng = np.random.default_rng(n + f)
    x = rng.standard_normal((n, f)).astype(np.float32)
    if not full:
        x[rng.random((n, f)) < 0.4] = 0
    d = synth.dense_to_csr(x, np.zeros(n, np.float32))
    trees = _random_trees(rounds, k, depth, f, rng)
    want = orc.predict_raw(d, trees, 0.3, 0.25)
    assert np.array_equal(predict_raw(d, trees, 0.3, 0.25), want)


# the walk from the matrix keeps more than 48 KB of leaf values in shared memory, a limit that every device has of its own
def test_large_direct_walk_on_every_device(gpu):
    import torch
    from thundergbm_b200.booster import predict_raw
    if torch.cuda.device_count() < 2:
        pytest.skip('needs two GPUs')
    rng = np.random.default_rng(1)
    d = synth.dense_to_csr(rng.standard_normal((20_000, 12)).astype(np.float32), np.zeros(20_000, np.float32))
    trees = _random_trees(100, 7, 4, 12, rng)
    got = []
    for dev in (0, 1, 0):
        torch.cuda.set_device(dev)
        got.append(predict_raw(d, trees, 0.3, 0.0))
    torch.cuda.set_device(0)
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


# a matrix of no columns has no cells and may be a null pointer: rows of missing values, like a CSR that stores nothing
@pytest.mark.parametrize('n', [5, 3_000_000])   # walked directly, by ranks
def test_matrix_without_columns(gpu, n):
    import ctypes as C
    from thundergbm_b200.thundergbm import TGBMModel
    x = _matrix(1000, 4, 0.5, np.float32)
    m = TGBMModel(depth=5, n_trees=30, learning_rate=0.5, verbose=0, objective='reg:linear', tree_method='hist').fit(x, np.arange(1000) % 7)
    got = np.full(n, np.nan, np.float32)
    m._lib.dense_predict_scikit(n, 0, None, 0, got.ctypes.data_as(C.c_void_p), C.byref(m.model), m.n_trees, m.tree_per_iter, b'reg:linear', m.num_class,
                                m.learning_rate, None, 0)
    assert not m._lib.tgbm_last_error()
    want = m.predict(sp.csr_matrix((n, 4), dtype=np.float32))
    assert np.array_equal(got, want)


# the labels of a model are those it was fitted with, whatever becomes of the caller's array
@pytest.mark.parametrize('n', [300, 70_000])   # counted before, and beside the training
def test_labels_of_the_model_are_its_own(gpu, n):
    from thundergbm_b200.thundergbm import TGBMRegressor
    x = _matrix(n, 3, 0, np.float32)
    y = np.arange(n, dtype=np.float32) % 251
    m = TGBMRegressor(depth=3, n_trees=2, verbose=0, tree_method='hist').fit(x, y)
    y[:] = 1
    assert m.group_label == [0.0] * 251


def test_failed_training_says_why(gpu):
    from thundergbm_b200.thundergbm import TGBMRegressor
    x = _matrix(70_000, 3, 0, np.float32)
    with pytest.raises(RuntimeError, match='depth must be in'):
        TGBMRegressor(depth=40, n_trees=2, verbose=0, tree_method='hist').fit(x, x[:, 0])
