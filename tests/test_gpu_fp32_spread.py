"""fp32 mode on gradients of very different sizes: rounds whose gradients do not fit the integer grid are built from float
sums, so the weights follow the float64 ones to the rounding of float sums (tests/common.py: sum_noise)."""
import numpy as np
import pytest

from common import sum_noise
from thundergbm_b200.synth import CsrData

pytestmark = pytest.mark.gpu


def _csr(cols, stored, y):
    """Rows of `cols` where `stored`, the rest missing."""
    ptr = np.concatenate([[0], np.cumsum(stored.sum(1))]).astype(np.int32)
    return CsrData(cols.shape[0], cols.shape[1], ptr, np.nonzero(stored)[1].astype(np.int32), cols[stored].astype(np.float32), np.asarray(y, np.float32))


def _rounds(d, **p):
    """(trees, node of every row, scores before the round) of every round, one boost() each."""
    from thundergbm_b200.booster import Booster
    b = Booster(d, hist_mode='fp32', keep_nid=1, **p)
    scores = [np.full(d.n_rows, np.float32(b.info.base_score))]
    for _ in range(p['n_trees']):
        b.boost(1)
        scores.append(b.ypred()[0].copy())
    trees, nid = b.trees()[:, 0], b.nid()
    b.close()
    return trees, nid, scores


def _rows_below(nid, node, depth):
    at = nid.astype(np.int64).copy()
    hit = at == node
    for _ in range(depth):
        at = np.where(at > 0, (at - 1) // 2, 0)
        hit |= at == node
    return hit


# Three labels of 1e9: one row without values, which goes the default way with the two rows of the last bin (the two largest
# values share one), as min_child_weight keeps it from being alone.  The other side of the root split is summed without them,
# and so is everything below; lambda leaves half of the three labels for the next round, every time.
@pytest.mark.parametrize('n', [4001, 40_001])       # a tree per launch, level kernels
@pytest.mark.parametrize('layout', ['dense', 'sparse'])
def test_outliers_among_normal_labels(gpu, monkeypatch, n, layout):
    monkeypatch.setenv('TGBM_LAYOUT', layout)
    r = np.random.default_rng(n)
    x = np.stack([r.integers(1, 9, n), r.integers(1, 5, n)], 1)
    y = 3.0 * (x[:, 0] > 4) - 2.0 * (x[:, 1] > 2) + r.standard_normal(n)
    stored = np.ones((n, 2), bool)
    usual = np.ones(n, bool)
    usual[[7, 11, 12]] = False
    y[~usual] = 1e9
    stored[7] = False
    x[11:13, 0] = 9, 10
    stored[11:13, 1] = False
    depth = 3
    rounds = 12 if layout == 'sparse' else 7     # (from ten on the CSR layout has its values by column)
    trees, nid, scores = _rounds(_csr(x, stored, y), depth=depth, n_trees=rounds, max_num_bin=16, learning_rate=1.0, objective='reg:linear', gamma=0.0,
                                 min_child_weight=2.0, **{'lambda': 3.0})
    for t in (5, 6):
        g = (scores[t] - y.astype(np.float32)).astype(np.float64)
        assert abs(g[7]) > 1e6 and np.abs(g[usual]).max() < 10
        dg, _ = sum_noise(np.stack([g, np.ones(n)], 1)[usual], int(usual.sum()))
        checked = 0
        for i, node in enumerate(trees[t]):
            rows = _rows_below(nid[t], i, depth)
            if not node['is_valid'] or not rows.any() or not usual[rows].all():
                continue
            assert node['sum_h'] == rows.sum()
            assert abs(float(node['base_weight']) + g[rows].sum() / (rows.sum() + 3)) <= dg / rows.sum() + 1e-6
            checked += 1
        assert checked >= 3


# One such label loses half of what is left of it per round: the first rounds need float sums, the later ones do not.
def test_rounds_change_over(gpu):
    from thundergbm_b200.booster import Booster
    n, rounds = 50_000, 45
    r = np.random.default_rng(5)
    x = np.stack([r.integers(1, 9, n), r.integers(1, 5, n)], 1)
    y = 3.0 * (x[:, 0] > 4) - 2.0 * (x[:, 1] > 2) + r.standard_normal(n)
    stored = np.ones((n, 2), bool)
    y[7] = 1e9
    stored[7] = False
    y = y.astype(np.float32)
    got = []
    for step in (1, 9, rounds):
        b = Booster(_csr(x, stored, y), hist_mode='fp32', depth=3, n_trees=rounds, max_num_bin=16, learning_rate=1.0, objective='reg:linear')
        for done in range(step, rounds + 1, step):
            b.boost(step)
            if step < rounds:   # read in between: the metric is that of the scores
                e = y.astype(np.float64) - b.ypred()[0]
                assert b.info.rounds_done == done and abs(b.metrics()[-1] - np.sqrt(np.mean(e * e))) <= 1e-5 * b.metrics()[-1]
        got.append(b.metrics())
        assert got[-1].size == rounds and b.trees().shape[0] == rounds
        b.close()
    for m in got:   # (the score of that row is a float near 1e9: in steps of 64)
        assert np.allclose(m, got[0], rtol=1e-3, atol=4 * 64 / np.sqrt(n))
        assert m[-1] < 1.01   # the noise of the labels


# Rows that the model is sure of, beside rows that it cannot tell apart, and no regularisation: a leaf of the former has
# weight -sum g / sum h of values that are a millionth of the largest.  The grid moves every gradient by at most 2^-31 and
# every hessian by at most 2^-32 (the largest are 1/2 and 1/4), equal ones alike.  (Float sums cannot do that: what the root's
# sums and those over its bins differ by, 2^-24 of a hundred, counts as missing rows of the leaf.)
def test_confident_rows_without_regularisation(gpu):
    n = 1000
    x = np.concatenate([np.full(n, 1), 2 + np.arange(n) // 2 % 2])[:, None]   # (2 and 3 share a bin)
    y = np.concatenate([np.zeros(n), np.arange(n) % 2])
    trees, nid, scores = _rounds(_csr(x, np.ones((2 * n, 1), bool), y), depth=1, n_trees=14, learning_rate=1.0, objective='binary:logistic', gamma=0.0,
                                 min_child_weight=0.0, **{'lambda': 0.0})
    for t in range(2, 14):
        p = 1 / (1 + np.exp(-scores[t][0].astype(np.float64)))   # of a row of the former, label 0
        h = p * (1 - p)
        want, moved = -p / h, (2.0 ** -31 + 2.0 ** -32 * p / h) / h
        got = float(trees[t, 1]['base_weight'])
        assert trees[t, 1]['is_valid'] and abs(got - want) <= 1.01 * moved + 1e-6, (t, got, want)
    assert p < 1e-5


def test_gradients_that_are_not_numbers(gpu):
    n = 3000
    r = np.random.default_rng(2)
    x = r.integers(1, 9, (n, 3))
    y = x[:, 0] + r.standard_normal(n)
    y[5] = np.nan
    trees, _, scores = _rounds(_csr(x, np.ones((n, 3), bool), y), depth=3, n_trees=4, learning_rate=0.5, objective='reg:linear')
    assert np.isnan(trees[:, 0]['base_weight']).all()   # as float sums have it, in every round
    assert np.isnan(scores[-1]).all()


# the first round of a softmax objective: its trees are built side by side from float sums, in cells spread out or, where they
# are too many for that, close together.  All rows of a class carry the same gradient, so the nodes' sums are counts.
@pytest.mark.parametrize('classes,features,depth', [(3, 2, 1), (3, 5, 4), (7, 40, 6), (12, 33, 9)])
@pytest.mark.parametrize('layout', ['dense', 'sparse'])
def test_first_round_of_several_trees(gpu, monkeypatch, classes, features, depth, layout):
    from thundergbm_b200.booster import Booster
    monkeypatch.setenv('TGBM_LAYOUT', layout)
    n = 6007
    r = np.random.default_rng(classes)
    x = np.where(r.random((n, features)) < 0.5, 1.0, r.integers(1, 250, (n, features)))   # one bin with half of the rows
    y = r.integers(0, classes, n)
    b = Booster(_csr(x, r.random((n, features)) < 0.8, y), hist_mode='fp32', keep_nid=1, depth=depth, n_trees=1, max_num_bin=255, learning_rate=1.0,
                objective='multi:softmax', num_class=classes, min_child_weight=0.0, gamma=0.0)
    b.boost(1)
    trees, nid = b.trees()[0], b.nid().reshape(classes, n)
    b.close()
    g = 1 / classes - (y[None, :] == np.arange(classes)[:, None])
    h = 2 / classes * (1 - 1 / classes)
    for k in range(classes):
        # m values added one after the other, every addition rounding the running sum by half a unit at most: m 2^-24 of the sum.
        # (Equal values drift: the rounding errors do not cancel.)  A level's sums inherit what their ancestors' were off.
        noise_g, noise_h = n * 2.0 ** -24 * np.abs(g[k]).sum(), n * 2.0 ** -24 * n * h
        assert (trees[k]['is_valid'] != 0).sum() >= 3
        for node in np.nonzero(trees[k]['is_valid'])[0]:
            rows = _rows_below(nid[k], node, depth)
            assert abs(trees[k]['sum_g'][node] - g[k][rows].sum()) <= noise_g * (depth + 1)
            assert abs(trees[k]['sum_h'][node] - h * rows.sum()) <= noise_h * (depth + 1)


# rows to their children in row order: every block's place in a child's list from the rows of the blocks before, added up by the block
# or, from 8192 (block, child) pairs on, by a pass of its own; the last level's children of 9 blocks are on that side, those of 8 at it
@pytest.mark.parametrize('n', [8192, 9001])
@pytest.mark.parametrize('layout', ['dense', 'sparse'])
def test_row_lists_of_many_children(gpu, monkeypatch, n, layout):
    from thundergbm_b200.booster import Booster
    monkeypatch.setenv('TGBM_LAYOUT', layout)
    depth, classes, r = 12, 3, np.random.default_rng(n)
    x = r.integers(1, 120, (n, 6))
    y = r.integers(0, classes, n)
    b = Booster(_csr(x, r.random((n, 6)) < 0.9, y), hist_mode='fp32', keep_nid=1, depth=depth, n_trees=1, max_num_bin=255, learning_rate=1.0,
                objective='multi:softmax', num_class=classes, min_child_weight=0.0, gamma=0.0)
    b.boost(1)
    trees, nid = b.trees()[0], b.nid().reshape(classes, n)
    b.close()
    h = 2 / classes * (1 - 1 / classes)
    for k in range(classes):
        valid = trees[k]['is_valid'] != 0
        assert valid[1023:2047].sum() > 100 and valid[2047:4095].sum() > 100   # (it is as deep as it is meant to be)
        _, noise = sum_noise(np.stack([np.zeros(n), np.full(n, h)], 1), n // 50)   # of one level; inherited by the levels below
        rows = np.zeros(valid.size)
        np.add.at(rows, nid[k], 1)
        for node in range(valid.size // 2 - 1, -1, -1):   # the rows of the children were the node's
            rows[node] += rows[2 * node + 1] + rows[2 * node + 2]
        assert rows[0] == n and np.abs(trees[k]['sum_h'][valid] - h * rows[valid]).max() <= noise * (depth + 1) < h / 2
