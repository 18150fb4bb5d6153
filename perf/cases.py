"""Work that a user of this package has it do, as measurable cases.

Training goes through `Booster` (create from a host CSR, boost, read back) and through the scikit-learn style front end
(`TGBMRegressor.fit` on a NumPy matrix at its default learning rate of 1, then `predict`); prediction through the front end and through
`predict_raw`.  All of these take host arrays, so a pass is the whole call: upload, cut points, binning, boosting rounds
or tree walk, read-back.  The data sets are seeded synthetic ones with the shapes and value distributions of the
benchmark configurations (Higgs, covtype, a sparse text-like set, MSLR) and of the small regression sets of the tests.

Two histogram arithmetics: `fp32`, the library's default, and `exact`, the deterministic one.  fp32 sums floats in
arrival order: two runs of one training differ in the last bits, a near-tie between two splits then falls one way or the
other, and the trees that follow grow on other gradients.  After a few rounds of a noisy classification task the node
records, and the scores of single rows, of two runs of the SAME library on the same data are no longer comparable
(measured: scores 3 to 60 % apart in the 2-norm), while the metric that the library reports for every round agrees to
a few parts in a thousand.  Such trainings are therefore compared by these metrics, for every round; the exact
trainings, the regressions of the front end and the predictions by everything that they return.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

from thundergbm_b200.booster import Booster, predict_raw
from thundergbm_b200.synth import CsrData
from thundergbm_b200.thundergbm import TGBMModel, TGBMRegressor

_LABELS = 5  # relevance grades of the ranked data


def _case(name, do, data, rows, features, depth, rounds, **more):
    c = {} if name is None else dict(name=name)
    c.update(do=do, data=data, rows=rows, features=features, depth=depth, rounds=rounds, bins=255,
             rate=0.1, objective='reg:linear', arithmetic='fp32', builder='hist', classes=1, bagging=0, columns=1.0)
    c.update(more)
    return c


def listed():
    return [
        # one row scored by a service that keeps its model: latency
        _case('predict 1 row', 'predict', 'dense', 1, 28, 6, 100),
        # class probabilities for a batch of odd size, one-hot features (absent ones are missing values)
        _case('predict softprob 50003x54', 'predict', 'covtype', 50_003, 54, 8, 30, objective='multi:softprob', classes=7),
        # a whole data set scored from the CSR it is kept in
        _case('predict_raw 4M x28', 'predict_raw', 'higgs', 4_000_000, 28, 8, 100, objective='binary:logistic'),
        # the reference's shipped fixture by shape: 1605 rows of 0/1 features, all parameters at their defaults
        _case('fit 1605x119', 'fit', 'binary', 1_605, 119, 6, 40, rate=1.0),
        # small dense regression at the front end's defaults
        _case('fit 10000x32', 'fit', 'dense', 10_000, 32, 6, 40, rate=1.0),
        # a NumPy matrix of ordinary size through fit() and predict()
        _case('fit 400009x28', 'fit', 'dense', 400_009, 28, 6, 40, rate=1.0),
        # the headline benchmark: Higgs shape, default arithmetic, 100 rounds
        _case('train higgs 10.5M x28', 'train', 'higgs', 10_500_000, 28, 8, 100, objective='binary:logistic'),
        # the same data at a tenth of the rows in the deterministic arithmetic
        _case('train higgs 1M x28 exact', 'train', 'higgs', 1_050_000, 28, 8, 100, objective='binary:logistic',
              arithmetic='exact'),
        # seven trees per round, integer and one-hot columns
        _case('train covtype 581012x54', 'train', 'covtype', 581_012, 54, 8, 20, objective='multi:softmax', classes=7),
        # wide sparse text-like data, 64 bins
        _case('train sparse 1M x100000', 'train', 'sparse', 1_000_000, 100_000, 6, 40, objective='binary:logistic',
              bins=64, rate=0.3),
        # learning to rank, ragged query groups
        _case('train ranked 300k x136', 'train', 'ranked', 300_000, 136, 8, 20, objective='rank:ndcg'),
        # every distinct value a split candidate (tree_method=exact) on data of the size it is used for
        _case('train exact splits 200k x28', 'train', 'higgs', 200_000, 28, 6, 10, objective='binary:logistic',
              arithmetic='exact', builder='exact'),
    ]


def draw(rng):
    """One more case of the same ranges; cost bounded by the largest listed one."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(['predict', 'predict', 'predict_raw', 'fit', 'fit', 'train', 'train', 'train', 'sparse', 'ranked', 'exact'])
    depth = rng.randint(4, 8)
    if kind == 'predict':
        rows = log_int(1, 300_000)
        if rng.random() < 0.3:
            return _case(None, 'predict', 'covtype', rows, 54, depth, log_int(5, 40), objective='multi:softprob', classes=7)
        features = log_int(4, 150)
        return _case(None, 'predict', 'dense', max(1, min(rows, 20_000_000 // features)), features, depth, log_int(10, 200))
    if kind == 'predict_raw':
        return _case(None, 'predict_raw', 'higgs', log_int(1_000, 4_000_000), 28, depth, log_int(10, 150), objective='binary:logistic')
    if kind == 'fit':
        if rng.random() < 0.3:
            return _case(None, 'fit', 'binary', log_int(800, 4_000), log_int(60, 200), rng.randint(4, 7), log_int(10, 60), rate=1.0)
        features = log_int(5, 150)
        rows = min(log_int(1_000, 400_000), 12_000_000 // features)
        return _case(None, 'fit', 'dense', rows, features, rng.randint(4, 8), log_int(10, 60), rate=1.0, bins=rng.choice([255, 255, 64]))
    if kind == 'train':
        data = rng.choice(['higgs', 'higgs', 'covtype'])
        arithmetic = rng.choice(['fp32', 'fp32', 'exact'])
        fewest = 50_000 if arithmetic == 'fp32' else 5_000  # the metric of a few thousand rows is too coarse to compare fp32 runs by
        sampled = rng.random() < 0.25  # bagging with some of the columns left out
        extra = dict(bagging=1, columns=0.2) if sampled else {}
        if data == 'covtype':
            return _case(None, 'train', data, log_int(fewest, 581_012), 54, depth, log_int(5, 20), objective='multi:softmax',
                         classes=7, arithmetic=arithmetic, **extra)
        return _case(None, 'train', data, log_int(fewest, 5_000_000), 28, depth, log_int(10, 60), objective='binary:logistic',
                     arithmetic=arithmetic, bins=rng.choice([255, 255, 128]), **extra)
    if kind == 'sparse':
        return _case(None, 'train', 'sparse', log_int(20_000, 1_000_000), log_int(2_000, 100_000), rng.randint(4, 7), log_int(10, 40),
                     objective='binary:logistic', bins=64, rate=0.3, arithmetic=rng.choice(['fp32', 'exact']))
    if kind == 'ranked':
        arithmetic = rng.choice(['fp32', 'exact'])
        return _case(None, 'train', 'ranked', log_int(50_000 if arithmetic == 'fp32' else 10_000, 300_000), log_int(40, 136), depth,
                     log_int(5, 20), objective='rank:ndcg', arithmetic=arithmetic)
    return _case(None, 'train', 'higgs', log_int(5_000, 200_000), 28, rng.randint(4, 7), log_int(4, 12), objective='binary:logistic',
                 arithmetic='exact', builder='exact')


# ------------------------------------------------------------------ inputs
def _rand(seed):
    return torch.Generator(device='cuda').manual_seed(seed)


def _higgs(n, f, gen):
    """Kinematic-like columns: three quarters normal (half of them folded), the rest log-normal; a noisy linear label."""
    x = torch.randn(n, f, generator=gen, device='cuda')
    k = 3 * f // 4
    x[:, 0:k:2].abs_()
    x[:, k:].mul_(0.5).exp_()
    w = torch.zeros(f, device='cuda')
    w[::3] = torch.randn(len(range(0, f, 3)), generator=gen, device='cuda')
    s = x @ w + 0.5 * x[:, 0] * x[:, -1] - 0.4 * x[:, 1 % f] * x[:, 2 % f]
    y = torch.rand(n, generator=gen, device='cuda') < torch.sigmoid(s - s.median())
    x[x == 0] = 1e-30
    return x, y.float()


def _dense(n, f, gen):
    """Uniform columns, linear target with one product term and noise."""
    x = torch.rand(n, f, generator=gen, device='cuda').clamp_min_(1e-7)
    w = torch.randn(f, generator=gen, device='cuda')
    y = x @ w + 0.5 * x[:, 0] * x[:, 1] + 0.1 * torch.randn(n, generator=gen, device='cuda')
    return x, y


def _binary(n, f, gen):
    """0/1 columns, about one in nine set (a zero is a missing value), a target of two levels with noise."""
    x = (torch.rand(n, f, generator=gen, device='cuda') < 0.117).float()
    w = torch.randn(f, generator=gen, device='cuda')
    s = x @ w + torch.randn(n, generator=gen, device='cuda')
    return x, torch.where(s > s.median(), 1.0, -1.0)


def _covtype(n, f, gen):
    """Ten integer columns of different ranges, a one-hot group of four, a Zipf one-hot group of the rest; seven classes."""
    assert f > 14
    cap = 200 + (torch.rand(10, generator=gen, device='cuda') * 3800).floor()
    x = torch.zeros(n, f, device='cuda')
    x[:, :10] = (torch.rand(n, 10, generator=gen, device='cuda') * (cap + 1)).floor()
    row = torch.arange(n, device='cuda')
    x[row, 10 + torch.randint(0, 4, (n,), generator=gen, device='cuda')] = 1
    zipf = 1.0 / torch.arange(1, f - 13, device='cuda').pow(1.3)
    x[row, 14 + _from_table(zipf, n, gen)] = 1
    scale = torch.ones(f, device='cuda')
    scale[:10] = 1 / cap
    w = torch.randn(f, 7, generator=gen, device='cuda')
    gumbel = -torch.log(-torch.log(torch.rand(n, 7, generator=gen, device='cuda').clamp(1e-7, 1 - 1e-7)))
    return x, ((x * scale) @ w + gumbel).argmax(1).float()


def _from_table(weight, n, gen):
    """n indices drawn with probabilities proportional to `weight`."""
    c = (weight.double() / weight.double().sum()).cumsum(0)
    u = torch.rand(n, generator=gen, device='cuda', dtype=torch.float64)
    return torch.searchsorted(c, u).clamp_max_(weight.numel() - 1)


def _csr(x, y, group=None):
    """CSR of the values that are not zero, on the host."""
    n, f = x.shape
    keep = x != 0
    ptr = torch.zeros(n + 1, dtype=torch.int32, device='cuda')
    ptr[1:] = keep.sum(1).cumsum(0)
    if bool(keep.all()):
        val, col = x.reshape(-1), torch.arange(f, dtype=torch.int32, device='cuda').repeat(n)
    else:
        val, col = x[keep], torch.arange(f, dtype=torch.int32, device='cuda').expand(n, f)[keep]
    g = np.zeros(0, np.int32) if group is None else group
    return CsrData(n, f, ptr.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy(), y.float().cpu().numpy(), g)


def _sparse(n, f, gen):
    """About 40 values a row, all 1.0, columns with a heavy-tailed popularity, labels from a few thousand of the columns."""
    per_row = torch.poisson(torch.full((n,), 40.0, device='cuda'), generator=gen).long().clamp_min_(1)
    row = torch.repeat_interleave(torch.arange(n, device='cuda'), per_row)
    weight = torch.arange(1, f + 1, device='cuda').double().pow(-1.1)
    weight = weight / weight.sum() + 0.5 / f
    key = torch.unique(row * f + _from_table(weight, row.numel(), gen))
    row, col = key // f, key % f
    ptr = torch.zeros(n + 1, dtype=torch.int32, device='cuda')
    ptr[1:] = torch.bincount(row, minlength=n).cumsum(0)
    w = torch.zeros(f, device='cuda')
    used = torch.randperm(f, generator=gen, device='cuda')[:2000]
    w[used] = torch.randn(used.numel(), generator=gen, device='cuda')
    s = torch.zeros(n, device='cuda').index_add_(0, row, w[col])
    y = torch.rand(n, generator=gen, device='cuda') < torch.sigmoid(s)
    return CsrData(n, f, ptr.cpu().numpy(), col.int().cpu().numpy(), np.ones(col.numel(), np.float32), y.float().cpu().numpy())


def _ranked(n, f, gen, seed):
    """Count columns and log-normal scores in query groups of about 120 rows, five relevance grades."""
    h = f // 2
    x = torch.empty(n, f, device='cuda')
    x[:, :h] = torch.poisson(torch.full((n, h), 5.0, device='cuda'), generator=gen)
    z = torch.randn(n, f - h, generator=gen, device='cuda')
    x[:, h:] = z.exp()
    w = torch.randn(f, generator=gen, device='cuda')
    s = torch.cat([(x[:, :h] - 5) / 5 ** 0.5, z], 1) @ w / f ** 0.5 + 0.5 * torch.randn(n, generator=gen, device='cuda')
    order = s.sort().values
    edges = order[[int(q * (n - 1)) for q in (0.52, 0.84, 0.97, 0.99)]]
    y = torch.bucketize(s, edges).clamp_max_(_LABELS - 1)
    r, group = np.random.default_rng(seed), []
    left = n
    while left > 0:
        group.append(min(left, max(1, int(r.poisson(120)))))
        left -= group[-1]
    return _csr(x, y, np.asarray(group, np.int32))


_MAKE = {'higgs': _higgs, 'dense': _dense, 'binary': _binary, 'covtype': _covtype}


def _matrix(data, n, f, gen):
    x, y = _MAKE[data](n, f, gen)
    return x.cpu().numpy(), y.cpu().numpy()


def _params(case):
    return {'depth': case['depth'], 'n_trees': case['rounds'], 'max_num_bin': case['bins'], 'learning_rate': case['rate'],
            'objective': case['objective'], 'hist_mode': case['arithmetic'], 'tree_method': case['builder'],
            'bagging': case['bagging'], 'column_sampling_rate': case['columns'], 'sample_seed': 7,
            'lambda': 1.0, 'gamma': 1.0, 'min_child_weight': 1.0}


def _front_end(case):
    return dict(depth=case['depth'], n_trees=case['rounds'], learning_rate=case['rate'], max_num_bin=case['bins'],
                objective=case['objective'], num_class=case['classes'], tree_method='hist', verbose=0)


_TRAIN_ROWS = 30_000  # rows that the models of the prediction cases are trained on


def prepare(case, seed):
    gen = _rand(seed)
    n, f, do = case['rows'], case['features'], case['do']
    if do == 'train':
        if case['data'] == 'sparse':
            d = _sparse(n, f, gen)
        elif case['data'] == 'ranked':
            d = _ranked(n, f, gen, seed)
        else:
            d = _csr(*_MAKE[case['data']](n, f, gen))
        return dict(case=case, data=d, params=_params(case))
    if do == 'fit':
        x, y = _matrix(case['data'], n, f, gen)
        return dict(case=case, x=x, y=y, params=_front_end(case))
    # prediction: the trained model is in hand (trained in the deterministic arithmetic: the same model every time)
    m = _TRAIN_ROWS
    if do == 'predict_raw':
        x, y = _MAKE[case['data']](n + m, f, gen)
        b = Booster(_csr(x[n:], y[n:]), **{**_params(case), 'hist_mode': 'exact'})
        b.boost(case['rounds'])
        trees, base = b.trees(), b.info.base_score
        b.close()
        return dict(case=case, data=_csr(x[:n], y[:n]), trees=trees, base=base)
    x, y = _matrix(case['data'], n + m, f, gen)
    model = TGBMModel(**_front_end(case)) if case['classes'] > 1 else TGBMRegressor(**_front_end(case))
    before = os.environ.get('TGBM_HIST_MODE')
    os.environ['TGBM_HIST_MODE'] = 'exact'
    try:
        model.fit(x[n:], y[n:])
    finally:
        if before is None:
            del os.environ['TGBM_HIST_MODE']
        else:
            os.environ['TGBM_HIST_MODE'] = before
    return dict(case=case, model=model, x=np.ascontiguousarray(x[:n]))


# ------------------------------------------------------------------ one pass
def run(state):
    case = state['case']
    do = case['do']
    if do == 'predict':
        return state['model'].predict(state['x'])
    if do == 'predict_raw':
        return predict_raw(state['data'], state['trees'], case['rate'], state['base'])
    if do == 'fit':
        return TGBMRegressor(**state['params']).fit(state['x'], state['y']).predict(state['x'])
    b = Booster(state['data'], **state['params'])
    b.boost(case['rounds'])
    trees = b.trees()  # the model, which the caller is after
    out = dict(metrics=b.metrics(), base=b.info.base_score)
    if case['arithmetic'] == 'exact':
        out['scores'] = b.ypred()
        for k in ('split_feature_id', 'split_value', 'default_right', 'is_leaf', 'is_valid', 'is_pruned', 'base_weight', 'gain',
                  'sum_g', 'sum_h'):
            out[k] = np.ascontiguousarray(trees[k])
    b.close()
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    n, f, k, depth, rounds = case['rows'], case['features'], case['classes'], case['depth'], case['rounds']
    stored = {'sparse': 30.0, 'covtype': 12.0, 'binary': 0.117 * f}.get(case['data'], float(f))  # values of a row
    nodes = 2.0 ** (depth + 1) - 1
    trees = float(rounds * k)
    if case['do'] in ('predict', 'predict_raw'):
        row = 4.0 * f if case['do'] == 'predict' else 8.0 * stored + 4
        # a comparison per tree and level
        return dict(bytes=n * (row + 4.0 * k) + 16.0 * nodes * trees, flops=n * trees * depth)
    # per tree: the bin of every stored value and the gradient pair of every row once for the root, for half of the rows
    # at every level below it; (row, bin) of every row per level to move it; score and gradient once.  Adds: two per
    # value and histogram.  (the exact builder: every value once per level)
    value = 4.0 if case['data'] == 'sparse' or case['builder'] == 'exact' else 1.0
    share = float(depth) if case['builder'] == 'exact' else 1.0 + 0.5 * (depth - 1)
    per_tree = n * ((stored * value + 8) * share + 9.0 * (depth - 1) + 20.0)
    once = n * ((4.0 * f if case['do'] == 'fit' else 8.0 * stored + 4) + 8) + n * stored * value
    return dict(bytes=once + trees * (per_tree + 48.0 * nodes), flops=trees * 2.0 * n * stored * share)


def tolerance(case):
    if case['do'] in ('predict', 'predict_raw'):
        return {'rel': 1e-6}  # the same comparisons, at most another order of the sums of float leaf values
    if case['arithmetic'] == 'exact':
        return {'rel': 1e-5, 'max': 1e-4}  # integer sums decide the trees; metrics and weights are 32-bit floats
    if case['do'] == 'fit':
        return {'rel': 1e-2, 'max': 0.9}  # rows below a node whose two best splits tie may get another leaf
    return {'rel': 1e-2, 'max': 4e-2}  # the metrics of two fp32 runs, see above
