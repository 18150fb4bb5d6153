"""Sizes at which the training kernels change over: edges of tiles, warps and shared memory, and the sizes on either side of
the rules that choose between them.  Against the CPU oracle bit for bit, or against NumPy where the result is a plain count."""
import numpy as np
import pytest

from thundergbm_b200.synth import CsrData

pytestmark = pytest.mark.gpu


def _csr(x, y):
    n, f = x.shape
    return CsrData(n, f, (np.arange(n + 1) * f).astype(np.int32), np.tile(np.arange(f, dtype=np.int32), n), np.ascontiguousarray(x, np.float32).ravel(),
                   np.asarray(y, np.float32))


def _holes(x, y, keep):
    """The same with only the kept entries stored."""
    n, f = x.shape
    ptr = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return CsrData(n, f, ptr, np.nonzero(keep)[1].astype(np.int32), np.ascontiguousarray(x[keep], np.float32), np.asarray(y, np.float32))


def _data(n, f, classes, seed, holes=0.2, levels=40):
    r = np.random.default_rng(seed)
    x = r.integers(1, levels, (n, f)).astype(np.float32)   # few distinct values: ties and runs
    y = r.integers(0, classes, n) if classes > 1 else x[:, 0] + 3 * (x[:, -1] > 20) + r.random(n)
    return _holes(x, y, r.random((n, f)) >= holes) if holes else _csr(x, y)


def _same_as_oracle(orc, d, **p):
    from thundergbm_b200.booster import Booster
    o = orc.train(d, hist_mode=1, keep_nid=0, **p)
    b = Booster(d, hist_mode='exact', **p)
    b.boost(p['n_trees'])
    assert b.trees().tobytes() == o.trees.tobytes()
    assert np.array_equal(b.ypred(), o.ypred)
    assert np.array_equal(b.metrics(), o.metric)
    b.close()


# one cluster builds the tree up to 32768 rows (each of its CTAs moves them for itself up to 4096), the level kernels from there on
@pytest.mark.parametrize('n,f,depth,classes,extra', [
    (1, 1, 1, 1, {}), (2, 3, 6, 1, {}), (31, 5, 4, 3, {}), (1023, 33, 6, 1, {}), (1025, 130, 9, 1, {}), (8191, 8, 10, 1, {}),
    (3001, 600, 3, 1, {}), (4096, 20, 7, 1, {}), (4097, 17, 6, 7, dict(bagging=1, sample_seed=3)), (5000, 64, 7, 1, dict(column_sampling_rate=0.3, sample_seed=5)),
    (32768, 20, 6, 1, {}), (32769, 20, 6, 1, {})])
def test_small_trees(gpu, orc, n, f, depth, classes, extra):
    d = _data(n, f, classes, n + f)
    p = dict(depth=depth, n_trees=3, max_num_bin=64, learning_rate=0.5, objective='multi:softmax' if classes > 1 else 'reg:linear', num_class=classes, **extra)
    _same_as_oracle(orc, d, **p)


# tiles of 1024 entries, several columns in one and one column over several; groups that end at a tile's edge
@pytest.mark.parametrize('n,f,depth,levels', [(1, 1, 2, 3), (1023, 1, 3, 500), (1024, 1, 6, 2), (1025, 2, 6, 10 ** 6), (512, 7, 4, 40), (300, 150, 9, 8),
                                              (40_000, 3, 8, 10 ** 6)])
@pytest.mark.parametrize('holes', [0, 0.5])
def test_exact_splits(gpu, orc, n, f, depth, levels, holes):
    d = _data(n, f, 1, 7 * n + f, holes, levels)
    if holes:
        d.y[: n // 3] = 0   # nodes that stop early: their entries leave
    _same_as_oracle(orc, d, depth=depth, n_trees=3, learning_rate=0.5, objective='reg:linear', tree_method='exact')


# from 2^21 rows on the columns of a full matrix are sorted one by one
@pytest.mark.parametrize('n', [(1 << 21) - 1, 1 << 21, (1 << 21) + 4097])
def test_cut_points_of_full_columns(gpu, n):
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(n)
    x = np.stack([r.standard_normal(n), r.integers(-3, 4, n), np.full(n, -0.0), r.integers(0, 300, n) * 1e-3, np.linspace(-1, 1, n)], 1).astype(np.float32)
    x[5, 2] = 0.0
    b = Booster(_csr(x, x[:, 0]), depth=3, n_trees=1, max_num_bin=255, objective='reg:linear')
    val, ptr = b.cuts()
    for j in range(x.shape[1]):
        u = np.unique(x[:, j])
        s = len(u) // 255
        want = u if s == 0 else u[np.arange(255) * s]
        assert np.array_equal(val[ptr[j]:ptr[j + 1]], want)
    b.close()


# more rows per CTA than the 16-bit halves of one window hold: 150 groups of columns leave one CTA each
def test_window_of_the_halved_sums(gpu):
    from thundergbm_b200.booster import Booster
    n, f = 70_001, 4 * 1200
    r = np.random.default_rng(1)
    cols = r.integers(1, 6, (n, 4)).astype(np.float32)
    x = np.tile(cols, (1, f // 4))
    b = Booster(_csr(x, 1e3 * cols[:, 0] + cols[:, 1]), depth=3, n_trees=3, max_num_bin=16, objective='reg:linear', hist_mode='fp32', keep_nid=1)
    b.boost(3)
    trees, nid = b.trees()[:, 0], b.nid().reshape(3, n)
    assert (b.quant_scale()[1:] != 1).all()   # the later rounds did sum on the grid
    for t in range(1, 3):   # hessian 1: a node's sum is its number of rows
        for i in np.unique(nid[t]):
            at, rows = int(i), nid[t] == i
            assert trees[t, at]['sum_h'] == rows.sum()
        assert trees[t, 0]['sum_h'] == n
    b.close()


# column ids travel as 16-bit numbers where all of them fit; page-locked arrays are copied as they are
@pytest.mark.parametrize('top', [65535, 65536])
def test_column_ids_of_a_large_csr(gpu, top):
    import torch
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(top)
    n = 150_001
    col = np.sort(r.choice(2000, (n, 5), replace=True) * 2 + np.arange(5), 1).astype(np.int32)
    keep = np.concatenate([np.ones((n, 1), bool), np.diff(col, axis=1) > 0], 1)
    keep[0] = True
    col[0] = [0, 1, 2, 3, 4]
    col[n // 2, -1] = top
    keep[n // 2] = [True, False, False, False, True]
    d = _holes(r.integers(1, 9, (n, 5)).astype(np.float32), col[:, 0] % 7 + r.random(n), keep)
    d.n_cols, d.col = top + 1, col[keep]
    pinned = CsrData(n, top + 1, *[torch.from_numpy(a).pin_memory().numpy() for a in (d.row_ptr, d.col, d.val, d.y)])
    got = []
    for data in (d, pinned):
        b = Booster(data, depth=4, n_trees=2, max_num_bin=16, objective='reg:linear', hist_mode='exact')
        b.boost(2)
        assert b.info.n_features == top + 1
        got.append((b.trees().tobytes(), b.ypred().tobytes()))
        b.close()
    assert got[0] == got[1]


# CSR layout: rows around the 32 values that a warp adds up at a time
@pytest.mark.parametrize('longest', [1, 32, 33, 64, 65, 400])
def test_rows_of_the_csr_layout(gpu, orc, monkeypatch, longest):
    monkeypatch.setenv('TGBM_LAYOUT', 'sparse')
    r = np.random.default_rng(longest)
    n, f = 3001, 400
    keep = r.random((n, f)).argsort(1) < r.integers(0, longest + 1, n)[:, None]
    keep[0] = np.arange(f) < longest
    x = r.integers(1, 9, (n, f)).astype(np.float32)
    d = _holes(x, (x * keep)[:, :20].sum(1) + r.random(n), keep)
    _same_as_oracle(orc, d, depth=6, n_trees=3, max_num_bin=16, learning_rate=0.5, objective='reg:linear')


# the trees of a round stand side by side in as much memory as there is, one by one if need be: the same trees
def test_softmax_trees_in_little_memory(gpu):
    import torch
    from thundergbm_b200 import _lib
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(3)
    x = r.standard_normal((3000, 30)).astype(np.float32)
    d = _csr(x, (x[:, 0] > 0) + 2 * (x[:, 1] > 0) + 3 * (x[:, 2] > 1))
    got = []
    for fill in (False, True):
        _lib.lib().tgbm_release_device_memory()
        torch.cuda.empty_cache()
        filler = torch.empty(torch.cuda.mem_get_info()[0] - (1500 << 20), dtype=torch.uint8, device='cuda') if fill else None
        b = Booster(d, depth=12, n_trees=2, objective='multi:softmax', num_class=7, hist_mode='exact')   # 0.6 GB per tree
        b.boost(2)
        got.append((b.trees().tobytes(), b.ypred().tobytes()))
        b.close()
        del filler
    torch.cuda.empty_cache()
    assert got[0] == got[1]


# chunks of 1024 rows with remainders, few and many children, several chunks per block; trees side by side in chunks of 2048 rows
@pytest.mark.parametrize('n,f,depth,classes,layout', [(1, 3, 3, 1, 'sparse'), (255, 5, 4, 1, 'sparse'), (1025, 5, 6, 1, 'sparse'), (2049, 3, 9, 1, 'sparse'),
                                                      (32_769, 4, 1, 1, 'dense'), (33_793, 4, 2, 1, 'dense'), (40_961, 5, 10, 1, 'dense'),
                                                      (180_225, 4, 5, 7, 'dense')])
def test_rows_to_children(gpu, orc, monkeypatch, n, f, depth, classes, layout):
    monkeypatch.setenv('TGBM_LAYOUT', layout)
    p = dict(depth=depth, n_trees=3, max_num_bin=64, learning_rate=0.5, objective='multi:softmax' if classes > 1 else 'reg:linear', num_class=classes)
    _same_as_oracle(orc, _data(n, f, classes, n), **p)


# the CSR layout with its columns sorted (from ten trees on) and without: more bins than the shared ones (columns of one value,
# of a few, of runs that span several warps), columns too long for the nodes that split on them, and rows that store a column twice
# (no sorted columns)
@pytest.mark.parametrize('n,f,depth,twice', [(700, 14_000, 4, False), (3000, 60, 5, False), (40_000, 130, 6, False), (2000, 60, 4, True)])
@pytest.mark.parametrize('trees', [9, 10])
def test_columns_of_the_csr_layout(gpu, orc, monkeypatch, n, f, depth, twice, trees):
    monkeypatch.setenv('TGBM_LAYOUT', 'sparse')
    r = np.random.default_rng(n)
    share = np.clip(1.5 / np.arange(1, f + 1) ** 0.6, 3 / n, 0.98)     # popular columns first, rare ones last
    keep = r.random((n, f)) < share
    keep[:, 0] = True
    x = r.integers(1, 250 if f < 200 else 3, (n, f)).astype(np.float32)
    y = x[:, 0] / 100 + keep[:, 1] + 2 * keep[:, f // 2] + (x[:, f // 3] > 1) * keep[:, f // 3] + r.random(n)
    d = _holes(x, y, keep)
    if twice:   # every row gets its first value once more, the same one: whichever counts, the row goes the same way
        at = d.row_ptr[:-1]
        d = CsrData(n, f, (d.row_ptr + np.arange(n + 1)).astype(np.int32), np.insert(d.col, at, d.col[at]), np.insert(d.val, at, d.val[at]), d.y)
    _same_as_oracle(orc, d, depth=depth, n_trees=trees, max_num_bin=255, learning_rate=0.5, objective='reg:linear', num_class=1, min_child_weight=0.5)


# blocks of the split search that take one feature or four: features of 64, 65 and 1 bins, none at all, numbers of them that leave a
# block part empty, left-out columns in one of four
@pytest.mark.parametrize('widths,extra', [([64] * 4, {}), ([65, 64, 1], {}), ([2], {}), ([1] * 6 + [200], {}), ([0, 3, 0, 70, 64, 2, 9], {}),
                                          ([2] * 21, dict(column_sampling_rate=0.4, sample_seed=2))])
def test_blocks_of_the_split_search(gpu, orc, widths, extra):
    n, r = 33_000, np.random.default_rng(len(widths))     # (beyond the sizes of a tree per launch)
    x = np.stack([r.integers(1, w + 1, n) if w else np.ones(n) for w in widths], 1).astype(np.float32)
    keep = r.random(x.shape) < np.where(np.array(widths) > 0, 0.85, 0.0)
    y = x @ r.normal(size=len(widths)) + keep[:, 0] + r.random(n)
    _same_as_oracle(orc, _holes(x, y, keep), depth=6, n_trees=2, max_num_bin=255, learning_rate=0.5, objective='reg:linear', num_class=1, **extra)


# columns that exclude each other share a byte of the row-major matrix: groups of one-hot columns, of columns with several bins that
# just fit a byte or do not, an empty column between them, one row that stores two of a group, rows whose columns come unordered
@pytest.mark.parametrize('widths,both,shuffle', [([1] * 60 + [30], False, False), ([85] * 3 + [1] * 50, False, False), ([86] * 3 + [1] * 50, False, True),
                                                 ([5] * 20 + [0] + [5] * 20, False, False), ([2] * 50, True, False)])
@pytest.mark.parametrize('mode', ['exact', 'fp32'])
def test_columns_that_share_a_byte(gpu, orc, widths, both, shuffle, mode):
    from thundergbm_b200.booster import Booster
    n, f, r = 33_000, len(widths) + 2, np.random.default_rng(len(widths))
    x, keep = np.zeros((n, f), np.float32), np.zeros((n, f), bool)
    of = r.choice(np.nonzero(widths)[0], n)           # every row stores one of the group
    row = np.arange(n)
    x[row, of] = 1 + r.integers(0, np.array(widths)[of])
    keep[row, of] = r.random(n) < 0.9
    if both:
        x[7, 3] = x[7, 30] = 1
        keep[7, [3, 30]] = True
    x[:, -2:] = r.integers(1, 200, (n, 2))            # two columns of their own
    keep[:, -2:] = r.random((n, 2)) < 0.8
    d = _holes(x, x[:, -1] / 50 + np.sin(of) + x.sum(1) / 100 + r.random(n), keep)
    in_order = d                                      # (what the oracle expects)
    if shuffle:
        ptr, col, val = d.row_ptr, d.col.copy(), d.val.copy()
        for i in range(0, n, 3):
            col[ptr[i]:ptr[i + 1]], val[ptr[i]:ptr[i + 1]] = d.col[ptr[i]:ptr[i + 1]][::-1], d.val[ptr[i]:ptr[i + 1]][::-1]
        d = CsrData(n, f, ptr, col, val, d.y)
    p = dict(depth=6, n_trees=3, max_num_bin=255, learning_rate=0.5, objective='reg:linear', num_class=1)
    o = orc.train(in_order, hist_mode=int(mode == 'exact'), **p)
    b = Booster(d, hist_mode=mode, **p)
    cut_val, cut_ptr, bins = orc.bin_only(in_order, 255)
    assert np.array_equal(b.bins(), orc.bins_to_dense(in_order, bins, cut_ptr, b.info.fpad))
    b.boost(3)
    if mode == 'exact':
        assert b.trees().tobytes() == o.trees.tobytes() and np.array_equal(b.ypred(), o.ypred)
    root, want = b.trees()[0, 0][0], o.trees[0, 0][0]
    assert root['split_feature_id'] == want['split_feature_id'] and root['split_bid'] == want['split_bid']
    assert np.max(np.abs(b.metrics() - o.metric)) <= 1e-4 * np.max(o.metric)
    b.close()


# binning: full rows with and without 16-byte alignment, groups of 32 with remainders, CSR rows of few and of many values; features
# of 1, 2, 254 and more distinct values, infinities and zeros of either sign
@pytest.mark.parametrize('n,f,holes', [(1, 1, 0), (257, 4, 0), (1000, 33, 0), (300, 64, 0), (16_384, 30, 0.1), (16_385, 67, 0.3), (17_000, 40, 0.6)])
def test_bins(gpu, n, f, holes):
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(n + f)
    x = r.standard_normal((n, f)).astype(np.float32)
    for j, levels in enumerate([1, 2, 253, 254, 255, 256, 600]):
        if j < f:
            x[:, j] = r.integers(0, levels, n) - levels // 2
    if n > 100:
        x[5:9, f - 1] = np.inf, -np.inf, 0.0, -0.0
    keep = r.random((n, f)) >= holes
    d = _holes(x, r.random(n), keep) if holes else _csr(x, r.random(n))
    b = Booster(d, depth=2, n_trees=1, objective='reg:linear', tree_method='hist')
    cut, ptr = b.cuts()
    got = b.bins()
    want = np.full(got.shape, 255, np.uint8)
    for j in range(f):
        c = cut[ptr[j]:ptr[j + 1]]
        if len(c):
            want[:, j] = np.where(keep[:, j], np.minimum(np.searchsorted(c, x[:, j], 'right'), len(c) - 1), 255)
    assert np.array_equal(got, want)
    b.close()


# query groups of one document to more than a block's threads, at the sizes where the sort changes its exchanges; groups of one
# label, and of one document among others of another label (all of them draw it)
@pytest.mark.parametrize('sizes', [[1, 2, 3, 31, 32, 33], [64, 65, 127, 128, 129, 1], [255, 256, 257, 40], [600, 5, 1025], [50] * 40])
@pytest.mark.parametrize('objective', ['rank:ndcg', 'rank:pairwise'])
def test_query_groups(gpu, orc, sizes, objective):
    n, r = sum(sizes), np.random.default_rng(len(sizes))
    x = r.integers(1, 20, (n, 6)).astype(np.float32)
    y = np.minimum(r.poisson(x[:, 0] / 10), 4)
    end = np.cumsum(sizes)
    y[end[-1] - sizes[-1]:] = 1              # the last group: one label ...
    if sizes[-1] > 1:
        y[-1] = 2                            # ... but for one document
    y[end[1] - sizes[1]:end[1]] = 3
    d = _csr(x, y)
    d.group = np.array(sizes, np.int32)
    _same_as_oracle(orc, d, depth=4, n_trees=4, max_num_bin=32, learning_rate=0.3, objective=objective, min_child_weight=0.0)


# NaNs with the sign set are the first cut point of a column, and no value compares above them
@pytest.mark.parametrize('n,f,holes', [(300, 33, 0), (17_000, 40, 0.2)])
def test_bins_of_columns_with_nans(gpu, n, f, holes):
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(f)
    nan = np.copysign(np.float32(np.nan), np.float32(-1))
    x = r.integers(1, 4, (n, f)).astype(np.float32)
    x[:, 0] = 1
    x[::3, :3] = nan
    x[:, 3] = nan
    x[::3, 4] = np.nan
    keep = r.random((n, f)) >= holes
    d = _holes(x, r.random(n), keep) if holes else _csr(x, r.random(n))
    b = Booster(d, depth=2, n_trees=1, objective='reg:linear', tree_method='hist')
    cut, ptr = b.cuts()
    got = b.bins()
    b.close()
    want = np.full(got.shape, 255, np.uint8)
    for j in range(f):
        c = cut[ptr[j]:ptr[j + 1]]
        assert np.isnan(c[0]) == (j < 4)
        lo, hi = np.zeros(n, int), np.full(n, len(c) - 1)
        for _ in range(9):
            mid = (lo + hi) // 2
            up = c[mid] <= x[:, j]
            lo, hi = np.where((lo < hi) & up, mid + 1, lo), np.where((lo < hi) & ~up, mid, hi)
        want[:, j] = np.where(keep[:, j], lo, 255)
    assert np.array_equal(got, want)


# a row that stores a column twice: the last value counts, whether a thread walks the row or the lanes of a warp share it.  Columns
# that ascend but for the repeats, in any order, and repeats a window of lanes or more apart
@pytest.mark.parametrize('n,f,per', [(3000, 40, 30), (16_384, 40, 30), (16_385, 218, 70), (17_000, 3, 100)])
@pytest.mark.parametrize('order', ['sorted', 'any', 'apart'])
def test_columns_stored_twice(gpu, n, f, per, order):
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(n + f)
    col = r.integers(0, f, (n, per))
    if order != 'any':
        col.sort(1)
        col[::2] = np.arange(per) * f // per     # (every other row: no repeats where it has no more values than there are columns)
    if order == 'apart':
        col[:, -1] = col[:, 0]
        col[1::3, per // 2] = col[1::3, 0]
    x = r.integers(1, 200, (n, per)).astype(np.float32)
    d = CsrData(n, f, (np.arange(n + 1) * per).astype(np.int32), col.astype(np.int32).ravel(), x.ravel(), r.random(n).astype(np.float32))
    b = Booster(d, depth=2, n_trees=1, objective='reg:linear', tree_method='hist')
    cut, ptr = b.cuts()
    got = b.bins()
    b.close()
    want = np.full(got.shape, 255, np.uint8)
    row = np.arange(n)
    for k in range(per):     # one value after the other
        c = col[:, k]
        for j in np.unique(c):
            at, cuts = row[c == j], cut[ptr[j]:ptr[j + 1]]
            want[at, j] = np.minimum(np.searchsorted(cuts, x[at, k], 'right'), len(cuts) - 1)
    assert np.array_equal(got, want)



def _trained_in(d, spare, rounds, **p):
    """Trees and scores of a training that finds `spare` bytes of free device memory (0: all there is)."""
    import torch
    from thundergbm_b200 import _lib
    from thundergbm_b200.booster import Booster
    _lib.lib().tgbm_release_device_memory()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - spare, dtype=torch.uint8, device='cuda') if spare else None
    b = Booster(d, n_trees=rounds, hist_mode='exact', objective='reg:linear', **p)
    b.boost(rounds)
    got = b.trees().tobytes(), b.ypred().tobytes()
    b.close()
    del filler
    torch.cuda.empty_cache()
    return got


# the values by column (240 MB that stay, 360 more while they are sorted) only where the level buffers (1.6 GB) leave room for them
def test_columns_of_the_csr_layout_in_little_memory(gpu):
    r = np.random.default_rng(1)
    n, per, f = 750_000, 40, 20_000
    col = (np.arange(per) * (f // per) + r.integers(0, f // per, (n, per))).astype(np.int32)
    d = CsrData(n, f, np.arange(0, n * per + 1, per, dtype=np.int32), col.ravel(), np.ones(n * per, np.float32), (col[:, 0] % 5 + r.random(n)).astype(np.float32))
    assert _trained_in(d, 0, 12, depth=12) == _trained_in(d, 1850 << 20, 12, depth=12)


# the bytes by slot (224 MB here) beside those by feature (twice 256 MB) only where there is room for them
def test_columns_that_share_a_byte_in_little_memory(gpu):
    r = np.random.default_rng(1)
    n, f = 1_000_000, 256
    a, b = r.integers(40, f, n), r.integers(40, f - 1, n)
    b += b >= a
    col = np.stack([r.integers(0, 40, n), np.minimum(a, b), np.maximum(a, b)], 1).astype(np.int32)   # forty exclude each other
    d = CsrData(n, f, np.arange(0, 3 * n + 1, 3, dtype=np.int32), col.ravel(), r.integers(1, 4, 3 * n).astype(np.float32),
                (col[:, 0] % 5 + r.random(n)).astype(np.float32))
    assert _trained_in(d, 0, 2, depth=4) == _trained_in(d, 640 << 20, 2, depth=4)


# shared memory that the kernels may ask for grows with the depth and, for ranking, with the longest query group: it is allowed to a
# kernel, not to a booster, so a booster made in between must not take away what another one needs
@pytest.mark.parametrize('layout,n,deep,shallow', [('dense', 33_000, 9, 2), ('dense', 33_000, 14, 12), ('dense', 33_000, 11, 10), ('sparse', 3000, 9, 2)])
def test_boosters_of_different_depths_side_by_side(gpu, orc, monkeypatch, layout, n, deep, shallow):
    from thundergbm_b200.booster import Booster
    monkeypatch.setenv('TGBM_LAYOUT', layout)
    d = _data(n, 4, 1, deep)
    for mode in ('exact', 'fp32'):
        p = [dict(depth=x, n_trees=2, max_num_bin=64, learning_rate=0.5, objective='reg:linear') for x in (deep, shallow)]
        b = [Booster(d, hist_mode=mode, **q) for q in p]
        for x, q in zip(b, p):
            x.boost(2)
            if mode == 'exact':
                o = orc.train(d, hist_mode=1, keep_nid=0, **q)
                assert x.trees().tobytes() == o.trees.tobytes() and np.array_equal(x.ypred(), o.ypred)
            assert x.info.rounds_done == 2 and np.isfinite(x.metrics()).all()
            x.close()


def test_rankings_of_different_group_sizes_side_by_side(gpu, orc):
    from thundergbm_b200.booster import Booster
    r = np.random.default_rng(4)
    p = dict(depth=3, n_trees=2, max_num_bin=32, learning_rate=0.5, objective='rank:ndcg')
    data = []
    for longest in (4096, 1300):
        d = _csr(r.integers(1, 20, (longest + 9, 3)), r.integers(0, 4, longest + 9))
        d.group = np.array([9, longest], np.int32)
        data.append(d)
    b = [Booster(d, hist_mode='exact', **p) for d in data]
    for x, d in zip(b, data):
        x.boost(2)
        assert x.trees().tobytes() == orc.train(d, hist_mode=1, keep_nid=0, **p).trees.tobytes()
        x.close()


def _profiled(d, rounds, **p):
    from thundergbm_b200.booster import Booster
    b = Booster(d, n_trees=rounds, objective='reg:linear', **p)
    b.set_profile(True)
    b.boost(rounds)
    got = b.profile()
    b.close()
    return got


# what the counters call the bytes of a row: one per column, or per group of columns that share it
def test_bytes_of_the_profile(gpu):
    n, r = 40_000, np.random.default_rng(2)
    x, keep = np.zeros((n, 62), np.float32), np.zeros((n, 62), bool)
    of = r.integers(0, 60, n)
    x[np.arange(n), of] = 1
    keep[np.arange(n), of] = True
    x[:, 60:] = r.integers(1, 200, (n, 2))
    keep[:, 60:] = True
    d = _holes(x, of % 7 + r.random(n), keep)
    assert _profiled(d, 2, depth=3).hist_root_bytes == 2 * n * (3 + 8)          # sixty share one, two have their own
    assert _profiled(_csr(x[:, 55:], d.y), 2, depth=3).hist_root_bytes == 2 * n * (7 + 8)


# launches that move rows: one a level but the last; two, and a third for many children, in float rounds; of the CSR layout with its
# values by column one more at every level
@pytest.mark.parametrize('layout,mode,trees,each', [('dense', 'exact', 10, [1, 1, 1, 0]), ('dense', 'fp32', 1, [2, 2, 2, 0]), ('sparse', 'exact', 9, [1, 1, 1, 0]),
                                                    ('sparse', 'exact', 10, [2, 2, 2, 1])])
def test_launches_of_the_profile(gpu, monkeypatch, layout, mode, trees, each):
    monkeypatch.setenv('TGBM_LAYOUT', layout)
    got = _profiled(_data(33_000, 5, 1, 3), trees, depth=4, hist_mode=mode)
    assert got.partition_launches == trees * sum(each) and got.partition_ms > 0 and got.kernel_launches > got.partition_launches + got.hist_launches
