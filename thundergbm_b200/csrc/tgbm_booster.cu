// Host orchestration of the boosting loop: every launch of a round is queued on one stream and
// nothing in boost() waits for the device, so the level loop never round-trips through the host
// (the reference synchronises after every launch, include/thundergbm/util/device_lambda.cuh:49).
#include "tgbm_booster.h"

#include <cub/cub.cuh>
#include <cub/device/device_merge.cuh>
#include <cuda/std/functional>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <cstring>

#include "tgbm_input.h"
#include "tgbm_kernels.cuh"
#include "tgbm_level.cuh"
#include "tgbm_hist_f32.cuh"
#include "tgbm_small.cuh"
#include "tgbm_exact.cuh"
#include "tgbm_rank.cuh"

namespace tgbm {

struct BoosterImpl {
    GBMParam p;
    const Comm *comm = nullptr;
    cudaStream_t stream = nullptr;
    int objective = REG_LINEAR;
    int N = 0, F = 0, Fpad = 0, B = 0, K = 1, n_nodes = 0, depth = 0;
    long long N_global = 0;
    long long row_offset = 0;  // global id of local row 0
    size_t Npad = 0;
    int num_class = 1;
    float base_score = 0;
    int rounds = 0;
    int num_sms = 148;
    int window_rows = 0;
    bool profile_on = false;

    std::vector<float> h_cut_val;
    std::vector<int> h_cut_ptr;
    std::vector<float> label;

    DeviceRows in;   // the stored values on the device, held from upload_rows() to the end of binning
    DevBuf<unsigned char> bins, binsT;
    // slots of `bins`: features, or neighbouring ones that share a byte (k_last_before)
    int S = 0, Spad = 0;
    std::vector<int> h_slot_ptr;   // first bin of every slot
    DevBuf<int> slot_ptr;
    void bundle_columns();
    // wide sparse data: CSR of global bin ids instead of the two dense matrices
    bool sparse = false;
    long long nnz_local = 0;
    DevBuf<int> sp_row_ptr, sp_bin, chunk_bin0;
    DevBuf<int> col_row, col_bin, col_ptr;   // the same values by column (SparseColumns)
    SparseColumns columns() const { return SparseColumns{col_row.p, col_bin.p, col_ptr.p}; }
    void sort_columns();
    int n_chunks = 0;
    DevBuf<float> cut_val, y, ypred, metric;
    DevBuf<int> cut_ptr, cut_fid;
    DevBuf<float2> gh;
    DevBuf<int2> ghq;
    DevBuf<unsigned> maxbits;
    DevBuf<unsigned long long> root_sum;
    DevBuf<QuantInfo> qinfo, qinfo_log;
    DevBuf<TreeNode> nodes, model;
    // the trees of a round are built in batches of `batch` (see Batch): one tree's share of the buffers below lies a
    // stride behind the one before
    int batch = 1;
    Batch bufs{};
    DevBuf<int> rec_idx;
    DevBuf<unsigned short> nid;
    DevBuf<int> seg_begin[2], seg_cnt[2], origin[2];
    DevBuf<float> leaf_weight;
    DevBuf<AssignRule> leaf_rule;
    DevBuf<int> nid_keep;
    DevBuf<long long> hist_full, hist_built;
    // fp32 mode: the same two buffers hold float pairs; `hist_spread` receives the built histograms, their cells
    // `f32_stride(pairs)` float2 apart (see tgbm_hist_f32.cuh)
    bool f32 = false;
    // the round sums floats value by value; fp32 mode's later rounds sum integers on a grid of FINE_BITS bits
    bool float_round(int round) const { return f32 && (exact || round < FINE_FROM_ROUND || force_float); }
    bool force_float = false;  // the round's gradients do not fit the grid (settle)
    bool last_float = false;   // hist_full holds float pairs
    size_t last_tree_full = 0; // where the histograms of the tree built last start in it
    DevBuf<float2> hist_spread;
    DevBuf<double> sum_partial;
    CutOffsets f32_cuts{};                 // fp32 dense kernel: first bin of every feature, passed by value
    bool f32_staged = true;                // fp32 dense kernel, gather levels: record tiles staged by bulk copies
    DevBuf<int> bag_count;                 // bagging: multiplicity of every gradient entry in the round's bootstrap sample
    DevBuf<unsigned char> ignored_all;     // column sampling: [round][feature] mask of the features left out
    // Distance of two cells of a built histogram, in cells: 32 (one 8-byte cell per 256 bytes) wherever the spread
    // buffer has room.  The L2 performs reductions to cells that share a line one after the other: a microbenchmark of
    // the bare reductions (10.5 M rows x 28) runs at 87 / 165 / 176 / 190 / 165 G/s with 8 / 64 / 128 / 256 / 512 bytes
    // between the cells of one node, and the whole boosting round got 13 % shorter going from 64 to 256 bytes.
    size_t spread_cells = 0;   // float2 cells of hist_spread
    int f32_stride(int pairs) const {
        int s = 32;
        while (s > 1 && (size_t)s * pairs * std::max(B, 1) > spread_cells) s >>= 1;
        return s;
    }
    bool prune_in_smem = true;
    TreeCtl stat_base{};  // counters of `ctl` when profiling was switched on
    DevBuf<RoundState> rstate;          // device copy of `rounds`
    cudaGraph_t round_graph = nullptr;  // one boosting round (gradients, K trees, metric) as captured in its steady state
    cudaGraphExec_t round_exec = nullptr;
    long long round_graph_launches = 0;
    bool graphs_allowed = true;
    void run_round(int round);
    void queue_round(int round);   // its launches one by one
    void wait() const;
    bool settle();
    DevBuf<int4> eval_items;  // k_eval: features a block each, or four of few bins (n_eval_items = 0: all a block each)
    int n_eval_items = 0;
    DevBuf<int> eval_ticket;  // k_eval: finished blocks per sibling pair, zero between launches
    int assign_ctas = 1, assign_rpt = 4;
    DevBuf<int> assign_table;   // float rounds: rows per block and child
    auto assign_kernel(int level, bool ordered) const {
        auto pick = [&](auto many, auto k0, auto k1, auto k2) { return level == 0 ? k0 : level == 1 ? k1 : level == 2 ? k2 : many; };
        if (ordered && sparse) return pick(k_assign<true, 4, 0, true>, k_assign<true, 4, 1, true>, k_assign<true, 4, 2, true>, k_assign<true, 4, 3, true>);
        if (ordered) return pick(k_assign<false, 4, 0, true>, k_assign<false, 4, 1, true>, k_assign<false, 4, 2, true>, k_assign<false, 4, 3, true>);
        if (sparse) return pick(k_assign<true, 4, 0, false>, k_assign<true, 4, 1, false>, k_assign<true, 4, 2, false>, k_assign<true, 4, 3, false>);
        if (assign_rpt == 8) return pick(k_assign<false, 8, 0, false>, k_assign<false, 8, 1, false>, k_assign<false, 8, 2, false>, k_assign<false, 8, 3, false>);
        return pick(k_assign<false, 4, 0, false>, k_assign<false, 4, 1, false>, k_assign<false, 4, 2, false>, k_assign<false, 4, 3, false>);
    }
    bool grad_max_ready = false;        // maxbits holds the maxima of the next round's gradients
    bool metric_partial_ready = false;  // metric_partial holds the finished round's partial sums
    int metric_blocks() const { return std::max(1, std::min((N + 255) / 256, std::min(num_sms * 8, METRIC_PARTS))); }   // of 256 threads: one full wave
    DevBuf<SplitRec> recs;
    DevBuf<TreeCtl> ctl;
    DevBuf<double> metric_partial, metric_sum;
    RankState rank;

    struct TimedEvent { cudaEvent_t a, b; int kind; long long launches; };
    std::vector<TimedEvent> events;
    HistProfile profile_acc;  // kernel times of the events already read and destroyed
    long long launches = 0;

    ~BoosterImpl() {
        if (stream) cudaStreamSynchronize(stream);    // nothing of this booster is in flight when its buffers go
        for (auto &e : events) { cudaEventDestroy(e.a); cudaEventDestroy(e.b); }
        if (round_exec) cudaGraphExecDestroy(round_exec);
        if (round_graph) cudaGraphDestroy(round_graph);
        if (stream) cudaStreamDestroy(stream);
    }

    // ---------------------------------------------------------------- init helpers
    void upload_rows(const DataSet &ds);
    void find_cuts_and_bins(const DataSet &ds);
    // tree_method = exact (tgbm_exact.cuh)
    bool exact = false;
    long long ex_nnz = 0;
    // stored values by column, largest first ([0]), and grouped by (column, node) at the levels below the root (two in turn)
    DevBuf<unsigned> ex_key[3];
    DevBuf<int> ex_row[3];
    DevBuf<float> ex_val[3];
    DevBuf<unsigned char> ex_pre, ex_tile_pre, ex_run;   // prefix sums: see k_exact_sum; ex_run: sums and prefixes of the blocks' runs
    DevBuf<unsigned> ex_lr;
    DevBuf<ExPair<int>> ex_tile_lr, ex_run_lr;
    DevBuf<int2> ex_group, ex_gh[3];                // (group ranges; gradient pairs of the entries, float or quantised)
    DevBuf<uint2> ex_side;
    DevBuf<int> ex_live, ex_nid, ex_any, ex_ticket;   // ex_live[level]: entries of the level
    DevBuf<unsigned long long> ex_best;
    void init_exact();
    template <typename T> void exact_levels(int k, const void *gh_rows);
    void build_tree_exact(int round, int k);
    void column_builder_candidates(DevBuf<unsigned long long> &ukeys, DevBuf<long long> &ucopies, long long &nu);
    void init_base_score();
    void gradient(int round);
    void build_trees(int round, int k0, int n_trees);
    SmallPlan small{};   // cluster > 0: trees of integer rounds are built by k_small_tree
    auto small_kernel() const { return N <= SMALL_LOCAL ? k_small_tree<true> : k_small_tree<false>; }
    void plan_small_trees();
    void launch_small_trees(int k0, int n_trees);
    void round_metric(int round);
};

static inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }
constexpr size_t PRUNE_SMEM = 200 * 1024;   // node tables that k_prune holds in shared memory
// shared memory of k_assign at a level: rules, counts, offsets (up to depth 13: 32 bytes per node), staged rows
static inline size_t assign_smem(int level, int rpt) {
    const size_t nl = (size_t)1 << level;
    return sizeof(ChunkRule) * (nl + 1) + sizeof(unsigned) * ASSIGN_THREADS * rpt + 3 * sizeof(int) * (2 * nl + 1);
}

void BoosterImpl::upload_rows(const DataSet &ds) {
    // fewer threads per rank when the ranks of one process upload side by side
    in.upload(ds, stream, num_sms, comm && comm->active() ? std::max(1, upload_threads() / comm->world) : upload_threads());
    nnz_local = (long long)in.nnz;
    // the largest column gives the feature count when the caller did not count (dataset.cpp:54-57), a negative one would
    // send the binning kernels out of bounds
    TGBM_CHECK(in.min_col >= 0, "negative column index in the CSR input");
    if (F < 0) F = std::max(1, in.max_col + 1);
    else TGBM_CHECK(in.max_col < F, "column index beyond the feature count");
}

// ------------------------------------------------------------------------------------------------
// Cut-point candidates of the reference's column-sharded builder (HistCut::get_cut_points3 + unique_by_flag,
// src/thundergbm/hist_cut.cu:104-187, run by each of its `column_shards` devices on the columns
// SparseColumns::csr2csc_gpu gives it, src/thundergbm/sparse_columns.cu:95-102).  In: the distinct (feature, value)
// keys in ascending order with their multiplicities.  Out: per feature the candidates, largest first, as keys
// (feature, complement of the value's ordered image), from which the usual stride selection picks the cut points.
void BoosterImpl::column_builder_candidates(DevBuf<unsigned long long> &ukeys, DevBuf<long long> &ucopies, long long &nu) {
    if (nu == 0) return;
    const int D = p.column_shards;
    const int grid = std::min(ceil_div(nu, 256), num_sms * 16);
    // copies before every key, per feature the largest value and the copies before its first key
    DevBuf<long long> before, ustart, fbefore;
    DevBuf<float> fmax;
    before.alloc(nu + 1); ustart.alloc(F + 1); fbefore.alloc(F + 1); fmax.alloc(F);
    TGBM_CUDA(cudaMemsetAsync(ucopies.p + nu, 0, sizeof(long long), stream));
    auto scan = [&](const long long *in, long long *out, long long n) {
        size_t tb = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, n, stream);
        DevBuf<unsigned char> tmp;
        tmp.alloc(std::max<size_t>(tb, 1));
        cub::DeviceScan::ExclusiveSum(tmp.p, tb, in, out, n, stream);
        TGBM_CUDA(cudaStreamSynchronize(stream));
    };
    scan(ucopies.p, before.p, nu + 1);
    long long total = 0;
    TGBM_CUDA(cudaMemcpyAsync(&total, before.p + nu, sizeof(long long), cudaMemcpyDeviceToHost, stream));
    k_feature_bounds<<<ceil_div(F + 1, 128), 128, 0, stream>>>(ukeys.p, nu, F, ustart.p);
    TGBM_CUDA(cudaStreamSynchronize(stream));
    k_feature_max_before<<<ceil_div(F + 1, 128), 128, 0, stream>>>(ukeys.p, ustart.p, before.p, nu, total, F, fmax.p, fbefore.p);
    std::vector<float> h_fmax(F);
    std::vector<long long> h_fbefore(F + 1);
    TGBM_CUDA(cudaMemcpyAsync(h_fmax.data(), fmax.p, sizeof(float) * F, cudaMemcpyDeviceToHost, stream));
    TGBM_CUDA(cudaMemcpyAsync(h_fbefore.data(), fbefore.p, sizeof(long long) * (F + 1), cudaMemcpyDeviceToHost, stream));
    TGBM_CUDA(cudaStreamSynchronize(stream));
    std::vector<ColumnShift> h_cs(F);
    std::vector<int> h_first(D), h_cols(D);
    std::vector<long long> h_sbefore(D);
    const int ave = F / D;
    for (int d = 0; d < D; ++d) {
        const int first = d * ave, ncol = d < D - 1 ? ave : F - first;
        h_first[d] = first; h_cols[d] = ncol; h_sbefore[d] = h_fbefore[first];
        float m = -INFINITY;
        for (int f = first; f < first + ncol; ++f) m = std::max(m, h_fmax[f]);
        // hist_cut.cu:109: the reference gives up when the shifted values leave the int range
        TGBM_CHECK(!(ncol > 0 && m > -INFINITY) || (double)m + (double)ncol * ((double)m + 1) < 2147483647.0,
                   "feature values too large for the column-sharded builder's value shift");
        for (int f = first; f < first + ncol; ++f)
            h_cs[f] = ColumnShift{d, first, m + 1.0f, h_fbefore[first + ncol] - h_fbefore[f + 1]};
    }
    DevBuf<ColumnShift> cs;
    DevBuf<int> shard_first, shard_cols;
    DevBuf<long long> shard_before;
    cs.alloc(F); shard_first.alloc(D); shard_cols.alloc(D); shard_before.alloc(D);
    TGBM_CUDA(cudaMemcpyAsync(cs.p, h_cs.data(), sizeof(ColumnShift) * F, cudaMemcpyHostToDevice, stream));
    TGBM_CUDA(cudaMemcpyAsync(shard_first.p, h_first.data(), sizeof(int) * D, cudaMemcpyHostToDevice, stream));
    TGBM_CUDA(cudaMemcpyAsync(shard_cols.p, h_cols.data(), sizeof(int) * D, cudaMemcpyHostToDevice, stream));
    TGBM_CUDA(cudaMemcpyAsync(shard_before.p, h_sbefore.data(), sizeof(long long) * D, cudaMemcpyHostToDevice, stream));
    // shift, sort per device (descending t), copies before every entry of the sorted array
    DevBuf<unsigned long long> k1, k2;
    DevBuf<long long> c2;
    k1.alloc(nu); k2.alloc(nu); c2.alloc(nu + 1);
    k_shift_keys<<<grid, 256, 0, stream>>>(ukeys.p, nu, cs.p, k1.p);
    {
        int end_bit = 32;
        while ((1ll << (end_bit - 32)) < D && end_bit < 64) ++end_bit;
        size_t tb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, k1.p, k2.p, ucopies.p, c2.p, nu, 0, end_bit, stream);
        DevBuf<unsigned char> tmp;
        tmp.alloc(std::max<size_t>(tb, 1));
        cub::DeviceRadixSort::SortPairs(tmp.p, tb, k1.p, k2.p, ucopies.p, c2.p, nu, 0, end_bit, stream);
        TGBM_CUDA(cudaStreamSynchronize(stream));
    }
    scan(c2.p, before.p, nu);
    DevBuf<unsigned long long> n_heads;
    n_heads.alloc(1);
    n_heads.zero(stream);
    k_unshift_keys<<<grid, 256, 0, stream>>>(k2.p, before.p, nu, cs.p, shard_first.p, shard_cols.p, shard_before.p,
                                             k1.p, n_heads.p);
    unsigned long long h_heads = 0;
    TGBM_CUDA(cudaMemcpyAsync(&h_heads, n_heads.p, sizeof(h_heads), cudaMemcpyDeviceToHost, stream));
    {
        size_t tb = 0;
        cub::DeviceRadixSort::SortKeys(nullptr, tb, k1.p, k2.p, nu, 0, 64, stream);
        DevBuf<unsigned char> tmp;
        tmp.alloc(std::max<size_t>(tb, 1));
        cub::DeviceRadixSort::SortKeys(tmp.p, tb, k1.p, k2.p, nu, 0, 64, stream);
        TGBM_CUDA(cudaStreamSynchronize(stream));
    }
    nu = (long long)h_heads;
    ukeys.alloc(std::max<long long>(nu, 1));
    if (nu) TGBM_CUDA(cudaMemcpyAsync(ukeys.p, k2.p, sizeof(unsigned long long) * nu, cudaMemcpyDeviceToDevice, stream));
    TGBM_CUDA(cudaStreamSynchronize(stream));
}

// ------------------------------------------------------------------------------------------------
// Cut points (HistCut::get_cut_points_single, src/thundergbm/hist_cut.cu:205-286) and the bin matrix.
// Radix sort of (feature, value) keys and DeviceSelect::Unique come from CUB; this runs once, before
// the boosting loop.  With several ranks every rank contributes its sorted distinct keys, all ranks merge the lists and
// derive identical cut points from the union, so the bins equal the single-GPU ones.
// A matrix without missing values is sorted column by column from BY_COLUMN_ROWS rows on: below, the launches of one sort
// per column cost more than the shorter keys save.  28 columns of 1.05 / 2.1 / 10.5 M rows: 1.9 / 2.8 / 9.1 ms, as one sort
// of 64-bit keys 1.7 / 3.4 / 16.6 ms.
constexpr int BY_COLUMN_ROWS = 1 << 21;
constexpr int SORT_LANES = 4;   // columns sorted side by side
// CSR rows binned by k_bin_rows: from so many rows on laying out the search trees of all columns pays, from so many values a row
// a warp per row (300 k rows x 136: 1.3 ms with a thread per row, 0.2 so; 581 k rows x 12 values: 0.09 against 0.16)
constexpr int BIN_ROWS_FROM = 16384, BIN_ROWS_VALUES = 24;
// CSR layout: trees from which on sorting the values by column pays.  What it takes, ms, and saves per tree, us: 1 M rows x 30 of
// 100 k columns of very different popularity 1.05 and 240, 100 k rows 0.19 and 30; columns alike, 40 values of 5 k columns in 200 k
// rows 0.38 and 27, of 10 k in 20 k rows 0.14 and 46; 12 distinct values, 20 of 1 k columns in 500 k rows 0.29 and 27.  Even after 3 to
// 16 trees, then; a training of ten is between 6 % faster and 2 % slower.
constexpr int COLUMNS_TREES = 10;

// streams that start after what `main` holds now; join() makes `main` wait for them
struct SideStreams {
    std::vector<cudaStream_t> st;
    cudaStream_t main;
    cudaEvent_t ev = nullptr;
    SideStreams(cudaStream_t m, int n) : main(m) {
        TGBM_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        TGBM_CUDA(cudaEventRecord(ev, main));
        for (int i = 0; i < n; ++i) {
            cudaStream_t s = nullptr;
            TGBM_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
            st.push_back(s);
            TGBM_CUDA(cudaStreamWaitEvent(s, ev, 0));
        }
    }
    void join() {
        for (cudaStream_t s : st) {
            TGBM_CUDA(cudaEventRecord(ev, s));
            TGBM_CUDA(cudaStreamWaitEvent(main, ev, 0));
        }
    }
    ~SideStreams() {
        for (cudaStream_t s : st) { cudaStreamSynchronize(s); cudaStreamDestroy(s); }
        if (ev) cudaEventDestroy(ev);
    }
};

// Fewer bytes per row for the histogram kernels, which take 32 slots of a row at a time whatever they hold: used where whole
// groups of 32 go.  (581 k rows x 54 columns, 44 of them two one-hot groups: 12 slots.)  The matrix by feature stays where there is
// no memory for another one beside it.
void BoosterImpl::bundle_columns() {
    S = F; Spad = Fpad;
    h_slot_ptr = h_cut_ptr;
    // (a full matrix has no two columns that exclude each other; up to SMALL_ROWS the trees are mostly built without these rows)
    if (in.full_cols == F || Fpad == 32 || F > 8192 || N <= SMALL_ROWS) return;
    DevBuf<int> last;
    last.alloc(F);
    TGBM_CUDA(cudaMemsetAsync(last.p, 0xff, sizeof(int) * F, stream));
    k_last_before<<<std::min(ceil_div(N, 256), num_sms * 4), 256, sizeof(int) * F, stream>>>(bins.p, N, Fpad, F, last.p);
    std::vector<int> h_last(F), slot(F), shift(F), ptr;
    TGBM_CUDA(cudaMemcpyAsync(h_last.data(), last.p, sizeof(int) * F, cudaMemcpyDeviceToHost, stream));
    TGBM_CUDA(cudaStreamSynchronize(stream));
    int a = -1;   // first feature of the running slot
    for (int f = 0; f < F; ++f) {
        if (a < 0 || h_last[f] >= a || h_cut_ptr[f + 1] - h_cut_ptr[a] > MISSING_BIN) { a = f; ptr.push_back(h_cut_ptr[f]); }
        slot[f] = (int)ptr.size() - 1;
        shift[f] = h_cut_ptr[f] - h_cut_ptr[a];
    }
    const int slots = (int)ptr.size(), pad = (slots + 31) / 32 * 32;
    if (pad == Fpad) return;
    ptr.push_back(B);
    DevBuf<int> d_slot, d_shift;
    DevBuf<unsigned char> packed;
    try {
        d_slot.alloc(F); d_shift.alloc(F); slot_ptr.alloc(slots + 1); packed.alloc((size_t)N * pad);
    } catch (const Error &) {
        slot_ptr.release();
        return;
    }
    TGBM_CUDA(cudaMemcpyAsync(d_slot.p, slot.data(), sizeof(int) * F, cudaMemcpyHostToDevice, stream));
    TGBM_CUDA(cudaMemcpyAsync(d_shift.p, shift.data(), sizeof(int) * F, cudaMemcpyHostToDevice, stream));
    TGBM_CUDA(cudaMemcpyAsync(slot_ptr.p, ptr.data(), sizeof(int) * ptr.size(), cudaMemcpyHostToDevice, stream));
    TGBM_CUDA(cudaMemsetAsync(packed.p, MISSING_BIN, packed.bytes(), stream));
    k_bundle<<<std::min(ceil_div(N, 256), num_sms * 8), 256, 0, stream>>>(bins.p, N, Fpad, F, d_slot.p, d_shift.p, pad, packed.p);
    TGBM_CUDA(cudaStreamSynchronize(stream));
    bins.take(packed);
    S = slots; Spad = pad;
    h_slot_ptr = ptr;
}

// The stored values of the CSR layout once more by column, for the kernels that look for the rows of a column: one sort by bin
// id, the rows stay in order.  Not where a row stores a column twice (which of its values counts is up to the search then), and
// only in memory that nothing else wants: after all that a training cannot do without, and beyond 512 MB within an eighth of what is
// free (asking takes 0.4 ms).
void BoosterImpl::sort_columns() {
    const size_t nnz = (size_t)nnz_local, kept = sizeof(int) * (2 * nnz + (size_t)B + 1);
    if (!nnz || nnz >= ((size_t)1 << 31)) return;
    if (kept > ((size_t)512 << 20)) {
        size_t free_bytes = 0, all_bytes = 0;
        TGBM_CUDA(cudaMemGetInfo(&free_bytes, &all_bytes));
        if (kept > free_bytes / 8) return;
    }
    const int grid = std::min(ceil_div(N, 8), num_sms * 16);
    DevBuf<int> twice, rows;
    twice.alloc(1);
    twice.zero(stream);
    k_rows_repeat<<<grid, 256, 0, stream>>>(sp_row_ptr.p, sp_bin.p, cut_fid.p, N, twice.p);
    int h_twice = 0;
    TGBM_CUDA(cudaMemcpyAsync(&h_twice, twice.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
    TGBM_CUDA(cudaStreamSynchronize(stream));
    if (h_twice) return;
    int end_bit = 1;
    while ((1ll << end_bit) < B) ++end_bit;
    size_t tb = 0;
    TGBM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, sp_bin.p, col_bin.p, rows.p, col_row.p, (long long)nnz, 0, end_bit, stream));
    DevBuf<unsigned char> tmp;
    try {
        rows.alloc(nnz); col_row.alloc(nnz); col_bin.alloc(nnz); tmp.alloc(std::max<size_t>(tb, 1)); col_ptr.alloc(B + 1);
    } catch (const Error &) {   // no room for them: the kernels search the rows
        col_row.release(); col_bin.release(); col_ptr.release();
        return;
    }
    k_value_rows<<<grid, 256, 0, stream>>>(sp_row_ptr.p, N, rows.p);
    TGBM_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, sp_bin.p, col_bin.p, rows.p, col_row.p, (long long)nnz, 0, end_bit, stream));
    k_bin_starts<<<std::min(ceil_div(B + 1, 256), num_sms * 8), 256, 0, stream>>>(col_bin.p, (int)nnz, B, col_ptr.p);
    TGBM_CUDA(cudaStreamSynchronize(stream));
}

void BoosterImpl::find_cuts_and_bins(const DataSet &ds) {
    const bool timing = getenv("TGBM_TIMING") != nullptr;  // phase times of the set-up on stderr
    auto t_prev = std::chrono::steady_clock::now();
    auto lap = [&](const char *what) {
        if (!timing) return;
        cudaStreamSynchronize(stream);
        const auto t = std::chrono::steady_clock::now();
        fprintf(stderr, "[tgbm init] %-28s %8.1f ms\n", what, std::chrono::duration<double, std::milli>(t - t_prev).count());
        t_prev = t;
    };
    const size_t nnz = (size_t)nnz_local;
    (void)ds;
    lap("H2D of the rows");
    long long nu = 0;
    DevBuf<unsigned long long> ukeys;
    const bool multi = comm && comm->active();
    std::string local_err;  // see Booster::init: local phases are followed by an agreement of all ranks
    auto agree = [&](const char *what) {
        if (multi) comm->agree(local_err, what, stream);
        else if (!local_err.empty()) throw Error(local_err);
    };
    const bool colb = p.column_shards > 0;   // the column-sharded builder's cut points need the multiplicity of every key
    DevBuf<long long> ucopies;
    std::vector<int> h_stride(F);
    h_cut_ptr.assign(F + 1, 0);
    DevBuf<int> d_stride;
    // strides and numbers of cut points from the number of distinct values of every feature
    auto lay_out_cuts = [&](auto &&distinct) {
        for (int f = 0; f < F; ++f) {
            const long long u = distinct(f), st = u / p.max_num_bin;
            h_stride[f] = (int)st;
            h_cut_ptr[f + 1] = h_cut_ptr[f] + (int)(st == 0 ? u : p.max_num_bin);
        }
        B = h_cut_ptr[F];
        d_stride.alloc(std::max(F, 1));
        cut_ptr.alloc(F + 1); cut_val.alloc(std::max(B, 1)); cut_fid.alloc(std::max(B, 1));
        TGBM_CUDA(cudaMemcpyAsync(d_stride.p, h_stride.data(), sizeof(int) * F, cudaMemcpyHostToDevice, stream));
        TGBM_CUDA(cudaMemcpyAsync(cut_ptr.p, h_cut_ptr.data(), sizeof(int) * (F + 1), cudaMemcpyHostToDevice, stream));
    };
    const bool by_column = in.full_cols > 0 && in.full_cols == F && !multi && !colb && N >= BY_COLUMN_ROWS;
    if (by_column) {
        const int chunks = ceil_div(N, COL_CHUNK);
        DevBuf<unsigned> a, c;
        DevBuf<int> heads, distinct;
        a.alloc(nnz); c.alloc(nnz); heads.alloc((size_t)chunks * F); distinct.alloc(F);
        k_order_columns<<<dim3(ceil_div(N, 64), ceil_div(F, 32)), 256, 0, stream>>>(in.val.p, N, F, a.p);
        size_t tb = 0;
        cub::DoubleBuffer<unsigned> keys(a.p, c.p);
        TGBM_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tb, keys, N, 0, 32, stream));
        tb = (std::max<size_t>(tb, 16) + 255) / 256 * 256;
        DevBuf<unsigned char> tmp;
        tmp.alloc(tb * SORT_LANES);
        int side = 0;
        {
            SideStreams lanes(stream, std::min(F, SORT_LANES));
            for (int f = 0; f < F; ++f) {
                const int q = f % SORT_LANES;
                keys = cub::DoubleBuffer<unsigned>(a.p + (size_t)f * N, c.p + (size_t)f * N);
                TGBM_CUDA(cub::DeviceRadixSort::SortKeys(tmp.p + q * tb, tb, keys, N, 0, 32, lanes.st[q]));
                TGBM_CHECK(f == 0 || keys.selector == side, "sorted columns in different buffers");
                side = keys.selector;
            }
            lanes.join();
        }
        const unsigned *sorted = side ? c.p : a.p;
        k_column_heads<<<dim3(chunks, F), 256, 0, stream>>>(sorted, N, heads.p);
        k_column_prefix<<<F, 1024, 0, stream>>>(heads.p, chunks, distinct.p);
        std::vector<int> h_distinct(F);
        TGBM_CUDA(cudaMemcpyAsync(h_distinct.data(), distinct.p, sizeof(int) * F, cudaMemcpyDeviceToHost, stream));
        TGBM_CUDA(cudaStreamSynchronize(stream));
        lap("columns sorted");
        lay_out_cuts([&](int f) { return (long long)h_distinct[f]; });
        k_column_cuts<<<dim3(chunks, F), 256, 0, stream>>>(sorted, N, heads.p, d_stride.p, cut_ptr.p, p.max_num_bin, cut_val.p, cut_fid.p);
        TGBM_CUDA(cudaStreamSynchronize(stream));
    } else {
        DevBuf<unsigned long long> keys, keys2;
        DevBuf<long long> copies, copies2;
        DevBuf<long long> d_nu;
        DevBuf<long long> counts, mine;
        try {
            keys.alloc(std::max<size_t>(nnz, 1)); keys2.alloc(std::max<size_t>(nnz, 1)); d_nu.alloc(1);
            if (colb) { copies.alloc(std::max<size_t>(nnz, 1)); copies2.alloc(std::max<size_t>(nnz, 1)); }
            if (multi) { counts.alloc(comm->world); mine.alloc(1); }
        } catch (const std::exception &e) { local_err = e.what(); }
        auto sort_unique = [&](size_t n) -> long long {  // keys -> keys (sorted distinct), returns the count
            if (n == 0) return 0;
            size_t tb = 0;
            int end_bit = 32;
            while ((1ll << (end_bit - 32)) < F && end_bit < 64) ++end_bit;
            if (colb) {  // ... and copies -> copies (summed over equal keys)
                cub::DeviceRadixSort::SortPairs(nullptr, tb, keys.p, keys2.p, copies.p, copies2.p, (long long)n, 0, end_bit, stream);
                DevBuf<unsigned char> tmp;
                tmp.alloc(std::max<size_t>(tb, 16));
                cub::DeviceRadixSort::SortPairs(tmp.p, tb, keys.p, keys2.p, copies.p, copies2.p, (long long)n, 0, end_bit, stream);
                size_t tb2 = 0;
                cub::DeviceReduce::ReduceByKey(nullptr, tb2, keys2.p, keys.p, copies2.p, copies.p, d_nu.p, cub::Sum(), (long long)n, stream);
                DevBuf<unsigned char> tmp2;
                tmp2.alloc(std::max<size_t>(tb2, 16));
                cub::DeviceReduce::ReduceByKey(tmp2.p, tb2, keys2.p, keys.p, copies2.p, copies.p, d_nu.p, cub::Sum(), (long long)n, stream);
                long long r = 0;
                TGBM_CUDA(cudaMemcpyAsync(&r, d_nu.p, sizeof(long long), cudaMemcpyDeviceToHost, stream));
                TGBM_CUDA(cudaStreamSynchronize(stream));
                return r;
            }
            cub::DeviceRadixSort::SortKeys(nullptr, tb, keys.p, keys2.p, (long long)n, 0, end_bit, stream);
            DevBuf<unsigned char> tmp;
            tmp.alloc(std::max<size_t>(tb, 16));
            cub::DeviceRadixSort::SortKeys(tmp.p, tb, keys.p, keys2.p, (long long)n, 0, end_bit, stream);
            size_t tb2 = 0;
            cub::DeviceSelect::Unique(nullptr, tb2, keys2.p, keys.p, d_nu.p, (long long)n, stream);
            DevBuf<unsigned char> tmp2;
            tmp2.alloc(std::max<size_t>(tb2, 16));
            cub::DeviceSelect::Unique(tmp2.p, tb2, keys2.p, keys.p, d_nu.p, (long long)n, stream);
            long long r = 0;
            TGBM_CUDA(cudaMemcpyAsync(&r, d_nu.p, sizeof(long long), cudaMemcpyDeviceToHost, stream));
            TGBM_CUDA(cudaStreamSynchronize(stream));
            return r;
        };
        if (local_err.empty()) {
            try {
                if (nnz) k_make_keys<<<std::min(ceil_div(nnz, 256), num_sms * 16), 256, 0, stream>>>(in.val.p, in.col.p, in.full_cols, nnz, keys.p);
                if (nnz && colb) k_fill_ll<<<std::min(ceil_div(nnz, 256), num_sms * 16), 256, 0, stream>>>(copies.p, nnz, 1);
                nu = sort_unique(nnz);
            } catch (const std::exception &e) { local_err = e.what(); }
        }
        agree("sorting its feature values");
        lap("  local sort + unique");
        if (multi) {
            // union of the ranks' distinct keys: all-gather (padded to the largest rank), then merge (or sort) + unique
            TGBM_CUDA(cudaMemcpyAsync(mine.p, &nu, sizeof(long long), cudaMemcpyHostToDevice, stream));
            comm->allgather(mine.p, counts.p, 1, Comm::I64, stream);
            std::vector<long long> hc(comm->world);
            TGBM_CUDA(cudaMemcpyAsync(hc.data(), counts.p, sizeof(long long) * comm->world, cudaMemcpyDeviceToHost, stream));
            comm->wait(stream);
            const long long mx = std::max<long long>(1, *std::max_element(hc.begin(), hc.end()));
            DevBuf<unsigned long long> padded, all;
            DevBuf<long long> padded_c, all_c;
            try {
                padded.alloc(mx); all.alloc((size_t)mx * comm->world);
                if (colb) { padded_c.alloc(mx); all_c.alloc((size_t)mx * comm->world); }
            } catch (const std::exception &e) { local_err = e.what(); }
            agree("making room for the ranks' feature values");
            TGBM_CUDA(cudaMemsetAsync(padded.p, 0xff, sizeof(unsigned long long) * mx, stream));
            if (nu) TGBM_CUDA(cudaMemcpyAsync(padded.p, keys.p, sizeof(unsigned long long) * nu, cudaMemcpyDeviceToDevice, stream));
            comm->allgather(padded.p, all.p, mx, Comm::I64, stream);
            lap("  all-gather of the distinct keys");
            if (colb) {
                TGBM_CUDA(cudaMemsetAsync(padded_c.p, 0, sizeof(long long) * mx, stream));
                if (nu) TGBM_CUDA(cudaMemcpyAsync(padded_c.p, copies.p, sizeof(long long) * nu, cudaMemcpyDeviceToDevice, stream));
                comm->allgather(padded_c.p, all_c.p, mx, Comm::I64, stream);
            }
            long long tot = 0;
            for (long long c : hc) tot += c;
            keys.alloc(std::max<long long>(tot, 1)); keys2.alloc(std::max<long long>(tot, 1));
            if (colb) { copies.alloc(std::max<long long>(tot, 1)); copies2.alloc(std::max<long long>(tot, 1)); }
            if (!colb && tot < INT_MAX) {
                // Every rank's list is sorted: the union is merged pairwise (log2 W passes over the keys) instead of
                // radix-sorted (five passes and a histogram), then made distinct.
                struct Run { const unsigned long long *p; long long n; };
                std::vector<Run> runs;
                for (int r = 0; r < comm->world; ++r)
                    if (hc[r]) runs.push_back({all.p + (size_t)r * mx, hc[r]});
                unsigned long long *bufs[2] = {keys.p, keys2.p};
                int into = 0;
                DevBuf<unsigned char> mtmp;
                while (runs.size() > 1) {
                    std::vector<Run> merged;
                    unsigned long long *out = bufs[into];
                    long long o = 0;
                    for (size_t i = 0; i + 1 < runs.size(); i += 2) {
                        size_t tb = 0;
                        cub::DeviceMerge::MergeKeys(nullptr, tb, runs[i].p, (int)runs[i].n, runs[i + 1].p, (int)runs[i + 1].n, out + o,
                                                    ::cuda::std::less<>{}, stream);
                        if (tb > mtmp.bytes() || !mtmp.p) mtmp.alloc(std::max<size_t>(tb, 16));
                        TGBM_CUDA(cub::DeviceMerge::MergeKeys(mtmp.p, tb, runs[i].p, (int)runs[i].n, runs[i + 1].p, (int)runs[i + 1].n, out + o,
                                                              ::cuda::std::less<>{}, stream));
                        merged.push_back({out + o, runs[i].n + runs[i + 1].n});
                        o += runs[i].n + runs[i + 1].n;
                    }
                    if (runs.size() & 1) {
                        const Run &last = runs.back();
                        TGBM_CUDA(cudaMemcpyAsync(out + o, last.p, sizeof(unsigned long long) * last.n, cudaMemcpyDeviceToDevice, stream));
                        merged.push_back({out + o, last.n});
                    }
                    runs.swap(merged);
                    into ^= 1;
                }
                nu = 0;
                if (!runs.empty()) {
                    size_t tb = 0;
                    cub::DeviceSelect::Unique(nullptr, tb, runs[0].p, bufs[into], d_nu.p, runs[0].n, stream);
                    DevBuf<unsigned char> tmp;
                    tmp.alloc(std::max<size_t>(tb, 16));
                    TGBM_CUDA(cub::DeviceSelect::Unique(tmp.p, tb, runs[0].p, bufs[into], d_nu.p, runs[0].n, stream));
                    TGBM_CUDA(cudaMemcpyAsync(&nu, d_nu.p, sizeof(long long), cudaMemcpyDeviceToHost, stream));
                    TGBM_CUDA(cudaStreamSynchronize(stream));
                    if (into == 1) std::swap(keys.p, keys2.p);   // the distinct keys are expected in `keys`
                }
            } else {
                long long o = 0;
                for (int r = 0; r < comm->world; ++r) {
                    if (hc[r]) TGBM_CUDA(cudaMemcpyAsync(keys.p + o, all.p + (size_t)r * mx, sizeof(unsigned long long) * hc[r], cudaMemcpyDeviceToDevice, stream));
                    if (hc[r] && colb) TGBM_CUDA(cudaMemcpyAsync(copies.p + o, all_c.p + (size_t)r * mx, sizeof(long long) * hc[r], cudaMemcpyDeviceToDevice, stream));
                    o += hc[r];
                }
                nu = sort_unique(tot);
            }
            lap("  union of the ranks' keys");
        }
        ukeys.alloc(std::max<long long>(nu, 1));
        if (nu) TGBM_CUDA(cudaMemcpyAsync(ukeys.p, keys.p, sizeof(unsigned long long) * nu, cudaMemcpyDeviceToDevice, stream));
        if (colb) {
            ucopies.alloc(std::max<long long>(nu, 1) + 1);
            if (nu) TGBM_CUDA(cudaMemcpyAsync(ucopies.p, copies.p, sizeof(long long) * nu, cudaMemcpyDeviceToDevice, stream));
        }
        TGBM_CUDA(cudaStreamSynchronize(stream));
    }
    if (!by_column) {
        if (colb) column_builder_candidates(ukeys, ucopies, nu);
        lap("sort + unique of the keys");
        // distinct values per feature -> stride and number of cut points per feature (host, F+1 numbers)
        DevBuf<long long> ustart;
        ustart.alloc(F + 1);
        k_feature_bounds<<<ceil_div(F + 1, 128), 128, 0, stream>>>(ukeys.p, nu, F, ustart.p);
        std::vector<long long> h_ustart(F + 1);
        TGBM_CUDA(cudaMemcpyAsync(h_ustart.data(), ustart.p, sizeof(long long) * (F + 1), cudaMemcpyDeviceToHost, stream));
        TGBM_CUDA(cudaStreamSynchronize(stream));
        lay_out_cuts([&](int f) { return h_ustart[f + 1] - h_ustart[f]; });
        if (nu) k_select_cuts<<<std::min(ceil_div(nu, 256), num_sms * 16), 256, 0, stream>>>(ukeys.p, nu, ustart.p, d_stride.p, cut_ptr.p,
                                                                                             p.max_num_bin, cut_val.p, cut_fid.p, colb ? 1 : 0);
        TGBM_CUDA(cudaStreamSynchronize(stream));   // the list of start positions goes
    }
    h_cut_val.resize(B);
    TGBM_CUDA(cudaMemcpyAsync(h_cut_val.data(), cut_val.p, sizeof(float) * B, cudaMemcpyDeviceToHost, stream));

    lap("cut point selection");
    // Layout: dense byte matrices (row-major + column-major) unless they would dwarf the data itself -- then the
    // reference's CSR of global bin ids.  TGBM_LAYOUT=dense|sparse overrides the choice (tests).
    {
        const double dense_bytes = 2.0 * (double)N * Fpad, csr_bytes = 4.0 * (double)nnz;
        sparse = F > 256 && dense_bytes > 4.0 * csr_bytes;
        if (const char *e = getenv("TGBM_LAYOUT")) {
            if (!strcmp(e, "sparse")) sparse = true;
            if (!strcmp(e, "dense")) sparse = false;
        }
        TGBM_CHECK(sparse || (long long)F * 32 <= (1 << 21), "the dense bin matrix supports at most 65536 features");
    }
    if (sparse) {
        in.need_csr(N, stream, num_sms);
        sp_row_ptr.alloc(N + 1);
        sp_bin.alloc(std::max<size_t>(nnz, 1));
        TGBM_CUDA(cudaMemcpyAsync(sp_row_ptr.p, in.row_ptr.p, sizeof(int) * (N + 1), cudaMemcpyDeviceToDevice, stream));
        if (nnz) k_bin_csr<<<std::min(ceil_div(nnz, 256), num_sms * 16), 256, 0, stream>>>(in.col.p, in.val.p, nnz, cut_ptr.p, cut_val.p, sp_bin.p, colb ? 1 : 0);
        // rows whose columns arrive unordered are put in ascending bin order (= ascending column order)
        if (nnz) {
            DevBuf<int> unsorted;
            unsorted.alloc(1);
            TGBM_CUDA(cudaMemsetAsync(unsorted.p, 0, sizeof(int), stream));
            k_rows_unsorted<<<std::min(ceil_div(N, 256), num_sms * 16), 256, 0, stream>>>(sp_row_ptr.p, sp_bin.p, N, unsorted.p);
            int h_unsorted = 0;
            TGBM_CUDA(cudaMemcpyAsync(&h_unsorted, unsorted.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
            TGBM_CUDA(cudaStreamSynchronize(stream));
            if (h_unsorted) {
                DevBuf<int> sorted_bin;
                sorted_bin.alloc(nnz);
                size_t tmp_bytes = 0;
                TGBM_CUDA(cub::DeviceSegmentedSort::SortKeys(nullptr, tmp_bytes, sp_bin.p, sorted_bin.p, (long long)nnz, (long long)N, sp_row_ptr.p,
                                                             sp_row_ptr.p + 1, stream));
                DevBuf<unsigned char> tmp;
                tmp.alloc(std::max<size_t>(tmp_bytes, 1));
                TGBM_CUDA(cub::DeviceSegmentedSort::SortKeys(tmp.p, tmp_bytes, sp_bin.p, sorted_bin.p, (long long)nnz, (long long)N, sp_row_ptr.p,
                                                             sp_row_ptr.p + 1, stream));
                TGBM_CUDA(cudaMemcpyAsync(sp_bin.p, sorted_bin.p, sizeof(int) * nnz, cudaMemcpyDeviceToDevice, stream));
                TGBM_CUDA(cudaStreamSynchronize(stream));
            }
        }
        // chunks of whole features with at most 256 bins for the split evaluation
        std::vector<int> cb(1, 0);
        int cur = 0;
        for (int f = 0; f < F; ++f) {
            const int nbf = h_cut_ptr[f + 1] - h_cut_ptr[f];
            if (cur + nbf > 256 && cur > 0) { cb.push_back(h_cut_ptr[f]); cur = 0; }
            cur += nbf;
        }
        if (cb.back() != B) cb.push_back(B);
        n_chunks = (int)cb.size() - 1;
        chunk_bin0.alloc(cb.size());
        TGBM_CUDA(cudaMemcpyAsync(chunk_bin0.p, cb.data(), sizeof(int) * cb.size(), cudaMemcpyHostToDevice, stream));
        TGBM_CUDA(cudaStreamSynchronize(stream));
    } else {
        bins.alloc((size_t)N * Fpad);
        binsT.alloc((size_t)F * Npad + ASSIGN_CHUNK);   // (k_assign reads the first column to the end of a chunk)
        const size_t tree_smem = sizeof(float) * (size_t)F * (BIN_TREE + 1);
        // a cut point that is a NaN with its sign set comes first, and no value is above it: what a search finds then depends on the
        // cut points that it looks at, so those of k_bin_dense decide
        bool ordered = !colb;
        for (int f = 0; f < F; ++f) ordered = ordered && !(h_cut_ptr[f] < h_cut_ptr[f + 1] && std::isnan(h_cut_val[h_cut_ptr[f]]));
        if (N && ordered && in.full_cols == F) {
            auto kern = F % 4 == 0 ? k_bin_full<true> : k_bin_full<false>;
            kern<<<dim3(std::min(ceil_div(N, 256), num_sms * 4), Fpad / 32), 256, 0, stream>>>(in.val.p, N, F, cut_ptr.p, cut_val.p, Fpad, Npad, bins.p, binsT.p);
        } else if (N && ordered && !in.full_cols && tree_smem <= BIN_ROWS_SMEM && N >= BIN_ROWS_FROM && nnz >= BIN_ROWS_VALUES * (size_t)N) {
            allow_shared(k_bin_rows, BIN_ROWS_SMEM);
            TGBM_CUDA(cudaMemsetAsync(bins.p, MISSING_BIN, bins.bytes(), stream));
            k_bin_rows<<<std::min(ceil_div(N, 32), num_sms), 1024, tree_smem, stream>>>(in.row_ptr.p, in.col.p, in.val.p, N, F, cut_ptr.p, cut_val.p, Fpad, bins.p);
            k_bins_by_column<<<dim3((unsigned)(Npad / 128), Fpad / 32), 256, 0, stream>>>(bins.p, N, F, Fpad, Npad, binsT.p);
        } else {
            TGBM_CUDA(cudaMemsetAsync(bins.p, MISSING_BIN, bins.bytes(), stream));
            TGBM_CUDA(cudaMemsetAsync(binsT.p, MISSING_BIN, binsT.bytes(), stream));
            if (N) k_bin_dense<<<ceil_div(N, 128), 128, 0, stream>>>(in.row_ptr.p, in.col.p, in.val.p, in.full_cols, N, cut_ptr.p, cut_val.p, Fpad, Npad, bins.p, binsT.p, colb ? 1 : 0);
        }
        bundle_columns();
    }
    TGBM_CUDA(cudaStreamSynchronize(stream));
    TGBM_CUDA(cudaGetLastError());
    in.release();
    lap("binning");
}

// ------------------------------------------------------------------------------------------------
// Exact builder, set-up: the stored values by column, largest first (SparseColumns::csr2csc_gpu,
// src/thundergbm/sparse_columns.cu:20-93 and :127) -- one stable radix sort of (column, complement of the value's ordered
// image) keys with the row ids as payload -- and the buffers of the level loop, sized once.
void BoosterImpl::init_exact() {
    const size_t nnz = (size_t)nnz_local;
    in.need_csr(N, stream, num_sms);
    ex_nnz = (long long)nnz;
    TGBM_CHECK(nnz < (1ull << 31), "the exact builder indexes stored values with 32 bits");
    TGBM_CHECK((double)F * (double)(1 << std::max(0, depth - 1)) < 4294967295.0, "columns x nodes of the last level must fit 32 bits");
    const size_t n1 = std::max<size_t>(nnz, 1), tiles = (n1 + EX_TILE - 1) / EX_TILE, padded = tiles * EX_TILE;   // whole tiles are loaded
    const int grid = std::max(1, std::min(ceil_div((long long)n1, 256), num_sms * 16));
    {
        DevBuf<unsigned long long> keys, keys2;
        DevBuf<int> rows;
        keys.alloc(n1); keys2.alloc(n1); rows.alloc(n1);
        ex_key[0].alloc(padded); ex_row[0].alloc(padded); ex_val[0].alloc(padded);
        if (N) k_value_rows<<<std::min(ceil_div(N, 8), num_sms * 16), 256, 0, stream>>>(in.row_ptr.p, N, rows.p);
        if (nnz) k_exact_csc_keys<<<grid, 256, 0, stream>>>(in.val.p, in.col.p, nnz, keys.p);
        int end_bit = 32;
        while ((1ll << (end_bit - 32)) < F && end_bit < 64) ++end_bit;
        if (nnz) {
            size_t tb = 0;
            cub::DeviceRadixSort::SortPairs(nullptr, tb, keys.p, keys2.p, rows.p, ex_row[0].p, (long long)nnz, 0, end_bit, stream);
            DevBuf<unsigned char> tmp;
            tmp.alloc(std::max<size_t>(tb, 1));
            TGBM_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, keys.p, keys2.p, rows.p, ex_row[0].p, (long long)nnz, 0, end_bit, stream));
            k_exact_csc_vals<<<grid, 256, 0, stream>>>(keys2.p, nnz, ex_val[0].p, ex_key[0].p);
            TGBM_CUDA(cudaStreamSynchronize(stream));
        }
    }
    in.release();
    // (not before the sort's buffers are gone: with them 2 G stored values would not fit)
    ex_gh[0].alloc(padded);
    for (int i = 1; i < (depth > 1 ? 3 : 1); ++i) { ex_key[i].alloc(padded); ex_row[i].alloc(padded); ex_val[i].alloc(padded); ex_gh[i].alloc(padded); }
    // no cut points, no bin matrix
    B = 0; sparse = false;
    h_cut_ptr.assign(F + 1, 0);
    cut_ptr.alloc(F + 1); cut_val.alloc(1); cut_fid.alloc(1);
    cut_ptr.zero(stream);
    const size_t max_nl = (size_t)1 << std::max(0, depth - 1);
    const size_t v = f32 ? sizeof(double) : sizeof(int), w = 8;
    ex_pre.alloc(2 * v * padded); ex_tile_pre.alloc(2 * w * tiles); ex_run.alloc(2 * 2 * w * num_sms * 8);
    ex_lr.alloc(padded); ex_tile_lr.alloc(tiles); ex_run_lr.alloc(2 * num_sms * 8);
    ex_group.alloc((size_t)F * max_nl + 1);
    ex_live.alloc(depth + 1);
    const int live = (int)nnz;
    TGBM_CUDA(cudaMemcpyAsync(ex_live.p, &live, sizeof(int), cudaMemcpyHostToDevice, stream));
    ex_nid.alloc(std::max(N, 1)); ex_side.alloc(N / 32 + 1);
    ex_best.alloc(max_nl);
    ex_best.zero(stream);
    ex_any.alloc(1);
    ex_any.zero(stream);
    ex_ticket.alloc(1);
    ex_ticket.zero(stream);
    allow_shared(k_exact_gain<float>, 64 * 1024);
    allow_shared(k_exact_gain<long long>, 64 * 1024);
    TGBM_CUDA(cudaStreamSynchronize(stream));
    TGBM_CUDA(cudaGetLastError());
}

// The level loop of one tree with the exact split search (TreeBuilder::build_approximate, tree_builder.cu:147-194, with
// ExactTreeBuilder::find_split / update_ins2node_id).  T = float: the reference's arithmetic; T = long long: sums of the
// quantised gradients, exact in any order.
template <typename T>
void BoosterImpl::exact_levels(int k, const void *gh_rows) {
    typedef typename ExKind<T>::V V;
    typedef typename ExKind<T>::W W;
    TGBM_CUDA(cudaMemsetAsync(ex_nid.p, 0, sizeof(int) * (size_t)std::max(N, 1), stream));
    if (!ex_nnz) return;   // no stored value: the root stays as it is
    const int tiles = std::max(1, ceil_div(ex_nnz, EX_TILE)), grid = std::min(tiles, num_sms * EX_SEARCH_BLOCKS), move_grid = std::min(tiles, num_sms * EX_MOVE_BLOCKS);
    const int row_grid = std::max(1, std::min(ceil_div(std::max(N, 1), 256), num_sms * 8));
    ExPair<V> *pre = reinterpret_cast<ExPair<V> *>(ex_pre.p);
    ExPair<W> *tile_pre = reinterpret_cast<ExPair<W> *>(ex_tile_pre.p), *run_sum = reinterpret_cast<ExPair<W> *>(ex_run.p), *run_pre = run_sum + num_sms * 8;
    ExPair<int> *run_cnt = ex_run_lr.p, *run_lr = ex_run_lr.p + num_sms * 8;
    typedef typename ExKind<T>::In In;
    auto gh_of = [&](int i) { return reinterpret_cast<In *>(ex_gh[i].p); };
    for (int level = 0; level < depth; ++level) {
        const int nl = 1 << level, a = level == 0 ? 0 : 1 + (level & 1), z = 1 + ((level + 1) & 1);   // this level's entries, the next one's
        const int *live = ex_live.p + level;
        launch_after(level == 0 ? k_exact_sum<T, true> : k_exact_sum<T, false>, grid, EX_THREADS, 0, stream, live, ex_key[a].p, ex_row[a].p,
                     static_cast<const In *>(gh_rows), gh_of(a), pre, tile_pre, run_sum, run_pre, ex_group.p, ex_ticket.p);
        const ExSearch<T> x{ex_key[a].p, ex_val[a].p, pre, tile_pre, run_pre, ex_group.p};
        launch_after(k_exact_gain<T>, grid, EX_THREADS, sizeof(unsigned long long) * (size_t)nl, stream, live, x, level, nodes.p, qinfo.p,
                     p.min_child_weight, p.lambda, p.rt_eps, ignored_all.p, rstate.p, F, ex_best.p, ex_any.p, ex_ticket.p);
        const int node_blocks = std::min(nl, 1024);
        launch_after(k_exact_move, dim3(std::max(1, row_grid / node_blocks), node_blocks), 256, 0, stream, ex_row[a].p, ex_val[a].p, ex_group.p, level, ex_nid.p,
                     nodes.p, ex_any.p);
        launch_after(k_exact_move_missing, row_grid, 256, 0, stream, ex_nid.p, N, level, nodes.p, ex_any.p, ex_side.p);
        launches += 4;
        if (level + 1 == depth) break;
        launch_after(k_exact_sides, move_grid, EX_THREADS, 0, stream, live, ex_row[a].p, ex_side.p, ex_lr.p, ex_tile_lr.p, run_cnt, run_lr, ex_live.p + level + 1,
                     ex_ticket.p);
        launch_after(k_exact_scatter<In>, move_grid, EX_THREADS, 0, stream, live, ex_key[a].p, ex_row[a].p, ex_val[a].p, gh_of(a), ex_lr.p, ex_tile_lr.p, run_lr, ex_group.p, ex_key[z].p,
                     ex_row[z].p, ex_val[z].p, gh_of(z));
        launches += 2;
    }
    (void)k;
}

void BoosterImpl::build_tree_exact(int round, int k) {
    const int tree_index = round * K + k;
    k_tree_init<<<ceil_div(n_nodes, 256), 256, 0, stream>>>(nodes.p, n_nodes, root_sum.p + 2 * k, qinfo.p, p.lambda, N,
                                                            seg_begin[0].p, seg_cnt[0].p, bufs.seg_stride, f32 ? 1 : 0, maxbits.p, 0, ctl.p);
    if (f32) exact_levels<float>(k, gh.p + (size_t)k * N);
    else exact_levels<long long>(k, ghq.p + (size_t)k * N);
    k_prune<<<1, 1024, prune_in_smem ? sizeof(TreeNode) * (size_t)n_nodes : 0, stream>>>(nodes.p, n_nodes, depth, p.gamma, prune_in_smem ? 1 : 0, model.p, K, k,
                                                                                         rstate.p, nullptr, nullptr, 0, 0, nullptr, 0, nullptr, nullptr);
    if (N) {
        int *nid_out = p.keep_nid ? nid_keep.p + (size_t)tree_index * N : nullptr;
        k_exact_predict<<<std::min(ceil_div(N, 256), num_sms * 8), 256, 0, stream>>>(ex_nid.p, N, nodes.p, p.learning_rate, ypred.p + (size_t)k * N, nid_out);
    }
    grad_max_ready = metric_partial_ready = false;
    launches += 3;
}

// ------------------------------------------------------------------------------------------------
Booster::Booster(const GBMParam &param, const Comm *comm) : impl_(new BoosterImpl) {
    impl_->p = param;
    impl_->comm = comm;
}
Booster::~Booster() = default;

void Booster::init(const DataSet &ds) {
    BoosterImpl &m = *impl_;
    GBMParam &p = m.p;
    m.objective = objective_from_name(p.objective);
    TGBM_CHECK(m.objective != OBJ_UNKNOWN, "undefined objective " + p.objective);
    TGBM_CHECK(p.depth >= 1 && p.depth <= MAX_DEPTH, "depth must be in [1, " + std::to_string(MAX_DEPTH) + "]");
    TGBM_CHECK(p.max_num_bin >= 1 && p.max_num_bin <= 255, "max_num_bin must be in [1, 255] (bin ids are bytes, 255 marks a missing value)");
    TGBM_CHECK(p.quant_bits >= 8 && p.quant_bits <= 20, "quant_bits must be in [8, 20]");
    TGBM_CHECK(p.hist_mode == 0 || p.hist_mode == 1, "hist_mode must be 0 (fp32) or 1 (exact)");
    m.f32 = p.hist_mode == 0;
    // Every phase that can fail on one rank alone (a check of this rank's input, an allocation) runs under `locally`
    // and is followed by an agreement of all ranks, so that no rank enters a collective its peers will never join.
    const bool multi = m.comm && m.comm->active();
    std::string local_err;
    auto locally = [&](auto &&phase) {
        if (!local_err.empty()) return;
        try { phase(); } catch (const std::exception &e) { local_err = e.what(); }
    };
    auto agree = [&](const char *what) {
        if (multi) m.comm->agree(local_err, what, m.stream);
        else if (!local_err.empty()) throw Error(local_err);
    };
    auto check_rows = [&] { TGBM_CHECK(ds.n_rows <= MAX_HIST_ROWS, "at most " + std::to_string(MAX_HIST_ROWS) + " rows per GPU"); };
    if (p.tree_method == "hist") locally(check_rows);
    if (!multi) agree("");   // (nothing has been allocated; ranks tell each other below)
    TGBM_CHECK(p.column_sampling_rate > 0.f, "column_sampling_rate must be positive");
    int dev = 0;
    TGBM_CUDA(cudaGetDevice(&dev));
    TGBM_CUDA(cudaDeviceGetAttribute(&m.num_sms, cudaDevAttrMultiProcessorCount, dev));
    TGBM_CUDA(cudaStreamCreateWithFlags(&m.stream, cudaStreamNonBlocking));
    m.N = ds.n_rows;
    m.F = ds.n_features;
    m.depth = p.depth;
    m.n_nodes = (1 << (p.depth + 1)) - 1;
    m.label = ds.label;
    // (buffers of the collectives are allocated inside the local phases too: between an agreement and the launch of the
    // collective no rank makes a call that could wait for another device -- cudaMalloc can, once peer access is on)
    DevBuf<long long> mine, all;
    locally([&] {
        if (need_group_file(m.objective)) RankState::validate(ds, m.N);
        m.upload_rows(ds);
        if (p.tree_method == "auto" && m.F <= 20000) check_rows();   // (it will be the histogram builder)
        if (multi) { mine.alloc(3); all.alloc(3 * (size_t)m.comm->world); }
    });
    agree("loading its rows");

    // global row count, this rank's row offset, global feature count, query groups before this rank's
    m.N_global = m.N;
    long long most_rows = m.N;   // of a rank
    m.row_offset = 0;
    long long first_group = 0, total_groups = (long long)ds.group.size();
    if (multi) {
        long long h[3] = {m.N, m.F, (long long)ds.group.size()};
        TGBM_CUDA(cudaMemcpyAsync(mine.p, h, sizeof(h), cudaMemcpyHostToDevice, m.stream));
        m.comm->allgather(mine.p, all.p, 3, Comm::I64, m.stream);
        std::vector<long long> ha(3 * (size_t)m.comm->world);
        TGBM_CUDA(cudaMemcpyAsync(ha.data(), all.p, sizeof(long long) * ha.size(), cudaMemcpyDeviceToHost, m.stream));
        m.comm->wait(m.stream);
        m.N_global = 0;
        total_groups = 0;
        for (int r = 0; r < m.comm->world; ++r) {
            if (r < m.comm->rank) { m.row_offset += ha[3 * r]; first_group += ha[3 * r + 2]; }
            m.N_global += ha[3 * r];
            most_rows = std::max(most_rows, ha[3 * r]);
            m.F = std::max<int>(m.F, (int)ha[3 * r + 1]);
            total_groups += ha[3 * r + 2];
        }
    }
    TGBM_CHECK(m.N_global < (1ll << 31), "row count must fit 32 bits");
    TGBM_CHECK(m.F >= 1, "data set has no features");
    m.Fpad = (m.F + 31) / 32 * 32;
    m.Npad = ((size_t)m.N + 127) / 128 * 128;

    // number of classes / trees per round (src/thundergbm/trainer.cu:26-37)
    m.K = 1;
    if (need_group_label(m.objective)) {
        p.num_class = (int)ds.label.size();
        if (p.num_class > 2) m.K = p.num_class;
    } else if (m.objective == REG_LINEAR || m.objective == REG_LOGISTIC) {
        p.num_class = 1;
    }
    p.tree_per_rounds = m.K;
    // with two labels the reference's Softmax::get_gradient aborts on a size check (multiclass_obj.cu:9); binary:logistic is the 2-class objective
    TGBM_CHECK(!((m.objective == MULTI_SOFTMAX || m.objective == MULTI_SOFTPROB) && p.num_class <= 2),
               "multi:softmax / multi:softprob need more than two classes; use binary:logistic for two");
    m.num_class = p.num_class;

    const bool timing = getenv("TGBM_TIMING") != nullptr;
    auto t_mark = std::chrono::steady_clock::now();
    auto lap = [&](const char *what) {
        if (!timing) return;
        cudaStreamSynchronize(m.stream);
        const auto t = std::chrono::steady_clock::now();
        fprintf(stderr, "[tgbm init] %-28s %8.1f ms\n", what, std::chrono::duration<double, std::milli>(t - t_mark).count());
        t_mark = t;
    };
    if (p.tree_method == "auto") p.tree_method = m.F > 20000 ? "exact" : "hist";   // src/thundergbm/trainer.cu:19-23
    TGBM_CHECK(p.tree_method == "hist" || p.tree_method == "exact", "unknown tree_method " + p.tree_method);
    m.exact = p.tree_method == "exact";
    if (m.exact) {
        TGBM_CHECK(!multi, "the exact builder runs on one GPU");
        locally([&] { m.init_exact(); });
        agree("sorting its columns");
    } else {
        m.find_cuts_and_bins(ds);
    }
    lap("= cuts and bins, with frees");

    locally([&] {
    const int N = m.N, K = m.K, depth = m.depth;
    const size_t n1 = std::max<size_t>(N, 1);
    m.y.alloc(n1); m.ypred.alloc(n1 * K); m.gh.alloc(n1 * K); m.ghq.alloc(n1 * K);
    upload_h2d(m.y.p, ds.yv ? ds.yv : ds.y.data(), sizeof(float) * (size_t)N, m.stream, std::min(4, upload_threads()));
    if (ds.labels_raw && N) {  // label value -> class index (dataset.cpp:83-101), on the device
        DevBuf<float> d_label;
        d_label.alloc(std::max<size_t>(ds.label.size(), 1));
        TGBM_CUDA(cudaMemcpyAsync(d_label.p, ds.label.data(), sizeof(float) * ds.label.size(), cudaMemcpyHostToDevice, m.stream));
        k_map_labels<<<std::min(ceil_div(N, 256), m.num_sms * 8), 256, 0, m.stream>>>(m.y.p, N, d_label.p, (int)ds.label.size());
        TGBM_CUDA(cudaStreamSynchronize(m.stream));
    }
    m.ypred.zero(m.stream);
    m.maxbits.alloc(2); m.root_sum.alloc(2 * (size_t)K + 2); m.qinfo.alloc(1);
    m.maxbits.zero(m.stream); m.root_sum.zero(m.stream);
    if (p.bagging) {
        TGBM_CHECK((unsigned long long)std::max(p.num_class, 1) * (unsigned long long)m.N_global < (1ull << 32), "bagging: num_class x rows must fit 32 bits");
        m.bag_count.alloc(n1 * K);
    }
    if (p.column_sampling_rate < 1.f) {
        // Shard::column_sampling (src/thundergbm/builder/shard.cu:8-23), once per round for all trees of the round:
        // max(1, int(F * rate)) randomly chosen features are put into the IGNORED set -- the reference's rate is the
        // share that is left out.  Its shuffle draws from std::rand(); here the features with the smallest hash of
        // (seed, round, feature) are taken, for all rounds in advance (the boosting loop never returns to the host).
        const int F = m.F, rounds = std::max(p.n_trees, 1);
        const int n_ignored = std::max(1, (int)(F * p.column_sampling_rate));
        std::vector<unsigned char> mask((size_t)rounds * F, 0);
        std::vector<std::pair<uint32_t, int>> key(F);
        for (int r = 0; r < rounds; ++r) {
            for (int f = 0; f < F; ++f) key[f] = {mix32(p.sample_seed ^ 0xC01A5EEDu, (uint32_t)r, 0u, (uint32_t)f), f};
            std::nth_element(key.begin(), key.begin() + std::min(n_ignored, F) - 1, key.end());
            for (int i = 0; i < std::min(n_ignored, F); ++i) mask[(size_t)r * F + key[i].second] = 1;
        }
        m.ignored_all.alloc(mask.size());
        TGBM_CUDA(cudaMemcpyAsync(m.ignored_all.p, mask.data(), mask.size(), cudaMemcpyHostToDevice, m.stream));
        TGBM_CUDA(cudaStreamSynchronize(m.stream));
    }
    m.qinfo_log.alloc(std::max(p.n_trees, 1) + 1);
    const size_t B1 = std::max(m.B, 1);
    const int max_pairs = std::max(1, 1 << std::max(0, depth - 2));
    {
        // trees built side by side: all of a round's while their buffers stay within 6 GB, and within an eighth of what is free
        // on a single GPU (ranks must agree on the number)
        Batch &b = m.bufs;
        b.half = (int)n1;
        b.nodes_stride = m.n_nodes;
        b.seg_stride = (size_t)1 << depth;
        // left children in the first half, right children in the second; the bulk copies that stage a unit of row ids read
        // up to a unit beyond the last one, from a 16-byte boundary
        b.rec_stride = (2 * n1 + 2 * F32_THREADS + 3) / 4 * 4;
        b.nid_stride = (n1 + ASSIGN_CHUNK - 1) / ASSIGN_CHUNK * ASSIGN_CHUNK;
        b.gh_stride = N;
        b.full_stride = (((size_t)1 << depth) - 1) * B1 * 2;
        b.built_stride = max_pairs * B1 * 2;
        b.recs_stride = m.exact ? 1 : ((size_t)1 << (depth - 1)) * (m.sparse ? std::max(m.n_chunks, 1) : m.F);
        b.ticket_stride = max_pairs;
        b.rule_stride = (size_t)1 << (depth - 1);
        // (the same number on every rank: it decides the order of the collectives)
        const double per_tree = 10.0 * (double)(std::max(most_rows, 1ll) + F32_THREADS) + 8.0 * (b.full_stride + b.built_stride);
        double room = 6e9;
        if (K * per_tree > 512e6 && K > 1 && !multi) {   // (asking takes 0.4 ms)
            size_t free_bytes = 0, all_bytes = 0;
            TGBM_CUDA(cudaMemGetInfo(&free_bytes, &all_bytes));
            room = std::min(room, free_bytes / 8.0);
        }
        m.batch = m.exact ? 1 : std::max(1, std::min(K, (int)(room / per_tree)));
        // Eight rows a thread from 1.2 M rows on (four and eight, us a launch: 600 k rows 5.3 and 5.3, 1.2 M 8.3 and 7.2, 3 M 15.8 and 15.1;
        // training rounds differ by 1 % at most)
        m.assign_rpt = !m.sparse && (long long)N * m.batch >= 4ll * m.num_sms * 8 * ASSIGN_THREADS ? 8 : 4;
        m.assign_ctas = std::max(1, std::min(ceil_div(N, ASSIGN_THREADS * m.assign_rpt), m.num_sms * (m.sparse || m.assign_rpt == 8 ? 4 : 6) / m.batch));
        const size_t T = m.batch;
        m.nodes.alloc(T * b.nodes_stride); b.nodes = m.nodes.p;
        for (int i = 0; i < 2; ++i) {
            m.seg_begin[i].alloc(T * b.seg_stride); m.seg_cnt[i].alloc(T * b.seg_stride); m.origin[i].alloc(T * b.seg_stride);
            m.seg_begin[i].zero(m.stream); m.seg_cnt[i].zero(m.stream);
            b.seg_begin[i] = m.seg_begin[i].p; b.seg_cnt[i] = m.seg_cnt[i].p; b.origin[i] = m.origin[i].p;
        }
        m.rec_idx.alloc(T * b.rec_stride); b.rec_idx = m.rec_idx.p;
        m.nid.alloc(T * b.nid_stride); b.nid = m.nid.p;
        m.nid.zero(m.stream);   // (what lies behind the rows stays so)
        m.leaf_weight.alloc(T * b.nodes_stride); b.weight = m.leaf_weight.p;
        m.leaf_rule.alloc(T * b.rule_stride); b.rule = m.leaf_rule.p;
        if (m.f32 && !m.exact) m.assign_table.alloc(T * m.assign_ctas * b.rule_stride);   // (a level's children are at most the last level's nodes)
        m.hist_full.alloc(T * b.full_stride); b.hist_full = m.hist_full.p;
        m.hist_built.alloc(T * b.built_stride); b.hist_built = m.hist_built.p;
        m.hist_built.zero(m.stream);   // the split search leaves it zeroed
        m.recs.alloc(T * b.recs_stride); b.recs = m.recs.p;
        m.eval_ticket.alloc(T * b.ticket_stride); b.ticket = m.eval_ticket.p;
        m.eval_ticket.zero(m.stream);
        m.ctl.alloc(1); b.ctl = m.ctl.p;
        m.ctl.zero(m.stream);
    }
    m.model.alloc((size_t)std::max(p.n_trees, 1) * K * m.n_nodes);
    m.metric.alloc(std::max(p.n_trees, 1));
    if (p.keep_nid) m.nid_keep.alloc(n1 * K * std::max(p.n_trees, 1));
    if (m.f32) {
        for (int f = 0; f < std::min(m.S, 256); ++f) m.f32_cuts.v[f] = m.h_slot_ptr[f];
        m.spread_cells = std::min<size_t>((size_t)32 * m.batch * max_pairs * B1, (size_t)8 << 20);   // 64 MB: they stay in L2
        m.hist_spread.alloc(m.spread_cells);
        m.hist_spread.zero(m.stream);
        m.sum_partial.alloc((size_t)SUM_BLOCKS * K * 2);
        const QuantInfo one{1.0, 1.0, 1.0, 1.0};
        TGBM_CUDA(cudaMemcpyAsync(m.qinfo.p, &one, sizeof(one), cudaMemcpyHostToDevice, m.stream));
        TGBM_CUDA(cudaStreamSynchronize(m.stream));
    }
    if (!m.exact && !m.sparse) {
        std::vector<int4> one, four;
        for (int f = 0; f < m.F; ++f) {
            if (m.h_cut_ptr[f + 1] - m.h_cut_ptr[f] > EVAL_SMALL) { one.push_back(make_int4(f, -2, -2, -2)); continue; }
            if (four.empty() || four.back().w >= 0) { four.push_back(make_int4(f, -1, -1, -1)); continue; }
            int4 &t = four.back();
            (t.y < 0 ? t.y : t.z < 0 ? t.z : t.w) = f;
        }
        if (four.size() > 1 || (four.size() == 1 && four[0].y >= 0)) {   // (the long ones first)
            one.insert(one.end(), four.begin(), four.end());
            m.n_eval_items = (int)one.size();
            m.eval_items.alloc(one.size());
            TGBM_CUDA(cudaMemcpyAsync(m.eval_items.p, one.data(), sizeof(int4) * one.size(), cudaMemcpyHostToDevice, m.stream));
            TGBM_CUDA(cudaStreamSynchronize(m.stream));
        }
    }
    m.rstate.alloc(1);
    m.rstate.zero(m.stream);
    m.graphs_allowed = getenv("TGBM_NO_GRAPH") == nullptr;
    m.f32_staged = getenv("TGBM_NO_BULK_COPY") == nullptr;
    m.metric_partial.alloc(m.metric_blocks()); m.metric_sum.alloc(1);
    m.window_rows = (1 << (31 - p.quant_bits)) - HIST_THREADS;
    TGBM_CHECK(m.window_rows >= HIST_THREADS, "quant_bits too large for the int32 accumulation window");
    constexpr size_t table = 4 * ((1 << (MAX_DEPTH - 2)) + 1);   // tiles before every pair of the deepest level
    allow_shared(k_hist<true, false>, HIST_EXACT_SMEM + table);
    allow_shared(k_hist<false, false>, HIST_EXACT_SMEM + table);
    allow_shared(k_hist<true, true>, HIST_FINE_SMEM + table);
    allow_shared(k_hist<false, true>, HIST_FINE_SMEM + table);
    if (assign_smem(std::max(0, depth - 2), m.assign_rpt) > 48 * 1024) {   // (depth 12 and beyond: one kernel for all levels with many children)
        allow_shared(m.assign_kernel(depth - 2, false), assign_smem(MAX_DEPTH - 2, ASSIGN_CHUNK / ASSIGN_THREADS));
        allow_shared(m.assign_kernel(depth - 2, true), assign_smem(MAX_DEPTH - 2, ASSIGN_CHUNK / ASSIGN_THREADS));
    }
    allow_shared(k_hist_sparse<true>, SPARSE_SMEM_BINS * 16 + table);
    allow_shared(k_hist_sparse<false>, SPARSE_SMEM_BINS * 16 + table);
    m.prune_in_smem = sizeof(TreeNode) * (size_t)m.n_nodes <= PRUNE_SMEM;  // up to depth 11
    if (m.prune_in_smem && sizeof(TreeNode) * (size_t)m.n_nodes > 40 * 1024)   // (the kernel has static shared memory beside it)
        allow_shared(k_prune, PRUNE_SMEM);
    m.plan_small_trees();
    if (need_group_file(m.objective)) m.rank.init(ds, m.objective, m.N, m.stream, first_group, total_groups);
    if (m.sparse && (long long)p.n_trees * K >= COLUMNS_TREES) m.sort_columns();
    });
    agree("allocating its training buffers");
    lap("training buffers");
    m.init_base_score();
    TGBM_CUDA(cudaStreamSynchronize(m.stream));
    TGBM_CUDA(cudaGetLastError());
    lap("base score");
}

// ------------------------------------------------------------------------------------------------
void BoosterImpl::gradient(int round) {
    const int tb = 256;
    const bool pointwise = objective == REG_LINEAR || objective == REG_LOGISTIC || objective == BINARY_LOGISTIC;
    const int logistic = objective == REG_LINEAR ? 0 : 1;
    // the pass that applied the previous tree has already found this round's gradient maxima
    const bool have_max = pointwise && grad_max_ready && round >= 0 && !float_round(round) && !p.bagging;
    grad_max_ready = false;
    // (root_sum and maxbits are zero here: k_round_end and k_tree_init leave them so)
    if (!have_max) {
        if (N) {
            const int gb = std::max(1, std::min(ceil_div(N, tb), num_sms * 8));
            switch (objective) {
            case REG_LINEAR: case REG_LOGISTIC: case BINARY_LOGISTIC:
                launch_after(k_grad_pointwise, gb, tb, 0, stream, y.p, ypred.p, N, logistic, gh.p, maxbits.p); break;
            case MULTI_SOFTMAX: case MULTI_SOFTPROB:
                launch_after(k_grad_softmax, gb, tb, 0, stream, y.p, ypred.p, N, K, gh.p, maxbits.p); break;
            case RANK_PAIRWISE: case RANK_NDCG:
                rank.gradient(rstate.p, p.rank_seed, ypred.p, gh.p, maxbits.p, stream); break;
            }
            ++launches;
        }
    }
    if (p.bagging && round >= 0 && N) {  // not for the base score (include/thundergbm/booster.h:69-73 comes before any sampling)
        bag_count.zero(stream);
        const unsigned long long m_total = (unsigned long long)std::max(p.num_class, 1) * (unsigned long long)N_global;
        k_bag_draw<<<num_sms * 8, 256, 0, stream>>>(m_total, p.sample_seed, rstate.p, N_global, row_offset, N, K, bag_count.p);
        maxbits.zero(stream);
        k_bag_scale<<<std::max(1, std::min(ceil_div((long long)N * K, 256), num_sms * 8)), 256, 0, stream>>>(gh.p, bag_count.p, (size_t)N * K, maxbits.p);
        launches += 2;
    }
    if (float_round(round)) {  // float gradients as they are; root sums in fp64, block partials combined in a fixed order
        launch_after(k_sum_gh, dim3(SUM_BLOCKS, K), 256, 0, stream, gh.p, N, sum_partial.p);
        launch_after(k_sum_gh_final, K, 32, 0, stream, sum_partial.p, SUM_BLOCKS, reinterpret_cast<double *>(root_sum.p));
        launches += 2;
        if (comm && comm->active()) comm->allreduce(root_sum.p, 2 * (size_t)K, Comm::F64, Comm::SUM, stream);
        return;
    }
    if (comm && comm->active()) comm->allreduce(maxbits.p, 2, Comm::U32, Comm::MAX, stream);
    const int blocks = std::max(1, std::min(ceil_div(N, tb), num_sms * 8));
    auto quantize = [&](auto kern, int bits) {
        launch_after(kern, dim3(blocks, K), tb, 0, stream, have_max ? nullptr : gh.p, N, maxbits.p, bits, (uint32_t)round, (uint32_t)row_offset,
                                                 ghq.p, root_sum.p, qinfo.p, y.p, ypred.p, logistic, round >= 0 ? rstate.p : nullptr, root_sum.p + 2 * K);
    };
    if (f32) quantize(k_quantize<true>, FINE_BITS);   // (its two words on the spread follow the root sums)
    else quantize(k_quantize<false>, p.quant_bits);
    ++launches;
    if (comm && comm->active()) comm->allreduce(root_sum.p, 2 * (size_t)K + (f32 ? 2 : 0), Comm::I64, Comm::SUM, stream);
}

// Base score (include/thundergbm/objective/regression_obj.h:35-53 and :95-114): gradients at y_pred = 0,
// w = -sum g / max(sum h, 1e-6) evaluated in double; binary:logistic maps it through sigmoid and logit
// with the host's libm, as the reference does.
void BoosterImpl::init_base_score() {
    base_score = 0;
    if (exact) return;   // include/thundergbm/booster.h:66-73: the reference computes a base score for tree_method = hist only
    if (!(objective == REG_LINEAR || objective == REG_LOGISTIC || objective == BINARY_LOGISTIC)) return;
    gradient(-1);
    unsigned long long hs[2];
    QuantInfo q;
    TGBM_CUDA(cudaMemcpyAsync(hs, root_sum.p, sizeof(hs), cudaMemcpyDeviceToHost, stream));
    TGBM_CUDA(cudaMemcpyAsync(&q, qinfo.p, sizeof(q), cudaMemcpyDeviceToHost, stream));
    TGBM_CUDA(cudaStreamSynchronize(stream));
    float fg, fh;
    if (f32) {
        double d[2];
        memcpy(d, hs, sizeof(d));
        fg = (float)d[0]; fh = (float)d[1];
    } else {
        fg = (float)((double)(long long)hs[0] * q.inv_sg); fh = (float)((double)(long long)hs[1] * q.inv_sh);
    }
    float w = (float)(-(double)fg / std::fmax((double)fh, 1e-6));
    if (objective == BINARY_LOGISTIC) {
        w = 1 / (1 + expf(-w));
        w = -logf(1.0f / w - 1.0f);
    }
    base_score = w;
    p.base_score = w;
    if (N) k_fill<<<std::min(ceil_div(N, 256), num_sms * 8), 256, 0, stream>>>(ypred.p, (size_t)N, w);
    root_sum.zero(stream); maxbits.zero(stream);
}

// Is the data small enough for a tree per launch (tgbm_small.cuh)?  Every CTA of the cluster walks all rows for its share of
// the features, so its time grows with rows x features per CTA and, deep down, with nodes x features per CTA, while a level
// of the level kernels takes 25-30 us at any size up to a few hundred thousand rows.
void BoosterImpl::plan_small_trees() {
    small = SmallPlan{};
    if (sparse || exact || (comm && comm->active()) || N < 1 || N > SMALL_ROWS || depth < 1 || F > 4096) return;
    SmallPlan pl{};
    pl.cluster = 1;
    while (pl.cluster < 16 && pl.cluster < F) pl.cluster *= 2;
    const int max_nl = 1 << (depth - 1);
    cudaFuncSetAttribute(small_kernel(), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (; pl.cluster >= 1; pl.cluster /= 2) {
        pl.feats = ceil_div(F, pl.cluster);
        pl.bins = 1;
        for (int f = 0; f < F; f += pl.feats) pl.bins = std::max(pl.bins, h_cut_ptr[std::min(F, f + pl.feats)] - h_cut_ptr[f]);
        if ((double)N * pl.feats > 8e4 || (double)max_nl * pl.feats > 512) return;
        const size_t budget = 200 * 1024, fixed = (sizeof(TreeNode) * (size_t)n_nodes + 15) / 16 * 16 + sizeof(SmallPost) * 2 * max_nl + (size_t)(N + 7) / 8 * 16 +
                     4 * (size_t)((max_nl + 3) / 4 * 4) + 4 * (size_t)(pl.feats + 1 + pl.bins) + 64;   // (64: roundings)
        pl.cells = small_feature_at(pl.bins, pl.feats);
        for (int f = 0; f < F; ++f) pl.most = std::max(pl.most, h_cut_ptr[f + 1] - h_cut_ptr[f]);
        const size_t per_node = 16 * (size_t)pl.cells + sizeof(SplitRec) * pl.feats;
        if (fixed + per_node > budget) return;
        pl.nodes_pass = (int)std::min<size_t>(max_nl, (budget - fixed) / per_node);
        if (max_nl > 8 * pl.nodes_pass) return;   // the rows would be walked over and over
        pl.smem = fixed + per_node * pl.nodes_pass;
        allow_shared(small_kernel(), budget);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = pl.cluster; cfg.blockDim = SMALL_THREADS; cfg.dynamicSmemBytes = pl.smem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = pl.cluster; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr; cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, small_kernel(), &cfg) == cudaSuccess && fit >= 1) {
            small = pl;
            return;
        }
        cudaGetLastError();   // no GPC has room for a cluster of this size: half of it
    }
}

void BoosterImpl::launch_small_trees(int k0, int n_trees) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = small.cluster * n_trees; cfg.blockDim = SMALL_THREADS; cfg.dynamicSmemBytes = small.smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = small.cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    const int2 *gq = ghq.p + (size_t)k0 * N;
    const unsigned long long *roots = root_sum.p + 2 * (size_t)k0;
    TGBM_CUDA(cudaLaunchKernelEx(&cfg, small_kernel(), (SmallPlan)small, N, Npad, F, depth, (const unsigned char *)binsT.p, (const int *)cut_ptr.p,
                                 (const float *)cut_val.p, gq, roots, (const QuantInfo *)qinfo.p, p.min_child_weight, p.lambda, p.rt_eps, p.gamma,
                                 (const unsigned char *)ignored_all.p, (const RoundState *)rstate.p, p.column_shards > 0 ? 1 : 0, nodes.p, model.p, K, k0,
                                 maxbits.p, f32 && k0 == 0 ? K : 0, ctl.p, hist_full.p, bufs.full_stride, nid.p, bufs.nid_stride, leaf_weight.p, leaf_rule.p, bufs.rule_stride));
    ++launches;
}

// Trees k0 .. k0 + n_trees - 1 of the round, level by level side by side (n_trees <= batch).
void BoosterImpl::build_trees(int round, int k0, int n_trees) {
    const bool float_sums = float_round(round), fine = f32 && !float_sums;
    last_float = float_sums;
    last_tree_full = (size_t)(n_trees - 1) * bufs.full_stride;
    Batch b = bufs;
    // float rounds: the float gradient pairs themselves (same 8 bytes)
    b.gh = float_sums ? reinterpret_cast<const int2 *>(gh.p + (size_t)k0 * N) : ghq.p + (size_t)k0 * N;
    const bool one_launch = small.cluster > 0 && !float_sums && !profile_on;
    if (one_launch) launch_small_trees(k0, n_trees);
    else {
    launch_after(k_tree_init, dim3(ceil_div(n_nodes, 256), n_trees), 256, 0, stream, nodes.p, n_nodes, root_sum.p + 2 * k0, qinfo.p, p.lambda, N,
                                                                           seg_begin[0].p, seg_cnt[0].p, b.seg_stride, float_sums ? 1 : 0, maxbits.p, fine && k0 == 0 ? K : 0, ctl.p);
    ++launches;
    }
    const int by_hessian = (comm && comm->active()) ? 1 : 0;
    const int colb = p.column_shards > 0 ? 1 : 0;  // candidates, tie rule and child sums of the column-sharded builder
    // one CTA per SM over all trees and groups of slots: every further CTA is one more flush per node
    const int G = sparse ? 1 : Spad / 32, hist_ctas = std::max(1, num_sms / (n_trees * G));
    const int *slots = slot_ptr.p ? slot_ptr.p : cut_ptr.p;
    for (int level = 0; level < depth && !one_launch; ++level) {
        const int nl = 1 << level, pairs = std::max(1, nl / 2), keep = level == 0 || level + 1 < depth;
        const size_t table = sizeof(int) * ((size_t)pairs + 1);
        // -- histogram of the root / of the smaller child of every pair, and the choice of the splits
        auto evaluate = [&](auto *built, size_t tree_cells, int bs) {
            using T = std::remove_pointer_t<decltype(built)>;
            if (sparse) {
                launch_after(k_eval_chunk<T>, dim3(n_chunks, pairs, n_trees), 64, 0, stream, level, b, n_chunks, B, chunk_bin0.p, cut_ptr.p, cut_val.p, cut_fid.p, built, tree_cells, bs,
                             qinfo.p, p.min_child_weight, p.lambda, ignored_all.p, rstate.p, F, colb, by_hessian, keep);
                launch_after(k_best_apply, dim3(nl, 1, n_trees), 32, 0, stream, level, b, n_chunks, cut_ptr.p, p.rt_eps, p.lambda, colb);
                launches += 2;
            } else {
                const bool items = sizeof(T) == 8 && n_eval_items > 0;
                auto kern = items ? k_eval<T, sizeof(T) == 8> : k_eval<T, false>;
                launch_after(kern, dim3(items ? n_eval_items : F, pairs, n_trees), EVAL_THREADS, 0, stream, level, b, items ? eval_items.p : nullptr, F, B, cut_ptr.p, built, tree_cells, bs, qinfo.p, p.min_child_weight, p.lambda,
                             cut_val.p, p.rt_eps, ignored_all.p, rstate.p, colb, by_hessian, keep);
                ++launches;
            }
        };
        auto timed = [&](int kind, auto &&work) {
            TimedEvent ev{};
            if (profile_on) {
                cudaEventCreate(&ev.a); cudaEventCreate(&ev.b);
                ev.kind = kind;
                cudaEventRecord(ev.a, stream);
            }
            const long long before = launches;
            work();
            ev.launches = launches - before;
            if (profile_on) { cudaEventRecord(ev.b, stream); events.push_back(ev); }
        };
        if (float_sums) {
            // Values are added one by one into cells `bs` float pairs apart
            const int bs = f32_stride(pairs * n_trees), ctas = std::max(1, num_sms * (2048 / F32_THREADS) / n_trees);
            const bool spread = bs != 1, multi = comm && comm->active();
            const size_t level_cells = (size_t)B * pairs, compact_cells = b.built_stride;
            float2 *compact = reinterpret_cast<float2 *>(hist_built.p), *cells = spread ? hist_spread.p : compact;
            const size_t tree_cells = spread ? level_cells * bs : compact_cells;
            // (the split search leaves the cells it reads zeroed; between ranks it reads the gathered ones)
            if (spread && multi) TGBM_CUDA(cudaMemsetAsync(cells, 0, sizeof(float2) * tree_cells * n_trees, stream));
            timed(level == 0 ? 0 : 1, [&] {
                if (sparse) {
                    auto kern = level == 0 ? k_hist_sparse_f32<false> : k_hist_sparse_f32<true>;
                    launch_after(kern, dim3(ctas, 1, n_trees), F32_THREADS, table, stream, level, b, sp_row_ptr.p, sp_bin.p, cells, tree_cells, B, bs, by_hessian);
                } else {
                    auto kern = level == 0 ? k_hist_f32<false> : k_hist_f32<true>;
                    launch_after(kern, dim3(ctas, G, n_trees), F32_THREADS, table, stream, level, b, bins.p, Spad, S, slots, cells, tree_cells, B, bs, f32_cuts, S <= 256,
                                 f32_staged ? 1 : 0, by_hessian);
                }
            });
            ++launches;
            if (multi) {
                // the ranks' sums meet in compact buffers: spread cells are gathered first (a pass over B x pairs cells)
                for (int t = 0; t < n_trees; ++t) {
                    if (spread) {
                        launch_after(k_compact_cells, std::min(ceil_div(level_cells, 256), num_sms * 8), 256, 0, stream, cells + t * tree_cells, compact + t * compact_cells,
                                     level_cells, bs);
                        ++launches;
                    }
                    comm->allreduce(compact + t * compact_cells, 2 * level_cells, Comm::F32, Comm::SUM, stream);
                }
                evaluate(reinterpret_cast<float *>(compact), 2 * compact_cells, 1);
            } else evaluate(reinterpret_cast<float *>(cells), 2 * tree_cells, bs);
        } else {
            timed(level == 0 ? 0 : 1, [&] {
                if (sparse && level == 0 && col_ptr.p) {
                    launch_after(k_hist_columns, dim3(std::max(1, num_sms * 8 / n_trees), 1, n_trees), 256, 0, stream, b, columns(), (int)nnz_local);
                } else if (sparse) {
                    auto kern = level == 0 ? k_hist_sparse<false> : k_hist_sparse<true>;
                    launch_after(kern, dim3(hist_ctas, 1, n_trees), SPARSE_THREADS, (size_t)std::min(B, SPARSE_SMEM_BINS) * 16 + table, stream, level, b, sp_row_ptr.p, sp_bin.p, B, by_hessian);
                } else {
                    auto kern = level == 0 ? (fine ? k_hist<false, true> : k_hist<false, false>) : (fine ? k_hist<true, true> : k_hist<true, false>);
                    launch_after(kern, dim3(hist_ctas, G, n_trees), HIST_THREADS, (fine ? HIST_FINE_SMEM : HIST_EXACT_SMEM) + table, stream, level, b, bins.p, Spad, S, slots, B, window_rows, by_hessian);
                }
            });
            ++launches;
            if (comm && comm->active())
                for (int t = 0; t < n_trees; ++t) comm->allreduce(hist_built.p + t * b.built_stride, 2 * (size_t)B * pairs, Comm::I64, Comm::SUM, stream);
            evaluate(hist_built.p, b.built_stride, 1);
        }
        // -- rows to their children (after the last level k_apply_tree does it)
        const bool by_columns = sparse && col_ptr.p, last = level == depth - 1;
        if (last && !by_columns) break;
        timed(2, [&] {
            if (by_columns) {
                const int node_blocks = std::min(nl, 1024);
                launch_after(k_assign_stored, dim3(std::max(1, num_sms * 8 / (node_blocks * n_trees)), node_blocks, n_trees), 256, 0, stream, level, b, columns(), cut_ptr.p, colb);
                ++launches;
            }
            if (last) return;
            auto assign = [&](int order) {
                launch_after(assign_kernel(level, float_sums), dim3(assign_ctas, 1, n_trees), ASSIGN_THREADS, assign_smem(level, assign_rpt), stream, level, b, N, binsT.p, Npad, sp_row_ptr.p,
                             sp_bin.p, cut_ptr.p, columns(), colb, order, assign_table.p);
                ++launches;
            };
            if (float_sums) {
                const bool add = 2ll * nl * assign_ctas <= ASSIGN_ADD;
                assign(ASSIGN_COUNT);
                if (!add) {
                    launch_after(k_assign_before, dim3(ceil_div(2 * nl, 32), 1, n_trees), 1024, 0, stream, assign_ctas, 2 * nl, assign_table.p);
                    ++launches;
                }
                assign(add ? ASSIGN_PLACE_ADD : ASSIGN_PLACE);
            } else assign(ASSIGN_ANY);
        });
    }
    if (!one_launch) {
        launch_after(k_prune, n_trees, 1024, prune_in_smem ? sizeof(TreeNode) * (size_t)n_nodes : 0, stream, nodes.p, n_nodes, depth, p.gamma, prune_in_smem ? 1 : 0,
                     model.p, K, k0, rstate.p, leaf_weight.p, leaf_rule.p, b.rule_stride, colb, seg_cnt[(depth - 1) & 1].p, b.seg_stride, cut_ptr.p, sparse ? col_ptr.p : nullptr);
        ++launches;
    }
    if (N) {
        float *yp = ypred.p + (size_t)k0 * N;
        int *nid_out = p.keep_nid ? nid_keep.p + ((size_t)round * K + k0) * N : nullptr;
        // One tree per round and a pointwise objective: the pass also adds up the round's metric and finds the maxima
        // of the next round's gradients (grid and order of additions are those of k_metric_partial).
        const bool fuse = K == 1 && (objective == REG_LINEAR || objective == REG_LOGISTIC || objective == BINARY_LOGISTIC);
        const dim3 ctas(fuse ? metric_blocks() : std::min(ceil_div(N, 256), num_sms * 8), n_trees);
        launch_after(sparse ? k_apply_tree<true> : k_apply_tree<false>, ctas, 256, 0, stream, b, N, depth - 1, binsT.p, Npad, sp_row_ptr.p, sp_bin.p,
                     cut_ptr.p, p.learning_rate, yp, nid_out, y.p, fuse ? objective : -1, metric_partial.p, maxbits.p, colb);
        ++launches;
        grad_max_ready = metric_partial_ready = fuse;
    }
}

void BoosterImpl::round_metric(int round) {
    const int log_len = (int)qinfo_log.n;
    if (need_group_file(objective)) {
        rank.metric(objective, ypred.p, nullptr, comm, N_global, stream);
        launch_after(k_round_end, 1, 32, 0, stream, objective, rank.sum.p, nullptr, 0, rank.n_group_total, metric.p, qinfo.p, qinfo_log.p, log_len, rstate.p, root_sum.p, 2 * K + 2, ctl.p);
        ++launches;
        return;
    }
    const int blocks = metric_blocks();
    if (!metric_partial_ready) {  // else the pass that applied the round's tree has left the partial sums
        launch_after(k_metric_partial, blocks, 256, 0, stream, objective, y.p, ypred.p, N, K, metric_partial.p);
        ++launches;
    }
    metric_partial_ready = false;
    const bool multi = comm && comm->active();
    if (multi) {
        k_metric_sum<<<1, 32, 0, stream>>>(metric_partial.p, blocks, metric_sum.p);
        comm->allreduce(metric_sum.p, 1, Comm::F64, Comm::SUM, stream);
        ++launches;
    }
    launch_after(k_round_end, 1, 32, 0, stream, objective, metric_sum.p, multi ? nullptr : metric_partial.p, blocks, N_global, metric.p, qinfo.p, qinfo_log.p,
                                      log_len, rstate.p, root_sum.p, 2 * K + 2, ctl.p);
    ++launches;
}

// One boosting round.  From the second round on the launch sequence no longer changes (which kernels run is decided
// by the objective and by flags that have reached their steady state; everything that depends on the data is decided
// on the device), so it is captured once into a CUDA graph and replayed: one launch per round instead of ~60, no
// gaps between the small per-level kernels.  Not with profiling events or a kept row->node table.  With a communicator
// the NCCL calls of the round are captured with it (every rank captures and replays the same sequence).
void BoosterImpl::queue_round(int round) {
    gradient(round);
    for (int k = 0; k < K; k += batch) {
        if (exact) build_tree_exact(round, k);
        else build_trees(round, k, std::min(batch, K - k));
    }
    round_metric(round);
}
void BoosterImpl::run_round(int round) {
    static const bool graph_with_comm = getenv("TGBM_NO_GRAPH_COMM") == nullptr;  // the round's collectives are captured with it
    // Ranks that are threads of ONE process do not replay graphs: instantiating a graph allocates device memory, and with
    // peer access enabled such a call can wait for the other devices of the process -- whose collective kernels may
    // already be waiting for this rank's.  (Between processes there is no such coupling.)
    const bool in_process_group = comm && comm->active() && comm->host;
    const bool graph_ok = graphs_allowed && round >= 1 && !profile_on && !p.keep_nid && !in_process_group &&
                          (graph_with_comm || !(comm && comm->active()));
    if (!graph_ok) { queue_round(round); return; }
    if (!round_exec) {
        const long long before = launches;
        TGBM_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        bool ok = true;
        try { queue_round(round); } catch (...) { ok = false; }
        cudaGraph_t g = nullptr;
        const cudaError_t rc = cudaStreamEndCapture(stream, &g);
        round_graph_launches = launches - before;
        launches = before;
        if (!ok || rc != cudaSuccess || !g) {  // fall back to plain launches for good
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            graphs_allowed = false;
            TGBM_CHECK(ok, "capturing a boosting round failed");
            queue_round(round);
            return;
        }
        round_graph = g;
        TGBM_CUDA(cudaGraphInstantiate(&round_exec, round_graph, 0));
    }
    TGBM_CUDA(cudaGraphLaunch(round_exec, stream));
    launches += round_graph_launches;
    last_float = float_round(round);
}

void BoosterImpl::wait() const {
    if (comm && comm->active()) comm->wait(stream);  // bounded: a rank may have left
    else TGBM_CUDA(cudaStreamSynchronize(stream));
}

// Fine rounds of fp32 mode are queued before it is known whether their gradients fit the grid.  One whose do not leaves the
// scores, the metric and the round counter alone (TreeCtl::coarse), and so does every round queued behind it.  Here, with the
// queue empty, it is built again from float sums, and the rounds after it are queued once more: in steps that start at one
// round and double, so that what is thrown away stays in proportion; one that does not fit either is found before it is built.
// Returns whether there was such a round.
bool BoosterImpl::settle() {
    if (!f32 || exact || rounds <= FINE_FROM_ROUND) return false;
    auto coarse = [&] {
        int v = 0;
        TGBM_CUDA(cudaMemcpyAsync(&v, &ctl.p->coarse, sizeof(int), cudaMemcpyDeviceToHost, stream));
        wait();
        return v != 0;
    };
    auto float_again = [&](int round) {
        static const QuantInfo one{1.0, 1.0, 1.0, 1.0};
        TGBM_CUDA(cudaMemsetAsync(&ctl.p->coarse, 0, sizeof(int), stream));
        TGBM_CUDA(cudaMemcpyAsync(qinfo.p, &one, sizeof(one), cudaMemcpyHostToDevice, stream));   // (what the log of the grids shows)
        force_float = true;
        queue_round(round);
        force_float = false;
    };
    bool again = false;
    for (int queued = rounds, step = 1;;) {
        if (coarse()) {
            RoundState at;
            TGBM_CUDA(cudaMemcpy(&at, rstate.p, sizeof(at), cudaMemcpyDeviceToHost));
            again = true;
            step = 1;
            float_again(at.round);
            for (queued = at.round + 1; queued < rounds; ++queued) {
                const bool have_max = grad_max_ready;
                gradient(queued);
                grad_max_ready = have_max;   // the maxima are still there
                k_grid_check<<<1, 1, 0, stream>>>(root_sum.p, K, ctl.p);
                root_sum.zero(stream);
                ++launches;
                if (!coarse()) break;
                float_again(queued);
            }
        } else if (queued == rounds) {
            return again;
        }
        for (int i = 0; i < step && queued < rounds; ++i) run_round(queued++);
        step *= 2;
    }
}

void Booster::boost(int n_rounds) {
    BoosterImpl &m = *impl_;
    TGBM_CHECK(m.rounds + n_rounds <= m.p.n_trees, "boost() beyond n_trees");
    for (int i = 0; i < n_rounds; ++i) {
        m.run_round(m.rounds);
        ++m.rounds;
    }
    TGBM_CUDA(cudaGetLastError());
    if (m.comm && m.comm->active()) m.settle();   // together: the ranks need not all ask for results, or at the same time
}

bool Booster::sync() {
    const bool again = impl_->settle();
    impl_->wait();
    TGBM_CUDA(cudaGetLastError());
    // bounded waits inside the kernels (bulk-copy barriers of the float histogram kernel) report here instead of spinning: the results of the run are not to be trusted
    if (impl_->ctl.p) {
        int err = 0;
        TGBM_CUDA(cudaMemcpy(&err, reinterpret_cast<const char *>(impl_->ctl.p) + offsetof(TreeCtl, error), sizeof(int), cudaMemcpyDeviceToHost));
        TGBM_CHECK(err == 0, "a bounded wait inside a kernel ran out (code " + std::to_string(err) + "); the trees of this run are invalid");
    }
    return again;
}

int Booster::rounds_done() const { return impl_->rounds; }
int Booster::trees_per_round() const { return impl_->K; }
int Booster::n_nodes() const { return impl_->n_nodes; }
int Booster::num_class() const { return impl_->num_class; }
float Booster::base_score() const { return impl_->base_score; }
int Booster::n_bins() const { return impl_->B; }
int Booster::n_features() const { return impl_->F; }
std::string Booster::tree_method() const { return impl_->p.tree_method; }
int Booster::fpad() const { return impl_->Fpad; }
cudaStream_t Booster::stream() const { return impl_->stream; }
void Booster::set_profile(bool on) {
    BoosterImpl &m = *impl_;
    if (on && !m.profile_on && m.ctl.p) {  // the byte counters of the plan kernels run all the time: remember where profiling starts
        sync();
        TGBM_CUDA(cudaMemcpy(&m.stat_base, m.ctl.p, sizeof(TreeCtl), cudaMemcpyDeviceToHost));
    }
    m.profile_on = on;
}

HistProfile Booster::profile() {
    BoosterImpl &m = *impl_;
    sync();
    HistProfile r;
    for (auto &e : m.events) {
        float ms = 0;
        cudaEventElapsedTime(&ms, e.a, e.b);
        if (e.kind == 2) { r.partition_ms += ms; r.partition_launches += e.launches; }
        else {
            r.hist_ms += ms; r.hist_launches += 1;
            if (e.kind == 0) { r.hist_root_ms += ms; r.hist_root_launches += 1; }
        }
    }
    // the timed events have been read: their times move into running totals and the events are destroyed, so that a
    // long profiled run does not pile them up
    for (auto &e : m.events) { cudaEventDestroy(e.a); cudaEventDestroy(e.b); }
    m.events.clear();
    m.profile_acc.hist_ms += r.hist_ms; m.profile_acc.hist_launches += r.hist_launches;
    m.profile_acc.hist_root_ms += r.hist_root_ms; m.profile_acc.hist_root_launches += r.hist_root_launches;
    m.profile_acc.partition_ms += r.partition_ms; m.profile_acc.partition_launches += r.partition_launches;
    r = m.profile_acc;
    TreeCtl c;
    TGBM_CUDA(cudaMemcpy(&c, m.ctl.p, sizeof(c), cudaMemcpyDeviceToHost));
    // algorithmic bytes: rows * (bin bytes + 8 gradient bytes [+ 4 row index]) + histograms * B * 16 written
    // bin bytes of a row: a byte per slot (S: a feature, or several that share it) dense; 4 per stored value + a row pointer in the CSR layout
    const double row_bytes = m.sparse ? 4.0 * (double)m.nnz_local / std::max(1, m.N) + 4.0 : (double)m.S;
    const TreeCtl &c0 = m.stat_base;
    r.hist_root_bytes = (double)(c.stat_rows_root - c0.stat_rows_root) * (row_bytes + 8);
    r.hist_bytes = r.hist_root_bytes + (double)(c.stat_rows_gather - c0.stat_rows_gather) * (row_bytes + 8 + 4) +
                   (double)(c.stat_hists - c0.stat_hists) * m.B * (m.last_float ? 8.0 : 16.0);
    r.partition_bytes = (double)(c.stat_part_rows - c0.stat_part_rows) * (4 + 1 + 4);
    r.hist_rows = (long long)((c.stat_rows_root - c0.stat_rows_root) + (c.stat_rows_gather - c0.stat_rows_gather));
    r.kernel_launches = m.launches;
    return r;
}

std::vector<std::vector<Tree>> Booster::get_model() {
    BoosterImpl &m = *impl_;
    sync();
    std::vector<TreeNode> h((size_t)m.rounds * m.K * m.n_nodes);
    if (!h.empty()) TGBM_CUDA(cudaMemcpy(h.data(), m.model.p, sizeof(TreeNode) * h.size(), cudaMemcpyDeviceToHost));
    std::vector<std::vector<Tree>> out(m.rounds);
    for (int r = 0; r < m.rounds; ++r) {
        out[r].resize(m.K);
        for (int k = 0; k < m.K; ++k) {
            const TreeNode *src = h.data() + ((size_t)r * m.K + k) * m.n_nodes;
            out[r][k].nodes.assign(src, src + m.n_nodes);
        }
    }
    return out;
}

template <typename T>
static std::vector<T> to_host(const T *p, size_t n) {
    std::vector<T> h(n);
    if (n) TGBM_CUDA(cudaMemcpy(h.data(), p, sizeof(T) * n, cudaMemcpyDeviceToHost));
    return h;
}

std::vector<float> Booster::get_metrics() { sync(); return to_host(impl_->metric.p, impl_->rounds); }
std::vector<float> Booster::get_ypred() { sync(); return to_host(impl_->ypred.p, (size_t)impl_->N * impl_->K); }
std::vector<float> Booster::get_cut_val() const { return impl_->h_cut_val; }
std::vector<int> Booster::get_cut_ptr() const { return impl_->h_cut_ptr; }
std::vector<unsigned char> Booster::get_bins() {
    sync();
    TGBM_CHECK(!impl_->sparse, "the booster holds the CSR layout: use get_bins_csr");
    const BoosterImpl &m = *impl_;
    if (m.S == m.F) return to_host(m.bins.p, (size_t)m.N * m.Fpad);
    const auto columns = to_host(m.binsT.p, (size_t)m.F * m.Npad);   // (several features share a byte of the other matrix)
    std::vector<unsigned char> rows((size_t)m.N * m.Fpad, MISSING_BIN);
    for (int f = 0; f < m.F; ++f)
        for (int r = 0; r < m.N; ++r) rows[(size_t)r * m.Fpad + f] = columns[(size_t)f * m.Npad + r];
    return rows;
}
std::vector<int> Booster::get_bins_csr() {
    sync();
    TGBM_CHECK(impl_->sparse, "the booster holds the dense layout: use get_bins");
    return to_host(impl_->sp_bin.p, (size_t)impl_->nnz_local);
}
bool Booster::is_sparse() const { return impl_->sparse; }
std::vector<int> Booster::get_nid() {
    sync();
    if (!impl_->p.keep_nid) return {};
    return to_host(impl_->nid_keep.p, (size_t)impl_->N * impl_->K * impl_->rounds);
}
std::vector<long long> Booster::get_root_hist() {
    sync();
    TGBM_CHECK(!impl_->f32, "fp32 mode keeps float histograms: use get_root_hist_f32");
    return to_host(impl_->hist_full.p + impl_->last_tree_full, (size_t)impl_->B * 2);
}
std::vector<float> Booster::get_root_hist_f32() {
    sync();
    TGBM_CHECK(impl_->f32, "exact mode keeps integer histograms: use get_root_hist");
    if (impl_->last_float) return to_host(reinterpret_cast<const float *>(impl_->hist_full.p + impl_->last_tree_full), (size_t)impl_->B * 2);
    const auto h = to_host(impl_->hist_full.p + impl_->last_tree_full, (size_t)impl_->B * 2);
    const QuantInfo q = to_host(impl_->qinfo.p, 1)[0];
    std::vector<float> out(h.size());
    for (size_t i = 0; i < h.size(); ++i) out[i] = (float)((double)h[i] * ((i & 1) ? q.inv_sh : q.inv_sg));
    return out;
}
std::vector<double> Booster::get_quant_scale() {
    sync();
    auto q = to_host(impl_->qinfo_log.p, impl_->rounds);
    std::vector<double> r;
    for (auto &v : q) { r.push_back(v.sg); r.push_back(v.sh); }
    return r;
}

}  // namespace tgbm
