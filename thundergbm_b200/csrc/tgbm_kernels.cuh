// CUDA kernels of the histogram tree builder (sm_100a).
//
// (the kernels of a tree level are in tgbm_level.cuh)
//
// Data layout in HBM (one rank = one contiguous block of rows):
//   bins   uint8 [N][Spad]   row-major bin ids by slot, Spad = slots rounded up to 32, 255 = missing.  A slot is a feature, or
//                            neighbouring features of which no row stores two (one-hot groups): its bins are theirs one after
//                            the other.  One 32-byte sector holds 32 slots of one row.
//   binsT  uint8 [F][Npad]   the same matrix column-major; read by k_assign, which
//                            needs one feature of many rows.
//   gh     float2 [K][N]     gradient pairs of the round, class-major like the reference.
//   ghq    int2   [K][N]     the same on the round's fixed-point grid.
//   nid    uint16 [N]        node of every row.
//   rec_idx [2N]             per-level row lists: rows grouped by tree node, roughly ascending inside a node.
//   hist   int64 [node][B][2] per-node histograms on the fixed-point grid.
//
// All sums on the fixed-point grid are integer sums, so they do not depend on the order of
// the atomics, on the CTA count or on the number of ranks.
#pragma once
#include <climits>

#include "tgbm_device.cuh"

namespace tgbm {

constexpr int HIST_THREADS = 1024;  // one CTA per SM: 64 KB of int32 accumulators + up to 128 KB of int64 totals
constexpr int ASSIGN_THREADS = 256, ASSIGN_CHUNK = 8 * ASSIGN_THREADS;   // rows that k_assign takes at a time, at most
constexpr int MISSING_BIN = 255;
constexpr int METRIC_PARTS = 1280;  // most partial sums of a round's metric (148 SMs x 8 blocks use 1184)
constexpr int FINE_BITS = 30;          // value bits of the grid of fp32 mode's later rounds
constexpr int FINE_WINDOW = 1 << 16;   // rows whose 16-bit low halves fit an unsigned accumulator
constexpr int FINE_FROM_ROUND = 1;     // fp32 mode: rounds before it sum floats value by value (k_hist_f32), and so do those that grid_too_coarse finds
constexpr int FINE_MEAN_BITS = 19;     // see grid_too_coarse

// Shares of the level's tiles per CTA of the dense histogram kernel: two when a CTA has HIST_SHARE_TILES tiles or more, else
// one.  Two balance the CTAs better (7 trees of 581 k rows side by side, 22 tiles per CTA: 50.6 ms per training against 52.6),
// but a CTA with few tiles then hands over the sums of twice as many nodes (1 M rows, 3 tiles per CTA: 54.3 ms against 52.2).
constexpr int HIST_SHARES = 2, HIST_SHARE_TILES = 8;

// Device copy of the booster's round counter: kernels whose work depends on the round read it here, so that the launch
// sequence of a round is the same every round and can be replayed as a CUDA graph.
struct RoundState {
    int round;
};

struct TreeCtl {  // device-side scalars of the booster
    unsigned long long stat_rows_root, stat_rows_gather, stat_hists, stat_part_rows;  // what the level kernels processed
    int error;   // non-zero when a bounded wait inside a kernel gave up; the host reads it after a sync
    int coarse;  // the running round's gradients do not fit the grid: scores, metric and round counter stay as they are
};

struct alignas(16) SplitRec {  // best candidate of one (node, feature)
    float gain;     // signed like the reference: negative = missing goes right
    int bin;        // local bin of the candidate, -1 = none
    float lg, lh;   // left sum without missing
    float mg, mh;   // missing sum of the feature in this node
    float value;    // where it splits
    int feature;
};

// ------------------------------------------------------------------ cut points
// key = feature id in the high word, order-preserving image of the float in the low word
static __global__ void k_make_keys(const float *__restrict__ val, const int *__restrict__ col, int full_cols, size_t nnz,
                            unsigned long long *__restrict__ keys) {
    // full_cols > 0: a matrix without missing values, `col` is not read
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nnz; i += (size_t)gridDim.x * blockDim.x) {
        unsigned u = __float_as_uint(val[i]);
        if (u == 0x80000000u) u = 0;  // -0.0f == 0.0f
        u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        const unsigned c = full_cols ? (unsigned)i % (unsigned)full_cols : (unsigned)col[i];
        keys[i] = ((unsigned long long)c << 32) | u;
    }
}

__device__ inline float key_to_float(unsigned long long k) {
    unsigned u = (unsigned)(k & 0xffffffffull);
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(u);
}

// ustart[f] = number of unique (feature,value) keys with feature < f
static __global__ void k_feature_bounds(const unsigned long long *__restrict__ ukeys, long long nu, int F, long long *__restrict__ ustart) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f > F) return;
    const unsigned long long target = (unsigned long long)(unsigned)f << 32;
    long long lo = 0, hi = nu;
    while (lo < hi) {
        const long long mid = lo + (hi - lo) / 2;
        if (ukeys[mid] < target) lo = mid + 1; else hi = mid;
    }
    ustart[f] = lo;
}

// HistCut::get_cut_points_single (src/thundergbm/hist_cut.cu:232-286): stride s = u / max_bin;
// s == 0 keeps every distinct value, else positions 0, s, ..., (max_bin-1) s
static __global__ void k_select_cuts(const unsigned long long *__restrict__ ukeys, long long nu, const long long *__restrict__ ustart,
                              const int *__restrict__ stride, const int *__restrict__ cut_ptr, int max_bin,
                              float *__restrict__ cut_val, int *__restrict__ cut_fid, int down) {
    // down: the keys carry the complement of the float's ordered image (candidates of the column-sharded builder,
    // largest value first)
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nu; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = ukeys[i];
        const int f = (int)(k >> 32);
        const long long t = i - ustart[f];
        const int s = stride[f];
        long long pos;
        if (s == 0) pos = t;
        else if (t % s == 0 && t / s < max_bin) pos = t / s;
        else continue;
        cut_val[cut_ptr[f] + pos] = key_to_float(down ? (k ^ 0xffffffffull) : k);
        cut_fid[cut_ptr[f] + pos] = f;
    }
}

// ------------------------------------------------------------------ cut points of the column-sharded builder
// HistCut::get_cut_points3 + unique_by_flag (src/thundergbm/hist_cut.cu:104-187), which every device of the
// reference runs on its own block of columns: each stored value v of local column j becomes t = v + j*(m+1), m the
// largest value on the device; all t of the device are sorted descending; the column ids are laid over the sorted
// array by COUNT, largest id first; runs of equal t keep their first entry; t goes back to t - j*(m+1) with the id
// found there.  Done here on the distinct (feature, value) keys with their multiplicities: the position of a key's
// first copy in the reference's sorted array is the number of copies before it.
struct ColumnShift {            // per feature
    int shard, first;           // device that owns it in the reference, first column of that device
    float step;                 // m + 1 of that device
    long long below;            // copies in the device's columns with a LARGER id: where this column's ids start
};
__device__ __forceinline__ unsigned float_order(float v) {
    unsigned u = __float_as_uint(v);
    if (u == 0x80000000u) u = 0;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float order_float(unsigned u) {
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(u);
}
// key (feature, value) -> (device, complement of the ordered image of t): ascending keys = descending t per device
static __global__ void k_shift_keys(const unsigned long long *__restrict__ ukeys, long long nu, const ColumnShift *__restrict__ cs,
                                    unsigned long long *__restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nu; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = ukeys[i];
        const int f = (int)(k >> 32);
        const ColumnShift c = cs[f];
        const float v = key_to_float(k), j = (float)(f - c.first);
        const float t = __fmaf_rn(j, c.step, v);  // one rounding: what nvcc makes of the reference's `v + j * step`
        out[i] = ((unsigned long long)(unsigned)c.shard << 32) | (unsigned)~float_order(t);
    }
}
// sorted shifted keys + the number of copies before each -> candidate keys (feature, complement of the ordered image of
// the value shifted back), all-ones for the entries that unique_by_key drops
static __global__ void k_unshift_keys(const unsigned long long *__restrict__ skeys, const long long *__restrict__ before, long long nu,
                                      const ColumnShift *__restrict__ cs, const int *__restrict__ shard_first,
                                      const int *__restrict__ shard_cols, const long long *__restrict__ shard_before,
                                      unsigned long long *__restrict__ out, unsigned long long *__restrict__ n_heads) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nu; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = skeys[i];
        if (i > 0 && skeys[i - 1] == k) { out[i] = ~0ull; continue; }
        const int d = (int)(k >> 32), first = shard_first[d];
        const long long pos = before[i] - shard_before[d];
        int lo = 0, hi = shard_cols[d] - 1;  // smallest local id whose ids start at or before pos (`below` falls as the id grows)
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (cs[first + mid].below <= pos) hi = mid; else lo = mid + 1;
        }
        const float t = order_float(~(unsigned)(k & 0xffffffffull)), j = (float)lo, step = cs[first + lo].step;
        const float v = __fmaf_rn(-j, step, t);
        out[i] = ((unsigned long long)(unsigned)(first + lo) << 32) | (unsigned)~float_order(v);
        atomicAdd(n_heads, 1ull);
    }
}
static __global__ void k_fill_ll(long long *p, size_t n, long long v) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}
// per feature: largest stored value (the last of its ascending keys) and the number of copies before its first key
static __global__ void k_feature_max_before(const unsigned long long *__restrict__ ukeys, const long long *__restrict__ ustart,
                                            const long long *__restrict__ before, long long nu, long long total, int F,
                                            float *__restrict__ fmax, long long *__restrict__ fbefore) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f > F) return;
    const long long a = ustart[f];
    fbefore[f] = a < nu ? before[a] : total;
    if (f < F) fmax[f] = ustart[f + 1] > a ? key_to_float(ukeys[ustart[f + 1] - 1]) : -INFINITY;
}

// HistTreeBuilder::get_bin_ids of the column-sharded builder (hist_tree_builder.cu:31-49): the cut points of a
// feature descend there; first position in [lo, hi] whose cut is <= v, hi when there is none
__device__ __forceinline__ int bin_search_down(const float *__restrict__ cut_val, int lo, int hi, float v) {
    while (lo != hi) {
        const int mid = lo + (hi - lo) / 2;
        if (cut_val[mid] <= v) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// HistTreeBuilder_single::get_bin_ids (hist_tree_builder_single.cu:81-119): clamped upper bound,
// bin = min(#cuts <= v, n_cuts - 1); stored as the feature-local id in both layouts
static __global__ void k_bin_dense(const int *__restrict__ row_ptr, const int *__restrict__ col, const float *__restrict__ val,
                            int full_cols, int n_rows, const int *__restrict__ cut_ptr, const float *__restrict__ cut_val, int Fpad,
                            size_t Npad, unsigned char *__restrict__ bins, unsigned char *__restrict__ binsT, int multi) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const int j0 = full_cols ? r * full_cols : row_ptr[r], j1 = full_cols ? j0 + full_cols : row_ptr[r + 1];
    for (int j = j0; j < j1; ++j) {
        const int f = full_cols ? j - j0 : col[j];
        const float v = val[j];
        const int b0 = cut_ptr[f];
        int lo = b0, hi = cut_ptr[f + 1] - 1;
        if (hi < lo) continue;
        if (multi) lo = bin_search_down(cut_val, lo, hi, v);
        else
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (cut_val[mid] <= v) lo = mid + 1; else hi = mid;
        }
        const unsigned char b = (unsigned char)(lo - b0);
        bins[(size_t)r * Fpad + f] = b;
        binsT[(size_t)f * Npad + r] = b;
    }
}

// The same with the cut points in shared memory.  (Above, neighbouring lanes read values a row apart and search the cut points
// through L1, a line per lane and step: 10.5 M full rows x 28 take 2.9 ms there and 1.1 here, 300 k CSR rows x 136 1.3 ms and 0.2.)
// The cut points of a feature are laid out as an implicit search tree of 255 nodes, level by level and padded with +inf; eight
// steps lead to the number of cut points <= v.
constexpr int BIN_TREE = 257;   // words from feature to feature: lanes on neighbouring features meet on different banks
__device__ __forceinline__ void bin_trees(const int *__restrict__ cut_ptr, const float *__restrict__ cut_val, int f0, int nf, float *tree) {
    for (int i = threadIdx.x; i < nf * 255; i += blockDim.x) {
        const int f = i / 255, k = i - f * 255, lv = 31 - __clz(k + 1), q = k + 1 - (1 << lv), mid = (2 * q + 1) * (128 >> lv) - 1, c = cut_ptr[f0 + f] + mid;
        tree[f * BIN_TREE + k] = c < cut_ptr[f0 + f + 1] ? cut_val[c] : INFINITY;
    }
}
__device__ __forceinline__ unsigned bin_of(const float *tree, int n, float v) {   // n: cut points; 255 if there are none
    int pos = 0;
#pragma unroll
    for (int step = 0; step < 8; ++step) pos = 2 * pos + (tree[pos] <= v ? 2 : 1);   // (a NaN goes to the first bin)
    return n ? (unsigned)min(pos - 255, n - 1) : (unsigned)MISSING_BIN;
}
// every value stored: a thread takes 32 features of a row; grid = (blocks, groups of 32).  VEC: rows on 16-byte boundaries
template <bool VEC>
static __global__ void __launch_bounds__(256)
k_bin_full(const float *__restrict__ val, int n_rows, int F, const int *__restrict__ cut_ptr, const float *__restrict__ cut_val, int Fpad, size_t Npad,
           unsigned char *__restrict__ bins, unsigned char *__restrict__ binsT) {
    __shared__ float tree[32 * BIN_TREE];
    __shared__ int cuts[32];
    const int f0 = blockIdx.y * 32, nf = min(32, F - f0);
    bin_trees(cut_ptr, cut_val, f0, nf, tree);
    if (threadIdx.x < nf) cuts[threadIdx.x] = cut_ptr[f0 + threadIdx.x + 1] - cut_ptr[f0 + threadIdx.x];
    __syncthreads();
    for (int r = blockIdx.x * 256 + threadIdx.x; r < n_rows; r += gridDim.x * 256) {
        const float *row = val + (size_t)r * F + f0;
        uint32_t w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            w[q] = 0xffffffffu;
            if (4 * q >= nf) continue;
            float v[4];
            if (VEC) {   // (F is a multiple of four, so is what is left of it)
                const float4 x = reinterpret_cast<const float4 *>(row)[q];
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = 4 * q + k < nf ? row[4 * q + k] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int f = 4 * q + k;
                if (f >= nf) continue;
                const unsigned b = bin_of(tree + f * BIN_TREE, cuts[f], v[k]);
                w[q] = (w[q] & ~(0xffu << (8 * k))) | (b << (8 * k));
                binsT[(size_t)(f0 + f) * Npad + r] = (unsigned char)b;
            }
        }
        uint4 *to = reinterpret_cast<uint4 *>(bins + (size_t)r * Fpad + f0);
        to[0] = make_uint4(w[0], w[1], w[2], w[3]);
        to[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}
// CSR rows: a warp per row, lanes over its values, row-major only (k_bins_by_column follows); `bins` comes filled with 255.
// Of a column that a row stores twice the last value counts, as above.  While the row's columns ascend no two lanes meet; from
// the first window on where they do not, windows are stored one after the other, and of lanes with the same column the last stores.
constexpr int BIN_ROWS_SMEM = 220 * 1024;
static __global__ void __launch_bounds__(1024, 1)
k_bin_rows(const int *__restrict__ row_ptr, const int *__restrict__ col, const float *__restrict__ val, int n_rows, int F, const int *__restrict__ cut_ptr,
           const float *__restrict__ cut_val, int Fpad, unsigned char *__restrict__ bins) {
    extern __shared__ float bin_sm[];   // [F][BIN_TREE], then the numbers of cut points
    int *cuts = reinterpret_cast<int *>(bin_sm + (size_t)F * BIN_TREE);
    bin_trees(cut_ptr, cut_val, 0, F, bin_sm);
    for (int f = threadIdx.x; f < F; f += 1024) cuts[f] = cut_ptr[f + 1] - cut_ptr[f];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    constexpr int U = 2;   // values in flight per lane
    for (int r = blockIdx.x * 32 + (threadIdx.x >> 5); r < n_rows; r += gridDim.x * 32) {
        const int j1 = row_ptr[r + 1];
        int last = -1;   // column before the window
        bool ascend = true;
        each_step(row_ptr[r], j1, 0, 32 * U, [&](unsigned j0) {   // (the same in the whole warp)
            int c[U];
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const unsigned j = j0 + 32 * u + lane;
                c[u] = j < (unsigned)j1 ? col[j] : INT_MAX;
                v[u] = j < (unsigned)j1 ? val[j] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool stored = c[u] != INT_MAX;
                const int left = __shfl_up_sync(0xffffffffu, c[u], 1);
                ascend = ascend && __all_sync(0xffffffffu, !stored || c[u] > (lane ? left : last));
                last = __shfl_sync(0xffffffffu, c[u], 31);
                const unsigned char b = stored ? (unsigned char)bin_of(bin_sm + c[u] * BIN_TREE, cuts[c[u]], v[u]) : (unsigned char)0;
                bool mine = stored;
                if (!ascend) {
                    const unsigned same = __match_any_sync(0xffffffffu, c[u]);
                    mine = mine && same >> lane == 1u;
                    __syncwarp();   // what earlier windows stored comes before
                }
                if (mine) bins[(size_t)r * Fpad + c[u]] = b;
            }
        });
    }
}
// bins [row][feature] -> binsT [feature][row], to the end of the padded rows; a block transposes 128 rows of 32 features
static __global__ void __launch_bounds__(256)
k_bins_by_column(const unsigned char *__restrict__ bins, int n_rows, int F, int Fpad, size_t Npad, unsigned char *__restrict__ binsT) {
    __shared__ __align__(4) unsigned char t[32][132];   // (read four bytes at a time)
    const int f0 = blockIdx.y * 32;
    const size_t r0 = (size_t)blockIdx.x * 128;
    {
        const int r = threadIdx.x >> 1, half = threadIdx.x & 1;
        uint4 v = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        if (r0 + r < (size_t)n_rows) v = *reinterpret_cast<const uint4 *>(bins + (r0 + r) * Fpad + f0 + 16 * half);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 16; ++k) t[16 * half + k][r] = (unsigned char)(w[k >> 2] >> (8 * (k & 3)));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * 32; i += 256) {   // (Npad is a multiple of 128)
        const int f = i >> 5, q = i & 31;
        if (f0 + f < F) *reinterpret_cast<uint32_t *>(binsT + (size_t)(f0 + f) * Npad + r0 + 4 * q) = *reinterpret_cast<const uint32_t *>(&t[f][4 * q]);
    }
}

// Neighbouring features of which no row stores two may share a byte of the row-major matrix (exclusive feature bundling, Ke et
// al., "LightGBM", NIPS 2017, section 4, without its tolerance for conflicts).  last[f] = the largest feature below f that a row
// with a value of f stores as well, -1 if none: [a, f] may share a byte if last is below a for all of them but a.
static __global__ void __launch_bounds__(256)
k_last_before(const unsigned char *__restrict__ bins, int n_rows, int Fpad, int F, int *__restrict__ last) {
    extern __shared__ int s_last[];   // [F]
    for (int f = threadIdx.x; f < F; f += 256) s_last[f] = -1;
    __syncthreads();
    for (int r = blockIdx.x * 256 + threadIdx.x; r < n_rows; r += gridDim.x * 256) {
        const uint4 *row = reinterpret_cast<const uint4 *>(bins + (size_t)r * Fpad);
        int before = -1;
        for (int q = 0; q < Fpad / 16; ++q) {
            const uint4 v = row[q];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                if (((w[k >> 2] >> (8 * (k & 3))) & 0xffu) == MISSING_BIN) continue;
                const int f = q * 16 + k;
                if (before > *(volatile int *)&s_last[f]) atomicMax(&s_last[f], before);
                before = f;
            }
        }
    }
    __syncthreads();
    for (int f = threadIdx.x; f < F; f += 256)
        if (s_last[f] >= 0) atomicMax(last + f, s_last[f]);
}
// the matrix by slot: feature f's bins start at `shift[f]` of slot `slot[f]`
static __global__ void __launch_bounds__(256)
k_bundle(const unsigned char *__restrict__ bins, int n_rows, int Fpad, int F, const int *__restrict__ slot, const int *__restrict__ shift, int Spad,
         unsigned char *__restrict__ out) {
    for (int r = blockIdx.x * 256 + threadIdx.x; r < n_rows; r += gridDim.x * 256) {
        const unsigned char *row = bins + (size_t)r * Fpad;
        unsigned char *to = out + (size_t)r * Spad;
        for (int f = 0; f < F; ++f)
            if (row[f] != MISSING_BIN) to[slot[f]] = (unsigned char)(row[f] + shift[f]);
    }
}

// Wide sparse data: the reference's own layout, one global bin id per stored value
// (hist_tree_builder_single.cu:113-119), sharing the CSR row pointers.
static __global__ void k_bin_csr(const int *__restrict__ col, const float *__restrict__ val, size_t nnz,
                                 const int *__restrict__ cut_ptr, const float *__restrict__ cut_val, int *__restrict__ out, int multi) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nnz; i += (size_t)gridDim.x * blockDim.x) {
        const int f = col[i];
        const float v = val[i];
        int lo = cut_ptr[f], hi = cut_ptr[f + 1] - 1;
        if (multi) lo = bin_search_down(cut_val, lo, hi, v);
        else
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (cut_val[mid] <= v) lo = mid + 1; else hi = mid;
        }
        out[i] = lo;
    }
}

// flag = 1 when some row's bin ids do not ascend (k_assign looks a feature up by binary search inside the row)
static __global__ void k_rows_unsorted(const int *__restrict__ row_ptr, const int *__restrict__ bin, int n_rows, int *__restrict__ flag) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        bool bad = false;
        for (int i = row_ptr[r] + 1; i < row_ptr[r + 1]; ++i) bad |= bin[i - 1] > bin[i];
        if (bad) *flag = 1;
    }
}

// flag = 1 when some row stores a column twice (bin ids ascend inside a row)
static __global__ void k_rows_repeat(const int *__restrict__ row_ptr, const int *__restrict__ bin, const int *__restrict__ cut_fid, int n_rows, int *__restrict__ flag) {
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += (gridDim.x * blockDim.x) >> 5) {
        bool bad = false;
        each_step(row_ptr[r], row_ptr[r + 1], 1 + lane, 32, [&](unsigned i) { bad |= cut_fid[bin[i - 1]] == cut_fid[bin[i]]; });
        if (bad) *flag = 1;
    }
}
// row of every stored value (CSR order)
static __global__ void k_value_rows(const int *__restrict__ row_ptr, int n_rows, int *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += (gridDim.x * blockDim.x) >> 5)
        each_step(row_ptr[r], row_ptr[r + 1], lane, 32, [&](unsigned j) { out[j] = r; });
}
// bin_ptr[x] = first of the sorted bin ids that is x or larger
static __global__ void k_bin_starts(const int *__restrict__ bin, int n, int n_bins, int *__restrict__ bin_ptr) {
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x <= n_bins; x += gridDim.x * blockDim.x) {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (bin[mid] < x) lo = mid + 1; else hi = mid;
        }
        bin_ptr[x] = lo;
    }
}

// y[i] <- index of y[i] among the ascending `label` values, 0 when it is not one of them
// (DataSet::group_label, src/thundergbm/dataset.cpp:83-101)
static __global__ void k_map_labels(float *__restrict__ y, int n, const float *__restrict__ label, int n_label) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = y[i];
        int lo = 0, hi = n_label;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (label[mid] < v) lo = mid + 1; else hi = mid;
        }
        y[i] = (lo < n_label && label[lo] == v) ? (float)lo : 0.f;
    }
}

// ------------------------------------------------------------------ objectives
// block-wide maximum of |g| and h, then one atomic pair per block (every thread of the block must call it)
__device__ inline void track_max(float ag, float h, unsigned *maxbits) {
    // non-negative floats order like their bit patterns
    __shared__ unsigned smax[2][32];
    unsigned a = __float_as_uint(ag), b = __float_as_uint(h);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) { smax[0][warp] = a; smax[1][warp] = b; }
    __syncthreads();
    if (warp == 0) {
        a = lane < nw ? smax[0][lane] : 0u;
        b = lane < nw ? smax[1][lane] : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        if (lane == 0) { atomicMax(maxbits, a); atomicMax(maxbits + 1, b); }
    }
}

// SquareLoss / LogisticLoss gradients (include/thundergbm/objective/regression_obj.h:129-154)
__device__ __forceinline__ float2 pointwise_gh(int logistic, float y, float yp) {
    if (logistic) {
        const float p = __fdiv_rn(1.0f, __fadd_rn(1.0f, portable_expf(-yp)));
        return make_float2(__fsub_rn(p, y), fmaxf(__fmul_rn(p, __fsub_rn(1.0f, p)), 1e-16f));
    }
    return make_float2(__fsub_rn(yp, y), 1.0f);
}

// one row's term of the training metric: squared error (pointwise_metric.cu:8-22), or 1 for a correct binary
// prediction (multiclass_metric.cu:9-46: sigmoid evaluated in double, class 1 above 0.5)
__device__ __forceinline__ double pointwise_metric_term(int objective, float y, float yp) {
    if (objective == BINARY_LOGISTIC) {
        // sigmoid(x) > 0.5 is decided by the sign of x except within rounding distance of zero
        const int k = fabsf(yp) > 1e-8f ? (yp > 0.f ? 1 : 0) : ((1.0 / (1.0 + exp(-(double)yp)) > 0.5) ? 1 : 0);
        return ((float)k == y) ? 1.0 : 0.0;
    }
    const float e = __fsub_rn(yp, y);
    return (double)__fmul_rn(e, e);
}

static __global__ void k_grad_pointwise(const float *y, const float *yp, int n, int logistic,
                                 float2 *gh, unsigned *maxbits) {
    chain_wait();
    float mg = 0.f, mh = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float2 v = pointwise_gh(logistic, y[i], yp[i]);
        const float g = v.x, h = v.y;
        gh[i] = make_float2(g, h);
        mg = fmaxf(mg, fabsf(g)); mh = fmaxf(mh, h);
    }
    track_max(mg, mh, maxbits);
}

// Softmax::get_gradient (src/thundergbm/objective/multiclass_obj.cu:7-35), class-major gh[k*N+i]
static __global__ void k_grad_softmax(const float *y, const float *yp, int n, int K,
                               float2 *gh, unsigned *maxbits) {
    chain_wait();
    float mg = 0.f, mh = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float mx = yp[i];
        for (int k = 1; k < K; ++k) mx = fmaxf(mx, yp[(size_t)k * n + i]);
        float sum = 0.f;
        for (int k = 0; k < K; ++k) sum = __fadd_rn(sum, portable_expf(__fsub_rn(yp[(size_t)k * n + i], mx)));
        const float yi = y[i];
        for (int k = 0; k < K; ++k) {
            const float p = __fdiv_rn(portable_expf(__fsub_rn(yp[(size_t)k * n + i], mx)), sum);
            const float g = ((float)k == yi) ? __fsub_rn(p, 1.0f) : p;
            const float h = fmaxf(__fmul_rn(__fmul_rn(2.0f, p), __fsub_rn(1.0f, p)), 1e-16f);
            gh[(size_t)k * n + i] = make_float2(g, h);
            mg = fmaxf(mg, fabsf(g));
            mh = fmaxf(mh, h);
        }
    }
    track_max(mg, mh, maxbits);
}

// Round the round's gradients to the fixed-point grid and sum them per class (root node sums,
// Tree::init2, src/thundergbm/tree.cu:31).  grid = (blocks, K)
//
// The rounding is dithered, q = floor(v * scale + u) with u in [0,1) a hash of (round, class, global row):
// round-to-nearest would move every row that carries the same gradient the same way (in the first round all rows
// of a class do), and those shifts would add up coherently in the histogram sums.
//
// FINE (fp32 mode from the second round on, FINE_BITS value bits): rounded to nearest, so a value moves by at most 2^-30 of
// the round's largest one, however small it is itself.  What that means for the sums depends on the spread of the values: `spread` (behind the root
// sums) collects what grid_too_coarse decides by.
//
// `gh` null: the gradients are those of a pointwise objective (`logistic` 0/1) and are computed again from y and the
// scores here -- the pass that found their maxima (k_apply_tree) did not store them.
template <bool FINE>
static __global__ void __launch_bounds__(256, 8)   // (the grid is one full wave of eight blocks per SM)
k_quantize(const float2 *gh, int n, const unsigned *maxbits, int quant_bits,
                           uint32_t round, uint32_t row_offset, int2 *ghq,
                           unsigned long long *root_sum, QuantInfo *qinfo,
                           const float *y, const float *yp, int logistic,
                           const RoundState *rs, unsigned long long *spread) {
    chain_wait();
    if (rs) round = (uint32_t)rs->round;  // the booster's rounds; the base-score pass gives its own
    const int k = blockIdx.y;
    const int eg = exp_above(__uint_as_float(maxbits[0])), eh = exp_above(__uint_as_float(maxbits[1]));
    const double sg = pow2d(quant_bits - eg), sh = pow2d(quant_bits - eh);
    if (blockIdx.x == 0 && k == 0 && threadIdx.x == 0) {
        qinfo->sg = sg; qinfo->sh = sh;
        qinfo->inv_sg = pow2d(eg - quant_bits); qinfo->inv_sh = pow2d(eh - quant_bits);
    }
    const bool in_float = sg < 1e38 && sh < 1e38;
    const float fg = (float)sg, fh = (float)sh;
    unsigned long long rounded = 0;
    bool bad = false;
    long long tg = 0, th = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float2 v = gh ? gh[(size_t)k * n + i] : pointwise_gh(logistic, y[i], yp[i]);
        int qg, qh;
        if (FINE) {
            // the scale is a power of two: where a float holds it, the product is exact in float, and the conversions to and from
            // double (a sixteenth of the float rate) can go
            bool off;   // the gradient is not on the grid (one of 23 bits and more counts as if it were)
            if (in_float) {
                const float pg = __fmul_rn(v.x, fg);
                qg = __float2int_rn(pg); qh = __float2int_rn(__fmul_rn(v.y, fh));
                off = fabsf(pg) < 4194304.f && __fadd_rn(__fadd_rn(pg, 12582912.f), -12582912.f) != pg;
            } else {
                const double pg = (double)v.x * sg;
                qg = __double2int_rn(pg); qh = __double2int_rn((double)v.y * sh);
                off = (double)qg != pg;
            }
            if (off) rounded += (unsigned)qh >> (31 - __clz(abs(qg) | 1));
            bad |= !(fabsf(v.x) + v.y < INFINITY);   // (hessians are not negative)
        } else {
        const uint32_t row = row_offset + (uint32_t)i;
        const double ug = (double)mix32(0x9E3779B9u, round, (uint32_t)k, row) * (1.0 / 4294967296.0);
        const double uh = (double)mix32(0x9E3779B9u + 1u, round, (uint32_t)k, row) * (1.0 / 4294967296.0);
        qg = (int)__double2ll_rd((double)v.x * sg + ug); qh = (int)__double2ll_rd((double)v.y * sh + uh);
        }
        ghq[(size_t)k * n + i] = make_int2(qg, qh);
        tg += qg; th += qh;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { tg += shfl_xor_ll(tg, o); th += shfl_xor_ll(th, o); }
    if (FINE && __any_sync(0xffffffffu, rounded != 0 || bad)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rounded += (unsigned long long)shfl_xor_ll((long long)rounded, o);
        bad = __any_sync(0xffffffffu, bad);
    }
    // one pair of atomics per block: all go to the same two words, and one pair per warp made 19 k of them at 1 M rows, 12 of
    // the kernel's 19 us
    __shared__ long long part[4][8];
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = tg; part[1][threadIdx.x >> 5] = th;
        if (FINE) { part[2][threadIdx.x >> 5] = (long long)rounded; part[3][threadIdx.x >> 5] = bad; }
    }
    __syncthreads();
    if (threadIdx.x < (FINE ? 4 : 2)) {
        long long t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[threadIdx.x][w];
        if (threadIdx.x < 2) atomicAdd(root_sum + 2 * k + threadIdx.x, (unsigned long long)t);
        else if (t) atomicAdd(spread + threadIdx.x - 2, (unsigned long long)t);
    }
}

// Is the grid of a fine round too coarse for its gradients?  Called by one thread, after k_quantize and the ranks' sums.
//
// root_sum[2 K]: 2 * hessian * 2^-bits summed over the gradients that the grid had to round, bits = those left of the value.
// 2^-bits bounds the relative error of a gradient, the hessian is the row's weight in -sum g / (sum h + lambda): divided by
// the sum of all hessians it is the mean relative error of what the leaf weights are made of.  On normal residuals with a few
// outliers, integer and float sums were both compared with float64 on the same gradients: the weights of the nodes without
// outliers are at least as good from the integers down to 2^-18 for 4 k rows (outliers 300 times the rest; their error in
// units of 2^-24 of the rms gradient, rms over the nodes: 0.4 against 1.3; 1.0 against 0.4 at 2^-16.7), down to 2^-15 for
// 400 k rows.  Lambda gradients come to 2^-21 to 2^-23, everything else of ordinary data to 2^-28 and less, since most
// gradients are multiples of the grid; one label of 1e9 among normal ones to 2^-1.
// Hessians need no such test: sum h + lambda loses at most 2^-31 of the largest per row, the float sums lose 2^-24 of the
// node's whole sum to one of its children (what the node's sum and the sum over its bins differ by counts as missing rows).
// root_sum[2 K + 1]: not zero if a gradient is not finite.  One is enough: float sums carry it on, the grid does not.
__device__ inline bool grid_too_coarse(const unsigned long long *root_sum, int K) {
    unsigned long long h = 0;
    for (int k = 0; k < K; ++k) h += root_sum[2 * k + 1];
    return root_sum[2 * K + 1] != 0 || root_sum[2 * K] > h >> (FINE_MEAN_BITS - 1);
}
// the same for a round that is not built yet
static __global__ void k_grid_check(const unsigned long long *root_sum, int K, TreeCtl *ctl) {
    if (grid_too_coarse(root_sum, K)) ctl->coarse = 1;
}


// ------------------------------------------------------------------ row and column sampling
// RowSampler::do_bagging (src/thundergbm/row_sampler.cu:9-35): M = size of the gradient array (num_class x rows) draws
// of a uniform index into that array, every entry's (g,h) multiplied by the number of times it was drawn.  The
// reference seeds thrust's generator from std::rand(); here draw j of round r is a counter-based hash, so that the
// CPU restatement and any number of ranks draw the same sample.  Every rank makes all the draws and keeps those that
// land in its own rows.  entry = class * n_global + global row.
static __global__ void k_bag_draw(unsigned long long m_total, uint32_t seed, const RoundState *__restrict__ rs, long long n_global,
                                  long long row_offset, int n_local, int K, int *__restrict__ count) {
    const uint32_t round = (uint32_t)rs->round;
    for (unsigned long long j = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; j < m_total; j += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t r = mix32(seed ^ 0xBA661D6Eu, round, (uint32_t)(j >> 32), (uint32_t)j);
        const unsigned long long e = ((unsigned long long)r * m_total) >> 32;
        const long long k = (long long)(e / (unsigned long long)n_global), row = (long long)(e % (unsigned long long)n_global) - row_offset;
        if (k < K && row >= 0 && row < n_local) atomicAdd(count + k * n_local + row, 1);
    }
}
// gh *= multiplicity; also the maxima of the scaled gradients for the fixed-point grid (every thread of the block calls track_max)
static __global__ void k_bag_scale(float2 *__restrict__ gh, const int *__restrict__ count, size_t n, unsigned *__restrict__ maxbits) {
    float mg = 0.f, mh = 0.f;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float2 v = gh[i];
        const float c = (float)count[i];
        v.x = __fmul_rn(v.x, c); v.y = __fmul_rn(v.y, c);
        gh[i] = v;
        mg = fmaxf(mg, fabsf(v.x)); mh = fmaxf(mh, v.y);
    }
    track_max(mg, mh, maxbits);
}

// ------------------------------------------------------------------ tree set-up
// The quantisation has used the round's maxima; those of the next round's gradients are collected from zero -- unless the
// round will be built again, on the same gradients.  fine_K > 0: the first trees of a fine round of fine_K trees.
__device__ inline void next_maxima(const unsigned long long *root_sum, int fine_K, unsigned *maxbits, TreeCtl *ctl) {
    const bool again = ctl->coarse, now = fine_K && grid_too_coarse(root_sum, fine_K);
    if (now) ctl->coarse = 1;
    if (!again && !now) maxbits[0] = maxbits[1] = 0;
}

// Tree::init2 (src/thundergbm/tree.cu:8-39)
// root_is_f64: fp32 mode, the root sums are doubles (k_sum_gh_final) instead of integers on the fixed-point grid
// grid.y = trees of the batch; seg tables: the root holds every row
static __global__ void k_tree_init(TreeNode *nodes, int n_nodes, const unsigned long long *root_sum,
                            const QuantInfo *q, float lambda, int n_rows, int *seg_begin,
                            int *seg_cnt, size_t seg_stride, int root_is_f64, unsigned *maxbits, int fine_K, TreeCtl *ctl) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && blockIdx.y == 0) next_maxima(root_sum, fine_K, maxbits, ctl);
    if (i >= n_nodes) return;
    const size_t tree = blockIdx.y;
    root_sum += 2 * tree;
    TreeNode t;
    memset(&t, 0, sizeof(t));
    t.final_id = i;
    t.split_feature_id = -1;
    t.parent_index = i == 0 ? -1 : (i - 1) / 2;
    if (i < n_nodes / 2) { t.is_leaf = 0; t.lch_index = 2 * i + 1; t.rch_index = 2 * i + 2; }
    else { t.is_leaf = 1; t.lch_index = -1; t.rch_index = -1; }
    if (i == 0) {
        if (root_is_f64) {
            t.sum_g = __double2float_rn(__longlong_as_double((long long)root_sum[0]));
            t.sum_h = __double2float_rn(__longlong_as_double((long long)root_sum[1]));
        } else {
            t.sum_g = q2f((long long)root_sum[0], q->inv_sg);
            t.sum_h = q2f((long long)root_sum[1], q->inv_sh);
        }
        t.is_valid = 1;
        t.base_weight = __fdiv_rn(-t.sum_g, __fadd_rn(t.sum_h, lambda));
        seg_begin[tree * seg_stride] = 0; seg_cnt[tree * seg_stride] = n_rows;
    }
    nodes[tree * n_nodes + i] = t;
}

// Exclusive prefix sums over n values inside one block of 1024 threads: out(i, prefix before i); returns the total.
// `scratch` holds 33 ints of shared memory.  Every thread of the block must call it.
template <typename In, typename Out>
__device__ inline int block_scan_excl(int n, In in, Out out, int *scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const int x = i < n ? in(i) : 0;
        int v = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
        __syncthreads();
        if (lane == 31) scratch[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int t = scratch[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, t, o); if (lane >= o) t += u; }
            scratch[lane] = t;
        }
        __syncthreads();
        const int incl = v + (warp ? scratch[warp - 1] : 0) + carry;
        if (i < n) out(i, incl - x);
        carry += scratch[31];
    }
    __syncthreads();
    return carry;
}

// ------------------------------------------------------------------ cut points of a matrix without missing values
// Every column is sorted for itself: 32-bit keys instead of 64-bit ones that carry the column, and four passes over them
// instead of five; distinct values are then counted and picked where they lie instead of being compacted first.
constexpr int COL_CHUNK = 4096;   // sorted keys per block

// values [n][c] -> order-preserving images by column [c][n]; a block transposes 64 rows of 32 columns
static __global__ void __launch_bounds__(256)
k_order_columns(const float *__restrict__ val, int n, int c, unsigned *__restrict__ out) {
    __shared__ unsigned t[64][33];
    const int r0 = blockIdx.x * 64, c0 = blockIdx.y * 32;
    for (int i = threadIdx.x; i < 64 * 32; i += 256) {
        const int r = r0 + (i >> 5), f = c0 + (i & 31);
        if (r < n && f < c) {
            unsigned u = __float_as_uint(val[(size_t)r * c + f]);
            if (u == 0x80000000u) u = 0;  // -0.0f == 0.0f
            t[i >> 5][i & 31] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 64 * 32; i += 256) {
        const int r = r0 + (i & 63), f = c0 + (i >> 6);
        if (r < n && f < c) out[(size_t)f * n + r] = t[i & 63][i >> 6];
    }
}

// distinct values that start in every chunk of a sorted column; grid = (chunks, columns)
static __global__ void __launch_bounds__(256)
k_column_heads(const unsigned *__restrict__ keys, int n, int *__restrict__ heads) {
    const unsigned *k = keys + (size_t)blockIdx.y * n;
    int cnt = 0;
    for (int u = 0; u < COL_CHUNK / 256; ++u) {
        const int i = blockIdx.x * COL_CHUNK + u * 256 + threadIdx.x;
        cnt += i < n && (i == 0 || k[i] != k[i - 1]);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    __shared__ int w[8];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int i = 0; i < 8; ++i) t += w[i];
        heads[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
    }
}

// exclusive prefix over the chunks of a column in place, and its number of distinct values; one block of 1024 threads each
static __global__ void __launch_bounds__(1024)
k_column_prefix(int *__restrict__ heads, int chunks, int *__restrict__ distinct) {
    __shared__ int scratch[33];
    int *h = heads + (size_t)blockIdx.x * chunks;
    const int total = block_scan_excl(chunks, [&](int i) { return h[i]; }, [&](int i, int before) { h[i] = before; }, scratch);
    if (threadIdx.x == 0) distinct[blockIdx.x] = total;
}

// k_select_cuts on the sorted columns; grid as in k_column_heads
static __global__ void __launch_bounds__(256)
k_column_cuts(const unsigned *__restrict__ keys, int n, const int *__restrict__ before, const int *__restrict__ stride,
              const int *__restrict__ cut_ptr, int max_bin, float *__restrict__ cut_val, int *__restrict__ cut_fid) {
    const unsigned *k = keys + (size_t)blockIdx.y * n;
    const int f = blockIdx.y, s = stride[f], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int rank0 = before[(size_t)f * gridDim.x + blockIdx.x];
    __shared__ int w[8];
    for (int u = 0; u < COL_CHUNK / 256; ++u) {
        const int i = blockIdx.x * COL_CHUNK + u * 256 + threadIdx.x;
        const unsigned key = i < n ? k[i] : 0u;
        const bool head = i < n && (i == 0 || key != k[i - 1]);
        const unsigned m = __ballot_sync(0xffffffffu, head);
        __syncthreads();
        if (lane == 0) w[warp] = __popc(m);
        __syncthreads();
        int t = rank0 + __popc(m & ((1u << lane) - 1u)), all = 0;
        for (int q = 0; q < 8; ++q) { if (q < warp) t += w[q]; all += w[q]; }
        if (head) {
            const int pos = s == 0 ? t : (t % s == 0 && t / s < max_bin ? t / s : -1);
            if (pos >= 0) {
                cut_val[cut_ptr[f] + pos] = key_to_float((unsigned long long)key);
                cut_fid[cut_ptr[f] + pos] = f;
            }
        }
        rank0 += all;
    }
}

// ------------------------------------------------------------------ splits as the rows meet them
// Direction (hist_tree_builder_single.cu:1003-1012; `rev`: the column-sharded builder's bins count down, left means bin >
// split bin, hist_tree_builder.cu:455-459): a row goes left iff x = (bin + shift) mod 256 is below the threshold (rev: not
// below).  The missing value's bin 255 thereby takes the default direction without a test of its own: unshifted it lies above
// every bin, shifted below.
struct AssignRule { int feature; unsigned test; };   // test = threshold << 1 | shift
constexpr unsigned ASSIGN_NONE = 0xffffffffu;        // test of a node that was not split
__device__ __forceinline__ AssignRule assign_rule(const TreeNode &nd, bool split, int rev) {
    const unsigned shift = rev ? (nd.default_right ? 1 : 0) : (nd.default_right ? 0 : 1);
    return split ? AssignRule{nd.split_feature_id, (((unsigned)nd.split_bid + shift + (rev ? 1u : 0u)) << 1) | shift} : AssignRule{0, ASSIGN_NONE};
}
__device__ __forceinline__ bool assign_left(unsigned test, unsigned bin, int rev) { return (((bin + (test & 1u)) & 0xffu) < (test >> 1)) != (rev != 0); }
// ------------------------------------------------------------------ end of tree
// Tree::prune_self / try_prune_leaf / reorder_nid (src/thundergbm/tree.cu:85-128).  The reference walks the
// leaves in index order and climbs while a parent has two leaf children and gain < gamma; the fixed point of that
// walk does not depend on the order, so the levels are processed bottom-up with one thread per node.  One block.
__device__ inline void prune_tree(TreeNode *sn, int n_nodes, int depth, float gamma, int *scratch) {   // called by 1024 threads
    for (int level = depth - 1; level >= 0; --level) {
        const int nl = 1 << level, off = nl - 1;
        for (int n = threadIdx.x; n < nl; n += blockDim.x) {
            TreeNode &p = sn[off + n];
            if (p.is_valid && !p.is_leaf) {
                TreeNode &l = sn[p.lch_index], &r = sn[p.rch_index];
                if (l.is_valid && l.is_leaf && r.is_valid && r.is_leaf && p.gain < gamma) {
                    l.is_pruned = 1; r.is_pruned = 1; p.is_leaf = 1;
                }
            }
        }
        __syncthreads();
    }
    block_scan_excl(n_nodes, [&](int i) { return (sn[i].is_valid && !sn[i].is_pruned) ? 1 : 0; },
                    [&](int i, int id) { if (sn[i].is_valid && !sn[i].is_pruned) sn[i].final_id = id; }, scratch);
    __syncthreads();
}
// Does k_assign_stored move the rows of a node that store its split column, bins [span.x, span.y)?  Not if the column is much
// longer than the node's list.  Rounds of nine kinds of data with other factors than 4: 0 (always searched) 2 to 28 % longer, 1 up to
// 4 % longer, 16 between 3 % shorter and 2 % longer, without a limit between 4 % shorter and 7 % longer (popular columns).
__device__ __forceinline__ bool by_column(const int *bin_ptr, int2 span, int rows) {
    return bin_ptr && (long long)bin_ptr[span.y] - bin_ptr[span.x] <= 4ll * rows;
}
// what k_apply_tree needs of a finished tree
__device__ inline void leave_rules(const TreeNode *sn, int n_nodes, int depth, int rev, float *weight, AssignRule *rule, const int *last_cnt, const int *cut_ptr,
                                   const int *bin_ptr) {
    for (int i = threadIdx.x; i < n_nodes; i += blockDim.x) {
        int k = i;
        while (k > 0 && sn[k].is_pruned) k = (k - 1) >> 1;
        weight[i] = sn[k].base_weight;
    }
    const int nl = 1 << (depth - 1);
    for (int i = threadIdx.x; i < nl; i += blockDim.x) {
        const TreeNode &nd = sn[nl - 1 + i];
        AssignRule r = assign_rule(nd, nd.is_valid && sn[nd.lch_index].is_valid, rev);
        if (bin_ptr && r.test != ASSIGN_NONE && by_column(bin_ptr, make_int2(cut_ptr[r.feature], cut_ptr[r.feature + 1]), last_cnt[i])) r.feature = -1;
        rule[i] = r;
    }
}
static __global__ void __launch_bounds__(1024)
k_prune(TreeNode *nodes, int n_nodes, int depth, float gamma, int table_in_smem, TreeNode *model, int K, int k0,
        const RoundState *rs, float *weight, AssignRule *rule, size_t rule_stride, int rev, const int *last_cnt, size_t cnt_stride, const int *cut_ptr,
        const int *bin_ptr) {
    chain_wait();
    // grid = trees of the batch.  The finished tree also goes to its slot of the model, tree (round * K + class).
    nodes += (size_t)blockIdx.x * n_nodes;
    model += ((size_t)rs->round * K + k0 + blockIdx.x) * n_nodes;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int scratch[33];
    // trees too large for shared memory (depth 12 to 14) are pruned in place in global memory; the 48-byte records are
    // copied as the 16-byte pieces they consist of
    TreeNode *sn = table_in_smem ? reinterpret_cast<TreeNode *>(sm) : nodes;
    const int pieces = n_nodes * (int)(sizeof(TreeNode) / 16);
    if (table_in_smem) {
        for (int i = threadIdx.x; i < pieces; i += blockDim.x) reinterpret_cast<int4 *>(sn)[i] = reinterpret_cast<const int4 *>(nodes)[i];
        __syncthreads();
    }
    prune_tree(sn, n_nodes, depth, gamma, scratch);
    if (weight) leave_rules(sn, n_nodes, depth, rev, weight + (size_t)blockIdx.x * n_nodes, rule + blockIdx.x * rule_stride, last_cnt + blockIdx.x * cnt_stride, cut_ptr, bin_ptr);
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
        const int4 t = reinterpret_cast<const int4 *>(sn)[i];
        if (table_in_smem) reinterpret_cast<int4 *>(nodes)[i] = t;
        reinterpret_cast<int4 *>(model)[i] = t;
    }
}

// ------------------------------------------------------------------ metrics
// per-block partial sums in a fixed order: RMSE (pointwise_metric.cu:8-22), binary error and
// multi-class accuracy (multiclass_metric.cu:9-46)
static __global__ void k_metric_partial(int objective, const float *__restrict__ y, const float *yp, int n, int K,
                                 double *partial) {
    chain_wait();
    __shared__ double ws[32];
    double s = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (objective == REG_LINEAR || objective == REG_LOGISTIC || objective == BINARY_LOGISTIC) {
            s += pointwise_metric_term(objective, y[i], yp[i]);
        } else {
            int mk = 0;
            float mp = yp[i];
            for (int k = 1; k < K; ++k) { const float v = yp[(size_t)k * n + i]; if (v > mp) { mp = v; mk = k; } }
            s += ((float)mk == y[i]) ? 1.0 : 0.0;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        partial[blockIdx.x] = t;
    }
}
// one warp: lane l adds partial[l], partial[l+32], ... in that order, then a fixed shuffle tree
static __global__ void k_metric_sum(const double *__restrict__ partial, int nb, double *__restrict__ out) {
    double t = 0;
    for (int i = threadIdx.x; i < nb; i += 32) t += partial[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) *out = t;
}
__device__ __forceinline__ float metric_from_sum(int objective, double s, long long n_total) {
    if (objective == REG_LINEAR || objective == REG_LOGISTIC) return sqrtf((float)s / (float)n_total);
    if (objective == BINARY_LOGISTIC) return 1.0f - (float)(long long)s / (float)n_total;
    if (objective == RANK_PAIRWISE || objective == RANK_NDCG) return (float)(s / (double)n_total);  // mean over the query groups
    return (float)(long long)s / (float)n_total;
}
static __global__ void k_metric_final(int objective, const double *__restrict__ sum, long long n_total, float *__restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *out = metric_from_sum(objective, *sum, n_total);
}

// End of a boosting round: the round's metric (for ranking `sum` and `n_total` are those of the query groups), the round's
// fixed-point grid for the log, and the device round counter moves on.  One warp; `partial` not null: the sum is that of the
// `nb` partial sums, added like k_metric_sum adds them.
static __global__ void k_round_end(int objective, const double *sum, const double *partial, int nb, long long n_total,
                                   float *metric, const QuantInfo *qinfo, QuantInfo *qinfo_log, int log_len,
                                   RoundState *rs,
                                   unsigned long long *root_sum, int n_root, const TreeCtl *ctl) {
    chain_wait();
    const int coarse = ctl->coarse;
    for (int i = threadIdx.x; i < n_root; i += 32) root_sum[i] = 0;   // the next round adds to them
    double t = 0;
    if (partial) {
        // (all loads first, then the additions in the usual order)
        double v[METRIC_PARTS / 32];
#pragma unroll
        for (int u = 0; u < METRIC_PARTS / 32; ++u) v[u] = (int)threadIdx.x + 32 * u < nb ? partial[threadIdx.x + 32 * u] : 0.0;
#pragma unroll
        for (int u = 0; u < METRIC_PARTS / 32; ++u) t += v[u];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (threadIdx.x == 0 && blockIdx.x == 0 && !coarse) {   // (else the round will be built again)
        const int r = rs->round;
        if (objective >= 0) metric[r] = metric_from_sum(objective, partial ? t : *sum, n_total);
        if (r < log_len) qinfo_log[r] = *qinfo;
        rs->round = r + 1;
    }
}

static __global__ void k_fill(float *p, size_t n, float v) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

}  // namespace tgbm
