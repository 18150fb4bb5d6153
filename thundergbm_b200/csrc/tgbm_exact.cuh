// The exact tree builder (tree_method = exact; ExactTreeBuilder, src/thundergbm/builder/exact_tree_builder.cu):
// every distinct stored value of a node is a split candidate.  Same level loop, node table, pruning and scores as
// the histogram builder; what differs is the split search and how the rows move.
//
// Data: the stored values by column, largest first (SparseColumns::csr2csc_gpu, sparse_columns.cu:20-93,127), built
// once.  The entries of a level stand grouped by `column * nodes_in_level + node of their row`, values descending inside a
// group; entries of rows that stopped are gone.  A group's children at the next level are its own entries parted in order,
// left ones first, so the groups are not sorted again: a level is
//   k_exact_sum      prefix sums of (g,h) over the entries, begin and end of every group
//   k_exact_gain     the last entry of each run of equal values is a candidate whose right child is the group's sum up to
//                    it (exact_tree_builder.cu:50-118); best candidate and split per node
//   k_exact_move     rows to child nodes, k_exact_move_missing the rows without a value
//   k_exact_sides    left / right / gone for every entry, counts before it
//   k_exact_scatter  entries to their places at the next level
// Bound by the 12 bytes of an entry and the row look-ups.  A radix sort of all keys and a scan by key per level took
// 1.4 of the 2.75 ms of a tree (200 k rows x 28, depth 6), the passes over unsorted copies another 0.7.
#pragma once
#include "tgbm_kernels.cuh"

namespace tgbm {

constexpr int EX_THREADS = 256, EX_ITEMS = 4, EX_TILE = EX_THREADS * EX_ITEMS;   // entries are handled in tiles, four neighbours per thread

// Blocks per SM of the passes over the entries, all resident at once: the two of a pair share the runs of tiles, so they have the same
// grid.  (Eight per SM, of which three to six fit, are 1.3 to 2.7 waves: 39 us for the sums of 5.6 M entries and 25 for the sides
// that take 29 and 21 so.  With 5 and 6 per SM 28 and 22, but the scatter 60 instead of 48; with 3 and 4 the gains 59 instead of 52.)
constexpr int EX_SEARCH_BLOCKS = 4, EX_MOVE_BLOCKS = 5;

template <typename T> struct ExPair { T g, h; };
template <typename T> __device__ __forceinline__ ExPair<T> operator+(const ExPair<T> &a, const ExPair<T> &b) { return ExPair<T>{a.g + b.g, a.h + b.h}; }
template <typename T> __device__ __forceinline__ ExPair<T> operator-(const ExPair<T> &a, const ExPair<T> &b) { return ExPair<T>{a.g - b.g, a.h - b.h}; }
// In = gradient pair of a row, V = sums inside a tile (1024 quantised values of at most 20 bits fit an int), W = sums.
// The float arithmetic adds in double, so that a group's sum may be taken as the difference of two prefixes.
template <typename T> struct ExKind;
template <> struct ExKind<long long> { typedef int2 In; typedef int V; typedef long long W; };
template <> struct ExKind<float> { typedef float2 In; typedef double V; typedef double W; };
__device__ __forceinline__ float exact_cell(long long v, const GridScale &s) { return s(v); }
__device__ __forceinline__ float exact_cell(double v, const GridScale &) { return __double2float_rn(v); }

// four neighbours at once, 16 bytes per access (one access each of 8 bytes: every 32-byte sector four times)
template <typename E> __device__ __forceinline__ void exact_load4(const E *p, E (&v)[4]) {
    static_assert(sizeof(E) == 8 || sizeof(E) == 16, "");
    int4 w[sizeof(E) / 4];
#pragma unroll
    for (int u = 0; u < (int)(sizeof(E) / 4); ++u) w[u] = reinterpret_cast<const int4 *>(p)[u];
    memcpy(v, w, sizeof(w));
}
template <typename E> __device__ __forceinline__ void exact_store4(E *p, const E (&v)[4]) {
    static_assert(sizeof(E) == 8 || sizeof(E) == 16, "");
    int4 w[sizeof(E) / 4];
    memcpy(w, v, sizeof(w));
#pragma unroll
    for (int u = 0; u < (int)(sizeof(E) / 4); ++u) reinterpret_cast<int4 *>(p)[u] = w[u];
}

// (column, complement of the value's ordered image): ascending keys = columns ascending, values descending
static __global__ void k_exact_csc_keys(const float *__restrict__ val, const int *__restrict__ col, size_t nnz, unsigned long long *__restrict__ keys) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nnz; i += (size_t)gridDim.x * blockDim.x)
        keys[i] = ((unsigned long long)(unsigned)col[i] << 32) | (unsigned)~float_order(val[i]);
}
static __global__ void k_exact_csc_vals(const unsigned long long *__restrict__ keys, size_t nnz, float *__restrict__ val, unsigned *__restrict__ col) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nnz; i += (size_t)gridDim.x * blockDim.x) {
        val[i] = order_float(~(unsigned)(keys[i] & 0xffffffffull));
        col[i] = (unsigned)(keys[i] >> 32);
    }
}

// sum over the threads before this one, and over all; `s` holds EX_THREADS / 32 pairs
template <typename V>
__device__ __forceinline__ ExPair<V> exact_block_scan(const ExPair<V> &x, ExPair<V> &total, ExPair<V> *s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ExPair<V> v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const ExPair<V> u{__shfl_up_sync(0xffffffffu, v.g, o), __shfl_up_sync(0xffffffffu, v.h, o)};
        if (lane >= o) v = v + u;
    }
    __syncthreads();   // `s` of the scan before has been read
    if (lane == 31) s[warp] = v;
    ExPair<V> before{__shfl_up_sync(0xffffffffu, v.g, 1), __shfl_up_sync(0xffffffffu, v.h, 1)};
    if (lane == 0) before = ExPair<V>{0, 0};
    __syncthreads();
    total = ExPair<V>{0, 0};
    ExPair<V> base{0, 0};
#pragma unroll
    for (int w = 0; w < EX_THREADS / 32; ++w) {
        if (w == warp) base = total;
        total = total + s[w];
    }
    return base + before;
}

// The block that finishes last goes on alone (nobody waits for it): true there, with all other blocks' writes visible.
__device__ __forceinline__ bool exact_last_block(int *ticket) {
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
        if (s_last) { *ticket = 0; __threadfence(); }
    }
    __syncthreads();
    return s_last;
}

// A block takes a run of neighbouring tiles.  It adds up its own run as it goes (tile_pre[t]: sum of the run before tile t),
// and the block that finishes last turns the runs' sums into prefixes: what stands before a tile is the sum of the two.
// (Prefixes of all 5469 tiles by the last block took 15 of the 45 us of a pass over 5.6 M entries.)
__device__ __forceinline__ int exact_run(int tiles) { return max(1, (tiles + (int)gridDim.x - 1) / (int)gridDim.x); }

// exclusive prefixes of n sums by one block, eight neighbours per thread and round; returns the total
template <typename W>
__device__ __forceinline__ ExPair<W> exact_scan_runs(const ExPair<W> *sums, ExPair<W> *pre, int n, ExPair<W> *s) {
    ExPair<W> carry{0, 0};
    for (int base = 0; base < n; base += 8 * EX_THREADS) {
        const int a = base + 8 * (int)threadIdx.x;
        ExPair<W> v[8], mine{0, 0}, total;
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = a + u < n ? ExPair<W>{__ldcg(&sums[a + u].g), __ldcg(&sums[a + u].h)} : ExPair<W>{0, 0};
#pragma unroll
        for (int u = 0; u < 8; ++u) mine = mine + v[u];
        ExPair<W> run = carry + exact_block_scan<W>(mine, total, s);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (a + u < n) pre[a + u] = run;
            run = run + v[u];
        }
        carry = carry + total;
    }
    return carry;
}

// pre[i] = (g,h) sum of the tile's entries up to and with i, tile_pre and run_pre as above, group[key] = first entry, end.
// The root fetches the gradients by row (GATHER, a 32-byte sector for 8 bytes) and writes them down; from there on they
// travel with the entries.
template <typename T, bool GATHER>
static __global__ void __launch_bounds__(EX_THREADS, EX_SEARCH_BLOCKS)
k_exact_sum(const int *live, const unsigned *key, const int *row, const typename ExKind<T>::In *gh_rows,
            typename ExKind<T>::In *gh, ExPair<typename ExKind<T>::V> *pre,
            ExPair<typename ExKind<T>::W> *tile_pre, ExPair<typename ExKind<T>::W> *run_sum, ExPair<typename ExKind<T>::W> *run_pre, int2 *group, int *ticket) {
    typedef typename ExKind<T>::V V;
    typedef typename ExKind<T>::W W;
    chain_wait();
    __shared__ ExPair<V> s[EX_THREADS / 32];
    __shared__ ExPair<W> sw[EX_THREADS / 32];
    const unsigned n = (unsigned)*live;
    const int tiles = (int)((n + EX_TILE - 1) / EX_TILE), lane = threadIdx.x & 31, per = exact_run(tiles);
    ExPair<W> run{0, 0};
    for (int t = blockIdx.x * per, t_end = min(tiles, t + per); t < t_end; ++t) {
        const unsigned i0 = (unsigned)t * EX_TILE + threadIdx.x * EX_ITEMS;
        const uint4 k4 = *reinterpret_cast<const uint4 *>(key + i0);   // (the arrays end with a whole tile)
        const unsigned k[4] = {k4.x, k4.y, k4.z, k4.w};
        typename ExKind<T>::In v[4];
        if (GATHER) {
            const int4 r4 = *reinterpret_cast<const int4 *>(row + i0);
            const int r[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = i0 + u < n ? gh_rows[r[u]] : typename ExKind<T>::In{0, 0};
            exact_store4(gh + i0, v);
        } else {
            exact_load4(gh + i0, v);
        }
        ExPair<V> p[4], sum{0, 0}, total;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i0 + u < n) sum = sum + ExPair<V>{(V)v[u].x, (V)v[u].y};
            p[u] = sum;
        }
        unsigned before = __shfl_up_sync(0xffffffffu, k[3], 1), after = __shfl_down_sync(0xffffffffu, k[0], 1);
        if (lane == 0 && i0 > 0 && i0 < n) before = key[i0 - 1];
        if (lane == 31 && i0 + 4 < n) after = key[i0 + 4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned i = i0 + u;
            if (i >= n) break;
            if (i == 0 || k[u] != (u ? k[u - 1] : before)) group[k[u]].x = (int)i;
            if (i + 1 == n || k[u] != (u < 3 ? k[u + 1] : after)) group[k[u]].y = (int)i + 1;
        }
        const ExPair<V> base = exact_block_scan<V>(sum, total, s);
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = base + p[u];
        exact_store4(pre + i0, p);
        if (threadIdx.x == 0) tile_pre[t] = run;
        run = run + ExPair<W>{(W)total.g, (W)total.h};
    }
    if (threadIdx.x == 0) run_sum[blockIdx.x] = run;
    if (exact_last_block(ticket)) exact_scan_runs<W>(run_sum, run_pre, (int)gridDim.x, sw);
}

// what the split search reads
template <typename T> struct ExSearch {
    const unsigned *key;
    const float *val;
    const ExPair<typename ExKind<T>::V> *pre;
    const ExPair<typename ExKind<T>::W> *tile_pre, *run_pre;
    const int2 *group;
};
// sum of the entries before entry i
template <typename T>
__device__ __forceinline__ ExPair<typename ExKind<T>::W> exact_before(const ExSearch<T> &x, unsigned i, int per) {
    typedef typename ExKind<T>::W W;
    if (i == 0) return ExPair<W>{0, 0};
    const ExPair<typename ExKind<T>::V> p = x.pre[i - 1];
    const int t = (int)((i - 1) / EX_TILE);
    return x.run_pre[t / per] + x.tile_pre[t] + ExPair<W>{(W)p.g, (W)p.h};
}

// right-child candidate sums and missing sums of a node
struct ExCand { float rg, rh, mg, mh; };
template <typename W>
__device__ __forceinline__ ExCand exact_cand(const TreeNode &nd, const ExPair<W> &right, const ExPair<W> &total, const GridScale &inv_sg, const GridScale &inv_sh) {
    // exact_tree_builder.cu:160-167 (missing = node sum - sum of the stored values)
    return ExCand{exact_cell(right.g, inv_sg), exact_cell(right.h, inv_sh),
                  __fsub_rn(nd.sum_g, exact_cell(total.g, inv_sg)), __fsub_rn(nd.sum_h, exact_cell(total.h, inv_sh))};
}
__device__ __forceinline__ float exact_gain(float parent, float pg, float ph, const ExCand &c, float mcw, float lam) {
    // exact_tree_builder.cu:186-209 (gain, default direction)
    const float gl = fmaxf(0.f, split_gain(parent, pg, ph, c.rg, c.rh, mcw, lam));
    const float rg2 = __fadd_rn(c.rg, c.mg), rh2 = __fadd_rn(c.rh, c.mh);
    const float gr = fmaxf(0.f, split_gain(parent, pg, ph, rg2, rh2, mcw, lam));
    return gl > gr ? gl : -gr;
}
// the children's terms of the gain with fast divisions (2 units in the last place), the larger of the two directions
__device__ __forceinline__ float exact_terms(float pg, float ph, const ExCand &c, float lam) {
    const float lg = pg - c.rg, lh = ph - c.rh, rg2 = c.rg + c.mg, rh2 = c.rh + c.mh, lg2 = pg - rg2, lh2 = ph - rh2;
    return fmaxf(__fdividef(lg * lg, lh + lam) + __fdividef(c.rg * c.rg, c.rh + lam), __fdividef(lg2 * lg2, lh2 + lam) + __fdividef(rg2 * rg2, rh2 + lam));
}

// SplitPoint of the best candidate and TreeBuilder::update_tree (exact_tree_builder.cu:262-296, :137-151 for the split
// value; tree_builder.cu:9-60) of node n of the level.
template <typename T>
__device__ __forceinline__ void exact_apply(const ExSearch<T> &x, int level, int n, unsigned long long b, TreeNode *nodes, const GridScale &inv_sg, const GridScale &inv_sh,
                                            float mcw, float lam, float rt_eps, int per) {
    const int off = (1 << level) - 1;
    TreeNode &nd = nodes[off + n];
    if (!nd.is_valid || b == 0) return;   // no stored value in the node: SplitPoint::nid = -1, the node stays as it is
    const unsigned j = 0xffffffffu - (unsigned)(b & 0xffffffffull), key = x.key[j];
    const int2 range = x.group[key];
    const ExPair<typename ExKind<T>::W> base = exact_before(x, (unsigned)range.x, per);
    const ExCand c = exact_cand(nd, exact_before(x, j + 1, per) - base, exact_before(x, (unsigned)range.y, per) - base, inv_sg, inv_sh);
    const float parent = __fdiv_rn(__fmul_rn(nd.sum_g, nd.sum_g), __fadd_rn(nd.sum_h, lam));
    const float gn = exact_gain(parent, nd.sum_g, nd.sum_h, c, mcw, lam);
    const float gain = __uint_as_float((unsigned)(b >> 32));   // |gn|, or 0 for a column left out of the round
    if (gain > rt_eps) {
        const float v = x.val[j];
        nd.gain = gain;
        nd.split_feature_id = (int)(key >> level);
        nd.split_bid = 0;
        nd.split_value = (int)j + 1 == range.y ? __fsub_rn(__fsub_rn(v, fabsf(x.val[range.x])), rt_eps)
                                               : __fmul_rn(__fadd_rn(v, x.val[j + 1]), 0.5f);
        TreeNode &l = nodes[nd.lch_index], &rc = nodes[nd.rch_index];
        l.is_valid = 1; rc.is_valid = 1;
        float rgs = c.rg, rhs = c.rh;
        if (gn < 0.f) { rgs = __fadd_rn(rgs, c.mg); rhs = __fadd_rn(rhs, c.mh); nd.default_right = 1; }
        else nd.default_right = 0;
        rc.sum_g = rgs; rc.sum_h = rhs;
        l.sum_g = __fsub_rn(nd.sum_g, rgs); l.sum_h = __fsub_rn(nd.sum_h, rhs);
        l.base_weight = __fdiv_rn(-l.sum_g, __fadd_rn(l.sum_h, lam));
        rc.base_weight = __fdiv_rn(-rc.sum_g, __fadd_rn(rc.sum_h, lam));
    } else {
        nd.is_leaf = 1;
        nodes[nd.lch_index].is_valid = 0;
        nodes[nd.rch_index].is_valid = 0;
    }
}

// Gain of every candidate and the best one per node: key = |gain| bits << 32 | ~position, so that the largest key is
// the largest |gain| and among equals the smallest sorted position (exact_tree_builder.cu:218-258: smaller partition
// id, i.e. smaller column, then larger value).  Per block the keys meet in shared memory (one slot per node of the
// level), warps whose lanes all sit in one node reduce first.
// What is the same for a group's candidates is worked out when a thread meets the group.
// Two exact divisions per direction are what a candidate costs: one that cannot reach its block's best so far is left out
// by a bound with fast divisions, whose margin (1e-5) is far above their error.
template <typename T>
static __global__ void __launch_bounds__(EX_THREADS, EX_SEARCH_BLOCKS)
k_exact_gain(const int *live, const ExSearch<T> x, int level, TreeNode *nodes, const QuantInfo *q, float mcw, float lam, float rt_eps,
             const unsigned char *__restrict__ ignored_all, const RoundState *rs, int F,
             unsigned long long *best, int *any_split, int *ticket) {
    typedef typename ExKind<T>::W W;
    chain_wait();
    extern __shared__ unsigned long long ex_best[];
    const int nl = 1 << level, off = nl - 1, lane = threadIdx.x & 31;
    for (int n = threadIdx.x; n < nl; n += EX_THREADS) ex_best[n] = 0;
    __syncthreads();
    const unsigned char *ignored = ignored_all ? ignored_all + (size_t)rs->round * F : nullptr;
    const GridScale inv_sg(cell_inv<T>(q, 0)), inv_sh(cell_inv<T>(q, 1));
    const unsigned n_live = (unsigned)*live;
    const int tiles = (int)((n_live + EX_TILE - 1) / EX_TILE), per = exact_run(tiles);
    unsigned cur = 0xffffffffu;      // group the values below belong to
    unsigned end = 0;
    ExPair<W> base{0, 0};
    float pg = 0.f, ph = 0.f, parent = 0.f, mg = 0.f, mh = 0.f;
    bool skipped = false;
    for (int t = blockIdx.x * per, t_end = min(tiles, t + per); t < t_end; ++t) {   // (neighbouring tiles: the threads seldom change the group)
        const unsigned i0 = (unsigned)t * EX_TILE + threadIdx.x * EX_ITEMS;
        const uint4 k4 = *reinterpret_cast<const uint4 *>(x.key + i0);
        const float4 v4 = *reinterpret_cast<const float4 *>(x.val + i0);
        const unsigned k[4] = {k4.x, k4.y, k4.z, k4.w};
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
        float after = __shfl_down_sync(0xffffffffu, v[0], 1);
        if (lane == 31 && i0 + 4 < n_live) after = x.val[i0 + 4];
        const ExPair<W> tile_base = x.run_pre[blockIdx.x] + x.tile_pre[t];
        ExPair<typename ExKind<T>::V> pr[4];
        exact_load4(x.pre + i0, pr);
        unsigned long long cand = 0;
        int cn = -1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned i = i0 + u;
            if (i >= n_live) continue;
            const int n = (int)(k[u] & (unsigned)(nl - 1));
            if (k[u] != cur) {
                cur = k[u];
                const int2 range = x.group[cur];
                end = (unsigned)range.y;
                base = exact_before(x, (unsigned)range.x, per);
                const ExPair<W> total = exact_before(x, end, per) - base;
                pg = nodes[off + n].sum_g; ph = nodes[off + n].sum_h;
                mg = __fsub_rn(pg, exact_cell(total.g, inv_sg)); mh = __fsub_rn(ph, exact_cell(total.h, inv_sh));
                parent = __fdiv_rn(__fmul_rn(pg, pg), __fadd_rn(ph, lam));
                skipped = ignored && ignored[cur >> level];
            }
            if (i + 1 != end && (u < 3 ? v[u + 1] : after) == v[u]) continue;   // not the last of its run
            float gn = 0.f;
            if (!skipped) {
                const ExPair<W> right = ExPair<W>{tile_base.g + (W)pr[u].g, tile_base.h + (W)pr[u].h} - base;
                const float bar = __uint_as_float((unsigned)(*(volatile unsigned long long *)&ex_best[n] >> 32));
                ExCand c;
                c.rg = exact_cell(right.g, inv_sg); c.rh = exact_cell(right.h, inv_sh);
                c.mg = mg; c.mh = mh;
                if (bar > 0.f && exact_terms(pg, ph, c, lam) * 1.00001f < (bar + parent) * 0.99999f) continue;
                gn = exact_gain(parent, pg, ph, c, mcw, lam);
            }
            const unsigned long long mine = ((unsigned long long)__float_as_uint(fabsf(gn)) << 32) | (0xffffffffu - i);
            if (cn >= 0 && cn != n) { atomicMax(&ex_best[cn], cand); cand = 0; }
            cn = n;
            cand = mine > cand ? mine : cand;
        }
        // warps in one node (the usual case) send one key
        const unsigned has = __ballot_sync(0xffffffffu, cn >= 0);
        if (!has) continue;
        const int n0 = __shfl_sync(0xffffffffu, cn, __ffs(has) - 1);
        if (__all_sync(0xffffffffu, cn == n0 || cn < 0)) {
            const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(cand >> 32));
            const unsigned lo = __reduce_max_sync(0xffffffffu, cn >= 0 && (unsigned)(cand >> 32) == hi ? (unsigned)cand : 0u);
            if (lane == 0) atomicMax(&ex_best[n0], ((unsigned long long)hi << 32) | lo);
        } else if (cn >= 0) {
            atomicMax(&ex_best[cn], cand);
        }
    }
    __syncthreads();
    for (int n = threadIdx.x; n < nl; n += EX_THREADS)
        if (ex_best[n]) atomicMax(&best[n], ex_best[n]);
    __threadfence();
    if (!exact_last_block(ticket)) return;
    if (threadIdx.x == 0) *any_split = 0;
    for (int n = threadIdx.x; n < nl; n += EX_THREADS) {
        const unsigned long long b = __ldcg(&best[n]);
        best[n] = 0;
        exact_apply<T>(x, level, n, b, nodes, inv_sg, inv_sh, mcw, lam, rt_eps, per);
    }
}

// ExactTreeBuilder::update_ins2node_id (exact_tree_builder.cu:303-340): a row that stores the split feature of its
// node goes by the value.  Those are the entries of the group (split feature, node).  grid = (blocks, nodes)
static __global__ void k_exact_move(const int *row, const float *val, const int2 *group, int level,
                                    int *nid, const TreeNode *nodes, int *any_split) {
    chain_wait();
    const int nl = 1 << level, off = nl - 1;
    for (int n = blockIdx.y; n < nl; n += gridDim.y) {
        const TreeNode &nd = nodes[off + n];
        if (nd.is_leaf || !nd.is_valid || nd.split_feature_id < 0) continue;
        const int2 range = group[((unsigned)nd.split_feature_id << level) + (unsigned)n];
        const float split = nd.split_value;
        const int l = nd.lch_index, r = nd.rch_index;
        for (unsigned i = (unsigned)range.x + blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)range.y; i += gridDim.x * blockDim.x)
            nid[row[i]] = val[i] < split ? l : r;
        if (blockIdx.x == 0 && threadIdx.x == 0) *any_split = 1;
    }
}
// ... and ExactTreeBuilder::ins2node_id_all_reduce (:394-409): the rows still in a splittable node of the level follow
// its default direction; skipped when no row moved at this level (tree_builder.cu:174-181 leaves the loop first).
// side[r / 32]: bit r % 32 of x / y = row r is now in a left / right child of the level.  Entries look their rows up there:
// two bits per row stay in L1 (200 k rows: 50 KB) where the node ids do not.
static __global__ void k_exact_move_missing(int *nid, int n_rows, int level, const TreeNode *nodes, const int *any_split, uint2 *side) {
    chain_wait();
    const bool any = *any_split != 0;
    const int nl = 1 << level, off = nl - 1;
    for (int r0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; r0 < n_rows; r0 += gridDim.x * blockDim.x) {   // whole warps
        const int r = r0 + (threadIdx.x & 31);
        int at = r < n_rows ? nid[r] : -1;
        if (any && at >= off && at < off + nl) {
            const TreeNode &nd = nodes[at];
            if (!nd.is_leaf && nd.is_valid) nid[r] = at = nd.default_right ? nd.rch_index : nd.lch_index;
        }
        const int c = at - (2 * nl - 1);
        const bool in = at >= 0 && c >= 0 && c < 2 * nl;
        const unsigned l = __ballot_sync(0xffffffffu, in && !(c & 1)), rr = __ballot_sync(0xffffffffu, in && (c & 1));
        if ((threadIdx.x & 31) == 0) side[r0 >> 5] = make_uint2(l, rr);
    }
}

// lr[i] = entries of the tile up to and with i that go left (low half) and right (high half); tile_lr, run_lr: those before
// tile t in its run, and before the run
static __global__ void __launch_bounds__(EX_THREADS, EX_MOVE_BLOCKS)
k_exact_sides(const int *live, const int *row, const uint2 *side, unsigned *lr,
              ExPair<int> *tile_lr, ExPair<int> *run_cnt, ExPair<int> *run_lr, int *next_live, int *ticket) {
    chain_wait();
    __shared__ ExPair<int> s[EX_THREADS / 32];
    const unsigned n = (unsigned)*live;
    const int tiles = (int)((n + EX_TILE - 1) / EX_TILE), per = exact_run(tiles);
    ExPair<int> run{0, 0};
    for (int t = blockIdx.x * per, t_end = min(tiles, t + per); t < t_end; ++t) {
        const unsigned i0 = (unsigned)t * EX_TILE + threadIdx.x * EX_ITEMS;
        const int4 r4 = *reinterpret_cast<const int4 *>(row + i0);
        const int r[4] = {r4.x, r4.y, r4.z, r4.w};
        uint2 c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = i0 + u < n ? side[r[u] >> 5] : make_uint2(0, 0);
        ExPair<int> p[4], sum{0, 0}, total;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            sum = sum + ExPair<int>{(int)((c[u].x >> (r[u] & 31)) & 1u), (int)((c[u].y >> (r[u] & 31)) & 1u)};
            p[u] = sum;
        }
        const ExPair<int> base = exact_block_scan<int>(sum, total, s);
        unsigned o[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) o[u] = (unsigned)(base.g + p[u].g) | ((unsigned)(base.h + p[u].h) << 16);
        *reinterpret_cast<uint4 *>(lr + i0) = make_uint4(o[0], o[1], o[2], o[3]);
        if (threadIdx.x == 0) tile_lr[t] = run;
        run = run + total;
    }
    if (threadIdx.x == 0) run_cnt[blockIdx.x] = run;
    if (exact_last_block(ticket)) {
        const ExPair<int> all = exact_scan_runs<int>(run_cnt, run_lr, (int)gridDim.x, s);
        if (threadIdx.x == 0) *next_live = all.g + all.h;
    }
}

// Entry i of group [b, e) goes to (entries kept before b) + (lefts of the group before it), or behind all lefts of the group.
// Neighbouring lanes hold neighbouring entries, so that either side's stores run on.
template <typename In>
static __global__ void __launch_bounds__(EX_THREADS, EX_MOVE_BLOCKS)
k_exact_scatter(const int *live, const unsigned *key, const int *row, const float *val, const In *gh, const unsigned *lr, const ExPair<int> *tile_lr,
                const ExPair<int> *run_lr, const int2 *group, unsigned *key_out, int *row_out, float *val_out, In *gh_out) {
    chain_wait();
    const unsigned n = (unsigned)*live;
    const int tiles = (int)((n + EX_TILE - 1) / EX_TILE), per = exact_run(tiles);
    auto before = [&](unsigned i) {   // lefts and rights before entry i
        if (i == 0) return ExPair<int>{0, 0};
        const unsigned v = lr[i - 1];
        const int t = (int)((i - 1) / EX_TILE);
        return run_lr[t / per] + tile_lr[t] + ExPair<int>{(int)(v & 0xffffu), (int)(v >> 16)};
    };
    unsigned cur = 0xffffffffu;
    int left0 = 0, right0 = 0;   // place of a left (right) entry = its lefts (rights) before + this
    for (int t = blockIdx.x * per, t_end = min(tiles, t + per); t < t_end; ++t) {
        unsigned k[EX_ITEMS], l[EX_ITEMS], p[EX_ITEMS];
        int r[EX_ITEMS];
        float v[EX_ITEMS];
        In g[EX_ITEMS];
#pragma unroll
        for (int u = 0; u < EX_ITEMS; ++u) {
            const unsigned in_tile = u * EX_THREADS + threadIdx.x, i = (unsigned)t * EX_TILE + in_tile;
            l[u] = p[u] = 0;
            if (i < n) {
                l[u] = lr[i]; p[u] = in_tile ? lr[i - 1] : 0u;
                k[u] = key[i]; r[u] = row[i]; v[u] = val[i]; g[u] = gh[i];
            }
        }
        const ExPair<int> tb = run_lr[blockIdx.x] + tile_lr[t];
#pragma unroll
        for (int u = 0; u < EX_ITEMS; ++u) {
            if (l[u] == p[u]) continue;   // gone
            if (k[u] != cur) {
                cur = k[u];
                const int2 range = group[cur];
                left0 = before((unsigned)range.x).h;    // kept before the group, less the lefts before it
                right0 = before((unsigned)range.y).g;   // ... and all lefts of the group, less the rights before it
            }
            const bool left = (l[u] & 0xffffu) != (p[u] & 0xffffu);
            const int d = left ? left0 + tb.g + (int)(p[u] & 0xffffu) : right0 + tb.h + (int)(p[u] >> 16);
            key_out[d] = 2 * k[u] + (left ? 0u : 1u);
            row_out[d] = r[u];
            val_out[d] = v[u];
            gh_out[d] = g[u];
        }
    }
}

// TreeBuilder::predict_in_training (tree_builder.cu:62-74) from the row -> node table
static __global__ void k_exact_predict(const int *nid, int n_rows, const TreeNode *nodes, float lr,
                                       float *yp, int *nid_out) {
    chain_wait();
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        int n = nid[r];
        if (nid_out) nid_out[r] = n;
        while (n != -1 && nodes[n].is_pruned) n = nodes[n].parent_index;
        yp[r] = __fmaf_rn(lr, nodes[n].base_weight, yp[r]);
    }
}

}  // namespace tgbm
