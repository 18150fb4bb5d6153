// Kernels of one tree level: histogram build, split search, row partition.
//
// A level is three launches -- k_hist (or its CSR / float forms), k_eval, k_assign -- that hand over to each other through
// the segment tables alone (seg_begin, seg_cnt: where the row list of every node of the level sits).
// What used to be planned by single-block kernels between them (which sibling to build, tile lists, prefix sums: 14 + 5 us
// a level, most of the time of a small training) every block now works out for itself from those tables, in shared memory,
// while its first loads are on their way.
//
// Trees of one round do not depend on each other (softmax builds one per class from the same scores), so every kernel
// takes a batch of them: blockIdx.z is the tree, the buffers of consecutive trees lie `Batch::*_stride` apart.
#pragma once
#include "tgbm_kernels.cuh"

namespace tgbm {

struct Batch {
    TreeNode *nodes;
    int *seg_begin[2], *seg_cnt[2];   // by level parity
    int *origin[2];                   // by level parity: rows of the nodes before a node, where its children's lists start
    int *rec_idx;                     // row ids of the level's lists, left children in the first half, right ones in the second
    unsigned short *nid;              // node of every row
    const int2 *gh;                   // gradient pairs by row
    long long *hist_full, *hist_built;
    SplitRec *recs;
    int *ticket;
    float *weight;                    // finished tree: weight of the deepest surviving node on the way to a node
    AssignRule *rule;                 // ... and the splits of the last level
    TreeCtl *ctl;
    size_t nodes_stride, seg_stride, rec_stride, nid_stride, gh_stride, full_stride, built_stride, recs_stride, ticket_stride, rule_stride;
    int half;                         // offset of the right children in rec_idx
};

// ------------------------------------------------------------------ work lists
// Exclusive prefix sums over n values inside one block of NT threads: out(i, prefix before i); returns the total.
// `scratch` holds 33 values of shared memory.  Every thread of the block must call it.
template <int NT, typename V, typename In, typename Out>
__device__ __forceinline__ V block_prefix(int n, In in, Out out, V *scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    V carry = 0;
    for (int base = 0; base < n; base += NT) {
        const int i = base + threadIdx.x;
        const V x = i < n ? in(i) : V(0);
        V v = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const V u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
        __syncthreads();
        if (lane == 31) scratch[warp] = v;
        __syncthreads();
        if (n - base <= 32) {   // one warp holds them all
            const V total = scratch[0];
            if (i < n) out(i, v - x + carry);
            carry += total;
            break;
        }
        if (warp == 0) {
            V t = lane < NT / 32 ? scratch[lane] : V(0);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const V u = __shfl_up_sync(0xffffffffu, t, o); if (lane >= o) t += u; }
            scratch[lane] = t;
        }
        __syncthreads();
        if (i < n) out(i, v + (warp ? scratch[warp - 1] : V(0)) + carry - x);
        carry += scratch[NT / 32 - 1];
    }
    __syncthreads();
    return carry;
}

// Which child of pair j of a level >= 1 is built (the other one is the parent minus it): the one with fewer rows, ties ->
// left (hist_tree_builder_single.cu:466); -1: neither holds rows.  With several ranks the row counts are rank-local, so
// every rank takes the child with the smaller hessian sum from the replicated node table -- the same choice everywhere
// without a collective; the histogram sums are integers, so built and subtracted ones are identical either way.
__device__ __forceinline__ int built_side(int level, int j, const int *seg_cnt, const TreeNode *nodes, int by_hessian) {
    if (by_hessian) {
        const int off = (1 << level) - 1;
        const TreeNode &l = nodes[off + 2 * j], &r = nodes[off + 2 * j + 1];
        if (!l.is_valid || !r.is_valid) return -1;
        return l.sum_h > r.sum_h ? 1 : 0;
    }
    const int2 c = *reinterpret_cast<const int2 *>(seg_cnt + 2 * j);
    return max(c.x, c.y) == 0 ? -1 : (c.x > c.y ? 1 : 0);
}

// The histograms a level builds and their tiles of `TILE` records: s_base[j] = tiles before pair j, s_base[pairs] = total.
// `node(j)`: the built node of the pair or -1.  The block that reports adds to the byte counters of the roofline.
template <int NT, int TILE>
__device__ __forceinline__ int hist_items(int level, const Batch &b, size_t tree, int by_hessian, int *s_base, int *scratch, bool report) {
    const int pairs = level == 0 ? 1 : 1 << (level - 1);
    const int *cnt = b.seg_cnt[level & 1] + tree * b.seg_stride;
    const TreeNode *nodes = b.nodes + tree * b.nodes_stride;
    __shared__ unsigned long long s_rows;
    __shared__ int s_hists;
    if (threadIdx.x == 0) { s_rows = 0; s_hists = 0; }
    __syncthreads();
    const int total = block_prefix<NT>(pairs,
        [&](int j) {
            const int r = level == 0 ? 0 : built_side(level, j, cnt, nodes, by_hessian);
            const int n = r < 0 ? 0 : cnt[level == 0 ? 0 : 2 * j + r];
            if (report && r >= 0) { atomicAdd(&s_rows, (unsigned long long)n); atomicAdd(&s_hists, 1); }
            return (n + TILE - 1) / TILE;
        },
        [&](int j, int before) { s_base[j] = before; }, scratch);
    if (threadIdx.x == 0) {
        s_base[pairs] = total;
        if (report) {
            atomicAdd(level == 0 ? &b.ctl->stat_rows_root : &b.ctl->stat_rows_gather, s_rows);
            atomicAdd(&b.ctl->stat_hists, (unsigned long long)s_hists);
        }
    }
    __syncthreads();
    return total;
}

// Order in which the dense histogram kernel visits the level's tiles.
// The tiles are dealt out to shares, one or two per CTA, in proportion to the items' sizes (cumulative rounding, so
// the shares of different items are disjoint; an item too small for a share of its own rides on one).  Inside an item
// tile t belongs to share v0 + t mod k.  CTA c owns its consecutive shares and visits, item by item, the tiles
// of its shares in ascending order: every CTA walks each of its (one or two, rarely more) lists once, front to back,
// and since all CTAs carry about the same number of tiles, all lists are walked at the same relative pace.  Row ids
// ascend inside every list (to the chunks of k_assign), so at any time the whole GPU gathers rows from one moving window of the bin matrix:
// DRAM pages and 64-byte sectors get shared between nodes.  A pure gather of 5.2 M of 10.5 M rows in 8 to 64 lists
// takes 72 us this way and 100 to 110 us list after list.
__device__ __forceinline__ void hist_share(const int *s_base, int w, int total, int n_shares, int &v0, int &k) {
    const unsigned half = (unsigned)total / 2, a = (unsigned)s_base[w] * (unsigned)n_shares + half, z = (unsigned)s_base[w + 1] * (unsigned)n_shares + half;
    v0 = (int)(a / (unsigned)total);
    k = (int)(z / (unsigned)total) - v0;
    if (k <= 0) { k = 1; v0 = min(v0, n_shares - 1); }
}

// Permute the 16 bin bytes of a half row so that byte j of the register array is the bin of slot (j XOR key),
// key = 0..15: at step j the 16 lane pairs of a warp then address 16 different slots of either half.  Key bits 0-1
// permute the bytes inside every word (one PRMT each), bits 2-3 exchange whole words.
__device__ __forceinline__ void xor_permute_half(uint32_t (&w)[4], int key) {
    const uint32_t sel = (key & 2) ? ((key & 1) ? 0x0123u : 0x1032u) : ((key & 1) ? 0x2301u : 0x3210u);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __byte_perm(w[i], 0u, sel);
    const int hi = key >> 2;
#pragma unroll
    for (int s = 1; s <= 2; s <<= 1) {
        uint32_t t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = (hi & s) ? w[i ^ s] : w[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = t[i];
    }
}

// ------------------------------------------------------------------ histogram build, dense layout
// Root: hist_tree_builder_single.cu:203-216, deeper levels: :485-505.
// Persistent CTAs, one per SM; grid = (ctas, feature groups of 32, trees).  A lane holds one 16-feature half of two rows;
// the shared-memory accumulators are laid out [bin][32 features] so that the bank is the feature index, and at step j the
// 32 lanes of a warp handle 32 different features, so every shared atomic of a warp hits 32 different banks.
//
// !FINE (exact mode, values of at most quant_bits bits): accumulators are int32.  Before they could overflow
// (`window_rows` rows of at most 2^quant_bits each) they are drained into int64 totals, also in shared memory.
// FINE (fp32 mode after its first round, values of FINE_BITS bits and a sign): a value is added in two halves, the low 16
// bits to an unsigned accumulator and the rest to a signed one.  Two plain 32-bit atomics per component are the cheapest
// exact 31-bit addition there is: the bare shared-memory atomics of 294 M (row, feature) pairs take 0.134 ms so, 0.188 ms
// as one returning atomic with a carry test, 0.290 ms as one 64-bit atomic, 0.320 ms as float atomics (compare-and-swap
// loops); 0.073 ms with one 32-bit atomic per component.  FINE_WINDOW rows fill the low halves.
//
// When a CTA is done with a node its sums are laid out [feature][bin][g,h] as int64 in shared memory and added to the
// node's histogram by one bulk reduction per feature (cp.reduce.async.bulk: the L2 takes whole lines; 148 CTAs flushing
// 28 x 255 cells: 4.3 us into one node, 2.8 us into 64; 21.7 and 10.7 us as one RED.64 per cell and component, whose
// lanes hit 32 different sectors).
constexpr int HIST_SEQ = 32;                                           // tiles of a CTA laid down at a time
constexpr int HIST_CELLS = 256 * 32;                                   // per component
constexpr int HIST_STAGE = 256 * 16 + 16;                              // bytes of a feature's int64 pairs; the pad keeps 8 lanes' 16-byte stores in different banks
constexpr int HIST_FINE_SMEM = 32 * HIST_STAGE;                        // 4 int32 accumulators per cell (128 KB), staged in place
constexpr int HIST_EXACT_SMEM = 2 * HIST_CELLS * 4 + 32 * HIST_STAGE;  // 2 int32 accumulators, then int64 totals = staging area

__device__ __forceinline__ void bulk_add_u64(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.u64 [%0], [%1], %2;"
                 ::"l"(dst), "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(bytes) : "memory");
}

// The rare parts of the kernel are functions of their own: inlined, their registers made the loop that adds up the rows
// spill (64 registers per thread is all there is; 180 bytes spilled, 126 us per launch in exact mode at 10.5 M rows).

// What they need stands in shared memory for the same reason.
struct HistTiles {
    const int *s_base, *seg_begin, *seg_cnt, *cut_ptr;
    const TreeNode *nodes;
    long long *slab;
    int level, total, n_shares, va, vb, ib, ie, by_hessian;   // the CTA owns shares [va, vb), items ib .. ie may have some of them
    int f0, nf, B;                                            // first feature of the group, features, bins of all features
};
// the CTA's t-th tile: first record, records (0 = no more), pair
__device__ __noinline__ int4 hist_tile(const HistTiles &x, int t) {
    for (int w = x.ib; w <= x.ie; ++w) {
        const int T = x.s_base[w + 1] - x.s_base[w];
        if (!T) continue;
        int v0, k;
        hist_share(x.s_base, w, x.total, x.n_shares, v0, k);
        const int ra = max(x.va, v0) - v0, width = min(x.vb, v0 + k) - v0 - ra;
        if (width <= 0) continue;
        const int n = (T / k) * width + min(max(T % k - ra, 0), width);   // the share's tiles: `width` neighbours of every k
        if (t >= n) { t -= n; continue; }
        const int at = (ra + (t / width) * k + t % width) * HIST_THREADS;
        const int node = x.level == 0 ? 0 : 2 * w + built_side(x.level, w, x.seg_cnt, x.nodes, x.by_hessian);
        return make_int4(x.seg_begin[node] + at, min(HIST_THREADS, x.seg_cnt[node] - at), w, 0);
    }
    return make_int4(0, 0, 0, 0);
}

// exact mode: int32 window -> int64 totals, same [bin][feature] layout
__device__ __noinline__ void hist_drain(unsigned char *hist_sm, bool drained) {
    int *acc = reinterpret_cast<int *>(hist_sm);
    long long *tot = reinterpret_cast<long long *>(hist_sm + 2 * HIST_CELLS * 4);
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < 2 * HIST_CELLS; i += HIST_THREADS) {
        const int v = acc[i];
        tot[i] = drained ? tot[i] + v : v;
        acc[i] = 0;
    }
    __syncthreads();
}

// the CTA's sums of a pair's built node to its histogram
template <bool FINE>
__device__ __noinline__ void hist_flush(const HistTiles &x, unsigned char *hist_sm, int pair, bool drained, bool again) {
    const int lane = threadIdx.x & 31;
    int *acc = reinterpret_cast<int *>(hist_sm), *high = acc + 2 * HIST_CELLS;
    unsigned char *stage = hist_sm + (FINE ? 0 : 2 * HIST_CELLS * 4);
    const long long *tot = reinterpret_cast<const long long *>(stage);
    long long vg[8], vh[8];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int s = ((threadIdx.x >> 5) + 32 * q) * 32 + lane;
        if (FINE) {
            vg[q] = ((long long)high[s] << 16) + (unsigned)acc[s]; vh[q] = ((long long)high[HIST_CELLS + s] << 16) + (unsigned)acc[HIST_CELLS + s];
        } else {
            vg[q] = acc[s]; vh[q] = acc[HIST_CELLS + s];
            if (drained) { vg[q] += tot[s]; vh[q] += tot[HIST_CELLS + s]; }
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q)
        *reinterpret_cast<longlong2 *>(stage + lane * HIST_STAGE + ((threadIdx.x >> 5) + 32 * q) * 16) = make_longlong2(vg[q], vh[q]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        const int b0 = lane < x.nf ? x.cut_ptr[x.f0 + lane] : 0, nb = lane < x.nf ? x.cut_ptr[x.f0 + lane + 1] - b0 : 0;   // the lane's feature
        if (nb > 0) bulk_add_u64(x.slab + ((size_t)pair * x.B + b0) * 2, stage + lane * HIST_STAGE, (uint32_t)nb * 16);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    if (!again) return;
    __syncthreads();
    for (int i = threadIdx.x; i < (FINE ? 4 : 2) * HIST_CELLS * 4 / 16; i += HIST_THREADS) reinterpret_cast<int4 *>(hist_sm)[i] = make_int4(0, 0, 0, 0);
    __syncthreads();
}

template <bool GATHER, bool FINE>
static __global__ void __launch_bounds__(HIST_THREADS, 1)
k_hist(int level, const Batch b, const unsigned char *__restrict__ bins, int Fpad, int F, const int *__restrict__ cut_ptr, int B,
       int window_rows, int by_hessian) {
    extern __shared__ __align__(128) unsigned char hist_sm[];
    int *acc = reinterpret_cast<int *>(hist_sm);          // g, h (FINE: low halves)
    int *s_base = reinterpret_cast<int *>(hist_sm + (FINE ? HIST_FINE_SMEM : HIST_EXACT_SMEM));
    __shared__ int scratch[33], s_ib, s_ie;
    __shared__ int4 s_seq[HIST_SEQ + 4];
    __shared__ HistTiles tiles;
    const int group = blockIdx.y, f0 = group * 32, lane = threadIdx.x & 31;
    const size_t tree = blockIdx.z;
    constexpr int ZERO_BYTES = FINE ? 4 * HIST_CELLS * 4 : 2 * HIST_CELLS * 4;   // the accumulators
    for (int i = threadIdx.x; i < ZERO_BYTES / 16; i += HIST_THREADS)
        reinterpret_cast<int4 *>(hist_sm)[i] = make_int4(0, 0, 0, 0);
    chain_wait();
    if (threadIdx.x == 0) { s_ib = 0x7fffffff; s_ie = -1; }
    const int total = hist_items<HIST_THREADS, HIST_THREADS>(level, b, tree, by_hessian, s_base, scratch, blockIdx.x == 0 && group == 0);
    if (total == 0) return;
    const int pairs = level == 0 ? 1 : 1 << (level - 1);
    const int per_cta = total >= HIST_SHARE_TILES * (int)gridDim.x ? HIST_SHARES : 1;
    const int n_shares = (int)gridDim.x * per_cta, va = (int)blockIdx.x * per_cta, vb = va + per_cta;
    const int *seg_begin = b.seg_begin[level & 1] + tree * b.seg_stride, *seg_cnt = b.seg_cnt[level & 1] + tree * b.seg_stride;
    const TreeNode *nodes = b.nodes + tree * b.nodes_stride;
    for (int w = threadIdx.x; w < pairs; w += HIST_THREADS) {   // items with a share among this CTA's
        if (s_base[w + 1] == s_base[w]) continue;
        int v0, k;
        hist_share(s_base, w, total, n_shares, v0, k);
        if (v0 < vb && v0 + k > va) { atomicMin(&s_ib, w); atomicMax(&s_ie, w); }
    }
    __syncthreads();
    if (s_ie < 0) return;
    // HIST_SEQ tiles at a time are laid down in shared memory
    if (threadIdx.x == 0)
        tiles = HistTiles{s_base, seg_begin, seg_cnt, cut_ptr, nodes, b.hist_built + tree * b.built_stride, level, total, n_shares, va, vb, s_ib, s_ie, by_hessian,
                          f0, min(32, F - f0), B};
    __syncthreads();
    int seq0 = 0;   // position of s_seq[0]
    if (threadIdx.x < HIST_SEQ + 4) s_seq[threadIdx.x] = hist_tile(tiles, (int)threadIdx.x);
    __syncthreads();

    const int *rec_idx = b.rec_idx + tree * b.rec_stride;
    const int2 *gh = b.gh + tree * b.gh_stride;

    bool drained = false;   // the totals hold something: few rows per node and CTA need none, so they are not zeroed either

    // Two lanes share a row: lane l loads the 16-byte half (l & 1) of the rows at tile positions
    // warp*32 + (l >> 1) ("A") and 16 further on ("B").  One load instruction of a warp therefore touches 16 rows
    // (16 sectors) instead of 32 half-used ones, which halves the L1 wavefronts the gathered rows cost.
    const int qa = (threadIdx.x & ~31) | (lane >> 1), qb = qa + 16;  // the lane's two tile positions
    const uint32_t laneoff = ((uint32_t)(lane & 1) << 6) | ((uint32_t)(lane >> 1) << 2);  // 4 * (16*half + key)
    // Software pipeline over the CTA's tiles.  While tile i is accumulated, the bin rows of tile i+1 are on their
    // way into registers, those of tile i+2 have been asked into L2 (a prefetch holds no register), and the row ids
    // of tile i+3 are being fetched.  The gather levels are bound by the bytes in flight (a loaded DRAM access takes
    // 2-3 us here): one tile per warp in registers alone sustains only ~2.4 TB/s of sector traffic.
    auto ids = [&](int i, int &ra, int &rb) {   // row ids of the lane's two positions in tile i, -1 = no record
        const int4 e = s_seq[i - seq0];
        ra = qa < e.y ? (GATHER ? rec_idx[e.x + qa] : e.x + qa) : -1;
        rb = qb < e.y ? (GATHER ? rec_idx[e.x + qb] : e.x + qb) : -1;
    };
    const size_t half_off = (size_t)f0 + 16u * (lane & 1);
    uint4 na = make_uint4(0, 0, 0, 0), nb = na;
    int2 nva = make_int2(0, 0), nvb = nva;
    int r1a, r1b, r2a, r2b, pair_next = 0;
    bool noka = false, nokb = false;
    auto load_rows = [&](int i) {   // rows of tile i (ids r1a, r1b) -> registers
        pair_next = s_seq[i - seq0].z;
        noka = r1a >= 0; nokb = r1b >= 0;
        if (noka) { na = *reinterpret_cast<const uint4 *>(bins + (size_t)r1a * Fpad + half_off); nva = gh[r1a]; }
        if (nokb) { nb = *reinterpret_cast<const uint4 *>(bins + (size_t)r1b * Fpad + half_off); nvb = gh[r1b]; }
    };
    // rows with ids r2a, r2b -> L2; one lane of each pair asks for the row's sector.  (Asking for the gradients too costs more
    // than it brings, 67.5 against 66.1 ms per training of 10.5 M rows: lines of eight rows, most are there already.)
    auto prefetch_rows = [&]() {
        if (GATHER && !(lane & 1)) {
            if (r2a >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(bins + (size_t)r2a * Fpad + f0));
            if (r2b >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(bins + (size_t)r2b * Fpad + f0));
        }
    };
    if (s_seq[0].y == 0) return;   // more shares than tiles
    ids(0, r1a, r1b);
    ids(1, r2a, r2b);
    load_rows(0);
    prefetch_rows();
    r1a = r2a; r1b = r2b;
    ids(2, r2a, r2b);
    int pair_cur = pair_next, since = 0;
    for (int i = 0; s_seq[i - seq0].y > 0; ++i) {
        const uint4 a = na, bb = nb;
        const int2 va2 = nva, vb2 = nvb;
        const bool oka = noka, okb = nokb;
        const int pair_this = pair_next;
        load_rows(i + 1);
        prefetch_rows();
        r1a = r2a; r1b = r2b;
        ids(i + 3, r2a, r2b);
        if (i + 1 - seq0 == HIST_SEQ) {
            __syncthreads();
            seq0 = i + 1;
            if (threadIdx.x < HIST_SEQ + 4) s_seq[threadIdx.x] = hist_tile(tiles, seq0 + (int)threadIdx.x);
            __syncthreads();
        }
        if (pair_this != pair_cur || (FINE && since + HIST_THREADS > FINE_WINDOW)) {  // another node: hand the finished one over
            hist_flush<FINE>(tiles, hist_sm, pair_cur, drained, true);
            drained = false;
            pair_cur = pair_this;
            since = 0;
        } else if (!FINE && since + HIST_THREADS > window_rows) {
            hist_drain(hist_sm, drained);
            drained = true;
            since = 0;
        }
        since += HIST_THREADS;
        // Step j adds a row to (bin of feature 16*half + (j ^ key), that feature), key = lane >> 1: the 32 lanes of a
        // warp address 32 different features = 32 different banks.  Byte offset of the accumulator:
        // bin * 128 | feature * 4 -- the bin field comes straight out of the packed word with one shift and one
        // mask.  No test for missing values: bin 255 (missing, and the padding columns beyond F) lands in row 255
        // of the table, which no feature ever reads back.
        char *const gbase = reinterpret_cast<char *>(acc);
        auto add = [&](uint32_t off, const int2 v) {
            if (FINE) {
                atomicAdd(reinterpret_cast<unsigned *>(gbase + off), (unsigned)v.x & 0xffffu);
                atomicAdd(reinterpret_cast<unsigned *>(gbase + off + HIST_CELLS * 4), (unsigned)v.y & 0xffffu);
                atomicAdd(reinterpret_cast<int *>(gbase + off + 2 * HIST_CELLS * 4), v.x >> 16);
                atomicAdd(reinterpret_cast<int *>(gbase + off + 3 * HIST_CELLS * 4), v.y >> 16);
            } else {
                atomicAdd(reinterpret_cast<int *>(gbase + off), v.x);
                atomicAdd(reinterpret_cast<int *>(gbase + off + HIST_CELLS * 4), v.y);
            }
        };
        auto add_row = [&](const uint4 &row, const int2 v) {
            uint32_t w[4] = {row.x, row.y, row.z, row.w};
            xor_permute_half(w, lane >> 1);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const uint32_t word = w[j >> 2];
                const uint32_t binoff = ((j & 3) == 0 ? (word << 7) : (word >> (8 * (j & 3) - 7))) & 0x7f80u;
                add(binoff | (laneoff ^ (4u * j)), v);
            }
        };
        if (oka) add_row(a, va2);
        if (okb) add_row(bb, vb2);
    }
    hist_flush<FINE>(tiles, hist_sm, pair_cur, drained, false);
}

// ------------------------------------------------------------------ histogram build, CSR of global bin ids
// A histogram of ~100k bins does not fit in shared memory, so the first SPARSE_SMEM_BINS bins are accumulated per CTA in
// shared memory and the rest goes straight to the node's histogram with global int64 atomics.  That pays where columns are
// numbered by frequency, as vocabularies usually are: 23 of 36 values per row of the generated data then hit the first bins.
// With ids in another order (hashed, alphabetical) the shared part gets what falls there by chance; the results are the same.
// (The histogram is L2-resident: 16 B per bin.)  One warp per row, lanes over its values; the shared accumulators are the low and high halves of k_hist<., true> in either mode (exact values are narrower), which costs
// four plain atomics per value: the int64 atomics they replace are compare-and-swap loops (root of 1 M rows x 30 values: 370 us).
constexpr int SPARSE_SMEM_BINS = 12288;  // 192 KB: low and high halves of g and h
constexpr int SPARSE_THREADS = 1024;     // one CTA per SM

template <bool GATHER>
static __global__ void __launch_bounds__(SPARSE_THREADS, 1)
k_hist_sparse(int level, const Batch b, const int *__restrict__ row_ptr, const int *__restrict__ bin, int B, int by_hessian) {
    extern __shared__ __align__(16) int sh_sparse[];  // [4][nsm]: low g, low h, high g, high h; then s_base
    __shared__ int scratch[33];
    const int nsm = min(B, SPARSE_SMEM_BINS);
    int *s_base = sh_sparse + 4 * nsm;
    const size_t tree = blockIdx.z;
    for (int i = threadIdx.x; i < 4 * nsm; i += SPARSE_THREADS) sh_sparse[i] = 0;
    chain_wait();
    const int total = hist_items<SPARSE_THREADS, HIST_THREADS>(level, b, tree, by_hessian, s_base, scratch, blockIdx.x == 0);
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int t_begin = min(total, (int)blockIdx.x * per), t_end = min(total, t_begin + per);
    if (t_begin >= t_end) return;
    const int pairs = level == 0 ? 1 : 1 << (level - 1);
    const int *seg_begin = b.seg_begin[level & 1] + tree * b.seg_stride, *seg_cnt = b.seg_cnt[level & 1] + tree * b.seg_stride;
    const TreeNode *nodes = b.nodes + tree * b.nodes_stride;
    const int *rec_idx = b.rec_idx + tree * b.rec_stride;
    const int2 *gh = b.gh + tree * b.gh_stride;
    long long *slab = b.hist_built + tree * b.built_stride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto flush = [&](int pair, bool again) {
        __syncthreads();
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(slab + (size_t)pair * B * 2);
        for (int i = threadIdx.x; i < 2 * nsm; i += SPARSE_THREADS) {   // consecutive lanes: consecutive words of the histogram
            const int s = (i & 1) * nsm + (i >> 1);
            const long long v = ((long long)sh_sparse[2 * nsm + s] << 16) + (unsigned)sh_sparse[s];
            if (v) atomicAdd(dst + i, (unsigned long long)v);
            if (again) { sh_sparse[s] = 0; sh_sparse[2 * nsm + s] = 0; }
        }
        if (again) __syncthreads();
    };
    int w = 0;
    {
        int lo = 0, hi = pairs - 1;   // last item that starts at or before t_begin
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (s_base[mid] <= t_begin) lo = mid; else hi = mid - 1;
        }
        w = lo;
    }
    int w_cur = w, since = 0, node = -1, begin = 0, count = 0;
    for (int t = t_begin; t < t_end; ++t) {
        while (t >= s_base[w + 1]) ++w;
        if (w != w_cur || since + HIST_THREADS > FINE_WINDOW) { flush(w_cur, true); since = 0; }
        since += HIST_THREADS;
        if (w != w_cur || node < 0) {
            w_cur = w;
            node = level == 0 ? 0 : 2 * w + built_side(level, w, seg_cnt, nodes, by_hessian);
            begin = seg_begin[node]; count = seg_cnt[node];
        }
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(slab + (size_t)w * B * 2);
        const int first = (t - s_base[w]) * HIST_THREADS;
        const int last = min(count, first + HIST_THREADS);
        // A warp takes every 32nd row of the tile.  Three rows are in flight per warp: the row pointers and gradients
        // of the row after next, the first 32 bin ids of the next row, and the row being accumulated -- a row is a
        // chain of three dependent loads (record -> row pointers -> bin ids) and would otherwise cost three memory
        // latencies each.
        constexpr int W = SPARSE_THREADS / 32;
        auto meta = [&](int q, int &j0, int &j1, int2 &v) {
            j0 = j1 = 0; v = make_int2(0, 0);
            if (q < last) {
                const int p = begin + q;
                const int r = GATHER ? rec_idx[p] : p;
                v = gh[r];
                j0 = row_ptr[r]; j1 = row_ptr[r + 1];
            }
        };
        int q = first + warp;
        int j0, j1, nj0, nj1, mj0, mj1;
        int2 v, nv, mv;
        meta(q, j0, j1, v);
        meta(q + W, nj0, nj1, nv);
        int b0 = lane < j1 - j0 ? bin[j0 + lane] : -1;
        for (; q < last; q += W) {
            meta(q + 2 * W, mj0, mj1, mv);
            const int nb0 = lane < nj1 - nj0 ? bin[nj0 + lane] : -1;
            int x = b0;
            each_step(j0, j1, lane, 32, [&](unsigned j) {
                if (j != (unsigned)j0 + lane) x = bin[j];
                if (x < nsm) {
                    atomicAdd(reinterpret_cast<unsigned *>(sh_sparse + x), (unsigned)v.x & 0xffffu);
                    atomicAdd(reinterpret_cast<unsigned *>(sh_sparse + nsm + x), (unsigned)v.y & 0xffffu);
                    atomicAdd(sh_sparse + 2 * nsm + x, v.x >> 16);
                    atomicAdd(sh_sparse + 3 * nsm + x, v.y >> 16);
                } else {
                    atomicAdd(dst + 2 * x, (unsigned long long)(long long)v.x);
                    atomicAdd(dst + 2 * x + 1, (unsigned long long)(long long)v.y);
                }
            });
            j0 = nj0; j1 = nj1; v = nv; b0 = nb0;
            nj0 = mj0; nj1 = mj1; nv = mv;
        }
    }
    flush(w_cur, false);
}

// The same stored values by column (rows ascend inside a bin), where no row stores a column twice: built once, see
// BoosterImpl::sort_columns.
struct SparseColumns {
    const int *row, *bin;   // [values] sorted by bin
    const int *bin_ptr;     // [bins + 1] first value of every bin; null: not there
};

// Root histogram bin by bin: a warp takes COLUMN_RUN neighbouring values, adds up those of a bin in registers and hands over two
// sums per bin.  What it costs is the gradients, 8 bytes from anywhere in an array that stays in L2, a 32-byte sector each (popular
// columns: up to four rows a sector): 36 M values of 1 M rows take 165 us, 5.6 TB/s of L2 sectors.  Row by row (k_hist_sparse) they
// take 198 us: 181 for the 23 M values that meet in shared memory, where popular columns make the same few cells hot.  Bins of a
// few values only: two reductions per value as there.  Against the rows, 20 rounds, ms: 50 k rows x 30 values, two or one to a bin
// 15.9 and 29.1 (16.3, 29.5), 1 M rows x 10 in 12 k bins 8.7 (9.5), 20 k rows x 40 in 10 k bins 3.6 (3.8), 200 k rows x 40 in 5 k bins,
// all in shared memory there, 7.5 (7.2).  grid = (blocks, 1, trees)
constexpr int COLUMN_RUN = 1024;
static __global__ void __launch_bounds__(256)
k_hist_columns(const Batch b, const SparseColumns c, int nnz) {
    chain_wait();
    const size_t tree = blockIdx.z;
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the byte counters, see hist_items
        atomicAdd(&b.ctl->stat_rows_root, (unsigned long long)b.seg_cnt[0][tree * b.seg_stride]);
        atomicAdd(&b.ctl->stat_hists, 1ull);
    }
    const int2 *gh = b.gh + tree * b.gh_stride;
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(b.hist_built + tree * b.built_stride);
    const int lane = threadIdx.x & 31;
    for (long long run = (long long)(blockIdx.x * 8 + (threadIdx.x >> 5)) * COLUMN_RUN; run < nnz; run += (long long)gridDim.x * 8 * COLUMN_RUN) {
        const int end = (int)min((long long)nnz, run + COLUMN_RUN);
        int cur = -1;   // bin that g and h belong to, the same in the whole warp
        long long g = 0, h = 0;
        auto hand_over = [&]() {
            if (cur < 0) return;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { g += shfl_xor_ll(g, o); h += shfl_xor_ll(h, o); }
            if (lane < 2) atomicAdd(dst + 2 * (size_t)cur + lane, (unsigned long long)(lane ? h : g));
            g = h = 0;
        };
        constexpr int U = 4;   // windows of 32 values in flight
        each_step((int)run, end, 0, 32 * U, [&](unsigned e0) {
            int x[U], r[U];
            int2 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const unsigned e = e0 + 32 * u + lane;
                x[u] = e < (unsigned)end ? c.bin[e] : -1;
                r[u] = e < (unsigned)end ? c.row[e] : -1;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = r[u] >= 0 ? gh[r[u]] : make_int2(0, 0);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                unsigned left = __ballot_sync(0xffffffffu, x[u] >= 0);
                const int before = __shfl_up_sync(0xffffffffu, x[u], 1);
                const int starts = __popc(__ballot_sync(0xffffffffu, x[u] >= 0 && lane > 0 && x[u] != before));
                if (starts > 4) {
                    if (x[u] >= 0) {
                        atomicAdd(dst + 2 * (size_t)x[u], (unsigned long long)(long long)v[u].x);
                        atomicAdd(dst + 2 * (size_t)x[u] + 1, (unsigned long long)(long long)v[u].y);
                    }
                    continue;
                }
                while (left) {
                    const int bin = __shfl_sync(0xffffffffu, x[u], __ffs(left) - 1);
                    if (bin != cur) { hand_over(); cur = bin; }
                    const bool mine = x[u] == bin;
                    if (mine) { g += v[u].x; h += v[u].y; }
                    left &= ~__ballot_sync(0xffffffffu, mine);
                }
            }
        });
        hand_over();
    }
}

// ------------------------------------------------------------------ split evaluation
// Histogram cells are `long long` sums on the round's fixed-point grid (exact mode) or `float` sums (fp32 mode, the
// reference's own arithmetic: GHPair of floats, include/thundergbm/common.h:43-59).  The evaluation kernels are
// written once over the cell type.
template <typename T> __device__ __forceinline__ double cell_inv(const QuantInfo *q, int h);
template <> __device__ __forceinline__ double cell_inv<long long>(const QuantInfo *q, int h) { return h ? q->inv_sh : q->inv_sg; }
template <> __device__ __forceinline__ double cell_inv<float>(const QuantInfo *, int) { return 1.0; }
__device__ __forceinline__ float cell_f(long long v, const GridScale &s) { return s(v); }
__device__ __forceinline__ float cell_f(float v, const GridScale &) { return v; }
__device__ __forceinline__ long long shfl_up_t(long long v, int d) { return shfl_up_ll(v, d); }
__device__ __forceinline__ float shfl_up_t(float v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ long long shfl_t(long long v, int src) { return shfl_ll(v, src); }
__device__ __forceinline__ float shfl_t(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// one child's sums (g, h); the other child is the node minus it, `parent` the node's own term
__device__ __forceinline__ float split_gain(float parent, float pg, float ph, float g, float h, float mcw, float lam) {
    const float g2 = __fsub_rn(pg, g), h2 = __fsub_rn(ph, h);
    if (h >= mcw && h2 >= mcw)
        return __fsub_rn(__fadd_rn(__fdiv_rn(__fmul_rn(g, g), __fadd_rn(h, lam)), __fdiv_rn(__fmul_rn(g2, g2), __fadd_rn(h2, lam))), parent);
    return 0.f;
}

// split value of a feature's candidate, from the feature's cut points
__device__ __forceinline__ float split_below(float first) { return (float)((double)__fsub_rn(first, fabsf(first)) - 1e-5); }   // of the first bin
__device__ __forceinline__ float split_at(const float *cuts, int bin, int multi) {
    if (multi) return cuts[bin];   // the column-sharded builder: the cut point itself (tree_builder.cu:9-60)
    return bin ? cuts[bin - 1] : split_below(cuts[0]);
}
// SplitPoint of candidate r (feature-local bin) into node nid of sums (sum_g, sum_h) and its children: TreeBuilder::update_tree.
// The table is a heap (Tree::init2): no index is read from it.
__device__ __forceinline__ void apply_split(TreeNode *nodes, int nid, const SplitRec &r, float sum_g, float sum_h, float rt_eps, float lam, int multi) {
    TreeNode &nd = nodes[nid], &left = nodes[2 * nid + 1], &right = nodes[2 * nid + 2];
    const float gain = fabsf(r.gain);
    if (!(gain > rt_eps)) {
        nd.is_leaf = 1;
        left.is_valid = 0;
        right.is_valid = 0;
        return;
    }
    const bool default_right = r.gain < 0.f;
    nd.gain = gain;
    nd.split_feature_id = r.feature;
    nd.split_bid = (unsigned char)r.bin;
    nd.split_value = r.value;
    nd.default_right = default_right ? 1 : 0;
    // the record's sums are the left child's -- the right one's where the column-sharded builder's candidates are taken
    // (`multi`, tree_builder.cu:9-60) --, the other child is the node minus it
    float g = r.lg, h = r.lh;
    if (default_right == (multi != 0)) { g = __fadd_rn(g, r.mg); h = __fadd_rn(h, r.mh); }
    const float og = __fsub_rn(sum_g, g), oh = __fsub_rn(sum_h, h), w = __fdiv_rn(-g, __fadd_rn(h, lam)), ow = __fdiv_rn(-og, __fadd_rn(oh, lam));
    left.is_valid = 1; right.is_valid = 1;
    left.sum_g = multi ? og : g; left.sum_h = multi ? oh : h; left.base_weight = multi ? ow : w;
    right.sum_g = multi ? g : og; right.sum_h = multi ? h : oh; right.base_weight = multi ? w : ow;
}

// Per-node argmax over the records, SplitPoint decode and update_tree (hist_tree_builder_single.cu:365-389 and :847-902) of node n
// of the level, whose sums the caller knows.  Called by one whole warp; the records may have been written by other blocks of the
// running kernel: they are read past L1.  chunked: F is the number of chunks and a record's bin is a global bin index
// (k_eval_chunk); otherwise one record per feature with a feature-local bin (k_eval).  Ties go to the smaller global bin.
// Up to BEST_WHOLE columns a lane keeps the record of its best: nothing waits for another load.  Of more it reads the first quarter of
// the records and the winner's once more (5.9 k columns: 96 us with whole records, 36 so).
constexpr int BEST_WHOLE = 128;
__device__ __forceinline__ SplitRec load_rec(const SplitRec *p) {
    int4 w[2] = {__ldcg(reinterpret_cast<const int4 *>(p)), __ldcg(reinterpret_cast<const int4 *>(p) + 1)};
    SplitRec r;
    memcpy(&r, w, sizeof(r));
    return r;
}
__device__ __forceinline__ void best_apply_node(int level, int n, int F, const SplitRec *recs, TreeNode *nodes, float sum_g, float sum_h, float rt_eps, float lam,
                                                const int *__restrict__ cut_ptr, int chunked, int multi) {
    const int lane = threadIdx.x & 31, nid = (1 << level) - 1 + n;
    unsigned long long key = 0;
    SplitRec best;
    int from = -1;   // of many columns: where the lane's best is
    recs += (size_t)n * F;
    auto better = [&](float gain, int bin, int f) {
        const unsigned long long k = bin < 0 ? 0 : ((unsigned long long)__float_as_uint(fabsf(gain)) << 32) | (unsigned)(0x7fffffff - (chunked ? bin : f));
        if (k <= key) return false;
        key = k;
        return true;
    };
    if (F <= BEST_WHOLE)
        for (int f = lane; f < F; f += 32) {
            const SplitRec r = load_rec(recs + f);
            if (better(r.gain, r.bin, f)) best = r;
        }
    else
#pragma unroll 8
        for (int f = lane; f < F; f += 32) {
            const int2 w = __ldcg(reinterpret_cast<const int2 *>(recs + f));   // gain and bin
            if (better(__int_as_float(w.x), w.y, f)) from = f;
        }
    // a record with gain 0 still has a key > 0, so 0 means "no record"
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    if (lo == 0) {  // no feature has a cut point: nothing to split on
        if (lane == 0) {
            nodes[nid].is_leaf = 1;
            nodes[2 * nid + 1].is_valid = 0;
            nodes[2 * nid + 2].is_valid = 0;
        }
        return;
    }
    if (key != (((unsigned long long)hi << 32) | lo)) return;   // one lane holds it
    if (from >= 0) best = load_rec(recs + from);
    if (chunked) best.bin -= cut_ptr[best.feature];
    apply_split(nodes, nid, best, sum_g, sum_h, rt_eps, lam, multi);
}

// Where the row lists of node n's children start, their lengths zeroed for k_assign to count up.  A node's children take
// the places of its own rows in either half of the lists, and the rows before it are known from its pair alone.
__device__ __forceinline__ void open_children(int level, int n, const Batch &b, size_t tree) {
    const size_t t = tree * b.seg_stride;
    const int in = level & 1, o = level == 0 ? 0 : b.origin[in ^ 1][t + (n >> 1)] + ((n & 1) ? b.seg_cnt[in][t + n - 1] : 0);
    b.origin[in][t + n] = o;
    *reinterpret_cast<int2 *>(b.seg_begin[in ^ 1] + t + 2 * n) = make_int2(o, b.half + o);
    *reinterpret_cast<int2 *>(b.seg_cnt[in ^ 1] + t + 2 * n) = make_int2(0, 0);
}

// CSR layout: one warp per node of the level, after k_eval_chunk
static __global__ void __launch_bounds__(32)
k_best_apply(int level, const Batch b, int F, const int *__restrict__ cut_ptr, float rt_eps, float lam, int multi) {
    chain_wait();
    const size_t tree = blockIdx.z;
    if (threadIdx.x == 0) open_children(level, blockIdx.x, b, tree);
    TreeNode *nodes = b.nodes + tree * b.nodes_stride;
    const TreeNode &nd = nodes[(1 << level) - 1 + blockIdx.x];
    if (nd.is_valid) best_apply_node(level, blockIdx.x, F, b.recs + tree * b.recs_stride, nodes, nd.sum_g, nd.sum_h, rt_eps, lam, cut_ptr, 1, multi);
}

// Sibling subtraction, per-feature prefix scan, missing sums, gains and per-feature argmax
// (hist_tree_builder_single.cu:257-347 for the root, :538-540 and :614-704 for sibling pairs), then, by the block that
// finishes a pair last (`ticket`, left at zero), the choice among the features and the tree update of the pair's nodes.
// grid = (items, pairs, trees), an item is a feature or, of features of up to EVAL_SMALL bins, four, a warp each (`items`: the
// features, -2 behind a single one, -1 for a warp without; PACKED = false: an item per feature, in a kernel of its own, as asking
// costs: 390 -> 367 us for the last level of 300 k rows x 28, depth 14; one-hot columns have one or two bins, and
// a block each made 24 k blocks of a level of seven trees: 109 us, 44 of 54 columns with two bins); a thread owns two bins of both
// children.  The gains are the work of this kernel -- four IEEE
// divisions per bin and child -- and its time is latency: few bins per thread keep a block's chain short, few threads per
// block keep many blocks resident.  The built histogram is zeroed as it is read, ready for the next level's reductions.
//
// multi: the column-sharded builder's candidates (hist_tree_builder.cu:299-352): the INCLUSIVE prefix along the
// bins (they count down from the largest values there) is the right child, the left one is the node minus it,
// missing values join the right child when that gains at least as much; the record then carries the right sums.
// bs: distance of two cells of `built` in cells (1 unless the fp32 histogram kernel spread them out); tree_cells: from tree to
// tree, in T.
// ignored: the round's column-sampling mask (Shard::column_sampling, src/thundergbm/builder/shard.cu:8-23; the
// masked features take no part in the split search, hist_tree_builder_single.cu:304,663), or null.
constexpr int EVAL_THREADS = 128, EVAL_BINS = 2, EVAL_SMALL = 32 * EVAL_BINS;
template <typename T> struct CellPair;
template <> struct CellPair<long long> { typedef longlong2 type; };
template <> struct CellPair<float> { typedef float2 type; };
template <typename T, bool PACKED>
static __global__ void __launch_bounds__(EVAL_THREADS, 8)
k_eval(int level, const Batch b, const int4 *__restrict__ items, int F, int B, const int *__restrict__ cut_ptr, T *built_all, size_t tree_cells, int bs,
       const QuantInfo *q, float mcw, float lam, const float *__restrict__ cut_val, float rt_eps,
       const unsigned char *__restrict__ ignored_all, const RoundState *rs, int multi, int by_hessian, int keep) {
    // keep = 0 at the last level: no level subtracts from its histograms, so they are not stored
    constexpr int WARPS = EVAL_THREADS / 32, NB = EVAL_BINS;
    __shared__ T s_sum[4][sizeof(T) == 4 ? 32 : WARPS];
    __shared__ unsigned long long s_key[2][WARPS];
    const int j = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4 item = PACKED ? items[blockIdx.x] : make_int4(blockIdx.x, -2, -2, -2);
    const bool packed = PACKED && item.y != -2;
    const int f = !packed || warp == 0 ? item.x : warp == 1 ? item.y : warp == 2 ? item.z : item.w, i0 = (packed ? lane : (int)threadIdx.x) * NB;
    const size_t tree = blockIdx.z;
    TreeNode *nodes = b.nodes + tree * b.nodes_stride;
    SplitRec *recs = b.recs + tree * b.recs_stride;
    int *ticket = b.ticket + tree * b.ticket_stride;
    const int b0 = cut_ptr[max(f, 0)], nb = f < 0 ? 0 : cut_ptr[f + 1] - b0, off = (1 << level) - 1, n_children = level == 0 ? 1 : 2;
    // the cut points around the thread's bins: the split value goes with the record
    float cut[NB + 1];
#pragma unroll
    for (int n = 0; n <= NB; ++n) cut[n] = i0 + n - 1 < nb && i0 < nb ? cut_val[b0 + max(i0 + n - 1, 0)] : 0.f;
    chain_wait();
    const int br = level == 0 ? 0 : built_side(level, j, b.seg_cnt[level & 1] + tree * b.seg_stride, nodes, by_hessian);
    if (blockIdx.x == 0 && (int)threadIdx.x < n_children) open_children(level, level == 0 ? 0 : 2 * j + (int)threadIdx.x, b, tree);
    const bool ignored = ignored_all && f >= 0 && ignored_all[(size_t)rs->round * F + f];
    T *full = reinterpret_cast<T *>(b.hist_full + tree * b.full_stride) + (size_t)off * B * 2;
    T *built = built_all + tree * tree_cells + ((size_t)j * B + b0) * 2 * bs;
    using Pair = typename CellPair<T>::type;
    // every load of the block is on its way before the first one is waited for (nothing here may alias: the compiler does
    // not know and would wait between a store and the next load)
    Pair cell[NB], above[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        const bool mine = i0 + n < nb && br >= 0;
        cell[n] = above[n] = Pair{0, 0};
        if (mine) cell[n] = *reinterpret_cast<const Pair *>(built + (size_t)2 * bs * (i0 + n));
        if (mine && level > 0) above[n] = *reinterpret_cast<const Pair *>(full + 2 * (b0 + i0 + n) - (size_t)(1 << (level - 1)) * B * 2 + (size_t)j * B * 2);
    }
    bool valid[2];
    float sum_g[2], sum_h[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const TreeNode &nd = nodes[off + (level == 0 ? 0 : 2 * j + c)];
        valid[c] = nd.is_valid; sum_g[c] = nd.sum_g; sum_h[c] = nd.sum_h;
    }
    const GridScale inv_sg(cell_inv<T>(q, 0)), inv_sh(cell_inv<T>(q, 1));
    T v[4][NB];   // g, h of the left child, g, h of the right one
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        const T cg = cell[n].x, ch = cell[n].y, og = above[n].x - cg, oh = above[n].y - ch;
        if (i0 + n < nb && br >= 0) {
            *reinterpret_cast<Pair *>(built + (size_t)2 * bs * (i0 + n)) = Pair{0, 0};
            T *own = full + 2 * (b0 + i0 + n);
            if (level == 0) *reinterpret_cast<Pair *>(own) = cell[n];   // what the next level subtracts from
            else if (keep) {
                *reinterpret_cast<Pair *>(own + (size_t)(2 * j + br) * B * 2) = cell[n];
                *reinterpret_cast<Pair *>(own + (size_t)(2 * j + 1 - br) * B * 2) = Pair{og, oh};
            }
        }
        v[0][n] = br == 1 ? og : cg; v[1][n] = br == 1 ? oh : ch;
        v[2][n] = br == 1 ? cg : og; v[3][n] = br == 1 ? ch : oh;
    }
    const SplitRec none{0.f, -1, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
    const bool skip = nb == 0 || br < 0 || ignored;   // the same in the whole block, or warp
    if (skip) {
        const int c = packed ? lane : (int)threadIdx.x;
        if (c < n_children && f >= 0) {
            recs[(size_t)(level == 0 ? 0 : 2 * j + c) * F + f] = none;
            __threadfence();
        }
    } else {
        T base[4], tot[4], groups[4] = {0, 0, 0, 0};   // sum before the thread's first bin (float cells: in its group, before its group), sum over all bins
        if constexpr (sizeof(T) == 4) {
            // float cells (first round): eight bins one after the other, then a scan over the 32 groups of eight -- the order
            // of additions this mode's parity with the reference was established with
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                T before = 0;   // sum of the group's bins before the thread's, group = four threads
                T run = v[c][0] + v[c][1];
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                    const T u = shfl_up_t(run, 1);
                    if ((lane & 3) == k) { before = u; run = (u + v[c][0]) + v[c][1]; }
                }
                if ((lane & 3) == 3) s_sum[c][threadIdx.x >> 2] = run;
                base[c] = before;
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                T t = s_sum[c][lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const T u = shfl_up_t(t, o); if (lane >= o) t += u; }
                tot[c] = shfl_t(t, 31);
                const int group = threadIdx.x >> 2;
                const T g = shfl_t(t, max(group - 1, 0));
                groups[c] = group == 0 ? T(0) : g;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const T own = v[c][0] + v[c][1];
                T incl = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const T u = shfl_up_t(incl, o); if (lane >= o) incl += u; }
                if (lane == 31) s_sum[c][warp] = incl;
                base[c] = incl - own;
                tot[c] = packed ? shfl_t(incl, 31) : T(0);
            }
            if (!packed) {
                __syncthreads();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    T all = 0;
#pragma unroll
                    for (int w = 0; w < WARPS; ++w) { if (w == warp) base[c] += all; all += s_sum[c][w]; }
                    tot[c] = all;
                }
            }
        }
        float best_gain[2], keep_g[2], keep_h[2], miss_g[2], miss_h[2], value[2];
        unsigned long long key[2], top[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            key[c] = 0;
            if (c >= n_children) continue;
            const float pg = sum_g[c], ph = sum_h[c];
            const float parent = __fdiv_rn(__fmul_rn(pg, pg), __fadd_rn(ph, lam));
            const float mg = __fsub_rn(pg, cell_f(tot[2 * c], inv_sg)), mh = __fsub_rn(ph, cell_f(tot[2 * c + 1], inv_sh));
            miss_g[c] = mg; miss_h[c] = mh;
            T run_g = base[2 * c], run_h = base[2 * c + 1];
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                const int i = i0 + n;
                T g = groups[2 * c] + run_g, h = groups[2 * c + 1] + run_h;
                if (multi) { g += v[2 * c][n]; h += v[2 * c + 1][n]; }
                run_g += v[2 * c][n]; run_h += v[2 * c + 1][n];
                const float kg = cell_f(g, inv_sg), kh = cell_f(h, inv_sh);   // left sums (multi: right sums) without missing
                const float kg2 = __fadd_rn(kg, mg), kh2 = __fadd_rn(kh, mh);
                const float a = split_gain(parent, pg, ph, kg, kh, mcw, lam), z = split_gain(parent, pg, ph, kg2, kh2, mcw, lam);
                const float gl = fmaxf(0.f, multi ? a : z), gr = fmaxf(0.f, multi ? z : a);   // missing values go left / right
                const float gn = gl > gr ? gl : -gr;
                // arg-abs-max, ties -> smaller bin (hist_tree_builder_single.cu:330-335)
                const unsigned long long kk = ((unsigned long long)__float_as_uint(fabsf(gn)) << 32) | (unsigned)(0x7fffffff - i);
                if (valid[c] && i < nb && kk > key[c]) {
                    key[c] = kk; best_gain[c] = gn; keep_g[c] = kg; keep_h[c] = kh;
                    value[c] = multi ? cut[n + 1] : i ? cut[n] : split_below(cut[n]);
                }
            }
            // largest key of the warp: the gain first, then the bin among the lanes that hold it
            const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key[c] >> 32));
            const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key[c] >> 32) == hi ? (unsigned)key[c] : 0u);
            top[c] = ((unsigned long long)hi << 32) | lo;
            if (lane == 0) s_key[c][warp] = top[c];
        }
        if (!packed) __syncthreads();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (c >= n_children) continue;
            unsigned long long mk = top[c];
            if (!packed) {
#pragma unroll
                for (int w = 0; w < WARPS; ++w) mk = s_key[c][w] > mk ? s_key[c][w] : mk;
            }
            SplitRec *r = recs + (size_t)(level == 0 ? 0 : 2 * j + c) * F + f;
            // the thread that writes the record also makes it visible before the block's ticket is
            if (mk == 0) { if (packed ? lane == 0 : threadIdx.x == 0) { *r = none; __threadfence(); } }   // the node is not valid
            else if (key[c] == mk) {
                *r = SplitRec{best_gain[c], 0x7fffffff - (int)(unsigned)(mk & 0xffffffffull), keep_g[c], keep_h[c], miss_g[c], miss_h[c], value[c], f};
                __threadfence();
            }
        }
    }
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(&ticket[j], 1) == (int)gridDim.x - 1;
        if (last) ticket[j] = 0;
    }
    __syncthreads();
    if (!last || warp >= n_children || !(warp ? valid[1] : valid[0])) return;
    __threadfence();
    best_apply_node(level, level == 0 ? 0 : 2 * j + warp, F, recs, nodes, warp ? sum_g[1] : sum_g[0], warp ? sum_h[1] : sum_h[0], rt_eps, lam, cut_ptr, 0, multi);
}

// The same evaluation for data with many narrow features: one block handles a chunk of whole features whose bins
// add up to at most 256 (a 100k-column one-hot-like data set has one or two bins per feature; a block per feature
// would launch millions of near-empty blocks).  The scan is segmented by feature; the record of a (node, chunk) keeps
// the GLOBAL bin index of its best candidate.  grid = (chunks, pairs); block = 64.
template <typename T>
static __global__ void __launch_bounds__(64)
k_eval_chunk(int level, const Batch b_, int n_chunks, int B, const int *__restrict__ chunk_bin0, const int *__restrict__ cut_ptr,
             const float *__restrict__ cut_val, const int *__restrict__ cut_fid, T *built_all, size_t tree_cells, int bs, const QuantInfo *q, float mcw, float lam,
             const unsigned char *__restrict__ ignored_all, const RoundState *rs, int F, int multi, int by_hessian, int keep) {
    chain_wait();
    const size_t tree = blockIdx.z;
    const TreeNode *nodes = b_.nodes + tree * b_.nodes_stride;
    SplitRec *recs = b_.recs + tree * b_.recs_stride;
    T *full = reinterpret_cast<T *>(b_.hist_full + tree * b_.full_stride) + (size_t)((1 << level) - 1) * B * 2;
    T *built = built_all + tree * tree_cells;
    __shared__ T sg[2][256], sh[2][256];
    const unsigned char *ignored = ignored_all ? ignored_all + (size_t)rs->round * F : nullptr;
    const int c = blockIdx.x, j = blockIdx.y;
    const int b0 = chunk_bin0[c], nb = chunk_bin0[c + 1] - b0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_children = level == 0 ? 1 : 2;
    const int node_local = level == 0 ? 0 : 2 * j + warp;
    const int off = (1 << level) - 1;
    const SplitRec none{0.f, -1, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
    const int br = level == 0 ? 0 : built_side(level, j, b_.seg_cnt[level & 1] + tree * b_.seg_stride, nodes, by_hessian);
    if (nb == 0 || br < 0) {
        if (lane == 0 && warp < n_children) recs[(size_t)node_local * n_chunks + c] = none;
        return;
    }
    {
        // (the loads of all four bins of a thread first: the stores below may alias them as far as the compiler knows)
        using Pair = typename CellPair<T>::type;
        Pair cell[4], above[4];
        T *bp = built + (size_t)j * B * 2 * bs;
        const T *pp = full - (level == 0 ? 0 : (size_t)(1 << (level - 1)) * B * 2) + (size_t)j * B * 2;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = threadIdx.x + 64 * u;
            if (i < nb) {
                cell[u] = *reinterpret_cast<const Pair *>(bp + (size_t)2 * bs * (b0 + i));
                if (level > 0) above[u] = *reinterpret_cast<const Pair *>(pp + 2 * (size_t)(b0 + i));
            }
        }
        T *fb = full + (level == 0 ? 0 : (size_t)(2 * j + br) * B * 2), *fo = full + (size_t)(2 * j + 1 - br) * B * 2;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = threadIdx.x + 64 * u;
            if (i >= nb) continue;
            *reinterpret_cast<Pair *>(bp + (size_t)2 * bs * (b0 + i)) = Pair{0, 0};   // zeroed as it is read, like in k_eval
            if (keep) *reinterpret_cast<Pair *>(fb + 2 * (size_t)(b0 + i)) = cell[u];   // not at the last level, like in k_eval
            const int side = level == 0 ? 0 : br;
            sg[side][i] = cell[u].x; sh[side][i] = cell[u].y;
            if (level > 0) {
                const T og = above[u].x - cell[u].x, oh = above[u].y - cell[u].y;
                sg[1 - br][i] = og; sh[1 - br][i] = oh;
                if (keep) *reinterpret_cast<Pair *>(fo + 2 * (size_t)(b0 + i)) = Pair{og, oh};
            }
        }
    }
    __syncthreads();
    if (warp >= n_children) return;
    const TreeNode nd = nodes[off + node_local];
    if (!nd.is_valid) {
        if (lane == 0) recs[(size_t)node_local * n_chunks + c] = none;
        return;
    }
    // lane-local pass over 8 consecutive bins; sums restart where a feature starts
    T eg[8], eh[8];       // exclusive prefix inside the feature, as far as the lane can see
    bool before_start[8];         // no feature start in this lane up to and including this bin -> add the carry
    T rg = 0, rh = 0;
    bool seen = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int b = lane * 8 + i;
        if (b < nb) {
            const int f = cut_fid[b0 + b];
            if (cut_ptr[f] == b0 + b) { rg = 0; rh = 0; seen = true; }
            eg[i] = rg; eh[i] = rh; before_start[i] = !seen;
            rg += sg[warp][b]; rh += sh[warp][b];
        } else { eg[i] = 0; eh[i] = 0; before_start[i] = false; }
    }
    // segmented inclusive scan of the lanes' open tails (rg, rh); flag = the lane contains a feature start
    T vg = rg, vh = rh;
    bool fl = seen;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T ug = shfl_up_t(vg, o), uh = shfl_up_t(vh, o);
        const int uf = __shfl_up_sync(0xffffffffu, (int)fl, o);
        if (lane >= o) {
            if (!fl) { vg += ug; vh += uh; }
            fl = fl || uf;
        }
    }
    T cg = shfl_up_t(vg, 1), ch = shfl_up_t(vh, 1);  // carry into this lane = inclusive value of lane-1
    if (lane == 0) { cg = 0; ch = 0; }
    // inclusive prefix per bin back into shared memory: the last bin of a feature then holds the feature total
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int b = lane * 8 + i;
        if (b < nb) {
            if (before_start[i]) { eg[i] += cg; eh[i] += ch; }
            const T ig = eg[i] + sg[warp][b], ih = eh[i] + sh[warp][b];
            sg[warp][b] = ig; sh[warp][b] = ih;
        }
    }
    __syncwarp();
    const float pg = nd.sum_g, ph = nd.sum_h, parent = __fdiv_rn(__fmul_rn(pg, pg), __fadd_rn(ph, lam));
    const GridScale inv_sg(cell_inv<T>(q, 0)), inv_sh(cell_inv<T>(q, 1));
    float best = 0.f, best_lg = 0.f, best_lh = 0.f, best_mg = 0.f, best_mh = 0.f;
    int best_bin = -1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int b = lane * 8 + i;
        if (b < nb && !(ignored && ignored[cut_fid[b0 + b]])) {
            const int f = cut_fid[b0 + b];
            const int lastb = cut_ptr[f + 1] - 1 - b0;
            const float mg = __fsub_rn(pg, cell_f(sg[warp][lastb], inv_sg)), mh = __fsub_rn(ph, cell_f(sh[warp][lastb], inv_sh));
            float gn, keep_g, keep_h;
            if (multi) {  // inclusive prefix = right child, see k_eval
                const float rg = cell_f(sg[warp][b], inv_sg), rh = cell_f(sh[warp][b], inv_sh);
                const float gl = fmaxf(0.f, split_gain(parent, pg, ph, rg, rh, mcw, lam));
                const float rg2 = __fadd_rn(rg, mg), rh2 = __fadd_rn(rh, mh);
                const float gr = fmaxf(0.f, split_gain(parent, pg, ph, rg2, rh2, mcw, lam));
                gn = gl > gr ? gl : -gr; keep_g = rg; keep_h = rh;
            } else {
                const float lg = cell_f(eg[i], inv_sg), lh = cell_f(eh[i], inv_sh);
                const float gr = fmaxf(0.f, split_gain(parent, pg, ph, lg, lh, mcw, lam));
                const float lg2 = __fadd_rn(lg, mg), lh2 = __fadd_rn(lh, mh);
                const float gl = fmaxf(0.f, split_gain(parent, pg, ph, lg2, lh2, mcw, lam));
                gn = gl > gr ? gl : -gr; keep_g = lg; keep_h = lh;
            }
            if (best_bin < 0 || fabsf(gn) > fabsf(best)) { best = gn; best_bin = b0 + b; best_lg = keep_g; best_lh = keep_h; best_mg = mg; best_mh = mh; }
        }
    }
    unsigned long long key = best_bin < 0 ? 0ull
                                          : (((unsigned long long)__float_as_uint(fabsf(best)) << 32) | (unsigned)(0x7fffffff - best_bin));
    unsigned long long mk = key;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = (unsigned long long)shfl_xor_ll((long long)mk, o);
        mk = other > mk ? other : mk;
    }
    if (mk == 0) { if (lane == 0) recs[(size_t)node_local * n_chunks + c] = none; }   // every column of the chunk is left out
    else if (key == mk) {
        const int f = cut_fid[best_bin];
        recs[(size_t)node_local * n_chunks + c] = SplitRec{best, best_bin, best_lg, best_lh, best_mg, best_mh, split_at(cut_val + cut_ptr[f], best_bin - cut_ptr[f], multi), f};
    }
}


// ------------------------------------------------------------------ rows to their children
// (replaces update_ins2node_id + the per-level radix sort, hist_tree_builder_single.cu:908-1020, :397-415)
// One pass over the rows in row order.  10.5 M rows: 35 us at the root, 41 to 53 below; moving records of row id and gradients
// instead, a pass to count and one to scatter them, took 64 to 88.  (The gradients by row cost the histogram kernels 8 of 58 ms
// per 100 trees; the final walk through all levels, 133 us, became one step of 81.)  Every row keeps its node (`nid`, two bytes), looks up the split, and its id is written
// to the list of its child.  The gradients are not moved: the histogram kernels fetch them by row.  A block handles a chunk of
// neighbouring rows: rank of every row among the chunk's rows of its child (ballots and one shared atomic per warp and child), one
// global atomic per child for the chunk's place in the list, and the ids, sorted by child in shared memory, go out as runs.
// The chunks of a list therefore stand in the order their blocks came by, roughly ascending; the sums do not depend on it.
// Rows of nodes that stopped splitting keep their node and are in no list.
// CSR layout: the row's bin among the bins [span.x, span.y) of a feature, searched in its ascending bin ids (hist_tree_builder_single.cu:941-966)
__device__ __forceinline__ unsigned csr_bin(const int *__restrict__ row_ptr, const int *__restrict__ bin, int2 span, int r) {
    const int c0 = span.x, c1 = span.y;
    if (c0 == c1) return MISSING_BIN;
    int lo = row_ptr[r], hi = row_ptr[r + 1];
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2, v = bin[mid];
        if (v >= c0 && v < c1) return (unsigned)(v - c0);
        if (v < c0) lo = mid + 1; else hi = mid;
    }
    return MISSING_BIN;
}

// The pass is bound by the instructions per row (127 in a first version with a test per row for every special case: 60 us at
// any level of 10.5 M rows), hence: rows that go nowhere have a dummy child behind the others, whose rows are ranked and staged
// like the rest and never read; a node's rule comes as one 16-byte word with the column's address; the next chunk's nodes and
// bins are on their way while a chunk is ranked.
// order: ASSIGN_ANY as above.  The float rounds keep the lists in row order, as what their sums come to depends on it (with lists in
// order to the chunk only, 7 % of trainings of 100 k rows fell on the other side of a near-tie that row order decides one
// way): ASSIGN_COUNT leaves the children's rows of every block's run of chunks in `table` ([blocks][2 nl] a tree), ASSIGN_PLACE
// starts from those of the blocks before, which it adds up (ASSIGN_PLACE_ADD) or finds there (k_assign_before has been).  1 M rows x 28:
// 12 to 14 us each of the two, 7 to 10 the one launch of ASSIGN_ANY (counting and scattering records took 7 and 9).
// RPT: rows per thread; eight where there are enough rows for it (BoosterImpl::assign_rpt).  The upper levels spill: 40 bytes with eight
// rows (BITS 1 to 3), 48 with four (BITS 2 and 3), of 64 and 40 registers.
// BITS: 1 to 3, the levels whose children (2^BITS) are few, ranked by ballots and one shared atomic per warp and child;
// 0: many children, one shared atomic per row, the lanes seldom meet.
enum AssignOrder { ASSIGN_ANY = 0, ASSIGN_COUNT = 1, ASSIGN_PLACE = 2, ASSIGN_PLACE_ADD = 3 };
struct alignas(16) ChunkRule {
    union {
        const unsigned char *col;   // dense: bins of the feature by row
        int2 span;                  // CSR: the feature's bins
    };
    unsigned code;                  // threshold << 23 | first child << 8 | shift
    unsigned pad;
};

// CSR layout with sorted columns: the rows that store the split column of their node go first, found in the column instead of
// searching the column in every row (1 M rows x 36 values: 45 us a level searching, five dependent reads a row).  grid = (blocks, nodes, trees)
static __global__ void __launch_bounds__(256)
k_assign_stored(int level, const Batch b, const SparseColumns c, const int *__restrict__ cut_ptr, int rev) {
    chain_wait();
    const size_t tree = blockIdx.z;
    const int nl = 1 << level;
    unsigned short *nid = b.nid + tree * b.nid_stride;
    for (int n = blockIdx.y; n < nl; n += gridDim.y) {
        const TreeNode &nd = b.nodes[tree * b.nodes_stride + nl - 1 + n];
        if (!nd.is_valid || nd.is_leaf) continue;
        const int2 span = make_int2(cut_ptr[nd.split_feature_id], cut_ptr[nd.split_feature_id + 1]);
        if (!by_column(c.bin_ptr, span, b.seg_cnt[level & 1][tree * b.seg_stride + n])) continue;
        // bins below the split bin go left (rev: those beyond it, the split bin itself goes right)
        const unsigned split = c.bin_ptr[span.x + nd.split_bid + (rev ? 1 : 0)];
        const unsigned short me = (unsigned short)(nl - 1 + n), left = (unsigned short)(2 * me + 1), right = (unsigned short)(2 * me + 2);
        each_step(c.bin_ptr[span.x], c.bin_ptr[span.y], blockIdx.x * 256 + threadIdx.x, gridDim.x * 256, [&](unsigned e) {
            const int r = c.row[e];
            if (nid[r] == me) nid[r] = (e < split) != (rev != 0) ? left : right;
        });
    }
}

// Row counts of the blocks -> those of the blocks before, child by child.  A block takes 32 children, a warp 1/32 of the table's
// rows of them.  Its 9 us (888 blocks) are latency.  Up to ASSIGN_ADD entries of the table every block of ASSIGN_PLACE_ADD adds up the
// rows before its own instead, which reads half of the table per block: 888 blocks with 8 children 2 us, with 16 and 32 30 on average,
// with 2048 6.4 ms.  grid = (children / 32, 1, trees)
constexpr int ASSIGN_ADD = 8192;
static __global__ void __launch_bounds__(1024)
k_assign_before(int blocks, int children, int *table) {
    chain_wait();
    __shared__ int part[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane, run = (blocks + 31) / 32;
    const int k0 = min(blocks, warp * run), k1 = min(blocks, k0 + run);
    int *at = table + (size_t)blockIdx.z * blocks * children + c;
    int sum = 0;
    if (c < children)
#pragma unroll 8
        for (int k = k0; k < k1; ++k) sum += at[(size_t)k * children];
    part[warp][lane] = sum;
    __syncthreads();
    if (c >= children) return;
    int before = 0;
    for (int w = 0; w < warp; ++w) before += part[w][lane];
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
        const int n = at[(size_t)k * children];
        at[(size_t)k * children] = before;
        before += n;
    }
}

template <bool SPARSE, int RPT, int BITS, bool ORDERED>
static __global__ void __launch_bounds__(ASSIGN_THREADS, SPARSE || RPT == 8 ? 4 : 6)
k_assign(int level, const Batch b, int n_rows, const unsigned char *__restrict__ binsT, size_t Npad, const int *__restrict__ sp_row_ptr,
         const int *__restrict__ sp_bin, const int *__restrict__ cut_ptr, const SparseColumns cols, int rev, int how, int *table) {
    const int order = !ORDERED ? (int)ASSIGN_ANY : how == ASSIGN_PLACE_ADD ? (int)ASSIGN_PLACE : how;
    constexpr int ROWS = RPT * ASSIGN_THREADS;   // at most 8192: 13 bits of a staged entry
    extern __shared__ __align__(16) unsigned char assign_sm[];
    __shared__ int scratch[33];
    if (BITS) level = BITS - 1;
    const int nl = 1 << level, lane = threadIdx.x & 31, in = level & 1;
    ChunkRule *rule = reinterpret_cast<ChunkRule *>(assign_sm);          // [nl + 1], the last one for rows of finished nodes
    unsigned *stage = reinterpret_cast<unsigned *>(rule + nl + 1);        // [ROWS] child << 13 | row of the chunk
    int *s_cnt = reinterpret_cast<int *>(stage + ROWS);                   // [2 nl + 1] rows of the chunk per child
    int *s_pre = s_cnt + 2 * nl + 1, *s_to = s_pre + 2 * nl + 1;          // [2 nl + 1] those before the child's; list position less that
    const size_t tree = blockIdx.z;
    const TreeNode *nodes = b.nodes + tree * b.nodes_stride + nl - 1;
    unsigned short *nid = b.nid + tree * b.nid_stride;
    const int *next_begin = b.seg_begin[in ^ 1] + tree * b.seg_stride;
    int *next_cnt = b.seg_cnt[in ^ 1] + tree * b.seg_stride, *list = b.rec_idx + tree * b.rec_stride;
    for (int i = threadIdx.x; i <= 2 * nl; i += ASSIGN_THREADS) s_cnt[i] = 0;
    chain_wait();
    const int chunks = (n_rows + ROWS - 1) / ROWS;
    unsigned at[RPT];   // level's node of the rows to come, nl: none
    auto load_nodes = [&](int chunk) {   // (the table ends with a whole chunk; what lies behind the rows stays at node 0)
        const unsigned short *p = nid + (size_t)chunk * ROWS + threadIdx.x;
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            if (BITS == 1) at[u] = chunk * ROWS + u * ASSIGN_THREADS + (int)threadIdx.x >= n_rows ? 3u : SPARSE ? (unsigned)p[u * ASSIGN_THREADS] : 0u;
            else at[u] = (unsigned)p[u * ASSIGN_THREADS];
        }
    };
    const int run = order == ASSIGN_ANY ? 1 : (chunks + (int)gridDim.x - 1) / (int)gridDim.x, step = order == ASSIGN_ANY ? (int)gridDim.x : 1;
    int chunk = blockIdx.x * run;
    const int chunk_end = order == ASSIGN_ANY ? chunks : min(chunks, chunk + run);
    if (chunk < chunk_end) load_nodes(chunk);
    for (int i = threadIdx.x; i <= nl; i += ASSIGN_THREADS) {
        AssignRule r{0, ASSIGN_NONE};
        if (i < nl) r = assign_rule(nodes[i], nodes[i].is_valid && !nodes[i].is_leaf, rev);
        const bool none = r.test == ASSIGN_NONE;   // always left, to the dummy
        ChunkRule x;
        if (SPARSE) {
            x.span = none ? make_int2(0, 0) : make_int2(cut_ptr[r.feature], cut_ptr[r.feature + 1]);
            if (!none && by_column(cols.bin_ptr, x.span, b.seg_cnt[in][tree * b.seg_stride + i])) x.span = make_int2(0, 0);   // who is still here stores no value
        }
        else x.col = binsT + (size_t)r.feature * Npad;
        x.code = none ? ((rev ? 0u : 256u) << 23) | ((unsigned)(2 * nl) << 8) : ((r.test >> 1) << 23) | ((unsigned)(2 * i) << 8) | (r.test & 1u);
        x.pad = 0;
        rule[i] = x;
    }
    // in s_to from here on: where the child's next rows go
    table += (tree * gridDim.x + blockIdx.x) * (size_t)(2 * nl);
    if (ORDERED && how == ASSIGN_PLACE_ADD)
        for (int i = threadIdx.x >> 5; i < 2 * nl; i += ASSIGN_THREADS / 32) {
            int before = 0;
            for (int k = lane; k < (int)blockIdx.x; k += 32) before += table[i - (long long)(k + 1) * (2 * nl)];
            before = __reduce_add_sync(0xffffffffu, before);
            if (lane == 0) s_to[i] = next_begin[i] + before;
        }
    else if (order == ASSIGN_PLACE)
        for (int i = threadIdx.x; i < 2 * nl; i += ASSIGN_THREADS) s_to[i] = next_begin[i] + table[i];
    if (blockIdx.x == 0 && order != ASSIGN_COUNT) {   // rows that are looked at, for the byte counter
        int rows = 0;
        for (int i = threadIdx.x; i < nl; i += ASSIGN_THREADS) rows += b.seg_cnt[in][tree * b.seg_stride + i];
        rows = __reduce_add_sync(0xffffffffu, rows);
        if (lane == 0 && rows) atomicAdd(&b.ctl->stat_part_rows, (unsigned long long)rows);
    }
    __syncthreads();
    unsigned code[RPT], bin[RPT];
    auto load_bins = [&](int chunk) {
        const int mine = chunk * ROWS + threadIdx.x;
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            const unsigned from = at[u] - (unsigned)(nl - 1);
            const ChunkRule q = rule[min(from, (unsigned)nl)];   // (a node further up: beyond nl)
            code[u] = q.code;
            // gone already, by its stored value
            if (SPARSE && from - (unsigned)nl < (unsigned)(2 * nl)) code[u] = ((rev ? 0u : 256u) << 23) | ((from - (unsigned)nl) << 8);
            const int r = mine + u * ASSIGN_THREADS;
            if (SPARSE) bin[u] = csr_bin(sp_row_ptr, sp_bin, q.span, r);
            else bin[u] = q.col[r];   // (behind the last row: the first column's, allocated to the end of a chunk)
        }
    };
    if (chunk < chunk_end) load_bins(chunk);
    for (; chunk < chunk_end; chunk += step) {
        const int row0 = chunk * ROWS;
        unsigned c[RPT];
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            const bool left = (((bin[u] + code[u]) & 0xffu) < (code[u] >> 23)) != (rev != 0);
            c[u] = (code[u] >> 8 & 0x7fffu) + (left ? 0u : 1u);
            if (order != ASSIGN_COUNT && (BITS == 1 || c[u] < (unsigned)(2 * nl)))
                nid[(size_t)row0 + u * ASSIGN_THREADS + threadIdx.x] = (unsigned short)(c[u] < (unsigned)(2 * nl) ? 2 * nl - 1 + c[u] : 0u);
        }
        const bool more = chunk + step < chunk_end;
        if (more) load_nodes(chunk + step);
        int rank[RPT];
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            if (order == ASSIGN_PLACE) {   // warp after warp
                const unsigned same = __match_any_sync(0xffffffffu, c[u]), below = same & ((1u << lane) - 1u);
                for (int w = 0; w < ASSIGN_THREADS / 32; ++w) {
                    if ((int)(threadIdx.x >> 5) == w) {
                        int first = 0;
                        if (below == 0) first = atomicAdd(&s_cnt[c[u]], __popc(same));
                        rank[u] = __shfl_sync(0xffffffffu, first, __ffs(same) - 1) + __popc(below);
                    }
                    __syncthreads();
                }
            } else if (BITS == 0) rank[u] = atomicAdd(&s_cnt[c[u]], 1);
            else {
                unsigned same = __ballot_sync(0xffffffffu, c[u] < (unsigned)(2 * nl));   // lanes with the same child
#pragma unroll
                for (int k = 0; k < BITS; ++k) {
                    const unsigned v = __ballot_sync(0xffffffffu, c[u] >> k & 1u);
                    same &= c[u] >> k & 1u ? v : ~v;
                }
                const unsigned below = same & ((1u << lane) - 1u);
                int first = 0;
                if (c[u] < (unsigned)(2 * nl) && below == 0) first = atomicAdd(&s_cnt[c[u]], __popc(same));
                rank[u] = __shfl_sync(0xffffffffu, first, __ffs(same) - 1) + __popc(below);
            }
        }
        if (more) load_bins(chunk + step);
        if (order == ASSIGN_COUNT) continue;
        __syncthreads();
        const int total = block_prefix<ASSIGN_THREADS>(2 * nl, [&](int i) { return s_cnt[i]; }, [&](int i, int before) { s_pre[i] = before; }, scratch);
        for (int i = threadIdx.x; i < 2 * nl; i += ASSIGN_THREADS) {   // (on its way while the rows are staged)
            const int n = s_cnt[i];
            s_cnt[i] = 0;
            if (order == ASSIGN_PLACE) {
                s_to[i] -= s_pre[i];
                s_cnt[i] = n;   // (for the next chunk's place, below)
            } else if (n) s_to[i] = next_begin[i] + atomicAdd(next_cnt + i, n) - s_pre[i];
        }
        if (threadIdx.x == 0) s_cnt[2 * nl] = 0;
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
            const unsigned v = (c[u] << 13) | (unsigned)(u * ASSIGN_THREADS + threadIdx.x);
            if (c[u] < (unsigned)(2 * nl)) stage[s_pre[c[u]] + rank[u]] = v;
        }
        __syncthreads();
#pragma unroll 4
        for (int i = threadIdx.x; i < total; i += ASSIGN_THREADS) {
            const unsigned w = stage[i];
            list[s_to[w >> 13] + i] = row0 + (int)(w & 8191u);
        }
        if (order == ASSIGN_PLACE) {
            __syncthreads();
            for (int i = threadIdx.x; i < 2 * nl; i += ASSIGN_THREADS) { s_to[i] += s_pre[i] + s_cnt[i]; s_cnt[i] = 0; }
            __syncthreads();
        }
    }
    if (order == ASSIGN_ANY) return;
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * nl; i += ASSIGN_THREADS) {
        if (order == ASSIGN_COUNT) table[i] = s_cnt[i];
        else if (blockIdx.x == gridDim.x - 1) next_cnt[i] = s_to[i] - next_begin[i];
    }
}

// ------------------------------------------------------------------ end of tree
// TreeBuilder::predict_in_training (src/thundergbm/builder/tree_builder.cu:62-74); nvcc contracts the reference's
// `y += lr * w` into one fused multiply-add, written out here.  The last level's split is applied on the way.  A node was split iff its children are valid; pruning only marks nodes, so the row's node is the
// one the reference's table would hold (`nid_out`) while the score takes the weight of the deepest node on the path that
// survived pruning (`weight`, left by leave_rules like the rules of the last level; feature < 0: who stores the split column has
// gone, see k_assign_stored).
constexpr int APPLY_RPT = 4;   // rows in flight per thread
template <bool SPARSE>
static __global__ void __launch_bounds__(256)
k_apply_tree(const Batch b, int n_rows, int last_level, const unsigned char *__restrict__ binsT, size_t Npad, const int *__restrict__ sp_row_ptr,
             const int *__restrict__ sp_bin, const int *__restrict__ cut_ptr, float lr, float *yp, int *__restrict__ nid_out,
             const float *__restrict__ y, int fuse_objective, double *metric_partial, unsigned *maxbits, int rev) {
    chain_wait();
    // fuse_objective >= 0 (a pointwise objective, one tree per round): the same pass adds up the round's training
    // metric (same grid, same order of additions as k_metric_partial) and finds the maxima of the next round's
    // gradients, so that neither needs a pass of its own over y and the scores.
    const bool fuse = fuse_objective >= 0;
    const int fuse_logistic = fuse_objective == REG_LINEAR ? 0 : 1;
    const size_t tree = blockIdx.y;
    unsigned short *nid = b.nid + tree * b.nid_stride;
    const float *weight = b.weight + tree * b.nodes_stride;
    const AssignRule *rule = b.rule + tree * b.rule_stride;
    yp += tree * n_rows;
    if (nid_out) nid_out += tree * n_rows;
    const bool coarse = b.ctl->coarse;   // the round will be built again
    if (coarse && !SPARSE) return;
    const unsigned nl = 1u << last_level, off = nl - 1u;
    double msum = 0;
    float mg = 0.f, mh = 0.f;
    const int step = gridDim.x * blockDim.x;
    for (int r0 = blockIdx.x * blockDim.x + threadIdx.x; r0 < n_rows; r0 += APPLY_RPT * step) {
        unsigned at[APPLY_RPT], bin[APPLY_RPT];
        float score[APPLY_RPT], yr[APPLY_RPT];
        AssignRule x[APPLY_RPT];
#pragma unroll
        for (int u = 0; u < APPLY_RPT; ++u) {
            const int r = r0 + u * step;
            const bool in = r < n_rows;
            at[u] = in && (SPARSE || last_level != 0) ? nid[r] : 0u;
            if (SPARSE && in) nid[r] = 0;   // the next tree's stored values look for the root there
            score[u] = in ? yp[r] : 0.f;
            yr[u] = in && fuse ? y[r] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < APPLY_RPT; ++u) x[u] = at[u] - off < nl ? rule[at[u] - off] : AssignRule{0, ASSIGN_NONE};
#pragma unroll
        for (int u = 0; u < APPLY_RPT; ++u) {
            const int r = r0 + u * step;
            bin[u] = 0;
            if (x[u].test == ASSIGN_NONE || r >= n_rows) continue;
            if (!SPARSE) bin[u] = binsT[(size_t)x[u].feature * Npad + r];
            else if (x[u].feature < 0) bin[u] = MISSING_BIN;
            else bin[u] = csr_bin(sp_row_ptr, sp_bin, make_int2(cut_ptr[x[u].feature], cut_ptr[x[u].feature + 1]), r);
        }
#pragma unroll
        for (int u = 0; u < APPLY_RPT; ++u) {
            const int r = r0 + u * step;
            if (r >= n_rows || coarse) break;
            if (x[u].test != ASSIGN_NONE) at[u] = 2 * at[u] + (assign_left(x[u].test, bin[u], rev) ? 1u : 2u);
            if (nid_out) nid_out[r] = (int)at[u];
            const float s = __fmaf_rn(lr, weight[at[u]], score[u]);
            yp[r] = s;
            if (fuse) {
                msum += pointwise_metric_term(fuse_objective, yr[u], s);
                const float2 v = pointwise_gh(fuse_logistic, yr[u], s);
                mg = fmaxf(mg, fabsf(v.x)); mh = fmaxf(mh, v.y);
            }
        }
    }
    if (fuse && !coarse) {
        __shared__ double part[8];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) msum += __shfl_xor_sync(0xffffffffu, msum, o);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = msum;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
            metric_partial[blockIdx.x] = t;
        }
        track_max(mg, mh, maxbits);
    }
}

}  // namespace tgbm
