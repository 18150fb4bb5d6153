// A whole tree in one launch, for data of a few thousand rows.
//
// With the kernels of tgbm_level.cuh a level of a small tree takes 30 us whatever it does: four launches, each a chain of
// dependent L2 accesses through segment tables, record lists and histograms in global memory.  Here ONE cluster of CTAs
// builds the tree.  Every CTA owns a share of the features and walks ALL rows for them, so histograms never meet across
// CTAs; the node of every row is kept in shared memory (each CTA its own copy, updated redundantly), the rows are not
// moved at all, every node's histogram is built (nothing is subtracted: the sums are integers and come out the same), and
// what the CTAs exchange per level is the best candidate of every node -- written to the own shared memory, read by the
// others through the cluster -- behind one cluster barrier.
//
// Bound by the shared-memory atomics of the rows x own features (four 32-bit halves per value, random banks; 12 k cycles a level
// for 10000 rows x 2 features a CTA) and by the split search (128 units of 255 bins a tree, 8 k cycles for 32 of them).
// 10000 rows x 32 features, depth 6: 124 us a tree (level kernels 185), 1605 rows x 119 features: 63 us (165).  64 registers, 28 to 32
// bytes of them spilled.  LOCAL: up to SMALL_LOCAL rows, which every CTA moves for itself; a kernel of its own, as either way of moving
// rows costs the other 3 % by its registers.
// Same integer sums, gains, tie rules and node records as the level kernels, bit for bit.
#pragma once
#include <cooperative_groups.h>

#include "tgbm_level.cuh"

namespace tgbm {

constexpr int SMALL_THREADS = 1024, SMALL_ROWS = 32768;   // most rows
constexpr int SMALL_LOCAL = 4 * SMALL_THREADS;            // rows that every CTA moves for itself

struct SmallPost {   // a CTA's best candidate of a node: |gain| bits << 32 | (0x7fffffff - feature), 0 = none
    unsigned long long key;
    SplitRec rec;
};

// A feature's bins stand one word further apart every eighth bin, so that the lanes of the split search, eight consecutive bins
// each, read from different banks (eight lanes on every bank they used cost a third of the search).
__host__ __device__ constexpr int small_at(int bin) { return bin + (bin >> 3); }
__host__ __device__ constexpr int small_feature_at(int first_bin, int f) { return small_at(first_bin) + f; }   // f-th feature of a CTA, bins before it

struct SmallPlan {   // sizes fixed by the host (BoosterImpl::plan_small_trees)
    int cluster, feats, bins;   // CTAs per tree, features per CTA, most bins of a CTA
    int cells;                  // words that these take
    int most;                   // most bins of a feature
    int nodes_pass;             // nodes whose histograms are in shared memory at a time
    size_t smem;
};

// Best candidate of one (node, feature), or of its `part` of `parts`: LANES neighbouring lanes own BPL consecutive bins each.  With
// parts the sums of the others come from `sums` ([parts] g, h), which small_sums has left.
struct SmallSums { long long g, h; };
template <int LANES, int BPL>
__device__ __forceinline__ void small_load(const int *cell, int words, int b0, int nb, long long (&g)[BPL], long long (&h)[BPL], SmallSums &own) {
    own = SmallSums{0, 0};
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        const int b = b0 + i;
        g[i] = h[i] = 0;
        if (b < nb) {
            const int *c = cell + small_at(b);
            g[i] = ((long long)c[2 * words] << 16) + (unsigned)c[0];
            h[i] = ((long long)c[3 * words] << 16) + (unsigned)c[words];
        }
        own.g += g[i]; own.h += h[i];
    }
}
template <int BPL>
__device__ __forceinline__ void small_sums(const int *cell, int words, int nb, int part, SmallSums *sums) {
    const int lane = threadIdx.x & 31;
    long long g[BPL], h[BPL];
    SmallSums t;
    small_load<32, BPL>(cell, words, (part * 32 + lane) * BPL, nb, g, h, t);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { t.g += shfl_xor_ll(t.g, o); t.h += shfl_xor_ll(t.h, o); }
    if (lane == 0) sums[part] = t;
}
// (Of up to four bins a lane in place, 0.4 us a level less than a call; the others are functions of their own: inlined, their arrays and
// what the kernel holds meanwhile do not fit 64 registers.)
struct SmallSearch {   // what is the same for all of them
    GridScale inv_sg, inv_sh;
    float mcw, lam;
    int multi, words;
};
template <int LANES, int BPL>
__device__ __forceinline__ void small_eval(const SmallSearch &x, const int *cell, int nb, float pg, float ph, int part, int parts, const SmallSums *sums, bool active,
                                        SplitRec *out) {
    const GridScale inv_sg = x.inv_sg, inv_sh = x.inv_sh;
    const float mcw = x.mcw, lam = x.lam;
    const int multi = x.multi, words = x.words;
    const int lane = threadIdx.x & (LANES - 1), b0 = (part * LANES + lane) * BPL;
    if (!active) nb = 0;
    long long g[BPL], h[BPL];
    SmallSums own;
    small_load<LANES, BPL>(cell, words, b0, nb, g, h, own);
    long long ig = own.g, ih = own.h;
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1) {
        const long long ug = shfl_up_ll(ig, o), uh = shfl_up_ll(ih, o);
        if (lane >= o) { ig += ug; ih += uh; }
    }
    long long all_g, all_h, rg = ig - own.g, rh = ih - own.h;
    if (parts == 1) {
        const int top = (threadIdx.x & 31) | (LANES - 1);
        all_g = shfl_ll(ig, top); all_h = shfl_ll(ih, top);
    } else {
        all_g = all_h = 0;
        for (int q = 0; q < parts; ++q) {
            if (q == part) { rg += all_g; rh += all_h; }
            all_g += sums[q].g; all_h += sums[q].h;
        }
    }
    const float mg = __fsub_rn(pg, inv_sg(all_g)), mh = __fsub_rn(ph, inv_sh(all_h));
    const float parent = __fdiv_rn(__fmul_rn(pg, pg), __fadd_rn(ph, lam));
    unsigned long long key = 0;
    float best = 0.f, keep_g = 0.f, keep_h = 0.f;
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        const int b = b0 + i;
        if (multi) { rg += g[i]; rh += h[i]; }
        const float kg = inv_sg(rg), kh = inv_sh(rh);   // see k_eval
        if (!multi) { rg += g[i]; rh += h[i]; }
        const float a = split_gain(parent, pg, ph, kg, kh, mcw, lam), z = split_gain(parent, pg, ph, __fadd_rn(kg, mg), __fadd_rn(kh, mh), mcw, lam);
        const float gl = fmaxf(0.f, multi ? a : z), gr = fmaxf(0.f, multi ? z : a);
        const float gn = gl > gr ? gl : -gr;
        const unsigned long long kk = ((unsigned long long)__float_as_uint(fabsf(gn)) << 32) | (unsigned)(0x7fffffff - b);
        if (b < nb && kk > key) { key = kk; best = gn; keep_g = kg; keep_h = kh; }
    }
    unsigned long long top;
    if (LANES == 32) {
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
        top = ((unsigned long long)hi << 32) | __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    } else {
        top = key;
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            const unsigned long long x = (unsigned long long)shfl_xor_ll((long long)top, o);
            top = x > top ? x : top;
        }
    }
    if (!active) return;
    if (top == 0) { if (lane == 0) out->bin = -1; }   // (a part without bins)
    else if (key == top) *out = SplitRec{best, 0x7fffffff - (int)(unsigned)top, keep_g, keep_h, mg, mh, 0.f, 0};
}

template <int LANES, int BPL>
__device__ __noinline__ void small_eval_call(const SmallSearch &x, const int *cell, int nb, float pg, float ph, int part, int parts, const SmallSums *sums, bool active,
                                             SplitRec *out) {
    small_eval<LANES, BPL>(x, cell, nb, pg, ph, part, parts, sums, active, out);
}

// grid = trees x plan.cluster, clusters of plan.cluster CTAs
template <bool LOCAL>
static __global__ void __launch_bounds__(SMALL_THREADS, 1)
k_small_tree(const SmallPlan plan, int N, size_t Npad, int F, int depth, const unsigned char *__restrict__ binsT, const int *__restrict__ cut_ptr,
             const float *__restrict__ cut_val, const int2 *ghq, const unsigned long long *root_sum, const QuantInfo *q, float mcw, float lam,
             float rt_eps, float gamma, const unsigned char *__restrict__ ignored_all, const RoundState *rs, int multi, TreeNode *nodes_out,
             TreeNode *model, int K, int k0, unsigned *maxbits, int fine_K, TreeCtl *ctl, long long *hist_full, size_t full_stride,
             unsigned short *nid, size_t nid_stride, float *weight, AssignRule *rule, size_t rule_stride) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char small_sm[];
    __shared__ int scratch[33], s_split;
    __shared__ __align__(8) unsigned char search_sm[sizeof(SmallSearch)];
    SmallSearch &s_search = *reinterpret_cast<SmallSearch *>(search_sm);
    __shared__ SmallSums s_sums[SMALL_THREADS / 32];
    __shared__ SplitRec s_parts[SMALL_THREADS / 32];
    const int n_nodes = (1 << (depth + 1)) - 1, max_nl = 1 << (depth - 1);
    TreeNode *nodes = reinterpret_cast<TreeNode *>(small_sm);
    SmallPost *posts = reinterpret_cast<SmallPost *>(small_sm + (sizeof(TreeNode) * n_nodes + 15) / 16 * 16);   // [2][max_nl]
    SplitRec *recs = reinterpret_cast<SplitRec *>(posts + 2 * max_nl);                                       // [nodes_pass][feats]
    unsigned *split = reinterpret_cast<unsigned *>(recs + plan.nodes_pass * plan.feats);                 // [max_nl] what the level decided
    unsigned short *node_of = reinterpret_cast<unsigned short *>(split + (max_nl + 3) / 4 * 4);            // [N, eights]
    int *s_first = reinterpret_cast<int *>(node_of + (N + 7) / 8 * 8);                                           // [feats + 1] bins before the own features
    float *s_cut = reinterpret_cast<float *>(s_first + plan.feats + 1);                                          // [bins] their cut points
    int *acc = reinterpret_cast<int *>(s_cut + plan.bins);                                                       // [4][nodes_pass * cells]
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), tree = blockIdx.x / plan.cluster, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f0 = min(F, rank * plan.feats), nf = min(F, f0 + plan.feats) - f0, bin0 = cut_ptr[f0], words = plan.nodes_pass * plan.cells;
    const int share = (N + plan.cluster - 1) / plan.cluster, share0 = min(N, rank * share), share1 = min(N, share0 + share);   // rows whose node this CTA reports
    for (int r = threadIdx.x; r < N; r += SMALL_THREADS) node_of[r] = 0;
    for (int f = threadIdx.x; f <= plan.feats; f += SMALL_THREADS) s_first[f] = cut_ptr[min(F, f0 + f)] - bin0;
    chain_wait();
    if (blockIdx.x == 0 && threadIdx.x == SMALL_THREADS - 1) next_maxima(root_sum, fine_K, maxbits, ctl);   // (a thread that has nothing else to do yet)
    const int2 *gq = ghq + (size_t)tree * N;
    const GridScale inv_sg(q->inv_sg), inv_sh(q->inv_sh);
    if (threadIdx.x == 0) s_search = SmallSearch{inv_sg, inv_sh, mcw, lam, multi, words};
    const unsigned char *ignored = ignored_all ? ignored_all + (size_t)rs->round * F : nullptr;
    for (int i = threadIdx.x; i < n_nodes; i += SMALL_THREADS) {   // Tree::init2, as k_tree_init
        TreeNode t;
        memset(&t, 0, sizeof(t));
        t.final_id = i;
        t.split_feature_id = -1;
        t.parent_index = i == 0 ? -1 : (i - 1) / 2;
        if (i < n_nodes / 2) { t.is_leaf = 0; t.lch_index = 2 * i + 1; t.rch_index = 2 * i + 2; }
        else { t.is_leaf = 1; t.lch_index = -1; t.rch_index = -1; }
        if (i == 0) {
            t.sum_g = inv_sg((long long)root_sum[2 * tree]);
            t.sum_h = inv_sh((long long)root_sum[2 * tree + 1]);
            t.is_valid = 1;
            t.base_weight = __fdiv_rn(-t.sum_g, __fadd_rn(t.sum_h, lam));
        }
        nodes[i] = t;
    }
    __syncthreads();
    bool moved = false;
    unsigned short *my_nid = nid + (size_t)tree * nid_stride;
    for (int level = 0; level < depth; ++level) {
        const int nl = 1 << level, off = nl - 1;   // (a row's node: from `off` on when it is still on its way)
        SmallPost *post = posts + (level & 1) * max_nl;
        for (int n0 = 0; n0 < nl; n0 += plan.nodes_pass) {
            const int here = min(plan.nodes_pass, nl - n0);
            // -- histograms of nodes n0 .. n0 + here - 1 over the own features
            for (int i = threadIdx.x; i < here * plan.cells; i += SMALL_THREADS) { acc[i] = 0; acc[words + i] = 0; acc[2 * words + i] = 0; acc[3 * words + i] = 0; }
            __syncthreads();
            if (level == 0)   // (on their way while the rows are added up)
                for (int i = threadIdx.x; i < s_first[nf]; i += SMALL_THREADS)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(s_cut + i)), "l"(cut_val + bin0 + i) : "memory");
            const int first_node = off + n0;
            // rows and features in flight per thread.  (Four rows and two features for one or two features: 5 % longer at 5000 rows, 1 %
            // at 10000; four rows and one for eight features: 4 to 9 % longer)
            auto add = [&](auto rows_c, auto feats_c) {
                constexpr int U = decltype(rows_c)::value, V = decltype(feats_c)::value;
                for (int r0 = threadIdx.x; r0 < N; r0 += U * SMALL_THREADS) {
                    int n[U];
                    int2 v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int r = r0 + u * SMALL_THREADS;
                        n[u] = r < N ? (int)node_of[r] - first_node : -1;
                        if ((unsigned)n[u] >= (unsigned)here) n[u] = -1;
                        v[u] = r < N ? gq[r] : make_int2(0, 0);   // (does not wait for the node)
                    }
                    for (int f = 0; f < nf; f += V) {
                        unsigned char b[U][V];
#pragma unroll
                        for (int k = 0; k < V; ++k)
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                b[u][k] = n[u] >= 0 && f + k < nf ? binsT[(size_t)(f0 + f + k) * Npad + r0 + u * SMALL_THREADS] : (unsigned char)MISSING_BIN;
#pragma unroll
                        for (int k = 0; k < V; ++k)
#pragma unroll
                            for (int u = 0; u < U; ++u) {
                                if (b[u][k] == MISSING_BIN) continue;
                                int *cell = acc + n[u] * plan.cells + small_feature_at(s_first[f + k], f + k) + small_at(b[u][k]);
                                atomicAdd(reinterpret_cast<unsigned *>(cell), (unsigned)v[u].x & 0xffffu);
                                if (v[u].y & 0xffff) atomicAdd(reinterpret_cast<unsigned *>(cell + words), (unsigned)v[u].y & 0xffffu);   // (a hessian of 1 has no low half)
                                atomicAdd(cell + 2 * words, v[u].x >> 16);
                                atomicAdd(cell + 3 * words, v[u].y >> 16);
                            }
                    }
                }
            };
            if (nf > 2) add(std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{});
            else add(std::integral_constant<int, 4>{}, std::integral_constant<int, 1>{});
            __syncthreads();
            if (level == 0) asm volatile("cp.async.wait_all;" ::: "memory");
            if (level == 0) {   // the root's histogram stays readable (tgbm_booster_get_root_hist)
                long long *full = hist_full + tree * full_stride;
                for (int f = warp; f < nf; f += SMALL_THREADS / 32)
                    for (int i = s_first[f] + lane; i < s_first[f + 1]; i += 32) {
                        const int *c = acc + small_feature_at(s_first[f], f) + small_at(i - s_first[f]);
                        full[2 * (size_t)(bin0 + i)] = ((long long)c[2 * words] << 16) + (unsigned)c[0];
                        full[2 * (size_t)(bin0 + i) + 1] = ((long long)c[3 * words] << 16) + (unsigned)c[words];
                    }
            }
            // -- best candidate of every (node, feature): a warp each; eight lanes where no feature has more than eight bins; several
            // warps where there are fewer units than warps (a unit of 255 bins is 15 k cycles for one warp alone; always two bins per lane and
            // four passes per warp were slower, 145 us a tree instead of 121)
            const int units = here * nf;
            const int parts_log = plan.most <= 128 ? 0 : units * 4 <= SMALL_THREADS / 32 ? 2 : units * 2 <= SMALL_THREADS / 32 ? 1 : 0, parts = 1 << parts_log;
            const int lanes_log = plan.most <= 8 ? 3 : 5;   // (shifts: a division by a variable is 200 cycles in every level's chain)
            auto unit = [&](int u, int &n, int &f, const int *&cell, int &nb) {
                n = nf == 1 ? u : u / nf; f = u - n * nf;
                const int first = s_first[f];
                nb = s_first[f + 1] - first;
                cell = acc + n * plan.cells + small_feature_at(first, f);
                return nodes[off + n0 + n].is_valid && nb > 0 && !(ignored && ignored[f0 + f]);
            };
            if (parts > 1) {   // (all units at once)
                const int u = warp >> parts_log, part = warp & (parts - 1);
                int n = 0, f = 0, nb = 0;
                const int *cell = acc;
                const bool active = u < units && unit(u, n, f, cell, nb);
                if (active) {
                    if (parts == 4) small_sums<2>(cell, words, nb, part, s_sums + u * parts);
                    else small_sums<4>(cell, words, nb, part, s_sums + u * parts);
                }
                __syncthreads();
                if (active) {
                    const TreeNode &nd = nodes[off + n0 + n];
                    if (parts == 4) small_eval_call<32, 2>(s_search, cell, nb, nd.sum_g, nd.sum_h, part, parts, s_sums + u * parts, true, s_parts + warp);
                    else small_eval_call<32, 4>(s_search, cell, nb, nd.sum_g, nd.sum_h, part, parts, s_sums + u * parts, true, s_parts + warp);
                } else if (lane == 0) s_parts[warp].bin = -1;
                __syncthreads();
                for (int x = threadIdx.x; x < units; x += SMALL_THREADS) {   // the earlier part among equals
                    SplitRec best = s_parts[x * parts];
                    for (int q = 1; q < parts; ++q) {
                        const SplitRec &r = s_parts[x * parts + q];
                        if (r.bin >= 0 && (best.bin < 0 || fabsf(r.gain) > fabsf(best.gain))) best = r;
                    }
                    recs[x / nf * plan.feats + x % nf] = best;
                }
            } else {
                for (int u0 = 0; u0 < units; u0 += SMALL_THREADS >> lanes_log) {
                    const int u = u0 + ((int)threadIdx.x >> lanes_log);
                    int n = 0, f = 0, nb = 0;
                    const int *cell = acc;
                    const bool active = u < units && unit(u, n, f, cell, nb);
                    const TreeNode &nd = nodes[off + n0 + n];
                    SplitRec *out = recs + n * plan.feats + f;
                    const float pg = nd.sum_g, ph = nd.sum_h;
                    if (lanes_log == 3) {
                        if (u < units && !active && (lane & 7) == 0) out->bin = -1;
                        if (__any_sync(0xffffffffu, active)) small_eval<8, 1>(s_search, cell, nb, pg, ph, 0, 1, nullptr, active, out);
                        continue;
                    }
                    if (!active) { if (u < units && lane == 0) out->bin = -1; continue; }   // (the same in the whole warp)
                    if (nb <= 32) small_eval<32, 1>(s_search, cell, nb, pg, ph, 0, 1, nullptr, true, out);
                    else if (nb <= 128) small_eval<32, 4>(s_search, cell, nb, pg, ph, 0, 1, nullptr, true, out);
                    else small_eval_call<32, 8>(s_search, cell, nb, pg, ph, 0, 1, nullptr, true, out);
                }
            }
            __syncthreads();
            for (int n = threadIdx.x; n < here; n += SMALL_THREADS) {   // ... and of the own features
                SmallPost p;
                p.key = 0;
                for (int f = 0; f < nf; ++f) {
                    const SplitRec r = recs[n * plan.feats + f];
                    if (r.bin < 0) continue;
                    const unsigned long long k = ((unsigned long long)__float_as_uint(fabsf(r.gain)) << 32) | (unsigned)(0x7fffffff - (f0 + f));
                    if (k > p.key) { p.key = k; p.rec = r; p.rec.value = split_at(s_cut + s_first[f], r.bin, multi); p.rec.feature = f0 + f; }
                }
                post[n0 + n] = p;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) s_split = 0;
        cluster.sync();   // every CTA's candidates are in place (and its reads of the level before are done)
        // sixteen lanes per node: each reads one CTA's candidate
        for (int base = (int)(threadIdx.x & ~31u); base < nl * 16; base += SMALL_THREADS) {
            const int n = (base + lane) >> 4, c = lane & 15;
            const bool valid = n < nl && nodes[off + n].is_valid;
            unsigned long long best = valid && c < plan.cluster ? cluster.map_shared_rank(post, c)[n].key : 0;
            int from = c;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                const unsigned long long other = (unsigned long long)shfl_xor_ll((long long)best, o);
                const int f = __shfl_xor_sync(0xffffffffu, from, o);
                if (other > best) { best = other; from = f; }
            }
            if (c == 0 && n < nl) {
                split[n] = 0;
                if (valid) {
                    TreeNode &nd = nodes[off + n];
                    if (best == 0) nd.is_leaf = 1;   // no feature has a cut point: nothing to split on
                    else {
                        const SplitRec r = cluster.map_shared_rank(post, from)[n].rec;
                        apply_split(nodes, off + n, r, nd.sum_g, nd.sum_h, rt_eps, lam, multi);
                    }
                    if (!nd.is_leaf) {
                        s_split = 1;
                        split[n] = 0x80000000u | (nd.default_right ? 0x40000000u : 0u) | ((unsigned)nd.split_feature_id << 8) | nd.split_bid;
                    }
                }
            }
            __syncwarp();
        }
        __syncthreads();
        if (!s_split || level == depth - 1) break;   // the same in every CTA (k_apply_tree makes the last move)
        // -- rows to the children.  Few of them: every CTA for itself, four rows a thread (a share each takes as long for 5000 rows and
        // 1.2 k cycles longer for 200: what it writes has to be seen by the other CTAs)
        if (LOCAL) {
            unsigned at[4], sp[4];
            unsigned char b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = (int)threadIdx.x + u * SMALL_THREADS;
                at[u] = r < N ? (unsigned)node_of[r] : 0u;
                sp[u] = r < N && at[u] >= (unsigned)off ? split[at[u] - off] : 0u;   // 0: not split
                b[u] = sp[u] ? binsT[(size_t)((sp[u] >> 8) & 0x3fffffu) * Npad + r] : (unsigned char)0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!sp[u]) continue;
                const unsigned char bid = (unsigned char)sp[u];
                const bool left = b[u] == MISSING_BIN ? !(sp[u] & 0x40000000u) : (multi ? b[u] > bid : b[u] < bid);
                node_of[threadIdx.x + u * SMALL_THREADS] = (unsigned short)(2 * at[u] + (left ? 1u : 2u));
            }
            __syncthreads();
            continue;
        }
        // More: a share of them per CTA, written to the table that the tree leaves behind and read back whole
        // (every CTA for itself: a warp's 32 rows are in up to 32 nodes, so in as many columns; 10 k cycles a level for 10000 rows)
        for (int r = share0 + (int)threadIdx.x; r < share1; r += SMALL_THREADS) {
            const unsigned at = node_of[r], sp = at >= (unsigned)off ? split[at - off] : 0u;   // 0: not split
            unsigned to = at;
            if (sp) {
                const unsigned char b = binsT[(size_t)((sp >> 8) & 0x3fffffu) * Npad + r], bid = (unsigned char)sp;
                const bool left = b == MISSING_BIN ? !(sp & 0x40000000u) : (multi ? b > bid : b < bid);
                to = 2 * at + (left ? 1u : 2u);
            }
            my_nid[r] = (unsigned short)to;
        }
        cluster.sync();
        for (int i = threadIdx.x; i < (N + 7) / 8; i += SMALL_THREADS)   // (past L1: other SMs wrote it; the table is padded)
            reinterpret_cast<uint4 *>(node_of)[i] = __ldcg(reinterpret_cast<const uint4 *>(my_nid) + i);
        __syncthreads();
        moved = true;
    }
    cluster.sync();   // nobody reads this CTA's candidates any more
    if (!moved)   // moved here, or a tree that is its root
        for (int r = share0 + (int)threadIdx.x; r < share1; r += SMALL_THREADS) my_nid[r] = node_of[r];
    if (rank != 0) return;
    // -- pruning and the finished tree (k_prune)
    if (threadIdx.x == 0) {
        atomicAdd(&ctl->stat_rows_root, (unsigned long long)N);
        atomicAdd(&ctl->stat_hists, 1ull);
    }
    prune_tree(nodes, n_nodes, depth, gamma, scratch);
    leave_rules(nodes, n_nodes, depth, multi, weight + (size_t)tree * n_nodes, rule + tree * rule_stride, nullptr, nullptr, nullptr);
    TreeNode *out = nodes_out + (size_t)tree * n_nodes, *mod = model + ((size_t)rs->round * K + k0 + tree) * n_nodes;
    for (int i = threadIdx.x; i < n_nodes * (int)(sizeof(TreeNode) / 16); i += SMALL_THREADS) {
        const int4 t = reinterpret_cast<const int4 *>(nodes)[i];
        reinterpret_cast<int4 *>(out)[i] = t;
        reinterpret_cast<int4 *>(mod)[i] = t;
    }
}

}  // namespace tgbm
