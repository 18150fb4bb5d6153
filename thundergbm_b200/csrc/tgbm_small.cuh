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
// Bound by the shared-memory atomics of the rows x own features (four 32-bit halves per value, random banks) and by the
// division chains of the split search.  10000 rows x 32 features, depth 6:
// 130 us a tree against 185 us; 1605 rows x 119 features: 85 us against 165 us.
// Same integer sums, gains, tie rules and node records as the level kernels, bit for bit.
#pragma once
#include <cooperative_groups.h>

#include "tgbm_level.cuh"

namespace tgbm {

constexpr int SMALL_THREADS = 1024;

struct SmallPost {   // a CTA's best candidate of a node: |gain| bits << 32 | (0x7fffffff - feature), 0 = none
    unsigned long long key;
    SplitRec rec;
};

struct SmallPlan {   // sizes fixed by the host (see small_plan in the booster)
    int cluster, feats, bins;   // CTAs per tree, features per CTA, most bins of a CTA
    int nodes_pass;             // nodes whose histograms are in shared memory at a time
    size_t smem;
};

// best candidate of one (node, feature): the lanes of a warp own BPL consecutive bins each
template <int BPL>
__device__ __forceinline__ void small_eval(const int *cell, int words, int nb, float pg, float ph, const GridScale &inv_sg, const GridScale &inv_sh, float mcw,
                                           float lam, int multi, SplitRec *out) {
    const int lane = threadIdx.x & 31;
    long long g[BPL], h[BPL], tg = 0, th = 0;
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        const int b = lane * BPL + i;
        g[i] = h[i] = 0;
        if (b < nb) {
            g[i] = ((long long)cell[2 * words + b] << 16) + (unsigned)cell[b];
            h[i] = ((long long)cell[3 * words + b] << 16) + (unsigned)cell[words + b];
        }
        tg += g[i]; th += h[i];
    }
    long long ig = tg, ih = th;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long ug = shfl_up_ll(ig, o), uh = shfl_up_ll(ih, o);
        if (lane >= o) { ig += ug; ih += uh; }
    }
    const long long all_g = shfl_ll(ig, 31), all_h = shfl_ll(ih, 31);
    const float mg = __fsub_rn(pg, inv_sg(all_g)), mh = __fsub_rn(ph, inv_sh(all_h));
    const float parent = __fdiv_rn(__fmul_rn(pg, pg), __fadd_rn(ph, lam));
    long long rg = ig - tg, rh = ih - th;
    unsigned long long key = 0;
    float best = 0.f, keep_g = 0.f, keep_h = 0.f;
#pragma unroll
    for (int i = 0; i < BPL; ++i) {
        const int b = lane * BPL + i;
        if (multi) { rg += g[i]; rh += h[i]; }
        const float kg = inv_sg(rg), kh = inv_sh(rh);   // see k_eval
        if (!multi) { rg += g[i]; rh += h[i]; }
        const float a = split_gain(parent, pg, ph, kg, kh, mcw, lam), z = split_gain(parent, pg, ph, __fadd_rn(kg, mg), __fadd_rn(kh, mh), mcw, lam);
        const float gl = fmaxf(0.f, multi ? a : z), gr = fmaxf(0.f, multi ? z : a);
        const float gn = gl > gr ? gl : -gr;
        const unsigned long long kk = ((unsigned long long)__float_as_uint(fabsf(gn)) << 32) | (unsigned)(0x7fffffff - b);
        if (b < nb && kk > key) { key = kk; best = gn; keep_g = kg; keep_h = kh; }
    }
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    if (key == (((unsigned long long)hi << 32) | lo)) *out = SplitRec{best, 0x7fffffff - (int)lo, keep_g, keep_h, mg, mh};
}

// grid = trees x plan.cluster, clusters of plan.cluster CTAs
static __global__ void __launch_bounds__(SMALL_THREADS, 1)
k_small_tree(const SmallPlan plan, int N, size_t Npad, int F, int depth, const unsigned char *__restrict__ binsT, const int *__restrict__ cut_ptr,
             const float *__restrict__ cut_val, const int2 *ghq, const unsigned long long *root_sum, const QuantInfo *q, float mcw, float lam,
             float rt_eps, float gamma, const unsigned char *__restrict__ ignored_all, const RoundState *rs, int multi, TreeNode *nodes_out,
             TreeNode *model, int K, int k0, unsigned *maxbits, int fine_K, TreeCtl *ctl, long long *hist_full, size_t full_stride,
             unsigned short *nid, size_t nid_stride, float *weight, AssignRule *rule, size_t rule_stride) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char small_sm[];
    __shared__ int scratch[33], s_split;
    const int n_nodes = (1 << (depth + 1)) - 1, max_nl = 1 << (depth - 1);
    TreeNode *nodes = reinterpret_cast<TreeNode *>(small_sm);
    SmallPost *posts = reinterpret_cast<SmallPost *>(small_sm + (sizeof(TreeNode) * n_nodes + 15) / 16 * 16);   // [2][max_nl]
    SplitRec *recs = reinterpret_cast<SplitRec *>(posts + 2 * max_nl);                                       // [nodes_pass][feats]
    unsigned *split = reinterpret_cast<unsigned *>(recs + (plan.nodes_pass * plan.feats + 1) / 2 * 2);   // [max_nl] what the level decided
    unsigned short *node_of = reinterpret_cast<unsigned short *>(split + (max_nl + 3) / 4 * 4);            // [N, eights]
    int *acc = reinterpret_cast<int *>(node_of + (N + 7) / 8 * 8);                                               // [4][nodes_pass * bins]
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), tree = blockIdx.x / plan.cluster, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f0 = min(F, rank * plan.feats), nf = min(F, f0 + plan.feats) - f0, bin0 = cut_ptr[f0], words = plan.nodes_pass * plan.bins;
    const int share = (N + plan.cluster - 1) / plan.cluster, share0 = min(N, rank * share), share1 = min(N, share0 + share);   // rows whose node this CTA reports
    for (int r = threadIdx.x; r < N; r += SMALL_THREADS) node_of[r] = 0;
    chain_wait();
    if (blockIdx.x == 0 && threadIdx.x == SMALL_THREADS - 1) next_maxima(root_sum, fine_K, maxbits, ctl);   // (a thread that has nothing else to do yet)
    const int2 *gq = ghq + (size_t)tree * N;
    const GridScale inv_sg(q->inv_sg), inv_sh(q->inv_sh);
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
    for (int level = 0; level < depth; ++level) {
        const int nl = 1 << level, off = nl - 1;   // (a row's node: from `off` on when it is still on its way)
        SmallPost *post = posts + (level & 1) * max_nl;
        for (int n0 = 0; n0 < nl; n0 += plan.nodes_pass) {
            const int here = min(plan.nodes_pass, nl - n0);
            // -- histograms of nodes n0 .. n0 + here - 1 over the own features
            for (int i = threadIdx.x; i < here * plan.bins; i += SMALL_THREADS) { acc[i] = 0; acc[words + i] = 0; acc[2 * words + i] = 0; acc[3 * words + i] = 0; }
            __syncthreads();
            constexpr int U = 4;   // rows in flight per thread
            for (int r0 = threadIdx.x; r0 < N; r0 += U * SMALL_THREADS) {
                int n[U];
                int2 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = r0 + u * SMALL_THREADS;
                    n[u] = r < N ? (int)node_of[r] - off - n0 : -1;
                    if ((unsigned)n[u] >= (unsigned)here) n[u] = -1;
                    v[u] = r < N ? gq[r] : make_int2(0, 0);   // (does not wait for the node)
                }
                for (int f = 0; f < nf; ++f) {
                    const unsigned char *col = binsT + (size_t)(f0 + f) * Npad;
                    const int first = cut_ptr[f0 + f] - bin0;
                    int b[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) b[u] = r0 + u * SMALL_THREADS < N ? col[r0 + u * SMALL_THREADS] : MISSING_BIN;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (b[u] == MISSING_BIN || n[u] < 0) continue;
                        int *cell = acc + n[u] * plan.bins + first + b[u];
                        atomicAdd(reinterpret_cast<unsigned *>(cell), (unsigned)v[u].x & 0xffffu);
                        if (v[u].y & 0xffff) atomicAdd(reinterpret_cast<unsigned *>(cell + words), (unsigned)v[u].y & 0xffffu);   // (a hessian of 1 has no low half)
                        atomicAdd(cell + 2 * words, v[u].x >> 16);
                        atomicAdd(cell + 3 * words, v[u].y >> 16);
                    }
                }
            }
            __syncthreads();
            if (level == 0) {   // the root's histogram stays readable (tgbm_booster_get_root_hist)
                long long *full = hist_full + tree * full_stride;
                for (int i = threadIdx.x; i < cut_ptr[f0 + nf] - bin0; i += SMALL_THREADS) {
                    full[2 * (size_t)(bin0 + i)] = ((long long)acc[2 * words + i] << 16) + (unsigned)acc[i];
                    full[2 * (size_t)(bin0 + i) + 1] = ((long long)acc[3 * words + i] << 16) + (unsigned)acc[words + i];
                }
            }
            // -- best candidate of every (node, feature): a warp each
            for (int u = warp; u < here * nf; u += SMALL_THREADS / 32) {
                const int n = u / nf, f = u - n * nf;
                const TreeNode &nd = nodes[off + n0 + n];
                SplitRec *out = recs + n * plan.feats + f;
                const int first = cut_ptr[f0 + f], nb = cut_ptr[f0 + f + 1] - first;
                if (!nd.is_valid || nb == 0 || (ignored && ignored[f0 + f])) { if (lane == 0) out->bin = -1; continue; }
                const int *cell = acc + n * plan.bins + first - bin0;
                const float pg = nd.sum_g, ph = nd.sum_h;
                if (nb <= 32) small_eval<1>(cell, words, nb, pg, ph, inv_sg, inv_sh, mcw, lam, multi, out);
                else if (nb <= 128) small_eval<4>(cell, words, nb, pg, ph, inv_sg, inv_sh, mcw, lam, multi, out);
                else small_eval<8>(cell, words, nb, pg, ph, inv_sg, inv_sh, mcw, lam, multi, out);
            }
            __syncthreads();
            for (int n = threadIdx.x; n < here; n += SMALL_THREADS) {   // ... and of the own features
                SmallPost p;
                p.key = 0;
                for (int f = 0; f < nf; ++f) {
                    const SplitRec r = recs[n * plan.feats + f];
                    if (r.bin < 0) continue;
                    const unsigned long long k = ((unsigned long long)__float_as_uint(fabsf(r.gain)) << 32) | (unsigned)(0x7fffffff - (f0 + f));
                    if (k > p.key) { p.key = k; p.rec = r; }
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
                        apply_split(nodes, off + n, 0x7fffffff - (int)(unsigned)(best & 0xffffffffull), r, cut_ptr, cut_val, rt_eps, lam, multi);
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
        // -- rows to the children
        // (every CTA for itself: moving a share each and storing it into all sixteen copies took twice the time)
        constexpr int R = 8;   // rows in flight per thread
        for (int r0 = threadIdx.x; r0 < N; r0 += R * SMALL_THREADS) {
            unsigned at[R], sp[R];
            unsigned char b[R];
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int r = r0 + u * SMALL_THREADS;
                at[u] = r < N ? node_of[r] : 0u;
                sp[u] = r < N && at[u] >= (unsigned)off ? split[at[u] - off] : 0u;   // 0: not split
                b[u] = sp[u] ? binsT[(size_t)((sp[u] >> 8) & 0x3fffffu) * Npad + r] : (unsigned char)0;
            }
#pragma unroll
            for (int u = 0; u < R; ++u) {
                if (!sp[u]) continue;
                const unsigned char bid = (unsigned char)sp[u];
                const bool left = b[u] == MISSING_BIN ? !(sp[u] & 0x40000000u) : (multi ? b[u] > bid : b[u] < bid);
                node_of[r0 + u * SMALL_THREADS] = (unsigned short)(2 * at[u] + (left ? 1u : 2u));
            }
        }
        __syncthreads();
    }
    for (int r = share0 + (int)threadIdx.x; r < share1; r += SMALL_THREADS) nid[(size_t)tree * nid_stride + r] = node_of[r];
    cluster.sync();   // nobody reads this CTA's candidates any more
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
