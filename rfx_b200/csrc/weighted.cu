// Case-wise weighting and RF-GAP proximity.
//
// Case-wise (use_casewise, the reference's bootstrap-frequency weighting):
//   tnodewt   per terminal node, the mean bootstrap multiplicity of the
//             in-bag samples that reach it, walked with the rule of
//             grow_tree_single's tnodewt block (src/rf_random_forest.cpp:
//             1049-1102); float(sum) / float(count), 0 for other nodes.
//   votes     q[i][jtr] += tnodewt[nodextr] per OOB tree, in tree order
//             (:1107-1153) — one thread per sample, trees in order.
//   pair sums C[i][j] += nin[j] / nodesize for OOB i and in-bag j of a leaf,
//             nodesize = the leaf's in-bag multiplicities summed, FP64
//             (src/rf_proximity.cpp:195-222); S = C + C^T is written as the
//             packed upper triangle.
//   importance (src/rf_varimp.cpp:138-148, 203-236): right, rightimp, qimp
//             and qimpm weighted by tnodewt of the node the (permuted) walk
//             reaches.
// RF-GAP (src/rf_proximity.cpp:238-391): pGAP(i,j) = (1/|S_i|) sum over the
//   trees where i is OOB of c_j / |M_i| for the in-bag samples j of i's node,
//   then P = (pGAP + pGAP^T) / 2; nodes are the per-tree node ids the
//   reference keeps (OOB: testreebag, in-bag: find_terminal_node), so any node
//   id matches, the root included.
//
// Every float and double sum runs in the reference's order, so the results
// are bit-identical to it: one warp owns a row's window and adds tree after
// tree (within one tree a row meets each column at most once, so its lanes
// never share a slot), votes and qimp/qimpm loop over trees in order per
// sample, rightimp loops over a tree's OOB samples in order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <string>

#include "walks.cuh"

namespace rfx {
namespace {

// Weighted pair-sum rows: columns of a window (two FP64 sums each; 1,024 = 16
// KB, 13 warps an SM: 1.32 ms at n = 5,000 / 500 trees, 512 took 1.66 and
// 2,048 1.59) and ranges whose loads are in flight together.
constexpr int WR_WINDOW = 1024;
constexpr int WR_BATCH = 4;

// tnodewt: one thread per (sample, tree) of the in-bag samples; integer sums
// (exact, so the order of the float sums of the reference does not matter).
__global__ void tnodewt_walk_kernel(const float* __restrict__ X, int n, int p, const DNode* __restrict__ nodes,
                                    const int64_t* __restrict__ offs, const int32_t* __restrict__ nnode,
                                    const int32_t* __restrict__ catgoleft, int maxcat, const int32_t* __restrict__ nin,
                                    int32_t* __restrict__ wsum, int32_t* __restrict__ wcnt) {
    const int t = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = nin[(size_t)t * n + i];
    if (c <= 0) return;
    const int64_t o = offs[t];
    const int nn = nnode[t];
    const DNode* tn = nodes + o;
    const int32_t* cgl = catgoleft ? catgoleft + o * maxcat : nullptr;
    const float* xr = X + (size_t)i * p;
    int cur = 0;
    for (int guard = 0; guard < nn + 1; ++guard) {  // a grown tree reaches a leaf within nnode steps
        const DNode nd = load_node(tn, cur);
        if (node_status(nd.meta) != 1) break;
        const int m = node_var(nd.meta);
        const float x = __ldg(xr + m);
        bool left;
        if (node_cat(nd.meta)) {
            const int idx = __float2int_rz(__fadd_rn(x, 0.5f));
            left = idx >= 0 && idx < maxcat && cgl_at(cgl, maxcat, cur, idx) == 1;
        } else {
            left = x <= nd.split;
        }
        cur = left ? nd.left : nd.right;
        if (cur < 0 || cur >= nn) break;
    }
    if (cur >= 0 && cur < nn && node_status(load_node(tn, cur).meta) == -1) {
        atomicAdd(wsum + o + cur, c);
        atomicAdd(wcnt + o + cur, 1);
    }
}

__global__ void tnodewt_final_kernel(int64_t N, const int32_t* __restrict__ wsum, const int32_t* __restrict__ wcnt,
                                     float* __restrict__ tnodewt) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= N) return;
    const int k = wcnt[g];
    tnodewt[g] = k > 0 ? __fdiv_rn((float)wsum[g], (float)k) : 0.0f;
}

// weight of an OOB vote that ends on node nd of a tree with nn nodes
__device__ __forceinline__ float vote_w(const float* __restrict__ tw, int nd, int nn) {
    return (nd >= 0 && nd < nn) ? __ldg(tw + nd) : 1.0f;
}

// Case-wise OOB votes: q[i][class] += weight over the OOB trees in order; the
// class of an OOB walk is the class of the node testreebag ends on (the root
// on its fallback path, whose node id is 0).  The chain of loads per (tree,
// sample) (bag flag, node, class and weight) does not depend on the order of
// the sums, so a CTA of 32 samples fetches CV_TREES trees at once into shared
// memory; then thread (sample, g) adds the classes = g (mod 8) tree after tree.
// n = 3,001 / 300 trees: 52 us (220 us with one thread per sample and the
// loads in its chain).
constexpr int CV_TREES = 64;
__global__ void __launch_bounds__(256)
casewise_votes_kernel(const int32_t* __restrict__ leafnode, const uint8_t* __restrict__ inbag,
                      const int64_t* __restrict__ offs, const int32_t* __restrict__ nnode,
                      const int32_t* __restrict__ nodeclass, const float* __restrict__ tnodewt, int n, int T,
                      int nclass, float* __restrict__ q) {
    extern __shared__ float qs[];  // 32 * nclass
    __shared__ float s_w[CV_TREES][32];
    __shared__ int8_t s_c[CV_TREES][32];  // class, -1 for none
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float* my = qs + (size_t)lane * nclass;  // this sample's sums; thread w owns the classes = w (mod 8)
    for (int c = w; c < nclass; c += 8) my[c] = 0.0f;
    for (int tb = 0; tb < T; tb += CV_TREES) {
        constexpr int PER = CV_TREES / 8;
        int nd[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int t = tb + u * 8 + w;
            const size_t ti = (size_t)t * n + i;
            nd[u] = t < T && i < n && !__ldg(inbag + ti) ? __ldg(leafnode + ti) : -1;
        }
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int t = tb + u * 8 + w;
            int cls = -1;
            float wt = 0.0f;
            if (nd[u] >= 0) {
                const int64_t o = offs[t];
                cls = __ldg(nodeclass + o + nd[u]);
                wt = vote_w(tnodewt + o, nd[u], nnode[t]);
                if (cls >= nclass) cls = -1;
            }
            s_c[u * 8 + w][lane] = (int8_t)max(cls, -1);
            s_w[u * 8 + w][lane] = wt;
        }
        __syncthreads();
        const int nt = min(CV_TREES, T - tb);
#pragma unroll 8
        for (int u = 0; u < nt; ++u) {
            const int cls = s_c[u][lane];
            if (cls >= 0 && (cls & 7) == w) my[cls] = __fadd_rn(my[cls], s_w[u][lane]);
        }
        __syncthreads();
    }
    if (i < n)
        for (int c = w; c < nclass; c += 8) q[(size_t)i * nclass + c] = my[c];
}

// Sum of the bootstrap multiplicities of every key's members (per tree, per
// key of the leaf lists).
__global__ void key_mass_kernel(const int64_t* __restrict__ segbase, const int32_t* __restrict__ segoff,
                                const int32_t* __restrict__ memb, const int32_t* __restrict__ nin, int n,
                                long long* __restrict__ mass) {
    const int t = blockIdx.x;
    const int64_t sb = segbase[t];
    const int K = (int)(segbase[t + 1] - sb) - 1;
    const int32_t* so = segoff + sb;
    const int32_t* mt = memb + (size_t)t * n;
    const int32_t* nt = nin + (size_t)t * n;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        long long s = 0;
        for (int q = so[k]; q < so[k + 1]; ++q) s += nt[mt[q]];
        mass[sb + k] = s;
    }
}

enum { WR_CASEWISE = 0, WR_RFGAP = 1, WR_PLAIN = 2 };

// One row's part of one tree: the members of the opposite bag status in the
// row's leaf with ids above the row's (start within the tree's member list,
// count; the top bit of `len` marks an in-bag row), and the row's factor:
//   out-of-bag row: the in-bag key's mass m (case-wise) or 1 / m (RF-GAP);
//   in-bag row: the finished weight of the row in its leaf.
struct __align__(16) WRange {
    int lo;
    unsigned len;
    double w;
};
constexpr unsigned WR_INBAG = 0x80000000u;

// Range table of the rows [i0, i1), row-major (T entries a row), so that the
// row kernel reads its trees' entries coalesced and does no search, mass
// lookup or division per tree.  32 rows x 32 trees per CTA, transposed
// through shared memory.
template <int MODE>
__global__ void __launch_bounds__(256)
weighted_ranges_kernel(const int32_t* __restrict__ key, const int64_t* __restrict__ segbase,
                       const int32_t* __restrict__ segoff, const int32_t* __restrict__ memb,
                       const long long* __restrict__ mass, const int32_t* __restrict__ nin, int n, int T, int i0,
                       int i1, WRange* __restrict__ tab) {
    __shared__ WRange tile[32][33];
    const int ib = i0 + blockIdx.x * 32, tb = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int t = tb + r, i = ib + tx;
        WRange v{0, 0u, 0.0};
        const int k = t < T && i < i1 ? __ldg(key + (size_t)t * n + i) : -1;
        if (k >= 0) {
            const int64_t sb = segbase[t];
            const int32_t* so = segoff + sb;
            const int32_t* mt = memb + (size_t)t * n;
            int lo = __ldg(so + (k ^ 1)), hi = __ldg(so + (k ^ 1) + 1);
            const int end = hi;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__ldg(mt + mid) <= i) lo = mid + 1;
                else hi = mid;
            }
            const long long m = end > lo ? mass[sb + (k | 1)] : 0;  // the in-bag key of the leaf
            if (end > lo && (m > 0 || MODE == WR_PLAIN)) {
                v.lo = lo;
                v.len = (unsigned)(end - lo);
                if ((k & 1) == 0) {
                    v.w = MODE == WR_PLAIN ? 1.0 : MODE == WR_RFGAP ? __ddiv_rn(1.0, (double)m) : (double)m;
                } else {
                    const double c = (double)__ldg(nin + (size_t)t * n + i);
                    v.len |= WR_INBAG;
                    v.w = MODE == WR_PLAIN   ? 1.0
                          : MODE == WR_RFGAP ? __dmul_rn(c, __ddiv_rn(1.0, (double)m))
                                             : __ddiv_rn(c, (double)m);
                }
            }
        }
        tile[r][tx] = v;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int i = ib + r, t = tb + tx;
        if (i < i1 && t < T) tab[(size_t)(i - i0) * T + t] = tile[tx][r];
    }
}

// Weight of every in-bag member in member-list order (case-wise nin / mass,
// RF-GAP nin x (1 / mass)), so that the row kernel reads it beside the member
// instead of dividing per pair.
template <int MODE>
__global__ void member_weight_kernel(const int32_t* __restrict__ key, const int64_t* __restrict__ segbase,
                                     const int32_t* __restrict__ segoff, const int32_t* __restrict__ memb,
                                     const long long* __restrict__ mass, const int32_t* __restrict__ nin, int n,
                                     double* __restrict__ wm) {
    const int t = blockIdx.y;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t sb = segbase[t];
    if (q >= __ldg(segoff + segbase[t + 1] - 1)) return;  // members without a key follow the keyed ones
    const size_t tn = (size_t)t * n;
    const int j = __ldg(memb + tn + q);
    const int k = __ldg(key + tn + j);
    if (!(k & 1)) return;
    const double c = (double)__ldg(nin + tn + j), m = (double)mass[sb + k];
    wm[tn + q] = MODE == WR_RFGAP ? __dmul_rn(c, __ddiv_rn(1.0, m)) : __ddiv_rn(c, m);
}

// One warp per row i.
//   i out of bag: accA[j] += w(j) for the in-bag members j
//   i in-bag:     accB[j] += w(i) for the out-of-bag members j
// casewise: w(s) = nin[s] / nodesize (nodesize = mass of the in-bag key);
//           S[i][j] = accA[j] + accB[j].
// plain:    w = 1 (the reference's weights without use_casewise), as FP64.
// rfgap:    w(s) = nin[s] * (1 / M), M = mass of the in-bag key;
//           P[i][j] = (accA[j] / |S_i| + accB[j] / |S_j|) / 2, with the
//           reference's multiplication by 1 / |S|.
// Every sum runs in the warp's program order, tree after tree, with no barrier.
// The row is taken in windows of `win` columns whose sums sit in shared
// memory; the row's ranges keep their position in the table between windows
// (members ascend), so nothing is searched.  The warp takes 32 trees at a time
// (lane = tree) and adds the ranges that reach into the window one after the
// other, lanes on consecutive members: the columns of one range are distinct,
// so no lane meets another.  The loads of the next WR_BATCH ranges are in
// flight with the adds of the current ones.
// PRE: the in-bag members' weights come from member_weight_kernel (without
// room for them they are formed here).
// n = 5,000 / 500 trees / 1.1e8 weighted updates: 1.32 ms (20.0 ms with one CTA
// per row and window, a barrier and a chain of dependent loads per tree;
// 1.6 ms with elements of several ranges taken together and conflicts resolved
// by match.any, which serialises distinct values; 2.9 ms with elements staged
// for the four warps of a CTA).
template <int MODE, bool PRE>
__global__ void __launch_bounds__(32)
weighted_row_kernel(WRange* __restrict__ tab, int i0, const int32_t* __restrict__ memb,
                    const double* __restrict__ wm, const int32_t* __restrict__ nin, const int32_t* __restrict__ nout,
                    int n, int T, int win, double* __restrict__ out) {
    extern __shared__ double2 wr_acc[];  // per column: x = accA, y = accB
    const int i = i0 + blockIdx.x;
    const int lane = threadIdx.x;
    double* acc = reinterpret_cast<double*>(wr_acc);
    int4* row = reinterpret_cast<int4*>(tab + (size_t)blockIdx.x * T);
    const int64_t rowoff = (int64_t)i * n - ((int64_t)i * (i - 1)) / 2 - i;  // + j gives [i][j]
    const int sI = nout[i] / 2;  // trees where i is OOB
    const double invI = sI > 0 ? __ddiv_rn(1.0, (double)sI) : 0.0;
    for (int c0 = i; c0 < n; c0 += win) {
        const int c1 = min(n, c0 + win);
        const bool last = c1 == n;
        for (int k = lane; k < c1 - c0; k += 32) wr_acc[k] = make_double2(0.0, 0.0);
        __syncwarp();
        int4 nxt = lane < T ? row[lane] : make_int4(0, 0, 0, 0);
        for (int tb = 0; tb < T; tb += 32) {
            const int t = tb + lane;
            const int4 raw = nxt;
            if (tb + 32 < T) nxt = t + 32 < T ? row[t + 32] : make_int4(0, 0, 0, 0);
            int lo = raw.x, len = raw.y & 0x7fffffff;
            const int side = (unsigned)raw.y >> 31;
            const int j0 = len > 0 ? __ldg(memb + (size_t)t * n + lo) : n;
            unsigned todo = __ballot_sync(0xffffffffu, j0 < c1);
            if (!todo) continue;
            struct Batch {
                int c[WR_BATCH], cnt[WR_BATCH], j[WR_BATCH];
                double v[WR_BATCH];
            };
            auto fetch = [&](int c, int at, int sd, double wc, int& j, double& v) {
                const size_t q = (size_t)(tb + c) * n + at;
                j = __ldg(memb + q);
                v = wc;
                if (MODE != WR_PLAIN && !sd) {
                    if (PRE) {
                        v = __ldg(wm + q);
                    } else {
                        const double cj = (double)__ldg(nin + (size_t)(tb + c) * n + j);
                        v = MODE == WR_RFGAP ? __dmul_rn(cj, wc) : __ddiv_rn(cj, wc);
                    }
                }
            };
            auto take = [&](Batch& b) {
#pragma unroll
                for (int u = 0; u < WR_BATCH; ++u) {
                    const int c = todo ? __ffs(todo) - 1 : 0;
                    b.c[u] = c;
                    b.cnt[u] = todo ? __shfl_sync(0xffffffffu, len, c) : 0;
                    const int at = __shfl_sync(0xffffffffu, lo, c), sd = __shfl_sync(0xffffffffu, side, c);
                    const double wc = __hiloint2double(__shfl_sync(0xffffffffu, raw.w, c),
                                                       __shfl_sync(0xffffffffu, raw.z, c));
                    todo &= todo - 1;
                    b.j[u] = n;
                    b.v[u] = 0.0;
                    if (lane < b.cnt[u]) fetch(c, at + lane, sd, wc, b.j[u], b.v[u]);
                }
            };
            Batch cur;
            take(cur);
            while (cur.cnt[0] > 0) {
                Batch ahead;
                take(ahead);
#pragma unroll
                for (int u = 0; u < WR_BATCH; ++u) {
                    if (cur.cnt[u] == 0) break;
                    const int c = cur.c[u];
                    const int sd = __shfl_sync(0xffffffffu, side, c);
                    const bool in = cur.j[u] < c1;
                    double* a = acc + sd - 2 * c0;
                    if (in) a[2 * cur.j[u]] = __dadd_rn(a[2 * cur.j[u]], cur.v[u]);
                    int used = __popc(__ballot_sync(0xffffffffu, in));
                    if (used == 32 && cur.cnt[u] > 32) {  // the rest of a long range
                        const int at = __shfl_sync(0xffffffffu, lo, c);
                        const double wc = __hiloint2double(__shfl_sync(0xffffffffu, raw.w, c),
                                                           __shfl_sync(0xffffffffu, raw.z, c));
                        for (int off = 32;; off += 64) {
                            int j1 = n, j2 = n;
                            double v1 = 0.0, v2 = 0.0;
                            if (off + lane < cur.cnt[u]) fetch(c, at + off + lane, sd, wc, j1, v1);
                            if (off + 32 + lane < cur.cnt[u]) fetch(c, at + off + 32 + lane, sd, wc, j2, v2);
                            if (j1 < c1) a[2 * j1] = __dadd_rn(a[2 * j1], v1);
                            if (j2 < c1) a[2 * j2] = __dadd_rn(a[2 * j2], v2);
                            const int got = __popc(__ballot_sync(0xffffffffu, j1 < c1)) +
                                            __popc(__ballot_sync(0xffffffffu, j2 < c1));
                            used += got;
                            if (got < 64) break;
                        }
                    }
                    if (lane == c) {
                        lo += used;
                        len -= used;
                    }
                    __syncwarp();  // this tree's adds come before the next one's
                }
                cur = ahead;
            }
            // the ranges go on from here in the next window
            if (!last && t < T && lo != raw.x)
                *reinterpret_cast<int2*>(row + t) = make_int2(lo, len | (raw.y & (int)WR_INBAG));
        }
        for (int j = c0 + lane; j < c1; j += 32) {
            double v;
            if (j == i) {
                v = MODE == WR_RFGAP ? (sI == 0 ? 1.0 : 0.0) : 0.0;
            } else {
                const double2 ab = wr_acc[j - c0];
                if (MODE == WR_RFGAP) {
                    const int sJ = nout[j] / 2;
                    const double a = sI > 0 ? __dmul_rn(ab.x, invI) : ab.x;
                    const double bj = sJ > 0 ? __dmul_rn(ab.y, __ddiv_rn(1.0, (double)sJ)) : ab.y;
                    v = __ddiv_rn(__dadd_rn(a, bj), 2.0);
                } else {
                    v = __dadd_rn(ab.x, ab.y);
                }
            }
            out[rowoff + j] = v;
        }
        __syncwarp();  // the sums are cleared for the next window
    }
}

// RF-GAP keys: 2 * node + in-bag from the per-tree node ids.
__global__ void gap_key_kernel(const int32_t* __restrict__ leafnode, const uint8_t* __restrict__ inbag, int64_t cells,
                               int32_t* __restrict__ key) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= cells) return;
    const int nd = leafnode[e];
    key[e] = nd >= 0 ? 2 * nd + (inbag[e] ? 1 : 0) : -1;
}

// ---------------------------------------------------------------------------
// Case-wise importance
// ---------------------------------------------------------------------------

// One decision of the cpu_testreeimp walk (src/rf_varimp.cpp:45-103) at node
// nd (id kt) for value x: the child, or -2 where the reference breaks.
__device__ __forceinline__ int cw_decide(const DNode& nd, int kt, float x, const int32_t* __restrict__ cgl,
                                         int maxcat) {
    if (!node_cat(nd.meta)) return (x <= nd.split) ? nd.left : nd.right;
    const int jcat = __float2int_rz(__fadd_rn(x, 0.5f));
    if (jcat < 0 || jcat >= maxcat) return -2;
    return (cgl_at(cgl, maxcat, kt, jcat) == 1) ? nd.left : nd.right;
}

// The permuted walk from node kt on, feature mr taken from xp: the terminal
// node, or -1 when the reference breaks without assigning.  Both children of a
// node are loaded with the feature value (bounds checked at load).
__device__ __forceinline__ int cw_side_walk(const float* __restrict__ xr, const float* __restrict__ xp, int mr, int p,
                                            int kt, int budget, const DNode* __restrict__ tn,
                                            const int32_t* __restrict__ cgl, int maxcat) {
    if (budget <= 0) return -1;
    DNode nd = load_node_now(tn, kt);
    for (int s = 0; s < budget; ++s) {
        if (node_status(nd.meta) == -1) return kt;
        const int m = node_var(nd.meta);
        if (m >= p) return -1;
        const DNode cl = load_node_now(tn, nd.left);
        const DNode cr = load_node_now(tn, nd.right);
        const int nx = cw_decide(nd, kt, __ldg((m == mr ? xp : xr) + m), cgl, maxcat);
        if (nx < 0) return -1;
        nd = nx == nd.left ? cl : cr;
        kt = nx;
    }
    return -1;
}

// One thread per (tree, OOB position) of the trees [t0, t0 + gridDim.y): what
// every feature adds for this sample.  A permuted walk leaves the unpermuted
// path only at a node that splits on its feature, so one walk decides all
// features of a block of 64 W (a side walk for each that diverges) instead of
// one walk per feature:
//   base[t][i]   = weight of the testreebag node if its class is right, else 0;
//   val[t][i][k] = the same for the node that the walk with feature k permuted
//                  ends on (a feature the tree does not split on: base).
// A wrong vote's 0 leaves the ordered sums below unchanged (weights are >= 0).
// Side walks are queued and shared out over the CTA.  n = 3,001 / 300 trees /
// p = 20: 0.27 ms for the walks and both sums (4.6 ms with one walk per feature,
// a tree's samples and a sample's trees one after the other in one thread).
constexpr int CW_THREADS = 128;
constexpr int CW_QCAP = CW_THREADS * 6;
template <int W>
__global__ void __launch_bounds__(CW_THREADS)
cw_walk_kernel(const float* __restrict__ X, const int32_t* __restrict__ y, int n, int p, int t0,
               const DNode* __restrict__ nodes, const int32_t* __restrict__ nodeclass,
               const int64_t* __restrict__ offs, const int32_t* __restrict__ nnode,
               const int32_t* __restrict__ catgoleft, int maxcat, const uint64_t* __restrict__ iv, int ivw,
               const int32_t* __restrict__ joob, const int32_t* __restrict__ noob_arr,
               const int32_t* __restrict__ partner, const int32_t* __restrict__ leafnode,
               const float* __restrict__ tnodewt, float* __restrict__ base, float* __restrict__ val,
               uint32_t* __restrict__ err) {
    __shared__ int4 q_ent[CW_QCAP];  // {thread, feature, start node, step budget}
    __shared__ int q_n;
    __shared__ int s_i[CW_THREADS], s_ip[CW_THREADS], s_y[CW_THREADS];
    const int t = t0 + blockIdx.y;
    const int noob = noob_arr[t];
    const int r = blockIdx.x * CW_THREADS + threadIdx.x;
    if (blockIdx.x * CW_THREADS >= noob) return;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool active = r < noob;
    const int64_t o = offs[t];
    const int nn = nnode[t];
    const int nnv = nn > 0 ? nn : 1;
    const DNode* tn = nodes + o;
    const int32_t* tc = nodeclass + o;
    const float* tw = tnodewt + o;
    const int32_t* cgl = catgoleft ? catgoleft + o * maxcat : nullptr;
    const size_t trow = (size_t)blockIdx.y * n;
    uint32_t my_err = 0;
    int i = 0, ip = 0, yi = -1;
    float w_tb = 0.0f;
    if (active) {
        i = __ldg(joob + (size_t)t * n + r);
        ip = __ldg(partner + (size_t)t * n + i);
        yi = __ldg(y + i);
        const int nd = __ldg(leafnode + (size_t)t * n + i);
        if (__ldg(tc + nd) == yi) w_tb = vote_w(tw, nd, nn);
        base[trow + i] = w_tb;
        s_i[tid] = i;
        s_ip[tid] = ip;
        s_y[tid] = yi;
    }
    for (int fb = 0; fb < p; fb += 64 * W) {
        if (tid == 0) q_n = 0;
        __syncthreads();
        const int pw = min(64 * W, p - fb);
        uint64_t done[W];
#pragma unroll
        for (int q = 0; q < W; ++q) done[q] = 0ull;
        float w_imp = 0.0f;
        bool ok = false;
        if (active) {
            const float* xi = X + (size_t)i * p;
            const float* xp = X + (size_t)ip * p;
            int kt = 0;
            DNode nd = load_node_now(tn, 0);
            for (int step = 0; step < nnv; ++step) {
                if (node_status(nd.meta) == -1) {
                    ok = true;
                    break;
                }
                const int m = node_var(nd.meta);
                if (m >= p) break;
                const DNode cl = load_node_now(tn, nd.left);
                const DNode cr = load_node_now(tn, nd.right);
                const int dir = cw_decide(nd, kt, __ldg(xi + m), cgl, maxcat);
                const int mm = m - fb;
                if ((unsigned)mm < (unsigned)pw) {
                    const uint64_t bit = 1ull << (mm & 63);
                    uint64_t dw = 0;
#pragma unroll
                    for (int q = 0; q < W; ++q)
                        if (q == (mm >> 6)) dw = done[q];
                    if (!(dw & bit)) {
                        const int dp = cw_decide(nd, kt, __ldg(xp + m), cgl, maxcat);
                        if (dp != dir) {
#pragma unroll
                            for (int q = 0; q < W; ++q)
                                if (q == (mm >> 6)) done[q] |= bit;
                            const int slot = dp >= 0 ? atomicAdd(&q_n, 1) : 0;
                            if (dp >= 0 && slot < CW_QCAP) {
                                q_ent[slot] = make_int4(tid, m, dp, nnv - step - 1);
                            } else {
                                const int pn = dp < 0 ? -1 : cw_side_walk(xi, xp, m, p, dp, nnv - step - 1, tn, cgl, maxcat);
                                if (pn < 0) my_err |= ERR_STALE_JVR;
                                val[(trow + i) * p + m] = pn >= 0 && __ldg(tc + pn) == yi ? vote_w(tw, pn, nn) : 0.0f;
                            }
                        }
                    }
                }
                if (dir < 0) break;
                nd = dir == nd.left ? cl : cr;
                kt = dir;
            }
            if (ok && __ldg(tc + kt) == yi) w_imp = vote_w(tw, kt, nn);
            if (!ok) {
                // features that did not diverge break with the unpermuted walk
#pragma unroll
                for (int q = 0; q < W; ++q)
                    if (fb + 64 * q < p && (__ldg(iv + (size_t)t * ivw + (fb >> 6) + q) & ~done[q])) my_err |= ERR_STALE_JVR;
            }
        }
        __syncthreads();
        const int qn = min(q_n, CW_QCAP);
        for (int e = tid; e < qn; e += CW_THREADS) {
            const int4 en = q_ent[e];
            const int si = s_i[en.x];
            const int pn = cw_side_walk(X + (size_t)si * p, X + (size_t)s_ip[en.x] * p, en.y, p, en.z, en.w, tn, cgl,
                                        maxcat);
            if (pn < 0) my_err |= ERR_STALE_JVR;
            val[(trow + si) * p + en.y] = pn >= 0 && __ldg(tc + pn) == s_y[en.x] ? vote_w(tw, pn, nn) : 0.0f;
        }
        // the other features of the warp's rows, one row at a time across the lanes
        const unsigned rows = __ballot_sync(0xffffffffu, active);
        for (int l = 0; l < 32; ++l) {
            if (!((rows >> l) & 1u)) break;  // active lanes come first
            const int ri = __shfl_sync(0xffffffffu, i, l);
            const float ri_imp = __shfl_sync(0xffffffffu, w_imp, l), ri_tb = __shfl_sync(0xffffffffu, w_tb, l);
#pragma unroll
            for (int q = 0; q < W; ++q) {
                const uint64_t dw = __shfl_sync(0xffffffffu, done[q], l);
                if (64 * q >= pw) continue;
                const uint64_t used = __ldg(iv + (size_t)t * ivw + (fb >> 6) + q);
                for (int k = lane; k < 64 && 64 * q + k < pw; k += 32)
                    if (!((dw >> k) & 1ull))
                        val[(trow + ri) * p + fb + 64 * q + k] = (used >> k) & 1ull ? ri_imp : ri_tb;
            }
        }
        __syncthreads();  // the queue is filled again
    }
    if (my_err) atomicOr(err, my_err);
}

// rr[t][k] = (right - rightimp) / noob for the trees [t0, t0 + gridDim.y): the
// ordered sums over the tree's OOB samples of base and of val (0 for a feature
// the tree does not use); one thread per (tree, feature), sixteen samples'
// loads in flight.
__global__ void cw_tree_kernel(int n, int p, int t0, const uint64_t* __restrict__ iv, int ivw,
                               const int32_t* __restrict__ joob, const int32_t* __restrict__ noob_arr,
                               const float* __restrict__ base, const float* __restrict__ val,
                               float* __restrict__ rr) {
    const int t = t0 + blockIdx.y;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p) return;
    const bool used = (__ldg(iv + (size_t)t * ivw + (k >> 6)) >> (k & 63)) & 1ull;
    float out = 0.0f;
    if (used) {
        const int noob = noob_arr[t];
        const int32_t* jo = joob + (size_t)t * n;
        const float* bt = base + (size_t)blockIdx.y * n;
        const float* vt = val + (size_t)blockIdx.y * n * p + k;
        float right = 0.0f, rightimp = 0.0f;
        constexpr int RB = 16;
        int r = 0;
        int nx[RB];  // the next block's samples, loaded with the current block's values
#pragma unroll
        for (int u = 0; u < RB; ++u) nx[u] = u < noob ? __ldg(jo + u) : 0;
        for (; r + RB <= noob; r += RB) {
            float b[RB], v[RB];
#pragma unroll
            for (int u = 0; u < RB; ++u) {
                b[u] = __ldg(bt + nx[u]);
                v[u] = __ldg(vt + (size_t)nx[u] * p);
            }
#pragma unroll
            for (int u = 0; u < RB; ++u) nx[u] = r + RB + u < noob ? __ldg(jo + r + RB + u) : 0;
#pragma unroll
            for (int u = 0; u < RB; ++u) {
                right = __fadd_rn(right, b[u]);
                rightimp = __fadd_rn(rightimp, v[u]);
            }
        }
        for (; r < noob; ++r) {
            const int i = __ldg(jo + r);
            right = __fadd_rn(right, __ldg(bt + i));
            rightimp = __fadd_rn(rightimp, __ldg(vt + (size_t)i * p));
        }
        out = __fdiv_rn(__fsub_rn(right, rightimp), (float)noob);
    }
    rr[(size_t)t * p + k] = out;
}

// One thread per (sample, feature): qimpm[i][k] += val / noob over the trees
// [t0, t1) where i is OOB, in tree order; feature 0's thread also sums qimp[i]
// from base.  The sums of one chunk of trees go on in the next.
__global__ void cw_sample_kernel(int n, int p, int t0, int t1, const uint8_t* __restrict__ inbag,
                                 const int32_t* __restrict__ noob_arr, const float* __restrict__ base,
                                 const float* __restrict__ val, int impn, float* __restrict__ qimp,
                                 float* __restrict__ qimpm) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int cols = impn ? p : 1;
    if (idx >= (int64_t)n * cols) return;
    const int i = (int)(idx / cols), k = (int)(idx % cols);
    float acc = impn && t0 > 0 ? qimpm[(size_t)i * p + k] : 0.0f;
    float accq = k == 0 && t0 > 0 ? qimp[i] : 0.0f;
    constexpr int TB = 8;
    for (int tb = t0; tb < t1; tb += TB) {
        bool oob[TB];
        float v[TB], b[TB], fn[TB];
#pragma unroll
        for (int u = 0; u < TB; ++u) {
            const int t = tb + u;
            oob[u] = t < t1 && __ldg(inbag + (size_t)t * n + i) == 0;
        }
#pragma unroll
        for (int u = 0; u < TB; ++u) {
            const size_t ti = (size_t)(tb + u - t0) * n + i;
            v[u] = oob[u] && impn ? __ldg(val + ti * p + k) : 0.0f;
            b[u] = oob[u] && k == 0 ? __ldg(base + ti) : 0.0f;
            fn[u] = oob[u] ? (float)__ldg(noob_arr + tb + u) : 1.0f;
        }
#pragma unroll
        for (int u = 0; u < TB; ++u) {
            if (!oob[u]) continue;
            acc = __fadd_rn(acc, __fdiv_rn(v[u], fn[u]));
            if (k == 0) accq = __fadd_rn(accq, __fdiv_rn(b[u], fn[u]));
        }
    }
    if (impn) qimpm[(size_t)i * p + k] = acc;
    if (k == 0) qimp[i] = accq;
}

// avimp[k] and sqsd[k]: sums over the trees in order of rr and rr * rr.
__global__ void cw_feature_kernel(const float* __restrict__ rr, int p, int T, float* __restrict__ avimp,
                                  float* __restrict__ sqsd) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p) return;
    float a = 0.0f, s = 0.0f;
#pragma unroll 16
    for (int t = 0; t < T; ++t) {
        const float r = __ldg(rr + (size_t)t * p + k);
        a = __fadd_rn(a, r);
        s = __fadd_rn(s, __fmul_rn(r, r));
    }
    avimp[k] = a;
    sqsd[k] = s;
}

inline unsigned nblk(int64_t count, int b = 256) { return (unsigned)((count + b - 1) / b); }

}  // namespace

// Per-node tnodewt of the loaded forest into c->d_tnodewt (allocated here).
rfx_status launch_tnodewt(Ctx* c) {
    rfx_status st = dalloc(c, &c->d_tnodewt, (size_t)c->N);
    if (st) return st;
    Scratch sc(c);
    int32_t* wsum = sc.get<int32_t>((size_t)c->N);
    int32_t* wcnt = sc.get<int32_t>((size_t)c->N);
    if (!wsum || !wcnt) {
        set_error("case-wise weights: scratch allocation failed");
        return RFX_ERR_OOM;
    }
    RFX_CUDA(cudaMemsetAsync(wsum, 0, sizeof(int32_t) * (size_t)c->N, c->stream));
    RFX_CUDA(cudaMemsetAsync(wcnt, 0, sizeof(int32_t) * (size_t)c->N, c->stream));
    dim3 g(nblk(c->n), c->T);
    tnodewt_walk_kernel<<<g, 256, 0, c->stream>>>(c->d_X, c->n, c->p, c->d_nodes, c->d_offs, c->d_nnode,
                                                  c->d_catgoleft, c->maxcat, c->d_nin, wsum, wcnt);
    tnodewt_final_kernel<<<nblk(c->N), 256, 0, c->stream>>>(c->N, wsum, wcnt, c->d_tnodewt);
    RFX_CUDA(cudaGetLastError());
    c->launches += 2;
    return RFX_OK;
}

rfx_status launch_casewise_votes(Ctx* c, const int32_t* d_leafnode, float* d_q) {
    if (c->nclass > 64) {
        set_error("case-wise votes: at most 64 classes");
        return RFX_ERR_UNSUPPORTED;
    }
    const size_t smem = 32 * (size_t)c->nclass * sizeof(float);
    casewise_votes_kernel<<<nblk(c->n, 32), 256, smem, c->stream>>>(d_leafnode, c->d_inbag, c->d_offs, c->d_nnode,
                                                                    c->d_nodeclass, c->d_tnodewt, c->n, c->T,
                                                                    c->nclass, d_q);
    RFX_CUDA(cudaGetLastError());
    c->launches += 1;
    return RFX_OK;
}

// Device bytes that a call's range table, and a chunk of trees' values in the
// case-wise importance, may take; RFX_CW_MB (megabytes) overrides, e.g. to run
// small forests in many pieces.
static size_t piece_bytes() {
    const char* e = std::getenv("RFX_CW_MB");
    const long mb = e ? std::atol(e) : 0;
    return (size_t)(mb > 0 ? mb : 256) << 20;
}

template <int MODE>
static rfx_status weighted_rows(Ctx* c, const int32_t* key, const int64_t* segbase, const int32_t* segoff,
                                const int32_t* memb, const long long* mass, double* out) {
    const int n = c->n, T = c->T;
    // the range table holds as many rows as piece_bytes takes (all rows of
    // the sizes whose matrix fits easily), fewer where memory is short
    Scratch sc(c);
    const size_t row_bytes = sizeof(WRange) * (size_t)T;
    int rows = (int)std::min<size_t>((size_t)n, std::max<size_t>(32, piece_bytes() / row_bytes));
    WRange* tab = sc.get<WRange>((size_t)rows * T);
    while (!tab && rows > 1) {
        rows = (rows + 1) / 2;
        tab = sc.get<WRange>((size_t)rows * T);
    }
    if (!tab) {
        set_error("weighted pair sums: scratch allocation failed");
        return RFX_ERR_OOM;
    }
    // member weights; RFX_CW_WEIGHTS=0 takes the form that runs without room for them
    const char* pre = std::getenv("RFX_CW_WEIGHTS");
    const bool per_pair = MODE == WR_PLAIN || (pre && std::string(pre) == "0");
    double* wm = per_pair ? nullptr : sc.get<double>((size_t)n * T);
    if (wm) {
        member_weight_kernel<MODE><<<dim3((n + 255) / 256, T), 256, 0, c->stream>>>(key, segbase, segoff, memb, mass,
                                                                                    c->d_nin, n, wm);
        RFX_CUDA(cudaGetLastError());
        c->launches += 1;
    }
    const int win = std::min(WR_WINDOW, n);
    const size_t smem = (size_t)win * sizeof(double2);
    for (int i0 = 0; i0 < n; i0 += rows) {
        const int i1 = std::min(n, i0 + rows);
        weighted_ranges_kernel<MODE><<<dim3((i1 - i0 + 31) / 32, (T + 31) / 32), 256, 0, c->stream>>>(
            key, segbase, segoff, memb, mass, c->d_nin, n, T, i0, i1, tab);
        if (wm || MODE == WR_PLAIN)
            weighted_row_kernel<MODE, true><<<i1 - i0, 32, smem, c->stream>>>(tab, i0, memb, wm, c->d_nin, c->d_nout,
                                                                              n, T, win, out);
        else
            weighted_row_kernel<MODE, false><<<i1 - i0, 32, smem, c->stream>>>(tab, i0, memb, wm, c->d_nin, c->d_nout,
                                                                               n, T, win, out);
        RFX_CUDA(cudaGetLastError());
        c->launches += 2;
    }
    return RFX_OK;
}

// Weighted FP64 pair sums (mode 0 case-wise, 2 unweighted) or the RF-GAP
// matrix (mode 1), packed upper triangle, from leaf lists of keys `key`
// (segbase/segoff/memb of those keys).
rfx_status launch_weighted_rows(Ctx* c, int mode, const int32_t* key, const int64_t* segbase, const int32_t* segoff,
                                const int32_t* memb, int64_t nkeys, double* out) {
    Scratch sc(c);
    long long* mass = sc.get<long long>((size_t)nkeys);
    if (!mass) {
        set_error("weighted pair sums: scratch allocation failed");
        return RFX_ERR_OOM;
    }
    key_mass_kernel<<<c->T, 512, 0, c->stream>>>(segbase, segoff, memb, c->d_nin, c->n, mass);
    RFX_CUDA(cudaGetLastError());
    c->launches += 1;
    if (mode == WR_PLAIN) return weighted_rows<WR_PLAIN>(c, key, segbase, segoff, memb, mass, out);
    if (mode == WR_RFGAP) return weighted_rows<WR_RFGAP>(c, key, segbase, segoff, memb, mass, out);
    return weighted_rows<WR_CASEWISE>(c, key, segbase, segoff, memb, mass, out);
}

rfx_status launch_gap_keys(Ctx* c, const int32_t* d_leafnode, int32_t* d_key) {
    const int64_t cells = (int64_t)c->T * c->n;
    gap_key_kernel<<<nblk(cells), 256, 0, c->stream>>>(d_leafnode, c->d_inbag, cells, d_key);
    RFX_CUDA(cudaGetLastError());
    c->launches += 1;
    return RFX_OK;
}

// Case-wise importance: per chunk of trees the walks (base and val), then the
// ordered sums per (tree, feature) and per (sample, feature); the per-feature
// sums at the end.  Needs d_joob / d_partner (OOB lists and permutation
// partners) and the testreebag node ids.
rfx_status launch_casewise_varimp(Ctx* c, const int32_t* d_leafnode, int impn, float* d_avimp, float* d_sqsd,
                                  float* d_qimp, float* d_qimpm) {
    const int n = c->n, p = c->p, T = c->T;
    // a chunk's values take at most piece_bytes (one tree at least)
    Scratch sc(c);
    float* rr = sc.get<float>((size_t)T * p);
    const size_t per_tree = (size_t)n * (p + 1);
    int chunk = (int)std::min<size_t>((size_t)T, std::max<size_t>(1, piece_bytes() / (per_tree * sizeof(float))));
    chunk = std::min(chunk, 65535);  // grid y
    float* buf = rr ? sc.get<float>(per_tree * chunk) : nullptr;
    while (rr && !buf && chunk > 1) {
        chunk = (chunk + 1) / 2;
        buf = sc.get<float>(per_tree * chunk);
    }
    if (!rr || !buf) {
        set_error("case-wise importance: scratch allocation failed");
        return RFX_ERR_OOM;
    }
    float* base = buf;
    float* val = buf + (size_t)n * chunk;
    int max_noob = 1;
    for (int t = 0; t < T; ++t) max_noob = std::max(max_noob, c->h_noob[t]);
    const int ivw = c->iv_words;
    for (int t0 = 0; t0 < T; t0 += chunk) {
        const int nt = std::min(chunk, T - t0);
        const dim3 g((max_noob + CW_THREADS - 1) / CW_THREADS, nt);
        auto go = [&](auto kernel) {
            kernel<<<g, CW_THREADS, 0, c->stream>>>(c->d_X, c->d_y, n, p, t0, c->d_nodes, c->d_nodeclass, c->d_offs,
                                                    c->d_nnode, c->d_catgoleft, c->maxcat, c->d_iv, ivw, c->d_joob,
                                                    c->d_noob, c->d_partner, d_leafnode, c->d_tnodewt, base, val,
                                                    c->d_err);
        };
        if (ivw == 1) go(cw_walk_kernel<1>);
        else if (ivw == 2) go(cw_walk_kernel<2>);
        else go(cw_walk_kernel<4>);
        cw_tree_kernel<<<dim3((p + 31) / 32, nt), 32, 0, c->stream>>>(n, p, t0, c->d_iv, ivw, c->d_joob, c->d_noob,
                                                                      base, val, rr);
        cw_sample_kernel<<<nblk((int64_t)n * (impn ? p : 1), 128), 128, 0, c->stream>>>(
            n, p, t0, t0 + nt, c->d_inbag, c->d_noob, base, val, impn, d_qimp, d_qimpm);
        RFX_CUDA(cudaGetLastError());
        c->launches += 3;
    }
    cw_feature_kernel<<<nblk(p, 32), 32, 0, c->stream>>>(rr, p, T, d_avimp, d_sqsd);
    RFX_CUDA(cudaGetLastError());
    c->launches += 1;
    return RFX_OK;
}

}  // namespace rfx
