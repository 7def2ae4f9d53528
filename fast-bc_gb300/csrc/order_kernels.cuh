// The locality order of batched runs on large graphs, on the device: the recursive BFS bisection of
// host_order.hpp, and the same permutation (but for small parts of very many rounds, below).  A part (a range of
// the order) is laid out by a BFS from its first vertex that stays inside the part, then halved; parts of at most
// kOrdLeaf vertices are sorted by id.  One launch per level of the recursion: a part belongs to one block, or to a
// cluster of eight while there are few parts; all parts of a level run side by side.
//
// A BFS round costs three barriers: every open neighbour is claimed by the least position next to it (an atomicMin
// on its mark), the claims are counted and summed over the threads in their order, and the children appended at
// the sums.  So the order follows the queue and the rows alone.  Appending whatever a thread wins to a shared
// counter takes one barrier and 4.2, 9.5, 22 and 69 ms on the sizes below, but leaves a level in the order of the
// threads' timing: rows are sorted by the new ids, so a vertex's dependency was summed in another order for another
// handle of the same graph.  Bound by the rounds' latency (a vertex, its row, the marks of its neighbours, twice).
//
// Road-like graphs, the order, the relabelled rows and their quads together, by the host's threads (16 cores) and
// here: 65,536 vertices 20 and 5.9 ms, 262,144 34 and 15, 1,024,000 98 and 39, 4,194,304 500 and 128.
#pragma once
#include <cooperative_groups.h>

#include "brandes_kernels.cuh"
#include "cluster_build.cuh"

namespace fbc {

constexpr int kOrdLeaf = 16;
constexpr int kOrdMaxDeg = 64;  // a row is a thread's; graphs with longer rows are ordered on the host
constexpr int kOrdCluster = 8;

struct OrderArgs {
    const int32_t* rp;
    const int2* adj;
    const int32_t* ord;  // the order so far
    int32_t* tmp;        // this level's
    uint32_t* mark;      // per vertex: kOrdOpen | its part's number while unvisited; then who claimed it
    int32_t* err;        // set where a part took more rounds than it is given
    int32_t n, level, parts;
};

// Marks.  Part p of `level` halvings has the number 2^level + p, its halves twice that and one more, so that
// no two parts of the recursion share one.  A visited vertex has the position of the parent that claimed
// it (positions of different parts do not meet), a seed kOrdSeed.
constexpr uint32_t kOrdOpen = 0x80000000u, kOrdSeed = 0x7fffffffu;

// the range of part p of `level` halvings of [0, n)
__device__ __forceinline__ void order_range(int n, int level, int p, int& lo, int& hi) {
    lo = 0;
    hi = n;
    for (int b = level - 1; b >= 0; --b) {
        const int mid = lo + (hi - lo) / 2;
        if ((p >> b) & 1) lo = mid;
        else hi = mid;
    }
}

// BFS rounds and seeds a part may take: several times what a road-like part needs.  A part that needs more
// (a long path, many components) keeps its remaining vertices in their present order, and reports it when
// it is large: the state of 64K vertices is a few megabytes of the L2 cache, however it is ordered.
constexpr int kOrdReport = 65536;
__device__ __forceinline__ int order_rounds(int len) { return 256 + 8 * (int)sqrtf((float)len); }

__global__ void order_init_kernel(int32_t n, int32_t* ord, uint32_t* mark) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        ord[i] = i;
        mark[i] = kOrdOpen | 1u;
    }
}

// fn(x) over the destinations of row [e, e1), four loads in flight
template <class F>
__device__ __forceinline__ void order_row(const int2* adj, int e, int e1, F&& fn) {
    for (; e < e1; e += 4) {
        int xs[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) xs[t] = e + t < e1 ? __ldg(adj + e + t).x : -1;
        fn(xs);
    }
}

template <bool kCluster>
__global__ void __launch_bounds__(1024, 1) order_split_kernel(OrderArgs A) {
    namespace cg = cooperative_groups;
    // Every warp's children in a step of a round, in every block of the cluster (two in rotation), and the
    // first unvisited position a seed scan finds (three in rotation), in the first block.
    constexpr int kWarps = kCluster ? 32 * kOrdCluster : 32;
    __shared__ int sums[2][kWarps];
    __shared__ int best_s[3];
    int* best = best_s;
    int C = 1, r = 0;
    if constexpr (kCluster) {
        cg::cluster_group cl = cg::this_cluster();
        C = (int)cl.num_blocks();
        r = (int)cl.block_rank();
        best = cl.map_shared_rank(best_s, 0);
    }
    auto sync = [&]() {
        if constexpr (kCluster) cg::this_cluster().sync();
        else __syncthreads();
    };
    const int lane = threadIdx.x & 31;
    const int T = C * (int)blockDim.x, t0 = r * (int)blockDim.x + (int)threadIdx.x;
    const int W = T >> 5, gw = t0 >> 5, per = (W + 31) / 32;  // warps of the part, this one, a lane's share of them
    const bool lead = t0 == 0;
    int buf = 0;
    // Exclusive sum of c over the part's threads in their order, and its total.
    auto scan = [&](int c, int& total) {
        int x = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += y;
        }
        const int mine = __shfl_sync(kFull, x, 31);
        if constexpr (kCluster) {
            if (lane < C) cg::this_cluster().map_shared_rank(&sums[buf][gw], lane)[0] = mine;
        } else {
            if (lane == 0) sums[buf][gw] = mine;
        }
        sync();
        int part = 0;  // of this lane's warps, and of those before gw
        int before = 0;
        for (int k = lane * per; k < min((lane + 1) * per, W); ++k) {
            const int s = *(volatile int*)&sums[buf][k];
            part += s;
            if (k < gw) before += s;
        }
        buf ^= 1;
        total = __reduce_add_sync(kFull, part);
        return __reduce_add_sync(kFull, before) + x - c;
    };
    for (int p = (int)blockIdx.x / C; p < A.parts; p += (int)gridDim.x / C) {
        int lo, hi;
        order_range(A.n, A.level, p, lo, hi);
        const int len = hi - lo;
        const uint32_t num = (uint32_t)(A.parts + p), me = kOrdOpen | num;
        const int32_t* ord = A.ord + lo;
        int32_t* out = A.tmp + lo;
        if (len <= kOrdLeaf) {
            for (int i = t0; i < len; i += T) out[i] = ord[i];
            continue;
        }
        if (lead)
            for (int j = 0; j < 3; ++j) best[j] = len;
        sync();
        const int cap = order_rounds(len);
        int qh = 0, qt = 0, cur = 0, rounds = 0;
        int kb = 0;  // this scan's word
        bool over = false;
        while (qt < len) {
            if (++rounds > cap) {
                over = true;
                break;
            }
            if (qh == qt) {  // nothing left to expand: the next unvisited vertex, in the present order
                for (; cur < len; cur += T) {
                    const int i = cur + t0;
                    const bool open = i < len && __ldcg(A.mark + ord[i]) == me;
                    if (lead) best[kb == 2 ? 0 : kb + 1] = len;
                    const unsigned m = __ballot_sync(kFull, open);
                    if (m && lane == __ffs(m) - 1) atomicMin(&best[kb], i);
                    sync();
                    const int b = *(volatile int*)&best[kb];
                    kb = kb == 2 ? 0 : kb + 1;
                    if (b < len) {
                        cur = b + 1;
                        if (lead) {
                            const int s = ord[b];
                            __stcg(A.mark + s, kOrdSeed);
                            __stcg(out + qt, s);
                        }
                        ++qt;
                        break;
                    }
                }
                sync();
                if (qh == qt) break;  // cannot be: qt < len leaves a vertex to find
            }
            // every open neighbour goes to the frontier vertex of least position next to it ...
            const uint32_t top = (uint32_t)(lo + qt);
            for (int i = qh + t0; i < qt; i += T) {
                const uint32_t key = (uint32_t)(lo + i);
                const int v = __ldcg(out + i);
                order_row(A.adj, A.rp[v], A.rp[v + 1], [&](const int (&xs)[4]) {
                    uint32_t w[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) w[t] = xs[t] >= 0 ? __ldcg(A.mark + xs[t]) : 0u;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (xs[t] >= 0 && (w[t] == me || (w[t] > key && w[t] < top))) atomicMin(A.mark + xs[t], key);
                });
            }
            sync();
            // ... which appends it: in the order of the parents, and of their rows
            int at = qt;
            for (int base = qh; base < qt; base += T) {
                const int i = base + t0;
                const uint32_t key = (uint32_t)(lo + i);
                int e = 0, e1 = 0;
                if (i < qt) {
                    const int v = __ldcg(out + i);
                    e = A.rp[v];
                    e1 = A.rp[v + 1];
                }
                unsigned long long won = 0ull;  // of up to kOrdMaxDeg edges
                int k = 0;
                order_row(A.adj, e, e1, [&](const int (&xs)[4]) {
                    uint32_t w[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) w[t] = xs[t] >= 0 ? __ldcg(A.mark + xs[t]) : kOrdSeed;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (w[t] == key) won |= 1ull << (k + t);
                    k += 4;
                });
                int total;
                int pos = at + scan(__popcll(won), total);
                for (; won; won &= won - 1ull) {
                    const int x = __ldg(A.adj + e + __ffsll((long long)won) - 1).x;
                    if (pos < len) __stcg(out + pos, x);
                    ++pos;
                }
                at += total;
            }
            sync();
            qh = qt;
            qt = at;
        }
        sync();
        if (over) {  // the vertices not yet reached, in their present order
            if (lead && len > kOrdReport) atomicOr(A.err, 1);
            int at = qt;
            for (int base = 0; base < len; base += T) {
                const int i = base + t0;
                const int v = i < len ? ord[i] : -1;
                const bool open = v >= 0 && __ldcg(A.mark + v) == me;
                int total;
                const int pos = at + scan(open ? 1 : 0, total);
                if (open && pos < len) __stcg(out + pos, v);
                at += total;
            }
            sync();
        }
        // the marks of the halves
        for (int i = t0; i < len; i += T) {
            const int v = __ldcg(out + i);
            if ((unsigned)v < (unsigned)A.n) __stcg(A.mark + v, kOrdOpen | (2u * num + (i >= len / 2 ? 1u : 0u)));
        }
        sync();
    }
    if constexpr (kCluster) cg::this_cluster().sync();  // the blocks' words outlive their writers
}

// Leaves: the last level's parts sorted by id, a thread each (the first half's takes both halves where the part
// above them is a leaf itself); inv[new] = old, nw[old] = new.
__global__ void order_leaf_kernel(int32_t n, int32_t level, int32_t parts, const int32_t* __restrict__ ord, int32_t* inv,
                                  int32_t* nw) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < parts; p += gridDim.x * blockDim.x) {
        int lo, hi;
        if (level > 0) {
            order_range(n, level - 1, p >> 1, lo, hi);
            if (hi - lo <= kOrdLeaf && (p & 1)) continue;
        }
        if (level == 0 || hi - lo > kOrdLeaf) order_range(n, level, p, lo, hi);
        for (int i = lo; i < hi; ++i) {
            const int v = ord[i];
            int j = i;
            while (j > lo && inv[j - 1] > v) {
                inv[j] = inv[j - 1];
                --j;
            }
            inv[j] = v;
        }
        for (int i = lo; i < hi; ++i) nw[inv[i]] = i;
    }
}

// The relabelled CSR: degrees in the new order (scanned to row offsets by the caller), then the rows, each
// sorted by destination, packed as well where adj4 is given (ids below 2^24, weights below 256).
__global__ void order_degree_kernel(int32_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ inv, int32_t* deg) {
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
        const int v = inv[u];
        deg[u] = rp[v + 1] - rp[v];
    }
}

__global__ void order_rows_kernel(int32_t n, const int32_t* __restrict__ rp, const int2* __restrict__ adj,
                                  const int32_t* __restrict__ inv, const int32_t* __restrict__ nw,
                                  const int32_t* __restrict__ nrp, int2* nadj, uint32_t* adj4) {
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
        const int v = inv[u], e0 = rp[v], d = rp[v + 1] - e0, o = nrp[u];
        for (int i = 0; i < d; ++i) {
            const int2 a = __ldg(adj + e0 + i);
            const int2 b = make_int2(nw[a.x], a.y);
            int j = o + i;
            while (j > o && nadj[j - 1].x > b.x) {
                nadj[j] = nadj[j - 1];
                --j;
            }
            nadj[j] = b;
        }
        if (adj4)
            for (int i = o; i < o + d; ++i) adj4[i] = (uint32_t)nadj[i].x | ((uint32_t)nadj[i].y << 24);
    }
}

// Reverse weights: edge u -> x gets the weight of x -> u; *asym is set where there is none.
__global__ void order_revw_kernel(int32_t n, const int32_t* __restrict__ nrp, const int2* __restrict__ nadj, uint8_t* revw,
                                  int32_t* asym) {
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x)
        for (int e = nrp[u]; e < nrp[u + 1]; ++e) {
            const int x = __ldg(nadj + e).x, end = nrp[x + 1];
            int f = nrp[x];
            while (f < end && __ldg(nadj + f).x < u) ++f;
            if (f < end && __ldg(nadj + f).x == u) revw[e] = (uint8_t)__ldg(nadj + f).y;
            else *asym = 1;
        }
}

}  // namespace fbc
