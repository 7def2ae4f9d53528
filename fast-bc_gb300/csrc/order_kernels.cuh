// The locality order of batched runs on large graphs, on the device: recursive BFS bisection as in
// host_order.hpp.  A part (a range of the order) is laid out by a BFS from its first vertex that stays
// inside the part, then halved; parts of at most kOrdLeaf vertices are sorted by id.  One launch per level
// of the recursion: a part belongs to one block, or to a cluster of eight while there are few parts, and a
// BFS level costs that group one barrier.  Bound by the BFS levels' latency (a vertex, its row, the marks
// of its neighbours, one append); all parts of a level run side by side.
//
// Road-like graphs, the order and the relabelled rows together, by the host's threads (16 cores) before and
// here: 65,536 vertices 20 -> 5.5 ms, 262,144 34 -> 13, 1,024,000 98 -> 28, 4,194,304 500 -> 70 (58 of them
// in the launches, a third in the first three levels: 1,000 to 1,600 rounds of about 6 us).  The runs that
// use the order are as fast as with the host's.
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
    int32_t* mark;       // per vertex: part + 1 while unvisited, its negative once visited
    int32_t* err;        // set where a part took more rounds than it is given
    int32_t n, level, parts;
};

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

__global__ void order_init_kernel(int32_t n, int32_t* ord, int32_t* mark) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        ord[i] = i;
        mark[i] = 0;
    }
}

template <bool kCluster>
__global__ void __launch_bounds__(1024, 1) order_split_kernel(OrderArgs A) {
    namespace cg = cooperative_groups;
    // Appended entries of a round (three rotating words: one counts, the next is zero, the last is being
    // read) and the first unvisited position a seed scan finds (likewise), both in the first block.
    __shared__ int cnt_s[3];
    __shared__ int best_s[3];
    int* cnt = cnt_s;
    int* best = best_s;
    int C = 1, r = 0;
    if constexpr (kCluster) {
        cg::cluster_group cl = cg::this_cluster();
        C = (int)cl.num_blocks();
        r = (int)cl.block_rank();
        cnt = cl.map_shared_rank(cnt_s, 0);
        best = cl.map_shared_rank(best_s, 0);
    }
    auto sync = [&]() {
        if constexpr (kCluster) cg::this_cluster().sync();
        else __syncthreads();
    };
    const int lane = threadIdx.x & 31;
    const int T = C * (int)blockDim.x, t0 = r * (int)blockDim.x + (int)threadIdx.x;
    const bool lead = t0 == 0;
    const unsigned below = (1u << lane) - 1u;
    for (int p = (int)blockIdx.x / C; p < A.parts; p += (int)gridDim.x / C) {
        int lo, hi;
        order_range(A.n, A.level, p, lo, hi);
        const int len = hi - lo, me = p + 1;
        const int32_t* ord = A.ord + lo;
        int32_t* out = A.tmp + lo;
        if (len <= kOrdLeaf) {
            for (int i = t0; i < len; i += T) out[i] = ord[i];
            continue;
        }
        for (int i = t0; i < len; i += T) A.mark[ord[i]] = me;
        if (lead) {
            for (int j = 0; j < 3; ++j) {
                cnt[j] = 0;
                best[j] = len;
            }
        }
        sync();
        const int cap = order_rounds(len);
        int qh = 0, qt = 0, cur = 0, rounds = 0;
        int k = 0, kb = 0;  // this round's counter, this scan's word
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
                            __stcg(A.mark + s, -me);
                            __stcg(out + qt, s);
                        }
                        ++qt;
                        break;
                    }
                }
                sync();
                if (qh == qt) break;  // cannot be: qt < len leaves a vertex to find
            }
            if (lead) cnt[k == 2 ? 0 : k + 1] = 0;
            for (int base = qh + (t0 & ~31); base < qt; base += T) {
                const int i = base + lane;
                int e = 0, e1 = 0;
                if (i < qt) {
                    const int v = __ldcg(out + i);
                    e = A.rp[v];
                    e1 = A.rp[v + 1];
                }
                for (; __any_sync(kFull, e < e1); e += 4) {
                    int xs[4], mk[4];
                    bool push[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) xs[t] = e + t < e1 ? __ldg(A.adj + e + t).x : -1;
#pragma unroll
                    for (int t = 0; t < 4; ++t) mk[t] = xs[t] >= 0 ? __ldcg(A.mark + xs[t]) : 0;
                    unsigned m[4];
                    int tot = 0;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (mk[t] == me) mk[t] = atomicCAS(A.mark + xs[t], me, -me);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        push[t] = mk[t] == me;
                        m[t] = __ballot_sync(kFull, push[t]);
                        tot += __popc(m[t]);
                    }
                    if (tot == 0) continue;
                    int b = 0;
                    if (lane == 0) b = atomicAdd(&cnt[k], tot);
                    b = qt + __shfl_sync(kFull, b, 0);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int pos = b + __popc(m[t] & below);
                        if (push[t] && pos < len) __stcg(out + pos, xs[t]);
                        b += __popc(m[t]);
                    }
                }
            }
            sync();
            qh = qt;
            qt += *(volatile int*)&cnt[k];
            k = k == 2 ? 0 : k + 1;
        }
        sync();
        if (over) {  // the vertices not yet reached, in about their present order
            if (lead) {
                if (len > kOrdReport) atomicOr(A.err, 1);
                cnt[0] = 0;
            }
            sync();
            for (int base = t0 & ~31; base < len; base += T) {
                const int i = base + lane;
                const int v = i < len ? ord[i] : -1;
                const bool open = v >= 0 && __ldcg(A.mark + v) == me;
                const unsigned m = __ballot_sync(kFull, open);
                if (!m) continue;
                int b = 0;
                if (lane == 0) b = atomicAdd(&cnt[0], __popc(m));
                b = qt + __shfl_sync(kFull, b, 0);
                const int pos = b + __popc(m & below);
                if (open && pos < len) __stcg(out + pos, v);
                if (open) __stcg(A.mark + v, -me);  // no mark of an earlier level may equal a later part's
            }
            sync();
        }
    }
    if constexpr (kCluster) cg::this_cluster().sync();  // the first block's words outlive their readers
}

// Leaves: the last level's parts sorted by id, a thread each; inv[new] = old, nw[old] = new.
__global__ void order_leaf_kernel(int32_t n, int32_t level, int32_t parts, const int32_t* __restrict__ ord, int32_t* inv,
                                  int32_t* nw) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < parts; p += gridDim.x * blockDim.x) {
        int lo, hi;
        order_range(n, level, p, lo, hi);
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
