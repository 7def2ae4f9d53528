// Edge list -> CSR on the device, with the rules of DirectedWeightedGraph (DirectedWeightedGraph.h:
// 67-96, 136-170): n = 1 + the largest source id, a destination id >= n is an error, a weight
// must be > 0, and a repeated (source, destination) pair has its weights summed (in input
// order, as the host path does).  The engine then needs integer weights below 2^31.
//
// Rows are built by a counting scatter on the source id, each row is sorted by
// (destination, input index) -- one thread per row, rows of up to kRowMax edges (longer rows:
// the host path) -- and equal destinations are merged.
#pragma once
#include <cstdint>

namespace fbc {

constexpr int kRowMax = 1024;

// error bits
constexpr int kGbNegId = 1;      // negative vertex id
constexpr int kGbWeight = 2;     // weight <= 0 (or NaN)
constexpr int kGbDst = 4;        // destination >= n
constexpr int kGbLongRow = 8;    // a row longer than kRowMax (host path)
constexpr int kGbNonInt = 16;    // merged weight not an integer below 2^31

__global__ void gb_check_kernel(int64_t m, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                const double* __restrict__ w, int* maxsrc, int* err) {
    int mx = -1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        if (src[i] < 0 || dst[i] < 0) atomicOr(err, kGbNegId);
        if (!(w[i] > 0)) atomicOr(err, kGbWeight);
        mx = max(mx, src[i]);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(maxsrc, mx);
}

__global__ void gb_count_kernel(int64_t m, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                int32_t n, int32_t* deg, int* err) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        if (dst[i] >= n) atomicOr(err, kGbDst);
        atomicAdd(deg + src[i], 1);
    }
}

// keys[rs[src] + k] = (dst << 32 | i) in any order within the row (sorted afterwards)
__global__ void gb_scatter_kernel(int64_t m, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                  const int32_t* __restrict__ rs, int32_t* cursor, unsigned long long* keys) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t s = src[i];
        const int32_t k = atomicAdd(cursor + s, 1);
        keys[rs[s] + k] = ((unsigned long long)(uint32_t)dst[i] << 32) | (unsigned long long)(uint32_t)i;
    }
}

// sort each row's keys (insertion sort, rows <= kRowMax) and count its distinct destinations
__global__ void gb_sort_rows_kernel(int32_t n, const int32_t* __restrict__ rs, unsigned long long* keys,
                                    int32_t* ndeg, int* err) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t a = rs[v], b = rs[v + 1];
        if (b - a > kRowMax) {
            atomicOr(err, kGbLongRow);
            ndeg[v] = 0;
            continue;
        }
        for (int32_t i = a + 1; i < b; ++i) {
            const unsigned long long k = keys[i];
            int32_t j = i - 1;
            while (j >= a && keys[j] > k) {
                keys[j + 1] = keys[j];
                --j;
            }
            keys[j + 1] = k;
        }
        int32_t d = 0;
        for (int32_t i = a; i < b; ++i) d += (i == a || (keys[i] >> 32) != (keys[i - 1] >> 32));
        ndeg[v] = d;
    }
}

// merged rows: (dst, sum of its weights in input order) at rp[v] ..; per-graph statistics
__global__ void gb_merge_kernel(int32_t n, const int32_t* __restrict__ rs, const unsigned long long* __restrict__ keys,
                                const double* __restrict__ w, const int32_t* __restrict__ rp, int2* adj,
                                int32_t* indeg, int* maxw, unsigned long long* sumw, int* maxdeg, int* err) {
    int mw = 0, md = 0;
    unsigned long long sw = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t a = rs[v], b = rs[v + 1];
        int32_t o = rp[v];
        for (int32_t i = a; i < b;) {
            const uint32_t d = (uint32_t)(keys[i] >> 32);
            double x = 0.0;
            int32_t j = i;
            for (; j < b && (uint32_t)(keys[j] >> 32) == d; ++j) x += w[(uint32_t)keys[j]];
            int32_t wi = 0;
            if (x != floor(x) || x > 2147483647.0) atomicOr(err, kGbNonInt);
            else wi = (int32_t)x;
            adj[o++] = make_int2((int32_t)d, wi);
            atomicAdd(indeg + d, 1);
            mw = max(mw, wi);
            sw += (unsigned long long)wi;
            i = j;
        }
        md = max(md, o - rp[v]);
    }
    mw = __reduce_max_sync(0xffffffffu, mw);
    md = __reduce_max_sync(0xffffffffu, md);
    for (int d = 16; d > 0; d >>= 1) sw += __shfl_down_sync(0xffffffffu, sw, d);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(maxw, mw);
        atomicMax(maxdeg, md);
        atomicAdd(sumw, sw);  // one per warp: a per-thread add to one word serialises
    }
}

// How rich a graph is in ties: of the vertices within two edges of a sample of vertices, how many are reached by
// several shortest ones of these ways.  A warp per sampled vertex; of longer rows the first kTieRow edges.
constexpr int kTieRow = 16;
constexpr int kTieSamples = 1024;
constexpr int kTieWarps = 4;  // of a block
__global__ void __launch_bounds__(32 * kTieWarps) gb_ties_kernel(int32_t n, const int32_t* __restrict__ rp,
                                                                 const int2* __restrict__ adj, int* targets, int* tied) {
    __shared__ uint2 ways[kTieWarps][kTieRow * (kTieRow + 1)];  // (vertex, length)
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint2* const way = ways[wid];
    int nt = 0, nd = 0;
    const int samples = min(n, kTieSamples);
    for (int k = blockIdx.x * kTieWarps + wid; k < samples; k += gridDim.x * kTieWarps) {
        const int u = (int)((int64_t)k * n / samples);
        const int e = rp[u], deg = min(rp[u + 1] - e, kTieRow);
        int2 a = make_int2(0, 0);
        int f = 0, len = 0;
        if (lane < deg) {
            a = adj[e + lane];
            f = rp[a.x];
            len = min(rp[a.x + 1] - f, kTieRow);
        }
        int cnt = 0;
        for (int i = 0; i < deg; ++i) {
            const int x = __shfl_sync(0xffffffffu, a.x, i), w = __shfl_sync(0xffffffffu, a.y, i);
            const int fi = __shfl_sync(0xffffffffu, f, i), li = __shfl_sync(0xffffffffu, len, i);
            if (lane == li) way[cnt + li] = make_uint2((unsigned)x, (unsigned)w);
            if (lane < li) {
                const int2 b = adj[fi + lane];
                way[cnt + lane] = make_uint2((unsigned)b.x, (unsigned)w + (unsigned)b.y);
            }
            cnt += li + 1;
        }
        __syncwarp();
        for (int r = lane; r < cnt; r += 32) {
            const uint2 me = way[r];
            int same = 0;
            bool least = me.x != (unsigned)u;  // the first of the shortest ways to this vertex
            for (int q = 0; q < cnt; ++q) {
                const uint2 o = way[q];
                if (o.x != me.x) continue;
                if (o.y < me.y || (o.y == me.y && q < r)) least = false;
                same += o.y == me.y;
            }
            nd += least;
            nt += least && same > 1;
        }
        __syncwarp();
    }
    nt = __reduce_add_sync(0xffffffffu, nt);
    nd = __reduce_add_sync(0xffffffffu, nd);
    if (lane == 0 && nd) {
        atomicAdd(targets, nd);
        if (nt) atomicAdd(tied, nt);
    }
}

// Hops in which a search from a vertex (one a block) has met `few` and `many` vertices (0: never): in a plane four
// times the vertices take about twice the hops, in a small world a few more.  Along the first kTieRow edges of a row.
constexpr int kBallMost = 2048;   // `many` at most
constexpr int kBallQueue = 3072;
constexpr int kBallTable = 8192;  // vertices met, hashed
constexpr int kBallHops = 256;
constexpr int kBallStarts = 4;
__global__ void __launch_bounds__(256) gb_ball_kernel(int32_t n, const int32_t* __restrict__ rp, const int2* __restrict__ adj,
                                                      int few, int many, int* hops) {
    __shared__ int table[kBallTable], queue[kBallQueue], cnt;
    const int u = (int)((int64_t)(blockIdx.x + 1) * n / (kBallStarts + 1));
    for (int i = threadIdx.x; i < kBallTable; i += blockDim.x) table[i] = -1;
    __syncthreads();
    const auto slot = [](int x) { return (int)(((unsigned)x * 2654435761u) >> 19); };  // (13 bits)
    if (threadIdx.x == 0) {
        table[slot(u)] = u;
        queue[0] = u;
        cnt = 1;
    }
    __syncthreads();
    int lo = 0, hi = 1, h1 = 0, h2 = 0;
    for (int hop = 1; hop <= kBallHops; ++hop) {
        for (int i = lo + (int)threadIdx.x; i < hi; i += blockDim.x) {
            const int v = queue[i], e0 = rp[v], e1 = min(rp[v + 1], e0 + kTieRow);
            for (int e = e0; e < e1 && *(volatile int*)&cnt < kBallQueue; ++e) {
                const int x = adj[e].x;
                int s = slot(x);
                for (int p = 0; p < 64; ++p, s = (s + 1) & (kBallTable - 1)) {
                    const int old = atomicCAS(table + s, -1, x);
                    if (old == -1) {
                        const int at = atomicAdd(&cnt, 1);
                        if (at < kBallQueue) queue[at] = x;
                    }
                    if (old == -1 || old == x) break;
                }
            }
        }
        __syncthreads();
        const int met = min(cnt, kBallQueue);
        __syncthreads();
        if (!h1 && met >= few) h1 = hop;
        if (met >= many) h2 = hop;
        if (h2 || met == hi) break;
        lo = hi;
        hi = met;
    }
    if (threadIdx.x == 0) {
        hops[2 * blockIdx.x] = h2 ? h1 : 0;
        hops[2 * blockIdx.x + 1] = h2;
    }
}

// The CSR in the caller's types: 64-bit offsets, destinations, weights as doubles (each null: not wanted).
__global__ void gb_export_kernel(int32_t n, int64_t m, const int32_t* __restrict__ rp, const int2* __restrict__ adj,
                                 int64_t* __restrict__ rp64, int32_t* __restrict__ col, double* __restrict__ w) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    if (rp64)
        for (int64_t v = t0; v <= n; v += nt) rp64[v] = rp[v];
    if (!col && !w) return;
    for (int64_t e = t0; e < m; e += nt) {
        const int2 a = adj[e];
        if (col) col[e] = a.x;
        if (w) w[e] = (double)a.y;
    }
}

__global__ void gb_max_kernel(int32_t n, const int32_t* __restrict__ x, int* out) {
    int mx = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        mx = max(mx, x[v]);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(out, mx);
}

}  // namespace fbc
