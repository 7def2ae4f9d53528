// The k-means step of the clustered pivot selection on the device:
// PlusPlusKMeans::computeCentroids (libfastbc/include/kmeans/PlusPlusKMeans.h:76-147) with its
// k-means++ initialisation (PlusPlusKMeans.h:150-183) and stopping rule (PlusPlusKMeans.h:186-207),
// for many independent point sets (one per Louvain community) at once, one thread-block cluster per set.
//
// A point is a vertex's border vector, normalized (VertexInfo::normalize): integer lengths and
// integer path counts.  Between two points VertexInfo::squaredDistance is a sum of integer squares,
// computed here in integers -- the same value the reference's double sum holds exactly (sets whose
// sums could pass 2^53 are refused).  The rounded steps keep the reference's operation
// order, each product and sum rounded separately (no fused multiply-add):
//   * the running mean distance of the initialisation, cdist = cdist * (1 - 1/i) + d * (1/i);
//   * a centroid's mean vector, the exact member sums divided by the member count;
//   * the distance of the mean to a member, summed over the borders in order.
// Ties keep the reference's sequential choices: the first point of largest running distance, the
// first centroid of least distance, the first member (in point order) nearest to the mean.
// Every loop is bounded by k, the set size and max_iter + 1 Lloyd steps.
//
// What it does without, with the same result (the reference's algorithm repeats all of it; with k
// half the points, nearly all centroids coincide -- 4 to 6 distinct ones of 778 after the
// initialisation on a 1,557-point community, 46 at the end):
//   * the distances to a centroid chosen again in the initialisation (the last kKmRows distinct ones'
//     are kept);
//   * centroids on a point that an earlier centroid holds (never the first nearest);
//   * distances to centroids that did not move, for points whose own one did not move either;
//   * sums, means and member distances of centroids whose members did not change (the sums follow
//     the changes, exactly);
//   * FP64 distances to the mean, two a clock per SM, where integers decide: n^2 times the squared
//     distance of a member to the mean of n is an exact integer, and the reference's rounded value is
//     within a relative error bound of it, so only members within that bound of the least one are
//     computed in its arithmetic -- none where there is one such member.
// A cluster of up to eight blocks shares a set's points, because the sets are few and of very
// different sizes; distances are summed in 32 bits where the set's range allows it.  20 communities of
// a 108x108 grid (143 to 1,557 points, 45 to 124 borders): a call of 739 ms
// with one block per set and none of this takes 5.0 (on the device 735 and 4.1; 2.9 of 9.2 million cycles of
// the largest set are its 777 initialisation steps, each a choice among all its blocks).
#pragma once
#include <cooperative_groups.h>
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace fbc {

constexpr int kKmThreads = 512;
constexpr int kKmCluster = 8;   // most blocks of a set
constexpr int kKmTile = 8;      // centroids whose distances a thread sums at once
constexpr int kKmBlock = 512;   // borders of a staged centroid tile
constexpr int kKmRows = 8;      // kept distance rows of the initialisation

struct KMSet {
    int64_t in_off;    // first entry of the set in the input vectors (entry j * nb + i)
    int64_t x_off;     // first entry of the set's points in X: entry i * np + j = border i of point j
    int64_t ws_off;    // byte offset of the set's work area in KMParams::ws
    int64_t out_off;   // first output entry (k of them)
    int64_t p_off;     // first point of the set in the weight array
    int32_t np, nb, k;
    int32_t id;        // the caller's number of the set
};

// What the packing found in a set: a length that is no integer in [0, 2^31), the largest length and
// count magnitude.
struct KMMeta {
    int32_t bad;
    uint32_t lmax, cmax;
    int32_t pad;
};

struct KMParams {
    const KMSet* sets;
    const KMMeta* meta;       // by id
    const int2* X;            // (length, count) per border and point, sets back to back
    const int32_t* wt;        // point weights
    char* ws;
    double min_variance;
    int32_t max_iter;
    int32_t* out_idx;         // centroid c of set s: point index within the set
    int32_t* out_w;           // summed weights of its members in the last assignment
};

// Counters of a set shared by its blocks.
struct KMCtl {
    int32_t ndirty, nmoved, nkept, ncand, go;
};

// Work area of one set (all offsets 256-byte aligned).
struct KMWork {
    KMCtl* ctl;
    double* cdist;            // np: running distances of the initialisation
    unsigned long long* key;  // np: n^2 x squared distance to the mean, or bits of the rounded distance
    double* rows;             // kKmRows * np: distances to recent centroids; then a list of points
    long long* bd;            // np: distance to the assigned centroid
    int32_t* assign;          // np
    int32_t* was;             // np: the former assignment
    int32_t* first;           // np: first centroid on a point
    int32_t* cand;            // np: members whose rounded distances decide
    int32_t* cent;            // k: the centroids of the current Lloyd step
    int32_t* ncent;           // k: the next step's
    int32_t* cnt;             // k
    int32_t* wsum;            // k
    int32_t* bestj;           // k: first candidate, then first nearest member
    int32_t* ncand;           // k: candidates
    int32_t* dirty;           // k: members changed in this step
    int32_t* moved;           // k: moved by the last step
    int32_t* dlist;           // k: the dirty ones
    int2* mlist;              // k: (centroid, point) of moved ones that are the first on their point
    int2* ulist;              // k: the others that are
    unsigned long long* best; // k: least key
    unsigned long long* rbest;// k: least rounded distance (bits of a non-negative double)
    long long* sum;           // 2 * k * nb: member sums, lengths then counts
};

__host__ __device__ inline int64_t km_al(int64_t x) { return (x + 255) & ~int64_t(255); }
__host__ __device__ inline int64_t km_work_bytes(int64_t np, int64_t nb, int64_t k) {
    return 256 + 3 * km_al(np * 8) + km_al(kKmRows * np * 8) + 4 * km_al(np * 4) + 8 * km_al(k * 4) + 5 * km_al(k * 8) +
           km_al(2 * k * (nb > 0 ? nb : 1) * 8);
}
__device__ inline KMWork km_carve(char* p, int64_t np, int64_t nb, int64_t k) {
    KMWork w;
    auto take = [&](int64_t bytes) {
        char* q = p;
        p += km_al(bytes);
        return q;
    };
    w.ctl = (KMCtl*)take(256);
    w.cdist = (double*)take(np * 8);
    w.key = (unsigned long long*)take(np * 8);
    w.rows = (double*)take(kKmRows * np * 8);
    w.bd = (long long*)take(np * 8);
    w.assign = (int32_t*)take(np * 4);
    w.was = (int32_t*)take(np * 4);
    w.first = (int32_t*)take(np * 4);
    w.cand = (int32_t*)take(np * 4);
    w.cent = (int32_t*)take(k * 4);
    w.ncent = (int32_t*)take(k * 4);
    w.cnt = (int32_t*)take(k * 4);
    w.wsum = (int32_t*)take(k * 4);
    w.bestj = (int32_t*)take(k * 4);
    w.ncand = (int32_t*)take(k * 4);
    w.dirty = (int32_t*)take(k * 4);
    w.moved = (int32_t*)take(k * 4);
    w.dlist = (int32_t*)take(k * 8);
    w.mlist = (int2*)take(k * 8);
    w.ulist = (int2*)take(k * 8);
    w.best = (unsigned long long*)take(k * 8);
    w.rbest = (unsigned long long*)take(k * 8);
    w.sum = (long long*)take(2 * k * (nb > 0 ? nb : 1) * 8);
    return w;
}

// The range in which every squared distance is exact in a double, as the reference's sums are.
__host__ __device__ inline double km_range(int nb, uint32_t lmax, uint32_t cmax) {
    return (double)nb * ((double)lmax * (double)lmax + 4.0 * ((double)cmax * (double)cmax));
}

// Input vectors (point-major, lengths as doubles) -> X (border-major int pairs), checked, 32 x 32
// entries at a time through shared memory.  Block (x, y): part x of the sets y, y + gridDim.y, ...
__global__ void __launch_bounds__(256) km_pack_kernel(const KMSet* __restrict__ sets, int nsets, const double* __restrict__ len,
                                                      const int32_t* __restrict__ cnt, int2* __restrict__ X, KMMeta* meta) {
    __shared__ int2 tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int s = blockIdx.y; s < nsets; s += gridDim.y) {
        const KMSet S = sets[s];
        const int tj = (S.np + 31) / 32, ti = (S.nb + 31) / 32;
        int bad = 0;
        unsigned lm = 0, cm = 0;
        for (int64_t t = blockIdx.x; t < (int64_t)tj * ti; t += gridDim.x) {
            const int j0 = (int)(t / ti) * 32, i0 = (int)(t % ti) * 32;
            for (int r = ty; r < 32; r += 8)
                if (j0 + r < S.np && i0 + tx < S.nb) {
                    const int64_t e = S.in_off + (int64_t)(j0 + r) * S.nb + i0 + tx;
                    const double l = len[e];
                    const int c = cnt[e];
                    const bool ok = l >= 0.0 && l <= 2147483647.0 && l == floor(l);
                    bad |= !ok;
                    const int li = ok ? (int)l : 0;
                    lm = max(lm, (unsigned)li);
                    cm = max(cm, c < 0 ? 0u - (unsigned)c : (unsigned)c);
                    tile[r][tx] = make_int2(li, c);
                }
            __syncthreads();
            for (int r = ty; r < 32; r += 8)
                if (i0 + r < S.nb && j0 + tx < S.np) X[S.x_off + (int64_t)(i0 + r) * S.np + j0 + tx] = tile[tx][r];
            __syncthreads();
        }
        bad = __reduce_or_sync(0xffffffffu, bad);
        lm = __reduce_max_sync(0xffffffffu, lm);
        cm = __reduce_max_sync(0xffffffffu, cm);
        if (tx == 0) {
            if (bad) atomicOr(&meta[S.id].bad, 1);
            if (lm) atomicMax(&meta[S.id].lmax, lm);
            if (cm) atomicMax(&meta[S.id].cmax, cm);
        }
    }
}

// Shared memory of a block.
struct KMShared {
    int2 tile[kKmBlock][kKmTile];       // staged centroids: border-major
    unsigned long long sv[32];
    int sj[32];
    unsigned long long mv[2][kKmCluster];  // every block's candidate of an initialisation step
    int mj[2][kKmCluster];
    double p[2];                        // 1 / i of this and the next initialisation step
    int row_of[kKmRows];                // centroid of each kept row
    int nr;
    double var;
};

// (value, index): the largest value, the smallest index among equal ones.  Values are the bits of
// non-negative doubles, which order as the doubles do (an FP64 comparison costs sixteen issue slots).
__device__ __forceinline__ void km_max(unsigned long long& v, int& j, unsigned long long v2, int j2) {
    if (v2 > v || (v2 == v && j2 < j)) { v = v2; j = j2; }
}

// kNarrow: every squared distance of the set is below 2^32.
template <bool kNarrow>
struct KMeans {
    using Acc = typename std::conditional<kNarrow, uint32_t, long long>::type;
    const KMSet& S;
    const int2* X;
    const KMWork& W;
    KMShared& M;
    int rank, nblk;   // of the cluster
    int p0, p1;       // the block's points
    int exact_n;         // most members of a centroid whose keys decide (below)
    double slack0, slack1;

    // n^2 times the squared distance of a member to the mean of n members is a sum of squares of 32-bit
    // integers, exact in 64 bits up to some n.  The reference's rounded distance: a difference of
    // the mean and an entry is 0 when it is exactly so, else at least 1 / n, and off by at most
    // u * most (the mean's rounding; u = 2^-53, most: the set's largest length or count) and u of itself; the
    // square and the sum of 2 nb terms add u each.  So it is within eta = 2 n most u + (2 nb + 4) u of
    // the exact value, and the member nearest by it is within 3 eta of the exactly nearest one; twelve
    // eta leave room for the second order.
    __device__ void bounds(double range, double most) {
        const double u = 1.1102230246251565e-16;
        slack0 = 12.0 * (2.0 * S.nb + 4.0) * u;
        slack1 = 12.0 * 2.0 * most * u;
        double n = fmin(sqrt(9.0e18 / fmax(range, 1.0)), 2147483646.0 / (2.0 * fmax(most, 1.0)));
        n = fmin(n, (0.01 - slack0) / fmax(slack1, 1e-30));
        exact_n = n > 2147483646.0 ? 2147483646 : n < 1.0 ? 0 : (int)n;
    }
    // whether member j of centroid c (n members) may be the nearest to the mean
    __device__ bool candidate(int j, int c, int n) const {
        return n > exact_n || (double)W.key[j] <= (double)__ldcg(W.best + c) * (1.0 + (slack0 + slack1 * n));
    }

    __device__ static Acc term(int2 a, int2 b) {
        const int d = a.x - b.x, e = a.y - b.y;
        if constexpr (kNarrow) return (uint32_t)d * (uint32_t)d + (uint32_t)e * (uint32_t)e;
        else return (long long)d * d + (long long)e * e;
    }

    // Distances of the block's points (listed in `pts`, or p0 .. p1 when null) to the centroids of a
    // list, kKmTile at a time; each point's least (distance, centroid) so far is in (W.bd, W.assign).
    // Several lanes share a point where the block has few (each sums every G-th border).
    __device__ void nearest(const int2* list, int nlist, const int32_t* pts, int npts) {
        const int np = S.np, nb = S.nb;
        int G = 1;
        while (G < 8 && 2 * G * npts <= kKmThreads) G <<= 1;
        const int per = 32 / G;                    // points of a warp
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const int pl = lane % per, gl = lane / per;
        for (int t0 = 0; t0 < nlist; t0 += kKmTile) {
            int c[kKmTile];
            const int2 mine = t0 + (int)(threadIdx.x % kKmTile) < nlist ? __ldcg(list + t0 + threadIdx.x % kKmTile)
                                                                       : make_int2(-1, 0);
#pragma unroll
            for (int q = 0; q < kKmTile; ++q) c[q] = __shfl_sync(0xffffffffu, mine.x, q);
            const int passes = (npts + per * (kKmThreads / 32) - 1) / (per * (kKmThreads / 32));
            for (int ps = 0; ps < passes; ++ps) {
                const int at = (ps * (kKmThreads / 32) + wid) * per + pl;
                const bool on = at < npts;
                const int j = on ? (pts ? __ldcg(pts + at) : p0 + at) : p0;
                Acc acc[kKmTile];
#pragma unroll
                for (int q = 0; q < kKmTile; ++q) acc[q] = 0;
                for (int b0 = 0; b0 < nb; b0 += kKmBlock) {
                    const int bn = min(kKmBlock, nb - b0);
                    if (ps == 0 || nb > kKmBlock) {  // stage the tile (kept over the passes when it is whole)
                        __syncthreads();
                        for (int e = threadIdx.x; e < bn * kKmTile; e += kKmThreads) {
                            const int i = e / kKmTile, q = e % kKmTile;  // q = threadIdx.x % kKmTile
                            M.tile[i][q] = __ldg(X + (int64_t)(b0 + i) * np + mine.y);
                        }
                        __syncthreads();
                    }
#pragma unroll 4
                    for (int i = gl; i < bn; i += G) {
                        const int2 x = __ldg(X + (int64_t)(b0 + i) * np + j);
#pragma unroll
                        for (int q = 0; q < kKmTile; ++q) acc[q] += term(x, M.tile[i][q]);
                    }
                }
                for (int o = per; o < 32; o <<= 1) {
#pragma unroll
                    for (int q = 0; q < kKmTile; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
                }
                if (on && gl == 0) {
                    long long bd = W.bd[j];
                    int a = W.assign[j];
#pragma unroll
                    for (int q = 0; q < kKmTile; ++q)
                        if (c[q] >= 0) {
                            const long long d = (long long)acc[q];
                            if (d < bd || (d == bd && c[q] < a)) { bd = d; a = c[q]; }
                        }
                    W.bd[j] = bd;
                    W.assign[j] = a;
                }
            }
        }
        __syncthreads();
    }

    // ---------------------------------------------- k-means++ initialisation (_initPlusPlus)
    template <class Cluster>
    __device__ void init(Cluster& cl) {
        const int np = S.np, nb = S.nb, k = S.k, tid = threadIdx.x;
        const int lane = tid & 31, wid = tid >> 5;
        for (int j = p0 + tid; j < p1; j += kKmThreads) W.cdist[j] = 0.0;
        if (tid < kKmRows) M.row_of[tid] = -1;
        if (rank == 0 && tid == 0) W.cent[0] = 0;
        if (tid == 0) M.p[1] = 1.0;
        __syncthreads();
        int lc = 0, next = 0;
        const int nwarps = min(kKmThreads / 32, (p1 - p0 + 31) / 32);
        for (int i = 1; i < k; ++i) {
            int slot = -1;
#pragma unroll
            for (int r = 0; r < kKmRows; ++r)
                if (M.row_of[r] == lc) slot = r;
            const bool fresh = slot < 0;
            if (fresh) {
                slot = next;
                next = next + 1 == kKmRows ? 0 : next + 1;
            }
            double* const row = W.rows + (int64_t)slot * np;
            unsigned long long bv = 0ull;
            int bj = 0x7fffffff;
            const double p = wid < nwarps ? M.p[i & 1] : 0.0;
            const double q = 1.0 - p;
            for (int j = p0 + tid; j < p1; j += kKmThreads) {
                double d;
                if (fresh) {
                    Acc a = 0;
#pragma unroll 4
                    for (int b = 0; b < nb; ++b)
                        a += term(__ldg(X + (int64_t)b * np + j), __ldg(X + (int64_t)b * np + lc));
                    d = (double)a;
                    row[j] = d;
                } else {
                    d = row[j];
                }
                const double c = __dadd_rn(__dmul_rn(W.cdist[j], q), __dmul_rn(d, p));
                W.cdist[j] = c;
                km_max(bv, bj, (unsigned long long)__double_as_longlong(c), j);
            }
            // the block's candidate to every block of the cluster, then the same choice in all
            if (wid < nwarps) {
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long v2 = __shfl_xor_sync(0xffffffffu, bv, o);
                    const int j2 = __shfl_xor_sync(0xffffffffu, bj, o);
                    km_max(bv, bj, v2, j2);
                }
                if (lane == 0) { M.sv[wid] = bv; M.sj[wid] = bj; }
            }
            __syncthreads();
            if (fresh && tid == 0) M.row_of[slot] = lc;
            if (tid == kKmThreads - 1) M.p[(i + 1) & 1] = 1.0 / (double)(i + 1);  // while the others choose
            if (wid == 0) {
                bv = lane < nwarps ? M.sv[lane] : 0ull;
                bj = lane < nwarps ? M.sj[lane] : 0x7fffffff;
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long v2 = __shfl_xor_sync(0xffffffffu, bv, o);
                    const int j2 = __shfl_xor_sync(0xffffffffu, bj, o);
                    km_max(bv, bj, v2, j2);
                }
                if (lane < nblk) {
                    KMShared* R = cl.map_shared_rank(&M, lane);
                    R->mv[i & 1][rank] = bv;
                    R->mj[i & 1][rank] = bj;
                }
            }
            cl.sync();
            bv = 0ull;
            bj = 0x7fffffff;
            for (int r = 0; r < nblk; ++r) km_max(bv, bj, M.mv[i & 1][r], M.mj[i & 1][r]);
            lc = bj;
            if (rank == 0 && tid == 0) W.cent[i] = lc;
        }
    }

    // Lists of the centroids that are the first on their point: moved ones, and the others (in no
    // order; the comparisons carry the centroid's number).  One block.
    __device__ void lists() {
        const int k = S.k, tid = threadIdx.x;
        for (int c = tid; c < k; c += kKmThreads) W.first[__ldcg(W.cent + c)] = 0x7fffffff;
        if (tid == 0) { W.ctl->nmoved = 0; W.ctl->nkept = 0; }
        __syncthreads();
        for (int c = tid; c < k; c += kKmThreads) atomicMin(W.first + __ldcg(W.cent + c), c);
        __syncthreads();
        for (int c = tid; c < k; c += kKmThreads) {
            const int at = __ldcg(W.cent + c);
            if (__ldcg(W.first + at) != c) continue;
            if (__ldcg(W.moved + c)) W.mlist[atomicAdd(&W.ctl->nmoved, 1)] = make_int2(c, at);
            else W.ulist[atomicAdd(&W.ctl->nkept, 1)] = make_int2(c, at);
        }
    }

    template <class Cluster>
    __device__ void lloyd(Cluster& cl, const KMParams& P) {
        const int np = S.np, nb = S.nb, k = S.k, tid = threadIdx.x;
        const int lane = tid & 31, wid = tid >> 5;
        const int gtid = rank * kKmThreads + tid, gth = nblk * kKmThreads;
        const int64_t kb = (int64_t)k * nb;
        for (int64_t e = gtid; e < 2 * kb; e += gth) W.sum[e] = 0;
        for (int c = gtid; c < k; c += gth) {
            W.cnt[c] = 0;
            W.dirty[c] = 0;
            W.moved[c] = 1;
        }
        for (int j = p0 + tid; j < p1; j += kKmThreads) W.assign[j] = -1;
        cl.sync();
        if (rank == 0) lists();
        if (gtid == 0) W.ctl->ndirty = W.ctl->ncand = 0;
        cl.sync();
        int iter = 0;
        for (;;) {
            ++iter;
            // ---- every point's nearest centroid: against the moved ones; from the start when its own moved
            if (tid == 0) M.nr = 0;
            __syncthreads();
            int32_t* const again = reinterpret_cast<int32_t*>(W.rows) + p0;  // (the rows are done with)
            for (int j = p0 + tid; j < p1; j += kKmThreads) {
                const int a = W.assign[j];
                W.was[j] = a;
                if (a < 0 || __ldcg(W.moved + a)) {
                    W.bd[j] = 0x7fffffffffffffffll;
                    W.assign[j] = 0x7fffffff;
                    again[atomicAdd(&M.nr, 1)] = j;
                }
            }
            __syncthreads();
            nearest(W.mlist, __ldcg(&W.ctl->nmoved), nullptr, p1 - p0);
            nearest(W.ulist, __ldcg(&W.ctl->nkept), again, M.nr);
            // ---- counts and exact sums follow the changes, a warp per changed point
            for (int j = p0 + wid; j < p1; j += kKmThreads / 32) {
                const int was = W.was[j], now = W.assign[j];
                if (was == now) continue;
                for (int h = 0; h < 2; ++h) {
                    const int c = h ? now : was;
                    if (c < 0) continue;
                    if (lane == 0) {
                        atomicAdd(W.cnt + c, h ? 1 : -1);
                        if (atomicExch(W.dirty + c, 1) == 0) {
                            W.dlist[atomicAdd(&W.ctl->ndirty, 1)] = c;
                            W.best[c] = W.rbest[c] = ~0ull;
                            W.bestj[c] = 0x7fffffff;
                            W.ncand[c] = 0;
                        }
                    }
                    for (int i = lane; i < nb; i += 32) {
                        const int2 x = __ldg(X + (int64_t)i * np + j);
                        const long long l = h ? x.x : -(long long)x.x, m = h ? x.y : -(long long)x.y;
                        atomicAdd((unsigned long long*)(W.sum + (int64_t)c * nb + i), (unsigned long long)l);
                        atomicAdd((unsigned long long*)(W.sum + kb + (int64_t)c * nb + i), (unsigned long long)m);
                    }
                }
            }
            cl.sync();
            // ---- nearest member to the mean, of the centroids whose members changed: by the exact
            // integer distances first
            const int nd = __ldcg(&W.ctl->ndirty);
            for (int j = p0 + wid; j < p1; j += kKmThreads / 32) {
                const int c = W.assign[j];
                if (!__ldcg(W.dirty + c)) continue;
                const int n = __ldcg(W.cnt + c);
                if (n > exact_n) continue;
                const long long* sl = W.sum + (int64_t)c * nb;
                unsigned long long t = 0;
                for (int i = lane; i < nb; i += 32) {
                    const int2 x = __ldg(X + (int64_t)i * np + j);
                    const int a = (int)(__ldcg(sl + i) - (long long)n * x.x), b = (int)(__ldcg(sl + kb + i) - (long long)n * x.y);
                    t += (unsigned long long)((long long)a * a) + (unsigned long long)((long long)b * b);
                }
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) {
                    W.key[j] = t;
                    atomicMin(W.best + c, t);
                }
            }
            cl.sync();
            for (int j = p0 + tid; j < p1; j += kKmThreads) {
                const int c = W.assign[j];
                if (!__ldcg(W.dirty + c)) continue;
                const int n = __ldcg(W.cnt + c);
                if (!candidate(j, c, n)) continue;
                atomicAdd(W.ncand + c, 1);
                atomicMin(W.bestj + c, j);
            }
            cl.sync();
            // ---- several within the rounding: the reference's arithmetic decides, a warp per candidate
            for (int j = p0 + tid; j < p1; j += kKmThreads) {
                const int c = W.assign[j];
                if (!__ldcg(W.dirty + c) || __ldcg(W.ncand + c) < 2) continue;
                const int n = __ldcg(W.cnt + c);
                if (!candidate(j, c, n)) continue;
                W.cand[atomicAdd(&W.ctl->ncand, 1)] = j;
            }
            cl.sync();
            const int nc = __ldcg(&W.ctl->ncand);
            if (nc > 0) {
                for (int e = rank * (kKmThreads / 32) + wid; e < nc; e += nblk * (kKmThreads / 32)) {
                    const int j = __ldcg(W.cand + e), c = __ldcg(W.assign + j);
                    const double n = (double)__ldcg(W.cnt + c);
                    const long long* sl = W.sum + (int64_t)c * nb;
                    double s = 0.0;
                    for (int i0 = 0; i0 < nb; i0 += 32) {
                        double a = 0.0, b = 0.0;
                        if (i0 + lane < nb) {
                            const int2 x = __ldg(X + (int64_t)(i0 + lane) * np + j);
                            const double d = __dsub_rn(__ddiv_rn((double)__ldcg(sl + i0 + lane), n), (double)x.x);
                            const double f = __dsub_rn(__ddiv_rn((double)__ldcg(sl + kb + i0 + lane), n), (double)x.y);
                            a = __dmul_rn(d, d);
                            b = __dmul_rn(f, f);
                        }
                        const int m = min(32, nb - i0);
                        for (int i = 0; i < m; ++i) {
                            s = __dadd_rn(s, __shfl_sync(0xffffffffu, a, i));
                            s = __dadd_rn(s, __shfl_sync(0xffffffffu, b, i));
                        }
                    }
                    if (lane == 0) {  // s >= 0: bits order as values
                        W.key[j] = (unsigned long long)__double_as_longlong(s);
                        atomicMin(W.rbest + c, (unsigned long long)__double_as_longlong(s));
                    }
                }
                for (int q = gtid; q < nd; q += gth) {
                    const int c = __ldcg(W.dlist + q);
                    if (__ldcg(W.ncand + c) >= 2) W.bestj[c] = 0x7fffffff;
                }
                cl.sync();
                for (int e = gtid; e < nc; e += gth) {
                    const int j = __ldcg(W.cand + e), c = __ldcg(W.assign + j);
                    if (__ldcg(W.key + j) == __ldcg(W.rbest + c)) atomicMin(W.bestj + c, j);
                }
                cl.sync();
            }
            // ---- the largest move (_centroidVariance), the next step's centroids and lists
            if (rank == 0) {
                if (tid == 0) M.var = 0.0;
                __syncthreads();
                double var = 0.0;
                for (int q = wid; q < nd; q += kKmThreads / 32) {
                    const int c = __ldcg(W.dlist + q);
                    const int from = __ldcg(W.cent + c), to = __ldcg(W.cnt + c) ? __ldcg(W.bestj + c) : from;
                    long long d = 0;
                    if (to != from)
                        for (int i = lane; i < nb; i += 32)
                            d += (long long)term(__ldg(X + (int64_t)i * np + from), __ldg(X + (int64_t)i * np + to));
                    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                    var = fmax(var, (double)d);
                    if (lane == 0) W.ncent[c] = to;
                }
                if (lane == 0) M.sv[wid] = (unsigned long long)__double_as_longlong(var);
                __syncthreads();
                if (tid == 0) {
                    for (int w = 0; w < kKmThreads / 32; ++w) M.var = fmax(M.var, __longlong_as_double((long long)M.sv[w]));
                    W.ctl->ncand = 0;
                    W.ctl->go = M.var > P.min_variance && iter <= P.max_iter;
                }
                __syncthreads();
                if (M.var > P.min_variance && iter <= P.max_iter) {
                    for (int c = tid; c < k; c += kKmThreads) W.moved[c] = 0;
                    __syncthreads();
                    for (int q = tid; q < nd; q += kKmThreads) {
                        const int c = __ldcg(W.dlist + q);
                        const int to = __ldcg(W.ncent + c);
                        W.moved[c] = to != __ldcg(W.cent + c);
                        W.cent[c] = to;
                        W.dirty[c] = 0;
                    }
                    __syncthreads();
                    lists();
                    if (tid == 0) W.ctl->ndirty = 0;
                }
            }
            cl.sync();
            if (!__ldcg(&W.ctl->go)) break;
        }
        // weights of the last assignment; the centroids of that assignment are the result
        for (int c = gtid; c < k; c += gth) W.wsum[c] = 0;
        cl.sync();
        for (int j = p0 + tid; j < p1; j += kKmThreads) atomicAdd(W.wsum + W.assign[j], __ldg(P.wt + S.p_off + j));
        cl.sync();
        for (int c = gtid; c < k; c += gth) {
            P.out_idx[S.out_off + c] = __ldcg(W.cent + c);
            P.out_w[S.out_off + c] = __ldcg(W.wsum + c);
        }
    }
};

// One cluster per set (blocks of a cluster consecutive).
__global__ void __launch_bounds__(kKmThreads) kmeans_kernel(KMParams P) {
    __shared__ KMShared M;
    auto cl = cooperative_groups::this_cluster();
    const int nblk = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const KMSet S = P.sets[blockIdx.x / nblk];
    const KMMeta meta = P.meta[S.id];
    const double range = km_range(S.nb, meta.lmax, meta.cmax);
    if (meta.bad || range >= 9007199254740992.0) return;  // refused by the host (the whole cluster)
    const double most = fmax((double)meta.lmax, (double)meta.cmax);
    const KMWork W = km_carve(P.ws + S.ws_off, S.np, S.nb, S.k);
    const int part = (S.np + nblk - 1) / nblk;
    const int p0 = min(rank * part, S.np), p1 = min(p0 + part, S.np);
    if (range < 4294967296.0) {
        KMeans<true> K{S, P.X + S.x_off, W, M, rank, nblk, p0, p1};
        K.bounds(range, most);
        K.init(cl);
        cl.sync();
        K.lloyd(cl, P);
    } else {
        KMeans<false> K{S, P.X + S.x_off, W, M, rank, nblk, p0, p1};
        K.bounds(range, most);
        K.init(cl);
        cl.sync();
        K.lloyd(cl, P);
    }
    cl.sync();  // no block leaves while another may still write to its shared memory
}

}  // namespace fbc
