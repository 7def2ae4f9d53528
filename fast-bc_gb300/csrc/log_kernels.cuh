// Batched schedule, segments too large for the team kernel (team_kernels.cuh): one source per block,
// per-source state in a global-memory slot, blocks pulling units from a shared counter.  The same two
// passes over the rounds of a pop log as the team kernel (the last pops, equal distances popped
// again, are a topological order of the shortest-path DAG), laid out for what bounds large graphs: the
// sectors of DRAM and L2 that a source touches, for the sources in flight share them.
//   * distances: 4 bytes a vertex (dist | stamp) relaxed by one atomicMin each, and 4 for the log place
//     of its last pop; the log itself and the far pile are written and read in order.  Relaxations
//     that cannot lower a word are dropped after a load;
//   * path counts: the words again, 4 bytes a vertex of counts added without a return value; count and
//     tight-edge mask of a vertex go into its log entry, in order;
//   * dependencies: the coefficient c = (1 + delta) / sigma, 8 bytes a vertex, read by predecessors;
//     delta goes straight into BC (in the segment's order where one segment runs), leaves' not at all.
//   * rows as 16-byte quads of (destination:24 | weight:8): one load for up to four edges, no row
//     offsets; the fourth place of a longer row links to its next quad (an entry of weight 0).
// What bounds it is the chain of dependent loads of a round against the sources that share the L2: the
// passes over fixed data (counts, dependencies) load the next round's entries and rows a round ahead, and
// the number of sources per SM follows the size (log_form in fbc_gpu.cu).
// Against the frontier kernel (frontier_kernels.cuh), which keeps 8 + 16 bytes a vertex with an in-edge
// counter, counts and pushes per Kahn level, device time, FP32C, one GB300: 280 pivots of the 2048x2048
// grid 235.7 -> 180 ms; 1,309 pivots of the 256x256 grid 18.9 -> 14.0; the 16,384 sources of the 128x128
// grid 47.3 -> 34.0; communities of 4.5K to 20K vertices (50K sources, FP64) 107 -> 82.
// A source whose counts reach 2^24, whose distances outgrow a word, or of too many narrow rounds stops before its
// dependencies and is done by the kernels with wider fields.
#pragma once
#include <cooperative_groups.h>
#include "frontier_kernels.cuh"
#include "team_kernels.cuh"

namespace fbc {

constexpr uint32_t kQuadNone = 0x00ffffffu;  // an empty place (weight 0); other entries of weight 0 are links
constexpr int kLogRow = 16;                  // longest row (mask bits)
constexpr int kLogStamp = 10;                // stamp bits where the segment's bound does not leave more

// Quads of segments, one grid column per segment; `extra` counts the continuation quads taken.
struct LogQuads {
    uint4* quad;
    int32_t seg, pad;
};
__global__ void log_quads_kernel(const Seg* __restrict__ segs, const LogQuads* __restrict__ ts, int32_t* extra) {
    const LogQuads t = ts[blockIdx.x];
    const Seg sg = segs[t.seg];
    for (int v = blockIdx.y * blockDim.x + threadIdx.x; v < sg.n; v += gridDim.y * blockDim.x) {
        int e = sg.rp[v];
        const int e1 = sg.rp[v + 1];
        int at = v;
        for (;;) {
            const int left = e1 - e;
            const int k = left > 4 ? 3 : left;
            uint32_t r[4] = {kQuadNone, kQuadNone, kQuadNone, kQuadNone};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < k) {
                    const int2 a = __ldg(sg.adj + e + i);
                    r[i] = (uint32_t)a.x | ((uint32_t)a.y << 24);
                }
            e += k;
            int next = -1;
            if (left > 4) {
                next = sg.n + atomicAdd(extra + blockIdx.x, 1);
                r[3] = (uint32_t)next;
            }
            t.quad[at] = make_uint4(r[0], r[1], r[2], r[3]);
            if (next < 0) break;
            at = next;
        }
    }
}

__host__ __device__ inline int64_t log_rounds(int64_t cap) { return cap / 4 + 64; }  // kept rounds

// Slot of one source for segments of up to cap vertices.
template <class Prec>
struct LState {
    uint32_t* word;
    uint32_t* sig;            // last pop in the distance pass, then the path count
    uint32_t* log;            // 2 * cap pops
    uint2* ent;               // of each pop: (vertex | low mask bits << 24, path count)
    typename Prec::D* coef;
    uint8_t* mhi;             // mask bits of the ninth to sixteenth edge
    int* rnd;                 // first log place of each round
    uint32_t *far0, *far1;
};
template <class Prec>
__host__ __device__ inline int64_t lstate_bytes(int64_t cap) {
    auto al = [](int64_t x) { return (x + 255) & ~int64_t(255); };
    return 2 * al(cap * 4) + al(2 * cap * 4) + al(2 * cap * 8) + al(cap * (int64_t)sizeof(typename Prec::D)) + al(cap) +
           al((log_rounds(cap) + 2) * 4) + 2 * al(fqcap(cap) * 4);
}
template <class Prec>
__device__ inline LState<Prec> lstate_carve(char* p, int64_t cap) {
    auto al = [](int64_t x) { return (x + 255) & ~int64_t(255); };
    LState<Prec> s;
    auto take = [&](int64_t b) {
        char* q = p;
        p += al(b);
        return q;
    };
    s.word = (uint32_t*)take(cap * 4);
    s.sig = (uint32_t*)take(cap * 4);
    s.log = (uint32_t*)take(2 * cap * 4);
    s.ent = (uint2*)take(2 * cap * 8);
    s.coef = (typename Prec::D*)take(cap * (int64_t)sizeof(typename Prec::D));
    s.mhi = (uint8_t*)take(cap);
    s.rnd = (int*)take((log_rounds(cap) + 2) * 4);
    s.far0 = (uint32_t*)take(fqcap(cap) * 4);
    s.far1 = (uint32_t*)take(fqcap(cap) * 4);
    return s;
}

struct LogCtl {
    int near[3], far[3];  // pushes of a step, three in rotation
    int dmin, unit, bad;
};

__device__ __forceinline__ uint32_t gatom_min_if(bool c, uint32_t* a, uint32_t x) {  // 0 where not done
    uint32_t old;
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %3, 0;\n mov.u32 %0, 0;\n @q atom.global.min.u32 %0, [%1], %2;\n}"
                 : "=r"(old) : "l"(a), "r"(x), "r"((uint32_t)c) : "memory");
    return old;
}
__device__ __forceinline__ void gred_add_if(bool c, uint32_t* a, uint32_t x) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q red.global.add.u32 [%0], %1;\n}" ::"l"(a), "r"(x),
                 "r"((uint32_t)c) : "memory");
}

// Append up to four values a lane; whole warps; places from a counter in shared memory.  A push past
// the capacity is dropped (the caller sees the count).
__device__ __forceinline__ void lpush(const bool (&want)[4], const uint32_t (&x)[4], uint32_t* q, int at, int cap, int* cnt) {
    unsigned m[4];
    int tot = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        m[t] = __ballot_sync(kFull, want[t]);
        tot += __popc(m[t]);
    }
    if (tot == 0) return;
    const int lane = threadIdx.x & 31;
    int b = 0;
    if (lane == 0) b = atomicAdd(cnt, tot);
    b = at + __shfl_sync(kFull, b, 0);
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int p = b + __popc(m[t] & below);
        if (want[t] && p < cap) q[p] = x[t];
        b += __popc(m[t]);
    }
}

// A load of state that other threads of the source wrote: those of a cluster's other blocks are not in
// this block's L1.
template <bool kCluster, class T>
__device__ __forceinline__ T lload(const T* p) {
    if constexpr (kCluster) return __ldcg(p);
    else return *p;
}

// Narrow sources: those of more rounds to come than are kept stop early, and so do, where there are several waves
// of units on a segment whose sources the frontier kernel's blocks share by four, those of less than twenty pops a
// round; with less than 27 the segment's other units start there.  All sources, this kernel / that one, ms: 6 x
// 2,000 vertices 125 / 92, 12 x 1,500 164 / 136, 20 x 1,000 138 / 121, 32 x 600 90 / 86, 40 x 500 82 / 82, 64 x 300
// 60 / 68 (a square's corner has some fifty pops a round).
template <int kThreads>
__device__ __forceinline__ bool log_shared(const KParams& P, int n) {
    return P.gave && n <= 32768 && P.nunits > 4 * ((int64_t)gridDim.x * (blockDim.x / kThreads));
}

// One source by a team of kThreads threads (bar: its named barrier), or by the `threads` threads of a
// cluster of blocks, whose control words lie in the first block's shared memory.  tid numbers the team's
// threads, whole warps together.
template <class Prec, int kThreads, bool kCluster = false>
__device__ __forceinline__ void log_unit(const KParams& P, const Seg& sg, const Unit& u, const LState<Prec>& S, LogCtl& C,
                                         int64_t cap, int tid, int bar, int threads = kThreads) {
    const int nth = kCluster ? threads : kThreads;
    const int n = sg.n, lane = tid & 31;
    auto sync = [bar]() {
        if constexpr (kCluster)
            asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
        else
            asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kThreads) : "memory");
    };
    const uint4* __restrict__ quads = sg.quad;
    const int sb = sg.stamp_bits;
    const uint32_t smask = (1u << sb) - 1u;
    const int dinf = (int)(kNoEdge >> sb);
    const int src = u.src;
    const int logcap = (int)min((int64_t)2 * n, 2 * cap), farcap = (int)fqcap(cap), rndcap = (int)log_rounds(n);
    const uint4 none = make_uint4(kQuadNone, kQuadNone, kQuadNone, kQuadNone);
    auto linked = [](const uint4& q) { return (q.w >> 24) == 0u && q.w != kQuadNone; };
    int delta = sg.delta > 0 ? sg.delta : 1;
    int bad = 0, total = 0, nr = 0;

    // ---------------------------------------------------------------- distances
    for (;;) {
        for (int i = tid; i < n; i += nth) {
            S.word[i] = kNoEdge;
            S.sig[i] = kNoEdge;
        }
        if (tid == 0) {
            C.near[0] = C.far[0] = 0;
            C.bad = 0;
        }
        sync();
        if (tid == 0) {
            S.word[src] = 0u;
            S.log[0] = (uint32_t)src;
        }
        sync();
        int s = 0, e = 1, nfar = 0, fs = 0, c3 = 0;
        int T = min(delta, dinf);
        uint32_t stamp = smask - 1u, fst = smask - 1u;
        const int64_t capl = (int64_t)P.iter_mult * ((int64_t)n + 2);
        int64_t steps = 0;
        int flag = 0;
        bool full = false;
        nr = 0;
        for (;;) {
            if (stamp < 4u) {  // out of stamps: the far pile's vertices get the first one again, all others none
                for (int i = tid; i < n; i += nth) S.word[i] = __ldcg(S.word + i) | smask;
                sync();
                for (int i = tid; i < nfar; i += nth) {
                    const uint32_t v = lload<kCluster>((fs ? S.far1 : S.far0) + i);
                    S.word[v] = __ldcg(S.word + v) ^ 1u;  // listed once each
                }
                stamp = fst = smask - 1u;
                sync();
            }
            const int cs = c3;
            c3 = c3 == 2 ? 0 : c3 + 1;
            if (tid == 0) {  // the next step's (last read two barriers ago)
                C.near[c3] = 0;
                C.far[c3] = 0;
                C.dmin = kInf;
            }
            if (++steps > capl) { bad = kErrIter; break; }
            if (s < e) {
                if (nr == rndcap) { bad = kErrNarrow; break; }
                const uint32_t nst = --stamp;
                if (tid == 0) S.rnd[nr] = s;
                ++nr;
                uint32_t* const qf = fs ? S.far1 : S.far0;
                for (int b = s + (tid & ~31); b < e; b += nth) {
                    const int i = b + lane;
                    const bool act = i < e;
                    const uint32_t v = lload<kCluster>(S.log + (act ? i : s));
                    uint4 q = __ldg(quads + v);
                    const int dv = (int)(__ldcg(S.word + v) >> sb);  // may have dropped since the push
                    // only the last pop stays (an exchange: loading and storing the place separately makes
                    // the kernel three to four times slower: 16,384 vertices 34 -> 123 ms)
                    const uint32_t before = act ? atomicExch(S.sig + v, (uint32_t)i) : kNoEdge;
                    if (before != kNoEdge) S.log[before] = kNoEdge;
                    if (!act) q = none;
                    for (;;) {
                        uint32_t x[4], cur[4], key[4];
                        bool pn[4], pf[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            const uint32_t a = quad_at(q, t);
                            x[t] = a & 0xffffffu;
                            cur[t] = (a >> 24) ? __ldcg(S.word + x[t]) : 0u;
                        }
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            const uint32_t w = quad_at(q, t) >> 24;
                            const int nd = dv + (int)w;
                            const bool near = nd < T;
                            const uint32_t st = near ? nst : fst;
                            key[t] = ((uint32_t)nd << sb) | st;
                            const bool go = w != 0u && nd < dinf && key[t] < cur[t];
                            if (w != 0u && nd >= dinf) flag = kErrNarrow;  // distances outgrow the word
                            const uint32_t old = gatom_min_if(go, S.word + x[t], key[t]);
                            const bool up = key[t] < old && ((old ^ st) & smask) != 0u;
                            pn[t] = up && near;
                            pf[t] = up && !near;
                        }
                        // a queued vertex's row on its way to the L2 (3% on every size; to the L1: nothing)
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            if (pn[t] || pf[t]) asm volatile("prefetch.global.L2 [%0];" ::"l"(quads + x[t]));
                        lpush(pn, x, S.log, e, logcap, C.near + cs);
                        lpush(pf, x, qf, nfar, farcap, C.far + cs);
                        const bool link = linked(q);
                        if (!__any_sync(kFull, link)) break;
                        const uint4 q2 = __ldg(quads + (link ? q.w : v));
                        q = link ? q2 : none;
                    }
                }
                sync();
                s = e;
                e += *(volatile int*)&C.near[cs];
                nfar += *(volatile int*)&C.far[cs];
            } else {
                if (nfar == 0) break;
                if (many_rounds(n, nr) && e < (log_shared<kThreads>(P, n) ? 20 : 3) * nr) { bad = kErrNarrow; break; }
                // the threshold moves on to the bucket of the closest live far vertex
                sync();  // (C.dmin is set)
                const uint32_t* const qo = fs ? S.far1 : S.far0;
                uint32_t* const qf = fs ? S.far0 : S.far1;
                int dmin = kInf;
                for (int i = tid; i < nfar; i += nth) {
                    const int d = (int)(__ldcg(S.word + lload<kCluster>(qo + i)) >> sb);
                    if (d >= T) dmin = min(dmin, d);
                }
                dmin = __reduce_min_sync(kFull, dmin);
                if (lane == 0 && dmin != kInf) atomicMin(&C.dmin, dmin);
                sync();
                dmin = *(volatile int*)&C.dmin;
                if (dmin == kInf) break;
                const int Told = T;
                const int64_t tn = ((int64_t)dmin / delta + 1) * (int64_t)delta;
                T = tn > (int64_t)dinf ? dinf : (int)tn;
                const uint32_t nst = --stamp;
                fst = --stamp;
                for (int b = tid & ~31; b < nfar; b += nth) {
                    const int i = b + lane;
                    const uint32_t x[4] = {i < nfar ? lload<kCluster>(qo + i) : 0u, 0u, 0u, 0u};
                    const int d = i < nfar ? (int)(__ldcg(S.word + x[0]) >> sb) : -1;
                    const bool live = i < nfar && d >= Told;  // the far pile holds a vertex once per generation
                    const bool pn[4] = {live && d < T, false, false, false}, pf[4] = {live && d >= T, false, false, false};
                    if (live) S.word[x[0]] = ((uint32_t)d << sb) | (d < T ? nst : fst);
                    lpush(pn, x, S.log, e, logcap, C.near + cs);
                    lpush(pf, x, qf, 0, farcap, C.far + cs);
                }
                sync();
                e += *(volatile int*)&C.near[cs];
                nfar = *(volatile int*)&C.far[cs];
                fs ^= 1;
            }
            if (nfar > farcap) { bad = kErrNarrow; break; }
            if (e > logcap) { full = true; break; }
        }
        sync();
        if (flag) C.bad = flag;
        sync();
        if (!bad) bad = *(volatile int*)&C.bad;
        total = e;
        if (!full || bad) break;
        // more than two pops a vertex: again with narrower buckets (width 1 pops every vertex once)
        delta = max(1, delta >> 2);
        sync();
    }
    if (tid == 0 && !bad && many_rounds(n, 2 * nr) && total < 27 * nr && log_shared<kThreads>(P, n)) count_narrow(P, u.seg);

    if (!bad) {
        // --------------------------------------------------------------- path counts, in pop order
        if (u.bout >= 0)
            for (int j = tid; j < sg.nb; j += nth) {
                const int d = (int)(__ldcg(S.word + sg.border[j]) >> sb);
                P.bdist[u.bout + j] = d != dinf ? (double)d : 0.0;
            }
        if (tid == 0) S.rnd[nr] = total;
        for (int i = tid; i < n; i += nth) S.sig[i] = 0u;
        sync();
        if (tid == 0) S.sig[src] = 1u;
        sync();
        uint32_t high = 0u;
        int s = 0, e = lload<kCluster>(S.rnd + 1);
        // what a lane needs of its entry but the count: fixed by now, so the next round's is loaded
        // while this one ends (only the counts wait for the barrier)
        struct Pre {
            uint32_t v;
            uint4 q;
            uint32_t wv, wx[4];
        };
        auto load = [&](Pre& p, int i, int end) {
            const uint32_t v = lload<kCluster>(S.log + min(i, end - 1));
            const bool on = i < end && v != kNoEdge;
            p.v = on ? v : kNoEdge;
            p.q = on ? __ldg(quads + v) : none;
            p.wv = on ? lload<kCluster>(S.word + v) : 0u;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t a = quad_at(p.q, t);
                p.wx[t] = (a >> 24) ? lload<kCluster>(S.word + (a & 0xffffffu)) : kNoEdge;  // (final: the L1 may hold it)
            }
        };
        Pre nx;
        load(nx, s + tid, e);
        for (int r = 0; r < nr; ++r) {
            const int e2 = lload<kCluster>(S.rnd + min(r + 2, nr));
            for (int b = s + (tid & ~31); b < e; b += nth) {
                const int i = b + lane;
                if (b >= s + nth) load(nx, i, e);  // (a round wider than the team)
                const uint32_t v = nx.v;
                const bool on = v != kNoEdge;
                const int dv = (int)(nx.wv >> sb);
                const uint32_t sv = on ? __ldcg(S.sig + v) : 1u;
                high |= sv;
                unsigned mk = 0u;
                for (int p = 0;; p += 3) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t a = quad_at(nx.q, t);
                        const bool tight = (a >> 24) && dv + (int)(a >> 24) == (int)(nx.wx[t] >> sb);
                        if (tight) mk |= 1u << (p + t);
                        gred_add_if(tight, S.sig + (a & 0xffffffu), sv);
                    }
                    const bool link = linked(nx.q);
                    if (!__any_sync(kFull, link)) break;
                    nx.q = link ? __ldg(quads + nx.q.w) : none;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t a = quad_at(nx.q, t);
                        nx.wx[t] = (a >> 24) ? lload<kCluster>(S.word + (a & 0xffffffu)) : kNoEdge;
                    }
                }
                if (i < e) S.ent[i] = on ? make_uint2(v | (mk << 24), sv) : make_uint2(kNoEdge, 1u);
                if (on && sg.wide) S.mhi[v] = (uint8_t)(mk >> 8);
            }
            s = e;
            e = e2;
            if (s < e) load(nx, s + tid, e);
            sync();
        }
        // every count below 2^24 (so no sum over up to 255 in-edges wrapped)
        if (__any_sync(kFull, (high >> 24) != 0u)) C.bad = kErrNarrow;
        sync();
        bad = *(volatile int*)&C.bad;
        if (!bad && u.bout >= 0)
            for (int j = tid; j < sg.nb; j += nth) P.bsig[u.bout + j] = __ldcg(S.sig + sg.border[j]);
        sync();
    }
    if (!bad) {
        // --------------------------------------------------------- dependency
        const double card = u.card;
        double* const bc = P.bc_seg ? P.bc_seg : P.bc + sg.out_base;
        const int32_t* const gid = P.bc_seg ? nullptr : sg.gid;
        int hi = total, lo = lload<kCluster>(S.rnd + nr - 1);
        struct Pre {  // an entry and its row, loaded a round ahead
            uint2 en;
            uint32_t m;
            uint4 q;
        };
        auto load = [&](Pre& p, int i, int end) {
            p.en = i < end ? lload<kCluster>(S.ent + i) : make_uint2(kNoEdge, 1u);
            const bool on = p.en.x != kNoEdge;
            const uint32_t v = p.en.x & 0xffffffu;
            p.m = on ? p.en.x >> 24 : 0u;
            if (on && sg.wide) p.m |= (uint32_t)lload<kCluster>(S.mhi + v) << 8;
            p.q = p.m ? __ldg(quads + v) : none;
        };
        Pre nx;
        load(nx, lo + tid, hi);
        for (int r = nr - 1; r >= 0; --r) {
            const int lo2 = lload<kCluster>(S.rnd + max(r - 1, 0));
            for (int b = lo + (tid & ~31); b < hi; b += nth) {
                const int i = b + lane;
                if (b >= lo + nth) load(nx, i, hi);
                const bool on = nx.en.x != kNoEdge;
                const uint32_t v = nx.en.x & 0xffffffu;
                const uint32_t sv = nx.en.y;
                uint32_t m = nx.m;
                const bool inner = m != 0u && v != (uint32_t)src;
                typename Prec::Acc acc = Prec::zero();
                if (__any_sync(kFull, m)) {
                    for (;;) {  // in row order
                        const bool link = linked(nx.q) && (m >> 3) != 0u;
                        typename Prec::D c[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            const bool tight = ((m >> t) & 1u) && !(t == 3 && link);
                            c[t] = tight ? lload<kCluster>(S.coef + (quad_at(nx.q, t) & 0xffffffu)) : Prec::store(Prec::zero());
                        }
                        Prec::add_coefs(acc, c[0], c[1], c[2], c[3]);
                        if (!__any_sync(kFull, link)) break;
                        nx.q = link ? __ldg(quads + nx.q.w) : none;
                        m = link ? m >> 3 : 0u;
                    }
                }
                typename Prec::D c;
                if (!__any_sync(kFull, sv != 1u)) {
                    c = Prec::coef1(acc);
                } else {
                    acc = Prec::times(acc, sv);
                    c = Prec::coef(acc, sv);
                }
                if (on) S.coef[v] = c;
                if (inner) {  // (kept by vertex and added in one sweep at the end: a tenth slower on all sizes)
                    const double d = Prec::value(acc);
                    atomicAdd(bc + (gid ? __ldg(gid + v) : (int)v), card == 1.0 ? d : card * d);
                }
            }
            hi = lo;
            lo = lo2;
            if (r > 0) load(nx, lo + tid, hi);
            sync();
        }
    }
    if (tid == 0) count_unit(P, u.seg, bad == kErrNarrow);
    if (bad && tid == 0) {
        if (bad == kErrNarrow) request_retry(P, u, kErrNarrow);  // recomputed with wider fields
        else atomicOr(P.err, bad);
    }
    sync();
}

// The next unit that is worth starting here; the others go back (one thread).
__device__ __forceinline__ void log_pick(const KParams& P, LogCtl& C) {
    for (;;) {
        const int64_t ui = (int64_t)atomicAdd(P.next_unit, 1ull);
        C.unit = (int)ui;
        if (ui >= P.nunits) return;
        const Unit u = P.units[ui];
        if (!gave_up(P, u.seg)) return;
        request_retry(P, u, kErrNarrow);
    }
}

// kTeams teams of kThreads threads in a block, one source each.
template <class Prec, int kThreads, int kTeams, int kPerSM>
__global__ void __launch_bounds__(kThreads * kTeams, kPerSM) log_kernel(KParams P) {
    __shared__ LogCtl ctl[kTeams];
    const int team = threadIdx.x / kThreads, tid = threadIdx.x % kThreads;
    LogCtl& C = ctl[team];
    const LState<Prec> S = lstate_carve<Prec>(P.ws + ((int64_t)blockIdx.x * kTeams + team) * P.ws_stride, P.ws_n);
    for (;;) {
        if (tid == 0) log_pick(P, C);
        asm volatile("bar.sync %0, %1;" ::"r"(team), "n"(kThreads) : "memory");
        const int ui = *(volatile int*)&C.unit;
        if (ui >= P.nunits) break;
        const Unit u = P.units[ui];
        const Seg sg = P.segs[u.seg];
        log_unit<Prec, kThreads>(P, sg, u, S, C, P.ws_n, tid, team);  // (barriers inside)
    }
}

// One source per cluster of blocks: for fewer sources than the GPU has SMs.  A warp's neighbours in the
// log go to different blocks, so that a round of a thousand vertices is spread over all of them.
template <class Prec>
__global__ void __launch_bounds__(1024, 1) log_cluster_kernel(KParams P) {
    __shared__ LogCtl own;
    auto cl = cooperative_groups::this_cluster();
    const int nblk = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    LogCtl& C = *cl.map_shared_rank(&own, 0);
    const int tid = (((int)threadIdx.x >> 5) * nblk + rank) * 32 + ((int)threadIdx.x & 31);
    const LState<Prec> S = lstate_carve<Prec>(P.ws + (int64_t)(blockIdx.x / nblk) * P.ws_stride, P.ws_n);
    for (;;) {
        if (tid == 0) log_pick(P, C);
        cl.sync();
        const int ui = *(volatile int*)&C.unit;
        if (ui >= P.nunits) break;
        const Unit u = P.units[ui];
        const Seg sg = P.segs[u.seg];
        log_unit<Prec, 1024, true>(P, sg, u, S, C, P.ws_n, tid, 0, 1024 * nblk);
    }
    cl.sync();  // no block leaves while another may still read the first one's control words
}

}  // namespace fbc
