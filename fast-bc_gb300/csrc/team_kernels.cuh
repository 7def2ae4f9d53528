// Batched schedule, segments of which shared memory holds two or more sources' state (up to some 8,400
// vertices; one, up to 16,384, where there are at most four units an SM): a persistent kernel whose blocks pull (segment, chunk of sources) work items; the
// block's warps form teams, one source per team, every word of a source's state in shared memory.
//
// What bounds it is the chain of dependent accesses of each round (a few hundred rounds per source)
// and the instructions of a round, times the sources in flight, which shared memory limits.  So:
//   * two passes over the rounds instead of three over rounds and levels: the distance pass logs
//     every popped vertex, and a vertex met again at an equal distance (a further shortest path) is
//     popped again, so that the last pops, in log order, have every vertex after all its
//     shortest-path predecessors.  The path counts follow in that order round by round, without
//     in-edge counts, their atomics and the per-level pushes; the dependencies in its reverse.
//     (1% more pops on road grids; the log's rounds outnumber the DAG's levels by a fifth);
//   * 13.5 bytes of state per vertex, planes reused pass after pass:
//       plane 0   (dist | stamp) word                    -> low word of the coefficient
//       plane 1   log of the pops (16 bits, two per vertex; a pop that a later one replaces is cleared), with the
//                 rounds' first log places from its far end
//       plane 2   log place of the last pop              -> path count (32 bits) -> high word
//     and an 8-bit tight-edge mask (16 bits for rows of 9 to 16 edges).
//     Path counts stay below 2^24 here; a source that needs more, or has too many narrow rounds, stops
//     before its dependencies and is done by another kernel;
//   * no far pile: when a bucket is empty, the next bucket's vertices are found by a sweep over the words
//     (four a lane), which costs less than keeping a second queue up to date;
//   * the dependency pass keeps the coefficient c_w = (1 + delta_w) / sigma_w in the place of dist and
//     sigma_w: a predecessor needs nothing else of w, delta_v = sigma_v * sum of c_w over its tight
//     out-edges.  One division per vertex (exact by scaling when the count is a power of two);
//   * one 32-bit word holds distance and queue stamp, so a single native shared-memory atomicMin
//     relaxes an edge and tells whether the vertex is already queued (the host gives the number
//     of stamp bits; stamps are renewed when they run out);
//   * rows as 16-byte quads of (4 * destination:16 | weight:15 | sign), vertex v's first quad at index
//     v: one vector load fetches a row of up to four edges without row offsets; a longer row has a
//     link to its next quad in the fourth place.  The quads lie in shared memory too where four
//     sources still fit beside them;
//   * steps without divergent branches: predicated accesses, and vertex numbers times four, so that they
//     are byte offsets.  (With branches the same passes took a third longer.)
//   * teams of one warp synchronise with __syncwarp and keep their counters in registers; wider ones
//     use a named barrier and counters in shared memory, three of each kind in rotation so that a
//     step takes one barrier.
// Measured against the one-warp kernel at 24 bytes per vertex (batched_kernels.cuh) and the frontier
// kernel, device time of exact or community runs, FP32C, one GB300: 65,536 sources over 76 communities
// of 68 to 2,448 vertices 19.9 -> 5.8 ms; 4,096 vertices 1.8 ms; 8,372 vertices 11.6 -> 8.4 ms;
// all 16,384 sources of that many vertices (one source per SM) 54.7 against 47.3 ms of the frontier kernel and
// 34 of the log kernel, hence the limit at two sources where there are many.
#pragma once
#include "batched_kernels.cuh"

namespace fbc {

constexpr int kTeamThreads = 640;  // 20 warps of up to 96 registers (1,024 threads spill or are no faster)
constexpr int kTeamMax = 15;          // teams of several warps in a block (named barriers 1..15)
constexpr int kTeamRow = 16;          // longest row (mask bits)
constexpr int kTeamIndeg = 255;       // most in-edges of a vertex (sums of that many counts below 2^24 fit 32 bits)
constexpr int kTeamDistBits = 24;     // most distance bits of a word (eight or more stamp bits)
constexpr uint32_t kNoEdge = 0xffffffffu;    // an empty place of a quad (negative, as a link is)
constexpr uint32_t kLink = 0x80010000u;      // | index of the row's next quad
constexpr uint32_t kNoVertex = 0xffffu;
constexpr int kTeamMaxN = 16384;      // 4 * vertex in 16 bits

// Rows of a segment as quads: n first quads, then the continuations (`extra` of them, counted as they are built;
// 0 before).
struct TeamSeg {
    uint4* quad;
    int32_t seg;        // index into KParams::segs
    int32_t stamp_bits; // low bits of a word
    int32_t wide_mask;  // 16-bit masks (rows of more than 8 edges)
    int32_t extra;
};

struct TeamParams {
    KParams k;
    const TeamSeg* tsegs;
    const Chunk* chunks;      // Chunk::seg indexes tsegs
    int32_t nchunks;
    int32_t smem;             // dynamic shared memory of a block (bytes)
    unsigned long long* next_chunk;
};

__host__ __device__ inline int64_t team_n16(int64_t n) { return (n + 15) & ~int64_t(15); }
// shared-memory state of one source: the log has room for two pops a vertex and n / 4 rounds' starts, which lie in
// what the pops leave of it, so that narrow sources of more rounds fit (4 x 500 vertices, all sources, 5.8 -> 2.4 ms)
__host__ __device__ inline int64_t team_log_bytes(int64_t n16) { return 4 * n16 + al16(n16 / 2 + 130); }
__host__ __device__ inline int64_t team_bytes(int64_t n, bool wide_mask) {
    return (wide_mask ? 10 : 9) * team_n16(n) + team_log_bytes(team_n16(n));
}

// Quads of the team segments, one grid row of blocks per segment: the rows in their order, a row
// of more than four edges continued in quads taken from the segment's counter.
__global__ void team_quads_kernel(const Seg* __restrict__ segs, TeamSeg* ts) {
    const TeamSeg t = ts[blockIdx.x];
    const Seg sg = segs[t.seg];
    uint32_t* const q32 = reinterpret_cast<uint32_t*>(t.quad);
    for (int v = blockIdx.y * blockDim.x + threadIdx.x; v < sg.n; v += gridDim.y * blockDim.x) {
        int e = sg.rp[v];
        const int e1 = sg.rp[v + 1];
        int at = v;
        for (;;) {
            const int left = e1 - e;
            const int k = left > 4 ? 3 : left;
            uint32_t r[4] = {kNoEdge, kNoEdge, kNoEdge, kNoEdge};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < k) {
                    const int2 a = __ldg(sg.adj + e + i);
                    r[i] = (uint32_t)a.x << 2 | ((uint32_t)a.y << 16);
                }
            e += k;
            int next = -1;
            if (left > 4) {
                next = sg.n + atomicAdd(&ts[blockIdx.x].extra, 1);
                r[3] = kLink | (uint32_t)next;
            }
            reinterpret_cast<uint4*>(q32)[at] = make_uint4(r[0], r[1], r[2], r[3]);
            if (next < 0) break;
            at = next;
        }
    }
}

// The block's dynamic shared memory, named here so that every access below is seen to be one to
// shared memory (through a plain pointer the atomics become generic ones).
extern __shared__ __align__(16) char team_smem[];

// Predicated accesses with the condition's comparison inside, so that a step of a warp has no
// divergent branch (each costs about as much as a shared-memory round trip).  `a` is a
// shared-memory address.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t atom_min_ge0(uint32_t c, uint32_t a, uint32_t x) {  // where c >= 0; else 0
    uint32_t old;
    asm volatile("{\n .reg .pred q;\n setp.ge.s32 q, %3, 0;\n mov.u32 %0, 0;\n @q atom.shared.min.u32 %0, [%1], %2;\n}"
                 : "=r"(old) : "r"(a), "r"(x), "r"(c) : "memory");
    return old;
}
__device__ __forceinline__ void red_add_eq(uint32_t c, uint32_t d, uint32_t a, uint32_t x) {  // where c == d
    asm volatile("{\n .reg .pred q;\n setp.eq.u32 q, %2, %3;\n @q red.shared.add.u32 [%0], %1;\n}" ::"r"(a), "r"(x), "r"(c),
                 "r"(d) : "memory");
}
__device__ __forceinline__ void st16_lt(uint32_t c, uint32_t d, uint32_t a, uint32_t x) {  // where c < d
    asm volatile("{\n .reg .pred q;\n setp.lt.u32 q, %2, %3;\n @q st.shared.u16 [%0], %1;\n}" ::"r"(a), "h"((uint16_t)x),
                 "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void st8_lt(uint32_t c, uint32_t d, uint32_t a, uint32_t x) {
    asm volatile("{\n .reg .pred q;\n setp.lt.u32 q, %2, %3;\n @q st.shared.u8 [%0], %1;\n}" ::"r"(a), "r"(x), "r"(c),
                 "r"(d) : "memory");
}
// two words where c != 0, else zeros
__device__ __forceinline__ void ld2_if(uint32_t c, uint32_t a, uint32_t b, uint32_t& x, uint32_t& y) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %4, 0;\n mov.u32 %0, 0;\n mov.u32 %1, 0;\n"
                 " @q ld.shared.u32 %0, [%2];\n @q ld.shared.u32 %1, [%3];\n}"
                 : "=&r"(x), "=&r"(y) : "r"(a), "r"(b), "r"(c) : "memory");
}
__device__ __forceinline__ void st2_if(bool c, uint32_t a, uint32_t b, uint32_t x, uint32_t y) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %4, 0;\n @q st.shared.u32 [%0], %2;\n @q st.shared.u32 [%1], %3;\n}" ::"r"(a),
                 "r"(b), "r"(x), "r"(y), "r"((uint32_t)c) : "memory");
}
__device__ __forceinline__ void red_f64_if(bool c, double* a, double x) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q red.global.add.f64 [%0], %1;\n}" ::"l"(a), "d"(x),
                 "r"((uint32_t)c) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t x;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t x;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
    uint32_t x;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(x) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t x) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)x) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t x) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}

// Counters of a team of several warps.
struct TeamCtl {
    uint32_t cnt[3];  // pushes of a step, three in rotation
    int dmin[3];      // least distance beyond the bucket, with them
    int unit, bad;
};

__device__ __forceinline__ uint32_t quad_at(const uint4& q, int i) {
    return i == 0 ? q.x : i == 1 ? q.y : i == 2 ? q.z : q.w;
}
__device__ __forceinline__ bool quad_linked(const uint4& q) { return (int)q.w < 0 && q.w != kNoEdge; }

// kWarp: the team is one warp.  kRows: the quads are in shared memory (else global, read-only).
template <class Prec, bool kWarp, bool kRows>
struct TeamUnit {
    int tid, nth, lane, bar;
    const uint4* quads;  // global quads (kRows: at the start of team_smem)
    TeamCtl* C;

    __device__ __forceinline__ void sync() const {
        if constexpr (kWarp) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nth) : "memory");
    }
    __device__ __forceinline__ uint4 row(uint32_t i4) const {  // quad i4 / 4
        if constexpr (kRows) return *reinterpret_cast<const uint4*>(team_smem + 4u * i4);
        else return __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(quads) + 4u * i4));
    }
    __device__ __forceinline__ void fill(void* p, int words4, uint32_t x) const {
        for (int i = tid; i < words4; i += nth) reinterpret_cast<uint4*>(p)[i] = make_uint4(x, x, x, x);
    }
    // Append x[t] where want[t] at the 16-bit places `at`, at + 2, ... (addresses below end).  The
    // count of a one-warp team is a register (nn), else in shared memory (one add per warp).
    __device__ __forceinline__ void push(const bool (&want)[4], const uint32_t (&x)[4], uint32_t at, uint32_t end, int& nn,
                                         uint32_t* cnt) const {
        unsigned m[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) m[t] = __ballot_sync(kFull, want[t]);
        if ((m[0] | m[1] | m[2] | m[3]) == 0u) return;
        const unsigned below = (1u << lane) - 1u;
        if constexpr (kWarp) {
            at += 2u * (uint32_t)nn;
        } else {
            uint32_t old = 0u;
            if (lane == 0)
                old = atomicAdd(cnt, (uint32_t)(__popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3])));
            at += 2u * __shfl_sync(kFull, old, 0);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t p = at + 2u * (uint32_t)__popc(m[t] & below);
            st16_lt(want[t] ? p : kNoEdge, end, p, x[t]);
            const int c = __popc(m[t]);
            at += 2u * (uint32_t)c;
            if constexpr (kWarp) nn += c;
        }
    }
    __device__ __forceinline__ void run(const KParams& K, const Seg& sg, const Unit& u, const TeamSeg& ts, int off,
                                        int& delta);
};

template <class D>
struct CoefBits;
template <>
struct CoefBits<double> {
    __device__ static double get(uint32_t lo, uint32_t hi) { return __hiloint2double((int)hi, (int)lo); }
    __device__ static void put(double d, uint32_t& lo, uint32_t& hi) {
        lo = (uint32_t)__double2loint(d);
        hi = (uint32_t)__double2hiint(d);
    }
};
template <>
struct CoefBits<float2> {
    __device__ static float2 get(uint32_t lo, uint32_t hi) { return make_float2(__uint_as_float(lo), __uint_as_float(hi)); }
    __device__ static void put(float2 d, uint32_t& lo, uint32_t& hi) {
        lo = __float_as_uint(d.x);
        hi = __float_as_uint(d.y);
    }
};

// Whether a source is too narrow for the kernel after nr rounds of e pops together: one or two vertices a round, as on
// a path (all sources of one of 1,500 vertices: 6.8 ms, 9.9 with a bound on the rounds instead, which only the outer
// sources meet, and late); and, where there are several waves of units (so that most of the segment's are then not
// begun), rounds that the block's few sources cannot fill.  All sources, this kernel / the frontier kernel, ms: 10 x 700
// vertices (two at once on an SM, 12 to 22 pops a round) 36.2 / 26.9, 5 x 1,000 (three; 6 to 11) 33.7 / 21.6; but
// 16 x 350 (16 to 28) 11.2 / 12.8, 12 x 340 6.5 / 9.4, 8 x 500 (four; 9 to 15) 9.0 / 11.3.
constexpr int kTeamMany = 16;  // units a block
__device__ __forceinline__ bool team_narrow(const KParams& K, int n, int nr, int e) {
    return (n > 512 && 20 * e < 41 * nr) || (K.gave && K.nunits > kTeamMany * (int64_t)gridDim.x &&
                                             (float)n * (float)n * (float)nr > 2e6f * (float)e);
}

template <class Prec, bool kWarp, bool kRows>
__device__ __forceinline__ void TeamUnit<Prec, kWarp, kRows>::run(const KParams& K, const Seg& sg, const Unit& u,
                                                                  const TeamSeg& ts, int off, int& delta) {
    const int n = sg.n;
    const int n16 = (int)team_n16(n);
    char* const base = team_smem + off;
    uint32_t* const word = (uint32_t*)base;                // plane 0
    uint32_t* const sig = (uint32_t*)(base + 4 * n16);     // plane 2
    const bool wide = ts.wide_mask != 0;
    // addresses: planes 0 and 2, where a vertex was popped last (plane 2 in the distance pass), tight-edge masks,
    // the log (plane 1), the first round's start at its end (the next ones' below it)
    const uint32_t aword = smem_addr(base), asig = aword + 4u * (uint32_t)n16, alast = asig,
                   amask = aword + 8u * (uint32_t)n16, amask2 = amask + (uint32_t)n16,
                   alog = amask + (wide ? 2u : 1u) * (uint32_t)n16, arnd = alog + (uint32_t)team_log_bytes(n16) - 2u;
    const int sb = ts.stamp_bits;
    const uint32_t smask = (1u << sb) - 1u, one = 1u << sb;
    const int dinf = (int)(kNoEdge >> sb);                 // unreached: all distance bits set
    const uint32_t src4 = 4u * (uint32_t)u.src;
    const uint4 none = make_uint4(kNoEdge, kNoEdge, kNoEdge, kNoEdge);
    int bad = 0;
    int total = 0, nr = 0;  // pops, rounds

    // ---------------------------------------------------------------- distances
    for (;;) {
        fill(word, n16 >> 2, kNoEdge);
        fill(sig, n16 >> 3, kNoEdge);
        sync();
        int s = 0, e = 1, c3 = 0;
        if (tid == 0) {
            sts32(aword + src4, 0u);
            sts16(alog, src4);
            if constexpr (!kWarp) {
                C->cnt[0] = 0u;
                C->dmin[0] = dinf;
                C->bad = 0;
            }
        }
        sync();
        int T = min(delta, dinf);
        uint32_t stamp = smask;
        int left = (int)min((int64_t)K.iter_mult * ((int64_t)n + 2), (int64_t)kInf);  // steps left
        nr = 0;
        uint32_t logend = arnd;  // the next round's start, and the end of the log's free places
        bool full = false;
        for (;;) {
            const int cs = c3;
            uint32_t* const cnt = kWarp ? nullptr : C->cnt + cs;
            if constexpr (!kWarp) {
                c3 = c3 == 2 ? 0 : c3 + 1;
                if (tid == 0) {  // the next step's (last read two barriers ago)
                    C->cnt[c3] = 0u;
                    C->dmin[c3] = dinf;
                }
            }
            if (--left < 0) { bad = kErrIter; break; }
            const bool scan = s == e;
            int nn = 0, dmin = dinf;
            if (!scan) {
                if (stamp == 0u) {  // out of stamps: every vertex back to none (which is never a round's)
                    for (int i = tid; i < n; i += nth) word[i] |= smask;
                    stamp = smask;
                    sync();
                }
                const uint32_t st = --stamp;
                if (tid == 0) sts16(logend, (uint32_t)s);
                logend -= 2u;
                ++nr;
                for (int b = s + (tid & ~31); b < e; b += nth) {
                    const int i = b + lane;
                    const bool act = i < e;
                    const uint32_t v4 = lds16(alog + 2u * (uint32_t)(act ? i : s));
                    uint4 q = row(v4);
                    const int dv = (int)(lds32(aword + v4) >> sb);  // may have dropped since the push
                    const uint32_t before = lds16(alast + (v4 >> 1));
                    if (!act) q = none;
                    st16_lt((uint32_t)i, (uint32_t)e, alast + (v4 >> 1), (uint32_t)i);
                    st16_lt(act ? before : kNoVertex, kNoVertex, alog + 2u * before, kNoVertex);  // only the last pop stays
                    for (;;) {
                        uint32_t x4[4];
                        bool want[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            // a relaxation below the threshold carries the round's stamp (stamps fall,
                            // so an equal distance of an earlier round is met too: its vertex is
                            // popped again, after this predecessor); beyond it, no stamp
                            const uint32_t a = quad_at(q, t);
                            x4[t] = a & 0xffffu;
                            const int nd = dv + (int)(a >> 16);
                            const bool near = nd < T;
                            const uint32_t key = (uint32_t)nd * one + (near ? st : smask);
                            const uint32_t old = atom_min_ge0(a, aword + x4[t], key);
                            want[t] = near && key < old && (old & smask) != st;
                        }
                        push(want, x4, alog + 2u * (uint32_t)e, logend, nn, cnt);
                        const bool link = quad_linked(q);
                        if (!__any_sync(kFull, link)) break;
                        const uint32_t next = link ? 4u * (q.w & 0xffffu) : v4;
                        q = row(next);
                        if (!link) q = none;
                    }
                }
            } else {
                if (many_rounds(n, nr) && team_narrow(K, n, nr, e)) { bad = kErrNarrow; break; }
                // the bucket is empty: on to the next one, or to the one of the closest vertex beyond
                const int T0 = T;
                T = T0 >= dinf - delta ? dinf : T0 + delta;
                for (int b = (tid & ~31); b < (n16 >> 2); b += nth) {
                    const int i = b + lane;
                    const uint32_t x4[4] = {16u * (uint32_t)i, 16u * (uint32_t)i + 4u, 16u * (uint32_t)i + 8u,
                                            16u * (uint32_t)i + 12u};
                    bool want[4];
                    const uint4 w4 = i < (n16 >> 2) ? reinterpret_cast<const uint4*>(word)[i] : none;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int d = (int)(quad_at(w4, t) >> sb);
                        want[t] = d >= T0 && d < T;
                        if (d >= T) dmin = min(dmin, d);
                    }
                    push(want, x4, alog + 2u * (uint32_t)e, logend, nn, cnt);
                }
                dmin = __reduce_min_sync(kFull, dmin);
                if constexpr (!kWarp) {
                    if (lane == 0 && dmin != dinf) atomicMin(&C->dmin[cs], dmin);
                }
            }
            sync();
            if constexpr (!kWarp) nn = (int)*(volatile uint32_t*)cnt;
            if (scan && nn == 0) {
                if constexpr (!kWarp) dmin = *(volatile int*)&C->dmin[cs];
                if (dmin >= dinf) break;  // nothing further is reached
                T = dmin / delta * delta;  // that bucket's start
            }
            s = e;
            e += nn;
            if (alog + 2u * (uint32_t)e > logend) { full = true; break; }
        }
        sync();
        total = e;
        if (!full) break;
        // the log is full: again with narrower buckets (width 1 pops every vertex once, and there is room for
        // that and as many rounds)
        delta = max(1, delta >> 2);
    }

    if (tid == 0 && !bad && many_rounds(n, nr) && team_narrow(K, n, nr, total)) count_narrow(K, u.seg);
    if (!bad) {
        // --------------------------------------------------------------- path counts
        // round by round over the last pops (every tight predecessor's is in an earlier round):
        // the tight edges are found, noted in the vertex's mask and pass its count on
        if (u.bout >= 0)
            for (int j = tid; j < sg.nb; j += nth) {
                const int d = (int)(word[sg.border[j]] >> sb);
                K.bdist[u.bout + j] = d != dinf ? nonneg_int_to_double(d) : 0.0;
            }
        if (tid == 0) sts16(arnd - 2u * (uint32_t)nr, (uint32_t)total);
        fill(sig, n16 >> 2, 0u);
        sync();
        if (tid == 0) sts32(asig + src4, 1u);  // one path to the source
        sync();
        uint32_t high = 0u;  // bits of the counts
        int s = 0, e = (int)lds16(arnd - 2u);
        for (int r = 0; r < nr; ++r) {
            const int e2 = (int)lds16(arnd - 2u * (uint32_t)min(r + 2, nr));
            for (int b = s + (tid & ~31); b < e; b += nth) {
                const int i = b + lane;
                uint32_t v4 = lds16(alog + 2u * (uint32_t)min(i, e - 1));
                const bool on = i < e && v4 != kNoVertex;
                if (!on) v4 = src4;
                uint4 q = row(v4);
                const uint32_t dv = lds32(aword + v4) | smask;
                const uint32_t sv = lds32(asig + v4);
                if (!on) q = none;
                high |= sv;
                unsigned mk = 0u;
                for (int p = 0;; p += 3) {
                    // the place of no edge, or of a link, is tested against the vertex itself and never
                    // found tight (it adds to the distance)
                    uint32_t x4[4], wx[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t a = quad_at(q, t);
                        x4[t] = (int)a >= 0 ? a & 0xffffu : v4;
                        wx[t] = lds32(aword + x4[t]) | smask;
                    }
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t key = (quad_at(q, t) >> 16) * one + dv;
                        if (wx[t] == key) mk |= 1u << (p + t);
                        red_add_eq(wx[t], key, asig + x4[t], sv);
                    }
                    const bool link = quad_linked(q);
                    if (!__any_sync(kFull, link)) break;
                    q = row(link ? 4u * (q.w & 0xffffu) : v4);
                    if (!link) q = none;
                }
                const uint32_t gate = on ? 0u : 1u;
                st8_lt(gate, 1u, amask + (v4 >> 2), mk);
                if (wide) st8_lt(gate, 1u, amask2 + (v4 >> 2), mk >> 8);
            }
            s = e;
            e = e2;
            sync();
        }
        // every count below 2^24 (so no sum over up to 255 in-edges wrapped)
        bad = __any_sync(kFull, (high >> 24) != 0u) ? kErrNarrow : 0;
        if constexpr (!kWarp) {
            if (bad && lane == 0) atomicOr(&C->bad, bad);
            sync();
            bad = *(volatile int*)&C->bad;
        }
        if (!bad && u.bout >= 0)
            for (int j = tid; j < sg.nb; j += nth) K.bsig[u.bout + j] = sig[sg.border[j]];
        sync();
    }
    if (!bad) {
        // --------------------------------------------------------- dependency
        using CB = CoefBits<typename Prec::D>;
        const double card = u.card;
        const bool card1 = __double_as_longlong(card) == 0x3ff0000000000000ll;
        double* const bc = K.bc + sg.out_base;
        int hi = total, lo = (int)lds16(arnd - 2u * (uint32_t)(nr - 1));
        for (int r = nr - 1; r >= 0; --r) {
            const int lo2 = (int)lds16(arnd - 2u * (uint32_t)max(r - 1, 0));
            for (int b = lo + (tid & ~31); b < hi; b += nth) {
                const int i = b + lane;
                uint32_t v4 = lds16(alog + 2u * (uint32_t)min(i, hi - 1));
                const bool on = i < hi && v4 != kNoVertex;
                if (!on) v4 = src4;
                uint4 q = row(v4);
                uint32_t m = lds8(amask + (v4 >> 2));
                if (wide) m |= lds8(amask2 + (v4 >> 2)) << 8;
                uint32_t sv = lds32(asig + v4);
                if (!on) {
                    m = 0u;
                    sv = 1u;
                }
                const bool inner = m != 0u && v4 != src4;
                const int v = (int)(v4 >> 2);
                double* const o = bc + (sg.gid ? __ldg(sg.gid + v) : v);
                typename Prec::Acc acc = Prec::zero();
                for (;;) {  // in row order
                    const bool link = quad_linked(q) && (m >> 3) != 0u;
                    uint32_t cl[4], ch[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t x4 = quad_at(q, t) & 0xffffu;
                        ld2_if(t == 3 && link ? 0u : m & (1u << t), aword + x4, asig + x4, cl[t], ch[t]);
                    }
                    Prec::add_coefs(acc, CB::get(cl[0], ch[0]), CB::get(cl[1], ch[1]), CB::get(cl[2], ch[2]),
                                    CB::get(cl[3], ch[3]));
                    if (!__any_sync(kFull, link)) break;
                    q = row(link ? 4u * (q.w & 0xffffu) : v4);
                    m = link ? m >> 3 : 0u;
                }
                uint32_t cl, ch;
                if (!__any_sync(kFull, sv != 1u)) {  // every count of the warp is 1
                    CB::put(Prec::coef1(acc), cl, ch);
                } else {
                    acc = Prec::times(acc, sv);
                    CB::put(Prec::coef(acc, sv), cl, ch);
                }
                st2_if(on, aword + v4, asig + v4, cl, ch);
                const double val = Prec::value(acc);
                red_f64_if(inner, o, card1 ? val : card * val);
            }
            hi = lo;
            lo = lo2;
            sync();
        }
    }
    if (tid == 0) count_unit(K, u.seg, bad == kErrNarrow);
    if (bad && tid == 0) {
        if (bad == kErrNarrow) request_retry(K, u, kErrNarrow);  // recomputed with wider counts
        else atomicOr(K.err, bad);
    }
    sync();
}

// Teams of a block for a segment of n vertices: rows in shared memory where at least kRowTeams
// sources still fit beside them, S sources at once, W warps each -- one for up to 1,023 vertices and
// one more for every 512 after, for a round of fewer vertices leaves the others idle (870-vertex
// sources: 147 us a batch with one warp, 162 with two; 4,096: 3.0 ms with one, 1.8 with eight).
struct TeamSplit {
    bool rows;
    int S, W;
};
constexpr int kRowTeams = 4;
// Bucket width: twice the segment's.  A round costs a chain of accesses here whatever its width, and
// the path counts and dependencies repeat the rounds.
__device__ __forceinline__ int team_delta(int d) { return d > 0 ? (d > 0x1fffffff ? d : 2 * d) : 2; }
__device__ __forceinline__ TeamSplit team_split(int n, int nquads, bool wide, int smem, int count, int nwarps) {
    const int per = (int)team_bytes(n, wide);
    const int qb = 16 * nquads;
    const int sa = qb < smem ? (smem - qb) / per : 0;
    TeamSplit t;
    t.rows = sa >= kRowTeams || (sa >= 1 && sa >= count);
    t.S = min(t.rows ? sa : smem / per, min(count, nwarps));
    t.S = max(t.S, 1);
    t.W = max(1, min(nwarps / t.S, n >> 9));
    if (t.W > 1 && t.S > kTeamMax) t.W = 1;
    return t;
}

// The chunk's next unit that is worth starting here; the others go back (one thread).
__device__ __forceinline__ int team_pick(const KParams& K, const Unit* units, int count, int* next) {
    for (;;) {
        const int k = atomicAdd(next, 1);
        if (k >= count) return k;
        const Unit u = units[k];
        if (!gave_up(K, u.seg)) return k;
        request_retry(K, u, kErrNarrow);
    }
}

template <class Prec>
__global__ void __launch_bounds__(kTeamThreads, 1) team_kernel(TeamParams TP) {
    __shared__ int s_chunk, s_next;
    __shared__ TeamCtl ctl[kTeamMax];
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (;;) {
        if (threadIdx.x == 0) {
            s_chunk = (int)atomicAdd(TP.next_chunk, 1ull);
            s_next = 0;
        }
        __syncthreads();
        const int ci = s_chunk;
        if (ci >= TP.nchunks) break;
        const Chunk ch = TP.chunks[ci];
        const TeamSeg ts = TP.tsegs[ch.seg];
        const Seg sg = TP.k.segs[ts.seg];
        const int nq = sg.n + ts.extra;
        const TeamSplit sp = team_split(sg.n, nq, ts.wide_mask != 0, TP.smem, ch.count, nw);
        if (sp.rows)
            for (int i = threadIdx.x; i < nq; i += blockDim.x)
                reinterpret_cast<uint4*>(team_smem)[i] = __ldg(ts.quad + i);
        __syncthreads();
        const int team = w / sp.W;
        if (team < sp.S) {
            const int base = (sp.rows ? 16 * nq : 0) + team * (int)team_bytes(sg.n, ts.wide_mask != 0);
            const Unit* const units = TP.k.units + ch.first;
            const int lane = threadIdx.x & 31;
            if (sp.W == 1) {
                TeamUnit<Prec, true, true> U{lane, 32, lane, 0, nullptr, nullptr};
                TeamUnit<Prec, true, false> G{lane, 32, lane, 0, ts.quad, nullptr};
                int delta = team_delta(sg.delta);
                for (;;) {
                    int k = 0;
                    if (lane == 0) k = team_pick(TP.k, units, ch.count, &s_next);
                    k = __shfl_sync(kFull, k, 0);
                    if (k >= ch.count) break;
                    if (sp.rows) U.run(TP.k, sg, units[k], ts, base, delta);
                    else G.run(TP.k, sg, units[k], ts, base, delta);
                }
            } else {
                const int tid = threadIdx.x - team * sp.W * 32;
                TeamCtl* C = ctl + team;
                TeamUnit<Prec, false, true> U{tid, sp.W * 32, lane, team + 1, nullptr, C};
                TeamUnit<Prec, false, false> G{tid, sp.W * 32, lane, team + 1, ts.quad, C};
                int delta = team_delta(sg.delta);
                for (;;) {
                    if (tid == 0) C->unit = team_pick(TP.k, units, ch.count, &s_next);
                    U.sync();
                    const int k = *(volatile int*)&C->unit;
                    if (k >= ch.count) break;
                    if (sp.rows) U.run(TP.k, sg, units[k], ts, base, delta);
                    else G.run(TP.k, sg, units[k], ts, base, delta);
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace fbc
