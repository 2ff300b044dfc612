// ct_euclid.cu — exact Euclidean kNN (the reference's Euclidean cover-tree path,
// CoverTreeWrapper.insert / knn_query, src/lib.rs:207-223,331 and
// src/algo.rs:179-323, which prunes with 2^(level+1) radii the greedy batch
// insert does not guarantee; this search is exhaustive and exact).
//
// A work item is a tile of 32 queries against a chunk of the points, swept 256 points at a time
// by eight warps (two along the queries, four along the points); a thread holds 4 queries x 8
// points.  d^2 is the left-to-right sum of squared differences, as `Euclidean::distance_sq`
// (src/metric.rs:33-41), one FMA per axis; the returned distance is its square root.
//
// What bounds it: 2 d FP32 operations per pair and one minimum.  Two points run as one f32x2
// chain (points lie axis-major in shared memory, so a 16-byte read brings two such pairs and a
// warp's reads of an axis are one wavefront each); for d <= 4 the negated query coordinates stay
// in registers.  A query's 8 values are compared with its threshold through their minimum; the
// few that pass go to a per-query buffer, which a warp sorts and merges into the query's list in
// registers when the next step could overflow it (the dense tile's lists, ct_dense.cuh).
//
// A list filled from infinity takes k ln(n / k) insertions, which cost more than the distances
// at n = 32768.  So the chunk is first swept in part for thresholds only: each of a query's 32
// threads keeps the smallest value of its own points, and the k-th smallest of those minima
// bounds the k-th distance (about the 1.2 k-th neighbour of the sample).
//
// Few query tiles split the points; up to 8 chunks of a tile form a cluster, whose blocks merge
// the lists through distributed shared memory (no scratch, no second launch), more of them go
// through scratch and a counter.
//
// Few points (some 600 at most) and few queries take a warp per query instead: the tile's fixed chain
// (thresholds, then four queries' sorts per warp) is 6 to 12 us there against 1 to 3.
//
// Measured on GB300 (whole calls, queries = the points; before: a warp per query with a sorted list
// of k per lane, so that a warp ran k insertion steps for every point any lane took):
//   n = 32768, d = 3, k = 10     4.49 -> 0.71 ms (9.0 T lane operations/s of 39 measured; without
//                                the sampled thresholds 1.11 ms)
//   n = 65536, d = 3, k = 10    14.8  -> 2.30 ms;   n = 65536, d = 8, k = 50, predecessors 54.1 -> 3.3 ms
//   n = 1024,  d = 3, k = 10    23 us both (the host's share of a call)
//   n = 50,    d = 3, k = 10    16.5 us, 22.5 with the tile
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "ct_common.cuh"
#include "ct_dense.cuh"
#include "ct_internal.h"

namespace ct {
namespace {

using dense::u64;

constexpr int kEThreads = 256;
constexpr int kEWarps = kEThreads / 32;
constexpr int kEQ = 32;    // queries of a tile
constexpr int kEC = 256;   // points of a step
constexpr int kESlack = 16;
constexpr int kECap = kEC + kESlack;  // buffer keys per query, merged above kESlack
constexpr int kEMaxK = 64;
constexpr int kEMaxD = 16;

struct ESmem {
    size_t pts, qry, buf, list, tau, taud, cnt, total;
};
__host__ __device__ inline ESmem e_layout(int d, int k) {
    ESmem L;
    size_t off = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 15) & ~size_t(15); return o; };
    L.pts = take(sizeof(float) * 2 * kEC * d);  // two steps, axis-major
    L.qry = take(sizeof(float) * 2 * kEQ * d);  // negated, each value twice (an f32x2 operand)
    L.buf = take(sizeof(u64) * kEQ * kECap);
    L.list = take(sizeof(u64) * kEQ * k);
    L.tau = take(sizeof(u64) * kEQ);
    L.taud = take(sizeof(float) * kEQ);
    L.cnt = take(sizeof(int) * kEQ);
    L.total = off;
    return L;
}

struct EParams {
    const float* pts;
    const float* qry;
    long long n, nq;
    int d, k, predecessor;
    int sample;       // steps of a chunk swept first for the thresholds
    int split;        // point chunks per query tile
    long long chunk;  // points per chunk (a multiple of kEC)
    // The chunks' lists meet either in their cluster's shared memory (part == nullptr: the split blocks
    // of a tile are one cluster) or in scratch, merged by the block that finishes last.
    u64* part;        // [nq][split][k] sorted keys
    int* done;        // [tiles] finished chunks, zero at launch
    long long* out_idx;
    float* out_dist;
};

__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 sqr_add2(u64 a, u64 s) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(r) : "l"(a), "l"(s));
    return r;
}
__device__ __forceinline__ float half_of(u64 a, int h) { return __uint_as_float((unsigned)(a >> (32 * h))); }

// D = 1..4: that many axes, query operands in registers; D = 5..8: operands from shared memory, the
// axes unrolled; D = 0: any d.
template <int D>
__global__ void __launch_bounds__(kEThreads, 2) euclid_knn_kernel(EParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_last;
    const int d = D > 0 ? D : P.d, k = P.k;
    const ESmem S = e_layout(d, k);
    float* Pts = (float*)(smem_raw + S.pts);
    u64* Qry = (u64*)(smem_raw + S.qry);
    u64* Buf = (u64*)(smem_raw + S.buf);
    u64* List = (u64*)(smem_raw + S.list);
    u64* Tau = (u64*)(smem_raw + S.tau);
    float* TauD = (float*)(smem_raw + S.taud);
    int* Cnt = (int*)(smem_raw + S.cnt);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int qrow = (warp & 1) * 16 + (lane >> 3);        // queries qrow + 4a
    const int ccol = (warp >> 1) * 64 + (lane & 7) * 4;    // points ccol + i, ccol + 32 + i, i < 4
    const long long tiles = (P.nq + kEQ - 1) / kEQ;
    const long long tile = tiles - 1 - blockIdx.x / P.split;  // heavy tiles (predecessor mode) first
    const int ch = (int)(blockIdx.x % P.split);
    const long long q0 = tile * kEQ;
    const int nv = (int)(P.nq - q0 < kEQ ? P.nq - q0 : kEQ);

    for (int e = tid; e < kEQ * d; e += kEThreads) {
        const float x = e < nv * d ? -P.qry[q0 * d + e] : 0.f;
        Qry[e] = ((u64)__float_as_uint(x) << 32) | __float_as_uint(x);
    }
    for (int e = tid; e < kEQ; e += kEThreads) {
        // a distance of FLT_MAX or more (and NaN) is no neighbour
        Tau[e] = e < nv ? dense::make_key(CT_FLT_MAX, 0) : 0ULL;
        TauD[e] = e < nv ? CT_FLT_MAX : -1.f;
        Cnt[e] = 0;
    }
    for (int e = tid; e < kEQ * k; e += kEThreads) List[e] = dense::kNoKey;

    // points of the chunk; in predecessor mode query row i takes points j < i
    const long long cb = (long long)ch * P.chunk;
    long long ce = cb + P.chunk < P.n ? cb + P.chunk : P.n;
    if (P.predecessor) ce = ce < q0 + nv - 1 ? ce : q0 + nv - 1;
    const int nsteps = ce > cb ? (int)((ce - cb + kEC - 1) / kEC) : 0;

    // a step's points: read into registers one step ahead, stored axis-major (NaN past the end:
    // their distances pass no test)
    constexpr int kPer = kEC * (D > 0 ? D : kEMaxD) / kEThreads;
    float next[kPer];
    auto fetch = [&](int t) {
        const long long base = (cb + (long long)t * kEC) * d, lim = ce * d - base;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int e = tid + i * kEThreads;
            if (D > 0 || e < kEC * d) next[i] = e < lim ? __ldg(P.pts + base + e) : __int_as_float(0x7fc00000);
        }
    };
    const int r0 = tid / d, c0 = tid - r0 * d, dr = kEThreads / d, dc = kEThreads - dr * d;
    auto store = [&](float* dst) {
        int r = r0, c = c0;  // point and axis of element tid + i * kEThreads
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            if (D > 0 || r < kEC) dst[c * kEC + r] = next[i];
            r += dr; c += dc;
            if (c >= d) { c -= d; ++r; }
        }
    };
    if (nsteps > 0) {
        fetch(0);
        store(Pts);
    }
    __syncthreads();
    constexpr int DR = D >= 1 && D <= 4 ? D : 0;  // axes held in registers
    u64 q[4][DR > 0 ? DR : 1];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < DR; ++c) q[a][c] = Qry[(qrow + 4 * a) * d + c];
    // d^2 of the thread's 4 queries and 8 points: query a, points (ccol, +1), (+2, +3), (+32, +33),
    // (+34, +35)
    u64 s[4][4];
    auto distances = [&](const float* X) {
        auto axis = [&](int c, const u64(&qc)[4]) {
            const ulonglong2 x0 = *(const ulonglong2*)(X + c * kEC + ccol);
            const ulonglong2 x1 = *(const ulonglong2*)(X + c * kEC + ccol + 32);
            const u64 x[4] = {x0.x, x0.y, x1.x, x1.y};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[a][i] = sqr_add2(add2(x[i], qc[a]), D > 0 && c == 0 ? 0ULL : s[a][i]);
        };
        auto from_shared = [&](int c) {
            const u64 qc[4] = {Qry[qrow * d + c], Qry[(qrow + 4) * d + c], Qry[(qrow + 8) * d + c],
                               Qry[(qrow + 12) * d + c]};
            axis(c, qc);
        };
        if constexpr (DR > 0) {
#pragma unroll
            for (int c = 0; c < DR; ++c) {
                const u64 qc[4] = {q[0][c], q[1][c], q[2][c], q[3][c]};
                axis(c, qc);
            }
        } else if constexpr (D > 0) {
#pragma unroll
            for (int c = 0; c < D; ++c) from_shared(c);
        } else {
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[a][i] = 0ULL;
            for (int c = 0; c < d; ++c) from_shared(c);
        }
    };
    // ---- thresholds.  The smallest d^2 that each thread sees over the sampled steps is the distance
    // of a different point for each of a query's 32 threads (128 with a minimum per f32x2 pair), so
    // the k-th smallest of those minima bounds the k-th distance of the chunk.  The sweep below then
    // starts with a threshold few points pass, instead of filling every list from infinity.
    const int nsample = nsteps < P.sample ? nsteps : P.sample;
    if (nsample > 0) {
        float mn[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int i = 0; i < 4; ++i) mn[a][i] = CT_FLT_MAX;
        for (int t = 0; t < nsample; ++t) {
            // after the last sampled step the sweep starts over
            const int tn = t + 1 < nsample ? t + 1 : 0;
            fetch(tn);
            distances(Pts + (size_t)(t & 1) * kEC * d);
            const long long j0 = cb + (long long)t * kEC;
            if (P.predecessor && j0 + kEC > q0) {
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const bool ok = j0 + ccol + (i < 4 ? i : 28 + i) < q0 + qrow + 4 * a;
                        mn[a][i >> 1] = fminf(mn[a][i >> 1], ok ? half_of(s[a][i >> 1], i & 1) : CT_FLT_MAX);
                    }
            } else {
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        mn[a][i] = fminf(mn[a][i], fminf(half_of(s[a][i], 0), half_of(s[a][i], 1)));
            }
            store(Pts + (size_t)((t + 1) & 1) * kEC * d);
            __syncthreads();
        }
        // (the buffers hold the minima meanwhile: 32 threads along the points x 1 or 4 of them)
        u64* Min = Buf;
        const int at = (warp >> 1) * 8 + (lane & 7);
        const int per = k <= 16 ? 1 : 4;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            u64* row = Min + (qrow + 4 * a) * 128;
            if (per == 1) {
                row[at] = dense::make_key(fminf(fminf(mn[a][0], mn[a][1]), fminf(mn[a][2], mn[a][3])), at);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) row[at * 4 + i] = dense::make_key(mn[a][i], at * 4 + i);
            }
        }
        __syncthreads();
        for (int qi = warp; qi < nv; qi += kEWarps) {
            const u64* row = Min + qi * 128;
            u64 kth;
            if (per == 1) {
                u64 x[1] = {row[lane]};
                dense::warp_sort<1>(x);
                kth = __shfl_sync(0xffffffffu, x[0], k - 1);
            } else {
                u64 x[4] = {row[lane], row[32 + lane], row[64 + lane], row[96 + lane]};
                dense::warp_sort<4>(x);
                kth = __shfl_sync(0xffffffffu, k <= 32 ? x[0] : x[1], (k - 1) & 31);
            }
            const float td = __uint_as_float((unsigned)(kth >> 32));
            if (lane == 0 && td < CT_FLT_MAX) {
                Tau[qi] = dense::make_key(td, -1);  // (equal distances pass, whatever their index)
                TauD[qi] = td;
            }
        }
        __syncthreads();
    }
    const int flip = nsample & 1;  // the buffer that holds step 0
    for (int t = 0; t < nsteps; ++t) {
        if (t + 1 < nsteps) fetch(t + 1);
        distances(Pts + (size_t)((t + flip) & 1) * kEC * d);
        const long long j0 = cb + (long long)t * kEC;
        const bool edge = P.predecessor && j0 + kEC > q0;  // some points are not predecessors of every query
        const int trig = t + 1 < nsteps ? kESlack : 0;
        int full = 0;  // some buffer has to be merged before the next step
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int qi = qrow + 4 * a;
            const float td = TauD[qi];
            float mn = fminf(half_of(s[a][0], 0), half_of(s[a][0], 1));
#pragma unroll
            for (int i = 1; i < 4; ++i) mn = fminf(mn, fminf(half_of(s[a][i], 0), half_of(s[a][i], 1)));
            if (__any_sync(0xffffffffu, mn <= td)) {
                const u64 tau = Tau[qi];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float v = half_of(s[a][i >> 1], i & 1);
                    if (v <= td) {
                        const long long gc = j0 + ccol + (i < 4 ? i : 28 + i);
                        const u64 key = dense::make_key(v, (int)gc);
                        if (key < tau && (!edge || gc < q0 + qi)) {
                            const int at = atomicAdd(&Cnt[qi], 1);
                            Buf[qi * kECap + at] = key;
                            full |= at >= trig;
                        }
                    }
                }
            }
        }
        if (t + 1 < nsteps) store(Pts + (size_t)((t + 1 + flip) & 1) * kEC * d);
        if (!__syncthreads_or(full) && t + 1 < nsteps) continue;
        // warp w owns queries w, w + 8, ...; buffers that the next step could overflow are merged (after
        // the last step, all that hold a key)
        for (int qi = warp; qi < kEQ; qi += kEWarps) {
            const int cnt = Cnt[qi];
            if (cnt <= trig) continue;
            dense::merge_buffer(List + qi * k, k, Buf + qi * kECap, cnt);
            if (lane == 0) {
                const u64 kth = List[qi * k + k - 1];
                Cnt[qi] = 0;
                if (kth != dense::kNoKey) {
                    Tau[qi] = kth;
                    TauD[qi] = __uint_as_float((unsigned)(kth >> 32));
                }
            }
        }
        // the next step's pushes wait for the merges
        __syncthreads();
    }
    auto write = [&](long long g, int j, u64 key) {
        P.out_idx[g * k + j] = key == dense::kNoKey ? -1LL : (long long)(unsigned)key;
        P.out_dist[g * k + j] = key == dense::kNoKey ? CT_FLT_MAX : sqrtf(__uint_as_float((unsigned)(key >> 32)));
    };
    if (P.split > 1 && !P.part) {
        // every block of the cluster merges its share of the tile's queries
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        for (int qi = ch * kEWarps + warp; qi < nv; qi += P.split * kEWarps) {
            u64 a[2] = {dense::kNoKey, dense::kNoKey};
            for (int r = 0; r < P.split; ++r) {
                const u64* src = cl.map_shared_rank(List + qi * k, r);
                u64 x[2] = {lane < k ? src[lane] : dense::kNoKey, 32 + lane < k ? src[32 + lane] : dense::kNoKey};
                dense::warp_merge<2>(a, x);
            }
            if (lane < k) write(q0 + qi, lane, a[0]);
            if (32 + lane < k) write(q0 + qi, 32 + lane, a[1]);
        }
        cl.sync();  // no block leaves while another reads its lists
        return;
    }
    __syncwarp();
    for (int qi = warp; qi < nv; qi += kEWarps) {
        const long long g = q0 + qi;
        for (int j = lane; j < k; j += 32) {
            const u64 key = List[qi * k + j];
            if (P.split > 1) P.part[(g * P.split + ch) * k + j] = key;
            else write(g, j, key);
        }
    }
    if (P.split > 1) {
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(&P.done[tile], 1) == P.split - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            dense::merge_tile<kEThreads, true>(P.part, P.split, k, q0, nv, (u64*)smem_raw, P.out_idx, P.out_dist, k);
        }
    }
}

// The form for few points: one warp per query, eight queries per block.  Points are staged through shared
// memory; lane l scores points l, l + 32, ... and keeps its own K best (d^2, index) in registers, sorted (a
// lane sees its points in increasing index, so a tie keeps the lower index).  The warp merges its 32 lists
// with k rounds of a warp-wide (d^2, index) minimum.
constexpr int kSTile = 512;

__device__ __forceinline__ bool dl_less(float da, int ia, float db, int ib) {
    return da < db || (da == db && ia < ib);
}

template <int K>
__global__ void __launch_bounds__(kEThreads) euclid_small_kernel(EParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* tile = (float*)smem_raw;  // kSTile * d floats
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = P.d;
    const long long qi = (long long)blockIdx.x * kEWarps + warp;
    const bool active = qi < P.nq;
    float q[kEMaxD];
#pragma unroll
    for (int c = 0; c < kEMaxD; ++c) q[c] = (active && c < d) ? P.qry[qi * d + c] : 0.f;
    float bd[K];
    int bi[K];
#pragma unroll
    for (int j = 0; j < K; ++j) { bd[j] = CT_FLT_MAX; bi[j] = 0x7fffffff; }
    const long long limit = P.predecessor ? (active ? qi : 0) : P.n;
    // the block needs points below the largest limit of its queries
    const long long block_limit = P.predecessor ? min(P.n, ((long long)blockIdx.x + 1) * kEWarps) : P.n;
    for (long long t0 = 0; t0 < block_limit; t0 += kSTile) {
        const int tn = (int)min((long long)kSTile, block_limit - t0);
        __syncthreads();
        for (int e = threadIdx.x; e < tn * d; e += kEThreads) tile[e] = P.pts[t0 * d + e];
        __syncthreads();
        if (!active) continue;
        const int jn = (int)min((long long)tn, limit - t0);
        for (int j = lane; j < jn; j += 32) {
            float s = 0.f;
            for (int c = 0; c < d; ++c) {
                const float df = __fsub_rn(q[c], tile[j * d + c]);
                s = __fmaf_rn(df, df, s);
            }
            if (s < bd[K - 1]) {  // strict: an equal distance seen later has a larger index
                const int gj = (int)(t0 + j);
#pragma unroll
                for (int p = K - 1; p > 0; --p) {
                    const bool up = s < bd[p - 1];
                    const bool here = !up && s < bd[p];
                    bd[p] = up ? bd[p - 1] : (here ? s : bd[p]);
                    bi[p] = up ? bi[p - 1] : (here ? gj : bi[p]);
                }
                if (s < bd[0]) { bd[0] = s; bi[0] = gj; }
            }
        }
    }
    if (!active) return;
    int head = 0;
    for (int r = 0; r < P.k; ++r) {
        float hd = CT_FLT_MAX;
        int hi = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < K; ++j)
            if (j == head) { hd = bd[j]; hi = bi[j]; }
        float md = hd;
        int mi = hi;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float od = __shfl_xor_sync(0xffffffffu, md, off);
            const int oi = __shfl_xor_sync(0xffffffffu, mi, off);
            if (dl_less(od, oi, md, mi)) { md = od; mi = oi; }
        }
        if (hd == md && hi == mi && hi != 0x7fffffff) ++head;
        if (lane == 0) {
            const bool ok = mi != 0x7fffffff && md < CT_FLT_MAX;
            P.out_idx[qi * P.k + r] = ok ? (long long)mi : -1LL;
            P.out_dist[qi * P.k + r] = ok ? sqrtf(md) : CT_FLT_MAX;
        }
    }
}

// Where it is the faster form (n = 16 to 1500, 1 to 40000 queries, k = 1 to 24, d = 1 to 16, both timed): up
// to 600 - 8 k points (n = 400, 300 queries, d = 3: k = 1 15 against 19 us, k = 24 28 against 32; n = 700,
// k = 16 even), while one wave of warps takes the queries; and with eight queries at most, one per warp of
// the tile, for the shortest lists or more than 8 axes only.  A predecessor search sees no more points than
// it has queries.
bool small_form(long long n, long long nq, int d, int k, int predecessor) {
    if (predecessor) n = std::min(n, nq);
    return n + 8 * k <= 600 && k <= (nq > 8 || d > 8 ? 24 : 4) &&
           (double)nq * (double)n * k <= (nq <= 1000 ? 3e6 : 2e6);
}

template <int K>
cudaError_t launch_small(const EParams& P, cudaStream_t st) {
    const size_t smem = sizeof(float) * kSTile * (size_t)P.d;  // at most 32 KB
    euclid_small_kernel<K><<<(unsigned)((P.nq + kEWarps - 1) / kEWarps), kEThreads, smem, st>>>(P);
    return cudaGetLastError();
}

// Sampled steps of a chunk of L points: a sample of M points leaves about 1.2 k L / M points under
// the threshold, each worth some 480 pairs of distances (its warp's detour and its share of a
// merge) at d = 3, fewer where a pair costs more (about 2 d + 2 instructions), so M grows as
// sqrt(k L).
int sample_steps(double len, int k, int d) {
    return (int)std::ceil(std::min(len, std::sqrt(576.0 * 8.0 / (2.0 * d + 2.0) * k * len)) / kEC);
}

// Point chunks per query tile: whole waves of two blocks per SM against what every chunk repeats
// (its sample, the points under its threshold, its merge).
int choose_split(long long n, long long nq, int d, int k, int predecessor, int sms) {
    const double tiles = std::ceil((double)nq / kEQ), slots = 2.0 * sms;
    const long long most = std::max<long long>(1, std::min<long long>(64, n / kEC));
    int best = 1;
    double best_t = 0.0;
    for (int sp = 1; sp <= most; ++sp) {
        const double len = std::ceil((double)n / sp / kEC) * kEC;
        const double cost = 256.0 + 2.0 * sample_steps(len, k, d) * kEC + 30.0 * k;
        const double items = tiles * sp;
        const double t = predecessor ? std::max(items * (0.5 * len + cost) / slots, len + cost)
                                     : std::ceil(items / slots) * (len + cost);
        if (sp == 1 || t < best_t) {
            best = sp;
            best_t = t;
        }
        if (items > 8.0 * slots) break;
    }
    return best;
}

template <int D>
cudaError_t launch_d(const EParams& P, long long items, cudaStream_t st) {
    const size_t smem = e_layout(P.d, P.k).total;
    cudaError_t e = cudaFuncSetAttribute(euclid_knn_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)items);
    cfg.blockDim = dim3(kEThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = P.split;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = P.split > 1 && !P.part ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, euclid_knn_kernel<D>, P);
}

}  // namespace

cudaError_t launch_euclid_knn(const float* pts, long long n, int d, const float* qry, long long nq, int k,
                              int predecessor, long long* out_idx, float* out_dist, cudaStream_t st) {
    if (nq <= 0) return cudaSuccess;
    if (small_form(n, nq, d, k, predecessor)) {
        EParams S{};
        S.pts = pts; S.qry = qry; S.n = n; S.nq = nq; S.d = d; S.k = k; S.predecessor = predecessor;
        S.out_idx = out_idx; S.out_dist = out_dist;
        return k <= 16 ? launch_small<16>(S, st) : launch_small<32>(S, st);
    }
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    EParams P{};
    P.pts = pts; P.qry = qry; P.n = n; P.nq = nq; P.d = d; P.k = k; P.predecessor = predecessor;
    P.out_idx = out_idx; P.out_dist = out_dist;
    const long long tiles = (nq + kEQ - 1) / kEQ;
    auto set_split = [&](int sp) {
        P.chunk = std::max<long long>(kEC, ((n + sp - 1) / sp + kEC - 1) / kEC * kEC);
        P.split = (int)std::max<long long>(1, (n + P.chunk - 1) / P.chunk);
        P.sample = sample_steps((double)std::min(P.chunk, n), k, d);
    };
    set_split(choose_split(n, nq, d, k, predecessor, sms));
    // Up to 8 chunks of a tile are a cluster; more need scratch, which a captured call does without.
    unsigned char* scratch = nullptr;
    if (P.split > 8) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        e = cudaStreamIsCapturing(st, &cs);
        if (e != cudaSuccess) return e;
        const size_t done_bytes = (sizeof(int) * (size_t)tiles + 255) & ~size_t(255);
        if (cs != cudaStreamCaptureStatusNone ||
            cudaMallocAsync((void**)&scratch, done_bytes + sizeof(u64) * (size_t)nq * P.split * k, st) != cudaSuccess) {
            cudaGetLastError();
            scratch = nullptr;
            set_split(8);
        } else {
            P.done = (int*)scratch;
            P.part = (u64*)(scratch + done_bytes);
            e = cudaMemsetAsync(P.done, 0, sizeof(int) * (size_t)tiles, st);
        }
    }
    if (e == cudaSuccess) {
        const long long items = tiles * P.split;
        switch (d) {
            case 1: e = launch_d<1>(P, items, st); break;
            case 2: e = launch_d<2>(P, items, st); break;
            case 3: e = launch_d<3>(P, items, st); break;
            case 4: e = launch_d<4>(P, items, st); break;
            case 5: e = launch_d<5>(P, items, st); break;
            case 6: e = launch_d<6>(P, items, st); break;
            case 7: e = launch_d<7>(P, items, st); break;
            case 8: e = launch_d<8>(P, items, st); break;
            default: e = launch_d<0>(P, items, st); break;
        }
    }
    if (scratch) {
        const cudaError_t f = cudaFreeAsync(scratch, st);
        if (e == cudaSuccess) e = f;
    }
    return e;
}

int euclid_max_k() { return kEMaxK; }
int euclid_max_d() { return kEMaxD; }

}  // namespace ct
