// ct_dense.cuh — the plain FP32 dense tile shared by the single-tree kernel
// (ct_brute.cu), the cover-tree build (ct_build.cu) and the batched persistent kernel
// (ct_batch.cu).
//
// A tile is QT queries x a candidate range [cbeg, cend), swept CT candidates at a time;
// each thread holds a QPT x CPT block of query x candidate pairs.  The V dot product of a
// pair is evaluated in the exact order of the reference's `dot_f32_simd_inline`
// (src/metric.rs:601-643): sixteen lane accumulators, lane l summing elements 16c+l in c
// order with a separately rounded multiply and add, then comb[l] = acc0[l] + acc1[l] and
// the horizontal tree ((c0+c4)+(c2+c6)) + ((c1+c5)+(c3+c7)).
//
// What bounds it: 2 m separately rounded FP32 operations per pair on 128 lanes per SM.
//  - Lanes l and l + 8 run as the two halves of one f32x2 chain, so a multiply-add step
//    costs two instructions for two elements (one issue slot per element instead of two)
//    and the issue slots no longer limit the FP32 pipe.  The product is an FMA with a -0
//    addend that the compiler cannot see (a kernel argument): a b + (-0) rounds exactly as
//    a b, and a product made that way cannot be contracted into the following add (an
//    f32x2 multiply can, which would change the bits).
//  - V is stored so that those pairs are adjacent: column s (m/8) + 2c + h of vperm holds
//    element 16c + l, l = bitrev3(s) + 8h, with s the visiting order of the lane pairs that
//    the tree above needs (at most three partial sums are live).
//  - A warp covers 4 QPT queries x 8 CPT candidates (lanes 4 x 8): a 16-byte operand read
//    is one shared-memory wavefront on either side, so the operands of a step take a
//    quarter of the FP32 cycles.
//  - Candidate rows arrive through a ring of `ns` stages of up to `wmax` columns by 16-byte
//    cp.async, running ahead across candidate tiles.
//  - The epilogue bounds |rho| from below the exact arithmetic's cost (approximate square
//    root and exponential with a margin far above their error) and computes the reference's
//    distance only where the pair can still enter the query's top k.  Entering pairs are
//    appended to a per-query buffer; a warp sorts and merges a buffer in registers when it
//    could overflow, instead of merging every candidate tile.
// Measured on GB300 (whole calls): N=32768, m=256, k=50, predecessor mode 12.5 ms (22 TFLOP/s of
// separately rounded operations, 56% of the 39 T/s that these chains reach alone); 30.4 ms with
// one scalar chain per lane, 16 barriers and one merge per 64 candidates.  N=8192, m=64, k=50
// 1.07 ms, 3.31 ms before: at m = 64 the epilogue and the list insertions outweigh the products.
// The same loop with 4 x 4 pairs per thread and half the warps took 20.6 ms (the chains' latency
// shows), with one block per SM 14.1 ms (nothing overlaps the epilogue).
//
// Queries are either dataset rows named by id (qids) or external rows (new
// points: natural-layout V, raw coordinates and p), which the tile permutes,
// scales by the tree's inverse lengthscales and normalises while loading, with
// the arithmetic of the dataset's own setup (ct_setup.cu).
#pragma once
#include <type_traits>

#include "ct_common.cuh"

namespace ct {
namespace dense {

typedef unsigned long long u64;

constexpr u64 kNoKey = ~0ULL;                           // empty list entry: above every (dist, idx) key
constexpr u64 kNegZero2 = 0x8000000080000000ULL;       // (-0, -0): the addend of the packed products
constexpr int kPend = 512;     // pairs of a step that wait for their exact distance (more are evaluated in place)

// Tile configurations: QT queries x CT candidates per step, NT threads.  The 256-thread forms run
// two blocks to an SM, so that one block's epilogue and selection overlap the other's multiply-adds;
// the 512-thread forms take one SM (rows too wide for half an SM's shared memory), and so does a
// launch of the 32-row 256-thread form for rows too wide for the 512-thread one, whose ring and
// buffers are larger.  The 16-row forms serve few queries and the widest rows.
enum Cfg { kCfg32 = 0, kCfg16 = 1, kCfg32w = 2, kCfg16w = 3, kNumCfg = 4 };
template <int C>
struct CfgOf;
template <>
struct CfgOf<kCfg32> { static constexpr int NT = 256, QT = 32, CT = 64, QPT = 4, CPT = 2; };
template <>
struct CfgOf<kCfg16> { static constexpr int NT = 256, QT = 16, CT = 64, QPT = 2, CPT = 2; };
template <>
struct CfgOf<kCfg32w> { static constexpr int NT = 512, QT = 32, CT = 128, QPT = 4, CPT = 2; };
template <>
struct CfgOf<kCfg16w> { static constexpr int NT = 512, QT = 16, CT = 64, QPT = 2, CPT = 1; };
__host__ __device__ inline int cfg_qt(int c) { return c == kCfg32 || c == kCfg32w ? 32 : 16; }
__host__ __device__ inline int cfg_ct(int c) { return c == kCfg32w ? 128 : 64; }
__host__ __device__ inline int cfg_threads(int c) { return c == kCfg32w || c == kCfg16w ? 512 : 256; }

// Column of vperm that holds V column `col` (see the header).
__host__ __device__ __forceinline__ int perm_col(int col, int m) {
    const int c = col >> 4, l = col & 15, rp = l & 7, h = l >> 3;
    const int s = ((rp & 1) << 2) | (rp & 2) | (rp >> 2);
    return s * (m >> 3) + 2 * c + h;
}

// Stage geometry: G lane pairs per stage (NC = 1), or NC stages per lane pair (G = 1).
struct Geo {
    int rw;   // floats of a lane pair in a row (m / 8)
    int G, NC;
    int W;    // floats of a full stage row
    int stages;  // stages of a row
};
// Padded stage row: an odd number of 16-byte units (8 rows read without bank conflicts), the same
// for every m, so that the rows of an operand are immediate offsets from one address.
__host__ __device__ constexpr int stage_stride(int wmax) { return wmax + 4; }
__host__ __device__ inline Geo geometry(int m, int wmax) {
    Geo g;
    g.rw = m >> 3;
    g.G = 1;
    g.NC = 1;
    if (g.rw <= wmax) {
        while (g.G < 8 && g.rw * g.G * 2 <= wmax) g.G *= 2;
        g.W = g.rw * g.G;
    } else {
        g.NC = (g.rw + wmax - 1) / wmax;
        g.W = wmax;
    }
    g.stages = g.NC > 1 ? 8 * g.NC : 8 / g.G;
    return g;
}

// Candidate tiles whose (xs, norms, p) are held: the ring runs at most two stages ahead, into the
// next tile, or the one after it when a tile is one stage.
__host__ __device__ inline int cand_buffers(const Geo& g) { return g.stages >= 2 ? 2 : 3; }

struct Smem {
    // byte offsets
    size_t a, b, buf, list, tau, thr, xq, nq, pq, qid, cnt, cand, pend, npend, total;
};

__host__ __device__ inline Smem layout(int cfg, int m, int d, int k, int ns, int wmax, int slack, int pend) {
    Smem L;
    const int qt = cfg_qt(cfg), ct = cfg_ct(cfg);
    const Geo g = geometry(m, wmax);
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 15) & ~size_t(15); return o; };
    L.a = take(sizeof(float) * qt * g.stages * stage_stride(wmax));  // the query rows, stage by stage
    L.b = take(sizeof(float) * ns * ct * stage_stride(wmax));
    L.buf = take(sizeof(u64) * qt * (ct + slack));
    L.list = take(sizeof(u64) * qt * k);
    L.tau = take(sizeof(u64) * qt);
    L.thr = take(sizeof(float) * qt);
    L.xq = take(sizeof(float) * qt * d);
    L.nq = take(sizeof(float) * qt);
    L.pq = take(sizeof(float) * qt);
    L.qid = take(sizeof(int) * qt);
    L.cnt = take(sizeof(int) * qt);
    L.cand = take(sizeof(float) * cand_buffers(g) * ct * (d + 2));
    L.pend = take((sizeof(float) + sizeof(int)) * pend);
    L.npend = take(2 * sizeof(int));
    L.total = off;
    return L;
}

// Ring depth, stage width, buffer slack and pending pairs of a configuration at (m, d, k): the deepest
// ring and roomiest buffers that fit `limit` bytes (a query's buffer holds CT + slack keys and is merged
// above `slack`); narrow stages are the 16-row forms' last resort, and a short list of pending pairs
// their last (m = 1936 to 1968 with more than 50 coordinates; pairs past it are evaluated in place).
// False when nothing fits.
struct Ring {
    int ns, wmax, slack, pend;
};
__host__ inline bool pick_ring(int cfg, int m, int d, int k, size_t limit, Ring* r, size_t* total) {
    const Ring tries[8] = {{3, 64, 32, kPend}, {3, 64, 16, kPend}, {2, 64, 16, kPend}, {2, 64, 8, kPend},
                           {2, 64, 4, kPend},  {2, 16, 16, kPend}, {2, 16, 4, kPend},  {2, 16, 4, 64}};
    for (const Ring& t : tries) {
        if (t.wmax == 16 && cfg_qt(cfg) != 16) continue;
        const size_t need = layout(cfg, m, d, k, t.ns, t.wmax, t.slack, t.pend).total;
        if (need <= limit) {
            *r = t;
            *total = need;
            return true;
        }
    }
    return false;
}
// Shared memory a block of the configuration may use: half an SM's for the 256-thread forms (1 KiB
// per block is reserved), the per-block limit for the others; `fixed` bytes are the kernel's own.
__host__ inline size_t cfg_limit(int cfg, size_t optin, size_t per_sm, size_t fixed) {
    return (cfg_threads(cfg) == 256 ? per_sm / 2 - 1024 : optin) - fixed;
}

// ---------------------------------------------------------------- cp.async, f32x2
// `bytes` of the 16 (8, 4) are read, the rest is zero-filled (0: a candidate past the range).
__device__ __forceinline__ void cp_async16z(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8z(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4z(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait(int left) {  // at most `left` groups still in flight
    if (left >= 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// acc + a b per component, product and sum rounded separately (nz = (-0, -0), see the header)
__device__ __forceinline__ u64 mul_add2(u64 a, u64 b, u64 acc, u64 nz) {
    u64 p;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(a), "l"(b), "l"(nz));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(acc) : "l"(p), "l"(acc));
    return acc;
}
__device__ __forceinline__ float sum_halves(u64 a) {
    return __fadd_rn(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)));
}

// ---------------------------------------------------------------- top-k lists
// A key is (distance bits, index): distances are non-negative, so keys order as (dist, idx).
__device__ __forceinline__ u64 make_key(float dist, int idx) {
    return ((u64)__float_as_uint(dist) << 32) | (unsigned)idx;
}
// Ascending sort of 32 E keys held by a warp (element e * 32 + lane), bitonic.
template <int E>
__device__ __forceinline__ void warp_sort(u64 (&x)[E]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int f = e ^ (j >> 5);
                    if (f > e) {
                        const bool up = ((e * 32) & k) == 0;
                        const u64 lo = x[e] < x[f] ? x[e] : x[f], hi = x[e] < x[f] ? x[f] : x[e];
                        x[e] = up ? lo : hi;
                        x[f] = up ? hi : lo;
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const u64 o = __shfl_xor_sync(0xffffffffu, x[e], j);
                    const bool up = ((e * 32 + lane) & k) == 0;
                    const bool keep_min = ((lane & j) == 0) == up;
                    x[e] = (x[e] < o) == keep_min ? x[e] : o;
                }
            }
        }
    }
}
// The 32 E smallest of two ascending sequences, ascending, into a.
template <int E>
__device__ __forceinline__ void warp_merge(u64 (&a)[E], const u64 (&b)[E]) {
    const int lane = threadIdx.x & 31;
    u64 t[E];
#pragma unroll
    for (int e = 0; e < E; ++e) t[e] = __shfl_sync(0xffffffffu, b[E - 1 - e], 31 - lane);
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = a[e] < t[e] ? a[e] : t[e];  // bitonic
#pragma unroll
    for (int j = 16 * E; j > 0; j >>= 1) {
        if (j >= 32) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int f = e ^ (j >> 5);
                if (f > e) {
                    const u64 lo = a[e] < a[f] ? a[e] : a[f], hi = a[e] < a[f] ? a[f] : a[e];
                    a[e] = lo;
                    a[f] = hi;
                }
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const u64 o = __shfl_xor_sync(0xffffffffu, a[e], j);
                a[e] = (a[e] < o) == ((lane & j) == 0) ? a[e] : o;
            }
        }
    }
}
// Merge the cnt keys of buf into the sorted list of k keys (one warp; k <= 32 E).
template <int E>
__device__ __forceinline__ void merge_buffer_e(u64* list, int k, const u64* buf, int cnt) {
    const int lane = threadIdx.x & 31;
    u64 a[E];
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = e * 32 + lane < k ? list[e * 32 + lane] : kNoKey;
    for (int base = 0; base < cnt; base += 32 * E) {
        u64 x[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = base + e * 32 + lane;
            x[e] = i < cnt ? buf[i] : kNoKey;
        }
        if (E > 1 && cnt - base <= 32) {  // most buffers: one key per lane to sort
            u64 y[1] = {x[0]};
            warp_sort<1>(y);
            x[0] = y[0];
        } else {
            warp_sort<E>(x);
        }
        warp_merge<E>(a, x);
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (e * 32 + lane < k) list[e * 32 + lane] = a[e];
    __syncwarp();
}
static __device__ __noinline__ void merge_buffer(u64* list, int k, const u64* buf, int cnt) {
    if (k <= 32) merge_buffer_e<1>(list, k, buf, cnt);
    else if (k <= 64) merge_buffer_e<2>(list, k, buf, cnt);
    else merge_buffer_e<4>(list, k, buf, cnt);
}

// Merge S sorted partial lists of k keys (list s at part + s * k) into out_* (one query by nw
// warps of the block, this one their part_w-th; every thread of the block calls).  Lists whose
// head does not beat the current k-th are skipped.  scratch: k keys of shared memory per warp.
// SQRT: the keys hold squared distances.
template <int E, bool SQRT>
__device__ __forceinline__ void merge_lists_e(const u64* part, int S, int k, int part_w, int nw, u64* scratch,
                                              bool active, long long* out_idx, float* out_dist) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 a[E];
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = kNoKey;
    auto take = [&](const u64* src, bool global) {
        u64 x[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = e * 32 + lane;
            x[e] = i < k ? (global ? __ldcg(src + i) : src[i]) : kNoKey;
        }
        u64 kth = a[0];
#pragma unroll
        for (int e = 1; e < E; ++e) kth = ((k - 1) >> 5) == e ? a[e] : kth;
        kth = __shfl_sync(0xffffffffu, kth, (k - 1) & 31);
        const u64 head = __shfl_sync(0xffffffffu, x[0], 0);
        if (head < kth) warp_merge<E>(a, x);
    };
    if (active)
        for (int s = part_w; s < S; s += nw) take(part + (size_t)s * k, true);
    if (nw > 1) {
        if (active)
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (e * 32 + lane < k) scratch[(size_t)warp * k + e * 32 + lane] = a[e];
        __syncthreads();
        if (active && part_w == 0)
            for (int w = 1; w < nw; ++w) take(scratch + (size_t)(warp + w) * k, false);
    }
    if (active && part_w == 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int j = e * 32 + lane;
            if (j < k) {
                out_idx[j] = a[e] == kNoKey ? -1LL : (long long)(unsigned)a[e];
                const float v = __uint_as_float((unsigned)(a[e] >> 32));
                out_dist[j] = a[e] == kNoKey ? CT_FLT_MAX : SQRT ? sqrtf(v) : v;
            }
        }
    }
    if (nw > 1) __syncthreads();  // scratch is free again
}
// Final merge of a query tile by NT threads: queries [g0, g0 + nv), partial lists [query][S][k].
// Fewer queries than warps get several warps each.
template <int NT, bool SQRT = false>
__device__ inline void merge_tile(const u64* part, int S, int k, long long g0, int nv, u64* scratch,
                                  long long* out_idx, float* out_dist, long long out_stride) {
    int nw = 1;
    while (nw * 2 * nv <= NT / 32) nw *= 2;
    const int warp = threadIdx.x >> 5, per = NT / 32 / nw;  // queries per round
    for (int q0 = 0; q0 < nv; q0 += per) {
        const int qi = q0 + warp / nw;
        const bool active = qi < nv;
        const long long g = g0 + (active ? qi : 0);
        const u64* src = part + (size_t)g * S * k;
        long long* oi = out_idx + g * out_stride;
        float* od = out_dist + g * out_stride;
        if (k <= 32) merge_lists_e<1, SQRT>(src, S, k, warp % nw, nw, scratch, active, oi, od);
        else if (k <= 64) merge_lists_e<2, SQRT>(src, S, k, warp % nw, nw, scratch, active, oi, od);
        else merge_lists_e<4, SQRT>(src, S, k, warp % nw, nw, scratch, active, oi, od);
    }
}

struct Tile {
    // candidates: the tree's device-resident metric (ct_setup.cu layout)
    const float* vperm;
    const float* xs;
    const float* norms;
    const float* p;
    long long n;
    int m, d, k, kernel_type, predecessor;
    float var;
    // queries: dataset ids (qids != nullptr) or external rows
    const long long* qids;
    const float* qv;       // external: nq x m, natural column order
    const float* qcoords;  // external: nq x d, unscaled
    const float* qp;       // external: nq
    const float* inv_ls;   // external: d inverse lengthscales of the tree
    long long nq;
    long long q0;          // first query of the tile
    long long cbeg, cend;  // candidate range
    // results: row g writes out_*[g * out_stride + j], j < k; with `part` set, the sorted keys
    // go to part[g * part_stride + j] instead
    long long* out_idx;
    float* out_dist;
    long long out_stride;
    u64* part;
    long long part_stride;
    Ring ring;             // pick_ring
};

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Epilogue test value of a query whose k-th distance is t: the pair cannot have distance <= t
// when (R + eps)^2 < max(p_q p_c, 1e-18) thr, R the approximate |kv - dot|.  dist <= t needs
// |rho| >= 1 - t^2 (1 + 2e-7) - 6e-8 and |rho| = |kv - dot| / sqrt(pp) up to 2e-7; the margins
// below are an order of magnitude wider.  Negative (never skip) when the bound is void.
__device__ __forceinline__ float skip_threshold(float t) {
    const float T = (1.f - t * t * (1.f + 4e-6f)) - 2e-6f;
    return T > 0.f ? T * T * (1.f - 8e-6f) : -1.f;
}

// Place of vperm column `col` in a query row's stages (float offset; stage st of row r is at
// (st * QT + r) * stride).
__device__ __forceinline__ void stage_of(const Geo& g, int col, int& st, int& off) {
    if (g.NC > 1) {
        const int rp = col / g.rw, in = col - rp * g.rw, cc = in / g.W;
        st = rp * g.NC + cc;
        off = in - cc * g.W;
    } else {
        st = col / g.W;
        off = col - st * g.W;
    }
}

// One query tile against its candidate range.  VEC = 4: operands move 16 bytes at a time (m a
// multiple of 32); VEC = 2: 8 bytes (m an odd multiple of 16).  RW > 0: full stages of 64 columns
// (m = 64, 128, 256 or a multiple of 512; RW = 8, 16, 32, 64 columns of a lane pair in a stage),
// whose loads, multiply-adds and folds are straight-line code; RW = 0: any m.  All add the
// products in the same order, so all give the same bits.
// (A function of its own, not inlined: the batched kernel holds one per configuration, each with
// its own registers.)
template <int C, int VEC, int WMAX, int RW>
__device__ __noinline__ void run_tile_v(const Tile& P, u64 nz) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int QT = CfgOf<C>::QT, CT = CfgOf<C>::CT, QPT = CfgOf<C>::QPT, CPT = CfgOf<C>::CPT;
    constexpr int kThreads = CfgOf<C>::NT, kWarps = kThreads / 32;
    constexpr int WQ = QT / (4 * QPT);  // warps along the queries
    static_assert(WQ * (CT / (8 * CPT)) == kWarps, "warps cover the tile");
    constexpr int STR = stage_stride(WMAX);
    const int ns = P.ring.ns, slack = P.ring.slack, CAP = CT + slack;
    const int pend = WMAX == 16 ? P.ring.pend : kPend;
    const Smem S = layout(C, P.m, P.d, P.k, ns, WMAX, slack, pend);
    const Geo g = geometry(P.m, WMAX);
    const int ncand = cand_buffers(g);
    float* As = (float*)(smem_raw + S.a);
    float* Bs = (float*)(smem_raw + S.b);
    u64* Buf = (u64*)(smem_raw + S.buf);
    u64* List = (u64*)(smem_raw + S.list);
    u64* Tau = (u64*)(smem_raw + S.tau);
    float* Thr = (float*)(smem_raw + S.thr);
    float* Xq = (float*)(smem_raw + S.xq);
    float* Nq = (float*)(smem_raw + S.nq);
    float* Pq = (float*)(smem_raw + S.pq);
    int* Qid = (int*)(smem_raw + S.qid);
    int* Cnt = (int*)(smem_raw + S.cnt);
    float* Cand = (float*)(smem_raw + S.cand);
    float* PendDot = (float*)(smem_raw + S.pend);
    int* PendPair = (int*)(PendDot + pend);
    int* Npend = (int*)(smem_raw + S.npend);

    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int qrow = (warp % WQ) * 4 * QPT + (lane >> 3);  // queries qrow + 4a
    const int crow = (warp / WQ) * 8 * CPT + (lane & 7);   // candidates crow + 8b
    const int m = P.m, d = P.d, k = P.k;
    const bool ext = P.qids == nullptr;
    const long long q0 = P.q0;
    const int cl = (int)(P.cend < P.n ? P.cend : P.n);  // candidate limit (n < 2^31)
    const int cb = (int)P.cbeg;

    // ---- query scalars.  Qid: dataset id (internal), row of the call (external), -1 = padding
    for (int qi = tid; qi < QT; qi += kThreads) {
        const long long gq = q0 + qi;
        long long id = -1;
        if (gq < P.nq) {
            id = ext ? gq : P.qids[gq];
            if (!ext && (id < 0 || id >= P.n)) id = -1;  // ids outside [0, n) give an all-padding row
        }
        Qid[qi] = id < 0 ? -1 : ext ? qi : (int)id;
        Cnt[qi] = 0;
        Tau[qi] = id < 0 ? 0ULL : kNoKey;
        Thr[qi] = id < 0 ? __int_as_float(0x7f800000) : -1.f;
        if (ext) {
            float s = 0.f;
            for (int c = 0; c < d; ++c) {
                const float x = id >= 0 ? __fmul_rn(P.qcoords[id * d + c], P.inv_ls[c]) : 0.f;
                Xq[qi * d + c] = x;
                s = __fadd_rn(s, __fmul_rn(x, x));
            }
            Nq[qi] = s;
            Pq[qi] = id >= 0 ? P.qp[id] : 1.f;
        } else {
            Nq[qi] = id >= 0 ? P.norms[id] : 0.f;
            Pq[qi] = id >= 0 ? P.p[id] : 1.f;
        }
    }
    for (int e = tid; e < QT * k; e += kThreads) List[e] = kNoKey;
    if (tid < 2) Npend[tid] = 0;
    __syncthreads();
    // ---- query rows
    if (ext) {
        for (int e = tid; e < QT * m; e += kThreads) {
            const int qi = e / m, col = e - qi * m;
            int st, off;
            stage_of(g, perm_col(col, m), st, off);
            As[(st * QT + qi) * STR + off] = Qid[qi] >= 0 ? P.qv[(q0 + qi) * m + col] : 0.f;
        }
    } else {
        const int mv = m / VEC;  // VEC columns never straddle two stages (W is a multiple of VEC)
        for (int e = tid; e < QT * mv; e += kThreads) {
            const int qi = e / mv, c = (e - qi * mv) * VEC;
            const int id = Qid[qi];
            int st, off;
            stage_of(g, c, st, off);
            float* dst = As + (st * QT + qi) * STR + off;
            const float* src = P.vperm + (long long)id * m + c;
            if (VEC == 4) *(float4*)dst = id >= 0 ? *(const float4*)src : make_float4(0.f, 0.f, 0.f, 0.f);
            else *(float2*)dst = id >= 0 ? *(const float2*)src : make_float2(0.f, 0.f);
        }
        for (int e = tid; e < QT * d; e += kThreads) {
            const int id = Qid[e / d];
            Xq[e] = id >= 0 ? P.xs[(long long)id * d + e % d] : 0.f;
        }
    }
    // ids of the tile (dataset queries): candidates below minq need no predecessor or self test
    int maxq = -1, minq = 0x7fffffff;
    for (int qi = 0; qi < QT; ++qi) {
        const int id = Qid[qi];
        maxq = max(maxq, id);
        minq = id >= 0 ? min(minq, id) : minq;
    }
    const bool pred = P.predecessor && !ext;
    const int jend = pred ? (maxq < 0 ? cb : min(maxq, cl)) : cl;
    const int ntiles = jend > cb ? (jend - cb - 1) / CT + 1 : 0;
    if (ext) minq = 0x7fffffff;

    // ---- candidate stages: stage i holds stage i % stiles of candidate tile i / stiles
    const int stiles = g.stages;
    int is_tile = 0, is_st = 0, is_slot = 0, is_rp = 0, is_cc = 0;  // next stage to issue
    const int wvf = g.W / VEC;  // pieces of a full stage row; this thread's first one and its stride
    const int r0f = tid / wvf, c0f = tid - r0f * wvf, drf = kThreads / wvf, dcf = kThreads - drf * wvf;
    auto issue = [&]() {
        if (is_tile < ntiles) {
            const int j0 = cb + is_tile * CT, rem = cl - j0;  // candidates left
            float* dst = Bs + (size_t)is_slot * CT * STR;
            const int w = g.NC > 1 ? min(g.W, g.rw - is_cc * g.W) : g.W;       // floats of this stage
            const int col = g.NC > 1 ? is_rp * g.rw + is_cc * g.W : is_st * g.W;  // first column of vperm
            const float* src = P.vperm + (long long)j0 * m + col;
            if constexpr (RW > 0) {
                const int r = tid >> 4, c = (tid & 15) * 4;  // 16 pieces a row
                const float* sp = src + (long long)r * m + c;
                float* dp = dst + r * STR + c;
#pragma unroll
                for (int i = 0; i < CT; i += kThreads / 16) {
                    const bool ok = r + i < rem;
                    cp_async16z(dp + i * STR, ok ? sp : P.vperm, ok ? 16 : 0);
                    sp += (kThreads / 16) * (long long)m;
                }
            } else {
                int wv = wvf, r = r0f, c = c0f, dr = drf, dc = dcf;
                if (w != g.W) {  // the short last stage of a wide lane pair
                    wv = w / VEC;
                    r = tid / wv; c = tid - r * wv;
                    dr = kThreads / wv; dc = kThreads - dr * wv;
                }
                while (r < CT) {
                    const bool ok = r < rem;
                    const float* sp = src + (ok ? (long long)r * m : 0LL) + c * VEC;
                    if (VEC == 4) cp_async16z(dst + r * STR + c * VEC, sp, ok ? 16 : 0);
                    else cp_async8z(dst + r * STR + c * VEC, sp, ok ? 8 : 0);
                    r += dr; c += dc;
                    if (c >= wv) { c -= wv; ++r; }
                }
            }
            if (is_st == 0) {
                float* cd = Cand + (size_t)(is_tile % ncand) * CT * (d + 2);
                for (int e = tid; e < CT * d; e += kThreads) {
                    const bool ok = e < (long long)rem * d;
                    cp_async4z(cd + e, P.xs + (ok ? (long long)j0 * d + e : 0LL), ok ? 4 : 0);
                }
                for (int e = tid; e < CT; e += kThreads) {
                    const bool ok = e < rem;
                    cp_async4z(cd + CT * d + e, P.norms + (ok ? j0 + e : 0), ok ? 4 : 0);
                    cp_async4z(cd + CT * (d + 1) + e, P.p + (ok ? j0 + e : 0), ok ? 4 : 0);
                }
            }
            if (++is_cc >= g.NC) { is_cc = 0; ++is_rp; }
            if (++is_st >= stiles) { is_st = 0; is_rp = 0; is_cc = 0; ++is_tile; }
            is_slot = is_slot + 1 == ns ? 0 : is_slot + 1;
        }
        cp_async_commit();
    };
    for (int i = 0; i + 1 < ns; ++i) issue();
    int slot = 0;  // ring slot of the next stage to consume
    const float epsv = 2e-6f * fabsf(P.var);
    const float ee = __int_as_float(0x219392ee);  // 1e-9f * 1e-9f rounded to binary32
    // Exact distance of the pair (query qi, candidate cj of the tile at j0) and its insertion.
    auto offer = [&](int qi, int cj, int j0, float d2, float dot, float pc, bool self) {
        const float dist =
            self ? 0.f : residual_from_parts(kernel_value_batch(d2, P.var, P.kernel_type), dot, Pq[qi], pc);
        const u64 key = make_key(dist, j0 + cj);
        if (key < Tau[qi]) Buf[qi * CAP + atomicAdd(&Cnt[qi], 1)] = key;
    };

    for (int t = 0; t < ntiles; ++t) {
        const int j0 = cb + t * CT;
        // partial sums of the lane tree: h = the pending leaf, sA = c0+c4 / c1+c5, t0 = (c0+c4)+(c2+c6)
        float h[QPT][CPT], sA[QPT][CPT], t0[QPT][CPT];
        u64 acc[QPT][CPT];
        const float* Ap = As + qrow * STR - QT * STR;  // the current stage's rows (moved on when it arrives)
        const float* Bp = Bs;
        int off = 0;  // columns of the stage already summed
        // The stage that arrives now; the slot read before it is free for the stage ns - 1 ahead.
        auto next_stage = [&]() {
            cp_async_wait(ns - 2);
            __syncthreads();
            issue();
            Ap += QT * STR;
            Bp = Bs + (size_t)slot * CT * STR + crow * STR;
            slot = slot + 1 == ns ? 0 : slot + 1;
            off = 0;
        };
        auto step = [&](int c) {
            if (VEC == 4) {
                ulonglong2 av[QPT], bv[CPT];
#pragma unroll
                for (int a = 0; a < QPT; ++a) av[a] = *(const ulonglong2*)(Ap + 4 * a * STR + c);
#pragma unroll
                for (int b = 0; b < CPT; ++b) bv[b] = *(const ulonglong2*)(Bp + 8 * b * STR + c);
#pragma unroll
                for (int a = 0; a < QPT; ++a)
#pragma unroll
                    for (int b = 0; b < CPT; ++b) acc[a][b] = mul_add2(av[a].x, bv[b].x, acc[a][b], nz);
#pragma unroll
                for (int a = 0; a < QPT; ++a)
#pragma unroll
                    for (int b = 0; b < CPT; ++b) acc[a][b] = mul_add2(av[a].y, bv[b].y, acc[a][b], nz);
            } else {
                u64 av[QPT], bv[CPT];
#pragma unroll
                for (int a = 0; a < QPT; ++a) av[a] = *(const u64*)(Ap + 4 * a * STR + c);
#pragma unroll
                for (int b = 0; b < CPT; ++b) bv[b] = *(const u64*)(Bp + 8 * b * STR + c);
#pragma unroll
                for (int a = 0; a < QPT; ++a)
#pragma unroll
                    for (int b = 0; b < CPT; ++b) acc[a][b] = mul_add2(av[a], bv[b], acc[a][b], nz);
            }
        };
        // w columns from `off` on, in blocks of SP steps (no loop control inside a block)
        auto columns = [&](auto sp, int w) {
            constexpr int N = decltype(sp)::value * VEC;
            const int end = off + w;
#pragma unroll 1
            for (; off < end; off += N)
#pragma unroll
                for (int c = 0; c < N; c += VEC) step(off + c);
        };
        // One lane pair (s in visiting order): its chains over the whole row.
        auto lane_pair = [&](int s) {
#pragma unroll
            for (int a = 0; a < QPT; ++a)
#pragma unroll
                for (int b = 0; b < CPT; ++b) acc[a][b] = 0ULL;
            for (int cc = 0; cc < g.NC; ++cc) {
                if (g.NC > 1 || (s & (g.G - 1)) == 0) next_stage();
                const int w = g.NC > 1 ? min(g.W, g.rw - cc * g.W) : g.rw;
                if (VEC == 4 && (w & 7) == 0) columns(std::integral_constant<int, 2>{}, w);
                else columns(std::integral_constant<int, 1>{}, w);
            }
        };
        // comb[l] = acc0[l] + acc1[l], folded into ((c0+c4)+(c2+c6)) + ((c1+c5)+(c3+c7)): the
        // finished lane pair s, and the finished pair of pairs s2, of the tree.
        auto each = [&](auto f) {
#pragma unroll
            for (int a = 0; a < QPT; ++a)
#pragma unroll
                for (int b = 0; b < CPT; ++b) f(a, b);
        };
        auto leaf = [&](bool odd) {
            if (!odd) each([&](int a, int b) { h[a][b] = sum_halves(acc[a][b]); });
            else each([&](int a, int b) { h[a][b] = __fadd_rn(h[a][b], sum_halves(acc[a][b])); });
        };
        auto node = [&](int s2) {
            if (s2 == 0 || s2 == 2) each([&](int a, int b) { sA[a][b] = h[a][b]; });
            else if (s2 == 1) each([&](int a, int b) { t0[a][b] = __fadd_rn(sA[a][b], h[a][b]); });
            else each([&](int a, int b) { h[a][b] = __fadd_rn(t0[a][b], __fadd_rn(sA[a][b], h[a][b])); });  // the dot
        };
        if constexpr (RW > 0) {
            constexpr int G = 64 / RW;  // lane pairs of a stage
#pragma unroll 1
            for (int st = 0; st < 8 / G; ++st) {
                next_stage();
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    each([&](int a, int b) { acc[a][b] = 0ULL; });
#pragma unroll
                    for (int c = 0; c < RW; c += 4) step(i * RW + c);
                    if constexpr (RW == 64) {  // the rest of a lane pair wider than a stage
                        for (int cc = 1; cc < g.NC; ++cc) {
                            next_stage();
#pragma unroll
                            for (int c = 0; c < RW; c += 4) step(c);
                        }
                    }
                    leaf(G == 1 ? (st & 1) : (i & 1));
                    if (G >= 2 && (i & 1)) {
                        if (G == 8) node(i >> 1);
                        else if (G == 4) node(2 * st + (i >> 1));
                        else node(st);
                    }
                }
                if (G == 1 && (st & 1)) node(st >> 1);
            }
        } else {
#pragma unroll 1
            for (int s2 = 0; s2 < 4; ++s2) {
                lane_pair(2 * s2);
                leaf(false);
                lane_pair(2 * s2 + 1);
                leaf(true);
                node(s2);
            }
        }
        // ---- epilogue
        const float* cx = Cand + (size_t)(t % ncand) * CT * (d + 2);
        const float* cn = cx + CT * d;
        const float* cp = cn + CT;
        float xd[QPT][CPT];  // x_q . x_c, left to right
        for (int c = 0; c < d; ++c) {
            float xc[CPT];
#pragma unroll
            for (int b = 0; b < CPT; ++b) xc[b] = cx[(crow + 8 * b) * d + c];
#pragma unroll
            for (int a = 0; a < QPT; ++a) {
                const float x = Xq[(qrow + 4 * a) * d + c];
#pragma unroll
                for (int b = 0; b < CPT; ++b) {
                    const float pr = __fmul_rn(x, xc[b]);
                    xd[a][b] = c == 0 ? pr : __fadd_rn(xd[a][b], pr);
                }
            }
        }
        float nc[CPT], pc[CPT];
#pragma unroll
        for (int b = 0; b < CPT; ++b) { nc[b] = cn[crow + 8 * b]; pc[b] = cp[crow + 8 * b]; }
        const bool edge = cl - j0 < CT || (!ext && minq - j0 < CT);  // some pair may be invalid or the query itself
        unsigned pass = 0;  // pairs that may enter their query's list
#pragma unroll
        for (int a = 0; a < QPT; ++a) {
            const int qi = qrow + 4 * a;
            const float nq = Nq[qi], pq = Pq[qi], thr = Thr[qi];
#pragma unroll
            for (int b = 0; b < CPT; ++b) {
                float d2 = __fsub_rn(__fadd_rn(nq, nc[b]), __fmul_rn(2.0f, xd[a][b]));
                d2 = d2 < 0.f ? 0.f : d2;
                xd[a][b] = d2;
                float kva;
                if (P.kernel_type == 0) {
                    kva = P.var * __expf(-0.5f * d2);
                } else {
                    const float ar = 2.2360679775f * sqrt_approx(d2);
                    kva = P.var * fmaf(ar * ar, 0.3333333333f, 1.f + ar) * __expf(-ar);
                }
                const float R = fabsf(kva - h[a][b]) + epsv;
                const float pp = __fmul_rn(pq, pc[b]);
                if (!(R * R < (pp > ee ? pp : ee) * thr)) pass |= 1u << (a * CPT + b);
            }
        }
        if (edge) {
#pragma unroll
            for (int a = 0; a < QPT; ++a) {
                const int qi = qrow + 4 * a, gq = Qid[qi];
#pragma unroll
                for (int b = 0; b < CPT; ++b) {
                    const int cj = crow + 8 * b, gc = j0 + cj;
                    const unsigned bit = 1u << (a * CPT + b);
                    if (cj >= cl - j0 || gq < 0 || (pred && gc >= gq)) pass &= ~bit;
                    else if (!ext && gc == gq) {
                        pass &= ~bit;
                        offer(qi, cj, j0, 0.f, 0.f, 0.f, true);
                    }
                }
            }
        }
        // Few pairs pass once the lists have filled.  They wait in a list that the whole block then
        // works off, one pair per thread, instead of each holding its warp through the exact
        // arithmetic (a division and three square roots).
        int* npend = Npend + (t & 1);
#pragma unroll
        for (int a = 0; a < QPT; ++a)
#pragma unroll
            for (int b = 0; b < CPT; ++b) {
                const bool mine = pass >> (a * CPT + b) & 1u;
                const unsigned who = __ballot_sync(0xffffffffu, mine);
                if (who == 0u) continue;
                int at = 0;
                if (lane == 0) at = atomicAdd(npend, __popc(who));
                at = __shfl_sync(0xffffffffu, at, 0) + __popc(who & ((1u << lane) - 1u));
                if (mine) {
                    if (at < pend) {
                        PendDot[at] = h[a][b];
                        PendPair[at] = (qrow + 4 * a) << 16 | (crow + 8 * b);
                    } else {
                        offer(qrow + 4 * a, crow + 8 * b, j0, xd[a][b], h[a][b], pc[b], false);
                    }
                }
            }
        __syncthreads();
        const int np = min(*npend, pend);
        if (tid == 0) Npend[(t & 1) ^ 1] = 0;
        if (np > 0) {
            for (int i = tid; i < np; i += kThreads) {
                const int qi = PendPair[i] >> 16, cj = PendPair[i] & 0xffff;
                const float d2 = coord_d2_batch(Xq + qi * d, cx + cj * d, d, Nq[qi], cn[cj]);
                offer(qi, cj, j0, d2, PendDot[i], cp[cj], false);
            }
            __syncthreads();
        }
        // ---- selection: warp w owns queries w, w + 8, ...; a buffer that the next tile could
        // overflow is merged (the last tile's buffers all are)
        const int trig = t + 1 < ntiles ? slack : 0;
        for (int qi = warp; qi < QT; qi += kWarps) {
            const int cnt = Cnt[qi];
            if (cnt <= trig) continue;
            merge_buffer(List + qi * k, k, Buf + qi * CAP, cnt);
            if (lane == 0) {
                const u64 kth = List[qi * k + k - 1];
                Cnt[qi] = 0;
                Tau[qi] = kth;
                Thr[qi] = kth == kNoKey ? -1.f : skip_threshold(__uint_as_float((unsigned)(kth >> 32)));
            }
        }
    }
    __syncwarp();
    // ---- results (dataset ids; -1 / FLT_MAX padding), each query by the warp that owns its list
    for (int qi = warp; qi < QT; qi += kWarps) {
        const long long gq = q0 + qi;
        if (gq >= P.nq) continue;
        for (int j = lane; j < k; j += 32) {
            const u64 key = List[qi * k + j];
            if (P.part) {
                P.part[gq * P.part_stride + j] = key;
            } else {
                P.out_idx[gq * P.out_stride + j] = key == kNoKey ? -1LL : (long long)(unsigned)key;
                P.out_dist[gq * P.out_stride + j] = key == kNoKey ? CT_FLT_MAX : __uint_as_float((unsigned)(key >> 32));
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

template <int C>
__device__ __forceinline__ void run_tile(const Tile& P, u64 nz) {
    if constexpr (C == kCfg32 || C == kCfg16) {  // (wider rows take the general loop or the 512-thread forms)
        if (P.ring.wmax == 64) {
            if (P.m == 64) return run_tile_v<C, 4, 64, 8>(P, nz);
            if (P.m == 128) return run_tile_v<C, 4, 64, 16>(P, nz);
            if (P.m == 256) return run_tile_v<C, 4, 64, 32>(P, nz);
        }
    } else {
        if (P.ring.wmax == 64 && (P.m & 511) == 0) return run_tile_v<C, 4, 64, 64>(P, nz);
    }
    if ((P.m & 31) == 0) {
        if (P.ring.wmax == 64) return run_tile_v<C, 4, 64, 0>(P, nz);
        if constexpr (CfgOf<C>::QT == 16) run_tile_v<C, 4, 16, 0>(P, nz);
    } else {
        if (P.ring.wmax == 64) return run_tile_v<C, 2, 64, 0>(P, nz);
        if constexpr (CfgOf<C>::QT == 16) run_tile_v<C, 2, 16, 0>(P, nz);
    }
}

}  // namespace dense
}  // namespace ct
