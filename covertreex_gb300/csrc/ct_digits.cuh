// ct_digits.cuh — exhaustive pass of the screened form on the tensor cores (included by
// ct_screen.cu, inside ct::screen).
//
// A query whose survivor list overflowed in the BF16 sweep (its residual variance is so small
// that the sweep's bound excludes nothing) is searched again over all its candidates with dot
// products that are exact up to 2e-9 or so: V as fixed-point numbers of five balanced 7-bit
// digits, v 2^-e = sum_i a_i 2^(-6 - 7 i), |a_i| <= 64.  Digits are exact BF16 values, a product
// of two is at most 2^12, and the products of one order s = i + j (at most 5 of them, over m
// columns) sum to integers below 2^24 for m <= kDigitMaxM: FP32 accumulation in the tensor core
// is exact.  Orders 0 .. 5 (19 products) have an accumulator each; what is left out is
//   sum over i + j >= 6:  at most 3.02 m 2^(12 - 54) 2^(2e), and
//   the digits' remainder: half a unit of 2^-34 per element, at most 2^(e - 35) sqrt(m) (|v_q| + |v_c|).
// The epilogue adds the accumulators exactly enough and evaluates the kernel value to kKvErr
// (f32x2 double-float steps on two candidates at a time), which gives certified bounds of |rho| some
// 30000 times tighter than the sweep's.
//
// Pass A sweeps every kDigitSample-th tile for thresholds only: each (row, chunk, group
// of columns) keeps its smallest upper bound of d^2; these belong to different candidates, so the
// k-th smallest of them bounds the k-th distance.  Pass B sweeps every tile and keeps the candidates
// whose lower bound reaches the threshold; the survivor pass (rescore_kernel) finishes them with
// the same exact distances as any other survivor.
//
// Layout: 128 queries x 64 candidates per tile, K in stages of 16 columns (one bulk copy for all digits of
// the queries' block, one for the candidates'), 7 MMAs a stage (a digit of the queries with up to four
// digits of the candidates is one product of N = 256), six accumulators of 64 columns.  The epilogue first
// moves the dots to shared memory as double-float, so that the next tile's products overlap its kernel
// values.  Row tiles are cut into chunks of equal size, dealt to one CTA per SM largest first.
//
// What bounds it: the tensor pipe, 64% active (304 clocks of products per 16 columns and tile against
// about 490).  Measured: 1024 queries over n = 32768, m = 512, D = 3, pass B 0.43 ms; with one MMA per
// pair of digits 0.75, with the kernel value in the exact distances' arithmetic 1.6, the epilogue not
// overlapped.  The compensated FP32 kernels need 9 ms for the same queries.  Whole calls: that one 11.3 ms
// before, 2.7 with this pass; n = 262144, m = 512, 1102 such queries 132 and 108; 4096 points against
// n = 131072, m = 256, 55 such queries 4.3 and 3.7.

constexpr int DS = 5;                       // digits
constexpr int DO = 6;                       // orders kept
constexpr int DN = 64;                      // candidates of a tile
constexpr int DSTAGES = 4;
constexpr int DK = 16;                      // columns of a stage: one MMA of each product
constexpr int DCHUNK_A = TQ * DK * 2, DCHUNK_B = DN * DK * 2;  // bytes of a digit's K-chunk
constexpr int DSTAGE_BYTES = DS * (DCHUNK_A + DCHUNK_B);
constexpr int kDigitMaxM = 800;             // 5 m 2^12 < 2^24
constexpr int kDigitSample = 4;
constexpr int kDigitDense = 128;            // tiles of pass A before it samples
constexpr int kDigitThreads = 64 + kEpiThreads;
constexpr int kDigitCap = 2048;             // survivors per (row, column half)
constexpr int kDigitMaxChunks = 304;        // of a row tile's candidates
constexpr int kDigitGroups = 4;             // column groups of a half with a minimum each
constexpr int kDigitCols = 4;               // columns of an accumulator load
constexpr int kCandF = 4 * kMaxD + 4;       // floats of two candidates: (h, h', l, l') of each scaled coordinate,
                                            // then 1/sqrt(p) and |v| of both
constexpr float kKvErr = 4e-10f;            // of the kernel value / variance (see kernel_mid2)

struct DigitParams {
    const bf16* a;       // digits of the queries, tiles of TQ rows
    const bf16* b;       // digits of the candidates (dataset order), tiles of DN rows
    const int* qid;      // row -> dataset id of its query (-1 padding)
    const int* qidx;     // row -> query of the call (index into qtau)
    const int4* items;   // (row tile, chunk, chunks of the row tile, chunks of the row tiles before)
    const int* cta_begin;  // items of a CTA: [cta_begin[b], cta_begin[b + 1])
    const int2* tile_chunks;  // per row tile: (chunks, chunks of the row tiles before)
    const long long* cend;  // per row tile: candidates [0, cend)
    int ntiles;          // candidate tiles of b
    const float* scale;  // 2^e
    float nz;            // -0: a product as fma(x, y, -0) is never contracted with what follows
    int* surv; float* survb; int* cnt;  // [row][2][kDigitCap], [row][2]
    float* minima;       // per row tile: [row][chunk][2][kDigitGroups]
    long long base;      // dataset row of b's row 0
    int* status;
};

struct DigitSmem {
    size_t stages, mins, cand, dots, tab, bars, tmem_slot, total;
};
__host__ __device__ inline DigitSmem digit_smem() {
    DigitSmem L;
    size_t off = 0;
    L.stages = off; off += (size_t)DSTAGES * DSTAGE_BYTES;
    L.mins = off; off += sizeof(float) * kDigitGroups * kEpiThreads;
    L.cand = off; off += sizeof(float) * kCandF * 16 * kEpiWarps;
    L.dots = off; off += sizeof(float2) * (DN / 2) * kEpiThreads;
    L.tab = off; off += sizeof(float2) * 16;
    L.bars = off; off += (2 * DSTAGES + 3) * 8;
    L.tmem_slot = off; off += 16;
    L.total = off + 1024;
    return L;
}

// Scale of the search, from the largest row norm (so of every |v|) of the dataset and the queries, which is
// below kDigitMaxNorm (digit_fit).
__global__ void digit_scale_kernel(const unsigned* __restrict__ vn_max, float* __restrict__ scale) {
    const float v = __uint_as_float(*vn_max);
    int e = 0;
    if (v > 0.f) frexpf(v * 0.9924f, &e);  // v < 64.5 / 64 2^e: the leading digit is at most 64
    *scale = ldexpf(1.f, e > -50 ? e : -50);
}
__global__ void gather_max_bits_kernel(const float* __restrict__ x, const int* __restrict__ rows, long long n,
                                       unsigned* __restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n && rows[i] >= 0) atomicMax(out, __float_as_uint(x[rows[i]]));
}

// Element offset in a digit matrix of tr-row tiles: a tile's K-block of DK columns holds its digits one after
// another (one bulk copy brings all of them), each as row groups of 8 of core matrices of 8 x 8.
__host__ __device__ inline size_t digit_offset(long long row, int col, int digit, int tr, int m) {
    const long long block = row / tr * (m / DK) + col / DK;
    return ((size_t)block * DS + digit) * (size_t)(tr * DK) + (row % tr >> 3) * (8 * DK) + ((col >> 3) & 1) * 64 +
           (row & 7) * 8 + (col & 7);
}

// Digits of V rows in that layout, in tiles of tr: row r < rows is V row rowmap[r] (none:
// row0 + r); negative entries and the rows up to rows_pad are zero.  A warp takes 16 rows x 16 columns, so
// that a digit's 512 bytes are contiguous (n = 262144, m = 512: 0.29 ms, 6.5 TB/s; 1.2 with lanes along a row).
__global__ void digit_split_kernel(const float* __restrict__ v, int m, const int* __restrict__ rowmap, long long row0,
                                   long long rows, long long rows_pad, int tr, const float* __restrict__ scale,
                                   bf16* __restrict__ out) {
    const float inv = 64.f / *scale;
    const int blocks = m / DK;
    const long long total = rows_pad / 16 * blocks * 32;  // rows_pad: a multiple of 64
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long g = (t >> 5) / blocks;
        const long long r = g * 16 + (t >> 4 & 1) * 8 + (t & 7);
        const int col = (int)((t >> 5) - g * blocks) * DK + (int)(t >> 3 & 1) * 8;
        const int src = r >= rows ? -1 : rowmap ? rowmap[r] : (int)(row0 + r);
        float x[8];
        load8(v, src, m, col, x);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] *= inv;  // exact
        const size_t off = digit_offset(r, col, 0, tr, m);
#pragma unroll
        for (int s = 0; s < DS; ++s) {
            __align__(16) bf16 dg[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float a = rintf(x[e]);
                dg[e] = __float2bfloat16_rn(a);
                x[e] = (x[e] - a) * 128.f;  // exact: a remainder of at most 1/2, shifted
            }
            *(uint4*)(out + off + (size_t)s * tr * DK) = *(const uint4*)dg;
        }
    }
}

// Four columns of the tile: the row's accumulators of the six orders.
__device__ __forceinline__ void digit_orders(uint32_t taddr, float (&o)[DO][kDigitCols]) {
    uint32_t r[DO * kDigitCols];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%24];\n"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%25];\n"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%26];\n"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12,%13,%14,%15}, [%27];\n"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16,%17,%18,%19}, [%28];\n"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20,%21,%22,%23}, [%29];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
        : "r"(taddr), "r"(taddr + DN), "r"(taddr + 2 * DN), "r"(taddr + 3 * DN), "r"(taddr + 4 * DN),
          "r"(taddr + 5 * DN)
        : "memory");
#pragma unroll
    for (int i = 0; i < DO * kDigitCols; ++i) o[i / kDigitCols][i % kDigitCols] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float2 two2(float a) { return make_float2(a, a); }
// a - b, a + b with the rounding errors (TwoSum) of two sums at once.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, two2(-1.f), a); }
__device__ __forceinline__ float2 two_sum2(float2 a, float2 b, float2& err) {
    const float2 s = __fadd2_rn(a, b), z = sub2(s, a);
    err = __fadd2_rn(sub2(a, sub2(s, z)), sub2(b, z));
    return s;
}

// Kernel values of two pairs, as sums kh + kl, from (h, h', l, l') of the candidates' coordinates and
// (h, l) of the negated query's; the coordinates are scaled so that their squared distance is d2 / 2
// (RBF) or 5 d2 (Matern 5/2).  Squared distance in double-float; e^x = 2^q T[j] (1 + r + r^2/2 + ...)
// with x = (16 q + j) ln2/16 + r, ln2/16 in two parts (the products of the first are exact), T in
// double-float, and the series to r^5 in FP32 on terms below 2.4e-4.  |error| <= 1.1e-10 of the variance
// (largest over 2e5 random pairs for each of 48 forms, scales 1e-3 to 1e3, D = 1, 3, 8, against an 80-bit
// evaluation); kKvErr is used.
template <int KT, int DP>
__device__ __forceinline__ void kernel_mid2(const float4* cand, const float2 (&nq)[DP], const float2* tab, float2 nz,
                                            float2& kh, float2& kl) {
    float2 S = two2(0.f), C = two2(0.f);
#pragma unroll
    for (int a = 0; a < DP; ++a) {
        const float4 c = cand[a];
        const float2 ch = make_float2(c.x, c.y);
        float2 e;
        const float2 s0 = two_sum2(ch, two2(nq[a].x), e);
        const float2 l0 = __fadd2_rn(e, __fadd2_rn(make_float2(c.z, c.w), two2(nq[a].y)));
        const float2 s = __fadd2_rn(s0, l0), l = sub2(l0, sub2(s, s0));
        const float2 p = __ffma2_rn(s, s, nz);
        const float2 pe = __ffma2_rn(__fadd2_rn(s, s), l, __ffma2_rn(s, s, __ffma2_rn(p, two2(-1.f), nz)));
        float2 se;
        S = two_sum2(S, p, se);
        C = __fadd2_rn(__fadd2_rn(C, pe), se);
    }
    if (KT == 1) {  // a = sqrt(5 d2): one Newton step from S rsqrt(S)
        S = make_float2(fmaxf(S.x, 1e-30f), fmaxf(S.y, 1e-30f));
        float2 r;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(S.x));
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(S.y));
        const float2 h = __ffma2_rn(S, r, nz);
        const float2 res = __fadd2_rn(__ffma2_rn(__ffma2_rn(h, two2(-1.f), nz), h, S), C);
        C = __ffma2_rn(res, __ffma2_rn(r, two2(0.5f), nz), nz);
        S = h;
    }
    // beyond e^-86 the value is 0 at this accuracy
    C = make_float2(S.x > 86.f ? 0.f : C.x, S.y > 86.f ? 0.f : C.y);
    S = make_float2(fminf(S.x, 86.f), fminf(S.y, 86.f));
    constexpr float kL1 = 2839.f / 65536.f;  // ln2 / 16 to 12 bits, and the rest
    constexpr float kL2 = (float)(0.69314718055994530942 / 16 - 2839.0 / 65536.0);
    const float2 t = __ffma2_rn(S, two2(-23.083120654223414f), two2(12582912.f));
    const float2 n = __fadd2_rn(t, two2(-12582912.f));
    const float2 r0 = __ffma2_rn(n, two2(-kL1), __ffma2_rn(S, two2(-1.f), nz));
    const float2 rl = __ffma2_rn(n, two2(-kL2), __ffma2_rn(C, two2(-1.f), nz));
    const float2 rs = __fadd2_rn(r0, rl), er = sub2(rl, sub2(rs, r0));
    float2 w = __ffma2_rn(rs, two2(1.f / 120.f), two2(1.f / 24.f));
    w = __ffma2_rn(rs, w, two2(1.f / 6.f));
    w = __ffma2_rn(rs, w, two2(0.5f));
    const float2 pl = __ffma2_rn(__ffma2_rn(rs, rs, nz), w, er);
    const int bx = __float_as_int(t.x), by = __float_as_int(t.y);
    const float2 tx = tab[bx & 15], ty = tab[by & 15];
    const float2 f = make_float2(__int_as_float((int)((unsigned)(bx >> 4) << 23) + 0x3f800000),
                                 __int_as_float((int)((unsigned)(by >> 4) << 23) + 0x3f800000));
    const float2 th = make_float2(tx.x, ty.x), tl = make_float2(tx.y, ty.y);
    const float2 p = __ffma2_rn(th, rs, nz);
    const float2 pe = __ffma2_rn(th, rs, __ffma2_rn(p, two2(-1.f), nz));
    const float2 s = __fadd2_rn(th, p), e = __fadd2_rn(p, sub2(th, s));
    const float2 lo = __fadd2_rn(__ffma2_rn(tl, rs, tl), __ffma2_rn(th, pl, __fadd2_rn(e, pe)));
    if (KT == 0) {
        kh = __ffma2_rn(s, f, nz);
        kl = __ffma2_rn(lo, f, nz);
        return;
    }
    // (1 + a + a^2 / 3) e^-a
    constexpr float k3h = (float)(1.0 / 3.0), k3l = (float)(1.0 / 3.0 - (double)(float)(1.0 / 3.0));
    const float2 q = __ffma2_rn(S, S, nz);
    const float2 qe = __ffma2_rn(__fadd2_rn(S, S), C, __ffma2_rn(S, S, __ffma2_rn(q, two2(-1.f), nz)));
    const float2 u = __ffma2_rn(q, two2(k3h), nz);
    const float2 ue = __ffma2_rn(qe, two2(k3h), __ffma2_rn(q, two2(k3l), __ffma2_rn(q, two2(k3h), __ffma2_rn(u, two2(-1.f), nz))));
    float2 e1, e2;
    const float2 s1 = two_sum2(two2(1.f), S, e1), s2 = two_sum2(s1, u, e2);
    const float2 pol = __fadd2_rn(__fadd2_rn(e1, e2), __fadd2_rn(C, ue));
    const float2 k = __ffma2_rn(s2, s, nz);
    const float2 ke = __ffma2_rn(pol, s, __ffma2_rn(s2, lo, __ffma2_rn(s2, s, __ffma2_rn(k, two2(-1.f), nz))));
    kh = __ffma2_rn(k, f, nz);
    kl = __ffma2_rn(ke, f, nz);
}

// KEEP = false: pass A (minima); true: pass B (survivors).  KT: kernel type; DP: coordinates read per
// candidate.
template <bool KEEP, int KT, int DP>
__global__ void __launch_bounds__(kDigitThreads, 1) digit_sweep_kernel(DigitParams P, RescoreParams R) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (sm::smem_u32(smem_raw) & 1023u)) & 1023u);
    const DigitSmem L = digit_smem();
    unsigned char* stage_base = smem + L.stages;
    float* mins = (float*)(smem + L.mins);
    float* cands = (float*)(smem + L.cand);
    float2* tab = (float2*)(smem + L.tab);
    float2* dots = (float2*)(smem + L.dots);
    uint64_t* full = (uint64_t*)(smem + L.bars);
    uint64_t* empty = full + DSTAGES;
    uint64_t* accf = empty + DSTAGES;
    uint64_t* acce = accf + 1;
    uint64_t* done = acce + 1;
    uint32_t* tmem_slot = (uint32_t*)(smem + L.tmem_slot);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = R.m / DK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < DSTAGES; ++s) { sm::mbar_init(&full[s], 1); sm::mbar_init(&empty[s], 1); }
        sm::mbar_init(accf, 1);
        sm::mbar_init(acce, kEpiWarps);
        sm::mbar_init(done, 1);
        sm::fence_barrier_init();
    }
    if (threadIdx.x < 16) {  // 2^(j / 16) in double-float
        const double x = exp2(threadIdx.x * 0.0625);
        tab[threadIdx.x] = make_float2((float)x, (float)(x - (double)(float)x));
    }
    if (warp == 1) {
        sm::tmem_alloc(tmem_slot, 512);
        sm::tmem_relinquish();
    }
    sm::tc_fence_before();
    __syncthreads();
    sm::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Candidate tiles of an item: every nch-th of the row tile's list from the chunk's own, so that the
    // minima of a row with few candidates spread over many chunks too.  Pass B lists every tile; pass A every
    // kDigitSample-th, but in predecessor search all of the first kDigitDense, since early rows have no
    // others.
    const int dense = R.predecessor ? kDigitDense : 0;
    auto range = [&](const int4& it, int& t1) {
        long long left = P.cend[it.x] - P.base;  // of this slab
        left = left < 0 ? 0 : (left + DN - 1) / DN;
        t1 = left < P.ntiles ? (int)left : P.ntiles;
        if (!KEEP && t1 > dense) t1 = dense + (t1 - dense + kDigitSample - 1) / kDigitSample;
    };
    auto tile_of = [&](int t) { return KEEP || t < dense ? t : dense + (t - dense) * kDigitSample; };
    const int item0 = P.cta_begin[blockIdx.x], item1 = P.cta_begin[blockIdx.x + 1];

    if (warp == 0) {
        if (lane == 0) {
            long long it = 0;
            bool alive = true;
            for (int item = item0; alive && item < item1; ++item) {
                const int4 im = P.items[item];
                int t1;
                range(im, t1);
                for (int t = im.y; alive && t < t1; t += im.z)
                    for (int c = 0; c < nk; ++c, ++it) {
                        const int s = (int)(it % DSTAGES);
                        if (!sm::mbar_wait(&empty[s], (unsigned)((it / DSTAGES) & 1) ^ 1u, P.status, 31)) { alive = false; break; }
                        unsigned char* dst = stage_base + (size_t)s * DSTAGE_BYTES;
                        sm::mbar_arrive_expect_tx(&full[s], DSTAGE_BYTES);
                        sm::bulk_g2s(dst, P.a + digit_offset((long long)im.x * TQ, c * DK, 0, TQ, R.m), DS * DCHUNK_A, &full[s]);
                        sm::bulk_g2s(dst + DS * DCHUNK_A, P.b + digit_offset((long long)tile_of(t) * DN, c * DK, 0, DN, R.m),
                                     DS * DCHUNK_B, &full[s]);
                    }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            static_assert(256 / DN == DS - 1, "the last digit's product with i = 1 is one of its own");
            long long it = 0;
            int lt = 0;
            bool alive = true;
            for (int item = item0; alive && item < item1; ++item) {
                const int4 im = P.items[item];
                int t1;
                range(im, t1);
                for (int t = im.y; alive && t < t1; t += im.z, ++lt) {
                    if (!sm::mbar_wait(acce, (unsigned)(lt & 1) ^ 1u, P.status, 32)) { alive = false; break; }
                    sm::tc_fence_after();
                    for (int c = 0; c < nk; ++c, ++it) {
                        const int s = (int)(it % DSTAGES);
                        if (!sm::mbar_wait(&full[s], (unsigned)((it / DSTAGES) & 1), P.status, 33)) { alive = false; break; }
                        sm::tc_fence_after();
                        unsigned char* st = stage_base + (size_t)s * DSTAGE_BYTES;
                        // digit i of the queries with digits 0 .. nj-1 of the candidates is one product with
                        // N = 64 nj: both the candidates' digits in shared memory and the orders i .. i + nj - 1
                        // in TMEM follow one another
#pragma unroll
                        for (int i = 0; i < DS; ++i) {
                            const uint64_t da = sm::smem_desc(st + i * DCHUNK_A, 128, 256);
                            constexpr int most = 256 / DN;  // digits of a product
                            const int nj = DO - i < DS ? DO - i : DS;
#pragma unroll
                            for (int j = 0; j < nj; j += most) {
                                const uint64_t db = sm::smem_desc(st + DS * DCHUNK_A + j * DCHUNK_B, 128, 256);
                                const int cols = (nj - j < most ? nj - j : most) * DN;
                                // the first product of an order starts its accumulator (order 5 starts at i = 1)
                                const bool first = c == 0 && (i == 0 || (i == 1 && j == DS - 1));
                                sm::mma_bf16(tmem_base + (uint32_t)((i + j) * DN), da, db, sm::idesc_bf16_f32(TQ, cols), !first);
                            }
                        }
                        sm::mma_commit(&empty[s]);
                    }
                    if (alive) sm::mma_commit(accf);
                }
            }
            sm::mma_commit(done);
            sm::mbar_wait(done, 0, P.status, 34);
        }
    } else {
        const int ew = warp - 2, quarter = warp & 3, half = ew >> 2;
        const int row = quarter * 32 + lane, et = ew * 32 + lane;
        float* cand = cands + ew * 16 * kCandF;
        const float sc = *P.scale, sc2 = sc * sc;
        const float2 nz = two2(P.nz);
        // coordinate scale: 1 / l times sqrt(1/2) (RBF) or sqrt(5)
        df il[DP];
#pragma unroll
        for (int a = 0; a < DP; ++a) {
            constexpr double f = KT == 0 ? 0.70710678118654752440 : 2.23606797749978969641;
            il[a] = a < R.d ? df_mul(df{R.inv_ls_df[2 * a], R.inv_ls_df[2 * a + 1]}, df{(float)f, (float)(f - (double)(float)f)})
                            : df{0.f, 0.f};
        }
        // The dot's error: left-out products, the FP32 sums with the orders 3 .. 5 (three
        // roundings of at most m 2^-43), remainders of the digits.  The kernel value's: kKvErr, and the rounding of the scaled coordinates (2^-46).
        const float xm = __uint_as_float(__ldg(R.xmax_max)), dd = (float)R.d;
        const float e0 = 4.7f * (float)R.m * 0x1p-42f * sc2 + 1e-12f * sc2;
        const float e1 = 1.02f * 0x1p-35f * sc * sqrtf((float)R.m);
        int lt = 0;
        bool alive = true;
        for (int item = item0; alive && item < item1; ++item) {
            const int4 im = P.items[item];
            const int rt = im.x;
            int t1;
            range(im, t1);
            const long long grow = (long long)rt * TQ + row;
            const int q = P.qid[grow], qi = P.qidx[grow];
            float2 nq[DP];
#pragma unroll
            for (int a = 0; a < DP; ++a) {
                const df u = df_mulf(il[a], q >= 0 && a < R.d ? R.coords[(size_t)q * R.d + a] : 0.f);
                nq[a] = make_float2(-u.h, -u.l);
            }
            const float isq = q >= 0 ? R.isp[q] : 1.f, vnq = q >= 0 ? R.vn[q] : 0.f;
            const float eq = (e0 + e1 * vnq + R.var * (kKvErr + 1e-13f * dd * (xm + (q >= 0 ? R.xmax[q] : 0.f)))) * 1.01f;
            const int lim = q < 0 ? 0 : R.predecessor ? q : (int)R.n;
            const float tq = q >= 0 ? __uint_as_float(__ldcg(&R.qtau[qi])) : 0.f;
            const float thr = (1.f - tq) * (1.f - 2e-6f) / isq;
            if (!KEEP)
                for (int i = 0; i < kDigitGroups; ++i) mins[i * kEpiThreads + et] = tq;  // itself a bound
            for (int t = im.y; t < t1; t += im.z, ++lt) {
                const int c0 = (int)P.base + tile_of(t) * DN + half * (DN / 2);
                {  // the half's candidates, one per lane, while the products are summed
                    const int c = c0 + lane;
                    const bool in = c < (int)R.n;
                    float x[DP];
#pragma unroll
                    for (int a = 0; a < DP; ++a) x[a] = in && a < R.d ? __ldg(R.coords + (size_t)c * R.d + a) : 0.f;
                    const float isc = in ? __ldg(R.isp + c) : 0.f, vnc = in ? __ldg(R.vn + c) : 0.f;
                    float* w = cand + (lane >> 1) * kCandF + (lane & 1);
                    __syncwarp();
#pragma unroll
                    for (int a = 0; a < DP; ++a) {
                        const df u = df_mulf(il[a], x[a]);
                        w[4 * a] = u.h;
                        w[4 * a + 2] = u.l;
                    }
                    w[4 * kMaxD] = isc;
                    w[4 * kMaxD + 2] = vnc;
                    __syncwarp();
                }
                if (!__all_sync(0xffffffffu, sm::mbar_wait(accf, (unsigned)(lt & 1), P.status, 35))) { alive = false; break; }
                sm::tc_fence_after();
                // minus the dots, as double-float: orders of weight 2^(-12 - 7 s) 2^(2e), the first three with
                // their errors; they move to shared memory so that the next tile's products can start
#pragma unroll 1
                for (int i0 = 0; i0 < DN / 2; i0 += kDigitCols) {
                    float o[DO][kDigitCols];
                    digit_orders(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * (DN / 2) + i0), o);
#pragma unroll
                    for (int j = 0; j < kDigitCols; j += 2) {
                        auto ord = [&](int i, float w) { return __ffma2_rn(make_float2(o[i][j], o[i][j + 1]), two2(-w * sc2), nz); };
                        float2 a1, a2;
                        const float2 b1 = two_sum2(ord(0, 0x1p-12f), ord(1, 0x1p-19f), a1);
                        const float2 dh = two_sum2(b1, ord(2, 0x1p-26f), a2);
                        const float2 dl = __fadd2_rn(__fadd2_rn(a1, a2),
                                                     __fadd2_rn(ord(3, 0x1p-33f), __fadd2_rn(ord(4, 0x1p-40f), ord(5, 0x1p-47f))));
                        dots[(i0 + j) * kEpiThreads + et] = dh;
                        dots[(i0 + j + 1) * kEpiThreads + et] = dl;
                    }
                }
                sm::tc_fence_before();
                __syncwarp();
                if (lane == 0) sm::mbar_arrive(acce);
#pragma unroll 1
                for (int i0 = 0; i0 < DN / 2; i0 += kDigitCols) {
                    float& gmin = mins[(i0 / (DN / 2 / kDigitGroups)) * kEpiThreads + et];
                    float gm = KEEP ? 0.f : gmin;
#pragma unroll
                    for (int j = 0; j < kDigitCols; j += 2) {
                        const float4* r = (const float4*)(cand + ((i0 + j) >> 1) * kCandF);
                        const float4 tail = r[kMaxD];
                        float2 kh, kl;
                        kernel_mid2<KT, DP>(r, nq, tab, nz, kh, kl);
                        const float2 dh = dots[(i0 + j) * kEpiThreads + et], dl = dots[(i0 + j + 1) * kEpiThreads + et];
                        // kernel value times the variance, with the product's error
                        const float2 var = two2(R.var);
                        const float2 vh = __ffma2_rn(kh, var, nz);
                        const float2 vl = __ffma2_rn(kl, var, __ffma2_rn(kh, var, __ffma2_rn(vh, two2(-1.f), nz)));
                        const float2 dif = __fadd2_rn(__fadd2_rn(vh, dh), __fadd2_rn(vl, dl));
                        const float2 Rr = make_float2(fabsf(dif.x), fabsf(dif.y));
                        const float2 e = __ffma2_rn(make_float2(tail.z, tail.w), two2(e1 * 1.01f), two2(eq));
                        if (KEEP) {
                            float2 hi = __ffma2_rn(Rr, two2(1.0000005f), e);
                            hi = __fmul2_rn(hi, make_float2(tail.x, tail.y));
#pragma unroll
                            for (int x = 0; x < 2; ++x) {
                                const int c = c0 + i0 + j + x;
                                const float h = x ? hi.y : hi.x;
                                if (c < lim && (!(h < thr) || c == q)) {  // (the query itself: d = 0)
                                    const int at = atomicAdd(&P.cnt[2 * grow + half], 1);
                                    if (at < kDigitCap) {
                                        P.surv[(2 * grow + half) * kDigitCap + at] = c;
                                        P.survb[(2 * grow + half) * kDigitCap + at] = c == q ? __int_as_float(0x7f800000) : h;
                                    }
                                }
                            }
                        } else {
                            const float2 lw = __ffma2_rn(Rr, two2(1.f - 5e-7f), make_float2(-e.x, -e.y));
#pragma unroll
                            for (int x = 0; x < 2; ++x) {
                                const int c = c0 + i0 + j + x;
                                const float rl = fmaxf(x ? lw.y : lw.x, 0.f) * fminf(isq * (x ? tail.y : tail.x), 1e9f) * (1.f - 2e-6f);
                                const float du2 = c == q ? 0.f : 1.f - fminf(rl, 1.f);
                                gm = c < lim ? fminf(gm, du2) : gm;
                            }
                        }
                    }
                    if (!KEEP) gmin = gm;
                }
            }
            if (!KEEP && q >= 0)
                for (int i = 0; i < kDigitGroups; ++i)
                    P.minima[(((size_t)im.w * TQ + (size_t)row * im.z + im.y) * 2 + half) * kDigitGroups + i] = mins[i * kEpiThreads + et];
        }
    }
    sm::tc_fence_before();
    __syncthreads();
    if (warp == 1) sm::tmem_dealloc(tmem_base, 512);
}

// Thresholds of pass B: the k-th smallest minimum of a row (one block per row, the minima in registers),
// widened by the double-float error of the exact distances, lowers its query's shared threshold.
__global__ void __launch_bounds__(256) digit_tau_kernel(DigitParams P, RescoreParams R, unsigned* __restrict__ qtau) {
    constexpr int kPer = (kDigitMaxChunks * 2 * kDigitGroups + 255) / 256;
    const long long r = blockIdx.x;
    const int q = P.qid[r];
    if (q < 0) return;
    const int2 tc = P.tile_chunks[r / TQ];
    const int n = tc.x * 2 * kDigitGroups;
    const float* mn = P.minima + (size_t)tc.y * TQ * 2 * kDigitGroups + (size_t)(r % TQ) * n;
    unsigned x[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) x[i] = i * 256 + threadIdx.x < n ? __float_as_uint(mn[i * 256 + threadIdx.x]) : 0xffffffffu;
    __shared__ int total[2];
    unsigned lo = 0, hi = 0x3f800001u;
    for (int it = 0; lo < hi; ++it) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        if (threadIdx.x == 0) total[it & 1] = 0;
        __syncthreads();
        int c = 0;
#pragma unroll
        for (int i = 0; i < kPer; ++i) c += x[i] <= mid;
        c = __reduce_add_sync(0xffffffffu, c);
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(&total[it & 1], c);
        __syncthreads();
        if (total[it & 1] >= R.k) hi = mid; else lo = mid + 1;
    }
    if (threadIdx.x == 0 && lo <= 0x3f800000u) {
        const float margin = 4e-12f * fmaxf(R.var, 1.f) * fminf(R.isp[q] * __uint_as_float(__ldg(R.isp_max)) * 1.01f, 1e9f) + 1e-12f;
        const float t2 = fminf(__fadd_ru(__fmul_ru(__uint_as_float(lo), 1.000004f), margin), 1.f);
        atomicMin(&qtau[P.qidx[r]], __float_as_uint(t2));
    }
}

// Results of the pass's rows into their queries' output rows (rows marked bad keep theirs).
__global__ void digit_scatter_kernel(const long long* __restrict__ idx, const float* __restrict__ dist,
                                     const int* __restrict__ qidx, const int* __restrict__ bad, long long rows, int k,
                                     long long* __restrict__ out_idx, float* __restrict__ out_dist) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= rows * k) return;
    const long long r = e / k;
    if (bad[r]) return;
    const long long o = (long long)qidx[r] * k + (e - r * k);
    out_idx[o] = idx[e];
    out_dist[o] = dist[e];
}
