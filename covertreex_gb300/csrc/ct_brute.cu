// ct_brute.cu — plain FP32 residual-correlation kNN, dense form for one tree.
//
// A work item is one query tile against one chunk of the candidates (in predecessor mode,
// of the candidates below the tile's largest query id).  The tile itself (dot-product
// order, distance epilogue, top-k lists) is dense::run_tile in ct_dense.cuh, shared with
// the batched persistent kernel.
//
// Launch shape.  An SM holds one or two blocks of a tile (registers and shared memory), so a call
// runs in waves.  choose_shape models the time of each tile height and
// candidate split as the larger of the mean load per block slot and the longest item, plus a fixed cost
// per item (loading the query rows, filling the lists, merging), and takes the smallest:
// tall tiles read the candidates least often, short ones and splits fill the chip when there
// are few queries.  Splitting needs scratch for the partial lists; the block that finishes a
// tile's last chunk merges them (a counter per tile, no block waits for another).
#include "ct_common.cuh"
#include "ct_dense.cuh"
#include "ct_internal.h"

#include <algorithm>
#include <cmath>

namespace ct {

namespace {

using dense::u64;

struct SplitArgs {
    int split;        // candidate chunks per query tile
    long long chunk;  // candidates per chunk
    u64* part;        // [nq][split][k] sorted keys (split > 1)
    int* done;        // [tiles] finished chunks, zero at launch
    dense::Ring ring;
    u64 nz;
};

template <int C>
__global__ void __launch_bounds__(dense::CfgOf<C>::NT, dense::CfgOf<C>::NT == 256 ? 2 : 1)
    brute_knn_kernel(BruteParams P, SplitArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int QT = dense::CfgOf<C>::QT;
    const long long tiles = (P.nq + QT - 1) / QT;
    // heavy tiles (large query ids in predecessor mode) first
    const long long tile = tiles - 1 - blockIdx.x / A.split;
    const int ch = (int)(blockIdx.x % A.split);
    const long long cend = P.cend > 0 ? P.cend : P.n;
    dense::Tile J;
    J.vperm = P.vperm; J.xs = P.xs; J.norms = P.norms; J.p = P.p;
    J.n = P.n; J.m = P.m; J.d = P.d; J.k = P.k; J.kernel_type = P.kernel_type; J.predecessor = P.predecessor;
    J.var = P.var;
    J.qids = P.qids; J.qv = nullptr; J.qcoords = nullptr; J.qp = nullptr; J.inv_ls = nullptr;
    J.nq = P.nq;
    J.q0 = tile * QT;
    J.cbeg = P.cbeg + ch * A.chunk;
    J.cend = J.cbeg + A.chunk < cend ? J.cbeg + A.chunk : cend;
    J.out_idx = P.out_idx; J.out_dist = P.out_dist; J.out_stride = P.k;
    J.part = A.split > 1 ? A.part + (long long)ch * P.k : nullptr;
    J.part_stride = (long long)A.split * P.k;
    J.ring = A.ring;
    dense::run_tile<C>(J, A.nz);
    if (A.split > 1) {
        __shared__ int s_last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(&A.done[tile], 1) == A.split - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            const int nv = (int)(P.nq - J.q0 < QT ? P.nq - J.q0 : QT);
            dense::merge_tile<dense::CfgOf<C>::NT>(A.part, A.split, P.k, J.q0, nv, (u64*)smem_raw, P.out_idx, P.out_dist, P.k);
        }
    }
}

// Cost of a work item beyond its pairs, in candidates of its own tile.  A query's list takes about
// k (1 + ln(L / k)) insertions over L candidates, each some 700 thread instructions (exact
// distance, its share of a sort and a merge), where a pair costs about m + 150; loading the query
// rows and writing the list adds a step.
double item_cost(double len, int m, int k) {
    return 64.0 + k * (1.0 + std::log(std::max(1.0, len / k))) * 700.0 / (m + 150.0);
}
constexpr size_t kFixedSmem = 64;  // the kernel's static shared memory

struct Shape {
    int cfg = -1, split = 1;
    dense::Ring ring{};
    size_t smem = 0;
};

struct Limits {
    size_t optin, per_sm;
    int sms;
};

Shape choose_shape(const BruteParams& P, long long cands, const Limits& L, bool scratch_ok) {
    Shape best;
    double best_t = 0.0;
    // time of a query-candidate pair with every block slot busy, relative to the 32-row tile
    // (the 16-row tiles reuse each operand half as often); the last is the 32-row tile with an SM to itself, for
    // rows too wide for the other 32-row forms (m = 528 to 1024) and calls of enough tiles to fill the chip
    // (4096 rows against 4096, k = 10: m = 768 1.3 times as fast as 16-row tiles, m = 1024 1.46 times)
    const double pair_cost[dense::kNumCfg + 1] = {1.0, 1.25, 1.1, 1.6, 1.15};
    for (int i = 0; i <= dense::kNumCfg; ++i) {
        if (i == dense::kNumCfg && P.nq < 512) break;
        const int c = i < dense::kNumCfg ? i : dense::kCfg32;
        Shape s;
        s.cfg = c;
        const size_t limit = i < dense::kNumCfg ? dense::cfg_limit(c, L.optin, L.per_sm, kFixedSmem) : L.optin - kFixedSmem;
        if (!dense::pick_ring(c, P.m, P.d, P.k, limit, &s.ring, &s.smem)) continue;
        const int qt = dense::cfg_qt(c), ct = dense::cfg_ct(c);
        const int bps = i < dense::kNumCfg && dense::cfg_threads(c) == 256 ? 2 : 1;
        const long long tiles = (P.nq + qt - 1) / qt;
        const double slots = (double)L.sms * bps;
        const int max_split =
            scratch_ok ? (int)std::max<long long>(1, std::min<long long>(128, cands / ct)) : 1;
        for (int sp = 1; sp <= max_split; ++sp) {
            const double chunk = std::ceil((double)cands / sp / ct) * ct, cost = item_cost(chunk, P.m, P.k);
            const double len = chunk + cost;  // longest item
            const double mean = (double)cands * (P.predecessor ? 0.5 : 1.0) / sp + cost;
            const double items = (double)tiles * sp;
            // equal items run in whole waves; predecessor tiles of falling length fill the gaps
            const double waves = P.predecessor ? std::max(items * mean / slots, len)
                                               : std::ceil(items / slots) * len;
            const double t = waves * qt * bps * pair_cost[i];
            if (best.cfg < 0 || t < best_t) {
                best = s;
                best.split = sp;
                best_t = t;
            }
            if (items > 16.0 * slots) break;
        }
    }
    return best;
}

bool device_limits(Limits* L) {
    int dev = 0, a = 0, b = 0, c = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&a, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&b, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return false;
    L->optin = (size_t)a;
    L->per_sm = (size_t)b;
    L->sms = c;
    return true;
}

template <int C>
cudaError_t launch_cfg(const BruteParams& P, const Shape& s, const SplitArgs& A, long long items, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(brute_knn_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
    if (e != cudaSuccess) return e;
    brute_knn_kernel<C><<<(unsigned)items, dense::CfgOf<C>::NT, s.smem, st>>>(P, A);
    return cudaGetLastError();
}

}  // namespace

bool brute_fits(int m, int d, int k) {
    Limits L;
    dense::Ring r;
    size_t total;
    if (!device_limits(&L)) return false;
    for (int c = 0; c < dense::kNumCfg; ++c)
        if (dense::pick_ring(c, m, d, k, dense::cfg_limit(c, L.optin, L.per_sm, kFixedSmem), &r, &total)) return true;
    return false;
}

cudaError_t launch_brute_knn(const BruteParams& P, bool scratch_ok, cudaStream_t stream) {
    const long long cend = P.cend > 0 ? P.cend : P.n;
    const long long cands = std::max<long long>(1, cend - P.cbeg);
    if (P.nq <= 0) return cudaSuccess;
    Limits L;
    if (!device_limits(&L)) return cudaGetLastError();
    cudaError_t e = cudaSuccess;
    if (scratch_ok) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        e = cudaStreamIsCapturing(stream, &cs);
        if (e != cudaSuccess) return e;
        scratch_ok = cs == cudaStreamCaptureStatusNone;
    }
    const Shape s = choose_shape(P, cands, L, scratch_ok);
    if (s.cfg < 0) return cudaErrorInvalidValue;
    const int qt = dense::cfg_qt(s.cfg), ct = dense::cfg_ct(s.cfg);
    const long long tiles = (P.nq + qt - 1) / qt;
    SplitArgs A{};
    A.ring = s.ring; A.nz = dense::kNegZero2;
    A.chunk = ((cands + s.split - 1) / s.split + ct - 1) / ct * ct;
    A.split = (int)((cands + A.chunk - 1) / A.chunk);
    unsigned char* scratch = nullptr;
    if (A.split > 1) {
        const size_t done_bytes = (sizeof(int) * (size_t)tiles + 255) & ~size_t(255);
        e = cudaMallocAsync((void**)&scratch, done_bytes + sizeof(u64) * (size_t)P.nq * A.split * P.k, stream);
        if (e != cudaSuccess) {  // no room for partial lists: one chunk per tile needs none
            cudaGetLastError();
            A.split = 1;
            A.chunk = (cands + ct - 1) / ct * ct;
            scratch = nullptr;
        } else {
            A.done = (int*)scratch;
            A.part = (u64*)(scratch + done_bytes);
            e = cudaMemsetAsync(A.done, 0, sizeof(int) * (size_t)tiles, stream);
        }
    }
    const long long items = tiles * A.split;
    if (scratch == nullptr) e = cudaSuccess;
    if (e == cudaSuccess) {
        switch (s.cfg) {
            case dense::kCfg32: e = launch_cfg<dense::kCfg32>(P, s, A, items, stream); break;
            case dense::kCfg16: e = launch_cfg<dense::kCfg16>(P, s, A, items, stream); break;
            case dense::kCfg32w: e = launch_cfg<dense::kCfg32w>(P, s, A, items, stream); break;
            default: e = launch_cfg<dense::kCfg16w>(P, s, A, items, stream); break;
        }
    }
    if (scratch) {
        const cudaError_t f = cudaFreeAsync(scratch, stream);
        if (e == cudaSuccess) e = f;
    }
    return e;
}

}  // namespace ct
