// ct_traverse.cu — plain FP32 form, cover-tree traversal (the query of
// single_residual_knn_query, src/algo.rs:612-1242, in its exhaustive parity mode,
// without the budget ladder), exact: it returns the dense form's neighbour lists
// bit for bit.
//
// One block owns one query at a time (persistent grid).  It keeps a depth-first stack of frames
// (a range of child indices and the subtree's bound) and its top-k list in shared memory and
// works in steps of kB candidates: the topmost frames' children (the roots when the stack is
// empty) are gathered, filtered in predecessor mode (a subtree whose minimum dataset id is not
// below the query's is skipped without a distance, src/algo.rs:900-916), their V rows scored by
// half-warps with the reference's batch-path f32 distance (lane l sums elements 16c + l,
// bit-identical to the dense form) and each candidate's normalisation, list key, bound and
// children looked up by a thread of its own.  Candidates that have children and are not pruned
// become frames.  A step costs a handful of dependent memory latencies whatever its width, so
// its width is what sets the rate while the tree fits in L2: N = 16384, m = 128, 256 queries
// 16.4 ms with a warp per query scoring 4 candidates at a time, 1.0 ms now.
//
// Prune (certified, ct_treebound.cuh): the subtree below a node a cannot hold a
// neighbour when
//   L = lower(d32(q, a), delta(q, a)) - si_up[a] > 0  and
//   lower(L, delta_max(q, subtree a)) > kth,
// where lower() is a certified lower bound of the ideal metric, si_up[a] a certified
// upper bound of the ideal distance from a to any descendant, and delta_max the FP32
// error bound of any pair (q, x) in the subtree (through sub_isp[a], the subtree's
// largest 1/sqrt(p)).  By the ideal metric's triangle inequality every x below a then
// has d32(q, x) > kth, so the pruned subtree cannot change the list: the result equals
// the dense form's.  The reference's own test, d(q, a) - max(si[a], 1e-3) > kth on
// FP32 values (src/algo.rs:814-818, 1113-1142), has no such guarantee.
#include <algorithm>

#include "ct_common.cuh"
#include "ct_dense.cuh"
#include "ct_internal.h"
#include "ct_tree.h"
#include "ct_treebound.cuh"

namespace ct {
namespace trav {

constexpr int kThreads = 256;
constexpr int kB = 128;  // candidates of a step
// A step pushes at most kB frames, and only the topmost batch of frames is consumed while it
// lasts, so the batches on the stack have strictly growing least depths: kB frames per level of
// the tree at most (levels fall strictly from 0 to -30; only duplicate points share the floor
// level).  A deeper tree is reported as an overflow error, never written past.
constexpr int kStack = kB * 40;
constexpr int kTopK = 64;
constexpr int kBufKeep = 64;            // keys a step may leave unmerged
constexpr int kBuf = kB + kBufKeep;

struct Params {
    const float* v;      // node-order natural V
    const float* xs;
    const float* norms;
    const float* p;
    const float* isp;    // node order: 1/sqrt(p), |v| (rounded up)
    const float* vn;
    const long long* order;  // node -> dataset id
    const long long* inv;    // dataset id -> node
    const long long* child_off;
    const long long* child_idx;
    const float* si_up;
    const float* sub_isp;
    const long long* sub_min;
    const long long* roots;
    long long n_roots;
    const long long* q_ids;
    long long nq, n;
    int m, d, k, kernel_type, predecessor;
    float var;
    BoundModel bound;
    long long* out_idx;
    float* out_dist;
    unsigned long long* evals;
    int* overflow;
};

struct Frame {
    int beg, end;  // child_idx range still to visit
    float lb;      // certified lower bound of every FP32 distance below it
};
struct Shared {
    Frame stack[kStack];
    dense::u64 list[kTopK];
    dense::u64 buf[kBuf];
    int cand[kB];
    float dot[kB];
    float xq[64];
    int fbeg[kB], ffirst[kB];  // the frames of a step: first child index, first candidate
    int wsum[kThreads / 32];
    int ncand, nframes, cnt, sp, overflow;
    dense::u64 tau;
};

__global__ void __launch_bounds__(kThreads) traverse_kernel(Params P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Shared& S = *(Shared*)smem_raw;
    float* vq = (float*)(smem_raw + ((sizeof(Shared) + 15) & ~size_t(15)));  // query row
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int l16 = lane & 15, hw = tid >> 4;
    const unsigned hmask = (lane & 16) ? 0xffff0000u : 0x0000ffffu;
    const int m = P.m, mc = P.m >> 4, k = P.k;
    unsigned long long evals = 0;
    for (long long qi = blockIdx.x; qi < P.nq; qi += gridDim.x) {
        const long long qd = P.q_ids[qi];
        const bool live = qd >= 0 && qd < P.n && !(P.predecessor && qd == 0);
        __syncthreads();  // the previous query's results have been written
        for (int j = tid; j < k; j += kThreads) S.list[j] = dense::kNoKey;
        if (tid == 0) { S.cnt = 0; S.sp = 0; S.tau = dense::kNoKey; S.overflow = 0; }
        const int qn = live ? (int)P.inv[qd] : 0;
        if (live) {
            for (int c = tid; c < m; c += kThreads) vq[c] = P.v[(size_t)qn * m + c];
            for (int c = tid; c < P.d; c += kThreads) S.xq[c] = P.xs[(size_t)qn * P.d + c];
        }
        const float nq = P.norms[qn], pq = P.p[qn], isq = P.isp[qn], vnq = P.vn[qn];
        const bool may_prune = isq <= kNoPruneIsp;
        long long next_root = live ? 0 : P.n_roots;
        __syncthreads();
        for (;;) {
            // ---- gather up to kB candidates from the topmost frames, or from the roots
            const int sp = S.sp;
            if (sp == 0 && next_root >= P.n_roots) break;
            const dense::u64 tau = S.tau;
            const float kth = tau == dense::kNoKey ? CT_FLT_MAX : __uint_as_float((unsigned)(tau >> 32));
            int c = -1;
            int total;
            if (sp == 0) {
                const long long left = P.n_roots - next_root;
                total = left < kB ? (int)left : kB;
                if (tid < total) c = (int)P.roots[next_root + tid];
                next_root += total;
                __syncthreads();  // every thread has read the stack state
            } else {
                // thread i looks at the i-th frame from the top; a pruned frame offers nothing
                int take = 0;
                Frame f{0, 0, 0.f};
                if (tid < kB && tid < sp) {
                    f = S.stack[sp - 1 - tid];
                    take = f.lb > kth ? 0 : min(f.end - f.beg, kB);
                }
                int incl = take;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (lane == 31) S.wsum[warp] = incl;
                __syncthreads();
                for (int w = 0; w < warp; ++w) incl += S.wsum[w];
                const int first = incl - take;  // candidates of the frames above this one
                // frames wholly or partly taken: those whose first candidate lies below kB
                if (tid < kB && tid < sp && first < kB) {
                    S.fbeg[tid] = f.beg;
                    S.ffirst[tid] = first;
                    const bool part = first + take > kB;
                    const bool last = tid + 1 == min(sp, kB) || incl >= kB;
                    if (part) S.stack[sp - 1 - tid].beg = f.beg + (kB - first);
                    if (last) {  // the deepest frame of the step
                        S.nframes = tid + 1;
                        S.ncand = min(incl, kB);
                        // a frame with children left stays, the ones above it go
                        const bool stays = part || (first + take == kB && f.lb <= kth && f.end - f.beg > take);
                        if (!part && stays) S.stack[sp - 1 - tid].beg = f.beg + take;
                        S.sp = sp - tid - (stays ? 0 : 1);
                    }
                }
                __syncthreads();
                total = S.ncand;
                if (tid < total) {
                    int lo = 0, hi = S.nframes - 1;  // last frame whose first candidate is <= tid
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (S.ffirst[mid] <= tid) lo = mid; else hi = mid - 1;
                    }
                    c = (int)P.child_idx[S.fbeg[lo] + (tid - S.ffirst[lo])];
                }
            }
            if (c >= 0 && P.predecessor && P.sub_min[c] >= qd) c = -1;
            // compact
            const unsigned okm = __ballot_sync(0xffffffffu, c >= 0);
            if (lane == 0) S.wsum[warp] = __popc(okm);
            __syncthreads();
            int at = __popc(okm & ((1u << lane) - 1u)), nc = 0;
            for (int w = 0; w < kThreads / 32; ++w) {
                if (w < warp) at += S.wsum[w];
                nc += S.wsum[w];
            }
            if (c >= 0) S.cand[at] = c;
            __syncthreads();
            // ---- V dots: half-warp h scores candidates h, h + 16, ..., four rows in flight
            for (int c0 = hw; c0 < nc; c0 += 64) {
                const float* row[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) row[u] = P.v + (size_t)S.cand[c0 + 16 * u < nc ? c0 + 16 * u : c0] * m + l16;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                for (int cc = 0; cc < mc; ++cc) {
                    const float a = vq[16 * cc + l16];
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[u] = __fadd_rn(__fmul_rn(a, __ldg(row[u] + 16 * cc)), acc[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float t = __shfl_down_sync(hmask, acc[u], 8, 16);
                    const float comb = __fadd_rn(acc[u], t);
                    t = __shfl_down_sync(hmask, comb, 4, 16);
                    const float s2 = __fadd_rn(comb, t);
                    t = __shfl_down_sync(hmask, s2, 2, 16);
                    const float u2 = __fadd_rn(s2, t);
                    t = __shfl_down_sync(hmask, u2, 1, 16);
                    if (l16 == 0 && c0 + 16 * u < nc) S.dot[c0 + 16 * u] = __fadd_rn(u2, t);
                }
            }
            __syncthreads();
            // ---- one candidate per thread: distance, list, bound, children
            bool push = false;
            Frame f{0, 0, 0.f};
            if (tid < nc) {
                const int node = S.cand[tid];
                const long long ds = P.order[node];
                const long long b0 = P.child_off[node], e0 = P.child_off[node + 1];
                const float nn = P.norms[node];
                float dist = 0.f;
                if (node != qn) {
                    const float d2 = coord_d2_batch(S.xq, P.xs + (size_t)node * P.d, P.d, nq, nn);
                    const float kv = kernel_value_batch(d2, P.var, P.kernel_type);
                    dist = residual_from_parts(kv, S.dot[tid], pq, P.p[node]);
                }
                if (!P.predecessor || ds < qd) {
                    const dense::u64 key = dense::make_key(dist, (int)ds);
                    if (key < tau) S.buf[atomicAdd(&S.cnt, 1)] = key;
                }
                if (e0 > b0) {
                    f.beg = (int)b0;
                    f.end = (int)e0;
                    if (may_prune) {
                        const float dqa = pair_delta(P.bound, nq, nn, vnq, P.vn[node], isq, P.isp[node]);
                        const float L = (dist_lower(dist, dqa) - P.si_up[node]) * (1.f - 5.0e-7f);
                        if (L > 0.f) {
                            const float dmax = pair_delta(P.bound, nq, P.bound.nmax, vnq, P.bound.vmax, isq,
                                                          P.sub_isp[node]);
                            f.lb = dist_lower(L, dmax);
                        }
                    }
                    push = !(f.lb > kth);
                }
            }
            evals += nc;
            const unsigned pm = __ballot_sync(0xffffffffu, push);
            if (lane == 0) S.wsum[warp] = __popc(pm);
            __syncthreads();
            const int sp0 = S.sp;
            int pos = sp0 + __popc(pm & ((1u << lane) - 1u)), np = 0;
            for (int w = 0; w < kThreads / 32; ++w) {
                if (w < warp) pos += S.wsum[w];
                np += S.wsum[w];
            }
            if (push && pos < kStack) S.stack[pos] = f;
            const int cnt = S.cnt;
            __syncthreads();
            if (tid == 0) {
                S.sp = min(sp0 + np, kStack);
                if (sp0 + np > kStack) S.overflow = 1;
            }
            if (warp == 1 && cnt > kBufKeep) {
                dense::merge_buffer(S.list, k, S.buf, cnt);
                if (lane == 0) { S.cnt = 0; S.tau = S.list[k - 1]; }
            }
            __syncthreads();
        }
        if (warp == 0) {
            dense::merge_buffer(S.list, k, S.buf, S.cnt);
            for (int j = lane; j < k; j += 32) {
                const dense::u64 key = S.list[j];
                P.out_idx[qi * k + j] = key == dense::kNoKey ? -1LL : (long long)(unsigned)key;
                P.out_dist[qi * k + j] = key == dense::kNoKey ? CT_FLT_MAX : __uint_as_float((unsigned)(key >> 32));
            }
            if (lane == 0 && S.overflow) atomicAdd(P.overflow, 1);
        }
    }
    if (tid == 0 && P.evals && evals) atomicAdd(P.evals, evals);
}

}  // namespace trav
}  // namespace ct

using namespace ct::trav;

int ct_tree::knn_tree(const int64_t* q_ids, int64_t nq, int k, int predecessor, int64_t* out_idx, float* out_dist,
                      ct_stats* stats, cudaStream_t st) {
    if (!has_tree) return set_err(CT_ERR_STATE, "%s", "tree form needs a tree (built without CT_BUILD_METRIC_ONLY)");
    if (k > kTopK) return set_err(CT_ERR_UNSUPPORTED, "tree form supports k <= %d", kTopK);
    if (m > 1024 || d > 64) return set_err(CT_ERR_UNSUPPORTED, "%s", "tree form supports m <= 1024, d <= 64");
    unsigned long long* evals = nullptr;
    int* overflow = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&evals, 8, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&overflow, 4, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(evals, 0, 8, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(overflow, 0, 4, st);
    Params P{};
    P.v = tvnat; P.xs = txs; P.norms = tnorms; P.p = tp; P.isp = tisp; P.vn = tvn; P.order = order; P.inv = inv;
    P.child_off = child_off; P.child_idx = child_idx; P.si_up = si_up; P.sub_isp = sub_isp; P.sub_min = sub_min;
    P.roots = roots; P.n_roots = n_roots; P.q_ids = (const long long*)q_ids; P.nq = nq; P.n = n;
    P.m = m; P.d = d; P.k = k; P.kernel_type = kernel_type; P.predecessor = predecessor ? 1 : 0; P.var = var;
    P.bound = bound;
    P.out_idx = (long long*)out_idx; P.out_dist = out_dist; P.evals = evals; P.overflow = overflow;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = ((sizeof(Shared) + 15) & ~size_t(15)) + sizeof(float) * (size_t)m;
    const long long blocks = std::min<long long>(nq, (long long)sms * 3);  // three blocks' stacks fit an SM
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    const bool timing = ct::timing_enabled();
    if (timing) { cudaEventCreate(&e0); cudaEventCreate(&e1); cudaEventRecord(e0, st); }
    if (e == cudaSuccess) {
        e = cudaFuncSetAttribute(traverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) traverse_kernel<<<(unsigned)blocks, kThreads, smem, st>>>(P);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    unsigned long long he = 0;
    int ho = 0;
    float ms = 0.f;
    if (timing && e == cudaSuccess) { cudaEventRecord(e1, st); cudaEventSynchronize(e1); cudaEventElapsedTime(&ms, e0, e1); }
    if (timing) { cudaEventDestroy(e0); cudaEventDestroy(e1); }
    if (e == cudaSuccess) {
        e = cudaMemcpyAsync(&he, evals, 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&ho, overflow, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    cudaFreeAsync(evals, st);
    cudaFreeAsync(overflow, st);
    if (e != cudaSuccess) return set_err(CT_ERR_CUDA, "tree traversal: %s", cudaGetErrorString(e));
    if (stats) {
        stats->distance_evals = (long long)he;
        stats->kernel_launches = 1;
        stats->device_ms = ms;
        stats->screen_ms = ms;
        stats->overflow_queries = ho;
    }
    if (ho > 0) return set_err(CT_ERR_STATE, "tree traversal: %d queries overflowed the %d-entry stack", ho, kStack);
    return CT_OK;
}
