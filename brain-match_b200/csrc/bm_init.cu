// bm_init.cu — greedy-similarity initial matching on the device.
//
// The algorithm of src/greedy-match.c:
//   features  per vertex: in-degree, out-degree, the number of distinct
//             vertices reachable in two out-steps and the number that reach
//             it in two in-steps (compute_vertex_features /
//             compute_2hop_metrics :213-293); duplicate edges count, as the
//             reference's adjacency lists keep them;
//   sort      both graphs' vertices by descending feature sum (:295-300,
//             :478-479), ties by ascending id;
//   greedy    each A vertex in that order takes the unmatched B vertex at the
//             smallest L1 feature distance, the first in B's sorted order on
//             ties (:442-447, :483-510).
// The result equals bm_greedy_match of the host library (bm_host.h), which
// restates the same steps on the CPU.
//
// Kernels: reach2_kernel gives each vertex to one CTA (taken from a counter,
// so hubs do not hold up a static share), which marks 2-hop targets in an
// n-bit shared-memory bitmap and counts them with popc.
//
// greedy_kernel is one CTA whose 32 warps hold 32 consecutive A vertices.  Each
// warp finds its vertex's nearest unmatched B vertex; then the vertices are
// committed in order up to the first whose choice an earlier one of the 32 has
// taken (a choice that is still free is still the nearest: matching others
// only removes candidates), and only warps with a new vertex or a taken choice
// search again.  A search starts where B's feature sum equals the vertex's and
// goes outwards both ways: the L1 distance is at least the difference of the
// sums, so a side ends where that difference exceeds the best distance.  The
// unmatched vertices are kept dense (compacted every 1,024 commits).  A
// block-wide argmin over all of B per A vertex took 131 ms at full scale;
// this one takes 22 ms.
#include <algorithm>
#include <climits>
#include <numeric>
#include <vector>

#include "bm_internal.cuh"

namespace {

constexpr int kReachThreads = 256;
constexpr int kGreedyThreads = 1024;

struct Adj {
    const int32_t* ptr;  // n+2
    const int32_t* idx;  // neighbour ids
};

__global__ void __launch_bounds__(kReachThreads) reach2_kernel(Adj out, Adj in, int32_t n, int* next,
                                                               int4* __restrict__ feat) {
    extern __shared__ uint32_t bits[];
    __shared__ int s_v;
    __shared__ int s_cnt;
    const uint32_t nw = (uint32_t)(n + 32) / 32u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = kReachThreads / 32;
    for (;;) {
        if (tid == 0) s_v = atomicAdd(next, 1) + 1;
        __syncthreads();
        const int32_t v = s_v;
        if (v > n) break;
        int counts[2];
        for (int dir = 0; dir < 2; dir++) {
            const Adj a = dir == 0 ? out : in;
            for (uint32_t i = tid; i < nw; i += kReachThreads) bits[i] = 0u;
            if (tid == 0) s_cnt = 0;
            __syncthreads();
            // warps take the first-step neighbours x, lanes stream x's list
            for (int32_t j = a.ptr[v] + warp; j < a.ptr[v + 1]; j += nwarps) {
                const int32_t x = a.idx[j];
                for (int32_t k = a.ptr[x] + lane; k < a.ptr[x + 1]; k += 32) {
                    const int32_t y = a.idx[k];
                    atomicOr(&bits[y >> 5], 1u << (y & 31));
                }
            }
            __syncthreads();
            int c = 0;
            for (uint32_t i = tid; i < nw; i += kReachThreads) c += __popc(bits[i]);
            for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            if (lane == 0) atomicAdd(&s_cnt, c);
            __syncthreads();
            counts[dir] = s_cnt;
            __syncthreads();
        }
        if (tid == 0)
            feat[v] = make_int4(in.ptr[v + 1] - in.ptr[v], out.ptr[v + 1] - out.ptr[v], counts[0], counts[1]);
    }
}

__device__ __forceinline__ long long l1(const int4& a, const int4& b) {
    return llabs((long long)a.x - b.x) + llabs((long long)a.y - b.y) + llabs((long long)a.z - b.z) +
           llabs((long long)a.w - b.w);
}

__device__ __forceinline__ long long total(const int4& f) { return (long long)f.x + f.y + f.z + f.w; }

// The nearest unmatched B vertex of one A vertex, by a warp: the smallest key
// = distance << 17 | sorted position, so ties go to the first position
// (n <= 131071 < 2^17; distances stay below 2^46).  cf, cpos: the `len`
// candidates left at the last compaction by descending sum; `used`: bits of
// the positions matched since.
__device__ unsigned long long nearest(const int4& f, const int4* cf, const int32_t* cpos, int32_t len,
                                      const uint32_t* used, int lane) {
    const long long ta = total(f);
    // the first candidate whose sum is at most ta: 32 probes a step
    int32_t lo = 0, hi = len;
    while (hi > lo) {
        const int32_t w = hi - lo, probe = lo + (int32_t)((long long)w * lane / 32);
        const unsigned above = __ballot_sync(0xffffffffu, total(cf[probe]) > ta);
        const int c = __popc(above);  // sums descend, so the first c probes are above
        if (c == 0) { hi = lo; break; }
        const int32_t nlo = lo + (int32_t)((long long)w * (c - 1) / 32) + 1;
        hi = c == 32 ? hi : lo + (int32_t)((long long)w * c / 32);
        lo = nlo;
    }
    int32_t r = lo, l = lo - 1;
    unsigned long long best = ~0ull;
    bool go_r = r < len, go_l = l >= 0;
    while (go_r || go_l) {
#pragma unroll
        for (int s = 0; s < 4; s++) {  // 64 candidates to the right, 64 to the left
            const int32_t j = (s & 1) ? l - 32 * (s >> 1) - lane : r + 32 * (s >> 1) + lane;
            if ((s & 1) ? (go_l && j >= 0) : (go_r && j < len)) {
                const int4 b = cf[j];
                const int32_t p = cpos[j];
                const unsigned long long key = ((unsigned long long)l1(f, b) << 17) | (unsigned long long)p;
                if (key < best && !((used[p >> 5] >> (p & 31)) & 1u)) best = key;
            }
        }
        r += 64;
        l -= 64;
        for (int o = 16; o; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
            best = t < best ? t : best;
        }
        const long long d = best == ~0ull ? LLONG_MAX : (long long)(best >> 17);
        go_r = go_r && r < len && ta - total(cf[min(r, len - 1)]) <= d;
        go_l = go_l && l >= 0 && total(cf[max(l, 0)]) - ta <= d;
    }
    return best;
}

constexpr int kGreedyCompact = 1024;  // commits between compactions

// fa, ida: A vertices in sorted order (features, ids); fb, idb: the same for
// B.  pi[ida[i]] = idb[j] for the position j chosen at step i.  cf, cpos:
// scratch of n entries each.
__global__ void __launch_bounds__(kGreedyThreads) greedy_kernel(const int4* __restrict__ fa,
                                                                const int32_t* __restrict__ ida,
                                                                const int4* __restrict__ fb,
                                                                const int32_t* __restrict__ idb, int32_t n, int4* cf,
                                                                int32_t* cpos, int32_t* __restrict__ pi) {
    extern __shared__ uint32_t used[];
    __shared__ unsigned long long s_key[32];
    __shared__ int32_t s_new[32];  // the slot's vertex needs a search
    __shared__ int32_t s_head, s_wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nw = (uint32_t)(n + 31) / 32u;
    for (uint32_t i = tid; i < nw; i += kGreedyThreads) used[i] = 0u;
    for (int32_t j = tid; j < n; j += kGreedyThreads) { cf[j] = fb[j]; cpos[j] = j; }
    if (tid < 32) s_new[tid] = 1;
    __syncthreads();
    int32_t head = 0, len = n, compacted = 0;
    while (head < n) {
        const int32_t i = head + ((warp - head) & 31);  // vertex i lives in slot i mod 32
        if (i < n && s_new[warp]) {
            const unsigned long long best = nearest(fa[i], cf, cpos, len, used, lane);
            if (lane == 0) s_key[warp] = best;
        }
        __syncthreads();
        if (warp == 0) {
            const int32_t v = head + lane, slot = v & 31;
            const int32_t j = v < n ? (int32_t)(s_key[slot] & 0x1FFFFull) : -1 - lane;
            const unsigned same = __match_any_sync(0xffffffffu, j);
            const unsigned clash = __ballot_sync(0xffffffffu, v >= n || (same & ((1u << lane) - 1u)) != 0u);
            const int done = clash ? __ffs(clash) - 1 : 32;
            if (lane < done) {
                atomicOr(&used[j >> 5], 1u << (j & 31));
                pi[ida[v]] = idb[j];
            }
            __syncwarp();
            s_new[slot] = lane < done || (v < n && ((used[j >> 5] >> (j & 31)) & 1u));
            if (lane == 0) s_head = head + done;
        }
        __syncthreads();
        head = s_head;
        if (head - compacted >= kGreedyCompact) {  // drop the matched candidates, in order
            compacted = head;
            int32_t base = 0;
            for (int32_t j0 = 0; j0 < len; j0 += kGreedyThreads) {
                const int32_t j = j0 + tid;
                int4 f = make_int4(0, 0, 0, 0);
                int32_t p = 0;
                bool keep = false;
                if (j < len) {
                    f = cf[j];
                    p = cpos[j];
                    keep = !((used[p >> 5] >> (p & 31)) & 1u);
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (lane == 0) s_wsum[warp] = __popc(m);
                __syncthreads();  // everything of this stretch is read
                int32_t before = base, all = 0;
                for (int w = 0; w < 32; w++) {
                    if (w < warp) before += s_wsum[w];
                    all += s_wsum[w];
                }
                if (keep) {
                    const int32_t at = before + __popc(m & ((1u << lane) - 1u));
                    cf[at] = f;
                    cpos[at] = p;
                }
                base += all;
                __syncthreads();
            }
            len = base;
        }
    }
}

// Plain adjacency (ids only, any order within a list: the features are counts)
// of both directions of an edge list.
__global__ void adj_count_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t m, int32_t n,
                                 int32_t* __restrict__ ocnt, int32_t* __restrict__ icnt, int* __restrict__ bad) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t s = src[e], d = dst[e];
        if ((uint32_t)(s - 1) >= (uint32_t)n || (uint32_t)(d - 1) >= (uint32_t)n) {
            *bad = 1;
            continue;
        }
        atomicAdd(ocnt + s, 1);
        atomicAdd(icnt + d, 1);
    }
}

// Exclusive sums of the counts of one direction (block 0: out, 1: in) into
// ptr[0..n+1] and the fill cursors.
__global__ void __launch_bounds__(1024) adj_scan_kernel(int32_t* cnt0, int32_t* cnt1, int32_t n, int32_t* ptr0, int32_t* ptr1) {
    __shared__ int32_t wsum[32];
    int32_t* cnt = blockIdx.x ? cnt1 : cnt0;
    int32_t* ptr = blockIdx.x ? ptr1 : ptr0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int32_t base = 0;
    for (int32_t v0 = 0; v0 <= n; v0 += 1024) {
        const int32_t v = v0 + tid, c = v <= n ? cnt[v] : 0;
        int32_t s = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (lane == 31) wsum[warp] = s;
        __syncthreads();
        int32_t before = base;
        for (int w = 0; w < 32; w++) {
            if (w < warp) before += wsum[w];
            base += wsum[w];
        }
        if (v <= n) {
            ptr[v] = before + s - c;
            cnt[v] = before + s - c;  // becomes the fill cursor
        }
        __syncthreads();
    }
    if (tid == 0) ptr[n + 1] = base;
}

__global__ void adj_fill_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t m,
                                int32_t* __restrict__ ocur, int32_t* __restrict__ icur, int32_t* __restrict__ oidx,
                                int32_t* __restrict__ iidx) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t s = src[e], d = dst[e];
        oidx[atomicAdd(ocur + s, 1)] = d;
        iidx[atomicAdd(icur + d, 1)] = s;
    }
}

struct DevBuf {
    std::vector<void*> p;
    ~DevBuf() { for (void* x : p) bm_cuda_free(x); }
    template <typename T>
    bool get(T** out, size_t count) {
        void* d = nullptr;
        if (bm_cuda_malloc(&d, sizeof(T) * std::max<size_t>(count, 1)) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        p.push_back(d);
        *out = static_cast<T*>(d);
        return true;
    }
};

// Features (n+1 int4: in, out, reach2, canreach2) of one graph on the device;
// *bad is set when an endpoint lies outside 1..n.
bm_status graph_features(bm_ctx* ctx, DevBuf& mem, int32_t n, int64_t m, const int32_t* src, const int32_t* dst,
                         std::vector<int4>& feat, bool* bad) {
    const size_t M = (size_t)m, V = (size_t)n + 2;
    int32_t *d_src, *d_dst, *d_optr, *d_oidx, *d_iptr, *d_iidx, *d_cnt;
    int* d_next;
    int4* d_feat;
    if (!mem.get(&d_src, M) || !mem.get(&d_dst, M) || !mem.get(&d_cnt, 2 * V) || !mem.get(&d_optr, V) ||
        !mem.get(&d_oidx, M) || !mem.get(&d_iptr, V) || !mem.get(&d_iidx, M) || !mem.get(&d_next, 2) ||
        !mem.get(&d_feat, (size_t)n + 1))
        return bm_fail(ctx, BM_OOM, "greedy matching: device allocation failed");
    if (m > 0) {
        BM_CUDA(ctx, cudaMemcpyAsync(d_src, src, sizeof(int32_t) * M, cudaMemcpyHostToDevice, ctx->stream));
        BM_CUDA(ctx, cudaMemcpyAsync(d_dst, dst, sizeof(int32_t) * M, cudaMemcpyHostToDevice, ctx->stream));
    }
    BM_CUDA(ctx, cudaMemsetAsync(d_cnt, 0, sizeof(int32_t) * 2 * V, ctx->stream));
    BM_CUDA(ctx, cudaMemsetAsync(d_next, 0, 2 * sizeof(int), ctx->stream));
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((m + 255) / 256, (int64_t)ctx->num_sms * 8));
    adj_count_kernel<<<grid, 256, 0, ctx->stream>>>(d_src, d_dst, m, n, d_cnt, d_cnt + V, d_next + 1);
    BM_LAUNCH_CHECK(ctx, "adj_count_kernel");
    int h_bad = 0;
    BM_CUDA(ctx, cudaMemcpyAsync(&h_bad, d_next + 1, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *bad = h_bad != 0;
    if (*bad) return BM_OK;
    adj_scan_kernel<<<2, 1024, 0, ctx->stream>>>(d_cnt, d_cnt + V, n, d_optr, d_iptr);
    BM_LAUNCH_CHECK(ctx, "adj_scan_kernel");
    adj_fill_kernel<<<grid, 256, 0, ctx->stream>>>(d_src, d_dst, m, d_cnt, d_cnt + V, d_oidx, d_iidx);
    BM_LAUNCH_CHECK(ctx, "adj_fill_kernel");
    BM_CUDA(ctx, cudaMemsetAsync(d_feat, 0, sizeof(int4) * ((size_t)n + 1), ctx->stream));
    const size_t smem = sizeof(uint32_t) * (((size_t)n + 32) / 32);
    if (smem > 48 * 1024)
        BM_CUDA(ctx, cudaFuncSetAttribute(reach2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    reach2_kernel<<<ctx->num_sms * 4, kReachThreads, smem, ctx->stream>>>(Adj{d_optr, d_oidx}, Adj{d_iptr, d_iidx}, n,
                                                                         d_next, d_feat);
    BM_LAUNCH_CHECK(ctx, "reach2_kernel");
    feat.resize((size_t)n + 1);
    BM_CUDA(ctx, cudaMemcpyAsync(feat.data(), d_feat, sizeof(int4) * ((size_t)n + 1), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    return BM_OK;
}

}  // namespace

extern "C" bm_status bm_greedy_match_dev(bm_ctx* ctx, int32_t n, int64_t mA, const int32_t* srcA,
                                         const int32_t* dstA, int64_t mB, const int32_t* srcB, const int32_t* dstB,
                                         int32_t* pi) {
    if (!ctx || !pi) return BM_INVALID_ARG;
    if (n < 1 || n > BM_MAX_N) return bm_fail(ctx, BM_INVALID_ARG, "n = %d outside 1..%d", n, BM_MAX_N);
    if (mA < 0 || mB < 0 || mA >= INT32_MAX || mB >= INT32_MAX || (mA > 0 && (!srcA || !dstA)) ||
        (mB > 0 && (!srcB || !dstB)))
        return bm_fail(ctx, BM_INVALID_ARG, "bad edge arrays");
    BM_CUDA(ctx, cudaSetDevice(ctx->device));
    DevBuf mem;
    std::vector<int4> fa, fb;
    bm_status s;
    bool badA = false, badB = false;
    if ((s = graph_features(ctx, mem, n, mA, srcA, dstA, fa, &badA)) != BM_OK) return s;
    if (!badA && (s = graph_features(ctx, mem, n, mB, srcB, dstB, fb, &badB)) != BM_OK) return s;
    if (badA || badB) {
        const int32_t* ends[4] = {srcA, dstA, srcB, dstB};
        const int64_t ms[4] = {mA, mA, mB, mB};
        for (int q = 0; q < 4; q++)
            for (int64_t e = 0; e < ms[q]; e++)
                if (ends[q][e] < 1 || ends[q][e] > n)
                    return bm_fail(ctx, BM_INVALID_ARG, "edge endpoint %d outside 1..%d", ends[q][e], n);
    }
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    // both graphs' vertices by descending feature sum, ties by id
    auto order = [&](const std::vector<int4>& f, std::vector<int32_t>& ids, std::vector<int4>& sorted) {
        ids.resize((size_t)n);
        std::iota(ids.begin(), ids.end(), 1);
        auto total = [&](int32_t v) {
            const int4& x = f[(size_t)v];
            return (long long)x.x + x.y + x.z + x.w;
        };
        std::stable_sort(ids.begin(), ids.end(), [&](int32_t p, int32_t q) { return total(p) > total(q); });
        sorted.resize((size_t)n);
        for (int32_t i = 0; i < n; i++) sorted[(size_t)i] = f[(size_t)ids[(size_t)i]];
    };
    std::vector<int32_t> ida, idb;
    std::vector<int4> sfa, sfb;
    order(fa, ida, sfa);
    order(fb, idb, sfb);
    int4 *d_fa, *d_fb, *d_cf;
    int32_t *d_ida, *d_idb, *d_pi, *d_cpos;
    if (!mem.get(&d_fa, (size_t)n) || !mem.get(&d_fb, (size_t)n) || !mem.get(&d_ida, (size_t)n) ||
        !mem.get(&d_idb, (size_t)n) || !mem.get(&d_pi, (size_t)n + 1) || !mem.get(&d_cf, (size_t)n) ||
        !mem.get(&d_cpos, (size_t)n))
        return bm_fail(ctx, BM_OOM, "greedy matching: device allocation failed");
    BM_CUDA(ctx, cudaMemcpyAsync(d_fa, sfa.data(), sizeof(int4) * (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(d_fb, sfb.data(), sizeof(int4) * (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(d_ida, ida.data(), sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(d_idb, idb.data(), sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    BM_CUDA(ctx, cudaMemsetAsync(d_pi, 0, sizeof(int32_t) * ((size_t)n + 1), ctx->stream));
    const size_t smem = sizeof(uint32_t) * (((size_t)n + 31) / 32);
    greedy_kernel<<<1, kGreedyThreads, smem, ctx->stream>>>(d_fa, d_ida, d_fb, d_idb, n, d_cf, d_cpos, d_pi);
    BM_LAUNCH_CHECK(ctx, "greedy_kernel");
    BM_CUDA(ctx, cudaMemcpyAsync(pi, d_pi, sizeof(int32_t) * ((size_t)n + 1), cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BM_OK;
}
