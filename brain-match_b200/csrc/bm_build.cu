// bm_build.cu — the device graph layout (bm_csr.hpp) built on the device from
// an edge list.
//
// The result is that of bm_build_host_csr, entry for entry (the hash table up
// to the order of equal probe sequences): lists sorted by (vertex, neighbour,
// edge index), A keeping every entry, B the last weight of a repeated edge,
// zero weights dropped, self-loops apart, lists padded to four entries.  Two
// stable radix sorts of the edge indices give the out- and the in-order; the
// edges kept are numbered along each order, which places them, and the two
// places of an edge are each other's twin.
//
// What bounds it: the copies of the edge list from the caller's pageable
// memory (36 MB at 3 M edges, about 4 ms) and of A's sorted lists back for the
// host-side selection; the sorts move 8 bytes an edge and pass, eight passes.
// Building the full-scale pair on the host took 190 ms for A and 390 ms for B;
// with each graph in one allocation (bm_graph_alloc) it takes 6.3-6.8 and 4.2-5.8
// ms so, the kernels 1.6 ms of them.
//
// Inputs that the layout rejects (ids, weights, a second self-loop of an A
// vertex, weighted degrees) only raise a flag here; the caller then has the
// host builder find the first offender and word the error.
#include <algorithm>
#include <vector>

#include "bm_internal.cuh"

namespace {

constexpr int kSortThreads = 512;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4,096 edges to a block
constexpr int kMaxDigits = 512;                       // 17-bit ids in two digits of at most 9 bits

enum { kBadInput = 1, kBadSelf = 2 };

// What the host needs to know before it sizes the lists.
struct BuildStats {
    int32_t flags;
    int32_t has_self;
    int32_t has_dup;
    int32_t max_deg;
    long long max_wdeg;
    int32_t m_real, m_out, m_in, pad;
};

__global__ void check_edges_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                   const int32_t* __restrict__ w, int64_t m, int32_t n, BuildStats* st) {
    bool bad = false;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x)
        bad |= (uint32_t)(src[e] - 1) >= (uint32_t)n || (uint32_t)(dst[e] - 1) >= (uint32_t)n ||
               (uint32_t)w[e] > (uint32_t)BM_MAX_W;
    if (bad) atomicOr(&st->flags, kBadInput);
}

// ---------------------------------------------------------- radix sort pass

// Edges per digit and tile: hist[d * tiles + tile].
__global__ void __launch_bounds__(kSortThreads) sort_count_kernel(const int32_t* __restrict__ perm,
                                                                  const int32_t* __restrict__ ids, int64_t m, int shift,
                                                                  int digits, int32_t* __restrict__ hist) {
    __shared__ int32_t cnt[kMaxDigits];
    for (int d = threadIdx.x; d < digits; d += kSortThreads) cnt[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    for (int i = threadIdx.x; i < kSortTile; i += kSortThreads) {
        const int64_t k = base + i;
        if (k < m) atomicAdd(&cnt[(ids[perm ? perm[k] : (int32_t)k] >> shift) & (digits - 1)], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < digits; d += kSortThreads) hist[(size_t)d * gridDim.x + blockIdx.x] = cnt[d];
}

// Block-wide exclusive sum of one value per thread; *all gets the total.
template <int THREADS>
__device__ __forceinline__ int32_t block_exclusive(int32_t v, int32_t* wsum, int32_t* all) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t s = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    int32_t before = 0, total = 0;
    for (int w = 0; w < THREADS / 32; w++) {
        if (w < warp) before += wsum[w];
        total += wsum[w];
    }
    __syncthreads();
    *all = total;
    return before + s - v;
}

// One block per digit: exclusive sums over the tiles, and the digit's total.
__global__ void __launch_bounds__(256) sort_scan_kernel(int32_t* __restrict__ hist, int32_t tiles,
                                                        int32_t* __restrict__ total) {
    __shared__ int32_t wsum[8];
    int32_t* h = hist + (size_t)blockIdx.x * tiles;
    int32_t base = 0;
    for (int32_t t0 = 0; t0 < tiles; t0 += 256) {
        const int32_t t = t0 + threadIdx.x, v = t < tiles ? h[t] : 0;
        int32_t all;
        const int32_t e = block_exclusive<256>(v, wsum, &all);
        if (t < tiles) h[t] = base + e;
        base += all;
    }
    if (threadIdx.x == 0) total[blockIdx.x] = base;
}

// Stable placement: an edge's rank in its tile is counted in (warp, round,
// lane) order, which is the order of the input.
__global__ void __launch_bounds__(kSortThreads) sort_place_kernel(const int32_t* __restrict__ perm,
                                                                  const int32_t* __restrict__ ids, int64_t m, int shift,
                                                                  int digits, const int32_t* __restrict__ hist,
                                                                  const int32_t* __restrict__ total,
                                                                  int32_t* __restrict__ out) {
    constexpr int W = kSortThreads / 32;
    __shared__ uint16_t cnt[W][kMaxDigits];
    __shared__ int32_t start[kMaxDigits];
    __shared__ int32_t wsum[W];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < W * kMaxDigits; i += kSortThreads) (&cnt[0][0])[i] = 0;
    int32_t all;
    const int32_t first = block_exclusive<kSortThreads>(tid < digits ? total[tid] : 0, wsum, &all);  // syncs
    if (tid < digits) start[tid] = first + hist[(size_t)tid * gridDim.x + blockIdx.x];
    __syncthreads();
    int32_t e[kSortItems], rank[kSortItems], dig[kSortItems];
    const int64_t base = (int64_t)blockIdx.x * kSortTile + warp * (32 * kSortItems) + lane;
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        const int64_t k = base + 32 * r;
        e[r] = k < m ? (perm ? perm[k] : (int32_t)k) : -1;
        dig[r] = e[r] >= 0 ? (ids[e[r]] >> shift) & (digits - 1) : kMaxDigits;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        const unsigned same = __match_any_sync(0xffffffffu, dig[r]);
        const unsigned below = same & ((1u << lane) - 1u);
        int32_t c = 0;
        if (e[r] >= 0) c = cnt[warp][dig[r]];
        rank[r] = c + __popc(below);
        __syncwarp();
        if (e[r] >= 0 && below == 0u) cnt[warp][dig[r]] = (uint16_t)(c + __popc(same));
        __syncwarp();
    }
    __syncthreads();
    if (tid < digits) {  // counts to exclusive sums over the warps
        int32_t s = 0;
        for (int w = 0; w < W; w++) {
            const int32_t c = cnt[w][tid];
            cnt[w][tid] = (uint16_t)s;
            s += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; r++)
        if (e[r] >= 0) out[start[dig[r]] + cnt[warp][dig[r]] + rank[r]] = e[r];
}

// -------------------------------------------------------------- edges kept

// A: every entry with a weight, self-loops apart.  B: of equal (source,
// target) the last, then the same.  `order`: the out-order.  Degrees and
// weighted degrees of the edges kept.
__global__ void keep_edges_kernel(const int32_t* __restrict__ order, const int32_t* __restrict__ src,
                                  const int32_t* __restrict__ dst, const int32_t* __restrict__ w, int64_t m, int side_b,
                                  uint8_t* __restrict__ keep, int32_t* __restrict__ self, int32_t* __restrict__ ocnt,
                                  int32_t* __restrict__ icnt, unsigned long long* __restrict__ wdeg, BuildStats* st) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = order[k], s = src[e], d = dst[e], we = w[e];
        bool ok = we != 0;
        if (side_b && k + 1 < m) {
            const int32_t f = order[k + 1];
            if (src[f] == s && dst[f] == d) ok = false;  // a later entry replaces it
        }
        if (ok && s == d) {
            ok = false;
            st->has_self = 1;
            if (atomicExch(self + s, we) != 0) atomicOr(&st->flags, kBadSelf);  // B: one entry is left, never a second
        }
        keep[e] = ok;
        if (!ok) continue;
        atomicAdd(ocnt + s, 1);
        atomicAdd(icnt + d, 1);
        atomicAdd(wdeg + s, (unsigned long long)we);
        atomicAdd(wdeg + d, (unsigned long long)we);
    }
}

// List offsets, padded to four entries (optr, iptr) and not (optr0, iptr0),
// and the totals.  One block.
__global__ void __launch_bounds__(1024) offsets_kernel(const int32_t* __restrict__ ocnt, const int32_t* __restrict__ icnt,
                                                       const int32_t* __restrict__ self,
                                                       const unsigned long long* __restrict__ wdeg, int32_t n,
                                                       int32_t* __restrict__ optr, int32_t* __restrict__ iptr,
                                                       int32_t* __restrict__ optr0, int32_t* __restrict__ iptr0,
                                                       BuildStats* st) {
    __shared__ int32_t wsum[32];
    int32_t base[4] = {0, 0, 0, 0};
    int32_t deg = 0;
    long long wd = 0;
    for (int32_t v0 = 0; v0 <= n; v0 += 1024) {
        const int32_t v = v0 + threadIdx.x;
        const int32_t o = v <= n ? ocnt[v] : 0, i = v <= n ? icnt[v] : 0;
        const int32_t val[4] = {(o + 3) & ~3, (i + 3) & ~3, o, i};
        int32_t* const ptr[4] = {optr, iptr, optr0, iptr0};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            int32_t all;
            const int32_t ex = block_exclusive<1024>(val[c], wsum, &all);
            if (v <= n) ptr[c][v] = base[c] + ex;
            base[c] += all;
        }
        if (v >= 1 && v <= n) {
            deg = max(deg, o + i);
            wd = max(wd, (long long)wdeg[v] + self[v]);
        }
    }
    atomicMax(&st->max_deg, deg);
    atomicMax(&st->max_wdeg, wd);
    if (threadIdx.x == 0) {
        optr[n + 1] = base[0];
        iptr[n + 1] = base[1];
        st->m_out = base[0];
        st->m_in = base[1];
        st->m_real = base[2];
    }
}

// Edges kept per tile of an order.
__global__ void __launch_bounds__(kSortThreads) kept_count_kernel(const int32_t* __restrict__ order,
                                                                  const uint8_t* __restrict__ keep, int64_t m,
                                                                  int32_t* __restrict__ count) {
    __shared__ int32_t total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    int32_t c = 0;
    for (int i = threadIdx.x; i < kSortTile; i += kSortThreads) {
        const int64_t k = (int64_t)blockIdx.x * kSortTile + i;
        if (k < m) c += keep[order[k]];
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) count[blockIdx.x] = total;
}

// The edges kept go to their lists: the number of kept edges before one in the
// order, less those of earlier vertices, is its place in its list.
__global__ void __launch_bounds__(kSortThreads) place_kernel(const int32_t* __restrict__ order,
                                                             const uint8_t* __restrict__ keep,
                                                             const int32_t* __restrict__ from,
                                                             const int32_t* __restrict__ to, const int32_t* __restrict__ w,
                                                             int64_t m, const int32_t* __restrict__ before,
                                                             const int32_t* __restrict__ ptr, const int32_t* __restrict__ ptr0,
                                                             uint32_t* __restrict__ ent, int32_t* __restrict__ place) {
    __shared__ int32_t wsum[kSortThreads / 32];
    int32_t base = before[blockIdx.x];
    for (int i = 0; i < kSortItems; i++) {
        const int64_t k = (int64_t)blockIdx.x * kSortTile + i * kSortThreads + threadIdx.x;
        const int32_t e = k < m ? order[k] : 0;
        const int32_t ok = k < m ? keep[e] : 0;
        int32_t all;
        const int32_t at = base + block_exclusive<kSortThreads>(ok, wsum, &all);
        base += all;
        if (!ok) continue;  // no barrier below
        const int32_t v = from[e], p = ptr[v] + (at - ptr0[v]);
        ent[p] = bm_pack((uint32_t)to[e], (uint32_t)w[e]);
        if (place) place[e] = p;
    }
}

// A: whether some sorted list names a neighbour more than once.
__global__ void repeats_kernel(const int32_t* __restrict__ ptr, const uint32_t* __restrict__ ent, int32_t n, BuildStats* st) {
    const int lane = threadIdx.x & 31;
    bool dup = false;
    for (int32_t v = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); v <= n; v += (int32_t)((gridDim.x * blockDim.x) >> 5)) {
        const int32_t hi = ptr[v + 1];
        for (int32_t j = ptr[v] + lane; j + 1 < hi; j += 32) {
            const uint32_t a = ent[j], b = ent[j + 1];
            dup |= b != 0u && bm_eid(a) == bm_eid(b);
        }
    }
    if (dup) st->has_dup = 1;
}

// B: twins of the id-sorted lists and the hash table.
__global__ void twins_hash_kernel(const uint8_t* __restrict__ keep, const int32_t* __restrict__ src,
                                  const int32_t* __restrict__ dst, const int32_t* __restrict__ w, int64_t m, int32_t n,
                                  const int32_t* __restrict__ opos, const int32_t* __restrict__ ipos,
                                  int32_t* __restrict__ otw, int32_t* __restrict__ itw, unsigned long long* tab, int log2) {
    const unsigned long long mask = (1ull << log2) - 1ull;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        if (!keep[e]) continue;
        otw[opos[e]] = ipos[e];
        itw[ipos[e]] = opos[e];
        const unsigned long long key = (unsigned long long)src[e] * (unsigned long long)(n + 1) + (unsigned long long)dst[e];
        const unsigned long long val = (key << 16) | (unsigned long long)w[e];
        // keys are distinct and the table at most half full: an empty slot comes
        for (unsigned long long s = bm_hash_slot0(key, log2);; s = (s + 1) & mask)
            if (atomicCAS(tab + s, BM_HASH_EMPTY, val) == BM_HASH_EMPTY) break;
    }
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

// Temporary device memory of one build: up to kStagedScratch in the context's
// staging buffer, which later calls use too (a fresh allocation and its release
// cost a new context milliseconds), above that one allocation given back at
// the end.
constexpr size_t kStagedScratch = (size_t)32 << 20;

struct Arena {
    char* base = nullptr;
    bool own = false;
    size_t used = 0;
    ~Arena() { if (own) bm_cuda_free(base); }
    template <typename T>
    T* take(size_t count) {
        T* p = reinterpret_cast<T*>(base + used);
        used += al256(sizeof(T) * std::max<size_t>(count, 1));
        return p;
    }
};

#define BUILD_TRY(x)                \
    do {                            \
        bm_status _s = (x);         \
        if (_s != BM_OK) return _s; \
    } while (0)

// Two stable passes by `ids` from `in` (null: the identity) to `out`; `mid`
// holds the first pass.
bm_status sort_by(bm_ctx* ctx, const int32_t* in, int32_t* mid, int32_t* out, const int32_t* ids, int64_t m, int bits,
                  int32_t* hist, int32_t* total) {
    const int d = (bits + 1) / 2, digits = 1 << d;
    const int32_t tiles = (int32_t)((m + kSortTile - 1) / kSortTile);
    const int32_t* from = in;
    int32_t* to = mid;
    for (int pass = 0; pass < 2; pass++) {
        sort_count_kernel<<<tiles, kSortThreads, 0, ctx->stream>>>(from, ids, m, pass * d, digits, hist);
        BM_LAUNCH_CHECK(ctx, "sort_count_kernel");
        sort_scan_kernel<<<digits, 256, 0, ctx->stream>>>(hist, tiles, total);
        BM_LAUNCH_CHECK(ctx, "sort_scan_kernel");
        sort_place_kernel<<<tiles, kSortThreads, 0, ctx->stream>>>(from, ids, m, pass * d, digits, hist, total, to);
        BM_LAUNCH_CHECK(ctx, "sort_place_kernel");
        from = to;
        to = out;
    }
    return BM_OK;
}

}  // namespace

// Builds a graph of the context's side B (side_b) or A into G (empty on entry;
// on failure the caller frees what it holds).  *rejected is set, and nothing
// else is to be used, when the layout rejects the input or there is no room
// for the build's scratch (41 bytes an edge).  1 <= n <= BM_MAX_N, 1 <= m.
bm_status bm_build_graph_dev(bm_ctx* ctx, bool side_b, int32_t n, int64_t m, const int32_t* src, const int32_t* dst,
                             const int32_t* w, DevGraph& G, bool* rejected) {
    *rejected = false;
    const int32_t tiles = (int32_t)((m + kSortTile - 1) / kSortTile);
    const size_t M = (size_t)m, V = (size_t)n + 2;
    Arena A;
    const size_t lists = M + 3 * V;  // padding adds at most three entries a list
    const size_t need = al256(sizeof(BuildStats)) + al256(4 * M) * 8 + al256(M) + al256(4 * (size_t)kMaxDigits * tiles) +
                        al256(4 * kMaxDigits) + al256(4 * (size_t)tiles) * 2 + al256(4 * V) * 4 + al256(8 * V) +
                        (side_b ? 0 : 3 * al256(4 * lists)) + 4096;
    if (need <= kStagedScratch) {
        BUILD_TRY(bm_stage(ctx, need));
        A.base = (char*)ctx->stage;
    } else if (bm_cuda_malloc(&A.base, need) != cudaSuccess) {
        cudaGetLastError();
        *rejected = true;
        return BM_OK;
    } else {
        A.own = true;
    }
    BuildStats* st = A.take<BuildStats>(1);
    int32_t* d_src = A.take<int32_t>(M);
    int32_t* d_dst = A.take<int32_t>(M);
    int32_t* d_w = A.take<int32_t>(M);
    int32_t* p0 = A.take<int32_t>(M);
    int32_t* p1 = A.take<int32_t>(M);
    int32_t* out_order = A.take<int32_t>(M);
    int32_t* in_order = A.take<int32_t>(M);
    int32_t* extra = A.take<int32_t>(M);
    uint8_t* keep = A.take<uint8_t>(M);
    int32_t* hist = A.take<int32_t>((size_t)kMaxDigits * tiles);
    int32_t* total = A.take<int32_t>(kMaxDigits);
    int32_t* kept_o = A.take<int32_t>(tiles);
    int32_t* kept_i = A.take<int32_t>(tiles);
    int32_t* ocnt = A.take<int32_t>(V);
    int32_t* icnt = A.take<int32_t>(V);
    int32_t* optr0 = A.take<int32_t>(V);
    int32_t* iptr0 = A.take<int32_t>(V);
    unsigned long long* wdeg = A.take<unsigned long long>(V);
    cudaStream_t sm = ctx->stream;
    BM_CUDA(ctx, cudaMemsetAsync(st, 0, sizeof(BuildStats), sm));
    BM_CUDA(ctx, cudaMemcpyAsync(d_src, src, 4 * M, cudaMemcpyHostToDevice, sm));
    BM_CUDA(ctx, cudaMemcpyAsync(d_dst, dst, 4 * M, cudaMemcpyHostToDevice, sm));
    BM_CUDA(ctx, cudaMemcpyAsync(d_w, w, 4 * M, cudaMemcpyHostToDevice, sm));
    const unsigned grid = (unsigned)std::min<int64_t>((m + 255) / 256, (int64_t)ctx->num_sms * 8);
    check_edges_kernel<<<grid, 256, 0, sm>>>(d_src, d_dst, d_w, m, n, st);
    BM_LAUNCH_CHECK(ctx, "check_edges_kernel");
    BuildStats h;
    BM_CUDA(ctx, cudaMemcpyAsync(&h, st, sizeof h, cudaMemcpyDeviceToHost, sm));
    BM_CUDA(ctx, cudaStreamSynchronize(sm));
    if (h.flags) {  // ids outside 1..n would index past the tables below
        *rejected = true;
        return BM_OK;
    }
    int bits = 1;
    while ((n >> bits) != 0) bits++;
    BUILD_TRY(sort_by(ctx, nullptr, p0, p1, d_dst, m, bits, hist, total));
    BUILD_TRY(sort_by(ctx, p1, p0, out_order, d_src, m, bits, hist, total));
    BUILD_TRY(sort_by(ctx, nullptr, p0, p1, d_src, m, bits, hist, total));
    BUILD_TRY(sort_by(ctx, p1, p0, in_order, d_dst, m, bits, hist, total));
    int64_t cap = 0;
    if (side_b)
        for (cap = 1024, G.hash_log2 = 10; cap < 2 * (m + 1); cap <<= 1) G.hash_log2++;
    BUILD_TRY(bm_graph_alloc(ctx, G, side_b, n, lists, lists, (size_t)cap));
    BM_CUDA(ctx, cudaMemsetAsync(G.self_w, 0, 4 * ((size_t)n + 1), sm));
    BM_CUDA(ctx, cudaMemsetAsync(ocnt, 0, 4 * V, sm));
    BM_CUDA(ctx, cudaMemsetAsync(icnt, 0, 4 * V, sm));
    BM_CUDA(ctx, cudaMemsetAsync(wdeg, 0, 8 * V, sm));
    keep_edges_kernel<<<grid, 256, 0, sm>>>(out_order, d_src, d_dst, d_w, m, side_b, keep, G.self_w, ocnt, icnt, wdeg, st);
    BM_LAUNCH_CHECK(ctx, "keep_edges_kernel");
    offsets_kernel<<<1, 1024, 0, sm>>>(ocnt, icnt, G.self_w, wdeg, n, G.out_ptr, G.in_ptr, optr0, iptr0, st);
    BM_LAUNCH_CHECK(ctx, "offsets_kernel");
    kept_count_kernel<<<tiles, kSortThreads, 0, sm>>>(out_order, keep, m, kept_o);
    BM_LAUNCH_CHECK(ctx, "kept_count_kernel");
    kept_count_kernel<<<tiles, kSortThreads, 0, sm>>>(in_order, keep, m, kept_i);
    BM_LAUNCH_CHECK(ctx, "kept_count_kernel");
    sort_scan_kernel<<<1, 256, 0, sm>>>(kept_o, tiles, total);
    BM_LAUNCH_CHECK(ctx, "sort_scan_kernel");
    sort_scan_kernel<<<1, 256, 0, sm>>>(kept_i, tiles, total);
    BM_LAUNCH_CHECK(ctx, "sort_scan_kernel");
    BM_CUDA(ctx, cudaMemcpyAsync(&h, st, sizeof h, cudaMemcpyDeviceToHost, sm));
    BM_CUDA(ctx, cudaStreamSynchronize(sm));
    if (h.flags || (!side_b && h.max_wdeg >= (1ll << 29))) {
        *rejected = true;
        return BM_OK;
    }
    const size_t mo = (size_t)h.m_out, mi = (size_t)h.m_in;
    G.n = n;
    G.m_out = h.m_out;
    G.m_in = h.m_in;
    G.m_real = h.m_real;
    G.max_deg = h.max_deg;
    G.max_wdeg = h.max_wdeg;
    G.has_self = h.has_self;
    uint32_t *oent, *ient;  // id-sorted
    int32_t* tmp = nullptr;
    if (side_b) {
        BM_CUDA(ctx, cudaMemsetAsync(G.hash, 0xFF, 8 * (size_t)cap, sm));
        BM_CUDA(ctx, cudaMemsetAsync(G.out_twin0, 0xFF, 4 * mo, sm));
        BM_CUDA(ctx, cudaMemsetAsync(G.in_twin0, 0xFF, 4 * mi, sm));
        oent = G.out_ent0;
        ient = G.in_ent0;
    } else {
        oent = A.take<uint32_t>(lists);
        ient = A.take<uint32_t>(lists);
        tmp = A.take<int32_t>(lists);
    }
    BM_CUDA(ctx, cudaMemsetAsync(oent, 0, 4 * mo, sm));
    BM_CUDA(ctx, cudaMemsetAsync(ient, 0, 4 * mi, sm));
    int32_t *opos = side_b ? p0 : nullptr, *ipos = side_b ? extra : nullptr;
    place_kernel<<<tiles, kSortThreads, 0, sm>>>(out_order, keep, d_src, d_dst, d_w, m, kept_o, G.out_ptr, optr0, oent, opos);
    BM_LAUNCH_CHECK(ctx, "place_kernel(out)");
    place_kernel<<<tiles, kSortThreads, 0, sm>>>(in_order, keep, d_dst, d_src, d_w, m, kept_i, G.in_ptr, iptr0, ient, ipos);
    BM_LAUNCH_CHECK(ctx, "place_kernel(in)");
    if (side_b) {
        twins_hash_kernel<<<grid, 256, 0, sm>>>(keep, d_src, d_dst, d_w, m, n, opos, ipos, G.out_twin0, G.in_twin0, G.hash,
                                                G.hash_log2);
        BM_LAUNCH_CHECK(ctx, "twins_hash_kernel");
        BM_CUDA(ctx, cudaStreamSynchronize(sm));
    } else {
        // A's device lists in bank-spread order (the row kernel's scatter); the
        // host copy keeps them sorted by neighbour id
        repeats_kernel<<<(unsigned)std::min((n + 8) / 8, ctx->num_sms * 8), 256, 0, sm>>>(G.out_ptr, oent, n, st);
        BM_LAUNCH_CHECK(ctx, "repeats_kernel");
        BM_CUDA(ctx, cudaMemcpyAsync(&h, st, sizeof h, cudaMemcpyDeviceToHost, sm));
        BUILD_TRY(bm_launch_spread(ctx, n, G.out_ptr, G.in_ptr, oent, ient, G.out_ent, G.in_ent, tmp));
        ctx->hA_optr.resize(V);
        ctx->hA_iptr.resize(V);
        ctx->hA_oent.resize(mo);
        ctx->hA_ient.resize(mi);
        BM_CUDA(ctx, cudaMemcpyAsync(ctx->hA_optr.data(), G.out_ptr, 4 * V, cudaMemcpyDeviceToHost, sm));
        BM_CUDA(ctx, cudaMemcpyAsync(ctx->hA_iptr.data(), G.in_ptr, 4 * V, cudaMemcpyDeviceToHost, sm));
        BM_CUDA(ctx, cudaMemcpyAsync(ctx->hA_oent.data(), oent, 4 * mo, cudaMemcpyDeviceToHost, sm));
        BM_CUDA(ctx, cudaMemcpyAsync(ctx->hA_ient.data(), ient, 4 * mi, cudaMemcpyDeviceToHost, sm));
        BM_CUDA(ctx, cudaStreamSynchronize(sm));
        G.has_dup = h.has_dup;
    }
    return BM_OK;
}
