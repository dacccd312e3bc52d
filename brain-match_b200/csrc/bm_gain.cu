// bm_gain.cu — one-sided gains of all rows kept across a search.
//
// G_u(f) = sum over u's A entries of min(w, B at f and the neighbour's image)
// is u's overlap if it alone took image f.  With the row table T[u][v] = G_u(pi v)
// and its transpose H (row hrow[v] holds G_u(pi v) for all u), the deltas of
// row u are read, not scattered:
//   delta(u, v) = T[u][v] + H[hrow u][v] - S(u) - S(v) + self-loop terms + direct edges:
// two streams of n values instead of about a million 2-hop entries.
//
// A swap of a and b changes G_u only for neighbours u of a or b, and only by
// the terms of the edges between them: with w0..w3 the weights of u -> a,
// u -> b, a -> u, b -> u and v0..v3 those of f -> pi a, f -> pi b, pi a -> f,
// pi b -> f, G_u(f) grows by
//   min(w0, v1) - min(w0, v0) + min(w1, v0) - min(w1, v1)
//   + min(w2, v3) - min(w2, v2) + min(w3, v2) - min(w3, v3).
// gain_lists_kernel lists, in order of their ids, the u with any w and the f
// with any v; gain_product_kernel adds the outer product to both tables (with
// the roles of rows and columns changed), consecutive threads on consecutive
// columns: the late swaps of a search are its hubs', whose lists cover much of
// a row, and updates in list order, a 32-byte sector each, took 431 us a batch
// of swaps of the full-scale search against 140 with the lists.  Then the swap
// itself: columns a and b of T change places, and rows of H by hrow.
//
// A search that accepts thousands of swaps a pass is better off scattering
// rows; one that accepts a few hundred and fewer is not (bm_gains_pay).
#include <algorithm>
#include <climits>

#include "bm_internal.cuh"

namespace {

constexpr int kBestThreads = 512;
constexpr int32_t kGainSwaps = 64;  // swaps whose lists are held at once

struct BestArgs {
    const int32_t* T;
    const int32_t* H;
    int64_t ld;
    const int32_t* hrow;
    GView A;
    HashView hb;
    const int32_t* selfB;
    const int32_t* pi;
    const int32_t* ov;
    int has_self;
    int32_t n;
    const int32_t* rows;
    bm_row_result* res;
};

// One row per block: the direct-edge terms are summed per column in shared
// memory, then the row's two streams are read once, 16 bytes at a time.
__global__ void __launch_bounds__(kBestThreads) gain_best_kernel(BestArgs a) {
    extern __shared__ __align__(16) int32_t corr[];
    __shared__ int32_t s_v[kBestThreads / 32];
    __shared__ int32_t s_d[kBestThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int32_t n = a.n, groups = (n + 4) / 4;
    const int32_t u = __ldg(a.rows + blockIdx.x);
    for (int32_t g = tid; g < groups; g += kBestThreads) reinterpret_cast<int4*>(corr)[g] = make_int4(0, 0, 0, 0);
    const int32_t fu = __ldg(a.pi + u);
    const int32_t o0 = __ldg(a.A.out_ptr + u), o1 = __ldg(a.A.out_ptr + u + 1);
    const int32_t i0 = __ldg(a.A.in_ptr + u), i1 = __ldg(a.A.in_ptr + u + 1);
    __syncthreads();
    for (int32_t j = tid; j < (o1 - o0) + (i1 - i0); j += kBestThreads) {
        const uint32_t e = j < o1 - o0 ? __ldg(a.A.out_ent + o0 + j) : __ldg(a.A.in_ent + i0 + (j - (o1 - o0)));
        if (!e) continue;  // list padding
        const int32_t x = bm_eid(e), w = bm_ew(e), fx = __ldg(a.pi + x);
        const int32_t c = imin(w, bm_hash_get(a.hb, fu, fx)) + imin(w, bm_hash_get(a.hb, fx, fu));
        if (c) atomicAdd(corr + x, c);
    }
    __syncthreads();
    const int4* trow = reinterpret_cast<const int4*>(a.T + (size_t)u * a.ld);
    const int4* hrow = reinterpret_cast<const int4*>(a.H + (size_t)__ldg(a.hrow + u) * a.ld);
    const int4* ov4 = reinterpret_cast<const int4*>(a.ov);
    const int32_t ovu = __ldg(a.ov + u);
    int32_t sau = 0, sbu = 0;
    if (a.has_self) { sau = __ldg(a.A.self_w + u); sbu = __ldg(a.selfB + fu); }
    // deltas stay below 2^31 (the row kernel's bound on weighted degrees)
    int32_t bd = INT_MIN, bv = INT_MAX;
#pragma unroll 4
    for (int32_t g = tid; g < groups; g += kBestThreads) {
        const int4 l = __ldcs(trow + g), h = __ldcs(hrow + g), o = __ldg(ov4 + g);
        const int4 c = reinterpret_cast<const int4*>(corr)[g];
        const int32_t ll[4] = {l.x, l.y, l.z, l.w}, hh[4] = {h.x, h.y, h.z, h.w}, oo[4] = {o.x, o.y, o.z, o.w},
                      cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int32_t v = 4 * g + k;
            if (v < 1 || v > n || v == u) continue;
            int32_t d = ll[k] + hh[k] - ovu - oo[k] + cc[k];
            if (a.has_self) {
                const int32_t sav = __ldg(a.A.self_w + v), sbv = __ldg(a.selfB + __ldg(a.pi + v));
                d += imin(sau, sbv) - imin(sau, sbu) + imin(sav, sbu) - imin(sav, sbv);
            }
            if (d > bd) { bd = d; bv = v; }  // columns ascend: the first of equal ones stays
        }
    }
    for (int o = 16; o; o >>= 1) {
        const int32_t d2 = __shfl_xor_sync(0xffffffffu, bd, o), v2 = __shfl_xor_sync(0xffffffffu, bv, o);
        if (d2 > bd || (d2 == bd && v2 < bv)) { bd = d2; bv = v2; }
    }
    if (lane == 0) { s_d[warp] = bd; s_v[warp] = bv; }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kBestThreads / 32; w++)
            if (s_d[w] > bd || (s_d[w] == bd && s_v[w] < bv)) { bd = s_d[w]; bv = s_v[w]; }
        bm_row_result r;
        r.row = u;
        r.first_pos = 0;
        r.npos = 0;
        r.first_delta = 0;
        r.best = bv == INT_MAX ? 0 : bv;
        r.best_delta = bv == INT_MAX ? 0 : bd;
        a.res[blockIdx.x] = r;
    }
}

// H = T transposed, 32 x 32 tiles; columns past n are left alone.
__global__ void __launch_bounds__(256) transpose_kernel(const int32_t* __restrict__ T, int32_t* __restrict__ H, int64_t ld,
                                                        int32_t n) {
    __shared__ int32_t t[32][33];
    const int32_t u0 = blockIdx.y * 32, c0 = blockIdx.x * 32, x = threadIdx.x & 31, y0 = threadIdx.x >> 5;
#pragma unroll
    for (int y = y0; y < 32; y += 8)
        if (u0 + y <= n && c0 + x <= n) t[y][x] = __ldcs(T + (size_t)(u0 + y) * ld + c0 + x);
    __syncthreads();
#pragma unroll
    for (int y = y0; y < 32; y += 8)
        if (c0 + y <= n && u0 + x <= n) __stcs(H + (size_t)(c0 + y) * ld + u0 + x, t[x][y]);
}

// One side's list of a swap: ids in ascending order with their four weights.
struct SwapList {
    int32_t* idx;
    uint2* w;  // x: w0 | w1 << 16, y: w2 | w3 << 16
    int32_t* count;
};

struct ListArgs {
    GView A;
    const uint32_t* Bout_ent;  // live: ids in A space
    const uint32_t* Bin_ent;
    const int4* ximg;
    int32_t n;
    const int32_t* pairs;
    int32_t* idx;    // [swap][side][cap]
    uint2* w;
    int32_t* count;  // [swap][side]
    int32_t cap;
};

constexpr int kListThreads = 1024;
constexpr int kListRange = 16384;  // ids marked at a time: 128 KB of weights

// blockIdx.y 0: the A side (u), 1: the B side (f, by the vertex that holds it).
__global__ void __launch_bounds__(kListThreads, 1) gain_lists_kernel(ListArgs a) {
    extern __shared__ __align__(16) uint16_t mark[];  // [kListRange][4]
    __shared__ int32_t wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, side = blockIdx.y;
    const int32_t sa = __ldg(a.pairs + 2 * blockIdx.x), sb = __ldg(a.pairs + 2 * blockIdx.x + 1);
    const size_t at = (size_t)(2 * blockIdx.x + side);
    int32_t* idx = a.idx + at * a.cap;
    uint2* out = a.w + at * a.cap;
    const uint32_t* ent[4];
    int32_t beg[4], end[4];
    const int4 xa = __ldg(a.ximg + sa), xb = __ldg(a.ximg + sb);
#pragma unroll
    for (int k = 0; k < 4; k++) {  // into a, into b, out of a, out of b
        const int32_t x = (k & 1) ? sb : sa;
        const int4 im = (k & 1) ? xb : xa;
        if (side == 0) {
            const int32_t* ptr = k < 2 ? a.A.in_ptr : a.A.out_ptr;
            ent[k] = k < 2 ? a.A.in_ent : a.A.out_ent;
            beg[k] = __ldg(ptr + x);
            end[k] = __ldg(ptr + x + 1);
        } else {
            ent[k] = k < 2 ? a.Bin_ent : a.Bout_ent;
            beg[k] = k < 2 ? im.x : im.z;
            end[k] = k < 2 ? im.y : im.w;
        }
    }
    int32_t total = 0;
    for (int32_t lo = 0; lo <= a.n; lo += kListRange) {
        for (int32_t i = tid; i < kListRange / 2; i += kListThreads)
            reinterpret_cast<uint4*>(mark)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++)
            for (int32_t j = beg[k] + tid; j < end[k]; j += kListThreads) {
                const uint32_t e = ent[k][j];
                const int32_t i = bm_eid(e) - lo;
                if (e && i >= 0 && i < kListRange) mark[4 * i + k] = (uint16_t)bm_ew(e);  // an id is in a list once
            }
        __syncthreads();
        for (int32_t i0 = 0; i0 < kListRange && lo + i0 <= a.n; i0 += kListThreads) {
            const uint2 m = reinterpret_cast<const uint2*>(mark)[i0 + tid];
            const bool any = (m.x | m.y) != 0u;
            const unsigned b = __ballot_sync(0xffffffffu, any);
            if (lane == 0) wsum[warp] = __popc(b);
            __syncthreads();
            int32_t before = total, all = 0;
            for (int w = 0; w < 32; w++) {
                if (w < warp) before += wsum[w];
                all += wsum[w];
            }
            if (any) {
                const int32_t p = before + __popc(b & ((1u << lane) - 1u));
                idx[p] = lo + i0 + tid;
                out[p] = m;
            }
            total += all;
            __syncthreads();
        }
    }
    if (tid == 0) a.count[at] = total;
}

struct ProductArgs {
    int32_t* T;
    int32_t* H;
    int64_t ld;
    const int32_t* hrow;
    const int32_t* idx;
    const uint2* w;
    const int32_t* count;
    int32_t cap;
};

constexpr int kProdThreads = 256;
constexpr int kProdCols = 4 * kProdThreads;  // columns of a tile: four a thread, kept in registers
constexpr int kProdRows = 64;

__device__ __forceinline__ int32_t swap_term(const uint2& w, const uint2& v) {
    const int32_t w0 = w.x & 0xFFFF, w1 = w.x >> 16, w2 = w.y & 0xFFFF, w3 = w.y >> 16;
    const int32_t v0 = v.x & 0xFFFF, v1 = v.x >> 16, v2 = v.y & 0xFFFF, v3 = v.y >> 16;
    return imin(w0, v1) - imin(w0, v0) + imin(w1, v0) - imin(w1, v1) + imin(w2, v3) - imin(w2, v2) + imin(w3, v2) -
           imin(w3, v3);
}

// blockIdx.y: swap; blockIdx.z 0: T (rows u, columns f), 1: H (rows f, columns
// u).  Swaps of one launch may meet in an entry, hence the atomics.
__global__ void __launch_bounds__(kProdThreads) gain_product_kernel(ProductArgs a) {
    __shared__ int64_t s_row[kProdRows];
    __shared__ uint2 s_w[kProdRows];
    const int tid = threadIdx.x, z = blockIdx.z;
    const size_t rl = 2 * (size_t)blockIdx.y + z, cl = 2 * (size_t)blockIdx.y + (1 - z);
    const int32_t nr = __ldg(a.count + rl), nc = __ldg(a.count + cl);
    const int32_t *ridx = a.idx + rl * a.cap, *cidx = a.idx + cl * a.cap;
    const uint2 *rw = a.w + rl * a.cap, *cw = a.w + cl * a.cap;
    int32_t* M = z ? a.H : a.T;
    const int32_t rt = (nr + kProdRows - 1) / kProdRows, ct = (nc + kProdCols - 1) / kProdCols;
    for (int32_t t = blockIdx.x; t < rt * ct; t += gridDim.x) {
        const int32_t r0 = (t / ct) * kProdRows, c0 = (t % ct) * kProdCols, rows = min(kProdRows, nr - r0);
        __syncthreads();
        if (tid < rows) {
            const int32_t id = __ldg(ridx + r0 + tid);
            s_row[tid] = (int64_t)(z ? __ldg(a.hrow + id) : id) * a.ld;
            s_w[tid] = __ldg(rw + r0 + tid);
        }
        int32_t col[4];
        uint2 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int32_t c = c0 + k * kProdThreads + tid;
            col[k] = c < nc ? __ldg(cidx + c) : 0;
            v[k] = c < nc ? __ldg(cw + c) : make_uint2(0u, 0u);  // no weights: no term
        }
        __syncthreads();
        for (int32_t r = 0; r < rows; r++) {
            const uint2 w = s_w[r];
            int32_t* row = M + s_row[r];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                // the term is the same with the roles changed
                const int32_t d = z ? swap_term(v[k], w) : swap_term(w, v[k]);
                if (d) atomicAdd(row + col[k], d);
            }
        }
    }
}

// After the swaps: their columns of T change places, and their rows of H.
__global__ void gain_swap_kernel(const int32_t* __restrict__ pairs, int32_t* T, int64_t ld, int32_t n, int32_t* hrow) {
    const int32_t a = __ldg(pairs + 2 * blockIdx.y), b = __ldg(pairs + 2 * blockIdx.y + 1);
    for (int32_t u = blockIdx.x * blockDim.x + threadIdx.x; u <= n; u += gridDim.x * blockDim.x) {
        int32_t* row = T + (size_t)u * ld;
        const int32_t x = row[a], y = row[b];
        row[a] = y;
        row[b] = x;
        if (u == 0) {
            const int32_t h = hrow[a];
            hrow[a] = hrow[b];
            hrow[b] = h;
        }
    }
}

__global__ void gain_iota_kernel(int32_t* a, int32_t lo, int32_t n) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = lo + i;
}

size_t best_smem(int32_t n) { return sizeof(int32_t) * 4 * (size_t)((n + 4) / 4); }

}  // namespace

void bm_gains_free(BmGains* g) {
    bm_cuda_free(g->mem);
    *g = BmGains();
}

bool bm_gains_possible(bm_ctx* ctx) {
    if (ctx->g[0].has_dup) return false;  // the terms of a repeated edge do not add up to one weight's
    if (ctx->semantics == BM_SEMANTICS_REF_CPU && ctx->g[0].has_self) return false;  // its self-loop terms are per pair
    return best_smem(ctx->n) + 1024 <= ctx->smem_optin;
}

// In units of scattered 2-hop entries (1.9e12 a second on a B200): a pass over
// the search's rows scatters theirs, `scatter` together; reading the tables
// costs about 4 a table entry, and an entry of a swap's product 4.  Products are
// taken as 64 times mean lists' (late swaps are hubs').  Filling the tables
// costs about half a pass over all W entries of the graph, whatever rows the
// search visits; it has to come back within the next four passes, or those that
// are left (`passes`, -1: no limit), and so has what does not depend on the
// sizes, the allocation, its release and the launches, about half a millisecond
// (five passes over 524 vertices: 1.47 ms with the tables, 0.90 ms without).
bool bm_gains_pay(const bm_ctx* ctx, const std::vector<int32_t>& order, int64_t pass_accepts, double passes) {
    if (ctx->h_rwork.size() != (size_t)ctx->n + 1) return false;
    double W = 0, scatter = 0;
    for (int32_t w : ctx->h_rwork) W += w;
    for (int32_t u : order) scatter += ctx->h_rwork[(size_t)u];
    const double n = ctx->n, d = (double)ctx->g[0].m_out / n, db = (double)ctx->g[1].m_out / n;
    const double update = 64.0 * d * db * 4.0;
    const double r = passes < 0 ? 4.0 : std::min(4.0, passes);
    const double fixed = 1e9;
    return r * ((double)pass_accepts * update + 4.0 * n * (double)order.size()) + 0.45 * W + 4.0 * n * n + fixed <
           0.9 * r * scatter;
}

// Fills the tables for the current mapping.  *ok is false, and nothing is
// held, when there is no room for them (at most half of the free memory).
bm_status bm_gains_build(bm_ctx* ctx, BmGains* g, bool* ok) {
    *ok = false;
    bm_gains_free(g);
    const int32_t n = ctx->n;
    const size_t ld = (size_t)((n + 1 + 3) & ~3);
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t tab = al(sizeof(int32_t) * ld * ((size_t)n + 1)), vec = al(sizeof(int32_t) * ld);
    const size_t lists = 2 * (size_t)kGainSwaps * ld;
    size_t free_b = 0, total_b = 0;
    BM_CUDA(ctx, cudaMemGetInfo(&free_b, &total_b));
    const size_t need = 2 * tab + 2 * vec + al(12 * lists) + al(8 * (size_t)kGainSwaps);
    if (need > free_b / 2) return BM_OK;
    if (bm_cuda_malloc(&g->mem, need) != cudaSuccess) {
        cudaGetLastError();
        return BM_OK;
    }
    char* base = (char*)g->mem;
    g->T = (int32_t*)base;
    g->H = (int32_t*)(base + tab);
    g->hrow = (int32_t*)(base + 2 * tab);
    int32_t* rows = (int32_t*)(base + 2 * tab + vec);
    g->list_w = (uint2*)(base + 2 * tab + 2 * vec);
    g->list_idx = (int32_t*)(g->list_w + lists);
    g->list_n = (int32_t*)(base + 2 * tab + 2 * vec + al(12 * lists));
    g->ld = (int64_t)ld;
    gain_iota_kernel<<<64, 256, 0, ctx->stream>>>(rows, 1, n);
    BM_LAUNCH_CHECK(ctx, "gain_iota_kernel");
    gain_iota_kernel<<<64, 256, 0, ctx->stream>>>(g->hrow, 0, n + 1);
    BM_LAUNCH_CHECK(ctx, "gain_iota_kernel");
    BM_CUDA(ctx, cudaMemsetAsync(g->T, 0, sizeof(int32_t) * ld, ctx->stream));
    bm_status s = bm_launch_rows_gen(ctx, rows, nullptr, n, nullptr, nullptr, g->T, g->ld, 0, nullptr, 0, nullptr, nullptr, true);
    if (s != BM_OK) return s;
    const unsigned t = (unsigned)((n + 32) / 32);
    transpose_kernel<<<dim3(t, t), 256, 0, ctx->stream>>>(g->T, g->H, g->ld, n);
    BM_LAUNCH_CHECK(ctx, "transpose_kernel");
    BM_CUDA(ctx, cudaFuncSetAttribute(gain_best_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)best_smem(n)));
    BM_CUDA(ctx, cudaFuncSetAttribute(gain_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * kListRange));
    *ok = true;
    return BM_OK;
}

// Best partner of each row (best, best_delta; the other fields are 0).  The
// rows are ids in 1..n.
bm_status bm_gains_rows_best(bm_ctx* ctx, const BmGains& g, const int32_t* d_rows, int32_t nrows, bm_row_result* d_res) {
    if (nrows <= 0) return BM_OK;
    const DevGraph &A = ctx->g[0], &B = ctx->g[1];
    const BestArgs a{g.T,     g.H,     g.ld,  g.hrow,  gview(A), hview(B), B.self_w, ctx->pi,
                     ctx->ov, A.has_self && B.has_self, ctx->n, d_rows,   d_res};
    gain_best_kernel<<<nrows, kBestThreads, best_smem(ctx->n), ctx->stream>>>(a);
    BM_LAUNCH_CHECK(ctx, "gain_best_kernel");
    return BM_OK;
}

// The swaps of d_pairs (independent) in the tables and in the mapping.
bm_status bm_gains_apply(bm_ctx* ctx, const BmGains& g, const int32_t* d_pairs, int32_t k) {
    if (k <= 0) return BM_OK;
    const DevGraph &A = ctx->g[0], &B = ctx->g[1];
    for (int32_t k0 = 0; k0 < k; k0 += kGainSwaps) {
        const int32_t kc = std::min(k - k0, kGainSwaps);
        const ListArgs la{gview(A), B.out_ent,  B.in_ent, ctx->ximg, ctx->n, d_pairs + 2 * k0,
                          g.list_idx, g.list_w, g.list_n, (int32_t)g.ld};
        gain_lists_kernel<<<dim3((unsigned)kc, 2), kListThreads, 8 * kListRange, ctx->stream>>>(la);
        BM_LAUNCH_CHECK(ctx, "gain_lists_kernel");
        const ProductArgs pa{g.T, g.H, g.ld, g.hrow, g.list_idx, g.list_w, g.list_n, (int32_t)g.ld};
        const unsigned parts = (unsigned)std::max(8, std::min(ctx->num_sms * 4, ctx->num_sms * 8 / kc));
        gain_product_kernel<<<dim3(parts, (unsigned)kc, 2), kProdThreads, 0, ctx->stream>>>(pa);
        BM_LAUNCH_CHECK(ctx, "gain_product_kernel");
    }
    const bm_status s = bm_launch_apply(ctx, d_pairs, k);
    if (s != BM_OK) return s;
    for (int32_t k0 = 0; k0 < k; k0 += 65535) {  // grid.y
        const unsigned kc = (unsigned)std::min(k - k0, 65535);
        gain_swap_kernel<<<dim3((unsigned)((ctx->n + 512) / 512), kc), 256, 0, ctx->stream>>>(d_pairs + 2 * k0, g.T, g.ld,
                                                                                            ctx->n, g.hrow);
        BM_LAUNCH_CHECK(ctx, "gain_swap_kernel");
    }
    return BM_OK;
}
