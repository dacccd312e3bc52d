// bm_apply.cu — commit swaps pi(a) <-> pi(b) on the device.
//
// The reference swaps two mapping entries and re-scores the whole graph after
// every accept (src/graph-alignment-optimized.c:556-576).  Here one CTA per
// swap updates only what the swap changes:
//   * S(v) for a, b and their A neighbours: each A entry incident to a or b
//     changes its contribution from min(w, B(old ends)) to min(w, B(new ends));
//     the difference is added to both endpoints' S;
//   * the relabelled B lists: every B entry that names image pi(a) now names
//     A vertex b and vice versa; the entries are found through the twin index
//     of the reverse direction, so the update costs O(deg_B);
//   * pi and pi^-1.
// Swaps in one launch must be pairwise independent (no shared vertex and no A
// edge between their endpoint sets), so no entry is touched by two swaps and
// no swap reads a mapping entry that another one writes.
#include <algorithm>

#include "bm_internal.cuh"

namespace {

constexpr int kApplyThreads = 512;

struct ApplyArgs {
    GView A;
    const int32_t* Bout_ptr;
    const int32_t* Bin_ptr;
    uint32_t* Bout_ent;
    uint32_t* Bin_ent;
    const int32_t* Bout_twin;
    const int32_t* Bin_twin;
    HashView hb;
    int32_t* pi;
    int32_t* pinv;
    int32_t* ov;
    int4* ximg;
};

// What the mapping arrays become.
__device__ __forceinline__ void finish_swap(const ApplyArgs& a, int32_t sa, int32_t sb, int32_t fa, int32_t fb) {
    a.pi[sa] = fb;
    a.pi[sb] = fa;
    a.pinv[fa] = sb;
    a.pinv[fb] = sa;
    a.ximg[sa] = bm_image_bounds(a.Bin_ptr, a.Bout_ptr, fb);
    a.ximg[sb] = bm_image_bounds(a.Bin_ptr, a.Bout_ptr, fa);
}

// The four A lists of a swap (S updates) and the four B lists of its images
// (relabelling) form one stream of entries over the threads of the swap's
// blocks, so that a swap is one chain of dependent loads, not eight.  A hub's
// 16,000 entries are shared by several blocks (blockIdx.y); the mapping arrays,
// which they all read, then change in a launch of their own
// (apply_finish_kernel), else at the end of the block.
__global__ void __launch_bounds__(kApplyThreads) apply_kernel(ApplyArgs a, const int32_t* __restrict__ pairs) {
    const int32_t sa = __ldg(pairs + 2 * blockIdx.x), sb = __ldg(pairs + 2 * blockIdx.x + 1);
    if (sa == sb) return;
    const int32_t fa = a.pi[sa], fb = a.pi[sb];
    const int4 xa = a.ximg[sa], xb = a.ximg[sb];
    // lists 0..3: out(sa), in(sa), out(sb), in(sb) of A; 4..7: B-in and B-out
    // of fa (whose entries now name sb), of fb (now sa)
    const int32_t beg[8] = {__ldg(a.A.out_ptr + sa), __ldg(a.A.in_ptr + sa), __ldg(a.A.out_ptr + sb),
                            __ldg(a.A.in_ptr + sb), xa.x, xa.z, xb.x, xb.z};
    const int32_t fin[8] = {__ldg(a.A.out_ptr + sa + 1), __ldg(a.A.in_ptr + sa + 1), __ldg(a.A.out_ptr + sb + 1),
                            __ldg(a.A.in_ptr + sb + 1), xa.y, xa.w, xb.y, xb.w};
    int32_t total = 0;
#pragma unroll
    for (int l = 0; l < 8; l++) total += fin[l] - beg[l];
    for (int32_t j = (int32_t)blockIdx.y * kApplyThreads + (int32_t)threadIdx.x; j < total;
         j += (int32_t)gridDim.y * kApplyThreads) {
        int l = 0;
        int32_t at = j;
        bool found = false;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int32_t len = fin[q] - beg[q];
            if (!found) {
                if (at < len) { l = q; at += beg[q]; found = true; }
                else at -= len;
            }
        }
        if (l >= 4) {
            const bool out = l & 1;  // twins of B-out entries are in the in-lists
            const int32_t t = out ? a.Bout_twin[at] : a.Bin_twin[at];
            if (t < 0) continue;  // list padding
            uint32_t* e = (out ? a.Bin_ent : a.Bout_ent) + t;
            *e = (*e & ~BM_ID_MASK) | (uint32_t)(l < 6 ? sb : sa);
            continue;
        }
        const bool out = !(l & 1), of_a = l < 2;
        const uint32_t ent = __ldg((out ? a.A.out_ent : a.A.in_ent) + at);
        if (ent == 0) continue;  // list padding
        const int32_t x = bm_eid(ent), w = bm_ew(ent);
        const int32_t me = of_a ? sa : sb, other = of_a ? sb : sa;
        const int32_t fme = of_a ? fa : fb, fnew = of_a ? fb : fa;  // my image before / after
        int32_t g0, h0, g1, h1;  // the B edge before and after
        if (x == other) {
            if (!out) continue;  // the edge other -> me is handled as other's out-entry
            g0 = fme; h0 = fnew; g1 = fnew; h1 = fme;
        } else {
            const int32_t gx = a.pi[x];
            g0 = out ? fme : gx; h0 = out ? gx : fme;
            g1 = out ? fnew : gx; h1 = out ? gx : fnew;
        }
        const int32_t d = imin(w, bm_hash_get(a.hb, g1, h1)) - imin(w, bm_hash_get(a.hb, g0, h0));
        if (d) { atomicAdd(a.ov + me, d); atomicAdd(a.ov + x, d); }
    }
    if (gridDim.y == 1) {
        __syncthreads();
        if (threadIdx.x == 0) finish_swap(a, sa, sb, fa, fb);
    }
}

__global__ void apply_finish_kernel(ApplyArgs a, const int32_t* __restrict__ pairs, int32_t k) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
        const int32_t sa = pairs[2 * i], sb = pairs[2 * i + 1];
        if (sa != sb) finish_swap(a, sa, sb, a.pi[sa], a.pi[sb]);
    }
}

}  // namespace

bm_status bm_launch_apply(bm_ctx* ctx, const int32_t* d_pairs, int32_t k) {
    if (k <= 0) return BM_OK;
    const DevGraph& B = ctx->g[1];
    ApplyArgs a;
    a.A = gview(ctx->g[0]);
    a.Bout_ptr = B.out_ptr;
    a.Bin_ptr = B.in_ptr;
    a.Bout_ent = B.out_ent;
    a.Bin_ent = B.in_ent;
    a.Bout_twin = B.out_twin;
    a.Bin_twin = B.in_twin;
    a.hb = hview(B);
    a.pi = ctx->pi;
    a.pinv = ctx->pinv;
    a.ov = ctx->ov;
    a.ximg = ctx->ximg;
    // blocks of a swap: about four entries a thread of the largest swap's lists
    // (A's and B's largest degrees twice), up to 32 blocks and while the swaps
    // leave room for them.  The late launches of a full-scale search, whose swaps
    // are hubs': 55 us in one block of 256 threads a swap, list by list, 11 us so;
    // a swap of the 2,000-vertex pair 12.5 and 5.3 us
    const int64_t most = 2 * ((int64_t)ctx->g[0].max_deg + B.max_deg);
    const unsigned parts = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>({(most + 2 * kApplyThreads - 1) / (4 * kApplyThreads), (int64_t)ctx->num_sms * 8 / k, 32}));
    apply_kernel<<<dim3((unsigned)k, parts), kApplyThreads, 0, ctx->stream>>>(a, d_pairs);
    BM_LAUNCH_CHECK(ctx, "apply_kernel");
    if (parts > 1) {
        apply_finish_kernel<<<(k + 255) / 256, 256, 0, ctx->stream>>>(a, d_pairs, k);
        BM_LAUNCH_CHECK(ctx, "apply_finish_kernel");
    }
    return BM_OK;
}
