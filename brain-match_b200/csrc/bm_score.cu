// bm_score.cu — full overlap score and per-vertex overlap, and the
// relabelling of B's lists into A space (with their bank-spread order and
// twins).
//
// score(pi) = sum over A entries (x->y, w) of min(w, w_B(pi x, pi y)), the sum
// of calculate_alignment_score (src/graph-alignment-optimized.c:292-307).
// Warps take fixed stretches of A's out-entries, whatever lists they fall in
// (a warp per vertex left a hub's 8,000 entries to one warp: 340 us at full
// scale, against 60 us so), look up w_B(pi u, pi x) in B's hash table and add
// min(w, w_B) to S(u) and S(x).  Self-loops are scored from the two
// self-weight arrays.
#include <algorithm>

#include "bm_internal.cuh"

namespace {

constexpr int kScoreThreads = 256;

constexpr int kScoreStretch = 256;  // out-entries of a warp's stretch

__global__ void __launch_bounds__(kScoreThreads)
score_kernel(GView A, HashView hb, const int32_t* __restrict__ selfB, const int32_t* __restrict__ pi, int32_t n,
             int32_t* __restrict__ ov, unsigned long long* __restrict__ total) {
    __shared__ unsigned long long block_sum[kScoreThreads / 32];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int32_t m = __ldg(A.out_ptr + n + 1);
    unsigned long long mine = 0;  // this thread's share of the score
    for (int32_t u = 1 + blockIdx.x * kScoreThreads + threadIdx.x; u <= n; u += gridDim.x * kScoreThreads) {
        const int32_t sw = __ldg(A.self_w + u);
        if (sw) mine += (unsigned long long)imin(sw, __ldg(selfB + __ldg(pi + u)));
    }
    for (int32_t c = blockIdx.x * (kScoreThreads / 32) + warp; (int64_t)c * kScoreStretch < m;
         c += gridDim.x * (kScoreThreads / 32)) {
        const int32_t j0 = c * kScoreStretch, j1 = imin(m, j0 + kScoreStretch);
        // the list that entry j0 falls in: the last u with out_ptr[u] <= j0
        int32_t lo = 0, hi = n;
        while (lo < hi) {
            const int32_t mid = (lo + hi + 1) >> 1;
            if (__ldg(A.out_ptr + mid) <= j0) lo = mid; else hi = mid - 1;
        }
        int32_t u = lo, end = __ldg(A.out_ptr + u + 1);
        for (int32_t j = j0 + lane; j - lane < j1; j += 32) {
            int32_t s = 0;
            if (j < j1) {
                while (j >= end) end = __ldg(A.out_ptr + ++u + 1);
                const uint32_t ent = __ldg(A.out_ent + j);
                if (ent) {  // else list padding
                    const int32_t x = bm_eid(ent);
                    s = imin(bm_ew(ent), bm_hash_get(hb, __ldg(pi + u), __ldg(pi + x)));
                    if (s) atomicAdd(ov + x, s);
                }
            }
            // entries of one list meet in one addition to S(u)
            mine += (unsigned long long)s;
            int same = 0;
            __match_all_sync(0xffffffffu, j < j1 ? u : -1, &same);
            if (same) {
                const int32_t t = __reduce_add_sync(0xffffffffu, s);
                if (lane == 0 && t) atomicAdd(ov + u, t);
            } else if (s) {
                atomicAdd(ov + u, s);
            }
        }
    }
    for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) block_sum[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < kScoreThreads / 32; i++) t += block_sum[i];
        if (t) atomicAdd(total, t);
    }
}

// One warp per B list g (out-lists, then in-lists): the list's entries
// relabelled into A space (id = pi^-1(B id)) and written in bank-spread order
// of their A ids, the rule of bm_bank_spread_lists (position p takes, where it
// can, an entry of bank ((p >> 2) + 8 (p & 3)) mod 32, else the next bank up
// that still has entries), so the row kernel's scatter over these lists meets
// fewer shared-memory bank conflicts.  pos[j] = the live position of the entry
// at position j of the id-sorted list; padding stays last and in place.  tmp
// (one int32 per entry) holds each bank's entries while they are placed.
//
// The rule is sequential only where some bank has run out: a full turn of 128
// positions takes exactly four entries of every bank, so as many turns as the
// smallest bank has fours are placed in parallel, and the rest step by step
// with the banks' fill levels in the lanes' registers (lane b: bank b) and the
// banks not yet empty as one ballot.  A thread per list took 2.4 ms a launch
// at full scale (a hub's 8,000 entries in one thread); both directions take
// 0.75 ms so.
//
// Without pinv the ids stay as they are and no positions are kept: the order
// of A's device lists.
struct SpreadArgs {
    const int32_t* ptr[2];
    const uint32_t* ent0[2];
    uint32_t* ent[2];
    int32_t* pos[2];
    int32_t* tmp[2];
    const int32_t* pinv;
    int32_t n;
};

template <bool RELABEL>
__device__ __forceinline__ void spread_place(const uint32_t* __restrict__ ent0, const int32_t* __restrict__ pinv,
                                             uint32_t* __restrict__ ent, int32_t* __restrict__ pos, int32_t i, int32_t at) {
    const uint32_t e = __ldg(ent0 + i);
    ent[at] = RELABEL ? bm_pack((uint32_t)__ldg(pinv + bm_eid(e)), (uint32_t)bm_ew(e)) : e;
    if (RELABEL) pos[i] = at;
}

template <bool RELABEL>
__global__ void __launch_bounds__(256) spread_relabel_kernel(SpreadArgs a) {
    const int lane = threadIdx.x & 31;
    const int dir = blockIdx.y;
    const int32_t* __restrict__ ent_ptr = a.ptr[dir];
    const uint32_t* __restrict__ ent0 = a.ent0[dir];
    uint32_t* __restrict__ ent = a.ent[dir];
    int32_t* __restrict__ pos = a.pos[dir];
    int32_t* tmp = a.tmp[dir];
    const int32_t* __restrict__ pinv = a.pinv;
    auto bank_of = [pinv](uint32_t e) { return (RELABEL ? __ldg(pinv + bm_eid(e)) : bm_eid(e)) & 31; };
    for (int32_t g = blockIdx.x * 8 + (threadIdx.x >> 5); g <= a.n; g += gridDim.x * 8) {
        const int32_t lo = __ldg(ent_ptr + g), hi = __ldg(ent_ptr + g + 1);
        if (lo == hi) continue;
        // padding is last, at most 3 entries
        const unsigned pad = __ballot_sync(0xffffffffu, lane < 3 && hi - 1 - lane >= lo && __ldg(ent0 + hi - 1 - lane) == 0u);
        const int32_t cnt = hi - lo - __popc(pad);
        int32_t num = 0;  // of bank `lane`
        for (int32_t i0 = lo; i0 < lo + cnt; i0 += 32) {
            const int32_t i = i0 + lane;
            const int b = i < lo + cnt ? bank_of(__ldg(ent0 + i)) : 32;
            const unsigned same = __match_any_sync(0xffffffffu, b);
            const int leader = __ffs(same) - 1;
            // the leader of every bank present tells its lane the count
            for (unsigned lead = __ballot_sync(0xffffffffu, b < 32 && lane == leader); lead; lead &= lead - 1) {
                const int src = __ffs(lead) - 1;
                const int bank = __shfl_sync(0xffffffffu, b, src), c = __shfl_sync(0xffffffffu, __popc(same), src);
                if (lane == bank) num += c;
            }
        }
        int32_t start = num;  // exclusive sums over the banks
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, start, o);
            if (lane >= o) start += t;
        }
        start += lo - num;
        int32_t head = start;
        for (int32_t i0 = lo; i0 < lo + cnt; i0 += 32) {
            const int32_t i = i0 + lane;
            const int b = i < lo + cnt ? bank_of(__ldg(ent0 + i)) : 32;
            const unsigned same = __match_any_sync(0xffffffffu, b);
            const int32_t at = __shfl_sync(0xffffffffu, head, b & 31) + __popc(same & ((1u << lane) - 1u));
            if (b < 32) tmp[at] = i;
            const int leader = __ffs(same) - 1;
            for (unsigned lead = __ballot_sync(0xffffffffu, b < 32 && lane == leader); lead; lead &= lead - 1) {
                const int src = __ffs(lead) - 1;
                const int bank = __shfl_sync(0xffffffffu, b, src), c = __shfl_sync(0xffffffffu, __popc(same), src);
                if (lane == bank) head += c;
            }
        }
        __syncwarp();
        // whole turns: position p of a turn takes the entry of its bank whose
        // rank is that of p's quad among the bank's four quads of a turn
        const int32_t turns = __reduce_min_sync(0xffffffffu, num) >> 2;
        for (int32_t p = lane; p < 128 * turns; p += 32) {
            const int q = (p & 127) >> 2, c = p & 3, b = (q + 8 * c) & 31;
            int r = 0;
#pragma unroll
            for (int o = 0; o < 4; o++) r += ((b - 8 * o) & 31) < q;
            const int32_t s = __shfl_sync(0xffffffffu, start, b);
            spread_place<RELABEL>(ent0, pinv, ent, pos, tmp[s + 4 * (p >> 7) + r], lo + p);
        }
        // the rest in order
        int32_t left = num - 4 * turns, at = start + 4 * turns;
        unsigned avail = __ballot_sync(0xffffffffu, left > 0);
        for (int32_t p0 = 128 * turns; p0 < cnt; p0 += 32) {
            int32_t mine = 0;
            const int32_t steps = imin(32, cnt - p0);
            for (int32_t k = 0; k < steps; k++) {
                const int32_t p = p0 + k;
                const int b0 = ((p >> 2) + 8 * (p & 3)) & 31;
                const int b = (b0 + __ffs(__funnelshift_r(avail, avail, b0)) - 1) & 31;
                const int32_t taken = __shfl_sync(0xffffffffu, at, b);
                if (lane == k) mine = taken;
                if (lane == b) { at++; left--; }
                avail = __ballot_sync(0xffffffffu, left > 0);
            }
            if (lane < steps) spread_place<RELABEL>(ent0, pinv, ent, pos, tmp[mine], lo + p0 + lane);
        }
        for (int32_t j = lo + cnt + lane; j < hi; j += 32) {
            ent[j] = 0u;
            if (RELABEL) pos[j] = j;
        }
        __syncwarp();
    }
}

// ximg[x] = the bounds of B's in- and out-lists at pi x, for every A vertex.
__global__ void image_bounds_kernel(const int32_t* __restrict__ pi, const int32_t* __restrict__ Bin_ptr,
                                    const int32_t* __restrict__ Bout_ptr, int32_t n, int4* __restrict__ ximg) {
    for (int32_t x = blockIdx.x * blockDim.x + threadIdx.x; x <= n; x += gridDim.x * blockDim.x)
        ximg[x] = x == 0 ? make_int4(0, 0, 0, 0) : bm_image_bounds(Bin_ptr, Bout_ptr, __ldg(pi + x));
}

// The twins of the live lists: the entry at live position pos_self[j] has its
// reverse-direction twin at live position pos_other[twin0[j]] (-1: padding).
__global__ void live_twins_kernel(const int32_t* __restrict__ twin0, const int32_t* __restrict__ pos_self,
                                  const int32_t* __restrict__ pos_other, int32_t* __restrict__ twin, int64_t m) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        const int32_t t0 = __ldg(twin0 + j);
        twin[__ldg(pos_self + j)] = t0 < 0 ? -1 : __ldg(pos_other + t0);
    }
}

}  // namespace

bm_status bm_launch_score(bm_ctx* ctx, int64_t* score_out) {
    const int32_t n = ctx->n;
    BM_CUDA(ctx, cudaMemsetAsync(ctx->ov, 0, sizeof(int32_t) * (size_t)ctx->nvec, ctx->stream));
    BM_CUDA(ctx, cudaMemsetAsync(ctx->d_score, 0, sizeof(unsigned long long), ctx->stream));
    int blocks = ctx->num_sms * 8;
    const int64_t need = std::max<int64_t>((n + kScoreThreads - 1) / kScoreThreads,
                                           (ctx->g[0].m_out + kScoreStretch * 8 - 1) / (kScoreStretch * 8));
    if (blocks > need) blocks = need > 0 ? (int)need : 1;
    score_kernel<<<blocks, kScoreThreads, 0, ctx->stream>>>(gview(ctx->g[0]), hview(ctx->g[1]), ctx->g[1].self_w,
                                                            ctx->pi, n, ctx->ov, ctx->d_score);
    BM_LAUNCH_CHECK(ctx, "score_kernel");
    unsigned long long h = 0;
    BM_CUDA(ctx, cudaMemcpyAsync(&h, ctx->d_score, sizeof h, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *score_out = (int64_t)h;
    return BM_OK;
}

// Exact semantics: the tracked score must equal the recomputed one, and a
// mismatch is a failed self-check.  Reference-delta semantics: the tracked
// score sums calculate_swap_delta values, which are not score differences on
// graphs with self-loops, so the recomputed score replaces it, as the
// reference's loop re-scores after every accept
// (src/graph-alignment-optimized.c:571-576).
bm_status bm_check_score(bm_ctx* ctx) {
    int64_t full = 0;
    bm_status s = bm_launch_score(ctx, &full);
    if (s != BM_OK) return s;
    const int64_t tracked = ctx->score;
    ctx->score = full;
    if (full != tracked && ctx->semantics == BM_SEMANTICS_EXACT)
        return bm_fail(ctx, BM_PARITY_FAIL, "tracked score %lld != recomputed score %lld", (long long)tracked,
                       (long long)full);
    return BM_OK;
}

bm_status bm_launch_spread(bm_ctx* ctx, int32_t n, const int32_t* optr, const int32_t* iptr, const uint32_t* oent,
                           const uint32_t* ient, uint32_t* out, uint32_t* in, int32_t* tmp) {
    const unsigned blocks = (unsigned)std::min((n + 8) / 8, ctx->num_sms * 8);
    // one direction after the other: they share tmp
    const SpreadArgs so{{optr, optr}, {oent, oent}, {out, out}, {nullptr, nullptr}, {tmp, tmp}, nullptr, n};
    spread_relabel_kernel<false><<<blocks, 256, 0, ctx->stream>>>(so);
    BM_LAUNCH_CHECK(ctx, "spread_kernel(out)");
    const SpreadArgs si{{iptr, iptr}, {ient, ient}, {in, in}, {nullptr, nullptr}, {tmp, tmp}, nullptr, n};
    spread_relabel_kernel<false><<<blocks, 256, 0, ctx->stream>>>(si);
    BM_LAUNCH_CHECK(ctx, "spread_kernel(in)");
    return BM_OK;
}

bm_status bm_launch_relabel(bm_ctx* ctx) {
    const DevGraph& B = ctx->g[1];
    image_bounds_kernel<<<(ctx->n + 1 + 255) / 256, 256, 0, ctx->stream>>>(ctx->pi, B.in_ptr, B.out_ptr, ctx->n, ctx->ximg);
    BM_LAUNCH_CHECK(ctx, "image_bounds_kernel");
    if (B.m_out + B.m_in == 0) return BM_OK;
    // the live twin arrays serve as the placement scratch, then are rebuilt
    const SpreadArgs sa{{B.out_ptr, B.in_ptr},   {B.out_ent0, B.in_ent0}, {B.out_ent, B.in_ent},
                        {B.out_pos, B.in_pos},   {B.out_twin, B.in_twin}, ctx->pinv, ctx->n};
    spread_relabel_kernel<true>
        <<<dim3((unsigned)std::min((ctx->n + 8) / 8, ctx->num_sms * 8), 2), 256, 0, ctx->stream>>>(sa);
    BM_LAUNCH_CHECK(ctx, "spread_relabel_kernel");
    const int tb = ctx->num_sms * 4;
    if (B.m_out > 0) {
        live_twins_kernel<<<tb, 256, 0, ctx->stream>>>(B.out_twin0, B.out_pos, B.in_pos, B.out_twin, B.m_out);
        BM_LAUNCH_CHECK(ctx, "live_twins_kernel(out)");
    }
    if (B.m_in > 0) {
        live_twins_kernel<<<tb, 256, 0, ctx->stream>>>(B.in_twin0, B.in_pos, B.out_pos, B.in_twin, B.m_in);
        BM_LAUNCH_CHECK(ctx, "live_twins_kernel(in)");
    }
    return BM_OK;
}
