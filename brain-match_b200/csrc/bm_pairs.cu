// bm_pairs.cu — exact swap deltas for an arbitrary list of pairs.
//
// Follows calculate_swap_delta (src/graph-alignment-optimized.c:321-408) in
// score-difference form.  With f_u = pi u, f_v = pi v, S the per-vertex overlap
// and B self-loops kept out of the hash (so w_B(f, f) = 0 there):
//
//   delta(u,v) =   sum_{x in out(u)} min(w, B(f_v, pi x)) + sum_{x in in(u)} min(w, B(pi x, f_v))
//                + sum_{y in out(v)} min(w, B(f_u, pi y)) + sum_{y in in(v)} min(w, B(pi y, f_u))
//                - S(u) - S(v)
//                + sum over A entries between u and v of [min(w, B(f_u,f_v)) + min(w, B(f_v,f_u))]
//                + self-loop terms.
//
// Self-loop terms, with s_x the A self-loop weight of x, b_x = B(f_x, f_x),
// p = B(f_u, f_v), q = B(f_v, f_u): exact semantics
//   min(s_u, b_v) - min(s_u, b_u) + min(s_v, b_u) - min(s_v, b_v);
// reference-delta semantics (what calculate_swap_delta returns: its out- and
// in-edge loops, :327-388, each meet the self-loop of a swapped vertex and
// compare the image after the swap, p or q, with the old image's b_x)
//   min(s_u, p) + min(s_u, q) + min(s_v, p) + min(s_v, q) - 2 min(s_u, b_u) - 2 min(s_v, b_v).
//
// The last sum repairs the direct edges u->v and v->u that S(u) and S(v) both
// counted (the reference handles them at :390-405).
//
// Two kernels.  pairs_kernel: one warp per pair (a block for a hub's), every
// lookup of B one probe sequence in the hash table (L2-resident).  It costs
// one random 32-byte sector per A entry, about 650 a pair on the full-scale
// pair, and that bounds it: 10.2 ms for 2^20 random pairs.  pairs_group_kernel: the pairs sorted by
// u, the four lists of u (A out, A in, relabelled B out, relabelled B in) as
// dense 16-bit weight tables in shared memory, and the four lists of every v
// streamed past them, so that each term is a coalesced entry and one
// shared-memory read:
//   sum_{x in out(u)} min(w, B(f_v, pi x)) = sum over B'-out(v) of min(b, A-out(u)[x]),
// B' being B with its ids relabelled into A space, and so on: 1.4 ms for the
// same pairs, sorting included.
#include <algorithm>

#include "bm_internal.cuh"

namespace {

constexpr int kPairThreads = 256;

struct PairArgs {
    GView A;
    const int32_t* selfB;
    HashView hb;
    const int32_t* pi;
    const int32_t* ov;
    int32_t n;
    int has_self;  // self-loop terms needed (A and B have self-loops; A alone in reference-delta mode)
    int refcpu;    // reference-delta semantics
};

// One pair's four lists as a single stream of entries: out(u), in(u), out(v),
// in(v); `end` are the running ends, `beg` the lists' starts less the entries
// before them.
struct PairLists {
    int4 beg, end;
};

__device__ __forceinline__ PairLists pair_lists(const PairArgs& a, int32_t u, int32_t v) {
    const int32_t o0 = __ldg(a.A.out_ptr + u), o1 = __ldg(a.A.out_ptr + u + 1);
    const int32_t i0 = __ldg(a.A.in_ptr + u), i1 = __ldg(a.A.in_ptr + u + 1);
    const int32_t p0 = __ldg(a.A.out_ptr + v), p1 = __ldg(a.A.out_ptr + v + 1);
    const int32_t j0 = __ldg(a.A.in_ptr + v), j1 = __ldg(a.A.in_ptr + v + 1);
    PairLists L;
    L.end.x = o1 - o0;
    L.end.y = L.end.x + (i1 - i0);
    L.end.z = L.end.y + (p1 - p0);
    L.end.w = L.end.z + (j1 - j0);
    L.beg = make_int4(o0, i0 - L.end.x, p0 - L.end.y, j0 - L.end.z);
    return L;
}

// One thread's share (entries t, t + STRIDE, ...) of the pair's overlaps
// after the swap and of the direct-edge repair.
template <int STRIDE>
__device__ __forceinline__ int32_t pair_share(const PairArgs& a, const PairLists& L, int32_t v, int32_t fu, int32_t fv,
                                              int t) {
    // at most the weighted degrees of u and v for the terms and twice u's for the
    // repair of its direct edges, each below 2^29: the pair's sum stays below 2^31
    int32_t s = 0;
#pragma unroll 2
    for (int32_t j = t; j < L.end.w; j += STRIDE) {
        const bool out = j < L.end.x || (j >= L.end.y && j < L.end.z);
        const bool of_u = j < L.end.y;
        const int32_t at = j + (of_u ? (out ? L.beg.x : L.beg.y) : (out ? L.beg.z : L.beg.w));
        const uint32_t ent = __ldg((out ? a.A.out_ent : a.A.in_ent) + at);
        if (ent == 0) continue;  // list padding
        const int32_t x = bm_eid(ent), w = bm_ew(ent);
        const int32_t gx = __ldg(a.pi + x), gm = of_u ? fv : fu;
        s += imin(w, out ? bm_hash_get(a.hb, gm, gx) : bm_hash_get(a.hb, gx, gm));
        if (of_u && x == v) s += imin(w, bm_hash_get(a.hb, fu, fv)) + imin(w, bm_hash_get(a.hb, fv, fu));
    }
    return s;
}

__device__ __forceinline__ int64_t pair_finish(const PairArgs& a, int64_t s, int32_t u, int32_t v, int32_t fu, int32_t fv) {
    s -= (int64_t)__ldg(a.ov + u) + (int64_t)__ldg(a.ov + v);
    if (a.has_self) {
        const int32_t su = __ldg(a.A.self_w + u), sv = __ldg(a.A.self_w + v);
        const int32_t bu = __ldg(a.selfB + fu), bv = __ldg(a.selfB + fv);
        if (a.refcpu) {
            const int32_t p = bm_hash_get(a.hb, fu, fv), q = bm_hash_get(a.hb, fv, fu);
            s += imin(su, p) + imin(su, q) + imin(sv, p) + imin(sv, q) - 2 * imin(su, bu) - 2 * imin(sv, bv);
        } else {
            s += imin(su, bv) - imin(su, bu) + imin(sv, bu) - imin(sv, bv);
        }
    }
    return s;
}

// A block takes `per` (1..8) pairs at a time, one to a warp; a pair of more
// than `heavy` entries waits and is then shared by the whole block, since one
// warp would walk a hub's lists for half a millisecond (1,852 random pairs of
// the full-scale pair: 600 us a warp each, 80 us so).
__global__ void __launch_bounds__(kPairThreads)
pairs_kernel(PairArgs a, const int32_t* __restrict__ pairs, int64_t k, int32_t per, int32_t heavy,
             int64_t* __restrict__ out) {
    constexpr int W = kPairThreads / 32;
    __shared__ int32_t s_heavy[W], s_sum[W], s_n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t i0 = (int64_t)blockIdx.x * per; i0 < k; i0 += (int64_t)gridDim.x * per) {
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        const int64_t i = i0 + warp;
        if (warp < per && i < k) {
            const int32_t u = __ldg(pairs + 2 * i), v = __ldg(pairs + 2 * i + 1);
            // ids outside 1..n (device-pointer callers) and u == v give 0
            if (u != v && u >= 1 && u <= a.n && v >= 1 && v <= a.n) {
                const PairLists L = pair_lists(a, u, v);
                if (L.end.w > heavy) {
                    if (lane == 0) s_heavy[atomicAdd(&s_n, 1)] = warp;
                } else {
                    const int32_t fu = __ldg(a.pi + u), fv = __ldg(a.pi + v);
                    const int32_t s = __reduce_add_sync(0xffffffffu, pair_share<32>(a, L, v, fu, fv, lane));
                    if (lane == 0) out[i] = pair_finish(a, s, u, v, fu, fv);
                }
            } else if (lane == 0) {
                out[i] = 0;
            }
        }
        __syncthreads();
        const int32_t nh = s_n;
        for (int32_t h = 0; h < nh; h++) {
            const int64_t ih = i0 + s_heavy[h];
            const int32_t u = __ldg(pairs + 2 * ih), v = __ldg(pairs + 2 * ih + 1);
            const int32_t fu = __ldg(a.pi + u), fv = __ldg(a.pi + v);
            const PairLists L = pair_lists(a, u, v);
            const int32_t s = __reduce_add_sync(0xffffffffu, pair_share<kPairThreads>(a, L, v, fu, fv, threadIdx.x));
            if (lane == 0) s_sum[warp] = s;
            __syncthreads();
            if (threadIdx.x == 0) {
                int64_t t = 0;
                for (int w = 0; w < W; w++) t += s_sum[w];
                out[ih] = pair_finish(a, t, u, v, fu, fv);
            }
            __syncthreads();
        }
    }
}

// ------------------------------------------------- pairs grouped by u

constexpr int kGrpPairs = 256;     // pairs of one u that a CTA takes together
constexpr int kGrpUnit = 512;      // quads (4 entries) of a pair's lists that a warp takes together: a typical
                                   // pair (about 160 quads) is one unit, a hub's lists are shared by the warps
constexpr int64_t kGrpChunk = 4 << 20;  // pairs sorted at once (bounds the scratch: 8 bytes a pair)

struct GroupArgs {
    PairArgs p;
    const uint4* Aout;  // A's lists and B's relabelled lists as quads
    const uint4* Ain;
    const uint4* Bout;
    const uint4* Bin;
    const int4* ximg;
    int32_t nv;              // table length
    const int32_t* off;      // sorted position of u's first pair (n + 2)
    const int32_t* item0;    // u's first item (n + 1)
    const int32_t* item_u;   // u of an item
    const int32_t* nitems;
    int32_t* next;           // claims of items past the blocks' first ones
    const int2* sorted;      // {v, index} by u
    int64_t* out;
};

// Pairs per u (count, not yet summed); out-of-range ids and u == v give 0.
// Equal u of a warp are counted with one atomic (lists of candidates per row
// come in runs of equal u).
__global__ void group_count_kernel(const int2* __restrict__ pairs, int64_t k, int32_t n, int32_t* __restrict__ cnt,
                                   int64_t* __restrict__ out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 - threadIdx.x % 32 < k; i0 += stride) {
        int32_t u = 0;
        if (i0 < k) {
            const int2 p = __ldg(pairs + i0);
            if (p.x != p.y && p.x >= 1 && p.x <= n && p.y >= 1 && p.y <= n) u = p.x;
            else out[i0] = 0;
        }
        const unsigned same = __match_any_sync(0xffffffffu, u);
        if (u && (int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(cnt + u, __popc(same));
    }
}

// Exclusive sums of the counts (off, and cursor = off) and of the items of
// kGrpPairs pairs (item0), and the u of every item.  One CTA.
__global__ void __launch_bounds__(1024) group_scan_kernel(const int32_t* __restrict__ cnt, int32_t n,
                                                          int32_t* __restrict__ off, int32_t* __restrict__ cursor,
                                                          int32_t* __restrict__ item0, int32_t* __restrict__ item_u,
                                                          int32_t* __restrict__ nitems) {
    __shared__ int32_t wsum[2][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int32_t base_c = 0, base_i = 0;
    for (int32_t v0 = 0; v0 <= n; v0 += 1024) {
        const int32_t v = v0 + tid;
        const int32_t c = (v >= 1 && v <= n) ? cnt[v] : 0, it = (c + kGrpPairs - 1) / kGrpPairs;
        int32_t sc = c, si = it;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t a = __shfl_up_sync(0xffffffffu, sc, o), b = __shfl_up_sync(0xffffffffu, si, o);
            if (lane >= o) { sc += a; si += b; }
        }
        if (lane == 31) { wsum[0][warp] = sc; wsum[1][warp] = si; }
        __syncthreads();
        int32_t pc = 0, pi = 0, tc = 0, ti = 0;
        for (int w = 0; w < 32; w++) {
            if (w < warp) { pc += wsum[0][w]; pi += wsum[1][w]; }
            tc += wsum[0][w];
            ti += wsum[1][w];
        }
        const int32_t ec = base_c + pc + sc - c, ei = base_i + pi + si - it;
        if (v <= n) {
            off[v] = ec;
            cursor[v] = ec;
            item0[v] = ei;
            for (int32_t j = 0; j < it; j++) item_u[ei + j] = v;
        }
        base_c += tc;
        base_i += ti;
        __syncthreads();
    }
    if (tid == 0) { off[n + 1] = base_c; *nitems = base_i; }
}

__global__ void group_place_kernel(const int2* __restrict__ pairs, int64_t k, int32_t n, int32_t* __restrict__ cursor,
                                   int2* __restrict__ sorted) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 - lane < k; i0 += stride) {
        int32_t u = 0, v = 0;
        if (i0 < k) {
            const int2 p = __ldg(pairs + i0);
            if (p.x != p.y && p.x >= 1 && p.x <= n && p.y >= 1 && p.y <= n) { u = p.x; v = p.y; }
        }
        const unsigned same = __match_any_sync(0xffffffffu, u);
        const int leader = __ffs(same) - 1;
        int32_t at = 0;
        if (u && lane == leader) at = atomicAdd(cursor + u, __popc(same));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (u) sorted[at + __popc(same & ((1u << lane) - 1u))] = make_int2(v, (int32_t)i0);
    }
}

// Writes (or clears) u's entries of one list in its table.
template <int kGrpThreads>
__device__ __forceinline__ void table_list(uint16_t* tab, const uint4* ent, int32_t b, int32_t e, bool set) {
    for (int32_t q = (b >> 2) + (int32_t)threadIdx.x; q < (e >> 2); q += kGrpThreads) {
        const uint4 x = __ldg(ent + q);
        const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int c = 0; c < 4; c++) tab[bm_eid(v[c])] = set ? (uint16_t)bm_ew(v[c]) : (uint16_t)0;  // padding: entry 0
    }
}

// What bounds it: reading every v's lists from L2 (2.7 GB for 2^20 random
// pairs of the full-scale pair) and the shared-memory reads of random 16-bit
// table entries; the tables of u are written and cleared once per item.
template <int kGrpThreads>
__global__ void __launch_bounds__(kGrpThreads, kGrpThreads == 1024 ? 1 : 2) pairs_group_kernel(GroupArgs a) {
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ int4 s_beg[kGrpPairs], s_end[kGrpPairs];  // per pair: list starts less the quads before, running ends
    __shared__ int32_t s_unit[kGrpPairs + 1];            // exclusive sums of the pairs' units
    __shared__ int32_t s_acc[kGrpPairs];
    __shared__ int32_t s_w[kGrpPairs / 32];
    __shared__ int32_t s_item, s_claim;
    uint16_t* T = reinterpret_cast<uint16_t*>(gsm);
    uint16_t *T0 = T, *T1 = T + a.nv, *T2 = T + 2 * a.nv, *T3 = T + 3 * a.nv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const GView& A = a.p.A;
    for (int32_t i = tid; i < a.nv / 2; i += kGrpThreads) reinterpret_cast<uint4*>(gsm)[i] = make_uint4(0, 0, 0, 0);
    const int32_t nitems = __ldg(a.nitems);
    __syncthreads();
    // a block's first item is its own number, the later ones are claimed: s_item is
    // written only at the head of an item and read between its barriers
    int32_t item = (int32_t)blockIdx.x;
    while (item < nitems) {
        const int32_t u = __ldg(a.item_u + item);
        const int32_t p0 = __ldg(a.off + u) + (item - __ldg(a.item0 + u)) * kGrpPairs;
        const int32_t np = imin(kGrpPairs, __ldg(a.off + u + 1) - p0);
        const int4 xu = __ldg(a.ximg + u);
        const int32_t uo0 = __ldg(A.out_ptr + u), uo1 = __ldg(A.out_ptr + u + 1);
        const int32_t ui0 = __ldg(A.in_ptr + u), ui1 = __ldg(A.in_ptr + u + 1);
        if (tid == 0) { s_item = (int32_t)gridDim.x + atomicAdd(a.next, 1); s_claim = 0; }
        table_list<kGrpThreads>(T0, a.Aout, uo0, uo1, true);
        table_list<kGrpThreads>(T1, a.Ain, ui0, ui1, true);
        table_list<kGrpThreads>(T2, a.Bout, xu.z, xu.w, true);
        table_list<kGrpThreads>(T3, a.Bin, xu.x, xu.y, true);
        // the pairs' lists as one stream of quads each, cut into units
        int32_t v = 0, idx = 0, units = 0;
        if (tid < kGrpPairs) {
            if (tid < np) {
                const int2 p = __ldg(a.sorted + p0 + tid);
                v = p.x;
                idx = p.y;
                const int4 xv = __ldg(a.ximg + v);
                const int32_t o0 = __ldg(A.out_ptr + v) >> 2, o1 = __ldg(A.out_ptr + v + 1) >> 2;
                const int32_t i0 = __ldg(A.in_ptr + v) >> 2, i1 = __ldg(A.in_ptr + v + 1) >> 2;
                int4 e, b;
                e.x = (xv.w - xv.z) >> 2;
                e.y = e.x + ((xv.y - xv.x) >> 2);
                e.z = e.y + (o1 - o0);
                e.w = e.z + (i1 - i0);
                b.x = xv.z >> 2;
                b.y = (xv.x >> 2) - e.x;
                b.z = o0 - e.y;
                b.w = i0 - e.z;
                s_beg[tid] = b;
                s_end[tid] = e;
                units = (e.w + kGrpUnit - 1) / kGrpUnit;
            }
            s_acc[tid] = 0;
            int32_t s = units;
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t t = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += t;
            }
            if (lane == 31) s_w[warp] = s;
            s_unit[tid] = s - units;  // within the warp, completed below
        }
        __syncthreads();
        if (tid < kGrpPairs) {
            int32_t before = 0;
            for (int w = 0; w < warp; w++) before += s_w[w];
            const int32_t mine = s_unit[tid] + before;
            s_unit[tid] = mine;
            if (tid == kGrpPairs - 1) s_unit[kGrpPairs] = mine + units;
        }
        const int32_t next_item = s_item;
        __syncthreads();
        const int32_t total = s_unit[kGrpPairs];
        for (;;) {
            int32_t un = 0;
            if (lane == 0) un = atomicAdd(&s_claim, 1);
            un = __shfl_sync(0xffffffffu, un, 0);
            if (un >= total) break;
            int32_t lo = 0, hi = np - 1;  // the last pair whose first unit is at most un
            while (lo < hi) {
                const int32_t mid = (lo + hi + 1) >> 1;
                if (s_unit[mid] <= un) lo = mid; else hi = mid - 1;
            }
            const int4 b = s_beg[lo], e = s_end[lo];
            const int32_t q0 = (un - s_unit[lo]) * kGrpUnit, q1 = imin(e.w, q0 + kGrpUnit);
            int32_t sum = 0;
            for (int32_t q = q0 + lane; q < q1; q += 128) {
                uint4 x[4];
                int32_t tb[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int32_t r = q + 32 * j;
                    const uint4* src = r < e.x ? a.Bout + b.x : r < e.y ? a.Bin + b.y : r < e.z ? a.Aout + b.z : a.Ain + b.w;
                    tb[j] = r < e.x ? 0 : r < e.y ? a.nv : r < e.z ? 2 * a.nv : 3 * a.nv;
                    x[j] = r < q1 ? __ldg(src + r) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const uint32_t w[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
#pragma unroll
                    for (int c = 0; c < 4; c++) sum += imin((int32_t)T[tb[j] + bm_eid(w[c])], bm_ew(w[c]));
                }
            }
            sum = __reduce_add_sync(0xffffffffu, sum);
            if (lane == 0 && sum) atomicAdd(&s_acc[lo], sum);
        }
        __syncthreads();
        if (tid < np) {
            const int32_t wuv = T0[v], wvu = T1[v], p = T2[v], q = T3[v];
            int64_t s = (int64_t)s_acc[tid] + imin(wuv, p) + imin(wuv, q) + imin(wvu, p) + imin(wvu, q);
            s -= (int64_t)__ldg(a.p.ov + u) + (int64_t)__ldg(a.p.ov + v);
            if (a.p.has_self) {
                const int32_t su = __ldg(A.self_w + u), sv = __ldg(A.self_w + v);
                const int32_t bu = __ldg(a.p.selfB + __ldg(a.p.pi + u)), bv = __ldg(a.p.selfB + __ldg(a.p.pi + v));
                if (a.p.refcpu)
                    s += imin(su, p) + imin(su, q) + imin(sv, p) + imin(sv, q) - 2 * imin(su, bu) - 2 * imin(sv, bv);
                else
                    s += imin(su, bv) - imin(su, bu) + imin(sv, bu) - imin(sv, bv);
            }
            a.out[idx] = s;
        }
        __syncthreads();
        table_list<kGrpThreads>(T0, a.Aout, uo0, uo1, false);
        table_list<kGrpThreads>(T1, a.Ain, ui0, ui1, false);
        table_list<kGrpThreads>(T2, a.Bout, xu.z, xu.w, false);
        table_list<kGrpThreads>(T3, a.Bin, xu.x, xu.y, false);
        item = next_item;
        __syncthreads();
    }
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t group_smem(int32_t n) { return 4 * sizeof(uint16_t) * (size_t)(((n + 1) + 7) & ~7); }

// Sizes of the scratch of one chunk of k pairs.
struct GroupScratch {
    size_t cnt, off, cursor, item0, item_u, sorted, total;
    GroupScratch(int32_t n, int64_t k) {
        const size_t v = al256(sizeof(int32_t) * ((size_t)n + 2));
        cnt = 256;  // the claim counter and the item count come first
        off = cnt + v;
        cursor = off + v;
        item0 = cursor + v;
        item_u = item0 + v;
        sorted = item_u + al256(sizeof(int32_t) * ((size_t)n + (size_t)(k / kGrpPairs) + 2));
        total = sorted + al256(sizeof(int2) * (size_t)k);
    }
};

// Whether k pairs, each u of which comes in runs of at least `run`, go to the
// grouped kernel.  An item costs about 29 ns of the chip (its tables, barriers
// and latency; full-scale pair), an entry of a pair about 0.02 ns of the hash
// lookups' bandwidth: the grouped kernel pays when its items, at most one per
// u, cost less than the pairs' entries.  Lists with repeated neighbours have no
// dense table; the tables must fit in shared memory.
bool groups_pay(const bm_ctx* ctx, int64_t k, int64_t run) {
    const int32_t mode = ctx->path[BM_PATH_PAIR_GROUPS];
    if (mode < 0 || ctx->g[0].has_dup) return false;
    if (group_smem(ctx->n) + 16384 > ctx->smem_optin) return false;
    const double items = (double)std::min<int64_t>(ctx->n, (k + run - 1) / run);
    const double entries = 2.0 * (double)(ctx->g[0].m_out + ctx->g[0].m_in) / ctx->n;  // of an average pair
    return mode > 0 || ((double)k * entries * 0.02 >= 29.0 * items && k >= 1024);
}

size_t group_scratch(const bm_ctx* ctx, int64_t k) { return GroupScratch(ctx->n, std::min(k, kGrpChunk)).total; }

// The context's own scratch for k pairs; null without room for it.
void* context_scratch(bm_ctx* ctx, int64_t k) {
    // a capture's later replays would share it with whatever call comes then
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return nullptr;
    const size_t need = group_scratch(ctx, k);
    if (ctx->pscr_bytes >= need) return ctx->pscr;
    // The call does not wait for the device: an outgrown block, which launches
    // in flight may use, is put by until the stream is next idle (bm_set_graph).
    // Blocks double up to the largest, so those put by hold about as much
    // together as the one in use at most.
    const size_t size = std::max(need, std::min(group_scratch(ctx, kGrpChunk), 2 * ctx->pscr_bytes));
    void* block = nullptr;
    if (bm_cuda_malloc(&block, size) != cudaSuccess) {
        cudaGetLastError();  // no room for the sort: one warp per pair needs none
        return nullptr;
    }
    if (ctx->pscr) ctx->pscr_old.push_back(ctx->pscr);
    ctx->pscr = block;
    ctx->pscr_bytes = size;
    return block;
}

bm_status launch_groups(bm_ctx* ctx, const PairArgs& pa, const int32_t* d_pairs, int64_t k, int64_t* d_out, char* base) {
    const int32_t n = ctx->n;
    const DevGraph &A = ctx->g[0], &B = ctx->g[1];
    const GroupScratch L(n, std::min(k, kGrpChunk));
    // 1,024 threads when the tables leave room for one CTA on an SM, else as
    // many CTAs of 512 as fit: an item is a chain of short phases, which the
    // other CTAs fill
    const size_t smem = group_smem(n);
    const bool wide = 2 * (smem + 16384) > ctx->smem_optin;
    int resident = 1;
    if (wide) {
        BM_CUDA(ctx, cudaFuncSetAttribute(pairs_group_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    } else {
        BM_CUDA(ctx, cudaFuncSetAttribute(pairs_group_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        BM_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, pairs_group_kernel<512>, 512, smem));
    }
    for (int64_t i0 = 0; i0 < k; i0 += kGrpChunk) {
        const int64_t kc = std::min(k - i0, kGrpChunk);
        const int2* pairs = reinterpret_cast<const int2*>(d_pairs) + i0;
        GroupArgs a;
        a.p = pa;
        a.Aout = reinterpret_cast<const uint4*>(A.out_ent);
        a.Ain = reinterpret_cast<const uint4*>(A.in_ent);
        a.Bout = reinterpret_cast<const uint4*>(B.out_ent);
        a.Bin = reinterpret_cast<const uint4*>(B.in_ent);
        a.ximg = ctx->ximg;
        a.nv = ((n + 1) + 7) & ~7;
        a.next = (int32_t*)base;
        int32_t* nitems = (int32_t*)(base + 128);
        a.nitems = nitems;
        int32_t* cnt = (int32_t*)(base + L.cnt);
        int32_t* off = (int32_t*)(base + L.off);
        int32_t* cursor = (int32_t*)(base + L.cursor);
        int32_t* item0 = (int32_t*)(base + L.item0);
        int32_t* item_u = (int32_t*)(base + L.item_u);
        int2* sorted = (int2*)(base + L.sorted);
        a.off = off;
        a.item0 = item0;
        a.item_u = item_u;
        a.sorted = sorted;
        a.out = d_out + i0;
        BM_CUDA(ctx, cudaMemsetAsync(base, 0, L.off, ctx->stream));
        const unsigned blocks = (unsigned)std::min<int64_t>((kc + 255) / 256, (int64_t)ctx->num_sms * 8);
        group_count_kernel<<<blocks, 256, 0, ctx->stream>>>(pairs, kc, n, cnt, a.out);
        BM_LAUNCH_CHECK(ctx, "group_count_kernel");
        group_scan_kernel<<<1, 1024, 0, ctx->stream>>>(cnt, n, off, cursor, item0, item_u, nitems);
        BM_LAUNCH_CHECK(ctx, "group_scan_kernel");
        group_place_kernel<<<blocks, 256, 0, ctx->stream>>>(pairs, kc, n, cursor, sorted);
        BM_LAUNCH_CHECK(ctx, "group_place_kernel");
        if (wide) pairs_group_kernel<1024><<<ctx->num_sms, 1024, smem, ctx->stream>>>(a);
        else pairs_group_kernel<512><<<ctx->num_sms * std::max(1, resident), 512, smem, ctx->stream>>>(a);
        BM_LAUNCH_CHECK(ctx, "pairs_group_kernel");
    }
    return BM_OK;
}

}  // namespace

static bm_status launch_pairs(bm_ctx* ctx, const int32_t* d_pairs, int64_t k, int64_t* d_out, bool exact_only,
                              void* scratch) {
    PairArgs a;
    a.A = gview(ctx->g[0]);
    a.selfB = ctx->g[1].self_w;
    a.hb = hview(ctx->g[1]);
    a.pi = ctx->pi;
    a.ov = ctx->ov;
    a.n = ctx->n;
    a.refcpu = !exact_only && ctx->semantics == BM_SEMANTICS_REF_CPU;
    a.has_self = a.refcpu ? ctx->g[0].has_self : (ctx->g[0].has_self && ctx->g[1].has_self);
    if (scratch) return launch_groups(ctx, a, d_pairs, k, d_out, (char*)scratch);
    // one pair to a block while the pairs are fewer than the resident blocks
    const int64_t slots = (int64_t)ctx->num_sms * 8;
    const int32_t per = (int32_t)std::max<int64_t>(1, std::min<int64_t>(kPairThreads / 32, k / slots));
    const int64_t blocks = std::min<int64_t>((k + per - 1) / per, slots * 2);
    pairs_kernel<<<(unsigned)blocks, kPairThreads, 0, ctx->stream>>>(a, d_pairs, k, per, per == 1 ? 64 : 1024, d_out);
    BM_LAUNCH_CHECK(ctx, "pairs_kernel");
    return BM_OK;
}

bm_status bm_launch_pairs(bm_ctx* ctx, const int32_t* d_pairs, int64_t k, int64_t* d_out, bool exact_only, int64_t run) {
    if (k <= 0) return BM_OK;
    const bool grouped = ((uintptr_t)d_pairs & 7) == 0 && groups_pay(ctx, k, std::max<int64_t>(1, run));
    return launch_pairs(ctx, d_pairs, k, d_out, exact_only, grouped ? context_scratch(ctx, k) : nullptr);
}

extern "C" bm_status bm_delta_pairs_dev(bm_ctx* ctx, const int32_t* d_pairs, int64_t k, int64_t* d_deltas) {
    bm_status s = bm_require_mapped(ctx);
    if (s != BM_OK) return s;
    if (k < 0 || (k > 0 && (!d_pairs || !d_deltas))) return bm_fail(ctx, BM_INVALID_ARG, "bad pair buffers");
    return bm_launch_pairs(ctx, d_pairs, k, d_deltas);
}

extern "C" bm_status bm_delta_pairs(bm_ctx* ctx, const int32_t* pairs, int64_t k, int64_t* deltas) {
    bm_status s = bm_require_mapped(ctx);
    if (s != BM_OK) return s;
    if (k < 0 || (k > 0 && (!pairs || !deltas))) return bm_fail(ctx, BM_INVALID_ARG, "bad pair buffers");
    if (k == 0) return BM_OK;
    // an id x in 1..n leaves the top bits of x - 1 and of n - x clear; sums of
    // words, without comparisons or an early exit, are what the compiler turns into
    // vectors (with a loop of comparisons a call of 2^20 pairs took 3.7 or 4.15 ms,
    // by where the loop lay in the library; 3.4 ms so)
    const uint32_t un = (uint32_t)ctx->n;
    uint32_t out_of_range = 0;
    for (int64_t i = 0; i < 2 * k; i++) {
        const uint32_t x = (uint32_t)pairs[i];
        out_of_range |= (x - 1u) | (un - x);
    }
    const bool bad = out_of_range >> 31;
    for (int64_t i = 0; bad && i < 2 * k; i++)
        if (pairs[i] < 1 || pairs[i] > ctx->n)
            return bm_fail(ctx, BM_INVALID_ARG, "pair entry %lld = %d outside 1..%d", (long long)i, pairs[i], ctx->n);
    const size_t in_bytes = sizeof(int32_t) * 2 * (size_t)k;
    const size_t in_al = (in_bytes + 255) & ~(size_t)255;
    // the sort's scratch is part of the call's staging: a context's first list
    // grows its memory once
    const size_t io = in_al + al256(sizeof(int64_t) * (size_t)k);
    bool grouped = groups_pay(ctx, k, 1);
    s = bm_stage(ctx, io + (grouped ? group_scratch(ctx, k) : 0));
    if (s == BM_OOM && grouped) {
        cudaGetLastError();
        grouped = false;
        s = bm_stage(ctx, io);
    }
    if (s != BM_OK) return s;
    int32_t* d_pairs = (int32_t*)ctx->stage;
    int64_t* d_out = (int64_t*)((char*)ctx->stage + in_al);
    BM_CUDA(ctx, cudaMemcpyAsync(d_pairs, pairs, in_bytes, cudaMemcpyHostToDevice, ctx->stream));
    s = launch_pairs(ctx, d_pairs, k, d_out, false, grouped ? (char*)ctx->stage + io : nullptr);
    if (s != BM_OK) return s;
    BM_CUDA(ctx, cudaMemcpyAsync(deltas, d_out, sizeof(int64_t) * (size_t)k, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BM_OK;
}
