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
// n-bit shared-memory bitmap and counts them with popc.  Neighbours with more
// than n / 64 neighbours of their own (at least 64) have their list as a row of
// n bits in memory, and the CTA ORs those rows, 16 bytes a thread, in
// registers: a word of 32 bits takes about 0.6 of the time of one scattered
// bit, and a list of n / 53 neighbours breaks even.  Bits alone took 4.5 ms a
// graph at 18,524 vertices and 3,000,000 edges (2 x 2.4e9 targets), with the
// rows 1.5 ms (lines at n / 32 and n / 128 were not better).
//
// The greedy step goes in rounds of kRound A vertices.  shortlist_kernel, a
// warp a vertex over the whole device, lists the kList nearest of the B
// vertices that are left; then one warp of commit_kernel goes through the
// round's vertices and gives each the first on its list that is still free (the
// nearest: all that are not listed are further).  A vertex whose list is
// used up is searched for then.  Searches start where B's feature sum
// equals the vertex's and go outwards both ways: the L1 distance is at least
// the difference of the sums, so a side ends where that difference exceeds the
// distance to beat.  The unmatched vertices are kept dense, compacted after
// each round.  At 18,524 vertices a block-wide argmin over all of B per A vertex
// took 131 ms, searches by the committing CTA alone 22 ms, this takes 5.8 ms.
#include <algorithm>
#include <climits>

#include "bm_internal.cuh"

namespace {

constexpr int kReachThreads = 256;
constexpr int kGreedyThreads = 1024;
constexpr int kListThreads = 128;
constexpr int kRound = 256;   // A vertices between compactions of what is left of B
constexpr int kList = 64;     // shortlist entries: two a lane; one vertex in 80 uses all of them up (rounds of 1,024: one in 25)

constexpr int kReachRows = 512;  // bit rows of a stretch

struct Adj {
    const int32_t* ptr;   // n+2
    const int32_t* idx;   // neighbour ids: [ptr, hend) those with a bit row, [hend, next ptr) the others
    const int32_t* hend;  // n+1
    const int32_t* row;   // a vertex's bit row, -1: none
    const uint4* rows;    // n + 1 bits in 16-byte words each
};

__global__ void __launch_bounds__(kReachThreads) reach2_kernel(Adj out, Adj in, int32_t n, int copies, int* next,
                                                               int4* __restrict__ feat) {
    extern __shared__ __align__(16) uint32_t bits[];
    __shared__ int s_v;
    __shared__ int s_cnt;
    __shared__ int32_t s_row[kReachRows];
    const int32_t groups = (n + 128) / 128;  // 16-byte words of n + 1 bits
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = kReachThreads / 32;
    for (;;) {
        if (tid == 0) s_v = atomicAdd(next, 1) + 1;
        __syncthreads();
        const int32_t v = s_v;
        if (v > n) break;
        int counts[2];
        for (int dir = 0; dir < 2; dir++) {
            const Adj a = dir == 0 ? out : in;
            const int32_t j0 = a.ptr[v], jh = a.hend[v], j1 = a.ptr[v + 1];
            for (int32_t i = tid; i < groups; i += kReachThreads) reinterpret_cast<uint4*>(bits)[i] = make_uint4(0, 0, 0, 0);
            if (tid == 0) s_cnt = 0;
            // neighbours with a bit row, in stretches: each thread ORs its words of them
            for (int32_t c0 = j0; c0 < jh; c0 += kReachRows) {
                const int32_t nr = min(kReachRows, jh - c0);
                for (int32_t j = tid; j < nr; j += kReachThreads) s_row[j] = a.row[a.idx[c0 + j]];
                __syncthreads();
                for (int32_t q = tid; q < groups * copies; q += kReachThreads) {
                    const int32_t g = q % groups;
                    uint4 acc = make_uint4(0, 0, 0, 0);
#pragma unroll 8
                    for (int32_t j = q / groups; j < nr; j += copies) {
                        const uint4 r = __ldg(a.rows + (size_t)s_row[j] * groups + g);
                        acc.x |= r.x;
                        acc.y |= r.y;
                        acc.z |= r.z;
                        acc.w |= r.w;
                    }
                    if (acc.x) atomicOr(&bits[4 * g], acc.x);
                    if (acc.y) atomicOr(&bits[4 * g + 1], acc.y);
                    if (acc.z) atomicOr(&bits[4 * g + 2], acc.z);
                    if (acc.w) atomicOr(&bits[4 * g + 3], acc.w);
                }
                __syncthreads();
            }
            __syncthreads();
            // the others: warps take the neighbours x, lanes stream x's list
            for (int32_t j = jh + warp; j < j1; j += nwarps) {
                const int32_t x = a.idx[j];
                for (int32_t k = a.ptr[x] + lane; k < a.ptr[x + 1]; k += 32) {
                    const int32_t y = a.idx[k];
                    atomicOr(&bits[y >> 5], 1u << (y & 31));
                }
            }
            __syncthreads();
            int c = 0;
            for (int32_t i = tid; i < 4 * groups; i += kReachThreads) c += __popc(bits[i]);
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

// The first candidate whose sum is at most ta (len: none), by a warp: 32
// probes a step.
__device__ __forceinline__ int32_t first_at_most(long long ta, const int4* cf, int32_t len, int lane) {
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
    return lo;
}

// The nearest unmatched B vertex of one A vertex, by a warp: the smallest key
// = distance << 17 | sorted position, so ties go to the first position
// (n <= 131071 < 2^17; distances stay below 2^46).  cf, cpos: the `len`
// candidates left at the last compaction by descending sum; `used`: the
// positions matched since.
__device__ unsigned long long nearest(const int4& f, const int4* cf, const int32_t* cpos, int32_t len,
                                      const uint8_t* used, int lane) {
    const long long ta = total(f);
    int32_t r = first_at_most(ta, cf, len, lane), l = r - 1;
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
                if (key < best && !used[p]) best = key;
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

using Key = unsigned long long;

__device__ __forceinline__ void order(Key& a, Key& b) {
    const Key lo = a < b ? a : b;
    b = a < b ? b : a;
    a = lo;
}

// One step of a bitonic network over a warp's lanes.
__device__ __forceinline__ void lane_step(Key& k, int lane, int stride, bool up) {
    const Key o = __shfl_xor_sync(0xffffffffu, k, stride);
    k = (((lane & stride) == 0) == up) == (o < k) ? o : k;
}

// Keys of 64 elements, element 32 r + lane in register r: those of (p0, p1) in
// any order and the sorted (k0, k1) give the sorted 64 smallest in (k0, k1).
__device__ void merge64(Key& k0, Key& k1, Key p0, Key p1, int lane) {
#pragma unroll
    for (int size = 2; size <= 32; size *= 2)
#pragma unroll
        for (int stride = size / 2; stride > 0; stride /= 2) {
            lane_step(p0, lane, stride, (lane & size) == 0);              // lane < 32: the 32-sort ascends,
            lane_step(p1, lane, stride, size < 32 && (lane & size) == 0);  // the second one descends
        }
    order(p0, p1);
#pragma unroll
    for (int stride = 16; stride > 0; stride /= 2) {
        lane_step(p0, lane, stride, true);
        lane_step(p1, lane, stride, true);
    }
    const Key q0 = __shfl_sync(0xffffffffu, p1, 31 - lane), q1 = __shfl_sync(0xffffffffu, p0, 31 - lane);
    k0 = q0 < k0 ? q0 : k0;
    k1 = q1 < k1 ? q1 : k1;
    order(k0, k1);
#pragma unroll
    for (int stride = 16; stride > 0; stride /= 2) {
        lane_step(k0, lane, stride, true);
        lane_step(k1, lane, stride, true);
    }
}

// list[64 i ..]: the kList smallest keys of A vertex head + i over the
// candidates, ascending, then ~0.  A warp scans outwards from its start and
// holds the list in registers; candidates below its last key wait in shared
// memory until there are more than 32.
__global__ void __launch_bounds__(kListThreads) shortlist_kernel(const int4* __restrict__ fa, int32_t head, int32_t count,
                                                                 const int4* __restrict__ cf,
                                                                 const int32_t* __restrict__ cpos,
                                                                 const int32_t* __restrict__ d_len, Key* __restrict__ list) {
    __shared__ Key s_wait[kListThreads / 32][64];
    const int lane = threadIdx.x & 31;
    const int32_t i = blockIdx.x * (kListThreads / 32) + (threadIdx.x >> 5);
    if (i >= count) return;
    Key* wait = s_wait[threadIdx.x >> 5];
    const int4 f = fa[head + i];
    const long long ta = total(f);
    const int32_t len = *d_len;
    int32_t r = first_at_most(ta, cf, len, lane), l = r - 1;
    Key k0 = ~0ull, k1 = ~0ull, last = ~0ull;
    int waiting = 0;
    bool go_r = r < len, go_l = l >= 0;
    while (go_r || go_l) {
        Key key[2] = {~0ull, ~0ull};
        long long edge[2] = {0, 0};  // the sum of the last candidate of this step on either side
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int32_t j = s ? l - lane : r + lane;
            if (s ? go_l && j >= 0 : go_r && j < len) {
                const int4 b = cf[j];
                key[s] = ((Key)l1(f, b) << 17) | (Key)cpos[j];
                edge[s] = total(b);
            }
        }
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const unsigned m = __ballot_sync(0xffffffffu, key[s] < last);
            if (key[s] < last) wait[waiting + __popc(m & ((1u << lane) - 1u))] = key[s];
            waiting += __popc(m);
            __syncwarp();
            if (waiting > 32) {
                merge64(k0, k1, wait[lane], lane + 32 < waiting ? wait[lane + 32] : ~0ull, lane);
                last = __shfl_sync(0xffffffffu, k1, 31);
                waiting = 0;
                __syncwarp();
            }
        }
        r += 32;
        l -= 32;
        const long long d = last == ~0ull ? LLONG_MAX : (long long)(last >> 17);
        const long long er = __shfl_sync(0xffffffffu, edge[0], 31), el = __shfl_sync(0xffffffffu, edge[1], 31);
        go_r = go_r && r < len && ta - er <= d;
        go_l = go_l && l >= 0 && el - ta <= d;
    }
    if (waiting > 0) merge64(k0, k1, lane < waiting ? wait[lane] : ~0ull, ~0ull, lane);
    list[(size_t)kList * i + lane] = k0;
    list[(size_t)kList * i + 32 + lane] = k1;
}

// Commits A vertices [first, end) (features and ids in sorted order: fa, ida).
// pi[ida[i]] = idb[j] for the position j chosen at step i.  cf, cpos, *d_len:
// what is left of B, before and after.  One warp goes through the vertices (a
// shared-memory read, a vote and a store a vertex are the chain: 0.1 us); the block's
// others load the lists and drop the matched candidates.
__global__ void __launch_bounds__(kGreedyThreads) commit_kernel(const int4* __restrict__ fa,
                                                                const int32_t* __restrict__ ida,
                                                                const int32_t* __restrict__ idb, int32_t n, int32_t first,
                                                                int32_t end, const Key* __restrict__ list, int4* cf,
                                                                int32_t* cpos, int32_t* d_len, int32_t* __restrict__ pi) {
    extern __shared__ __align__(16) uint8_t s_dyn[];
    int32_t* s_list = reinterpret_cast<int32_t*>(s_dyn);     // positions, n: none
    uint8_t* used = s_dyn + sizeof(int32_t) * kRound * kList;  // positions matched in this round, and n
    __shared__ int32_t s_choice[kRound];
    __shared__ int32_t s_wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int32_t len = *d_len;
    for (int32_t i = tid; i <= n / 16; i += kGreedyThreads) reinterpret_cast<uint4*>(used)[i] = make_uint4(0, 0, 0, 0);
    for (int32_t k = tid; k < (end - first) * kList; k += kGreedyThreads) {
        const Key key = list[k];
        s_list[k] = key == ~0ull ? n : (int32_t)(key & 0x1FFFFull);
    }
    __syncthreads();
    if (tid == 0) used[n] = 1;
    if (warp == 0) {
        __syncwarp();
        int32_t p0 = s_list[lane], p1 = s_list[32 + lane];
        for (int32_t i = 0; i < end - first; i++) {
            const bool f0 = !used[p0], f1 = !used[p1];
            const int32_t ahead = kList * min(i + 1, end - first - 1) + lane;
            const int32_t q0 = s_list[ahead], q1 = s_list[ahead + 32];
            const unsigned m0 = __ballot_sync(0xffffffffu, f0), m1 = __ballot_sync(0xffffffffu, f1);
            int32_t p = m0 ? p0 : p1;
            bool mine = lane == __ffs(m0 ? m0 : m1) - 1;
            if (!(m0 | m1)) {
                p = (int32_t)(nearest(fa[first + i], cf, cpos, len, used, lane) & 0x1FFFFull);
                mine = lane == 0;
            }
            if (mine) {
                used[p] = 1;
                s_choice[i] = p;
            }
            __syncwarp();
            p0 = q0;
            p1 = q1;
        }
    }
    __syncthreads();
    for (int32_t i = first + tid; i < end; i += kGreedyThreads) pi[ida[i]] = idb[s_choice[i - first]];
    int32_t base = 0;  // drop the matched candidates, in order
    for (int32_t j0 = 0; j0 < len; j0 += kGreedyThreads) {
        const int32_t j = j0 + tid;
        int4 f = make_int4(0, 0, 0, 0);
        int32_t p = 0;
        bool keep = false;
        if (j < len) {
            f = cf[j];
            p = cpos[j];
            keep = !used[p];
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
    if (tid == 0) *d_len = base;
}

// Sorted positions (descending feature sum, ties by id) of both graphs'
// vertices (blockIdx.z: 0 A, 1 B) by counting who comes before: 2 n^2
// comparisons, and nothing goes to the host and back.  rank: 2 (n + 1), zero.
__global__ void __launch_bounds__(256) rank_kernel(const int4* __restrict__ feat, int32_t n, int32_t* __restrict__ rank) {
    __shared__ long long s_t[256];
    const int4* f = feat + (size_t)blockIdx.z * (n + 1);
    const int32_t v = 1 + blockIdx.x * 256 + threadIdx.x;
    const long long mine = v <= n ? total(f[v]) : 0;
    int32_t c = 0;
    for (int32_t x0 = 1 + blockIdx.y * 256; x0 <= n; x0 += gridDim.y * 256) {
        const int32_t y = x0 + threadIdx.x;
        __syncthreads();
        s_t[threadIdx.x] = y <= n ? total(f[y]) : LLONG_MIN;
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < 256; k++) c += s_t[k] > mine || (s_t[k] == mine && x0 + k < v);
    }
    if (v <= n && c) atomicAdd(rank + (size_t)blockIdx.z * (n + 1) + v, c);
}

// A's features and ids in sorted order; B's as the first candidates.
__global__ void sorted_kernel(const int4* __restrict__ feat, const int32_t* __restrict__ rank, int32_t n, int4* __restrict__ fa,
                              int32_t* __restrict__ ida, int32_t* __restrict__ idb, int4* __restrict__ cf,
                              int32_t* __restrict__ cpos, int32_t* __restrict__ d_len) {
    const int32_t v = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (v > n) return;
    const int32_t ra = rank[v], rb = rank[n + 1 + v];
    fa[ra] = feat[v];
    ida[ra] = v;
    cf[rb] = feat[n + 1 + v];
    cpos[rb] = rb;
    idb[rb] = v;
    if (v == 1) *d_len = n;
}

// Plain adjacency (ids only, any order within a list but for the vertices with
// a bit row: the features are counts) of both directions of an edge list.
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

struct Fill {  // one direction while it is built
    int32_t* cnt;   // n+1: counts, then the front cursor of each list
    int32_t* back;  // n+1: the back cursor
    int32_t* ptr;   // n+2
    int32_t* idx;
    int32_t* row;   // n+1
    uint32_t* rows;
};

// Exclusive sums of the counts of one direction (block 0: out, 1: in) into
// ptr[0..n+1] and the fill cursors; rows for vertices with more than `heavy`
// neighbours.
__global__ void __launch_bounds__(1024) adj_scan_kernel(Fill out, Fill in, int32_t n, int32_t heavy) {
    __shared__ int32_t wsum[32];
    __shared__ int32_t s_rows;
    const Fill d = blockIdx.x ? in : out;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_rows = 0;
    int32_t base = 0;
    for (int32_t v0 = 0; v0 <= n; v0 += 1024) {
        const int32_t v = v0 + tid, c = v <= n ? d.cnt[v] : 0;
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
            d.ptr[v] = before + s - c;
            d.cnt[v] = before + s - c;
            d.back[v] = before + s;
            d.row[v] = c > heavy ? atomicAdd(&s_rows, 1) : -1;
        }
        __syncthreads();
    }
    if (tid == 0) d.ptr[n + 1] = base;
}

__global__ void adj_fill_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ dst, int64_t m, int32_t n,
                                Fill out, Fill in) {
    const size_t words = 4 * (size_t)((n + 128) / 128);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t s = src[e], d = dst[e];
        if ((uint32_t)(s - 1) >= (uint32_t)n || (uint32_t)(d - 1) >= (uint32_t)n) continue;
        out.idx[out.row[d] >= 0 ? atomicAdd(out.cnt + s, 1) : atomicSub(out.back + s, 1) - 1] = d;
        in.idx[in.row[s] >= 0 ? atomicAdd(in.cnt + d, 1) : atomicSub(in.back + d, 1) - 1] = s;
        const int32_t rs = out.row[s], rd = in.row[d];
        if (rs >= 0) atomicOr(out.rows + rs * words + (d >> 5), 1u << (d & 31));
        if (rd >= 0) atomicOr(in.rows + rd * words + (s >> 5), 1u << (s & 31));
    }
}

// Memory of one call: a single block, cut into 256-byte aligned arrays.
struct Arena {
    char* mem = nullptr;
    size_t used = 0;
    ~Arena() { bm_cuda_free(mem); }
    template <typename T>
    void get(T** p, size_t count) {
        *p = mem ? reinterpret_cast<T*>(mem + used) : nullptr;
        used += (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~(size_t)255;
    }
};

struct Work {
    int32_t *src, *dst;
    Fill d[2];  // out, in
    int* misc;  // next vertex, bad endpoint, candidates left
    int4 *feat, *fa, *cf;
    int32_t *rank, *ida, *idb, *cpos, *pi;
    Key* list;
};

// heavy: a list longer than this has a bit row (at most m / (heavy + 1) lists).
void lay_out(Arena& a, Work& w, int32_t n, int64_t m, int32_t heavy) {
    const size_t M = (size_t)m, V = (size_t)n + 2;
    a.used = 0;
    a.get(&w.misc, 4);
    a.get(&w.src, M);
    a.get(&w.dst, M);
    for (Fill& f : w.d) {
        a.get(&f.cnt, V);
        a.get(&f.back, V);
        a.get(&f.ptr, V);
        a.get(&f.row, V);
        a.get(&f.idx, M);
        a.get(&f.rows, heavy == INT32_MAX ? 1 : (M / ((size_t)heavy + 1)) * 4 * (size_t)((n + 128) / 128));
    }
    a.get(&w.feat, 2 * V);
    a.get(&w.rank, 2 * V);
    a.get(&w.fa, V);
    a.get(&w.cf, V);
    a.get(&w.ida, V);
    a.get(&w.idb, V);
    a.get(&w.cpos, V);
    a.get(&w.pi, V);
    a.get(&w.list, (size_t)kRound * kList);
}

// Features (in, out, reach2, canreach2) of one graph into feat[1..n]; endpoints
// outside 1..n set misc[1] and are left out.
bm_status graph_features(bm_ctx* ctx, const Work& w, int32_t n, int64_t m, int32_t heavy, const int32_t* src,
                         const int32_t* dst, int4* feat) {
    const size_t M = (size_t)m, V = (size_t)n + 2;
    if (m > 0) {
        BM_CUDA(ctx, cudaMemcpyAsync(w.src, src, sizeof(int32_t) * M, cudaMemcpyHostToDevice, ctx->stream));
        BM_CUDA(ctx, cudaMemcpyAsync(w.dst, dst, sizeof(int32_t) * M, cudaMemcpyHostToDevice, ctx->stream));
    }
    const size_t groups = (size_t)((n + 128) / 128);
    for (const Fill& f : w.d) {
        BM_CUDA(ctx, cudaMemsetAsync(f.cnt, 0, sizeof(int32_t) * V, ctx->stream));
        if (heavy != INT32_MAX && m > heavy)
            BM_CUDA(ctx, cudaMemsetAsync(f.rows, 0, M / ((size_t)heavy + 1) * groups * 16, ctx->stream));
    }
    BM_CUDA(ctx, cudaMemsetAsync(w.misc, 0, sizeof(int), ctx->stream));
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((m + 255) / 256, (int64_t)ctx->num_sms * 8));
    adj_count_kernel<<<grid, 256, 0, ctx->stream>>>(w.src, w.dst, m, n, w.d[0].cnt, w.d[1].cnt, w.misc + 1);
    BM_LAUNCH_CHECK(ctx, "adj_count_kernel");
    adj_scan_kernel<<<2, 1024, 0, ctx->stream>>>(w.d[0], w.d[1], n, heavy);
    BM_LAUNCH_CHECK(ctx, "adj_scan_kernel");
    adj_fill_kernel<<<grid, 256, 0, ctx->stream>>>(w.src, w.dst, m, n, w.d[0], w.d[1]);
    BM_LAUNCH_CHECK(ctx, "adj_fill_kernel");
    const size_t smem = groups * 16;
    // rows ORed at once: the fewest of up to eight that leave the fewest threads of the last step idle
    int copies = 1;
    auto idle = [&](int c) { return (double)((groups * c + kReachThreads - 1) / kReachThreads * kReachThreads) / (groups * c); };
    for (int c = 2; c <= 8; c++)
        if (idle(c) < idle(copies)) copies = c;
    auto adj = [](const Fill& f) { return Adj{f.ptr, f.idx, f.cnt, f.row, reinterpret_cast<const uint4*>(f.rows)}; };
    reach2_kernel<<<ctx->num_sms * 8, kReachThreads, smem, ctx->stream>>>(adj(w.d[0]), adj(w.d[1]), n, copies, w.misc,
                                                                            feat);
    BM_LAUNCH_CHECK(ctx, "reach2_kernel");
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
    const int64_t m = std::max(mA, mB);
    int32_t heavy = std::max(64, n / 64);
    Arena mem;
    Work w;
    for (;;) {
        lay_out(mem, w, n, m, heavy);
        if (bm_cuda_malloc((void**)&mem.mem, mem.used) == cudaSuccess) break;
        cudaGetLastError();
        mem.mem = nullptr;
        if (heavy == INT32_MAX) return bm_fail(ctx, BM_OOM, "greedy matching: device allocation failed");
        heavy = INT32_MAX;  // without the bit rows
    }
    lay_out(mem, w, n, m, heavy);
    bm_status s;
    BM_CUDA(ctx, cudaMemsetAsync(w.misc, 0, 4 * sizeof(int), ctx->stream));
    BM_CUDA(ctx, cudaMemsetAsync(w.rank, 0, sizeof(int32_t) * 2 * ((size_t)n + 1), ctx->stream));
    BM_CUDA(ctx, cudaMemsetAsync(w.pi, 0, sizeof(int32_t) * ((size_t)n + 1), ctx->stream));
    if ((s = graph_features(ctx, w, n, mA, heavy, srcA, dstA, w.feat)) != BM_OK) return s;
    if ((s = graph_features(ctx, w, n, mB, heavy, srcB, dstB, w.feat + (n + 1))) != BM_OK) return s;
    const unsigned nb = (unsigned)((n + 255) / 256);
    rank_kernel<<<dim3(nb, std::min(nb, 16u), 2), 256, 0, ctx->stream>>>(w.feat, n, w.rank);
    BM_LAUNCH_CHECK(ctx, "rank_kernel");
    sorted_kernel<<<nb, 256, 0, ctx->stream>>>(w.feat, w.rank, n, w.fa, w.ida, w.idb, w.cf, w.cpos, w.misc + 2);
    BM_LAUNCH_CHECK(ctx, "sorted_kernel");
    const size_t smem = sizeof(int32_t) * kRound * kList + ((size_t)n / 16 + 1) * 16;
    BM_CUDA(ctx, cudaFuncSetAttribute(commit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int32_t head = 0; head < n; head += kRound) {
        const int32_t count = std::min(kRound, n - head);
        shortlist_kernel<<<(count + kListThreads / 32 - 1) / (kListThreads / 32), kListThreads, 0, ctx->stream>>>(
            w.fa, head, count, w.cf, w.cpos, w.misc + 2, w.list);
        BM_LAUNCH_CHECK(ctx, "shortlist_kernel");
        commit_kernel<<<1, kGreedyThreads, smem, ctx->stream>>>(w.fa, w.ida, w.idb, n, head, head + count, w.list, w.cf,
                                                                w.cpos, w.misc + 2, w.pi);
        BM_LAUNCH_CHECK(ctx, "commit_kernel");
    }
    int bad = 0;
    BM_CUDA(ctx, cudaMemcpyAsync(&bad, w.misc + 1, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (bad) {
        const int32_t* ends[4] = {srcA, dstA, srcB, dstB};
        const int64_t ms[4] = {mA, mA, mB, mB};
        for (int q = 0; q < 4; q++)
            for (int64_t e = 0; e < ms[q]; e++)
                if (ends[q][e] < 1 || ends[q][e] > n)
                    return bm_fail(ctx, BM_INVALID_ARG, "edge endpoint %d outside 1..%d", ends[q][e], n);
    }
    BM_CUDA(ctx, cudaMemcpyAsync(pi, w.pi, sizeof(int32_t) * ((size_t)n + 1), cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BM_OK;
}
