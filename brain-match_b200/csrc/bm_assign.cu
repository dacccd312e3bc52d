// bm_assign.cu — re-assignment of an A-independent vertex subset by an optimal
// linear assignment: the method of src/independent-hungarian/hungarianSubset.c
// (random independent subset :657-740, one-sided gains one_side_swap_delta
// :414-459, optimal_assignment with the Hungarian method hungarian.c:144-334,
// apply and re-score :760-795).
//
// For a subset T = {t_0..t_{k-1}} with no A edge between two members, the
// score change of giving each t_i the old image of t_sigma(i) is exactly
// sum_i c[i][sigma(i)] with c[i][j] = G_{t_i}(pi t_j) - S(t_i) (+ self-loop
// terms), G_u(f) = sum over u's A entries of min(w, B at f and the neighbour's
// image): every A edge touches at most one member, so the moves do not
// interact.  The reference skips self-loops in the gains and re-scores; here
// they are included, so the delta is exact.
//
// On the device: the gains of a member against all images come from the row
// kernel in its one-sided mode (the first two 2-hop terms only), read at the
// members' columns; the assignment is solved by the auction algorithm
// (Bertsekas) with epsilon scaling on benefits multiplied by k + 1, which makes
// the final epsilon = 1 phase exactly optimal for integer benefits, with prices,
// bids and owners in one CTA's shared memory; apply_perm_kernel then moves
// every changed member at once (S updates of its A entries, relabelled B
// entries naming its new image, pi and pi^-1).
#include <algorithm>
#include <chrono>
#include <climits>
#include <numeric>
#include <vector>

#include <cooperative_groups.h>

#include "bm_internal.cuh"
#include "bm_rng.hpp"

namespace cg = cooperative_groups;

namespace {

constexpr int kLapThreads = 1024;
constexpr int kLapMaxK = 4096;
constexpr int kLapIdBits = 13;  // person index in a bid key (k <= 4096 < 2^13)
constexpr int kPermThreads = 256;

// Bounded auction: `limit` SM clock cycles at most (by default kAuctionLimit,
// ~10 s); status 1 means it ran out.
constexpr long long kAuctionLimit = 20000000000ll;

// The auction: one CTA holds the state and runs the rounds; where a round has
// many bidders the CTAs of its cluster share their rows (each reads the prices
// and places its bids through distributed shared memory), since one SM reads
// the benefits at a small part of the L2's rate.  Every round all unassigned
// persons bid at the same prices; of a random subset's assignment three rounds
// in four have a single bidder (a chain of displaced persons), so a round's
// fixed cost is what bounds it: the list of bidders is carried from round to round instead of being
// searched for among all persons, the warps share the rows of few bidders
// (all 32 one row when there is one), and only the objects that got a bid are
// visited.  Values and prices are computed in 32 bits while they stay below
// 2^30 (benefits times k + 1 and every bid, checked), else in 64: the same
// integers, and the same assignment as one CTA's.  k = 1,542 of the full-scale
// pair: 33.5 ms with a warp a row and the searches and one CTA throughout, 14.6
// ms in one CTA as it is now, 13 ms with the cluster.
struct AuctionSmem {
    unsigned long long* bid;  // per object: bid << kLapIdBits | reversed person, 0: none
    int32_t* owner;           // per object
    int32_t* pobj;            // per person: its object or -1
    int32_t* list[2];         // bidders of this round and of the next
    int32_t* bidobj;          // per bidder of this round
    unsigned long long* key;  // per bidder of a shared round: its bid, or why there is none
};

// A round's orders to the other CTAs of the cluster.
struct AuctionCmd {
    int32_t nu;   // bidders; 0: done
    int32_t cur;  // which list
    int32_t wide; // 64-bit values
    long long eps;
};

constexpr int kLapCluster = 8;
constexpr int kLapShared = 24;  // a round of more bidders goes to the whole cluster: its two barriers and the copy of
                                // the prices cost about 4,000 cycles, a single CTA's 32 bidders 13,000
constexpr int kLapClusterMin = 256;  // a smaller matrix is solved by one CTA

template <typename T>
struct Top2 {
    T v1, v2;
    int32_t j1;
};

template <typename T>
__device__ __forceinline__ T lowest() { return sizeof(T) == 4 ? (T)INT_MIN : (T)LLONG_MIN; }

// Best and second-best of two disjoint parts; equal bests: the lower object.
template <typename T>
__device__ __forceinline__ void merge(Top2<T>& a, T v1, T v2, int32_t j1) {
    if (v1 > a.v1 || (v1 == a.v1 && j1 < a.j1)) {
        a.v2 = a.v1 > v2 ? a.v1 : v2;
        a.v1 = v1;
        a.j1 = j1;
    } else if (v1 > a.v2) {
        a.v2 = v1;
    }
}

template <typename T>
__device__ __forceinline__ void warp_merge(Top2<T>& t) {
    if constexpr (sizeof(T) == 4) {
        // three warp reductions: the best, its lowest object, and the best of
        // what is left (the winner's second and the others' bests)
        const T v1 = __reduce_max_sync(0xffffffffu, t.v1);
        const int32_t j1 = __reduce_min_sync(0xffffffffu, t.v1 == v1 ? t.j1 : INT_MAX);
        t.v2 = __reduce_max_sync(0xffffffffu, t.v1 == v1 && t.j1 == j1 ? t.v2 : t.v1);
        t.v1 = v1;
        t.j1 = j1;
    } else {
        for (int o = 16; o; o >>= 1) {
            const T v1 = __shfl_xor_sync(0xffffffffu, t.v1, o), v2 = __shfl_xor_sync(0xffffffffu, t.v2, o);
            const int32_t j1 = __shfl_xor_sync(0xffffffffu, t.j1, o);
            merge(t, v1, v2, j1);
        }
    }
}

// A thread's share (objects j0, j0 + step, ...) of person i's values.  BATCH
// loads are in flight together, the last ones under a predicate: a share is
// rarely longer than a batch, and a remainder loop would wait for each load.
template <int BATCH, typename T>
__device__ __forceinline__ Top2<T> scan_row(const int32_t* __restrict__ a, const T* price, int32_t k, T scale, int32_t i,
                                            int32_t j0, int32_t step) {
    Top2<T> t{lowest<T>(), lowest<T>(), INT_MAX};
    const int32_t* row = a + (size_t)i * (size_t)k;
    for (int32_t b = j0; b < k; b += BATCH * step) {
        int32_t x[BATCH];
#pragma unroll
        for (int r = 0; r < BATCH; r++) x[r] = b + r * step < k ? __ldg(row + b + r * step) : 0;
#pragma unroll
        for (int r = 0; r < BATCH; r++) {
            const int32_t j = b + r * step;
            // no branches: the warp's lanes rarely agree on them
            const T v = j < k ? (T)x[r] * scale - price[j] : lowest<T>();
            const T low = v < t.v1 ? v : t.v1;
            t.j1 = v > t.v1 ? j : t.j1;
            t.v1 = v > t.v1 ? v : t.v1;
            t.v2 = low > t.v2 ? low : t.v2;
        }
    }
    return t;
}

constexpr long long kNarrowMax = 1ll << 30;

// A bidder's bid from its best two values: 0 and its key, 1 too large for the
// keys, 2 too large for T.
template <typename T>
__device__ __forceinline__ int bid_key(const T* price, const Top2<T>& t, int32_t i, long long eps, unsigned long long* key) {
    const long long v2 = t.v2 == lowest<T>() ? (long long)t.v1 : (long long)t.v2;  // a single object
    const long long b = (long long)price[t.j1] + ((long long)t.v1 - v2) + eps;
    if (b >= (1ll << (63 - kLapIdBits))) return 1;
    if (sizeof(T) == 4 && b >= kNarrowMax) return 2;
    *key = ((unsigned long long)b << kLapIdBits) | (unsigned long long)((1 << kLapIdBits) - 1 - i);
    return 0;
}

template <typename T>
__device__ __forceinline__ int place_bid(const AuctionSmem& s, const T* price, const Top2<T>& t, int32_t q, int32_t i,
                                         long long eps) {
    unsigned long long key;
    const int st = bid_key(price, t, i, eps, &key);
    s.bidobj[q] = t.j1;
    if (!st) atomicMax(&s.bid[t.j1], key);
    return st;
}

// Bidders q0, q0 + step, ... of a round, a warp each.  SHARED: the bids are
// left by bidder, for the state's CTA to enter: 64-bit maxima on its shared
// memory from other CTAs, beside its own, lost bids.  (Keys are at least 1 << kLapIdBits, a lower
// value is bid_key's status.)
template <typename T, bool SHARED>
__device__ __forceinline__ void bid_rows(const int32_t* __restrict__ a, int32_t k, const AuctionSmem& s, const T* price,
                                         const int32_t* list, int32_t nu, int32_t q0, int32_t step, long long eps,
                                         int32_t* s_flag) {
    const int lane = threadIdx.x & 31;
    for (int32_t q = q0; q < nu; q += step) {
        const int32_t i = list[q];
        Top2<T> t = scan_row<16>(a, price, k, (T)k + 1, i, lane, 32);
        warp_merge(t);
        if (lane == 0) {
            if (SHARED) {
                unsigned long long key;
                const int st = bid_key(price, t, i, eps, &key);
                s.bidobj[q] = t.j1;
                s.key[q] = st ? (unsigned long long)st : key;
            } else {
                const int st = place_bid(s, price, t, q, i, eps);
                if (st) atomicMax(s_flag, st);
            }
        }
    }
}

// Rounds from the current phase on with values of type T; returns 0 when the
// last phase is done, 1 on failure, 2 when a bid no longer fits T (the round's
// bids are withdrawn: the wider type repeats the round).
template <typename T, int CL>
__device__ int auction_rounds(const int32_t* __restrict__ a, int32_t k, const AuctionSmem& s, T* price, long long& eps,
                              int& cur, int32_t& nu, long long t0, long long limit, Top2<T>* part, int32_t* s_count,
                              int32_t* s_flag, AuctionCmd* cmd) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int W = kLapThreads / 32;
    const T scale = (T)k + 1;
    for (;;) {
        while (nu > 0) {
            if (nu == 1) {
                // a chain: the bidder takes its best object unopposed and whoever
                // held that bids next.  The round ends with its flag and count being
                // read and no barrier behind that, so both are written between the
                // two barriers only, the clock's verdict too
                const int32_t i = s.list[cur][0];
                Top2<T> t = scan_row<kLapMaxK / kLapThreads>(a, price, k, scale, i, tid, kLapThreads);
                warp_merge(t);
                if (lane == 0) part[warp] = t;
                __syncthreads();
                if (warp == 0) {
                    t = part[lane];
                    warp_merge(t);
                    if (lane == 0) {
                        const int st = clock64() - t0 > limit ? 1 : place_bid(s, price, t, 0, i, eps);
                        const int32_t j = t.j1;
                        if (st) {
                            *s_flag = st;
                        } else {
                            price[j] = (T)(long long)(s.bid[j] >> kLapIdBits);
                            const int32_t old = s.owner[j];
                            s.owner[j] = i;
                            s.pobj[i] = j;
                            if (old >= 0) {
                                s.pobj[old] = -1;
                                s.list[cur][0] = old;
                            }
                            *s_count = old >= 0;
                        }
                        s.bid[j] = 0ull;
                    }
                }
                __syncthreads();
                const int flag = *s_flag;
                if (flag) {
                    __syncthreads();
                    if (tid == 0) *s_flag = 0;
                    __syncthreads();
                    return flag;
                }
                nu = *s_count;
                continue;
            }
            const int32_t* list = s.list[cur];
            int32_t* next = s.list[cur ^ 1];
            if (tid == 0) {
                *s_count = 0;
                if (clock64() - t0 > limit) *s_flag = 1;
            }
            if (nu <= W / 2) {
                // the warps in groups, a group to a bidder
                int32_t group = W;
                while (group * nu > W) group >>= 1;
                const int32_t q = warp / group;
                if (q < nu) {
                    Top2<T> t = scan_row<8>(a, price, k, scale, list[q], (warp - q * group) * 32 + lane, group * 32);
                    warp_merge(t);
                    if (lane == 0) part[warp] = t;
                }
                __syncthreads();
                if (warp < nu) {
                    Top2<T> t{lowest<T>(), lowest<T>(), INT_MAX};
                    if (lane < group) t = part[warp * group + lane];
                    warp_merge(t);
                    if (lane == 0) {
                        const int st = place_bid(s, price, t, warp, list[warp], eps);
                        if (st) *s_flag = st;
                    }
                }
            } else if (CL > 1 && nu > kLapShared) {
                if (tid == 0) *cmd = AuctionCmd{nu, cur, sizeof(T) == 8, eps};
                cg::this_cluster().sync();  // the order and the state are seen
                bid_rows<T, true>(a, k, s, price, list, nu, warp * CL, W * CL, eps, s_flag);
                cg::this_cluster().sync();  // all bids are left
                for (int32_t q = tid; q < nu; q += kLapThreads) {
                    const unsigned long long key = s.key[q];
                    if (key >> kLapIdBits) atomicMax(&s.bid[s.bidobj[q]], key);
                    else atomicMax(s_flag, (int32_t)key);
                }
            } else {
                bid_rows<T, false>(a, k, s, price, list, nu, warp, W, eps, s_flag);
            }
            __syncthreads();
            const int flag = *s_flag;
            if (flag) {
                for (int32_t q = tid; q < nu; q += kLapThreads) s.bid[s.bidobj[q]] = 0ull;
                __syncthreads();
                if (tid == 0) *s_flag = 0;
                __syncthreads();
                return flag;
            }
            // objects go to their highest bidder (the lowest person on ties); who
            // lost or was displaced bids again
            for (int32_t q = tid; q < nu; q += kLapThreads) {
                const int32_t i = list[q], j = s.bidobj[q];
                const unsigned long long key = s.bid[j];
                int32_t again = i;
                if ((1 << kLapIdBits) - 1 - (int32_t)(key & ((1ull << kLapIdBits) - 1)) == i) {
                    price[j] = (T)(long long)(key >> kLapIdBits);
                    again = s.owner[j];
                    if (again >= 0) s.pobj[again] = -1;
                    s.owner[j] = i;
                    s.pobj[i] = j;
                }
                if (again >= 0) next[atomicAdd(s_count, 1)] = again;
            }
            __syncthreads();
            for (int32_t q = tid; q < nu; q += kLapThreads) s.bid[s.bidobj[q]] = 0ull;
            nu = *s_count;
            cur ^= 1;
            __syncthreads();
        }
        if (eps == 1) return 0;
        eps = max(1ll, eps / 5);
        for (int32_t i = tid; i < k; i += kLapThreads) {
            s.pobj[i] = -1;
            s.owner[i] = -1;
            s.list[cur][i] = i;
        }
        nu = k;
        __syncthreads();
    }
}

// The other CTAs of the cluster: every shared round they copy the prices, bid
// for their part of the bidders and place the bids in the state's CTA.
template <typename T>
__device__ __forceinline__ void auction_help(const int32_t* __restrict__ a, int32_t k, const AuctionSmem& s, T* price,
                                             const T* price0, const AuctionCmd& c, int rank, int ncta) {
    for (int32_t j = threadIdx.x; j < k; j += kLapThreads) price[j] = price0[j];
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    bid_rows<T, true>(a, k, s, price, s.list[c.cur], c.nu, warp * ncta + rank, (kLapThreads / 32) * ncta, c.eps, nullptr);
}

// d_max: the largest |benefit| (at most 2^30).  total: the assignment's total.
template <int CL>
__device__ __forceinline__ void auction_body(const int32_t* __restrict__ a, int32_t k, const int32_t* __restrict__ d_max,
                                             int32_t* __restrict__ assign, int32_t* __restrict__ status,
                                             long long* __restrict__ total, long long limit) {
    extern __shared__ unsigned long long lsm[];
    __shared__ Top2<long long> part[kLapThreads / 32];
    __shared__ int32_t s_count, s_flag;
    __shared__ unsigned long long s_total;
    __shared__ AuctionCmd s_cmd;
    long long* price = reinterpret_cast<long long*>(lsm);
    const int tid = threadIdx.x;
    const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
    // the state: this CTA's shared memory in rank 0, rank 0's in the others
    auto state = [&](unsigned long long* base) {
        AuctionSmem s;
        s.bid = base + k;
        s.key = base + 2 * k;
        s.owner = reinterpret_cast<int32_t*>(base + 3 * k);
        s.pobj = s.owner + k;
        s.list[0] = s.pobj + k;
        s.list[1] = s.list[0] + k;
        s.bidobj = s.list[1] + k;
        return s;
    };
    if constexpr (CL > 1) {
        if (rank != 0) {
            cg::cluster_group cl = cg::this_cluster();
            unsigned long long* base0 = cl.map_shared_rank(lsm, 0);
            const AuctionSmem s = state(base0);
            const AuctionCmd* cmd0 = cl.map_shared_rank(&s_cmd, 0);
            for (;;) {  // ends with rank 0's rounds, which are bounded
                cl.sync();
                const AuctionCmd c = *cmd0;
                if (c.nu == 0) break;
                if (c.wide)
                    auction_help(a, k, s, price, reinterpret_cast<const long long*>(base0), c, rank, CL);
                else
                    auction_help(a, k, s, reinterpret_cast<int32_t*>(price), reinterpret_cast<const int32_t*>(base0), c,
                                 rank, CL);
                cl.sync();
            }
            cl.sync();  // rank 0's shared memory is read no more
            return;
        }
    }
    const AuctionSmem s = state(lsm);
    const long long t0 = clock64();
    const long long top = max(1, *d_max) * ((long long)k + 1);
    for (int32_t j = tid; j < k; j += kLapThreads) {
        price[j] = 0;
        s.bid[j] = 0ull;
        s.owner[j] = -1;
        s.pobj[j] = -1;
        s.list[0][j] = j;
    }
    if (tid == 0) { s_flag = 0; s_total = 0ull; }
    __syncthreads();
    long long eps = max(1ll, top / 5);
    int cur = 0;
    int32_t nu = k;
    int st = 2;
    if (top <= kNarrowMax)
        st = auction_rounds<int32_t, CL>(a, k, s, reinterpret_cast<int32_t*>(price), eps, cur, nu, t0, limit,
                                         reinterpret_cast<Top2<int32_t>*>(part), &s_count, &s_flag, &s_cmd);
    if (st == 2) {
        if (top <= kNarrowMax) {  // the prices so far, widened in place
            int32_t p[kLapMaxK / kLapThreads];
#pragma unroll
            for (int r = 0; r < kLapMaxK / kLapThreads; r++) {
                const int32_t j = tid + r * kLapThreads;
                p[r] = j < k ? reinterpret_cast<int32_t*>(price)[j] : 0;
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kLapMaxK / kLapThreads; r++) {
                const int32_t j = tid + r * kLapThreads;
                if (j < k) price[j] = p[r];
            }
            __syncthreads();
        }
        st = auction_rounds<long long, CL>(a, k, s, price, eps, cur, nu, t0, limit, part, &s_count, &s_flag, &s_cmd);
    }
    if constexpr (CL > 1) {
        if (tid == 0) s_cmd.nu = 0;
        cg::this_cluster().sync();
    }
    long long sum = 0;
    for (int32_t i = tid; i < k; i += kLapThreads) {
        const int32_t j = s.pobj[i];
        assign[i] = j;
        if (j >= 0) sum += a[(size_t)i * (size_t)k + (size_t)j];
    }
    atomicAdd(&s_total, (unsigned long long)sum);
    __syncthreads();
    if (tid == 0) {
        *status = st != 0;
        *total = (long long)s_total;
    }
    if constexpr (CL > 1) cg::this_cluster().sync();
}

__global__ void __launch_bounds__(kLapThreads) auction_kernel(const int32_t* a, int32_t k, const int32_t* d_max,
                                                              int32_t* assign, int32_t* status, long long* total,
                                                              long long limit) {
    auction_body<1>(a, k, d_max, assign, status, total, limit);
}

__global__ void __cluster_dims__(kLapCluster, 1, 1) __launch_bounds__(kLapThreads)
auction_cluster_kernel(const int32_t* a, int32_t k, const int32_t* d_max, int32_t* assign, int32_t* status,
                       long long* total, long long limit) {
    auction_body<kLapCluster>(a, k, d_max, assign, status, total, limit);
}

// The largest |benefit| of a matrix, added to *out by maximum.
__global__ void max_abs_kernel(const int32_t* __restrict__ a, int64_t count, int32_t* __restrict__ out) {
    int32_t m = 0;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = __ldg(a + q);
        m = max(m, v < 0 ? -v : v);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

struct PermArgs {
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

// One CTA per moved member u: old image g0, new image g1.  Members share no A
// edge, so every neighbour's image is fixed while the members move.
__global__ void __launch_bounds__(kPermThreads) apply_perm_kernel(PermArgs a, const int32_t* __restrict__ who,
                                                                  const int32_t* __restrict__ old_img,
                                                                  const int32_t* __restrict__ new_img) {
    const int32_t u = who[blockIdx.x], g0 = old_img[blockIdx.x], g1 = new_img[blockIdx.x];
    if (g0 == g1) return;
    for (int32_t j = a.A.out_ptr[u] + threadIdx.x; j < a.A.out_ptr[u + 1]; j += kPermThreads) {
        const uint32_t ent = a.A.out_ent[j];
        if (ent == 0) continue;
        const int32_t x = bm_eid(ent), w = bm_ew(ent);
        const int32_t gx = a.pi[x];
        const int32_t d = imin(w, bm_hash_get(a.hb, g1, gx)) - imin(w, bm_hash_get(a.hb, g0, gx));
        if (d) { atomicAdd(a.ov + u, d); atomicAdd(a.ov + x, d); }
    }
    for (int32_t j = a.A.in_ptr[u] + threadIdx.x; j < a.A.in_ptr[u + 1]; j += kPermThreads) {
        const uint32_t ent = a.A.in_ent[j];
        if (ent == 0) continue;
        const int32_t x = bm_eid(ent), w = bm_ew(ent);
        const int32_t gx = a.pi[x];
        const int32_t d = imin(w, bm_hash_get(a.hb, gx, g1)) - imin(w, bm_hash_get(a.hb, gx, g0));
        if (d) { atomicAdd(a.ov + u, d); atomicAdd(a.ov + x, d); }
    }
    // B entries naming the new image now name u (found through the twins)
    for (int dir = 0; dir < 2; dir++) {
        const int32_t* ptr = dir ? a.Bout_ptr : a.Bin_ptr;
        const int32_t* twin = dir ? a.Bout_twin : a.Bin_twin;
        uint32_t* other = dir ? a.Bin_ent : a.Bout_ent;
        for (int32_t j = ptr[g1] + threadIdx.x; j < ptr[g1 + 1]; j += kPermThreads) {
            const int32_t t = twin[j];
            if (t < 0) continue;
            other[t] = (other[t] & ~BM_ID_MASK) | (uint32_t)u;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a.pi[u] = g1;
        a.pinv[g1] = u;
        a.ximg[u] = bm_image_bounds(a.Bin_ptr, a.Bout_ptr, g1);
    }
}

size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t lap_smem(int32_t k) { return (size_t)k * (3 * 8 + 5 * 4); }

// What the auction leaves beside the assignment.
struct LapOut {
    long long total;
    int32_t status;
    int32_t max_abs;
};

bm_status lap_device(bm_ctx* ctx, const int32_t* d_a, int32_t k, int32_t* d_assign, LapOut* d_out) {
    const size_t smem = lap_smem(k);
    BM_CUDA(ctx, cudaMemsetAsync(d_out, 0, sizeof(LapOut), ctx->stream));
    const int64_t count = (int64_t)k * k;
    max_abs_kernel<<<(unsigned)std::min<int64_t>((count + 1023) / 1024, (int64_t)ctx->num_sms * 4), 256, 0, ctx->stream>>>(
        d_a, count, &d_out->max_abs);
    BM_LAUNCH_CHECK(ctx, "max_abs_kernel");
    const long long limit = ctx->wait_limit > 0 ? (long long)ctx->wait_limit : kAuctionLimit;
    if (k >= kLapClusterMin) {
        BM_CUDA(ctx, cudaFuncSetAttribute(auction_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        auction_cluster_kernel<<<kLapCluster, kLapThreads, smem, ctx->stream>>>(d_a, k, &d_out->max_abs, d_assign,
                                                                               &d_out->status, &d_out->total, limit);
        BM_LAUNCH_CHECK(ctx, "auction_cluster_kernel");
    } else {
        BM_CUDA(ctx, cudaFuncSetAttribute(auction_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        auction_kernel<<<1, kLapThreads, smem, ctx->stream>>>(d_a, k, &d_out->max_abs, d_assign, &d_out->status,
                                                              &d_out->total, limit);
        BM_LAUNCH_CHECK(ctx, "auction_kernel");
    }
    return BM_OK;
}

// Subset checks: ids in 1..n, distinct, no A edge between two members.
bm_status check_subset(bm_ctx* ctx, const int32_t* subset, int32_t k, BmMarks& mk) {
    mk.reset(ctx->n);
    for (int32_t i = 0; i < k; i++)
        if (subset[i] < 1 || subset[i] > ctx->n)
            return bm_fail(ctx, BM_INVALID_ARG, "subset[%d] = %d outside 1..%d", i, subset[i], ctx->n);
    for (int32_t i = 0; i < k; i++) {
        if (mk.marked(subset[i]))
            return bm_fail(ctx, BM_INVALID_ARG, "subset[%d] = %d repeats or shares an A edge with another member", i,
                           subset[i]);
        mk.mark_closed(ctx, subset[i]);
    }
    return BM_OK;
}

// Gains, assignment and apply for a checked subset; *delta, *changed.
bm_status assign_subset(bm_ctx* ctx, const int32_t* subset, int32_t k, int64_t* delta, int32_t* changed) {
    const size_t sb = al256(sizeof(int32_t) * (size_t)k), cb = al256(sizeof(int32_t) * (size_t)k * (size_t)k);
    bm_status s;
    if ((s = bm_stage(ctx, 5 * sb + cb + 256)) != BM_OK) return s;
    char* base = (char*)ctx->stage;
    int32_t* d_sub = (int32_t*)base;
    int32_t* d_asg = (int32_t*)(base + sb);
    int32_t* d_old = (int32_t*)(base + 2 * sb);
    int32_t* d_new = (int32_t*)(base + 3 * sb);
    int32_t* d_who = (int32_t*)(base + 4 * sb);
    int32_t* d_cost = (int32_t*)(base + 5 * sb);
    LapOut* d_out = (LapOut*)(base + 5 * sb + cb);
    BM_CUDA(ctx, cudaMemcpyAsync(d_sub, subset, sizeof(int32_t) * (size_t)k, cudaMemcpyHostToDevice, ctx->stream));
    if ((s = bm_launch_rows_gen(ctx, d_sub, nullptr, k, nullptr, nullptr, nullptr, 0, 0, d_sub, k, d_cost)) != BM_OK)
        return s;
    if ((s = lap_device(ctx, d_cost, k, d_asg, d_out)) != BM_OK) return s;
    std::vector<int32_t> asg((size_t)k), old((size_t)k), pi((size_t)ctx->n + 1);
    LapOut out;
    BM_CUDA(ctx, cudaMemcpyAsync(asg.data(), d_asg, sizeof(int32_t) * (size_t)k, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(&out, d_out, sizeof out, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(pi.data(), ctx->pi, sizeof(int32_t) * pi.size(), cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int32_t i = 0; i < k; i++) old[(size_t)i] = pi[(size_t)subset[i]];  // old images of the members
    if (out.status) return bm_fail(ctx, BM_TIMEOUT, "auction did not finish within its bound");
    std::vector<int32_t> who, o_img, n_img;
    const int64_t d = out.total;
    std::vector<char> seen((size_t)k, 0);
    for (int32_t i = 0; i < k; i++) {
        const int32_t j = asg[(size_t)i];
        if (j < 0 || j >= k || seen[(size_t)j]) return bm_fail(ctx, BM_CUDA_ERROR, "auction returned no permutation");
        seen[(size_t)j] = 1;
        if (j != i) {
            who.push_back(subset[i]);
            o_img.push_back(old[(size_t)i]);
            n_img.push_back(old[(size_t)j]);
        }
    }
    const int32_t m = (int32_t)who.size();
    if (m > 0) {
        BM_CUDA(ctx, cudaMemcpyAsync(d_who, who.data(), sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, ctx->stream));
        BM_CUDA(ctx, cudaMemcpyAsync(d_old, o_img.data(), sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, ctx->stream));
        BM_CUDA(ctx, cudaMemcpyAsync(d_new, n_img.data(), sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, ctx->stream));
        const DevGraph& B = ctx->g[1];
        PermArgs pa{gview(ctx->g[0]), B.out_ptr, B.in_ptr, B.out_ent, B.in_ent, B.out_twin, B.in_twin, hview(B),
                    ctx->pi, ctx->pinv, ctx->ov, ctx->ximg};
        apply_perm_kernel<<<m, kPermThreads, 0, ctx->stream>>>(pa, d_who, d_old, d_new);
        BM_LAUNCH_CHECK(ctx, "apply_perm_kernel");
        BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    ctx->score += d;
    if (delta) *delta = d;
    if (changed) *changed = m;
    return BM_OK;
}

}  // namespace

extern "C" bm_status bm_lap_solve(bm_ctx* ctx, const int32_t* benefit, int32_t k, int32_t* assign, int64_t* total) {
    if (!ctx || !benefit || !assign) return BM_INVALID_ARG;
    if (k < 1 || k > kLapMaxK) return bm_fail(ctx, BM_INVALID_ARG, "k = %d outside 1..%d", k, kLapMaxK);
    BM_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t cb = al256(sizeof(int32_t) * (size_t)k * (size_t)k), ab = al256(sizeof(int32_t) * (size_t)k);
    bm_status s = bm_stage(ctx, cb + ab + 256);
    if (s != BM_OK) return s;
    int32_t* d_a = (int32_t*)ctx->stage;
    int32_t* d_asg = (int32_t*)((char*)ctx->stage + cb);
    LapOut* d_out = (LapOut*)((char*)ctx->stage + cb + ab);
    long long mx = 1;
    for (size_t q = 0; q < (size_t)k * (size_t)k; q++) {
        const long long v = benefit[q];
        mx = std::max(mx, v < 0 ? -v : v);
    }
    if (mx > (1ll << 30)) return bm_fail(ctx, BM_INVALID_ARG, "benefits must stay within +-2^30");
    BM_CUDA(ctx, cudaMemcpyAsync(d_a, benefit, sizeof(int32_t) * (size_t)k * (size_t)k, cudaMemcpyHostToDevice,
                                 ctx->stream));
    if ((s = lap_device(ctx, d_a, k, d_asg, d_out)) != BM_OK) return s;
    LapOut out;
    BM_CUDA(ctx, cudaMemcpyAsync(assign, d_asg, sizeof(int32_t) * (size_t)k, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(&out, d_out, sizeof out, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (out.status) return bm_fail(ctx, BM_TIMEOUT, "auction did not finish within its bound");
    if (total) *total = out.total;
    return BM_OK;
}

extern "C" bm_status bm_subset_assign(bm_ctx* ctx, const int32_t* subset, int32_t k, int64_t* delta,
                                      int32_t* changed) {
    bm_status s = bm_require_mapped(ctx);
    if (s != BM_OK) return s;
    if (!subset || k < 1 || k > kLapMaxK) return bm_fail(ctx, BM_INVALID_ARG, "k = %d outside 1..%d", k, kLapMaxK);
    if ((s = bm_rows_smem_check(ctx)) != BM_OK) return s;
    BmMarks mk;
    if ((s = check_subset(ctx, subset, k, mk)) != BM_OK) return s;
    return assign_subset(ctx, subset, k, delta, changed);
}

extern "C" bm_status bm_search_hungarian(bm_ctx* ctx, int32_t k, uint64_t seed, int32_t iterations,
                                         double time_budget_s, bm_progress* prog) {
    using clk = std::chrono::steady_clock;
    bm_status s = bm_require_mapped(ctx);
    if (s != BM_OK) return s;
    if (!prog) return bm_fail(ctx, BM_INVALID_ARG, "progress struct required");
    if (k < 2 || k > kLapMaxK) return bm_fail(ctx, BM_INVALID_ARG, "k = %d outside 2..%d", k, kLapMaxK);
    if ((s = bm_rows_smem_check(ctx)) != BM_OK) return s;
    const int32_t n = ctx->n;
    const auto t0 = clk::now();
    std::vector<uint64_t> keyv((size_t)n);
    std::vector<int32_t> order((size_t)n), subset;
    BmMarks mk;
    bm_status ret = BM_OK;
    const uint32_t key[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
    for (int32_t it = 0; iterations < 0 || it < iterations; it++) {
        if (time_budget_s > 0 && std::chrono::duration<double>(clk::now() - t0).count() >= time_budget_s) {
            ret = BM_TIMEOUT;
            break;
        }
        // a random order of the vertices (Philox keys, counter = vertex and
        // iteration), then greedily the members with disjoint closed A
        // neighbourhoods, the reference's random independent subset
        for (int32_t v = 1; v <= n; v++) {
            const uint32_t c[4] = {(uint32_t)v, (uint32_t)prog->launches, 0x48554E47u, 0u};
            uint32_t o[4];
            bm_philox4x32_10(c, key, o);
            keyv[(size_t)v - 1] = ((uint64_t)o[0] << 32) | o[1];
            order[(size_t)v - 1] = v;
        }
        std::sort(order.begin(), order.end(), [&](int32_t p, int32_t q) {
            const uint64_t a = keyv[(size_t)p - 1], b = keyv[(size_t)q - 1];
            return a != b ? a < b : p < q;
        });
        mk.reset(n);
        subset.clear();
        for (int32_t v : order) {
            if ((int32_t)subset.size() >= k) break;
            if (mk.marked(v)) continue;  // v is a member or next to one
            subset.push_back(v);
            mk.mark_closed(ctx, v);
        }
        int64_t d = 0;
        int32_t changed = 0;
        if ((s = assign_subset(ctx, subset.data(), (int32_t)subset.size(), &d, &changed)) != BM_OK) return s;
        prog->launches++;
        prog->accepts += changed;
        prog->rows_done += (int64_t)subset.size();
        prog->evaluated += (int64_t)subset.size() * (int64_t)subset.size();
    }
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    prog->seconds += std::chrono::duration<double>(clk::now() - t0).count();
    s = bm_check_score(ctx);
    prog->score = ctx->score;
    if (s != BM_OK) return s;
    return ret;
}
