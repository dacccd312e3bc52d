// bm_kset.cu — exact deltas of permutations of small vertex sets (k <= 8):
// the 3-vertex moves of src/graph-re-alignment-gpu-3-swap.cu:43-305 (best of
// the non-identity permutations of a triple, applied by apply_permutation
// :925-956) and the permutation sets of
// src/graph-alignment-permset-parallel.c:304-363,625-746 (all k! permutations
// of a random k-subset, the best one applied).  The reference's group delta
// counts an edge inside the group twice and is repaired by a full re-score
// (:698-730); here the delta is exact.
//
// For a set T = {t_0..t_{k-1}} with images f_i = pi(t_i) and a permutation
// sigma (member i takes the image of member sigma(i)):
//
//   delta(sigma) = sum_i (g[i][sigma i] - S(t_i)) + sum over A entries e = (t_i -> t_j, w)
//                  inside T of [h(si, sj) + h(i, j) - h(si, j) - h(i, sj)] + self-loop terms
//
// with g[i][q] = G_{t_i}(f_q) = sum_{x in out(t_i)} min(w, B(f_q, pi x)) +
// sum_{x in in(t_i)} min(w, B(pi x, f_q)) (old images everywhere, so
// g[i][i] = S(t_i)), h(p, q) = min(w, B(f_p, f_q)) and h(p, p) = 0.  The first
// sum moves every member's external and internal edges as if the other end
// stayed; the second repairs each internal edge to its true new value.
//
// One CTA per set.  The B rows of the members' images (out and in) mark, in a
// table indexed by the low bits of the id, which members' rows may hold it;
// the members' lists are then scanned once, and only an entry that meets a
// mark looks its weight up in the hash, atomics into g in shared memory.
// (Binary searches of the k-1 rows, staged in shared memory, for every entry
// took 146,000 of a set's cycles on average, this scan 53,000: what bounds it
// now is the latency of the lookups of hubs, which are in most rows.)
//
// The best permutation (largest delta, the first in lexicographic order on
// ties) is then found in one of two ways.  The delta is a sum of one term per
// member but for the internal entries.  With the images of a vertex cover of
// the internal entries fixed, every other member's term depends on its own
// image alone, and those members form an assignment problem, solved by a table
// over subsets of the images left: E[mask] = the best total of the members not
// yet placed when the images of mask are taken, 2^m values for m members,
// filled from the full mask down.  So the c members of a smallest cover are
// enumerated, k!/(k-c)! choices, a warp to a choice.  A sparse graph's random
// sets have c = 0 (one table of 256 values instead of 40,320 permutations at
// k = 8) or, with a hub among them, c = 1.  Past the limit of cover_limit(),
// for calls that want every permutation's delta, and for k < 6, the k!
// permutations are enumerated, each thread a contiguous block stepped by the
// lexicographic successor (the permutation packed in one register).
#include <climits>
#include <vector>

#include "bm_internal.cuh"

namespace {

constexpr int kKThreads = 256;
constexpr int kMaxK = 8;
constexpr int kMaxInternal = 256;

struct KsetArgs {
    GView A;
    HashView hb;
    const int32_t* selfB;
    int has_self;
    const int32_t* pi;
    const int32_t* ov;
    int32_t n;
    int32_t k;
    int32_t kfact;
    const int32_t* sets;
    int64_t nsets;
    long long* best_delta;
    int32_t* best_perm;  // nsets * k
    long long* all;      // nsets * kfact, optional
    int32_t* status;     // nonzero: some set was rejected (see bm_kset_eval)
    // B's rows in B ids
    const int32_t* Bout_ptr;
    const int32_t* Bin_ptr;
    const uint32_t* Bout_ent0;
    const uint32_t* Bin_ent0;
};

// Row marks per direction, indexed by the id's low bits: exact up to 16,384
// ids; beyond, two ids that share a mark cost a lookup that finds nothing.
constexpr int kMaskIds = 16384;
constexpr size_t kKsetSmem = 2 * kMaskIds;

__device__ __forceinline__ void decode_perm(int32_t p, int k, int32_t* s) {
    int32_t avail[kMaxK];
    int32_t f = 1;
    for (int i = 0; i < k; i++) avail[i] = i;
    for (int i = 2; i < k; i++) f *= i;  // (k-1)!
    for (int i = 0; i < k; i++) {
        const int32_t idx = (k - 1 - i) > 0 ? p / f : 0;
        if (k - 1 - i > 0) p -= idx * f;
        s[i] = avail[idx];
        for (int j = idx; j < k - 1 - i; j++) avail[j] = avail[j + 1];
        if (k - 1 - i > 0) f /= (k - 1 - i);
    }
}

// The permutations [p0, p1) of K members, in lexicographic order, evaluated
// from the gain table g (shared), the internal entries and the self-loop
// terms; the best (largest delta, lowest index) is returned in bd, bp.  A
// permutation is held as K 4-bit fields of one register (field i = s[i]), so
// that the lexicographic successor is shifts and masks rather than indexed
// register arrays.
__device__ __forceinline__ uint32_t nib(uint32_t S, int i) { return (S >> (4 * i)) & 15u; }

template <int K>
__device__ void enumerate_perms(const KsetArgs& a, int64_t set, int32_t p0, int32_t p1, const int32_t* g,
                                const int32_t* Bsub, const int32_t* sA, const int32_t* sB, int32_t ni,
                                const int32_t* ie_i, const int32_t* ie_j, const int32_t* ie_w, long long& bd,
                                int32_t& bp) {
    int32_t s0[kMaxK];
    decode_perm(p0, K, s0);
    uint32_t S = 0;
#pragma unroll
    for (int i = 0; i < K; i++) S |= (uint32_t)s0[i] << (4 * i);
    long long base = 0;  // sum of g[i][i]
#pragma unroll
    for (int i = 0; i < K; i++) base += g[i * K + i];
    if constexpr (K >= 4) {
        // Without internal entries, self-loop terms or per-permutation output,
        // six consecutive permutations (p0 and p1 multiples of 6) share the
        // first K - 3 fields and order the last three values a < b < c as abc,
        // acb, bac, bca, cab, cba: one successor step per six, nine table reads.
        if (ni == 0 && !a.has_self && !a.all && p0 % 6 == 0 && p1 % 6 == 0) {
            const int32_t* g0 = g + (K - 3) * K;
            const int32_t* g1 = g + (K - 2) * K;
            const int32_t* g2 = g + (K - 1) * K;
            for (int32_t p = p0; p < p1; p += 6) {
                long long sp = -base;
#pragma unroll
                for (int i = 0; i < K - 3; i++) sp += g[i * K + (int)nib(S, i)];
                const int x = (int)nib(S, K - 3), y = (int)nib(S, K - 2), z = (int)nib(S, K - 1);
                const long long d6[6] = {sp + g0[x] + g1[y] + g2[z], sp + g0[x] + g1[z] + g2[y],
                                         sp + g0[y] + g1[x] + g2[z], sp + g0[y] + g1[z] + g2[x],
                                         sp + g0[z] + g1[x] + g2[y], sp + g0[z] + g1[y] + g2[x]};
#pragma unroll
                for (int q = 0; q < 6; q++)
                    if (d6[q] > bd) { bd = d6[q]; bp = p + q; }
                // the group's last permutation (suffix z y x), then its successor
                S = (S & ~(0xFFFu << (4 * (K - 3)))) |
                    ((uint32_t)z << (4 * (K - 3))) | ((uint32_t)y << (4 * (K - 2))) | ((uint32_t)x << (4 * (K - 1)));
                int piv = -1;
#pragma unroll
                for (int i = 0; i < K - 1; i++)
                    if (nib(S, i) < nib(S, i + 1)) piv = i;
                if (piv < 0) break;
                const uint32_t sv = nib(S, piv);
                int j = piv + 1;
#pragma unroll
                for (int jj = 1; jj < K; jj++)
                    if (jj > piv && nib(S, jj) > sv) j = jj;
                const uint32_t sj = nib(S, j);
                S = (S & ~((15u << (4 * piv)) | (15u << (4 * j)))) | (sj << (4 * piv)) | (sv << (4 * j));
                uint32_t R = 0;
#pragma unroll
                for (int i = 0; i < K; i++) {
                    const int src = (i > piv) ? (K - 1 - (i - piv - 1)) : i;
                    R |= nib(S, src) << (4 * i);
                }
                S = R;
            }
            return;
        }
    }
    for (int32_t p = p0; p < p1; p++) {
        long long d = -base;
#pragma unroll
        for (int i = 0; i < K; i++) d += g[i * K + (int)nib(S, i)];
        for (int32_t e = 0; e < ni; e++) {
            const int i = ie_i[e], j = ie_j[e], w = ie_w[e];
            const int si = (int)nib(S, i), sj = (int)nib(S, j);
            d += imin(w, Bsub[si * K + sj]) + imin(w, Bsub[i * K + j]) - imin(w, Bsub[si * K + j]) -
                 imin(w, Bsub[i * K + sj]);
        }
        if (a.has_self) {
#pragma unroll
            for (int i = 0; i < K; i++) d += imin(sA[i], sB[nib(S, i)]) - imin(sA[i], sB[i]);
        }
        if (a.all) a.all[set * a.kfact + p] = d;
        if (d > bd) { bd = d; bp = p; }
        // lexicographic successor: pivot = last i with s[i] < s[i+1]; swap it
        // with the last larger field after it; reverse the fields after it
        int piv = -1;
#pragma unroll
        for (int i = 0; i < K - 1; i++)
            if (nib(S, i) < nib(S, i + 1)) piv = i;
        if (piv < 0) break;
        const uint32_t sp = nib(S, piv);
        int j = piv + 1;
#pragma unroll
        for (int jj = 1; jj < K; jj++)
            if (jj > piv && nib(S, jj) > sp) j = jj;
        const uint32_t sj = nib(S, j);
        S = (S & ~((15u << (4 * piv)) | (15u << (4 * j)))) | (sj << (4 * piv)) | (sp << (4 * j));
        // reverse fields piv+1 .. K-1
        uint32_t R = 0;
#pragma unroll
        for (int i = 0; i < K; i++) {
            const int src = (i > piv) ? (K - 1 - (i - piv - 1)) : i;
            R |= nib(S, src) << (4 * i);
        }
        S = R;
    }
}

// The c-th choice of images for the members of `cover` (in member order, images
// in lexicographic order of the choice), as 4-bit fields at the members'
// places; `used` gets the images taken.
__device__ __forceinline__ uint32_t decode_choice(int32_t c, int k, uint32_t cover, int32_t count, uint32_t& used) {
    uint32_t S = 0;
    used = 0;
    int32_t radix = count;  // choices of the members from here on
    int left = k;
    for (uint32_t m = cover; m; m &= m - 1, left--) {
        const int i = __ffs(m) - 1;
        radix /= left;
        int idx = c / radix;
        c -= idx * radix;
        uint32_t avail = ~used & ((1u << k) - 1u);
        for (; idx > 0; idx--) avail &= avail - 1;
        const uint32_t q = (uint32_t)__ffs(avail) - 1u;
        S |= q << (4 * i);
        used |= 1u << q;
    }
    return S;
}

constexpr int kCoverChoices = 336;  // 8 * 7 * 6: the most choices of a cover (see cover_limit)

// The largest cover that is enumerated; -1: always the permutations.  A choice
// costs a warp about 300 instructions, a permutation a thread about 100, so
// k!/(k-c)! choices on 8 warps stay below k! permutations on 256 threads up to
// c = 3 at k = 8 (336 choices against 40,320), 2 at k = 7 and 1 at k = 6.
__device__ __forceinline__ int cover_limit(int k) { return k - 5 > 0 ? k - 5 : -1; }

struct CoverSmem {
    long long E[1024];                  // 256 values for c = 0, else 128 to a warp
    int32_t W[kKThreads / 32][64];      // gains of the members left, by the images left
    long long val[kCoverChoices];
    unsigned key;
    int cover;
};

// Change of an internal entry's term when its ends take images si and sj.
__device__ __forceinline__ int32_t repair(int32_t w, const int32_t* Bsub, int k, int i, int j, int si, int sj) {
    return imin(w, Bsub[si * k + sj]) + imin(w, Bsub[i * k + j]) - imin(w, Bsub[si * k + j]) - imin(w, Bsub[i * k + sj]);
}

// The place-th set bit of m.
__device__ __forceinline__ int nth_bit(uint32_t m, int place) {
    for (; place > 0; place--) m &= m - 1;
    return __ffs(m) - 1;
}

// One choice of the cover's images (fields S, images `used`): the gains of the
// members left in W, the table in E, by the threads t, t + STRIDE, ... of a
// warp or the whole CTA; returns the choice's best total (E[0] and the cover's
// own terms).
template <int STRIDE>
__device__ long long cover_choice(int k, const int32_t* g, const int32_t* Bsub, const int32_t* sA, const int32_t* sB,
                                  int32_t ni, const int32_t* ie_i, const int32_t* ie_j, const int32_t* ie_w,
                                  uint32_t cover, uint32_t S, uint32_t used, int t, int32_t* W, long long* E) {
    const uint32_t full = (1u << k) - 1u, rest = full & ~cover, left = full & ~used;
    const int m = __popc(rest);
    auto sync = [] { if (STRIDE == 32) __syncwarp(); else __syncthreads(); };
    sync();  // the last choice's tables are no longer read
    for (int e = t; e < m * m; e += STRIDE) {
        const int i = nth_bit(rest, e / m), q = nth_bit(left, e % m);
        int32_t d = g[i * k + q] + imin(sA[i], sB[q]);
        for (int32_t n = 0; n < ni; n++) {
            const int x = ie_i[n], y = ie_j[n];
            if (x == i) d += repair(ie_w[n], Bsub, k, x, y, q, (int)nib(S, y));
            else if (y == i) d += repair(ie_w[n], Bsub, k, x, y, (int)nib(S, x), q);
        }
        W[e] = d;
    }
    if (t == 0) E[(1 << m) - 1] = 0;
    sync();
    for (int lev = m - 1; lev >= 0; lev--) {
        for (int mask = t; mask < (1 << m) - 1; mask += STRIDE) {
            if (__popc((unsigned)mask) != lev) continue;
            long long best = LLONG_MIN;
            for (uint32_t av = ((1u << m) - 1u) & ~(uint32_t)mask; av; av &= av - 1) {
                const int q = __ffs(av) - 1;
                const long long v = (long long)W[lev * m + q] + E[mask | (1 << q)];
                if (v > best) best = v;
            }
            E[mask] = best;
        }
        sync();
    }
    long long v = E[0];
    for (uint32_t c = cover; c; c &= c - 1) {
        const int i = __ffs(c) - 1, q = (int)nib(S, i);
        v += (long long)g[i * k + q] + imin(sA[i], sB[q]);
    }
    for (int32_t n = 0; n < ni; n++) {
        const int x = ie_i[n], y = ie_j[n];
        if (((cover >> x) & 1u) && ((cover >> y) & 1u))
            v += repair(ie_w[n], Bsub, k, x, y, (int)nib(S, x), (int)nib(S, y));
    }
    return v;
}

// The first permutation in lexicographic order that completes a choice to its
// best total, as a field string with member 0 foremost.
__device__ uint32_t cover_key(int k, uint32_t cover, uint32_t S, uint32_t used, const int32_t* W, const long long* E) {
    const uint32_t full = (1u << k) - 1u, left = full & ~used;
    const int m = __popc(left);
    uint32_t key = 0, mask = 0;
    int lev = 0;
    for (int i = 0; i < k; i++) {
        int q = (int)nib(S, i);
        if (!((cover >> i) & 1u)) {
            int a = 0;
            for (uint32_t av = ((1u << m) - 1u) & ~mask; av; av &= av - 1) {
                a = __ffs(av) - 1;
                if ((long long)W[lev * m + a] + E[mask | (1u << a)] == E[mask]) break;
            }
            mask |= 1u << a;
            lev++;
            q = nth_bit(left, a);
        }
        key |= (uint32_t)q << (28 - 4 * i);
    }
    return key;
}

// Best permutation of one set with the images of `cover` enumerated; whole
// CTA.  sA is zero when there are no self-loop terms.
__device__ void best_by_cover(const KsetArgs& a, int64_t set, const int32_t* g, const int32_t* Bsub, const int32_t* sA,
                              const int32_t* sB, int32_t ni, const int32_t* ie_i, const int32_t* ie_j,
                              const int32_t* ie_w, uint32_t cover, CoverSmem& cs) {
    const int k = a.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = __popc(cover);
    if (tid == 0) cs.key = 0xFFFFFFFFu;
    long long top;
    if (c == 0) {
        top = cover_choice<kKThreads>(k, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, 0u, 0u, 0u, tid, cs.W[0], cs.E);
        if (tid == 0) cs.key = cover_key(k, 0u, 0u, 0u, cs.W[0], cs.E);
    } else {
        int32_t count = 1;
        for (int t = 0; t < c; t++) count *= k - t;
        long long* E = cs.E + 128 * warp;
        for (int32_t ch = warp; ch < count; ch += kKThreads / 32) {
            uint32_t used;
            const uint32_t S = decode_choice(ch, k, cover, count, used);
            const long long v =
                cover_choice<32>(k, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, cover, S, used, lane, cs.W[warp], E);
            if (lane == 0) cs.val[ch] = v;
        }
        __syncthreads();
        top = LLONG_MIN;
        for (int32_t ch = lane; ch < count; ch += 32) top = max(top, cs.val[ch]);
        for (int o = 16; o; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        for (int32_t ch = warp; ch < count; ch += kKThreads / 32) {
            if (cs.val[ch] != top) continue;
            uint32_t used;
            const uint32_t S = decode_choice(ch, k, cover, count, used);
            if (count > kKThreads / 32)  // else the warp's tables are still this choice's
                cover_choice<32>(k, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, cover, S, used, lane, cs.W[warp], E);
            if (lane == 0) atomicMin(&cs.key, cover_key(k, cover, S, used, cs.W[warp], E));
        }
    }
    __syncthreads();
    if (tid < k) a.best_perm[set * k + tid] = (int32_t)((cs.key >> (28 - 4 * tid)) & 15u);
    if (tid == 0) {
        long long base = 0;
        for (int i = 0; i < k; i++) base += (long long)g[i * k + i] + imin(sA[i], sB[i]);
        a.best_delta[set] = top - base;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kKThreads, 4) kset_kernel(KsetArgs a) {
    extern __shared__ uint32_t rmask[];  // per id, the members whose B-out row holds it, then whose B-in row: bytes
    __shared__ CoverSmem cs;
    __shared__ uint32_t adj[kMaxK];  // members joined to member i by internal entries
    // the B rows (2q: B-out(f_q), 2q+1: B-in(f_q)) and the A lists (2i: out(t_i),
    // 2i+1: in(t_i)) as two streams of quads: running ends, and starts less the
    // quads before
    __shared__ int32_t r_beg[2 * kMaxK], r_end[2 * kMaxK], l_beg[2 * kMaxK], l_end[2 * kMaxK];
    __shared__ int32_t t[kMaxK], f[kMaxK], sA[kMaxK], sB[kMaxK];
    __shared__ int32_t g[kMaxK * kMaxK], Bsub[kMaxK * kMaxK];
    __shared__ int32_t n_int, bad;
    __shared__ int32_t ie_i[kMaxInternal], ie_j[kMaxInternal], ie_w[kMaxInternal];
    __shared__ long long red_d[kKThreads / 32];
    __shared__ int32_t red_p[kKThreads / 32];
    const int k = a.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int64_t set = blockIdx.x; set < a.nsets; set += gridDim.x) {
        if (tid == 0) n_int = bad = 0;
        if (tid < kMaxK) adj[tid] = 0u;
        for (int32_t i = tid; i < 2 * kMaskIds / 16; i += kKThreads)
            reinterpret_cast<uint4*>(rmask)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (tid < k) {
            const int32_t v = a.sets[set * k + tid];
            t[tid] = v;
            if (v < 1 || v > a.n) bad = 1;
        }
        if (tid < k * k) g[tid] = 0;
        __syncthreads();
        if (tid < k * k && tid / k < tid % k && t[tid / k] == t[tid % k]) bad = 1;
        __syncthreads();
        if (bad) {
            if (tid < k) a.best_perm[set * k + tid] = tid;
            if (tid == 0) { a.best_delta[set] = 0; atomicOr(a.status, 1); }
            if (a.all)
                for (int32_t p = tid; p < a.kfact; p += kKThreads) a.all[set * a.kfact + p] = 0;
            __syncthreads();
            continue;
        }
        if (tid < k) {
            f[tid] = a.pi[t[tid]];
            sA[tid] = a.has_self ? a.A.self_w[t[tid]] : 0;
        }
        __syncthreads();
        if (tid < k) sB[tid] = a.has_self ? a.selfB[f[tid]] : 0;
        if (tid < k * k) {
            const int p = tid / k, q = tid % k;
            Bsub[tid] = (p == q) ? 0 : bm_hash_get(a.hb, f[p], f[q]);
        }
        // ---- bounds of all rows and lists
        if (tid < 4 * k) {
            const bool row = tid < 2 * k;
            const int l = row ? tid : tid - 2 * k;
            const int32_t* ptr = row ? ((l & 1) ? a.Bin_ptr : a.Bout_ptr) : ((l & 1) ? a.A.in_ptr : a.A.out_ptr);
            const int32_t v = row ? f[l >> 1] : t[l >> 1];
            (row ? r_beg : l_beg)[l] = ptr[v] >> 2;
            (row ? r_end : l_end)[l] = ptr[v + 1] >> 2;
        }
        __syncthreads();
        if (tid == 0 || tid == 32) {
            int32_t* beg = tid ? l_beg : r_beg;
            int32_t* end = tid ? l_end : r_end;
            int32_t sum = 0;
            for (int l = 0; l < 2 * k; l++) {
                const int32_t b = beg[l];
                beg[l] = b - sum;
                sum += end[l] - b;
                end[l] = sum;
            }
        }
        __syncthreads();
        const int nl = 2 * k;
        auto list_of = [nl](const int32_t* end, int32_t q) {  // the list that quad q of a stream falls in
            int l = 0;
#pragma unroll
            for (int step = 8; step; step >>= 1)
                if (l + step < nl && end[l + step - 1] <= q) l += step;
            return l;
        };
        // ---- marks of the B rows
        for (int32_t q = tid; q < r_end[nl - 1]; q += kKThreads) {
            const int r = list_of(r_end, q), dir = r & 1;
            const uint4 e4 = __ldg(reinterpret_cast<const uint4*>(dir ? a.Bin_ent0 : a.Bout_ent0) + r_beg[r] + q);
            const uint32_t en4[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (en4[c] == 0) continue;
                const uint32_t at = dir * kMaskIds + ((uint32_t)bm_eid(en4[c]) & (kMaskIds - 1));
                atomicOr(rmask + (at >> 2), 1u << (8 * (at & 3) + (r >> 1)));
            }
        }
        __syncthreads();
        // ---- gains and internal entries: a thread a quad at a time; the lookups
        // of its four entries run in one loop, so that a warp's lanes do theirs
        // together
        for (int32_t q = tid; q < l_end[nl - 1]; q += kKThreads) {
            const int l = list_of(l_end, q), i = l >> 1, dir = l & 1;
            const uint4 e4 = __ldg(reinterpret_cast<const uint4*>(dir ? a.A.in_ent : a.A.out_ent) + l_beg[l] + q);
            const uint32_t en4[4] = {e4.x, e4.y, e4.z, e4.w};
            int32_t gx4[4];
            uint32_t found = 0;  // byte c: the rows that entry c meets
#pragma unroll
            for (int c = 0; c < 4; c++) gx4[c] = __ldg(a.pi + bm_eid(en4[c]));
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const uint32_t m = reinterpret_cast<const uint8_t*>(rmask)[dir * kMaskIds + (gx4[c] & (kMaskIds - 1))];
                found |= (en4[c] ? m & ~(1u << i) : 0u) << (8 * c);
            }
            if (dir == 0)
                for (int m = 0; m < k; m++) {
                    const uint32_t tm = (uint32_t)t[m];
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if ((en4[c] & BM_ID_MASK) == tm) {
                            const int32_t slot = atomicAdd(&n_int, 1);
                            if (slot < kMaxInternal) { ie_i[slot] = i; ie_j[slot] = m; ie_w[slot] = bm_ew(en4[c]); }
                            atomicOr(&adj[i], 1u << m);
                            atomicOr(&adj[m], 1u << i);
                        }
                }
            for (; found; found &= found - 1) {
                const int b = __ffs(found) - 1, c = b >> 3, m = b & 7;
                const int32_t gx = c == 0 ? gx4[0] : c == 1 ? gx4[1] : c == 2 ? gx4[2] : gx4[3];
                const uint32_t en = c == 0 ? en4[0] : c == 1 ? en4[1] : c == 2 ? en4[2] : en4[3];
                // out: B(f_m, pi x); in: B(pi x, f_m)
                const int32_t d = imin(bm_ew(en), dir ? bm_hash_get(a.hb, gx, f[m]) : bm_hash_get(a.hb, f[m], gx));
                if (d) atomicAdd(&g[i * k + m], d);
            }
        }
        __syncthreads();
        if (tid < k) g[tid * k + tid] = a.ov[t[tid]];
        if (tid == 0 && n_int > kMaxInternal) { bad = 1; atomicOr(a.status, 2); }
        __syncthreads();
        const int32_t ni = bad ? 0 : n_int;
        const int climit = cover_limit(k);
        if (climit >= 0 && !a.all && !bad) {
            // the smallest vertex cover (the lowest mask on ties): a thread a mask
            if (tid == 0) cs.cover = 0x7FFFFFFF;
            __syncthreads();
            if (tid < (1 << k)) {
                bool covers = true;
                for (int i = 0; i < k; i++) covers &= ((tid >> i) & 1) || (adj[i] & ~(uint32_t)tid) == 0u;
                if (covers) atomicMin(&cs.cover, (__popc((unsigned)tid) << kMaxK) | tid);
            }
            __syncthreads();
            if ((cs.cover >> kMaxK) <= climit) {
                best_by_cover(a, set, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, (uint32_t)cs.cover & ((1u << kMaxK) - 1u), cs);
                continue;
            }
        }
        // ---- enumerate permutations
        int32_t per = (a.kfact + kKThreads - 1) / kKThreads;
        if (k >= 4) per = (per + 5) / 6 * 6;  // whole groups of six (see enumerate_perms)
        const int32_t p0 = tid * per, p1 = min(a.kfact, p0 + per);
        long long bd = LLONG_MIN;
        int32_t bp = INT_MAX;
        if (!bad && p0 < p1) {
            switch (k) {
                case 2: enumerate_perms<2>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
                case 3: enumerate_perms<3>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
                case 4: enumerate_perms<4>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
                case 5: enumerate_perms<5>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
                case 6: enumerate_perms<6>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
                case 7: enumerate_perms<7>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
                default: enumerate_perms<8>(a, set, p0, p1, g, Bsub, sA, sB, ni, ie_i, ie_j, ie_w, bd, bp); break;
            }
        }
        if (bad && a.all)
            for (int32_t p = tid; p < a.kfact; p += kKThreads) a.all[set * a.kfact + p] = 0;
        // ---- block argmax (largest delta, lowest index)
        for (int o = 16; o; o >>= 1) {
            const long long d2 = __shfl_xor_sync(0xffffffffu, bd, o);
            const int32_t p2 = __shfl_xor_sync(0xffffffffu, bp, o);
            if (d2 > bd || (d2 == bd && p2 < bp)) { bd = d2; bp = p2; }
        }
        if (lane == 0) { red_d[warp] = bd; red_p[warp] = bp; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kKThreads / 32; w++)
                if (red_d[w] > red_d[0] || (red_d[w] == red_d[0] && red_p[w] < red_p[0])) {
                    red_d[0] = red_d[w];
                    red_p[0] = red_p[w];
                }
            if (bad) { red_d[0] = 0; red_p[0] = 0; }
            a.best_delta[set] = red_d[0];
            int32_t s[kMaxK];
            decode_perm(red_p[0], k, s);
            for (int i = 0; i < k; i++) a.best_perm[set * k + i] = s[i];
        }
        __syncthreads();
    }
}

// Apply permutations of independent sets: member i of set takes the image of
// member perm[i].  S updates of every A entry touching a member (entries
// inside a set once, from the out-lists), relabelled B entries, then pi.
struct ApplySetsArgs {
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
    int32_t k;
    const int32_t* sets;
    const int32_t* perms;
};

__global__ void __launch_bounds__(kKThreads) apply_sets_kernel(ApplySetsArgs a) {
    __shared__ int32_t t[kMaxK], f[kMaxK], fn[kMaxK];
    const int k = a.k;
    const int64_t set = blockIdx.x;
    if (threadIdx.x < k) {
        t[threadIdx.x] = a.sets[set * k + threadIdx.x];
        f[threadIdx.x] = a.pi[t[threadIdx.x]];
    }
    __syncthreads();
    if (threadIdx.x < k) fn[threadIdx.x] = f[a.perms[set * k + threadIdx.x]];
    __syncthreads();
    for (int i = 0; i < k; i++) {
        for (int dir = 0; dir < 2; dir++) {
            const int32_t* ptr = dir ? a.A.in_ptr : a.A.out_ptr;
            const uint32_t* ent = dir ? a.A.in_ent : a.A.out_ent;
            const int32_t b = ptr[t[i]], e = ptr[t[i] + 1];
            for (int32_t j = b + threadIdx.x; j < e; j += kKThreads) {
                const uint32_t en = ent[j];
                if (en == 0) continue;
                const int32_t x = bm_eid(en), w = bm_ew(en);
                int xq = -1;
                for (int q = 0; q < k; q++)
                    if (t[q] == x) xq = q;
                if (dir == 1 && xq >= 0) continue;  // inside the set: counted from the out-list
                const int32_t gx_old = a.pi[x];
                const int32_t gx_new = xq >= 0 ? fn[xq] : gx_old;
                int32_t d;
                if (dir == 0)
                    d = imin(w, bm_hash_get(a.hb, fn[i], gx_new)) - imin(w, bm_hash_get(a.hb, f[i], gx_old));
                else
                    d = imin(w, bm_hash_get(a.hb, gx_new, fn[i])) - imin(w, bm_hash_get(a.hb, gx_old, f[i]));
                if (d) { atomicAdd(a.ov + t[i], d); atomicAdd(a.ov + x, d); }
            }
        }
    }
    // image f[q] is now held by the member i with fn[i] == f[q]
    for (int i = 0; i < k; i++) {
        const int32_t img = fn[i];
        const uint32_t label = (uint32_t)t[i];
        for (int dir = 0; dir < 2; dir++) {
            const int32_t* ptr = dir ? a.Bout_ptr : a.Bin_ptr;
            const int32_t* twin = dir ? a.Bout_twin : a.Bin_twin;
            uint32_t* other = dir ? a.Bin_ent : a.Bout_ent;
            const int32_t b = ptr[img], e = ptr[img + 1];
            for (int32_t j = b + threadIdx.x; j < e; j += kKThreads) {
                const int32_t tw = twin[j];
                if (tw < 0) continue;
                other[tw] = (other[tw] & ~BM_ID_MASK) | label;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int i = 0; i < k; i++) {
            a.pi[t[i]] = fn[i];
            a.pinv[fn[i]] = t[i];
            a.ximg[t[i]] = bm_image_bounds(a.Bin_ptr, a.Bout_ptr, fn[i]);
        }
}

int32_t factorial(int k) {
    int32_t f = 1;
    for (int i = 2; i <= k; i++) f *= i;
    return f;
}

}  // namespace

bm_status bm_launch_kset(bm_ctx* ctx, int32_t k, const int32_t* d_sets, int64_t nsets, long long* d_best,
                         int32_t* d_perm, long long* d_all, int32_t* d_status) {
    if (nsets <= 0) return BM_OK;
    KsetArgs a;
    a.A = gview(ctx->g[0]);
    a.hb = hview(ctx->g[1]);
    a.selfB = ctx->g[1].self_w;
    a.has_self = ctx->g[0].has_self && ctx->g[1].has_self;
    a.pi = ctx->pi;
    a.ov = ctx->ov;
    a.n = ctx->n;
    a.k = k;
    a.kfact = factorial(k);
    a.Bout_ptr = ctx->g[1].out_ptr;
    a.Bin_ptr = ctx->g[1].in_ptr;
    a.Bout_ent0 = ctx->g[1].out_ent0;
    a.Bin_ent0 = ctx->g[1].in_ent0;
    a.sets = d_sets;
    a.nsets = nsets;
    a.best_delta = d_best;
    a.best_perm = d_perm;
    a.all = d_all;
    a.status = d_status;
    // a block per set: sets differ widely in cost (hubs, covers), and the
    // hardware hands out blocks as they finish
    const int64_t blocks = nsets < (1 << 20) ? nsets : (1 << 20);
    BM_CUDA(ctx, cudaFuncSetAttribute(kset_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKsetSmem));
    BM_CUDA(ctx, cudaFuncSetAttribute(kset_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      (int)cudaSharedmemCarveoutMaxShared));
    kset_kernel<<<(unsigned)blocks, kKThreads, kKsetSmem, ctx->stream>>>(a);
    BM_LAUNCH_CHECK(ctx, "kset_kernel");
    return BM_OK;
}

bm_status bm_launch_apply_sets(bm_ctx* ctx, int32_t k, const int32_t* d_sets, const int32_t* d_perms, int32_t nsets) {
    if (nsets <= 0) return BM_OK;
    const DevGraph& B = ctx->g[1];
    ApplySetsArgs a;
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
    a.k = k;
    a.sets = d_sets;
    a.perms = d_perms;
    apply_sets_kernel<<<nsets, kKThreads, 0, ctx->stream>>>(a);
    BM_LAUNCH_CHECK(ctx, "apply_sets_kernel");
    return BM_OK;
}

extern "C" bm_status bm_kset_eval(bm_ctx* ctx, int32_t k, const int32_t* sets, int64_t nsets, int64_t* best_delta,
                                  int32_t* best_perm, int64_t* all_deltas) {
    bm_status s = bm_require_mapped(ctx);
    if (s != BM_OK) return s;
    if (k < 2 || k > kMaxK) return bm_fail(ctx, BM_INVALID_ARG, "k must be 2..%d", kMaxK);
    if (nsets < 0 || (nsets > 0 && (!sets || !best_delta || !best_perm)))
        return bm_fail(ctx, BM_INVALID_ARG, "bad set buffers");
    if (nsets == 0) return BM_OK;
    for (int64_t i = 0; i < nsets; i++)
        for (int a = 0; a < k; a++) {
            const int32_t v = sets[i * k + a];
            if (v < 1 || v > ctx->n) return bm_fail(ctx, BM_INVALID_ARG, "set %lld: id %d outside 1..%d", (long long)i, v, ctx->n);
            for (int b = 0; b < a; b++)
                if (sets[i * k + b] == v) return bm_fail(ctx, BM_INVALID_ARG, "set %lld repeats vertex %d", (long long)i, v);
        }
    const int32_t kf = factorial(k);
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t b_sets = al(sizeof(int32_t) * (size_t)(nsets * k));
    const size_t b_best = al(sizeof(long long) * (size_t)nsets);
    const size_t b_perm = al(sizeof(int32_t) * (size_t)(nsets * k));
    const size_t b_stat = 256;
    const size_t b_all = all_deltas ? al(sizeof(long long) * (size_t)nsets * (size_t)kf) : 0;
    if ((s = bm_stage(ctx, b_sets + b_best + b_perm + b_stat + b_all)) != BM_OK) return s;
    char* base = (char*)ctx->stage;
    int32_t* d_sets = (int32_t*)base;
    long long* d_best = (long long*)(base + b_sets);
    int32_t* d_perm = (int32_t*)(base + b_sets + b_best);
    int32_t* d_stat = (int32_t*)(base + b_sets + b_best + b_perm);
    long long* d_all = all_deltas ? (long long*)(base + b_sets + b_best + b_perm + b_stat) : nullptr;
    BM_CUDA(ctx, cudaMemcpyAsync(d_sets, sets, sizeof(int32_t) * (size_t)(nsets * k), cudaMemcpyHostToDevice, ctx->stream));
    BM_CUDA(ctx, cudaMemsetAsync(d_stat, 0, sizeof(int32_t), ctx->stream));
    if ((s = bm_launch_kset(ctx, k, d_sets, nsets, d_best, d_perm, d_all, d_stat)) != BM_OK) return s;
    int32_t hstat = 0;
    BM_CUDA(ctx, cudaMemcpyAsync(best_delta, d_best, sizeof(long long) * (size_t)nsets, cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(best_perm, d_perm, sizeof(int32_t) * (size_t)(nsets * k), cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaMemcpyAsync(&hstat, d_stat, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    if (all_deltas)
        BM_CUDA(ctx, cudaMemcpyAsync(all_deltas, d_all, sizeof(long long) * (size_t)nsets * (size_t)kf,
                                     cudaMemcpyDeviceToHost, ctx->stream));
    BM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (hstat & 2)
        return bm_fail(ctx, BM_UNSUPPORTED, "a set has more than %d A entries between its members", kMaxInternal);
    return BM_OK;
}

extern "C" bm_status bm_kset_eval_dev(bm_ctx* ctx, int32_t k, const int32_t* d_sets, int64_t nsets,
                                      int64_t* d_best_delta, int32_t* d_best_perm, int32_t* d_status) {
    bm_status s = bm_require_mapped(ctx);
    if (s != BM_OK) return s;
    if (k < 2 || k > kMaxK) return bm_fail(ctx, BM_INVALID_ARG, "k must be 2..%d", kMaxK);
    if (nsets < 0 || (nsets > 0 && (!d_sets || !d_best_delta || !d_best_perm || !d_status)))
        return bm_fail(ctx, BM_INVALID_ARG, "bad set buffers");
    return bm_launch_kset(ctx, k, d_sets, nsets, (long long*)d_best_delta, d_best_perm, nullptr, d_status);
}
