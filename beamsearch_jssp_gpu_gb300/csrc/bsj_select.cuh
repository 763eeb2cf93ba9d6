// bsj_select.cuh -- one-CTA top-K selection of a level (gpu modes): the routes of k_select,
// shared by the level kernels and by the resident search, whose levels with too many tied
// scores fall back to them.
#pragma once

#include "bsj_kernels.h"

namespace bsj {

#ifndef FULL_MASK
#define FULL_MASK 0xFFFFFFFFu
#endif

// ---- thread-block clusters and distributed shared memory ----
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// all threads of all CTAs of the cluster (release / acquire at cluster scope)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() { cluster_arrive(); cluster_wait(); }
// the shared-memory address of `p`'s counterpart in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(const void* p, unsigned rank)
{
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t ld_peer(const void* p, unsigned rank)
{
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_addr(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld_peer4(const void* p, unsigned rank)
{
    uint4 v;
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(peer_addr(p, rank))
                 : "memory");
    return v;
}

// ------------------------------------------------------------------------------------
// k_select: exact top-K + stable order per beam (gpu modes).
//
// The reference sorts all P*n (score, slot) pairs with a stable radix sort and keeps the
// first min(P*n, K) (gpu/v1/solver.cu:255-274).  Scores of skipped slots are 1e9f, above
// every real score, so the kept list is: the real candidates in ascending
// (score bits, slot) order, then -- only when fewer than min(P*n,K) are real -- the
// lowest-numbered skipped slots ("fillers").  Keys are unique 64-bit
// (score bits << 32 | slot), so the top-K set is exact: an MSD radix select finds the
// K-th key, survivors are compacted and bitonic-sorted in shared memory.
// ------------------------------------------------------------------------------------
struct SelSmem {
    uint32_t* hist;            // 16 KB: u32[4096] bucket counts | u16[32][256] digit counters | u32[16][256]
    uint32_t* tot;             // [256]
    unsigned long long* red;   // [64]
    int* misc;                 // [64]
    unsigned long long* A;     // [kLsdMax]   compacted survivors / radix-sort buffer
    unsigned long long* stg;   // [kStageKeys] staged candidate keys / radix-sort buffer / wide bitonic
    uint32_t rmin, rmax;       // min / max score bits of the level's keys (from k_step's chunk ranges)
};

constexpr int kLsdMax = 8192;      // largest survivor count for the radix sort
constexpr int kStageKeys = 16384;  // candidate keys staged in shared memory

__device__ __forceinline__ SelSmem sel_smem(uint8_t* base, uint32_t rmin = 0xFFFFFFFFu, uint32_t rmax = 0u)
{
    SelSmem s;
    s.rmin = rmin;
    s.rmax = rmax;
    s.hist = reinterpret_cast<uint32_t*>(base);
    s.tot = s.hist + 4096;
    s.red = reinterpret_cast<unsigned long long*>(s.tot + 256);
    s.misc = reinterpret_cast<int*>(s.red + 64);
    s.A = reinterpret_cast<unsigned long long*>(s.misc + 64);
    s.stg = s.A + kLsdMax;
    return s;
}

constexpr size_t kSelectSmemBytes =
    (size_t)(4096 + 256) * 4 + 64 * 8 + 64 * 4 + (size_t)(kLsdMax + kStageKeys) * 8;

// Block-wide exclusive scan of one int per thread; returns the prefix, *total the sum.
static __device__ int block_exclusive_scan(int v, int* total, int* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nwarps ? warp_sums[lane] : 0;
        int ws = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(FULL_MASK, ws, o);
            if (lane >= o) ws += y;
        }
        warp_sums[32 + lane] = ws - w;
        if (lane == 31) warp_sums[64] = ws;
    }
    __syncthreads();
    int res = warp_sums[32 + warp] + x - v;
    *total = warp_sums[64];
    __syncthreads();
    return res;
}

// Candidate keys of one beam live in per-chunk regions of cap keys each, filled to
// cpref[c+1]-cpref[c]; logical key i is found by a binary search over the prefix.
struct KeySrc {
    const unsigned long long* base;
    const int* cpref;  // shared memory, nch+1 entries
    int nch;
    int cap;
    __device__ __forceinline__ unsigned long long operator()(int i) const
    {
        int lo = 0, hi = nch;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (cpref[mid] <= i) lo = mid; else hi = mid;
        }
        return base[(size_t)lo * cap + (i - cpref[lo])];
    }
    // fn(key) on every key, warp per chunk (order not preserved)
    template <typename Fn>
    __device__ __forceinline__ void each_key(Fn fn) const
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        for (int c = warp; c < nch; c += nw) {
            const int c0 = cpref[c], nc = cpref[c + 1] - c0;
            const unsigned long long* src = base + (size_t)c * cap;
            for (int j = lane; j < nc; j += 32) fn(src[j]);
        }
    }
    // keys i0 .. i0+KPT-1 (~0 past V): one search, then walk the chunks
    template <int KPT>
    __device__ __forceinline__ void load_run(int i0, int V, unsigned long long (&out)[KPT]) const
    {
        int lo = 0, hi = nch;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (cpref[mid] <= i0) lo = mid; else hi = mid;
        }
#pragma unroll
        for (int q = 0; q < KPT; q++) {
            const int i = i0 + q;
            if (i < V) {
                while (lo + 1 < nch && cpref[lo + 1] <= i) lo++;
                out[q] = base[(size_t)lo * cap + (i - cpref[lo])];
            } else {
                out[q] = ~0ull;
            }
        }
    }
};

// ---- top-K selection -----------------------------------------------------------------
// 1. stage: the level's candidate keys (slot order) into shared memory, coalesced.
// 2. threshold: one histogram pass over 4096 linear buckets of the score bits gives the
//    bucket T holding rank R; every key of buckets <= T is kept (R plus the rest of T).
//    If that set is too large, MSD radix passes over the 64-bit keys find the R-th key
//    exactly instead.
// 3. compact the kept keys, stably (slot order preserved), with one block scan.
// 4. stable LSD radix sort by the score bits only -- the input is in slot order, so this
//    is exactly the reference's stable (score, slot) order -- and emit the first R.
constexpr int kNB = 4096;

__device__ __forceinline__ unsigned long long umin64(unsigned long long a, unsigned long long b) { return a < b ? a : b; }
__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) { return a < b ? b : a; }

__device__ __forceinline__ int pow2ceil(int c)
{
    return c <= 1 ? 1 : 1 << (32 - __clz(c - 1));
}

__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gmem_src)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem_src) : "memory");
}

// 1. all V keys, logical order, into stg (warp per chunk, consecutive lanes -> consecutive keys)
static __device__ void stage_keys(const KeySrc& ks, unsigned long long* stg)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int c = warp; c < ks.nch; c += nwarps) {
        const int c0 = ks.cpref[c], nc = ks.cpref[c + 1] - c0;
        const unsigned long long* src = ks.base + (size_t)c * ks.cap;
        for (int i = lane; i < nc; i += 32) cp_async8(stg + c0 + i, src + i);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
}

// Bucket of a score (bits) in [smin, smin + 4096 << shift); clamped, so a score outside the
// recorded range cannot index past the counts.
__device__ __forceinline__ uint32_t bucket_of(uint32_t sb, uint32_t smin, int shift)
{
    const uint32_t b = (sb - smin) >> shift;
    return b < (uint32_t)kNB ? b : (uint32_t)(kNB - 1);
}

// 2a. bucket threshold over 4096 linear buckets of the score bits between the level's
// min and max (S.rmin / S.rmax): returns the number of keys in buckets <= T; misc[2] = T,
// misc[4] = shift, misc[1] = smin.
// `each(fn)` calls fn on every key this thread is responsible for.
template <typename ForEach>
static __device__ int bucket_threshold_each(ForEach each, int R, const SelSmem& S)
{
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;
    uint32_t* cnt = S.hist;
    int* misc = S.misc;
    int* wsum = reinterpret_cast<int*>(S.red);
    (void)lane;
    for (int b = tid; b < kNB; b += nthr) cnt[b] = 0;
    if (tid == 0) misc[1] = (int)S.rmin;
    __syncthreads();
    const uint32_t smin = S.rmin, range = S.rmax - S.rmin;
    const int nbits = range ? 32 - __clz(range) : 0;
    const int shift = nbits > 12 ? nbits - 12 : 0;
    each([&](unsigned long long k) { atomicAdd(&cnt[bucket_of((uint32_t)(k >> 32), smin, shift)], 1u); });
    __syncthreads();
    constexpr int BPT = kNB / kSelectThreads;
    uint32_t c4[BPT];
    int sum = 0;
#pragma unroll
    for (int u = 0; u < BPT; u++) { c4[u] = cnt[tid * BPT + u]; sum += (int)c4[u]; }
    int tot;
    int base = block_exclusive_scan(sum, &tot, wsum);
#pragma unroll
    for (int u = 0; u < BPT; u++) {
        if (base < R && R <= base + (int)c4[u]) { misc[2] = tid * BPT + u; misc[3] = base + (int)c4[u]; }
        base += (int)c4[u];
    }
    if (tid == 0) misc[4] = shift;
    __syncthreads();
    return misc[3];
}

template <typename Get>
static __device__ int bucket_threshold(Get get, int V, int R, const SelSmem& S)
{
    const int tid = threadIdx.x, nthr = blockDim.x;
    return bucket_threshold_each([&](auto fn) { for (int i = tid; i < V; i += nthr) fn(get(i)); }, R, S);
}

// 2b. radix threshold: exact R-th key; returns (pmask, prefix) with keep = (k & pmask) <= prefix.
template <typename Get>
static __device__ void radix_threshold(Get get, int V, int R, const SelSmem& S, unsigned long long& pmask_out,
                                unsigned long long& prefix_out)
{
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long pmask = 0ull, prefix = 0ull;
    if (V > R && R > 0) {
        // --- min / max -> highest differing bit ---
        unsigned long long mn = ~0ull, mx = 0ull;
        for (int idx = tid; idx < V; idx += nthr) { unsigned long long k = get(idx); mn = min(mn, k); mx = max(mx, k); }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn = min(mn, __shfl_xor_sync(FULL_MASK, mn, o));
            mx = max(mx, __shfl_xor_sync(FULL_MASK, mx, o));
        }
        if (lane == 0) { S.red[warp] = mn; S.red[32 + warp] = mx; }
        __syncthreads();
        if (tid == 0) {
            unsigned long long a0 = ~0ull, a1 = 0ull;
            for (int w = 0; w < (nthr >> 5); w++) { a0 = min(a0, S.red[w]); a1 = max(a1, S.red[32 + w]); }
            S.red[0] = a0;
            S.red[32] = a1;
        }
        __syncthreads();
        mn = S.red[0];
        mx = S.red[32];
        __syncthreads();
        const int hb = 63 - __clzll((long long)(mn ^ mx));
        pmask = (hb >= 63) ? 0ull : ~((2ull << hb) - 1ull);
        prefix = mn & pmask;
        int shift = hb + 1;
        int rem = R;
        while (shift > 0) {
            const int db = shift < 8 ? shift : 8;
            shift -= db;
            const unsigned dm = (1u << db) - 1u;
            for (int t = tid; t < 16 * 256; t += nthr) S.hist[t] = 0;
            __syncthreads();
            uint32_t* hw = S.hist + (warp & 15) * 256;
            for (int idx = tid; idx < V; idx += nthr) {
                unsigned long long k = get(idx);
                if ((k & pmask) == prefix) atomicAdd(hw + ((unsigned)(k >> shift) & dm), 1u);
            }
            __syncthreads();
            for (int t = tid; t < 256; t += nthr) {
                uint32_t sum = 0;
                for (int w = 0; w < 16; w++) sum += S.hist[w * 256 + t];
                S.tot[t] = sum;
            }
            __syncthreads();
            if (warp == 0) {
                // 8 buckets per lane, lane-ordered
                uint32_t loc[8];
                uint32_t ls = 0;
#pragma unroll
                for (int u = 0; u < 8; u++) { loc[u] = S.tot[lane * 8 + u]; ls += loc[u]; }
                uint32_t inc = ls;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    uint32_t y = __shfl_up_sync(FULL_MASK, inc, o);
                    if (lane >= o) inc += y;
                }
                uint32_t before = inc - ls;
                // the bucket where the running count first reaches rem
                if ((int)before < rem && rem <= (int)inc) {
                    uint32_t cum = before;
                    for (int u = 0; u < 8; u++) {
                        if ((int)(cum + loc[u]) >= rem) {
                            S.misc[0] = lane * 8 + u;
                            S.misc[1] = (int)cum;
                            S.misc[2] = (int)loc[u];
                            break;
                        }
                        cum += loc[u];
                    }
                }
            }
            __syncthreads();
            const int dg = S.misc[0], cum = S.misc[1], cnt = S.misc[2];
            rem -= cum;
            prefix |= (unsigned long long)dg << shift;
            pmask |= (unsigned long long)dm << shift;
            __syncthreads();
            if (cnt == rem) break;
        }
    }

    pmask_out = pmask;
    prefix_out = prefix;
    __syncthreads();
}

// 3. stable compaction: each warp owns a contiguous range of the input, counted then
// written tile by tile with ballots; one block scan over the 32 warp totals.
template <typename Get, typename Keep>
static __device__ int compact_stable(Get get, int V, Keep keep, unsigned long long* dst, int cap, const SelSmem& S)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    int* wtot = S.misc + 16;   // [32]
    const int L = ((V + nwarps - 1) / nwarps + 31) & ~31;
    const int lo = warp * L, hi = min(V, lo + L);
    int c = 0;
    for (int i0 = lo; i0 < hi; i0 += 32) {
        const int i = i0 + lane;
        c += __popc(__ballot_sync(FULL_MASK, i < hi && keep(get(i))));
    }
    if (lane == 0) wtot[warp] = c;
    __syncthreads();
    if (warp == 0) {
        const int v = lane < nwarps ? wtot[lane] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= o) x += y;
        }
        if (lane < nwarps) wtot[lane] = x - v;
        if (lane == 31) S.misc[60] = x;
    }
    __syncthreads();
    int pos = wtot[warp];
    const unsigned lt = (1u << lane) - 1u;
    for (int i0 = lo; i0 < hi; i0 += 32) {
        const int i = i0 + lane;
        unsigned long long k = 0;
        bool f = false;
        if (i < hi) { k = get(i); f = keep(k); }
        const unsigned b = __ballot_sync(FULL_MASK, f);
        if (f && pos + __popc(b & lt) < cap) dst[pos + __popc(b & lt)] = k;
        pos += __popc(b);
    }
    const int total = S.misc[60];
    __syncthreads();
    return total;
}

// 3b. dense ranks.  The survivors of a level carry few distinct scores (~150-250 at
// 50x20, K=4096: scores are cmax/ns plus a noise of a few ulps) spread over ~2^20 ulps,
// so their score bits are replaced by the rank of the score among the distinct survivor
// scores -- strictly monotone, so the (score, slot) order is unchanged -- and the radix
// sort below needs one 8-bit pass (two above 256 distinct scores) instead of three.
// Distinct scores are marked in a bitmap over the occupied buckets <= T (2^shift bits
// each); a popcount prefix over the bitmap words gives each score's rank.  Returns false,
// keys untouched, when the bitmap would not fit.  Uses the staging area above the first
// kLsdMax keys (the radix sort's second buffer) for the bitmap, its prefix and the
// occupied-bucket index.
constexpr int kDenseOccOff = kLsdMax;              // u16[kNB] occupied-bucket index
constexpr int kDenseBmOff = kLsdMax + kNB / 4;     // u32[kDenseWords] bitmap, then its prefix
constexpr int kDenseWords = 4096;
static_assert(kDenseBmOff + kDenseWords <= kStageKeys, "dense-rank tables exceed the staging area");

// Dense-rank tables over the occupied buckets <= T: a bitmap of the distinct scores
// (2^shift bits per occupied bucket) and the popcount prefix of its words.
struct DenseTables {
    uint16_t* occ;   // [kNB] occupied-bucket index
    uint32_t* bm;    // [kDenseWords] bitmap
    uint32_t* wp;    // [kDenseWords] exclusive popcount prefix of bm
    int W;           // bitmap words per occupied bucket
    int shift;
    uint32_t smin, omask;
    __device__ __forceinline__ int word_of(uint32_t score_bits, uint32_t& bit) const
    {
        const uint32_t dd = score_bits - smin;
        const uint32_t off = dd & omask;
        bit = off & 31u;
        return (int)occ[dd >> shift] * W + (int)(off >> 5);
    }
    // rank of a score among the distinct scores marked in the bitmap
    __device__ __forceinline__ uint32_t rank_of(uint32_t score_bits) const
    {
        uint32_t bit;
        const int w = word_of(score_bits, bit);
        return wp[w] + (uint32_t)__popc(bm[w] & ((1u << bit) - 1u));
    }
};

// Builds the tables for the keys `each` visits whose bucket is <= T (`each(fn)` calls fn on
// every key this thread is responsible for).  Returns the number of distinct scores, or -1
// (tables unusable) when the bitmap would exceed kDenseWords words.
template <typename ForEach>
static __device__ int dense_build(ForEach each, int T, int shift, uint32_t smin, const SelSmem& S, DenseTables& D)
{
    const int tid = threadIdx.x, nthr = blockDim.x;
    D.W = shift > 5 ? 1 << (shift - 5) : 1;
    D.shift = shift;
    D.smin = smin;
    D.omask = (1u << shift) - 1u;
    int* wsum = reinterpret_cast<int*>(S.red);
    constexpr int BPT = kNB / kSelectThreads;
    int f[BPT], sum = 0;
#pragma unroll
    for (int u = 0; u < BPT; u++) {
        const int b = tid * BPT + u;
        f[u] = (b <= T && S.hist[b] != 0u) ? 1 : 0;
        sum += f[u];
    }
    int O;
    int base = block_exclusive_scan(sum, &O, wsum);
#pragma unroll
    for (int u = 0; u < BPT; u++) {
        D.occ[tid * BPT + u] = (uint16_t)base;
        base += f[u];
    }
    const int nw = O * D.W;
    if (nw > kDenseWords) return -1;   // O is the same in every thread
    for (int w = tid; w < nw; w += nthr) D.bm[w] = 0u;
    __syncthreads();
    const uint32_t lim = ((uint32_t)T + 1u) << shift;
    each([&](unsigned long long k) {
        const uint32_t sb = (uint32_t)(k >> 32);
        if (sb - smin < lim) {
            uint32_t bit;
            const int w = D.word_of(sb, bit);
            atomicOr(&D.bm[w], 1u << bit);
        }
    });
    __syncthreads();
    const int per = (nw + nthr - 1) / nthr;
    int c = 0;
    for (int k = 0; k < per; k++) {
        const int w = tid * per + k;
        if (w < nw) c += __popc(D.bm[w]);
    }
    int Dn;
    int pre = block_exclusive_scan(c, &Dn, wsum);
    for (int k = 0; k < per; k++) {
        const int w = tid * per + k;
        if (w < nw) {
            D.wp[w] = (uint32_t)pre;
            pre += __popc(D.bm[w]);
        }
    }
    __syncthreads();
    return Dn;
}

// 4'. One stable counting pass over the compacted survivors by their dense score rank (at
// most 256 distinct), scattered straight into `sel`.  The rank of each element comes from
// the dense tables as it is loaded: no min/max pass, no second buffer, no emit pass.
// Elements p = warp*32*E + e*32 + lane (warps own contiguous runs, E = ceil(count/1024))
// are ranked in element order against per-warp 16-bit digit counters with bit-ballot peer
// masks; each element's (rank, offset) goes back into its own A slot (bits 63..48 rank,
// 47..32 offset) so the loops stay rolled; a digit-major prefix over (digit, warp) gives
// the positions.
static __device__ void dense_sort_emit(unsigned long long* A, int count, int R, const DenseTables& D, uint32_t* sel,
                                       const SelSmem& S)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int E = (count + kSelectThreads - 1) / kSelectThreads;
    uint16_t* wh = reinterpret_cast<uint16_t*>(S.hist);   // [32][256]
    int* dtot = reinterpret_cast<int*>(S.tot);           // [256]
    for (int i = tid; i < 32 * 256 / 2; i += blockDim.x) S.hist[i] = 0u;
    __syncthreads();
#pragma unroll 1
    for (int e = 0; e < E; e++) {
        const int p = warp * 32 * E + e * 32 + lane;
        const bool valid = p < count;
        const unsigned long long x = valid ? A[p] : 0ull;
        const int d = valid ? (int)D.rank_of((uint32_t)(x >> 32)) : 0;
        unsigned grp = __ballot_sync(FULL_MASK, valid);
#pragma unroll
        for (int bit = 0; bit < 8; bit++) {
            const unsigned bb = __ballot_sync(FULL_MASK, (d >> bit) & 1);
            grp &= ((d >> bit) & 1) ? bb : ~bb;
        }
        const int r_in = __popc(grp & lt);
        int b = 0;
        if (valid) b = wh[warp * 256 + d];
        __syncwarp();
        if (valid && r_in == 0) wh[warp * 256 + d] = (uint16_t)(b + __popc(grp));
        __syncwarp();
        if (valid)
            A[p] = ((unsigned long long)d << 48) | ((unsigned long long)(b + r_in) << 32) | (x & 0xFFFFFFFFull);
    }
    __syncthreads();
    if (tid < 256) {
        int run = 0;
        for (int w = 0; w < 32; w++) {
            const int t = wh[w * 256 + tid];
            wh[w * 256 + tid] = (uint16_t)run;
            run += t;
        }
        dtot[tid] = run;
    }
    __syncthreads();
    if (warp == 0) {
        int v8[8], sum = 0;
#pragma unroll
        for (int u = 0; u < 8; u++) { v8[u] = dtot[lane * 8 + u]; sum += v8[u]; }
        int xx = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, xx, o);
            if (lane >= o) xx += y;
        }
        int run = xx - sum;
#pragma unroll
        for (int u = 0; u < 8; u++) { dtot[lane * 8 + u] = run; run += v8[u]; }
    }
    __syncthreads();
#pragma unroll 1
    for (int e = 0; e < E; e++) {
        const int p = warp * 32 * E + e * 32 + lane;
        if (p < count) {
            const unsigned long long x = A[p];
            const int dg = (int)(x >> 48);
            const int pos = dtot[dg] + (int)wh[warp * 256 + dg] + (int)((x >> 32) & 0xFFFFull);
            if (pos < R) sel[pos] = (uint32_t)(x & 0xFFFFFFFFull);
        }
    }
}

// 4. stable LSD radix sort of `count` (<= kLsdMax) keys by their score bits, first R out.
// Elements p = warp*32*E + e*32 + lane are ranked in element order against per-warp
// 16-bit digit counters with bit-ballot peer masks (no atomics); a digit-major prefix over
// (digit, warp) gives the scatter base.
template <int E>
static __device__ unsigned long long* lsd_sort(unsigned long long* A, unsigned long long* B, int count, const SelSmem& S)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    uint16_t* wh = reinterpret_cast<uint16_t*>(S.hist);   // [32][256]
    int* dtot = reinterpret_cast<int*>(S.tot);
    int* misc = S.misc;
    uint32_t mn = 0xFFFFFFFFu, mx = 0u;
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int p = warp * 32 * E + e * 32 + lane;
        if (p < count) { const uint32_t sb = (uint32_t)(A[p] >> 32); mn = min(mn, sb); mx = max(mx, sb); }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(FULL_MASK, mn, o));
        mx = max(mx, __shfl_xor_sync(FULL_MASK, mx, o));
    }
    if (tid == 0) { misc[8] = 0; misc[9] = (int)0xFFFFFFFFu; }
    __syncthreads();
    if (lane == 0) {
        atomicMax(reinterpret_cast<unsigned*>(&misc[8]), mx);
        atomicMin(reinterpret_cast<unsigned*>(&misc[9]), mn);
    }
    __syncthreads();
    const uint32_t smin = (uint32_t)misc[9];
    const uint32_t range = (uint32_t)misc[8] - smin;
    const int nbits = (count > 0 && range) ? 32 - __clz(range) : 0;
    for (int sh = 0; sh < nbits; sh += 8) {
        uint32_t* wh32 = S.hist;
        for (int i = tid; i < 32 * 256 / 2; i += blockDim.x) wh32[i] = 0;
        __syncthreads();
        unsigned long long x[E];
        int dg[E], off[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int p = warp * 32 * E + e * 32 + lane;
            const bool valid = p < count;
            x[e] = valid ? A[p] : 0ull;
            const int d = valid ? (int)(((((uint32_t)(x[e] >> 32)) - smin) >> sh) & 255u) : 0;
            // lanes holding the same digit: intersect the 8 bit-ballots
            unsigned grp = __ballot_sync(FULL_MASK, valid);
#pragma unroll
            for (int bit = 0; bit < 8; bit++) {
                const unsigned bb = __ballot_sync(FULL_MASK, (d >> bit) & 1);
                grp &= ((d >> bit) & 1) ? bb : ~bb;
            }
            const int r_in = __popc(grp & lt);
            int b = 0;
            if (valid) b = wh[warp * 256 + d];
            __syncwarp();
            if (valid && r_in == 0) wh[warp * 256 + d] = (uint16_t)(b + __popc(grp));
            __syncwarp();
            dg[e] = d;
            off[e] = b + r_in;
        }
        __syncthreads();
        // per digit: exclusive prefix over the 32 warps (thread d walks the warps; the
        // [warp][256] layout makes consecutive threads read consecutive counters)
        if (tid < 256) {
            int run = 0;
            for (int w = 0; w < 32; w++) {
                const int t = wh[w * 256 + tid];
                wh[w * 256 + tid] = (uint16_t)run;
                run += t;
            }
            dtot[tid] = run;
        }
        __syncthreads();
        if (warp == 0) {
            int v8[8], sum = 0;
#pragma unroll
            for (int u = 0; u < 8; u++) { v8[u] = dtot[lane * 8 + u]; sum += v8[u]; }
            int xx = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(FULL_MASK, xx, o);
                if (lane >= o) xx += y;
            }
            int run = xx - sum;
#pragma unroll
            for (int u = 0; u < 8; u++) { dtot[lane * 8 + u] = run; run += v8[u]; }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int p = warp * 32 * E + e * 32 + lane;
            if (p < count) B[dtot[dg[e]] + (int)wh[warp * 256 + dg[e]] + off[e]] = x[e];
        }
        __syncthreads();
        unsigned long long* t = A;
        A = B;
        B = t;
    }
    return A;
}

template <int E>
static __device__ void lsd_sort_emit(unsigned long long* A, unsigned long long* B, int count, int R, uint32_t* sel,
                              const SelSmem& S)
{
    const unsigned long long* out = lsd_sort<E>(A, B, count, S);
    for (int i = threadIdx.x; i < R; i += blockDim.x) sel[i] = (uint32_t)(out[i] & 0xFFFFFFFFull);
}

// in-thread compare-exchange stage of distance J (< E) on the blocked layout i = t*E + e
template <int E, int J>
__device__ __forceinline__ void bitonic_in_thread(unsigned long long (&x)[E], int t, int k)
{
#pragma unroll
    for (int e = 0; e < E; e++) {
        if ((e & J) == 0) {
            const bool up = ((t * E + e) & k) == 0;
            const unsigned long long a = x[e], b = x[e + J];
            if ((a > b) == up) { x[e] = b; x[e + J] = a; }
        }
    }
}

// Ascending bitonic sort of N = 1024*E keys, E per thread (thread t holds positions
// t*E .. t*E+E-1); xs is a shared exchange buffer of N keys, used striped (e*1024 + t) so
// cross-warp stages are bank-conflict free.
template <int E>
static __device__ void block_bitonic_reg(unsigned long long (&x)[E], unsigned long long* xs)
{
    // the longest in-thread distance below is 16: at 64 keys per thread padding ends up among the keys
    static_assert(E <= 32, "block_bitonic_reg sorts at most 32 keys per thread");
    const int t = threadIdx.x, lane = t & 31;
    const int N = E * kSelectThreads;
    for (int k = 2; k <= N; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j < E) {
                if (j == 1) bitonic_in_thread<E, 1>(x, t, k);
                else if (j == 2) bitonic_in_thread<E, (E > 2 ? 2 : 1)>(x, t, k);
                else if (j == 4) bitonic_in_thread<E, (E > 4 ? 4 : 1)>(x, t, k);
                else if (j == 8) bitonic_in_thread<E, (E > 8 ? 8 : 1)>(x, t, k);
                else bitonic_in_thread<E, (E > 16 ? 16 : 1)>(x, t, k);
            } else if (j < 32 * E) {
                const int lj = j / E;
                const bool low = (lane & lj) == 0;
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const bool up = ((t * E + e) & k) == 0;
                    const unsigned long long y = __shfl_xor_sync(FULL_MASK, x[e], lj);
                    x[e] = (low == up) ? umin64(x[e], y) : umax64(x[e], y);
                }
            } else {
                const int tj = j / E;
#pragma unroll
                for (int e = 0; e < E; e++) xs[e * kSelectThreads + t] = x[e];
                __syncthreads();
                const bool low = (t & tj) == 0;
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const bool up = ((t * E + e) & k) == 0;
                    const unsigned long long y = xs[e * kSelectThreads + (t ^ tj)];
                    x[e] = (low == up) ? umin64(x[e], y) : umax64(x[e], y);
                }
                __syncthreads();
            }
        }
    }
}

template <int E>
static __device__ void sort_emit_e(unsigned long long* sbuf, int count, int R, uint32_t* sel)
{
    const int t = threadIdx.x;
    unsigned long long x[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int idx = e * kSelectThreads + t;   // any bijection works for unsorted input
        x[e] = idx < count ? sbuf[idx] : ~0ull;
    }
    __syncthreads();
    block_bitonic_reg<E>(x, sbuf);
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int i = t * E + e;
        if (i < R) sel[i] = (uint32_t)(x[e] & 0xFFFFFFFFull);
    }
}

// Sort the `count` keys in sbuf and write the first R slots to sel (count <= 16384).
static __device__ void sort_and_emit(unsigned long long* sbuf, int count, int R, uint32_t* sel)
{
    const int N = pow2ceil(count);
    if (N <= kSelectThreads) sort_emit_e<1>(sbuf, count, R, sel);
    else if (N <= 2 * kSelectThreads) sort_emit_e<2>(sbuf, count, R, sel);
    else if (N <= 4 * kSelectThreads) sort_emit_e<4>(sbuf, count, R, sel);
    else if (N <= 8 * kSelectThreads) sort_emit_e<8>(sbuf, count, R, sel);
    else if (N <= 16 * kSelectThreads) sort_emit_e<16>(sbuf, count, R, sel);
    else if constexpr (kSelectThreads * 16 < kStageKeys) sort_emit_e<kStageKeys / kSelectThreads>(sbuf, count, R, sel);
}

// Fillers (v1 / v2 only): when fewer than min(P*n, K) children were scored, the
// reference's stable sort keeps the lowest-numbered unscored slots next, in slot order.
static __device__ void select_fillers(const SegDesc& d, const StepArgs& a, int P, int R, int keff, uint32_t* sel,
                               uint8_t* smem)
{
    if (keff <= R) return;
    int* wsum = reinterpret_cast<int*>(smem);
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int n = d.n;
    const int F = keff - R;
    const int W = d.words;
    const uint32_t* mk = a.masks + d.mask_off;
    int base = 0;
    for (int c0 = 0; c0 < P && base < F; c0 += nthr) {
        const int c = c0 + tid;
        int f = 0;
        if (c < P) {
            int pc = 0;
            for (int w = 0; w < W; w++) pc += __popc(mk[(int64_t)c * W + w]);
            f = n - pc;
        }
        int tot;
        const int off = block_exclusive_scan(f, &tot, wsum);
        if (c < P && base + off < F) {
            int out = R + base + off;
            const int lim = F - base - off;
            int got = 0;
            for (int b = 0; b < n && got < lim && got < f; b++) {
                uint32_t word = mk[(int64_t)c * W + (b >> 5)];
                if (!((word >> (b & 31)) & 1u)) {
                    sel[out + got] = kFillerFlag | (uint32_t)(c * n + b);
                    got++;
                }
            }
        }
        base += tot;
    }
}

// ---- large levels: more candidate keys than the staging area holds (V > kStageKeys) or
// more survivors than the 64-bit radix buffer (K > kLsdMax).  The keys stay in their chunk
// regions in global memory (L2-resident); survivors are compacted as 32-bit words
// (dense rank << 21 | slot) into the two 96 KB halves of the A/stg area, and sorted by the
// rank bits with a stable 8-bit radix pass that needs no per-element registers. ----
constexpr int kBigCap = kLsdMax + kStageKeys;  // u32 survivors per half of the A/stg area
constexpr int kSlotBits = 21;                                         // slot < K * n <= 2^21
constexpr int kBigMaxDistinct = 1 << (32 - kSlotBits);                // ranks in the top 11 bits
static_assert(2 * kBigCap * 4 == (kLsdMax + kStageKeys) * 8, "two kBigCap u32 halves fill the A/stg area");
static_assert(kNB / 2 + 2 * kDenseWords <= kBigCap, "dense tables must fit the second half");
static_assert((long long)kMaxBeam * kMaxJobs <= (1LL << kSlotBits), "slots must fit 21 bits");

// Stable compaction of the keys of buckets <= T (score bits - smin < lim), in slot order,
// each written as (dense rank << kSlotBits) | slot.  Warps own contiguous runs of chunks:
// one counting sweep, a scan of the warp totals, one writing sweep.
static __device__ int compact_ranked(const KeySrc& ks, uint32_t lim, uint32_t smin, const DenseTables& D, uint32_t* out,
                              int cap, const SelSmem& S)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int* wtot = S.misc + 16;   // [32]
    const int cpw = (ks.nch + nwarps - 1) / nwarps;
    const int c_lo = min(ks.nch, warp * cpw), c_hi = min(ks.nch, c_lo + cpw);
    int c = 0;
    for (int ch = c_lo; ch < c_hi; ch++) {
        const int nc = ks.cpref[ch + 1] - ks.cpref[ch];
        const unsigned long long* src = ks.base + (size_t)ch * ks.cap;
        for (int j0 = 0; j0 < nc; j0 += 32) {
            const int j = j0 + lane;
            const bool f = j < nc && ((uint32_t)(src[j] >> 32) - smin) < lim;
            c += __popc(__ballot_sync(FULL_MASK, f));
        }
    }
    if (lane == 0) wtot[warp] = c;
    __syncthreads();
    if (warp == 0) {
        const int v = lane < nwarps ? wtot[lane] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= o) x += y;
        }
        if (lane < nwarps) wtot[lane] = x - v;
        if (lane == 31) S.misc[60] = x;
    }
    __syncthreads();
    int pos = wtot[warp];
    const unsigned lt = (1u << lane) - 1u;
    for (int ch = c_lo; ch < c_hi; ch++) {
        const int nc = ks.cpref[ch + 1] - ks.cpref[ch];
        const unsigned long long* src = ks.base + (size_t)ch * ks.cap;
        for (int j0 = 0; j0 < nc; j0 += 32) {
            const int j = j0 + lane;
            unsigned long long k = 0;
            bool f = false;
            if (j < nc) {
                k = src[j];
                f = ((uint32_t)(k >> 32) - smin) < lim;
            }
            const unsigned b = __ballot_sync(FULL_MASK, f);
            const int at = pos + __popc(b & lt);
            if (f && at < cap) out[at] = (D.rank_of((uint32_t)(k >> 32)) << kSlotBits) | (uint32_t)(k & 0xFFFFFFFFull);
            pos += __popc(b);
        }
    }
    const int total = S.misc[60];
    __syncthreads();
    return total;
}

// One stable counting pass of src[0..count) into dst by the 8-bit digit at bit `sh`.
// Warps own contiguous element runs; a digit's rank inside a 32-element tile comes from the
// peers' bit ballots, across tiles and warps from per-warp 16-bit counters.  The tiles are
// walked twice (count, then scatter) so no element state is held across the prefix.
static __device__ void radix_pass32(const uint32_t* src, uint32_t* dst, int count, int sh, const SelSmem& S)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    uint16_t* wh = reinterpret_cast<uint16_t*>(S.hist);   // [32][256]
    int* dtot = reinterpret_cast<int*>(S.tot);           // [256]
    const unsigned lt = (1u << lane) - 1u;
    const int per = ((count + nwarps - 1) / nwarps + 31) & ~31;
    const int lo = min(count, warp * per), hi = min(count, lo + per);
    for (int i = tid; i < 32 * 256 / 2; i += blockDim.x) S.hist[i] = 0u;
    __syncthreads();
    auto peers = [&](bool valid, int dg) {
        unsigned grp = __ballot_sync(FULL_MASK, valid);
#pragma unroll
        for (int bit = 0; bit < 8; bit++) {
            const unsigned bb = __ballot_sync(FULL_MASK, (dg >> bit) & 1);
            grp &= ((dg >> bit) & 1) ? bb : ~bb;
        }
        return grp;
    };
    for (int i0 = lo; i0 < hi; i0 += 32) {
        const int i = i0 + lane;
        const bool valid = i < hi;
        const int dg = valid ? (int)((src[i] >> sh) & 255u) : 0;
        const unsigned grp = peers(valid, dg);
        if (valid && (grp & lt) == 0u) wh[warp * 256 + dg] = (uint16_t)(wh[warp * 256 + dg] + __popc(grp));
        __syncwarp();
    }
    __syncthreads();
    if (tid < 256) {
        int run = 0;
        for (int w = 0; w < nwarps; w++) {
            const int t = wh[w * 256 + tid];
            wh[w * 256 + tid] = (uint16_t)run;
            run += t;
        }
        dtot[tid] = run;
    }
    __syncthreads();
    if (warp == 0) {
        int v8[8], sum = 0;
#pragma unroll
        for (int u = 0; u < 8; u++) { v8[u] = dtot[lane * 8 + u]; sum += v8[u]; }
        int xx = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, xx, o);
            if (lane >= o) xx += y;
        }
        int run = xx - sum;
#pragma unroll
        for (int u = 0; u < 8; u++) { dtot[lane * 8 + u] = run; run += v8[u]; }
    }
    __syncthreads();
    for (int i0 = lo; i0 < hi; i0 += 32) {
        const int i = i0 + lane;
        const bool valid = i < hi;
        const uint32_t x = valid ? src[i] : 0u;
        const int dg = (int)((x >> sh) & 255u);
        const unsigned grp = peers(valid, dg);
        if (valid) dst[dtot[dg] + (int)wh[warp * 256 + dg] + __popc(grp & lt)] = x;
        __syncwarp();
        if (valid && (grp & lt) == 0u) wh[warp * 256 + dg] = (uint16_t)(wh[warp * 256 + dg] + __popc(grp));
        __syncwarp();
    }
    __syncthreads();
}

// The whole selection of a large level; false (nothing written) when it does not fit
// these buffers -- then the general path runs.
static __device__ bool select_large(SegState& st, int R, const KeySrc& ks, uint32_t* sel, const SelSmem& S)
{
    const int tid = threadIdx.x;
    auto each = [&](auto fn) { ks.each_key(fn); };
    const int count0 = bucket_threshold_each(each, R, S);
    const int T = S.misc[2], shift = S.misc[4];
    const uint32_t smin = (uint32_t)S.misc[1];
    __syncthreads();
    if (count0 > kBigCap) return false;
    uint32_t* buf1 = reinterpret_cast<uint32_t*>(S.A);
    uint32_t* buf2 = buf1 + kBigCap;
    DenseTables D;
    D.occ = reinterpret_cast<uint16_t*>(buf2);
    D.bm = buf2 + kNB / 2;
    D.wp = D.bm + kDenseWords;
    const int nd = dense_build(each, T, shift, smin, S, D);
    if (nd < 0 || nd > kBigMaxDistinct) return false;
    const uint32_t lim = ((uint32_t)T + 1u) << shift;
    int count = compact_ranked(ks, lim, smin, D, buf1, kBigCap, S);
    if (count != count0 || count < R) {
        if (tid == 0) atomicOr(&st.status, kStatusBadSelect);
        count = min(count, kBigCap);
    }
    const int nbits = nd > 1 ? 32 - __clz(nd - 1) : 0;
    uint32_t* src = buf1;
    uint32_t* dst = buf2;
    for (int sh = kSlotBits; sh < kSlotBits + nbits; sh += 8) {
        radix_pass32(src, dst, count, sh, S);
        uint32_t* t = src;
        src = dst;
        dst = t;
    }
    const int RR = R < count ? R : count;
    for (int i = tid; i < RR; i += blockDim.x) sel[i] = src[i] & ((1u << kSlotBits) - 1u);
    __syncthreads();
    return true;
}

// ---- direct staged selection: the common case of a level that fits the staging area.
// After the bucket threshold, the distinct scores of the keys of buckets <= T get dense
// ranks (at most 256 of them); one stable counting pass over the staged keys, in slot
// order, then gives every kept key its final position in (score, slot) order -- the
// reference's stable sort order -- and survivors below R go straight to `sel`.  Warps own
// contiguous runs of the staged keys: pass 1 walks each run tile by tile, ranking a key
// against its tile peers (bit ballots of the digit) and the warp's running per-digit
// counters, and writes (digit << 16 | offset) over the key's score bits; after a
// digit-major prefix over (digit, warp), pass 2 scatters in parallel.  No compaction
// buffer, no sort passes.  Returns false -- staged keys untouched, nothing written -- when
// the dense tables do not fit or there are more than 256 distinct scores; the general
// path then runs.  Taken for levels of up to kDirectMaxKeys keys. ----
constexpr int kDirectMaxDistinct = 256;
// Largest level (candidate keys) the direct path takes: beyond it, compacting the keys
// first and sorting the survivors is faster (a GB300 sweep over 18 shapes: the direct
// path wins 5-10 % up to ~4 K keys, loses from ~6 K on).
constexpr int kDirectMaxKeys = 4096;

static __device__ bool select_direct(unsigned long long* stg, int V, int R, int T, int shift, uint32_t smin, uint32_t* sel,
                              const SelSmem& S)
{
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    DenseTables D;
    D.occ = reinterpret_cast<uint16_t*>(S.A);
    D.bm = reinterpret_cast<uint32_t*>(S.A + kNB / 4);
    D.wp = D.bm + kDenseWords;
    auto each = [&](auto fn) {
        for (int i = tid; i < V; i += nthr) fn(stg[i]);
    };
    const int nd = dense_build(each, T, shift, smin, S, D);   // reads S.hist, ends synchronised
    if (nd < 0 || nd > kDirectMaxDistinct) return false;      // the same in every thread
    uint16_t* wh = reinterpret_cast<uint16_t*>(S.hist);       // [32][256] per-warp digit counters
    int* dtot = reinterpret_cast<int*>(S.tot);                // [256]
    for (int i = tid; i < 32 * 256 / 2; i += nthr) S.hist[i] = 0u;
    __syncthreads();
    const uint32_t lim = ((uint32_t)T + 1u) << shift;          // bucket <= T
    const unsigned lt = (1u << lane) - 1u;
    const int per = ((V + nwarps - 1) / nwarps + 31) & ~31;   // <= 512: offsets fit 16 bits
    const int lo = min(V, warp * per), hi = min(V, lo + per);
    // two tiles per step: their digits and peer sets are independent; only the counter
    // updates run in tile order
    auto tile = [&](int i, unsigned long long& k, int& dg, unsigned& grp) {
        k = ~0ull;
        dg = 0;
        bool kept = false;
        if (i < hi) {
            k = stg[i];
            const uint32_t sb = (uint32_t)(k >> 32);
            kept = (sb - smin) < lim;
            if (kept) dg = (int)D.rank_of(sb);
        }
        grp = __ballot_sync(FULL_MASK, kept);
#pragma unroll
        for (int bit = 0; bit < 8; bit++) {
            const unsigned bb = __ballot_sync(FULL_MASK, (dg >> bit) & 1);
            grp &= ((dg >> bit) & 1) ? bb : ~bb;
        }
        if (!kept) grp = 0u;
    };
    auto count = [&](int dg, unsigned grp) {
        int base = 0;
        if (grp) base = wh[warp * 256 + dg];
        __syncwarp();
        if (grp && (grp & lt) == 0u) wh[warp * 256 + dg] = (uint16_t)(base + __popc(grp));
        __syncwarp();
        return base + __popc(grp & lt);
    };
    for (int i0 = lo; i0 < hi; i0 += 64) {
        const int ia = i0 + lane, ib = i0 + 32 + lane;
        unsigned long long ka, kb;
        int da, db;
        unsigned ga, gb;
        tile(ia, ka, da, ga);
        tile(ib, kb, db, gb);
        const int oa = count(da, ga);
        const int ob = count(db, gb);
        if (ia < hi) stg[ia] = ga ? ((unsigned long long)(((uint32_t)da << 16) | (uint32_t)oa) << 32) | (ka & 0xFFFFFFFFull) : ~0ull;
        if (ib < hi) stg[ib] = gb ? ((unsigned long long)(((uint32_t)db << 16) | (uint32_t)ob) << 32) | (kb & 0xFFFFFFFFull) : ~0ull;
    }
    __syncthreads();
    // per digit: exclusive prefix over the warps, then over the digits
    if (tid < 256) {
        int run = 0;
        for (int w = 0; w < nwarps; w++) {
            const int t = wh[w * 256 + tid];
            wh[w * 256 + tid] = (uint16_t)run;
            run += t;
        }
        dtot[tid] = run;
    }
    __syncthreads();
    if (warp == 0) {
        int v8[8], sum = 0;
#pragma unroll
        for (int u = 0; u < 8; u++) { v8[u] = dtot[lane * 8 + u]; sum += v8[u]; }
        int xx = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, xx, o);
            if (lane >= o) xx += y;
        }
        int run = xx - sum;
#pragma unroll
        for (int u = 0; u < 8; u++) { dtot[lane * 8 + u] = run; run += v8[u]; }
    }
    __syncthreads();
    for (int i = tid; i < V; i += nthr) {
        const unsigned long long x = stg[i];
        const uint32_t h = (uint32_t)(x >> 32);
        if (h != 0xFFFFFFFFu) {
            const int dg = (int)(h >> 16);
            const int pos = dtot[dg] + (int)wh[(i / per) * 256 + dg] + (int)(h & 0xFFFFu);
            if (pos < R) sel[pos] = (uint32_t)(x & 0xFFFFFFFFull);
        }
    }
    __syncthreads();
    return true;
}

// lsd_sort_emit for any count <= kLsdMax (E = ceil(count / kSelectThreads) elements per thread)
static __device__ void lsd_sort_emit_n(unsigned long long* A, unsigned long long* B, int count, int R, uint32_t* sel,
                                const SelSmem& S)
{
    switch ((count + kSelectThreads - 1) / kSelectThreads) {
    case 0:
    case 1: lsd_sort_emit<1>(A, B, count, R, sel, S); break;
    case 2: lsd_sort_emit<2>(A, B, count, R, sel, S); break;
    case 3: lsd_sort_emit<3>(A, B, count, R, sel, S); break;
    case 4: lsd_sort_emit<4>(A, B, count, R, sel, S); break;
    case 5: lsd_sort_emit<5>(A, B, count, R, sel, S); break;
    case 6: lsd_sort_emit<6>(A, B, count, R, sel, S); break;
    case 7: lsd_sort_emit<7>(A, B, count, R, sel, S); break;
    case 8: lsd_sort_emit<8>(A, B, count, R, sel, S); break;
    default:
        if constexpr (kSelectThreads * 8 < kLsdMax) lsd_sort_emit<kLsdMax / kSelectThreads>(A, B, count, R, sel, S);
        break;
    }
}

// The first R slots of the level in (score, slot) order into sel; V keys, beam width K.
static __device__ void select_sorted(SegState& st, int K, int R, int V, int fz, const KeySrc& ks, uint32_t* sel,
                                     uint8_t* smem, uint32_t rmin, uint32_t rmax)
{
    const int tid = threadIdx.x;
    const SelSmem S = sel_smem(smem, rmin, rmax);
    // fz: route flags (0 = by level size); uniform over the block
    // routes taken, recorded by thread 0 with a reduction that returns nothing
    auto route = [&](uint32_t bit) { if (tid == 0) atomicOr(&st.select_paths, bit); };
    // staged (shared-memory) input when the level fits; larger levels take select_large
    const bool staged = (V <= kStageKeys) && (K <= kLsdMax);
    const bool try_large = (fz & kSelForceLarge) ? true : ((fz & kSelNoLarge) ? false : !staged);
    if (R > 0 && try_large && select_large(st, R, ks, sel, S)) {
        route(kPathLarge);   // done: survivors 0..R-1 written
    } else if (R > 0) {
        if (staged) stage_keys(ks, S.stg);
        const unsigned long long* stg = S.stg;
        auto get_s = [=](int i) { return stg[i]; };
        auto get_g = [=](int i) { return ks(i); };
        int count = staged ? bucket_threshold(get_s, V, R, S) : bucket_threshold(get_g, V, R, S);
        unsigned long long* dst = S.A;
        const int T = S.misc[2], shift = S.misc[4];
        const uint32_t smin = (uint32_t)S.misc[1];
        // survivors = the keys of buckets <= T
        const bool bucketed = count <= kLsdMax && !(fz & kSelForceRadix);
        __syncthreads();
        const bool direct = !(fz & (kSelNoDirect | kSelForceRadix)) && staged && V <= kDirectMaxKeys &&
                            count >= R && select_direct(S.stg, V, R, T, shift, smin, sel, S);
        if (direct) route(kPathDirect);
        if (!direct) {
            if (bucketed) {
                route(kPathBucket);
                const uint32_t lim = ((uint32_t)T + 1u) << shift;  // bucket <= T
                auto keep = [=](unsigned long long k) { return (((uint32_t)(k >> 32)) - smin) < lim; };
                count = staged ? compact_stable(get_s, V, keep, dst, kLsdMax, S)
                               : compact_stable(get_g, V, keep, dst, kLsdMax, S);
            } else {
                route(kPathRadix);
                if (tid == 0) st.select_fallbacks += 1;
                unsigned long long pmask, prefix;
                if (staged) radix_threshold(get_s, V, R, S, pmask, prefix);
                else radix_threshold(get_g, V, R, S, pmask, prefix);
                auto keep = [=](unsigned long long k) { return (k & pmask) <= prefix; };
                if (R > kLsdMax) dst = S.stg;  // only reached unstaged (K > kLsdMax)
                const int cap = (R > kLsdMax) ? kStageKeys : kLsdMax;
                count = staged ? compact_stable(get_s, V, keep, dst, cap, S)
                               : compact_stable(get_g, V, keep, dst, cap, S);
            }
            if (count < R || count > kStageKeys) {
                if (tid == 0) atomicOr(&st.status, kStatusBadSelect);
                count = count > kStageKeys ? kStageKeys : count;
            }
            const int RR = R < count ? R : count;
            if (count <= kLsdMax && !(fz & kSelBitonic)) {
                int nd = -1;
                DenseTables D;
                if (bucketed && !(fz & kSelNoDense)) {
                    // bucket counts are intact on the bucketed path (the radix path reuses them)
                    D.occ = reinterpret_cast<uint16_t*>(S.stg + kDenseOccOff);
                    D.bm = reinterpret_cast<uint32_t*>(S.stg + kDenseBmOff);
                    D.wp = D.bm + kDenseWords;
                    auto each = [&](auto fn) {
                        for (int i = tid; i < count; i += kSelectThreads) fn(dst[i]);
                    };
                    nd = dense_build(each, T, shift, smin, S, D);
                }
                if (nd >= 0 && nd <= 256 && !(fz & kSelRankLsd)) {
                    route(kPathDense);
                    dense_sort_emit(dst, count, RR, D, sel, S);
                } else {
                    if (nd >= 0) {
                        // more distinct scores than one 8-bit pass (or the route is forced):
                        // ranks into the keys, then LSD passes over the rank bits
                        route(kPathRankLsd);
                        for (int i = tid; i < count; i += kSelectThreads) {
                            const unsigned long long k = dst[i];
                            dst[i] = ((unsigned long long)D.rank_of((uint32_t)(k >> 32)) << 32) | (k & 0xFFFFFFFFull);
                        }
                        __syncthreads();
                    } else {
                        route(kPathRawLsd);
                    }
                    lsd_sort_emit_n(dst, S.stg, count, RR, sel, S);
                }
            } else {
                route(kPathBitonic);
                if (dst != S.stg) {
                    // survivors in A (count <= kLsdMax): the bitonic sort works in stg
                    for (int i = tid; i < count; i += kSelectThreads) S.stg[i] = dst[i];
                    __syncthreads();
                }
                sort_and_emit(S.stg, count, RR, sel);
            }
        }
    }
    __syncthreads();
}

static __device__ void select_gpu(const SegDesc& d, SegState& st, const StepArgs& a, int P, int V, const KeySrc& ks,
                                  uint8_t* smem, uint32_t rmin, uint32_t rmax)
{
    const int K = d.K;
    const int total = P * d.n;
    const int keff = (d.mode == MODE_CLEAN) ? (V < K ? V : K) : (total < K ? total : K);
    const int R = V < keff ? V : keff;
    uint32_t* sel = a.sel + d.sel_off;
    select_sorted(st, K, R, V, a.select_force, ks, sel, smem, rmin, rmax);
    select_fillers(d, a, P, R, keff, sel, smem);
    __syncthreads();
    if (threadIdx.x == 0) {
        st.P = keff;
        atomicAdd(reinterpret_cast<unsigned long long*>(&st.materialized), (unsigned long long)keff);
    }
}

}  // namespace bsj
