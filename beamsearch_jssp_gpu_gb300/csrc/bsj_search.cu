// bsj_search.cu -- the resident search: every level of a gpu-mode beam (v1, v2, clean) in one
// kernel, one thread-block cluster per beam.
//
// The level kernels pay, per level, two or three launches and a selection whose phases are
// chains of block-wide steps over all of the level's keys.  Here a cluster of C blocks (one
// block for narrow beams) keeps a beam for the whole search: block r owns the ranks
// [r*Pc, (r+1)*Pc) of every level, its candidate keys stay in its shared memory until the
// survivors among them are handed to the block that owns their position, and the blocks
// meet at two cluster barriers per level:
//
//   step    a group of G lanes per survivor: the parent's snapshot (L2) into shared memory by
//           one bulk copy, the selected operation applied, the child stored by one bulk copy,
//           its candidates found (a byte compare of the ready positions' machines against the
//           pivot machine), then a thread per candidate scores it; keys go to the block's list
//           and are counted into 512 score bins
//   #1      every block reads the others' packed counts -> V, the bin T that holds rank R, each bin's
//           first position; the keys of bins <= T go to the block(s) owning their bin's
//           positions, in any order
//   #2      keys are unique (score, slot) pairs, so a key's position is its bin's first
//           position plus the smaller keys of the bin: counted directly in small bins, within
//           groups of equal scores in larger ones, by a bitonic sort of the block's keys when
//           neither holds
//
// The bins are linear in the score bits over a range predicted from the previous level (the
// map is monotone whatever the range, so a poor prediction costs time, not correctness): a
// level whose largest bin comes out too large, or whose last survivor lies past the range, is
// counted again up to that survivor's bin, with linear bins and then with bins for tied scores
// (TieMap).  Levels whose bins still do not fit the blocks' buffers are dumped to global memory in
// slot order and sorted by the one-block routes of the level kernels.
//
// A snapshot is stored by ready position, not by job: position i holds the finish time of
// its job's last operation, the operation index and its machine, so that a level needs no
// job-indexed lookups and the pivot test reads four positions per word.  (For m = 1 the
// reference reads another job's finish time, which this layout does not keep: those beams
// use the level kernels.)
//
// What bounds it: the level's chain of dependent instructions and barriers (50x20 K=4096 on
// 16 blocks: ~25 K cycles per level), the blocks' differences at barrier #1, and for wide
// shares of long lists the children's stores (an SM writes ~30 bytes per cycle to L2).  512
// threads: 1 024 measured 9.8 against 8.1 us per level at 15x15 K=256 (barriers and issue
// slots), 256 12.0.  Snapshots by bulk copies: 256 of 448 bytes load in 2 350 cycles, by
// 16-byte cp.async in 4 280.  GB300, us per call, level kernels -> this: 15x15 K=256 3 332 ->
// 1 530; v1 20x15 K=1024 6 836 -> 2 950; v1 20x15 K=16384 64 083-75 838 -> 22 300;
// 50x20 K=4096 24 288 -> 12 410, 8 beams 28 182 -> 16 050; 100x20 K=4096 8 beams 66 166 ->
// 40 300.
#include <algorithm>
#include <mutex>
#include <type_traits>

#define BSJ_SELECT_THREADS 512   // = kSearchThreads
#include "bsj_select.cuh"

namespace bsj {

namespace {

constexpr int T = kSearchThreads;
constexpr int NB = kSearchBins;
static_assert(T == kSelectThreads, "the fallback's block routines assume their block size");
static_assert(NB == T, "one bin per thread in the bin scan");

// ops in shared memory: (duration << 8) | last-operation-of-its-job flag | machine
constexpr uint32_t kLastOp = 0x80u;
constexpr uint32_t kNoKey = 0xFFFFFFFFu;   // score bits of a pruned child
// a key: score bits << 32 | bin << kSlotBits | slot.  Bins are monotone in (score, slot), so keys
// order as without them.
constexpr uint32_t kSlotMask = (1u << kSlotBits) - 1u;
static_assert(NB <= 1 << (32 - kSlotBits), "bin and slot share a word");

__device__ __forceinline__ void st_peer32(const void* p, unsigned rank, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_addr(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ void st_peer64(const void* p, unsigned rank, unsigned long long v)
{
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(peer_addr(p, rank)), "l"(v) : "memory");
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- bulk copies of snapshots (global <-> shared memory), completing on a warp's mbarrier
__device__ __forceinline__ void bar_init(unsigned long long* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long* bar, int bytes)
{
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(
                     smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}
// Waits (bounded) for the phase; false when it never completed.  The whole warp calls it.
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, uint32_t phase)
{
    uint32_t done = 0;
    for (uint32_t it = 0; it < (1u << 16) && !done; it++)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done)
                     : "r"(smem_addr(bar)), "r"(phase)
                     : "memory");
    return __all_sync(FULL_MASK, done);
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, int bytes, unsigned long long* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, const void* src, int bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the thread's bulk stores have read their shared-memory source / are complete
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// orders generic-proxy accesses to shared memory with the bulk copies' (async-proxy) ones.  The
// beam buffers in global memory are written and read by bulk copies only (v1, whose child
// slots are written in place, stages them by cp.async), so no fence over global memory is
// needed: it cost ~900 cycles each.
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ int warp_inclusive(int x, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Exclusive prefix of v over the block, and its total; ws: 32 words the caller does not
// reuse before the next block barrier.  One block barrier.
__device__ __forceinline__ int block_exclusive(int v, int* ws, int lane, int warp)
{
    const int x = warp_inclusive(v, lane);
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    const int w = lane < warp ? ws[lane] : 0;
    return __reduce_add_sync(FULL_MASK, w) + x - v;
}
__device__ __forceinline__ int block_exclusive(int v, int* ws, int lane, int warp, int& total)
{
    const int x = warp_inclusive(v, lane);
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    const int w = lane < T / 32 ? ws[lane] : 0;
    total = __reduce_add_sync(FULL_MASK, w);
    return __reduce_add_sync(FULL_MASK, lane < warp ? w : 0) + x - v;
}

// The keys src[0..count) of one block in ascending order, E per thread (position t*E + e);
// those whose global position lies in [w0, w1) to sel.  src is the exchange buffer too.
template <int E>
__device__ void sort_window_e(unsigned long long* src, unsigned long long* xs, int count, int x0, int w0, int w1,
                              uint32_t* sel)
{
    const int t = threadIdx.x;
    unsigned long long x[E];
#pragma unroll
    for (int e = 0; e < E; e++) x[e] = e * T + t < count ? src[e * T + t] : ~0ull;
    __syncthreads();
    block_bitonic_reg<E>(x, xs);
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int i = t * E + e, p = x0 + i;
        if (i < count && p >= w0 && p < w1) sel[p - w0] = (uint32_t)x[e] & kSlotMask;
    }
}

__device__ __noinline__ void sort_window(unsigned long long* src, unsigned long long* xs, int count, int x0, int w0,
                                         int w1, uint32_t* sel)
{
    if (count <= T) sort_window_e<1>(src, xs, count, x0, w0, w1, sel);
    else if (count <= 2 * T) sort_window_e<2>(src, xs, count, x0, w0, w1, sel);
    else if (count <= 4 * T) sort_window_e<4>(src, xs, count, x0, w0, w1, sel);
    else if (count <= 8 * T) sort_window_e<8>(src, xs, count, x0, w0, w1, sel);
    else sort_window_e<16>(src, xs, count, x0, w0, w1, sel);
}
constexpr int kMaxAhead = 4;           // rounds whose parents are loaded at once
constexpr int kSortMax = 16 * T;      // keys sort_window takes
// Where the lines between the ranking routes lie, us per level (20x15 v1 K=1024 | 30x20 K=1000 |
// 37x11 clean K=1500 | 50x20 K=4096 | 20x15 K=16384):
// bins up to kPlainBinMax keys: every key counts the bin's smaller ones.  48: 11.1 | 9.2 | 9.9;
// 96: 10.4 | 8.8 | 9.8; 192: 10.3 | 9.0 | 10.5 (quadratic in the bin; 24 loses 4 % at 50x20).
constexpr int kPlainBinMax = 96;
// groups of equal scores up to kTieMax keys are ranked by counting, larger ones sorted with the
// whole window.  256: 14.0 | 35.2 for the last two; 512: 13.9 | 35.2; 1 024: 13.9 | 34.6.
constexpr int kTieMax = 1024;
// a bin larger than kRecountBin: the level is counted again over a closer score range, which costs
// a pass over the keys and two barriers.  384: 14.0 at 50x20 K=4096; 768 and 1 536: 13.5.
constexpr int kRecountBin = 1536;
constexpr int kMaxRecounts = 3;
// Tie bins follow a level whose ranking was slow for its ties: one that sorted a block's window though
// that spans few bins, or whose largest group of equal scores had more than kTieSlow keys.  ms per
// call, 50x20 K=4096, durations U[1, 99] | x 1 000: 384: 12.28 | 16.8, 192: 12.29 | 15.8, 96: 12.42 |
// 15.8.  They stay for 2, 4, .. kTieStay levels, as long as linear bins fail each time between (a tie
// bin costs a division and a pass over the keys: on every level of U[1, 99], 14.1).  Not below
// kTieBlocks blocks, whose pass takes 4 to 16 times as many keys per thread (levels that fit no bins
// get tie bins there too): 256 mixed searches 2 590 -> 2 905 per second, 150 of 100x20 K=4096 497 ->
// 452 ms; but 20 of 50x20 K=1024 on 4 blocks, durations 1 to 5: 20.3 ms without, 15.3 with.
constexpr int kTieBlocks = 4;
constexpr int kTieSlow = 192;
constexpr int kTieStay = 64;

// What a block keeps of its beam.  In shared memory, not registers: the level loop's live
// state would otherwise spill, and local memory does not fit the L1 the shared memory leaves.
struct BeamConst {
    int n, m, N, K, mode, words, S, bound, off_jr, off_op, off_mc, off_hdr, WL, P, parents;   // parents: entries `sel` may name
    uint32_t seed, paths;
    float inv_m, inv_s16;
    int levels, unit;   // unit: greatest common divisor of the durations
    float slack;        // 0.08 of the mean duration
    long long expanded, slots, mat;
    uint8_t *beam0, *beam1, *slot_base;
    uint32_t* hist;
    unsigned long long* spill;
};

// The level loop's state across the fallback's call (one copy per block: every thread holds the same).
struct LevelState {
    int seg, t, recount_ok, tm, lo, cnt, V, Vb, keff, R, Pn, w0, w1, Tb;
};

// Bins of a level with many tied scores.  Scores of one makespan c lie a few ulps apart (the noise),
// those of the next makespan thousands of ulps further: linear bins that span a few makespans put
// all of one into one bin.  These give every makespan of the window [c0, c0 + nc) (in units of the
// durations' common divisor) q bins: a bin for each of the nq scores c can have, in nsl parts
// by slot; or q parts of the noise's range where it has more scores than that.  The map
// is monotone in (score, slot) whatever its parameters: c is a rounded multiple of the score, the
// rest a difference to one number per c, and only keys of one score are told apart by slot.
// GB300, ms per call, one-block route or sorted windows -> tie bins (level kernels): 50x20 K=4096,
// durations 1: 49.5 -> 13.1 (35.5), 1..5: 53.7 -> 12.0 (23.4), 1..20: 28.8 -> 12.6 (23.6); 20x15
// K=1024, 1: 6.7 -> 2.6 (5.7), 1..2: 5.8 -> 4.1 (5.3); K=16384, 1..5: 34.0 -> 9.3 (28.3).
struct TieMap {
    int c0, nc, q, nq, nsl, unit;
    float per, ns, oscale, sscale;   // oscale: noise parts per unit of score, 0 = a bin per score
};

__device__ __forceinline__ int tie_bin(const TieMap& m, uint32_t sc, uint32_t slot)
{
    const float f = __uint_as_float(sc);
    const int c = __float2int_rn(__fmul_rn(f, m.per)), g = c - m.c0;
    if (g < 0) return 0;
    if (g >= m.nc) return NB - 1;
    const float base = __fdiv_rn(__int2float_rn((int)((uint32_t)c * (uint32_t)m.unit)), m.ns);
    if (m.oscale > 0.0f) return g * m.q + min(max((int)__fmul_rn(__fsub_rn(f, base), m.oscale), 0), m.nq - 1);
    const int o = (int)(sc - __float_as_uint(base));
    if (o < 0) return g * m.q;
    if (o >= m.nq) return g * m.q + m.q - 1;
    return g * m.q + o * m.nsl + min((int)__fmul_rn(__int2float_rn((int)slot), m.sscale), m.nsl - 1);
}

// The map of makespans c0 .. c0 + nc - 1 (nc <= NB), scores from flo on, P parents.
__device__ __forceinline__ void tie_map(TieMap& m, int c0, int nc, int unit, float ns, float flo, int P)
{
    const int most = NB / nc;
    // noise of up to 0.000000999 in steps of an ulp of the lowest score
    const float ulp = __uint_as_float(__float_as_uint(flo) + 1u) - flo;
    const int scores = 1 + (int)fminf(0.999e-6f / fmaxf(ulp, 1e-12f) + 0.5f, 1e6f);
    const int nq = min(scores, most), nsl = most / nq;
    m.c0 = c0;
    m.nc = nc;
    m.unit = unit;
    m.ns = ns;
    m.per = __fdiv_rn(ns, (float)unit);
    m.oscale = scores > most ? 1e6f * (float)most : 0.0f;
    m.nq = nq;
    m.nsl = nsl;
    m.q = nq * nsl;
    m.sscale = (float)nsl / (float)(P << 7);
}

// Fixed part of the dynamic shared memory (bytes); the rest of the layout is SearchCfg's.
constexpr int kRow = NB / 2 + 4;                  // words: 16-bit counts of two bins, then the valid children
constexpr int kOffHist = 0;                       // u32[NB] this block's keys per bin
constexpr int kOffPack = kOffHist + 4 * NB;       // u32[kRow] the same for the other blocks
constexpr int kOffTot = kOffPack + 4 * kRow;      // u32[NB] keys of all blocks
constexpr int kOffBase = kOffTot + 4 * NB;        // u32[NB] first position
constexpr int kOffCur = kOffBase + 4 * NB;        // u32[NB] next position
constexpr int kOffOwn = kOffCur + 4 * NB;         // u16[NB] first | last owning block << 8
constexpr int kOffNoise = kOffOwn + 2 * NB;       // f32[1000]
constexpr int kOffMagic = kOffNoise + 4000;       // u32[kMaxJobs + 1] floor((2^32 - 1) / r)
constexpr int kSubBins = 128;                     // bins of a block's window refined by exact score
constexpr int kSubs = 16;                         // scores per refined bin
static_assert(kSubBins * kSubs <= 1 << (32 - kSlotBits), "group and slot share a word");
constexpr int kOffSub = (kOffMagic + 4 * (kMaxJobs + 1) + 15) & ~15;   // u32[kSubBins][kSubs]
constexpr int kOffRef = kOffSub + 4 * kSubBins * kSubs;                // u32[kSubBins] a score of the bin
constexpr int kOffRows = (kOffRef + 4 * kSubBins + 15) & ~15;          // u32[blocks][kRow] every block's
constexpr size_t kFallbackBytes = ((kSelectSmemBytes + 15) & ~(size_t)15) + 4 * (kMaxChunks + 1);

// h % r for 1 <= r <= kMaxJobs
__device__ __forceinline__ int mod_small(uint32_t h, uint32_t r, const uint32_t* magic)
{
    uint32_t x = h - __umulhi(h, magic[r]) * r;   // the quotient is short by 2 at most
    x = x >= r ? x - r : x;
    x = x >= r ? x - r : x;
    return (int)x;
}

// The level's dumped keys (slot order, dense) through the one-block selection.
__device__ __noinline__ void sorted_fallback(SegState& st, int K, int R, int V, const unsigned long long* keys,
                                             uint32_t* sel, uint8_t* smem, uint32_t mn, uint32_t mx)
{
    int* const cpref = reinterpret_cast<int*>(smem + ((kSelectSmemBytes + 15) & ~(size_t)15));
    KeySrc ks;
    const int per = (V + kMaxChunks - 1) / kMaxChunks;
    const int cs = per < 64 ? 64 : (per + 31) & ~31;
    ks.base = keys;
    ks.cpref = cpref;
    ks.nch = (V + cs - 1) / cs;
    ks.cap = cs;
    for (int c = threadIdx.x; c <= ks.nch; c += T) cpref[c] = min(c * cs, V);
    __syncthreads();
    select_sorted(st, K, R, V, 0, ks, sel, smem, mn, mx);
}

template <bool V1, int G>
__global__ void __launch_bounds__(T, 1) k_search(StepArgs a, SearchCfg cf)
{
    using Mask = typename std::conditional<G == 1, unsigned long long, uint32_t>::type;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ BeamConst B;
    __shared__ uint4 s_pub[1];                 // min, max score bits (y, z)
    __shared__ __align__(8) unsigned long long s_bar[kMaxAhead * T / 32];   // per round and warp
    __shared__ LevelState s_keep;
    __shared__ TieMap s_tm[2];
    __shared__ int s_ws[2][32];
    __shared__ int s_T, s_first, s_maxbin, s_x0, s_x1, s_mymax, s_valid, s_lcount, s_tie;
    __shared__ int s_slow;             // ranking the last level with linear bins was slow
    __shared__ uint4 s_lin;            // score bins: plo, shift, tie; levels left with tie bins | the last stay << 16
    __shared__ int s_bad;              // a survivor entry or position that names nothing

    int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = cf.cluster;
    unsigned rank = C > 1 ? cluster_rank() : 0u;
    int seg = __ldg(cf.list + blockIdx.x / (unsigned)C);

    uint32_t* const hist = reinterpret_cast<uint32_t*>(smem + kOffHist);
    uint32_t* const packed = reinterpret_cast<uint32_t*>(smem + kOffPack);
    uint32_t* const rows = reinterpret_cast<uint32_t*>(smem + kOffRows);
    uint32_t* const total = reinterpret_cast<uint32_t*>(smem + kOffTot);
    uint32_t* const binbase = reinterpret_cast<uint32_t*>(smem + kOffBase);
    uint32_t* const cur = reinterpret_cast<uint32_t*>(smem + kOffCur);
    uint16_t* const own = reinterpret_cast<uint16_t*>(smem + kOffOwn);
    float* const noise = reinterpret_cast<float*>(smem + kOffNoise);
    uint32_t* const magic = reinterpret_cast<uint32_t*>(smem + kOffMagic);
    uint32_t* const ops = reinterpret_cast<uint32_t*>(smem + kOffRows + 4 * kRow * C);
    uint32_t* const masks = reinterpret_cast<uint32_t*>(smem + cf.off_mask);
    uint32_t* const sel = reinterpret_cast<uint32_t*>(smem + cf.off_sel);
    int4* const info = reinterpret_cast<int4*>(smem + cf.off_info);
    unsigned long long* const list = reinterpret_cast<unsigned long long*>(smem + cf.off_list);
    uint8_t* const stage = smem + cf.off_stage;
    unsigned long long* const buf = reinterpret_cast<unsigned long long*>(stage);   // after the step: keys by position

    auto csync = [&] {
        __syncwarp();
        if (C > 1) cluster_sync(); else __syncthreads();
    };
    auto load_tables = [&] {
        const SegDesc& d = a.segs[seg];
        const int m = d.m, N = d.N;
#pragma unroll 1
        for (int i = tid; i < N; i += T) {
            const uint32_t o = __ldg(a.ops + d.op_off + i);
            ops[i] = o | (i % m == m - 1 ? kLastOp : 0u);
        }
#pragma unroll 1
        for (int i = tid; i < 1000; i += T) noise[i] = __ldg(a.noise + i);
#pragma unroll 1
        for (int i = tid; i <= kMaxJobs; i += T) magic[i] = i ? 0xFFFFFFFFu / (uint32_t)i : 0u;
#pragma unroll 1
        for (int b = tid; b < NB; b += T) hist[b] = 0u;
    };

    if (tid == 0) {
        const SegDesc& d = a.segs[seg];
        const SearchLay L(d.n, d.m);
        B.n = d.n; B.m = d.m; B.N = d.N; B.K = d.K; B.mode = d.mode; B.words = d.words;
        B.S = L.bytes; B.off_jr = L.off_jr; B.off_op = L.off_op; B.off_mc = L.off_mc; B.off_hdr = L.off_hdr;
        B.bound = a.st[seg].bound;
        B.seed = d.seed;
        B.unit = d.unit;
        B.slack = d.slack;
        B.inv_m = 1.0f / (float)d.m;
        B.inv_s16 = 1.0f / (float)(L.bytes >> 4);
        B.WL = (((d.n + 3) >> 2) + G - 1) / G;   // ready-position words per lane
        B.P = 1;
        B.parents = 0;
        B.paths = cf.paths;
        B.levels = 0;
        B.expanded = B.slots = B.mat = 0;
        B.beam0 = a.beam_pool + d.beam_off[0];
        B.beam1 = a.beam_pool + d.beam_off[1];
        B.slot_base = a.slot_pool + d.slot_off;
        B.hist = a.hist + d.hist_off;
        B.spill = cf.spill + d.key_off;
        s_valid = 0;
        s_lcount = 0;
        s_slow = 0;
        s_bad = 0;
        s_lin = make_uint4(0u, 21u, 0u, 1u << 16);
    }
    load_tables();
    if (lane == 0)
        for (int k = 0; k < kMaxAhead; k++) bar_init(&s_bar[k * (T / 32) + warp]);
    __syncthreads();
    int n = B.n, S = B.S;
    const int SP = cf.stage_stride;
    bool usemask = B.mode != MODE_CLEAN;
    bool split = cf.rs * S > (64 << 10);   // children's stores in quarters
    int P = 1, Pc = 1, lo = rank == 0 ? 0 : 1, cnt = rank == 0 ? 1 : 0;
    if (usemask)
#pragma unroll 1
        for (int i = tid; i < cnt * B.words; i += T) masks[i] = 0u;
    uint32_t phase = 0;
    bool recount_ok = true;
    int tm = 0;           // the level's tie bins are s_tm[tm]'s
    csync();   // the cluster's shared memory is initialised before any remote access

    int sv = tid / G, gl = lane % G;
    int gsh = (lane / G) * G;

    for (int t = 0;; t++) {
        const uint32_t seed_t = B.seed + (uint32_t)t;
        // score bins: bin = (score bits - plo) >> shift, clamped, or tie bins
        uint32_t plo = s_lin.x;
        int shift = (int)s_lin.y;
        bool tie = s_lin.z != 0u;
        const bool lastlv = t == B.N - 1;
        const int rounds = Pc <= cf.rs ? 1 : (Pc + cf.rs - 1) / cf.rs;   // the same in every block
        // entries past list_cap live in global memory
        auto lget = [&](int i) { return i < cf.list_cap ? list[i] : B.spill[(int64_t)lo * n + i]; };
        auto lput = [&](int i, unsigned long long v) {
            if (i < cf.list_cap) list[i] = v; else B.spill[(int64_t)lo * n + i] = v;
        };
        auto linear_bin = [&](uint32_t sc) {
            const uint32_t b = sc < plo ? 0u : (sc - plo) >> shift;
            return b < (uint32_t)NB ? b : (uint32_t)(NB - 1);
        };
        auto bin_of = [&](unsigned long long k) { return (int)((uint32_t)k >> kSlotBits); };

        // ---- v1: survivors are copies of child slots, which this level's children overwrite.
        // With one round per block they are all in shared memory before the first is
        // written; otherwise they are first copied to the beam buffer.
        if (V1 && t > 0 && rounds > 1) {
            const int pieces = cnt * (S >> 4);
            auto piece = [&](int i, const uint4*& from, uint4*& to) {
                const int x = (int)(((float)i + 0.5f) * B.inv_s16), q = i - x * (S >> 4);
                const uint32_t e = sel[x] & ~kFillerFlag;
                // (an entry that is no survivor is reported in the step below)
                const int c = min((int)(e >> 7), B.parents - 1), b = min((int)(e & 127u), n - 1);
                from = reinterpret_cast<const uint4*>(B.slot_base + (int64_t)(c * n + b) * S) + q;
                to = reinterpret_cast<uint4*>(B.beam0 + (lo + x) * S) + q;
            };
#pragma unroll 1
            for (int i = tid; i < pieces; i += 4 * T) {
                const uint4* from[4];
                uint4 *to[4], v[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i + u * T < pieces) {
                        piece(i + u * T, from[u], to[u]);
                        v[u] = __ldcg(from[u]);
                    }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i + u * T < pieces) *to[u] = v[u];
            }
            csync();
        }

        // ---- step
        int nvalid = 0;
        // where the staging area holds the block's whole share, every round's parents are on
        // their way before the first round starts
        const bool ahead = !V1 && t > 0 && rounds > 1 && cf.ahead;
        if (ahead) {
            for (int rd = 0; rd < rounds; rd++) {
                const int rl = rd * cf.rs + sv;
                const bool head = gl == 0 && sv < cf.rs && rl < cnt && search_entry_ok(sel[rl], B.parents, n);
                const uint32_t heads = __ballot_sync(FULL_MASK, head);
                unsigned long long* bar = &s_bar[rd * (T / 32) + warp];
                if (lane == 0 && heads) bar_expect(bar, __popc(heads) * S);
                __syncwarp();
                if (head) {
                    proxy_fence();
                    bulk_load(stage + rl * SP, (t & 1 ? B.beam0 : B.beam1) + (int)((sel[rl] & ~kFillerFlag) >> 7) * S, S, bar);
                }
            }
        }
#pragma unroll 1
        for (int rd = 0; rd < rounds; rd++) {
            const int rl = rd * cf.rs + sv;
            const int r = lo + rl;
            bool act = sv < cf.rs && rl < cnt;
            uint32_t e = 0;
            uint8_t* const sb = stage + (!V1 && cf.ahead ? rl : sv) * SP;
            int32_t* const tr = reinterpret_cast<int32_t*>(sb);
            int32_t* const jr = reinterpret_cast<int32_t*>(sb + B.off_jr);
            uint16_t* const op = reinterpret_cast<uint16_t*>(sb + B.off_op);
            uint8_t* const mcb = sb + B.off_mc;
            uint4* const hdr = reinterpret_cast<uint4*>(sb + B.off_hdr);   // r | ns << 16, cmax, lineage, stamp
            if (t > 0) {
                // (an entry that is no survivor takes no part)
                if (act) e = sel[rl];
                const bool entry = search_entry_ok(e, B.parents, n);
                if (act && !entry) s_bad = 1;
                act = act && entry;
                if (V1) {
                    if (act) {
                        const int c = (int)((e & ~kFillerFlag) >> 7);
                        const uint8_t* src = rounds > 1 ? B.beam0 + r * S
                                                        : B.slot_base + (int64_t)(c * n + (int)(e & 127u)) * S;
#pragma unroll 1
                        for (int q = 16 * gl; q < S; q += 16 * G) cp_async16(sb + q, src + q);
                    }
                    cp_async_commit();
                    cp_async_wait_all();
                    __syncwarp();
                    if (rounds == 1) csync();   // every survivor is staged: slots may be written
                } else {
                    const uint32_t heads = __ballot_sync(FULL_MASK, act && gl == 0);
                    if (heads) {
                        const int k = ahead ? rd : 0;
                        unsigned long long* bar = &s_bar[k * (T / 32) + warp];
                        if (!ahead) {
                            if (lane == 0) bar_expect(bar, __popc(heads) * S);
                            __syncwarp();
                            if (act && gl == 0) {
                                const uint8_t* src = (t & 1 ? B.beam0 : B.beam1) + (int)((e & ~kFillerFlag) >> 7) * S;
                                if (rd > 0) bulk_wait_read();   // this slot's child of the last round
                                // the staging slot was last accessed through the generic proxy
                                proxy_fence();
                                bulk_load(sb, src, S, bar);
                            }
                        }
                        const bool ok = bar_wait(bar, (phase >> k) & 1u);
                        phase ^= 1u << k;
                        if (!ok) {
                            // a copy that never completed: its survivors take no further part
                            if (lane == 0) s_bad = 1;
                            act = false;
                        }
                    }
                    __syncwarp();
                }
            } else if (act) {
                // root (gpu_snapshot.cuh:34-44): first op of every job ready, in job order
                const int m = B.m;
#pragma unroll 1
                for (int q = gl; q < n; q += G) {
                    jr[q] = 0;
                    op[q] = (uint16_t)(q * m);
                    mcb[q] = (uint8_t)(ops[q * m] & 63u);
                }
#pragma unroll 1
                for (int q = gl; q < m; q += G) tr[q] = 0;
                if (gl == 0) *hdr = make_uint4((uint32_t)n, 0u, kMark, 0u);
                proxy_fence();
            }
            __syncwarp();
            bool fresh = act;   // a new state, to be stored
            // many children's stores are issued in quarters between the phases below: an SM writes
            // ~30 bytes per cycle, and a warp waits while the copy queue is full
            auto store_children = [&](int part) {
                if (!V1 && fresh && gl == 0 && !lastlv && (split ? ((lane / G) & 3) == part : part == 0)) {
                    proxy_fence();
                    bulk_store((t & 1 ? B.beam1 : B.beam0) + r * S, sb, S);
                    bulk_commit();
                }
            };
            uint4 h = act ? *hdr : make_uint4(0u, 0u, 0u, 0u);
            if (V1) {
                if (t > 0 && act && gl == 0) B.hist[(t - 1) * B.K + r] = h.w == (uint32_t)t ? h.z : kMark;
            } else {
                if (t > 0) {
                    // kernel_materialize_topk (gpu/v2_twophases/solver.cu:193-252): apply the op at
                    // ready position ii of the parent; a filler's branch is looked up in the
                    // parent's expansion, and one that does not exist leaves the rank's older state
                    const int c = (int)((e & ~kFillerFlag) >> 7);
                    int ii = (int)(e & 127u);
                    if (act && (e & kFillerFlag)) {
                        const int rr = (int)(h.x & 0xFFFFu);
                        int found = -1;
                        if (rr > 0) {
                            const int pm = mcb[mod_small(pivot_hash(seed_t - 1u + (uint32_t)c), (uint32_t)rr, magic)];
#pragma unroll 1
                            for (int i = 0, k = 0; i < rr; i++)
                                if (mcb[i] == pm && k++ == ii) { found = i; break; }
                        }
                        ii = found;
                    }
                    const bool apply = act && search_position_ok(ii, h.x);
                    int opx = 0, opl = 0, mcx = 0, mcl = 0, jrl = 0, fin = 0, last = 0;
                    uint32_t o = 0;
                    if (apply) {
                        last = (int)(h.x & 0xFFFFu) - 1;
                        opx = op[ii];
                        mcx = mcb[ii];
                        opl = op[last];
                        mcl = mcb[last];
                        jrl = jr[last];
                        o = ops[opx];
                        fin = max(tr[mcx], jr[ii]) + (int)(o >> 8);
                        const bool cont = !(o & kLastOp);
                        h.x = (uint32_t)(last + (cont ? 1 : 0)) | (((h.x >> 16) + 1u) << 16);
                        h.y = (uint32_t)max((int)h.y, fin);
                    }
                    __syncwarp();
                    if (apply && gl == 0) {
                        tr[mcx] = fin;
                        if (ii != last) {
                            op[ii] = (uint16_t)opl;
                            mcb[ii] = (uint8_t)mcl;
                            jr[ii] = jrl;
                        }
                        if (!(o & kLastOp)) {
                            op[last] = (uint16_t)(opx + 1);
                            mcb[last] = (uint8_t)(ops[opx + 1] & 63u);
                            jr[last] = fin;
                        }
                        *reinterpret_cast<uint2*>(hdr) = make_uint2(h.x, h.y);
                        B.hist[(t - 1) * B.K + r] = ((uint32_t)c << 8) | (uint32_t)(int)(((float)opx + 0.5f) * B.inv_m);
                    }
                    if (act && !apply) {
                        const uint4* s4 = reinterpret_cast<const uint4*>((t & 1 ? B.beam1 : B.beam0) + r * S);
#pragma unroll 1
                        for (int q = gl; q < (S >> 4); q += G) reinterpret_cast<uint4*>(sb)[q] = __ldcg(s4 + q);
                        if (gl == 0) {
                            B.hist[(t - 1) * B.K + r] = kMark;
                            if (B.mode == MODE_CLEAN || !(e & kFillerFlag)) s_bad = 1;
                        }
                    }
                    __syncwarp();
                    if (act && !apply) h = *hdr;
                    fresh = apply;
                }
                store_children(0);
            }

            // ---- expand for level t: pivot machine, candidate positions (gpu/v1/solver.cu:47-69)
            const int rr = (int)(h.x & 0xFFFFu);
            Mask mk = 0;
            if (rr > 0) {
                const int pm = mcb[mod_small(pivot_hash(seed_t + (uint32_t)r), (uint32_t)rr, magic)];
                if (gl == 0) {
                    const int ns1 = (int)(h.x >> 16) + 1;
                    info[sv] = make_int4(tr[pm], (int)h.y, __float_as_int(__int2float_rn(ns1)), ns1);
                }
                const uint32_t rep = (uint32_t)pm * 0x01010101u;
                const int WL = B.WL;
                const uint32_t* mw = reinterpret_cast<const uint32_t*>(mcb) + gl * WL;
                const int left = rr - 4 * gl * WL;
                // up to 32 positions per lane (64 where a lane takes the whole list)
#pragma unroll 1
                for (int k = 0; k < WL && 4 * k < left; k += 2) {
                    // (a word past the lane's last is inside the record; its bits are cut off)
                    const uint32_t w0 = mw[k], w1 = mw[k + 1];
                    mk |= (Mask)((((__vcmpeq4(w0, rep) & 0x01010101u) * 0x10204080u) >> 28) |
                                 ((((__vcmpeq4(w1, rep) & 0x01010101u) * 0x10204080u) >> 28) << 4)) << (4 * k);
                }
                const int most = min(4 * WL, left);
                if (most < (int)(8 * sizeof(Mask))) mk &= most > 0 ? ((Mask)1 << most) - 1 : (Mask)0;
            }
            store_children(1);
            // the warp's candidates take a run of the list (in any order of the warps: a key
            // carries its slot)
            const int cl = G == 1 ? __popcll(mk) : __popc((uint32_t)mk);
            const int inc = warp_inclusive(cl, lane);
            const int wtot = __shfl_sync(FULL_MASK, inc, 31);
            int base = 0;
            if (lane == 31 && inc) base = atomicAdd(&s_lcount, inc);
            base = __shfl_sync(FULL_MASK, base, 31);
            {
                int pos = base + inc - cl, i0 = 4 * gl * B.WL;
                int b = (inc - cl) - __shfl_sync(FULL_MASK, inc - cl, gsh);
                while (mk) {
                    const int i = i0 + (G == 1 ? __ffsll((long long)mk) : __ffs((int)mk)) - 1;
                    mk &= mk - 1;
                    lput(pos++, (unsigned long long)(((uint32_t)sv << 16) | ((uint32_t)i << 8) | (uint32_t)b++));
                }
            }
            __syncwarp();
            store_children(2);
            // ---- score (kernel_score_candidates, gpu/v1/solver.cu:72-127, v2 :68-123)
#pragma unroll 1
            for (int x0 = 0; x0 < wtot; x0 += 32) {
                const int x = base + x0 + lane;
                const bool has = x0 + lane < wtot;
                const uint32_t en = has ? (uint32_t)lget(x) : 0u;
                const int sv2 = (int)(en >> 16), i = (int)((en >> 8) & 255u), b = (int)(en & 255u);
                const uint8_t* sb2 = stage + (!V1 && cf.ahead ? rd * cf.rs + sv2 : sv2) * SP;
                bool valid = false;
                int fin = 0, cm = 0, opx = 0;
                if (has) {
                    const int4 f = info[sv2];
                    opx = reinterpret_cast<const uint16_t*>(sb2 + B.off_op)[i];
                    const int pred = reinterpret_cast<const int32_t*>(sb2 + B.off_jr)[i];
                    fin = max(f.x, pred) + (int)(ops[opx] >> 8);
                    cm = max(f.y, fin);
                    valid = cm < B.bound;   // gpu/v1/solver.cu:120
                    const int r2 = lo + rd * cf.rs + sv2;
                    unsigned long long key = ~0ull;
                    if (valid) {
                        const float q = __fdiv_rn(__int2float_rn(cm), __int_as_float(f.z));
                        const uint32_t sc = __float_as_uint(
                            __fadd_rn(q, noise[noise_hash(seed_t, (uint32_t)r2, (uint32_t)b) % 1000u]));
                        const uint32_t bin = linear_bin(sc);
                        key = ((unsigned long long)sc << 32) | (bin << kSlotBits) | ((uint32_t)r2 << 7) | (uint32_t)(V1 ? b : i);
                        if (!tie) atomicAdd(&hist[bin], 1u);
                        if (usemask) atomicOr(&masks[(rd * cf.rs + sv2) * B.words + (b >> 5)], 1u << (b & 31));
                        if (lastlv && f.w == B.N) {
                            const int job = (int)(((float)opx + 0.5f) * B.inv_m);
                            atomicMin(&a.st[seg].best, ((unsigned long long)(uint32_t)cm << 32) |
                                                    ((unsigned long long)(uint32_t)(r2 * n + b) << 8) | (uint32_t)job);
                            atomicMin(a.group_best + a.segs[seg].group, cm);
                        }
                    }
                    lput(x, key);
                }
                const uint32_t vb = __ballot_sync(FULL_MASK, valid);
                nvalid += __popc(vb);
                if (V1 && !lastlv) {
                    // every scored child's snapshot into its slot (gpu/v1/solver.cu:129-145):
                    // four lanes per child copy the parent, then write what the op changes
#pragma unroll 1
                    for (int y0 = 0; y0 < 32; y0 += 8) {
                        if (!((vb >> y0) & 255u)) continue;
                        const int from = y0 + (lane >> 2), q4 = lane & 3;
                        const uint32_t en2 = __shfl_sync(FULL_MASK, en, from);
                        const int fin2 = __shfl_sync(FULL_MASK, fin, from), cm2 = __shfl_sync(FULL_MASK, cm, from);
                        const bool on = (vb >> from) & 1u;
                        const int sv3 = (int)(en2 >> 16), i3 = (int)((en2 >> 8) & 255u), b3 = (int)(en2 & 255u);
                        const uint8_t* s3 = stage + sv3 * SP;
                        const int r3 = lo + rd * cf.rs + sv3;
                        uint8_t* dst = B.slot_base + ((int64_t)r3 * n + b3) * S;
                        if (on)
#pragma unroll 1
                            for (int q = q4; q < (S >> 4); q += 4)
                                reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<const uint4*>(s3)[q];
                        __syncwarp();
                        if (on) {
                            const uint4 h3 = *reinterpret_cast<const uint4*>(s3 + B.off_hdr);
                            const int last = (int)(h3.x & 0xFFFFu) - 1;
                            const int op3 = reinterpret_cast<const uint16_t*>(s3 + B.off_op)[i3];
                            const uint32_t o3 = ops[op3];
                            const bool cont = !(o3 & kLastOp);
                            uint16_t* dop = reinterpret_cast<uint16_t*>(dst + B.off_op);
                            int32_t* djr = reinterpret_cast<int32_t*>(dst + B.off_jr);
                            uint8_t* dmc = dst + B.off_mc;
                            if (q4 == 0) {
                                const int job = (int)(((float)op3 + 0.5f) * B.inv_m);
                                *reinterpret_cast<uint4*>(dst + B.off_hdr) =
                                    make_uint4((uint32_t)(last + (cont ? 1 : 0)) | (((h3.x >> 16) + 1u) << 16),
                                               (uint32_t)cm2, ((uint32_t)r3 << 8) | (uint32_t)job, (uint32_t)(t + 1));
                            } else if (q4 == 1) {
                                reinterpret_cast<int32_t*>(dst)[o3 & 63u] = fin2;
                                if (cont) djr[last] = fin2;
                            } else if (q4 == 2) {
                                if (i3 != last) {
                                    djr[i3] = reinterpret_cast<const int32_t*>(s3 + B.off_jr)[last];
                                    dop[i3] = reinterpret_cast<const uint16_t*>(s3 + B.off_op)[last];
                                    dmc[i3] = s3[B.off_mc + last];
                                }
                            } else if (cont) {
                                dop[last] = (uint16_t)(op3 + 1);
                                dmc[last] = (uint8_t)(ops[op3 + 1] & 63u);
                            }
                        }
                        __syncwarp();
                    }
                }
            }
            store_children(3);
            __syncwarp();
        }
        if (lane == 0 && nvalid) atomicAdd(&s_valid, nvalid);
        if (!V1) bulk_wait_read();   // the staging area is the key buffer from barrier #1 on
        if (tid == 0) {
            s_T = 0;
            s_first = NB;
            s_maxbin = 0;
            s_x0 = 1 << 30;   // no window: x0 + tid stays above s_x1
            s_x1 = 0;
            s_mymax = 0;
        }

        // ---- selection: V, threshold bin, positions
        int V, Vb, keff, R, Pn, w0, w1, H, Tb;   // Vb: valid children of lower blocks
        int tries = 0;
        int lcount;
        uint32_t slow;   // blocks whose ranking of the last level with linear bins was slow
        for (;;) {
            __syncthreads();
            lcount = s_lcount;
            if (tie || tries) {
                // the keys' bins in another map than the score's linear one
#pragma unroll 1
                for (int i = tid; i < lcount; i += T) {
                    const unsigned long long k = lget(i);
                    const uint32_t sc = (uint32_t)(k >> 32), slot = (uint32_t)k & kSlotMask;
                    if (sc == kNoKey) continue;
                    const uint32_t bin = tie ? (uint32_t)tie_bin(s_tm[tm], sc, slot) : linear_bin(sc);
                    lput(i, (k & ~0xFFFFFFFFull) | (bin << kSlotBits) | slot);
                    atomicAdd(&hist[bin], 1u);
                }
                __syncthreads();
            }
            uint32_t lower = 0, tot = 0;   // of bin tid
            if (C > 1) {
                // counts above 16 bits saturate; such a bin never fits the buffers, and V is exact
                if (tid < NB / 2) {
                    const uint2 c = reinterpret_cast<const uint2*>(hist)[tid];
                    reinterpret_cast<uint2*>(hist)[tid] = make_uint2(0u, 0u);
                    packed[tid] = min(c.x, 0xFFFFu) | (min(c.y, 0xFFFFu) << 16);
                } else if (tid == NB / 2) {
                    packed[NB / 2] = (uint32_t)s_valid | (uint32_t)s_slow << 24;
                }
                csync();   // #1
                for (int x = tid; x < C * (kRow / 4); x += T) {
                    const int p = (x * (65536 / (kRow / 4) + 1)) >> 16, j = 4 * (x - p * (kRow / 4));
                    *reinterpret_cast<uint4*>(&rows[p * kRow + j]) = ld_peer4(&packed[j], p);
                }
                __syncthreads();
                const uint32_t* col = rows + (tid >> 1);
                const int half = 16 * (tid & 1);
#pragma unroll 4
                for (int q = 0; q < C; q++) {
                    if (q == (int)rank) lower = tot;
                    tot += (col[q * kRow] >> half) & 0xFFFFu;
                }
                const uint32_t pv = lane < C ? rows[lane * kRow + NB / 2] : 0u;
                const uint32_t sum = __reduce_add_sync(FULL_MASK, pv);
                V = (int)(sum & 0xFFFFFFu);
                slow = sum >> 24;
                Vb = (int)(__reduce_add_sync(FULL_MASK, lane < (int)rank ? pv : 0u) & 0xFFFFFFu);
            } else {
                tot = hist[tid];
                hist[tid] = 0u;
                V = s_valid;
                Vb = 0;
                slow = (uint32_t)s_slow;
            }
            const int t0 = (int)tot, b0 = block_exclusive(t0, s_ws[0], lane, warp);
            keff = usemask ? min(P * n, B.K) : min(V, B.K);
            R = min(V, keff);
            Pn = (int)(((unsigned long long)(uint32_t)(keff + C - 1) * cf.c_magic) >> 20);
            w0 = (int)rank * Pn;
            w1 = min(w0 + Pn, R);   // positions [w0, w1) of the sort are this block's
            if (lastlv || R == 0) break;
            total[tid] = tot;
            binbase[tid] = (uint32_t)b0;
            cur[tid] = (uint32_t)b0 + lower;
            const bool in = t0 > 0 && b0 < R;
            if (C > 1 && in) {
                // first and last owner of the bin's positions
                const float inv = 1.0f / (float)Pn;
                auto owner = [&](int p) {
                    int q = (int)((float)p * inv);
                    q -= q * Pn > p ? 1 : 0;
                    q += (q + 1) * Pn <= p ? 1 : 0;
                    return q;
                };
                own[tid] = (uint16_t)(owner(b0) | (owner(min(b0 + t0, R) - 1) << 8));
            }
            const int wbig = (int)__reduce_max_sync(FULL_MASK, in ? tot : 0u);
            const uint32_t occ = __ballot_sync(FULL_MASK, t0 > 0);
            if (lane == 0 && wbig) atomicMax(&s_maxbin, wbig);
            if (occ && lane == __ffs(occ) - 1) atomicMin(&s_first, tid);
            if (in && b0 + t0 >= R) s_T = tid;
            if (in && b0 < w1 && b0 + t0 > w0) {
                atomicMin(&s_x0, b0);
                atomicMax(&s_x1, b0 + t0);
                atomicMax(&s_mymax, t0);
            }
            __syncthreads();
            H = s_maxbin;
            Tb = s_T;
            // too coarse, or a range that ends below the last survivor (its bin holds all that lie past it)
            const bool fit = Pn + 2 * H <= cf.buf_cap;
            const bool coarse = H > kRecountBin || !fit || (tries == 0 && Tb == NB - 1 && H > kPlainBinMax);
            if (!coarse || tries == (recount_ok ? kMaxRecounts : 1) || (fit && (tries > 1 || !recount_ok))) {
                // recounts that did not help: hardly any more of them for this beam while it lasts
                if (tries) recount_ok = !coarse;
                else if (!coarse) recount_ok = true;
                break;
            }
            // ---- again, over the range from the level's lowest score to the bin of the last
            // survivor: linear bins, then (at once, if the level had them or has one try only) tie bins
            tries++;
            uint32_t mn = 0xFFFFFFFFu, mx = 0u;
#pragma unroll 1
            for (int i = tid; i < lcount; i += T) {
                const uint32_t sc = (uint32_t)(lget(i) >> 32);
                if (sc != kNoKey) { mn = min(mn, sc); mx = max(mx, sc); }
            }
            if (tid == 0) s_pub[0] = make_uint4(0u, 0xFFFFFFFFu, 0u, 0u);
            mn = __reduce_min_sync(FULL_MASK, mn);
            mx = __reduce_max_sync(FULL_MASK, mx);
            __syncthreads();
            if (lane == 0) {
                atomicMin(&s_pub[0].y, mn);
                atomicMax(&s_pub[0].z, mx);
            }
            if (tid == 0) {
                s_T = 0;
                s_first = NB;
                s_maxbin = 0;
                s_x0 = 1 << 30;
                s_x1 = 0;
                s_mymax = 0;
            }
            csync();
            mn = 0xFFFFFFFFu;
            mx = 0u;
            if (lane < C) {
                const uint4 w = C > 1 ? ld_peer4(&s_pub[0], lane) : s_pub[0];
                mn = w.y;
                mx = w.z;
            }
            mn = __reduce_min_sync(FULL_MASK, mn);
            mx = __reduce_max_sync(FULL_MASK, mx);
            const bool was = tie;
            if (!was && Tb < NB - 1)
                mx = (uint32_t)min((unsigned long long)mx, plo + ((unsigned long long)(Tb + 1) << shift) - 1);
            if (was || tries > 1 || !recount_ok) {
                const float ns = (float)(t + 1), per = __fdiv_rn(ns, (float)B.unit);
                const int c0 = __float2int_rn(__uint_as_float(mn) * per);
                int c1 = __float2int_rn(__uint_as_float(mx) * per);
                if (was && Tb < NB - 1) c1 = min(c1, s_tm[tm].c0 + Tb / s_tm[tm].q);
                tie = (uint32_t)(c1 - c0) < (uint32_t)NB;
                if (tie) {
                    tm ^= 1;
                    if (tid == 0) tie_map(s_tm[tm], c0, c1 - c0 + 1, B.unit, ns, __uint_as_float(mn), P);
                }
            }
            if (!tie) {
                plo = mn;
                const int nbits = mx > plo ? 32 - __clz(mx - plo) : 0;
                shift = nbits > kSearchBinBits ? nbits - kSearchBinBits : 0;
            }
            if (tid == T - 32) {
                s_lin.x = plo;
                s_lin.y = (uint32_t)shift;
                s_lin.z = tie ? 1u : 0u;
            }
        }
        if (tid == 0) {
            B.expanded += V;
            B.slots += P * n;
            B.levels += 1;
            B.mat += lastlv ? 0 : keff;
            B.P = keff;
            B.parents = P;
            const bool large = V > kStageKeys || B.K > kLsdMax;
            if (R > 0 && !lastlv)
                B.paths |= (large ? kPathLarge : (cf.wide && C > 1 && V > kClusterMinKeys ? kPathCluster : kPathDirect)) |
                           (tries ? kPathRecount : 0u) | (tie ? kPathTieBins : 0u);
        }
        if (lastlv || keff == 0) break;    // clean: every child pruned
        if (!V1) bulk_wait();              // this level's children are in memory before barrier #2
        const bool fits = R == 0 || (H < 0xFFFF && Pn + 2 * H <= cf.buf_cap);
        // ---- the next level's bins: this level's kept scores, one operation later (in a warp that has
        // no keys to push where the share is small)
        if (tid == T - 32 && R == 0) s_lin.z = 0u;
        if (tid == T - 32 && R > 0) {
            const uint4 lin = s_lin;
            // linear bins did not do: some block ranked the last level slowly, or this one goes to one block
            const bool failed = slow != 0u || !fits;
            const float u = __fdividef(1.0f, (float)(t + 2));
            // f0, f1: the scores kept.  The lowest child keeps its makespan; above, half the kept range
            // and some more (a narrow beam's range is a few operations' differences wide, and a
            // prediction that misses it clamps all keys into one bin)
            float f0 = __uint_as_float(lin.x + ((uint32_t)s_first << lin.y));
            float f1 = __uint_as_float(lin.x + (((uint32_t)Tb + 1u) << lin.y) - 1u);
            int left = (int)(lin.w & 0xFFFFu), stay = (int)(lin.w >> 16), next_tie = 0;
            if (lin.z | (uint32_t)failed | (lin.w ^ (1u << 16))) {
                // tie bins for the next levels where linear ones did not do, and for twice as many
                // each time that they do not again
                if (lin.z) {
                    const TieMap& m = s_tm[tm];
                    const float score = __fdiv_rn((float)m.unit, m.ns);
                    f0 = (float)(m.c0 + min(s_first / m.q, m.nc)) * score;
                    f1 = (float)(m.c0 + min(Tb / m.q, m.nc) + 1) * score;
                }
                if (left > 0) left--;
                else if (lin.z || failed) left = stay = min(2 * stay, kTieStay);
                else stay = max(stay / 2, 1);
                if (left > 0) {
                    const float g0 = f0 - f0 * u, g1 = f1 + 0.5f * (f1 - f0) + B.slack * u;
                    const float ns = (float)(t + 2), per = __fdiv_rn(ns, (float)B.unit);
                    const int c0 = __float2int_rn(g0 * per), c1 = __float2int_rn(g1 * per);
                    next_tie = (uint32_t)(c1 - c0) < (uint32_t)NB ? 1 : 0;
                    if (next_tie) tie_map(s_tm[tm ^ 1], c0, c1 - c0 + 1, B.unit, ns, g0, keff);
                }
            }
            const float g0 = f0 - f0 * u, g1 = f1 + 0.5f * (f1 - f0) + B.slack * u;
            const uint32_t lo32 = __float_as_uint(g0), hi32 = __float_as_uint(g1);
            const int nbits = hi32 > lo32 ? 32 - __clz(hi32 - lo32) : 0;
            s_lin = make_uint4(lo32, (uint32_t)(nbits > kSearchBinBits ? nbits - kSearchBinBits : 0),
                               (uint32_t)next_tie, (uint32_t)(left | stay << 16));
        }
        if (R > 0 && fits) {
            // ---- keys of bins <= T to their positions' owners; buf[p - first position + H]
#pragma unroll 1
            for (int i = tid; i < lcount; i += T) {
                const unsigned long long k = lget(i);
                if ((uint32_t)(k >> 32) == kNoKey) continue;
                const int bin = bin_of(k);
                if (bin > Tb) continue;
                const int p = (int)atomicAdd(&cur[bin], 1u);
                if (C > 1) {
                    const uint32_t w = own[bin];
#pragma unroll 1
                    for (int q = (int)(w & 255u); q <= (int)(w >> 8); q++) st_peer64(&buf[p - q * Pn + H], q, k);
                } else {
                    buf[p + H] = k;
                }
            }
            uint32_t* const sub = reinterpret_cast<uint32_t*>(smem + kOffSub);
            uint32_t* const ref = reinterpret_cast<uint32_t*>(smem + kOffRef);
            {
#pragma unroll
                for (int u = 0; u < kSubBins * kSubs / 4 / T; u++)
                    reinterpret_cast<uint4*>(sub)[u * T + tid] = make_uint4(0u, 0u, 0u, 0u);
                if (tid == 0) s_tie = 0;
            }
            csync();   // #2
            const int x0 = s_x0, x1 = s_x1;
            if (tid == 0) s_slow = 0;
            unsigned long long* const win = buf + (H - w0);   // by global position
            if (s_mymax <= kPlainBinMax) {
                // small bins: two lanes per key count the smaller keys of its bin
#pragma unroll 1
                for (int xb = x0; xb < x1; xb += T / 2) {
                    const int x = xb + (tid >> 1);
                    int c = 0, f0 = 0;
                    unsigned long long k = 0;
                    if (x < x1) {
                        k = win[x];
                        const int bin = bin_of(k);
                        f0 = (int)binbase[bin];
                        const int ft = (int)total[bin];
                        const unsigned long long* y = win + f0;
#pragma unroll 2
                        for (int z = tid & 1; z < ft; z += 2) c += y[z] < k ? 1 : 0;
                    }
                    c += __shfl_xor_sync(FULL_MASK, c, 1);
                    const int p = f0 + c;
                    if (x < x1 && !(tid & 1) && p >= w0 && p < w1) sel[p - w0] = (uint32_t)k & kSlotMask;
                }
            } else {
                // larger bins hold a few scores, a few ulps apart (one makespan, different
                // noise): keys are placed by exact score within their bin, then each counts the
                // smaller slots among its equals
                uint32_t* const win2 = reinterpret_cast<uint32_t*>(buf + cf.buf_cap) + (H - w0);   // group, slot by position
                const int bin0 = x0 < x1 ? bin_of(win[x0]) : 0;
                const int nb = x0 < x1 ? bin_of(win[x1 - 1]) - bin0 + 1 : 0;
                bool ok = nb <= kSubBins;
                if (ok) {
#pragma unroll 1
                    for (int x = x0 + tid; x < x1; x += T) {
                        const unsigned long long k = win[x];
                        ref[bin_of(k) - bin0] = (uint32_t)(k >> 32);   // any score of the bin
                    }
                    __syncthreads();
#pragma unroll 1
                    for (int x = x0 + tid; x < x1; x += T) {
                        const unsigned long long k = win[x];
                        const int lb = bin_of(k) - bin0;
                        const uint32_t o = (uint32_t)(k >> 32) - ref[lb] + kSubs / 2;
                        if (o < (uint32_t)kSubs) atomicAdd(&sub[lb * kSubs + o], 1u);
                        else s_tie = 1 << 30;   // scores further apart than the table
                    }
                    __syncthreads();
                    // per bin: first position of each score; the largest group of equals
                    int most = 0;
                    if (tid < nb) {
                        uint32_t p = binbase[bin0 + tid];
#pragma unroll
                        for (int o = 0; o < kSubs; o++) {
                            const uint32_t c = sub[tid * kSubs + o];
                            sub[tid * kSubs + o] = p;
                            most = max(most, (int)c);
                            p += c;
                        }
                    }
                    most = (int)__reduce_max_sync(FULL_MASK, (uint32_t)most);
                    if (lane == 0 && most) atomicMax(&s_tie, most);
                    __syncthreads();
                    ok = s_tie <= kTieMax;
                }
                if (tid == 0 && !tie && C >= kTieBlocks && nb <= kSubBins && (!ok || s_tie > kTieSlow)) s_slow = 1;
                if (ok) {
#pragma unroll 1
                    for (int x = x0 + tid; x < x1; x += T) {
                        const unsigned long long k = win[x];
                        const uint32_t sc = (uint32_t)(k >> 32);
                        const int lb = bin_of(k) - bin0, g = lb * kSubs + (int)(sc - ref[lb]) + kSubs / 2;
                        const int p = (int)atomicAdd(&sub[g], 1u);   // afterwards sub[g] is the group's end
                        win2[p] = ((uint32_t)g << kSlotBits) | ((uint32_t)k & kSlotMask);
                    }
                    __syncthreads();
#pragma unroll 1
                    for (int xb = x0; xb < x1; xb += T / 2) {
                        const int x = xb + (tid >> 1);
                        int c = 0, f0 = 0;
                        uint32_t k = 0;
                        if (x < x1) {
                            k = win2[x];
                            const int g = (int)(k >> kSlotBits);
                            f0 = (int)((g & (kSubs - 1)) ? sub[g - 1] : binbase[bin0 + g / kSubs]);
                            const int f1 = (int)sub[g];
                            int z = f0 + (tid & 1);
                            if (f1 <= w0 || f0 >= w1) z = f1;   // another block's positions
                            for (; z + 6 < f1; z += 8) {
                                const uint32_t y0 = win2[z], y1 = win2[z + 2], y2 = win2[z + 4], y3 = win2[z + 6];
                                c += (y0 < k ? 1 : 0) + (y1 < k ? 1 : 0) + (y2 < k ? 1 : 0) + (y3 < k ? 1 : 0);
                            }
#pragma unroll 1
                            for (; z < f1; z += 2) c += win2[z] < k ? 1 : 0;
                        }
                        c += __shfl_xor_sync(FULL_MASK, c, 1);
                        const int p = f0 + c;
                        if (x < x1 && !(tid & 1) && p >= w0 && p < w1) sel[p - w0] = k & kSlotMask;
                    }
                } else {
                    sort_window(win + x0, buf, x1 - x0, x0, w0, w1, sel);
                    if (tid == 0) B.paths |= kPathWindowSort;
                }
            }
        } else if (R > 0) {
            // ---- a bin too large for the buffers: the level's keys, slot order, to global
            // memory, and the one-block selection in block 0 (whose tables share this
            // kernel's shared memory)
            const SegDesc& d = a.segs[seg];
            const int words = d.words;
            if (tid == 0) B.paths |= kPathOneBlock;
            if (usemask)
#pragma unroll 1
                for (int i = tid; i < cnt * words; i += T) a.masks[d.mask_off + (int64_t)lo * words + i] = masks[i];
            // slot order: a bit per candidate's ready position and survivor, prefix of their counts
            uint32_t* const bits = reinterpret_cast<uint32_t*>(stage);   // [cnt][words]
            int* const first = reinterpret_cast<int*>(bits + cnt * words);
            for (int i = tid; i < cnt * words; i += T) bits[i] = 0u;
            if (tid == 0) s_pub[0] = make_uint4(0u, 0xFFFFFFFFu, 0u, 0u);
            __syncthreads();
            uint32_t mn = 0xFFFFFFFFu, mx = 0u;
            for (int i = tid; i < lcount; i += T) {
                const unsigned long long k = lget(i);
                const uint32_t sc = (uint32_t)(k >> 32), sl = (uint32_t)k & kSlotMask;
                if (sc == kNoKey) continue;
                mn = min(mn, sc);
                mx = max(mx, sc);
                atomicOr(&bits[((int)(sl >> 7) - lo) * words + ((sl & 127u) >> 5)], 1u << (sl & 31u));
            }
            mn = __reduce_min_sync(FULL_MASK, mn);
            mx = __reduce_max_sync(FULL_MASK, mx);
            if (lane == 0) {
                atomicMin(&s_pub[0].y, mn);
                atomicMax(&s_pub[0].z, mx);
            }
            __syncthreads();
            unsigned long long* dump = a.keys + d.key_off + Vb;
            for (int c0 = 0, sum = 0; c0 < cnt; c0 += T) {
                const int c = c0 + tid;
                int f = 0, tot;
                if (c < cnt)
                    for (int w = 0; w < words; w++) f += __popc(bits[c * words + w]);
                const int off = block_exclusive(f, s_ws[(c0 / T) & 1], lane, warp, tot);
                if (c < cnt) first[c] = sum + off;
                sum += tot;
            }
            __syncthreads();
            for (int i = tid; i < lcount; i += T) {
                const unsigned long long k = lget(i);
                const uint32_t sl = (uint32_t)k & kSlotMask;
                if ((uint32_t)(k >> 32) == kNoKey) continue;
                const int c = (int)(sl >> 7) - lo;
                int p = first[c];
                for (uint32_t w = 0; w < ((sl & 127u) >> 5); w++) p += __popc(bits[c * words + w]);
                p += __popc(bits[c * words + ((sl & 127u) >> 5)] & ((1u << (sl & 31u)) - 1u));
                dump[p] = (k & ~0xFFFFFFFFull) | sl;
            }
            csync();
            __threadfence();
            mn = 0xFFFFFFFFu;
            mx = 0u;
            if (lane < C) {
                const uint4 w = C > 1 ? ld_peer4(&s_pub[0], lane) : s_pub[0];
                mn = w.y;
                mx = w.z;
            }
            mn = __reduce_min_sync(FULL_MASK, mn);
            mx = __reduce_max_sync(FULL_MASK, mx);
            // Nothing but the warps' copy phases stays in registers across the call: what does is
            // kept in local memory for the whole level loop (84-168 bytes per thread).  us per call
            // with and without: 15x15 K=256 1 654 -> 1 456, v1 20x15 K=1024 3 266 -> 2 932, 50x20
            // K=4096 13 602 -> 12 425, 8 beams 17 539 -> 16 042, 100x20 8 beams 43 166 -> 39 875 (figures
            // of the build that took them out).
            if (tid == 0)
                s_keep = LevelState{seg, t, recount_ok ? 1 : 0, tm, lo, cnt, V, Vb, keff, R,
                                    Pn, w0, w1, Tb};
            if (rank == 0) sorted_fallback(a.st[seg], d.K, R, V, a.keys + d.key_off, a.sel + d.sel_off, smem, mn, mx);
            csync();
            __threadfence();
            {
                const volatile LevelState& k = s_keep;
                const volatile BeamConst& b = B;
                seg = k.seg; t = k.t; recount_ok = k.recount_ok != 0; tm = k.tm; lo = k.lo; cnt = k.cnt; V = k.V; Vb = k.Vb; keff = k.keff; R = k.R;
                Pn = k.Pn; w0 = k.w0; w1 = k.w1; Tb = k.Tb;
                n = b.n; S = b.S;
                usemask = b.mode != MODE_CLEAN;
                split = cf.rs * S > (64 << 10);
                asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
                lane = tid & 31;
                warp = tid >> 5;
                sv = tid / G;
                gl = lane % G;
                gsh = (lane / G) * G;
                rank = C > 1 ? cluster_rank() : 0u;
            }
            load_tables();
            const SegDesc& d2 = a.segs[seg];
#pragma unroll 1
            for (int i = tid; i < w1 - w0; i += T) sel[i] = __ldcg(a.sel + d2.sel_off + w0 + i);
            if (usemask)
#pragma unroll 1
                for (int i = tid; i < cnt * d2.words; i += T)
                    masks[i] = __ldcg(a.masks + d2.mask_off + (int64_t)lo * d2.words + i);
            __syncthreads();
        }
        if (keff > R) {
            // ---- v1 / v2: the lowest-numbered unscored slots follow, in slot order
            const int F = keff - R, words = B.words;
            int before = lo * n - Vb;
#pragma unroll 1
            for (int c0 = 0; c0 < cnt && before < F; c0 += T) {
                const int c = c0 + tid;
                int f = 0;
                if (c < cnt) {
                    f = n;
#pragma unroll 1
                    for (int w = 0; w < words; w++) f -= __popc(masks[c * words + w]);
                }
                int tot;
                const int off = block_exclusive(f, s_ws[(c0 / T) & 1], lane, warp, tot);
                int g = before + off;
#pragma unroll 1
                for (int b = 0; b < n && f > 0 && g < F; b++) {
                    if ((masks[c * words + (b >> 5)] >> (b & 31)) & 1u) continue;
                    const int p = R + g, q = p / Pn;
                    const uint32_t e = kFillerFlag | ((uint32_t)(lo + c) << 7) | (uint32_t)b;
                    if (C > 1) st_peer32(&sel[p - q * Pn], q, e);
                    else sel[p] = e;
                    g++;
                    f--;
                }
                before += tot;
            }
            csync();
        }
        tm ^= 1;
        P = keff;
        Pc = Pn;
        lo = min(w0, P);
        cnt = min(Pc, P - lo);
        if (tid == 0) {
            s_valid = 0;
            s_lcount = 0;
        }
        if (usemask)
            for (int i = tid; i < cnt * B.words; i += T) masks[i] = 0u;
        __syncthreads();
    }
    if (rank == 0 && tid == 0) {
        SegState& st = a.st[seg];
        st.expanded += B.expanded;
        st.slots += B.slots;
        st.materialized += B.mat;
        st.levels += B.levels;
        st.P = B.P;
    }
    if (tid == 0) {
        atomicOr(&a.st[seg].select_paths, B.paths);
        if (s_bad) atomicOr(&a.st[seg].status, kStatusBadSelect);
    }
    csync();   // peers may read this block's counts until here
}

template <typename F>
cudaError_t for_each_search(F&& f)
{
    cudaError_t e = f(k_search<false, 1>);
    if (e == cudaSuccess) e = f(k_search<true, 1>);
    if (e == cudaSuccess) e = f(k_search<false, 2>);
    if (e == cudaSuccess) e = f(k_search<false, 4>);
    if (e == cudaSuccess) e = f(k_search<false, 8>);
    if (e == cudaSuccess) e = f(k_search<true, 2>);
    if (e == cudaSuccess) e = f(k_search<true, 4>);
    if (e == cudaSuccess) e = f(k_search<true, 8>);
    return e;
}

std::mutex g_search_mu;

}  // namespace

// Shared-memory layout of a launch; false when it does not fit `limit` dynamic bytes.
bool search_layout(SearchCfg& cf, int cluster, int lanes, int kmax, int nmax, int opsmax, int smax, size_t limit)
{
    const int pc = (kmax + cluster - 1) / cluster;
    const int words = (nmax + 31) / 32;
    cf.cluster = cluster;
    cf.lanes = lanes;
    cf.paths = kPathResident;
    for (int k = 0; k < (int)(sizeof(kSearchSizes) / sizeof(kSearchSizes[0])); k++)
        if (kSearchSizes[k] == cluster) cf.paths |= 1u << (kPathBlocks + k);
    cf.c_magic = ((1u << 20) + (uint32_t)cluster - 1) / (uint32_t)cluster;   // x / cluster, x < 2^15
    cf.stage_stride = smax + ((smax >> 4) & 1 ? 0 : 16);   // odd in 16-byte units: groups' words on distinct banks
    for (cf.rs = T / lanes; cf.rs >= 16; cf.rs /= 2) {
        size_t o = 0;
        auto take = [&](size_t bytes) { const size_t at = o; o = (o + bytes + 15) & ~(size_t)15; return (int)at; };
        take(kOffRows + 4 * (size_t)kRow * cluster);
        take(4 * (size_t)opsmax);
        cf.off_mask = take(4 * (size_t)pc * words);
        cf.off_sel = take(4 * (size_t)pc);
        cf.off_info = take(16 * (size_t)cf.rs);
        // the staging area doubles as the sort's two key buffers and holds the fallback's slot
        // bits; buffers for the block's positions and bins of ~1 000 keys on either side where
        // that leaves the list 16 keys per survivor
        const size_t want = (size_t)pc * nmax * 8;
        size_t stage = std::max(std::max((size_t)cf.rs * cf.stage_stride, (size_t)kSearchMinBuf * 12),
                                (size_t)pc * (words + 1) * 4);
        size_t roomy = kSearchMinBuf;
        while (roomy < (size_t)pc + 4096) roomy *= 2;
        if (o + roomy * 12 + std::min(want, (size_t)pc * 128) <= limit) stage = std::max(stage, roomy * 12);
        // the whole share staged at once (2 to kMaxAhead rounds of it) where that leaves the
        // list 6 keys per survivor (the levels of 50x20 hold 3.7; fitted there -- lists of few machines
        // hold more, 20 at 60x3, and keep part of them in L2: 60x3 K=4096 is faster than by the level
        // kernels all the same)
        const size_t whole = (size_t)pc * cf.stage_stride;
        cf.ahead = pc > cf.rs && pc <= kMaxAhead * cf.rs && o + whole + std::min(want, (size_t)pc * 48) <= limit ? 1 : 0;
        if (cf.ahead) stage = std::max(stage, whole);
        // wide shares: the largest buffer where a third more makes it (a bin too large for the buffer
        // sends the level to one block).  v1 100x8 K=16384: 577 -> 354 us per level
        const size_t most = (size_t)kSortMax * 12;
        if (pc >= 512 && stage < most && most - stage <= stage / 3 && o + most + (size_t)pc * 48 <= limit) stage = most;
        if (o + stage + (size_t)kSearchMinList * 8 > limit) continue;
        const size_t lst = std::min((want + 15) & ~(size_t)15, (limit - o - stage) & ~(size_t)15);
        cf.list_cap = (int)(lst / 8);
        cf.off_list = take(lst);
        cf.off_stage = (int)o;
        cf.smem = std::max(o + stage, kFallbackBytes);
        cf.buf_cap = kSortMax;   // a power of two: sort_window pads its keys to one
        while ((size_t)cf.buf_cap * 12 > cf.smem - o) cf.buf_cap /= 2;
        return cf.smem <= limit;
    }
    return false;
}

namespace {

// Clusters of `cluster` blocks the device runs at once (0 when that size cannot run).
int max_active_clusters(int cluster, size_t smem)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)cluster);
    c.blockDim = dim3(T);
    c.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    int num = 0;
    if (cudaOccupancyMaxActiveClusters(&num, k_search<false, 4>, &c) != cudaSuccess) { cudaGetLastError(); return 0; }
    return num;
}

}  // namespace

// What the current device offers the resident search, its kernels configured (once per
// device and process).
cudaError_t search_device(SearchDevice& out)
{
    constexpr int kMaxDevices = 64;
    static SearchDevice known[kMaxDevices];
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_search_mu);
    SearchDevice& d = known[dev];
    if (!d.smem) {
        e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return e;
        size_t fixed = 0;
        e = for_each_search([&](auto fn) {
            cudaFuncAttributes at;
            const cudaError_t r = cudaFuncGetAttributes(&at, fn);
            if (r == cudaSuccess) fixed = std::max(fixed, at.sharedSizeBytes);
            return r;
        });
        if (e != cudaSuccess) return e;
        const size_t smem = ((size_t)optin - fixed) & ~(size_t)15;
        e = for_each_search([&](auto fn) {
            cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (r == cudaSuccess) r = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            return r;
        });
        if (e != cudaSuccess) return e;
        for (int c : kSearchSizes) d.clusters[c] = max_active_clusters(c, smem);
        d.smem = smem;
    }
    out = d;
    return cudaSuccess;
}

// Fitted to single beams on GB300 on an earlier build; the sizes have become faster since by unequal
// factors, so these are estimates that choose among block counts, not times.  us per level over
// survivors per block (v2, 20x20): one block 64: 5.8, 128: 6.4, 256: 8.1, 384: 10.5, 512: 14.6,
// 1 024: 27.7, 2 048: 50.6; 2 blocks +1.9, 16 +3.8 (barriers); lists of 50 / 100 jobs cost 1.4 / 2
// times as much per survivor; v1 also writes the scored children (1 024: 62.4).  The number of
// machines is not in it.
double search_level_us(int n, int K, bool v1, int C)
{
    const double at[] = {64, 128, 256, 384, 512}, cost[] = {0, 0.7, 2.6, 5.2, 9.3}, slots[] = {0.9, 2.0, 4.8, 7.4, 10.0};
    const double per = (K + C - 1) / C;
    double f = 0, w = 0.9 * per / 64;
    if (per >= 512) {
        f = cost[4] + (per - 512) * 0.026;
        w = slots[4] + (per - 512) * 0.045;
    } else {
        for (int i = 0; i < 4; i++)
            if (per >= at[i] && per < at[i + 1]) {
                const double x = (per - at[i]) / (at[i + 1] - at[i]);
                f = cost[i] + x * (cost[i + 1] - cost[i]);
                w = slots[i] + x * (slots[i + 1] - slots[i]);
            }
    }
    return (C == 1 ? 5.6 : 7.3 + 0.14 * C) + 0.008 * n + f * std::max(1.0, 0.7 + 0.013 * n) + (v1 ? w * n / 20 : 0.0);
}

int search_lanes(int n, int K, int C)
{
    // a round of kSearchThreads / lanes survivors per block: narrow shares spread over more
    // lanes; a lane takes 32 ready positions at most, or 64 alone.  One lane for shares above
    // 256 where lists are short: 37x11, 375 per block 16.4 against 18.2 us per level with two,
    // 20x15, 1 024 per block 41 against 76, but 50x20, 342 per block 23.9 against 20.5.
    const int pc = (K + C - 1) / C;
    if (pc <= 64) return 8;
    if (n > 64 || pc <= 128) return 4;
    return pc <= 256 || n > 40 ? 2 : 1;
}

int search_blocks(const SearchDevice& dev, int n, int m, int K, bool v1, int cmax)
{
    const SearchLay L(n, m);
    int best = 0;
    for (int c : kSearchSizes) {
        // 12 only as the widest allowed: its odd shares leave lanes idle (v1 20x15 K=1024: 12.2 us
        // per level, 11.2 with 16)
        if ((c > cmax && best) || dev.clusters[c] < 1 || (c == 12 && cmax != 12)) continue;
        SearchCfg cf;
        if (!search_layout(cf, c, search_lanes(n, K, c), K, n, n * m, L.bytes, dev.smem)) continue;
        if (!best || search_level_us(n, K, v1, c) < 0.97 * search_level_us(n, K, v1, best)) best = c;
    }
    return best;
}

cudaError_t launch_search(const StepArgs& a, const SearchCfg& cf, int nbeams, bool v1, cudaStream_t stream)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)(nbeams * cf.cluster));
    c.blockDim = dim3(T);
    c.dynamicSmemBytes = cf.smem;
    c.stream = stream;
    cudaLaunchAttribute at[1];
    if (cf.cluster > 1) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cf.cluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        c.attrs = at;
        c.numAttrs = 1;
    }
    switch (cf.lanes) {
    case 1: return v1 ? cudaLaunchKernelEx(&c, k_search<true, 1>, a, cf) : cudaLaunchKernelEx(&c, k_search<false, 1>, a, cf);
    case 2: return v1 ? cudaLaunchKernelEx(&c, k_search<true, 2>, a, cf) : cudaLaunchKernelEx(&c, k_search<false, 2>, a, cf);
    case 4: return v1 ? cudaLaunchKernelEx(&c, k_search<true, 4>, a, cf) : cudaLaunchKernelEx(&c, k_search<false, 4>, a, cf);
    case 8: return v1 ? cudaLaunchKernelEx(&c, k_search<true, 8>, a, cf) : cudaLaunchKernelEx(&c, k_search<false, 8>, a, cf);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace bsj
