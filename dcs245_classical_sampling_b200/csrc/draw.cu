// FP64 inverse-CDF draw of the free bits from a complex128 block (sm_100a).
//
// Reference: `draw_checked`, source/sampling/sampling_protocol.py:44-88.  The reference
// computes weights w = re*re + im*im (two roundings, no FMA), the SEQUENTIAL cumulative sum
// S_i, divides by S_n, forces the last value to 1 and takes searchsorted(u, side='right'),
// i.e. the first i with u < S_i/S_n.  It cross-checks the chosen bin with math.fsum.
//
// Device method:
//   1. weights with the same two-rounding formula (__dmul_rn/__dadd_rn), plus double-double
//      (error-free TwoSum, Knuth; Dekker) partial sums per chunk;
//   2. exclusive double-double scan of the chunk sums -> total T (accurate to ~2^-104);
//   3. the chunk and element with P_{i-1} <= u*T < P_i (P = accurate prefix sums);
//   4. certification: a sequential FP64 sum of non-negative terms satisfies
//      |S_i - P_i| <= gamma_{i} P_i (Higham, Accuracy and Stability, Sec. 4.2), so if u lies
//      outside the error intervals of both bin edges, numpy's index is the same index.
//      Otherwise the block is flagged as a tie and an exact sequential FP64 pass (the same
//      operation order as numpy's cumsum, evaluated through integer maps) decides, without host sync.  On
//      request (DCS_DRAW_SEQUENTIAL) that pass runs for every block, so that the reported CDF
//      values are numpy's bit for bit (the production record rows derive a grid count from them);
//   5. the 53-bit grid total-variation diagnostic of the reference.
#include <cuda.h>
#include <string.h>

#include <mutex>

#include "common.cuh"

using dcs::after_previous;
using dcs::let_next_start;

namespace {

struct dd { double hi, lo; };

__device__ __forceinline__ dd two_sum(double a, double b) {
    const double s = __dadd_rn(a, b);
    const double bb = __dsub_rn(s, a);
    const double err = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
    return {s, err};
}
__device__ __forceinline__ dd fast_two_sum(double a, double b) {
    const double s = __dadd_rn(a, b);
    return {s, __dsub_rn(b, __dsub_rn(s, a))};
}
__device__ __forceinline__ dd dd_add(dd a, double b) {
    dd s = two_sum(a.hi, b);
    return fast_two_sum(s.hi, __dadd_rn(s.lo, a.lo));
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
    dd s = two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __dadd_rn(s.lo, __dadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ dd dd_mul(dd a, double b) {  // Dekker product with FMA error term
    const double p = __dmul_rn(a.hi, b);
    const double e = fma(a.hi, b, -p);
    return fast_two_sum(p, __dadd_rn(e, __dmul_rn(a.lo, b)));
}
// a / b for b != 0, inv = 1 / b.hi: a first quotient, and the exact remainder's (double-double long division, as
// in Hida, Li and Bailey's library), which is 2^-52 of it, so that neither needs a division of its own
__device__ __forceinline__ double dd_div(dd a, dd b, double inv) {
    const double q = a.hi * inv;
    const dd qb = dd_mul(b, q);
    const dd r = dd_add(a, dd{-qb.hi, -qb.lo});
    return fma(r.hi, inv, q);
}
__device__ __forceinline__ bool dd_lt(dd a, dd b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }

constexpr int kChunkLog = 11;
constexpr int kChunk = 1 << kChunkLog;
constexpr int kThreads = 256;
constexpr int kPer = kChunk / kThreads;

struct BlockState {  // per block scratch (device)
    dd total;
    int64_t chunk;
    int32_t status;
    int32_t pad;
};

// The sequential CDF as integer maps.  While the running FP64 sum S stays in one binade [2^e, 2^(e+1)) it
// is k q with q = 2^(e-52), and S <- fl(S + w) adds to k a whole number that depends on w and, only
// where w / q ends in exactly one half (ties go to even), on the parity of k.  So any stretch of
// additions inside one binade is a map (parity of k) -> increment of k, two maps in a row are again
// such a map, and stretches are composed in parallel, exactly.  A stretch is a sub-chunk of kSub elements
// and a chunk; S of its ends is known beforehand to (n + 16) 2^-52 relative from the compensated
// prefix sums (Higham, Accuracy and Stability, Sec. 4.2), which decides whether it lies in one binade.  Zero and the
// subnormal numbers are one more such stretch of whole multiples (e = -1023), in which additions are exact.
constexpr int kSub = 128;                       // elements per sub-chunk: 16 threads of kPer
constexpr int kSubs = kChunk / kSub;            // sub-chunks per chunk
constexpr int kSubThreads = kSub / kPer;
constexpr int32_t kMapWalk = INT32_MIN;         // crosses (or may cross) a binade: add its weights one by one
constexpr int32_t kMapNone = INT32_MIN + 1;     // all weights are zero: S does not change
struct SeqMap {
    long long d0, d1;  // increment of k for even / odd k
    int32_t e;         // the binade's exponent, kMapWalk or kMapNone
    int32_t pad;
};
struct SeqChunk {
    SeqMap map;
    double start;      // S before the chunk
};

// layout of the scratch area
struct Layout {
    size_t w, chunk_sum, state, tv_part, sq_part, chunk_map, sub_map, bytes;
};
__host__ __device__ constexpr Layout layout(int k, int nblocks) {
    const size_t n = (size_t)1 << k;
    const size_t nch = n >= (size_t)kChunk ? n / kChunk : 1;
    const size_t nsub = n >= (size_t)kSub ? n / kSub : 1;
    Layout L{};
    L.w = 0;
    L.chunk_sum = L.w + ((n * nblocks * sizeof(double) + 15) & ~(size_t)15);
    L.state = L.chunk_sum + nch * nblocks * sizeof(dd);
    L.tv_part = L.state + nblocks * sizeof(BlockState);
    L.sq_part = L.tv_part + nch * nblocks * sizeof(double);
    L.chunk_map = L.sq_part + nch * nblocks * sizeof(double);
    L.sub_map = L.chunk_map + nch * nblocks * sizeof(SeqChunk);
    L.bytes = L.sub_map + nsub * nblocks * sizeof(SeqMap);
    L.bytes = (L.bytes + 255) & ~(size_t)255;
    return L;
}

__device__ __forceinline__ dd shfl_up_dd(dd v, int off) {
    return {__shfl_up_sync(0xffffffffu, v.hi, off), __shfl_up_sync(0xffffffffu, v.lo, off)};
}

// sum over the CTA (kThreads threads), the same value in every thread
__device__ __forceinline__ dd block_sum_dd(dd v) {
    __shared__ dd red[kThreads / 32];
    for (int off = 16; off > 0; off >>= 1) {
        dd o{__shfl_xor_sync(0xffffffffu, v.hi, off), __shfl_xor_sync(0xffffffffu, v.lo, off)};
        v = dd_add(v, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[threadIdx.x & (kThreads / 32 - 1)];
    for (int off = kThreads / 64; off > 0; off >>= 1) {
        dd o{__shfl_xor_sync(0xffffffffu, v.hi, off), __shfl_xor_sync(0xffffffffu, v.lo, off)};
        v = dd_add(v, o);
    }
    __syncthreads();
    return v;
}

// Exclusive scan over the CTA's threads, on top of `carry`; `total` receives carry + the sum.  Two
// shuffle scans (inside the warps, then over the warp sums in every warp) instead of one thread
// walking the kThreads sums: a walk is kThreads dependent double-double additions.
__device__ __forceinline__ dd block_scan_dd(dd v, dd carry, dd* total) {
    __shared__ dd red[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    dd inc = v;
    for (int off = 1; off < 32; off <<= 1) {
        const dd o = shfl_up_dd(inc, off);
        if (lane >= off) inc = dd_add(o, inc);
    }
    if (lane == 31) red[warp] = inc;
    __syncthreads();
    dd s = lane < kThreads / 32 ? red[lane] : dd{0.0, 0.0};
    if (lane == 0) s = dd_add(carry, s);
    for (int off = 1; off < kThreads / 32; off <<= 1) {
        const dd o = shfl_up_dd(s, off);
        if (lane >= off) s = dd_add(o, s);
    }
    const int last = kThreads / 32 - 1;
    *total = {__shfl_sync(0xffffffffu, s.hi, last), __shfl_sync(0xffffffffu, s.lo, last)};
    const int from = warp ? warp - 1 : 0;
    dd before{__shfl_sync(0xffffffffu, s.hi, from), __shfl_sync(0xffffffffu, s.lo, from)};
    if (warp == 0) before = carry;
    dd ex = shfl_up_dd(inc, 1);
    if (lane == 0) ex = dd{0.0, 0.0};
    __syncthreads();
    return dd_add(before, ex);
}

// 1. weights + per-chunk double-double sums; part[] marks chunks with a nonfinite amplitude
__global__ void __launch_bounds__(kThreads)
k_weights(const double2* __restrict__ blocks, int k, double* __restrict__ w, dd* __restrict__ chunk_sum,
          double* __restrict__ part) {
    const int b = blockIdx.y;
    const uint64_t n = 1ull << k;
    const uint64_t start = (uint64_t)blockIdx.x * kChunk;
    const double2* v = blocks + ((uint64_t)b << k);
    double* wb = w + ((uint64_t)b << k);
    dd acc{0.0, 0.0};
    int bad = 0;
    let_next_start();
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint64_t i = start + threadIdx.x + (uint64_t)j * kThreads;
        if (i < n) {
            const double2 a = v[i];
            bad |= !isfinite(a.x) || !isfinite(a.y);
            const double wi = __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y));
            wb[i] = wi;
            acc = dd_add(acc, wi);
        }
    }
    const dd s = block_sum_dd(acc);
    const int anybad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        chunk_sum[(uint64_t)b * gridDim.x + blockIdx.x] = s;
        part[(uint64_t)b * gridDim.x + blockIdx.x] = anybad ? 1.0 : 0.0;
    }
}

// 2. chunk scan + chunk search, one CTA per block.  A 2^20 block has 512 chunks: one thread walking them
//    took 69 us (a dependent load, store and addition per chunk), the scan takes about 5.
__global__ void __launch_bounds__(kThreads)
k_scan_locate(dd* chunk_sum, int nch, const double* uniforms, BlockState* state, dcs_draw_result* res,
              const double* part) {
    let_next_start();
    after_previous();
    const int b = blockIdx.x;
    dd* cs = chunk_sum + (uint64_t)b * nch;
    __shared__ int at;
    if (threadIdx.x == 0) at = 0;
    dd run{0.0, 0.0};
    int bad = 0;
    for (int c0 = 0; c0 < nch; c0 += kThreads) {  // exclusive scan in place
        const int c = c0 + threadIdx.x;
        dd s{0.0, 0.0};
        if (c < nch) {
            s = cs[c];
            bad |= part[(uint64_t)b * nch + c] != 0.0;
        }
        dd total;
        const dd ex = block_scan_dd(s, run, &total);
        if (c < nch) cs[c] = ex;
        run = total;
    }
    const int nonfinite = __syncthreads_or(bad);
    const double u = uniforms[b];
    int status = 0;
    if (nonfinite || !(u >= 0.0 && u < 1.0)) status = DCS_E_ARG;
    else if (!(run.hi > 0.0) || !isfinite(run.hi)) status = DCS_E_CDF;
    if (!status) {
        // last chunk whose exclusive start is <= target (every thread reads back its own stores)
        const dd target = dd_mul(run, u);
        int mine = 0;
        for (int c = threadIdx.x; c < nch; c += kThreads)
            if (!dd_lt(target, cs[c])) mine = c;
        if (mine) atomicMax(&at, mine);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        BlockState& st = state[b];
        st.total = run;
        st.status = status;
        st.chunk = at;
        dcs_draw_result& r = res[b];
        memset(&r, 0, sizeof(r));
        r.uniform = u;
        r.index = -1;
        r.status = status;
        r.total_exact = status ? 0.0 : run.hi;
    }
}

// first map, then second
__device__ __forceinline__ void map_then(long long& a0, long long& a1, long long b0, long long b1) {
    a0 += (a0 & 1) ? b1 : b0;
    a1 += ((a1 + 1) & 1) ? b1 : b0;
}

// The maps of one chunk's sub-chunks and of the chunk (all threads of the CTA): thread t owns the
// weights loc[] of elements kPer t .. kPer t + kPer - 1 and `before`, the prefix sum before them.
__device__ __forceinline__ void chunk_maps(const double (&loc)[kPer], double before, uint64_t n, uint64_t c,
                                           uint64_t nch, SeqChunk* chunk_map, SeqMap* sub_map) {
    constexpr int kGroups = kThreads / kSubThreads;
    __shared__ SeqMap sm[kGroups];
    const int lane = threadIdx.x & 31;
    double mine = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) mine += loc[j];
    // ends of the sub-chunk (its kSubThreads threads are half a warp)
    const int first = lane & ~(kSubThreads - 1);
    const double lo = __shfl_sync(0xffffffffu, before, first);
    const double hi = __shfl_sync(0xffffffffu, before + mine, first + kSubThreads - 1);
    const unsigned some = __ballot_sync(0xffffffffu, mine > 0.0) >> first & ((1u << kSubThreads) - 1u);
    const double rel = ((double)n + 16.0) * 2.220446049250313e-16;  // twice the bound, in ulps of 2^-53
    const double s0 = lo * (1.0 - rel), s1 = hi * (1.0 + rel);
    const int e0 = (__double2hiint(s0) >> 20) - 1023, e1 = (__double2hiint(s1) >> 20) - 1023;
    const bool inside = some && e0 == e1 && e0 < 1000;
    long long d0 = 0, d1 = 0;
    if (inside) {
        // increments from an even and from an odd k of the same binade, 2^e and 2^e + q (inside a binade an
        // increment of k is one of the bit pattern)
        const double even = __hiloint2double((e0 + 1023) << 20, 0), odd = __hiloint2double((e0 + 1023) << 20, 1);
#pragma unroll
        for (int j = 0; j < kPer; ++j)
            map_then(d0, d1, __double_as_longlong(__dadd_rn(even, loc[j])) - __double_as_longlong(even),
                     __double_as_longlong(__dadd_rn(odd, loc[j])) - __double_as_longlong(odd));
    }
#pragma unroll
    for (int off = 1; off < kSubThreads; off <<= 1) {
        const long long o0 = __shfl_down_sync(0xffffffffu, d0, off), o1 = __shfl_down_sync(0xffffffffu, d1, off);
        if (!((lane & (kSubThreads - 1)) & (2 * off - 1))) map_then(d0, d1, o0, o1);
    }
    if (lane == first) {
        SeqMap m{d0, d1, inside ? e0 : (some ? kMapWalk : kMapNone), 0};
        sm[threadIdx.x / kSubThreads] = m;
        const uint64_t g = c * kSubs + threadIdx.x / kSubThreads;
        if (g * kSub < n) sub_map[g] = m;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // the chunk: one map if no sub-chunk leaves the binade of the others
        const SeqMap m = lane < kSubs ? sm[lane] : SeqMap{0, 0, kMapNone, 0};
        int e = m.e;
        bool walk = e == kMapWalk;
        long long c0 = m.d0, c1 = m.d1;
#pragma unroll
        for (int off = 1; off < kSubs; off <<= 1) {
            const int oe = __shfl_down_sync(0xffffffffu, e, off);
            const bool ow = __shfl_down_sync(0xffffffffu, (int)walk, off);
            const long long o0 = __shfl_down_sync(0xffffffffu, c0, off), o1 = __shfl_down_sync(0xffffffffu, c1, off);
            if (!(lane & (2 * off - 1))) {
                walk = walk || ow || (e != kMapNone && oe != kMapNone && e != oe);
                if (e == kMapNone) e = oe;
                map_then(c0, c1, o0, o1);
            }
        }
        if (lane == 0) chunk_map[c].map = SeqMap{c0, c1, walk ? kMapWalk : e, 0};
    }
    __syncthreads();
}

// 3. per chunk: 53-bit grid TV and sum of squared weights (partial sums), in the located chunk the
//    element search with its certification, and on request (maps) the sequential CDF's maps.  The three
//    need the same prefix sums of the chunk's weights.
__global__ void __launch_bounds__(kThreads, 3)  // (3 of them per SM: 64 blocks of 2^14 take 4 us longer with 2)
k_chunk(const double* w, int k, const dd* chunk_sum, int nch, const BlockState* state, dcs_draw_result* res, double* part,
        double* sq_part, SeqChunk* chunk_map, SeqMap* sub_map, int maps) {
    let_next_start();
    after_previous();
    const int b = blockIdx.y;
    const int c = blockIdx.x;
    const uint64_t n = 1ull << k;
    if (state[b].status) return;
    const dd T = state[b].total;
    const double mass = T.hi;
    const uint64_t start = (uint64_t)c * kChunk;
    const double* wb = w + ((uint64_t)b << k);
    double loc[kPer];
    dd acc{0.0, 0.0};
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint64_t i = start + (uint64_t)threadIdx.x * kPer + j;
        loc[j] = i < n ? wb[i] : 0.0;
        acc = dd_add(acc, loc[j]);
    }
    dd total;
    const dd before = block_scan_dd(acc, chunk_sum[(uint64_t)b * nch + c], &total);
    if (maps)
        chunk_maps(loc, before.hi, n, c, nch, chunk_map + (uint64_t)b * nch,
                   sub_map + (uint64_t)b * (n >= (uint64_t)kSub ? n / kSub : 1));
    dd run = before;
    const double two53 = 9007199254740992.0;
    // quotients by the total (> 0); totals whose reciprocal is infinite, subnormal or near it are scaled, exactly
    const double up = T.hi < 0x1p-900 ? 0x1p600 : T.hi > 0x1p900 ? 0x1p-600 : 1.0;
    const dd Ts{T.hi * up, T.lo * up};
    const double inv = 1.0 / Ts.hi;
    auto share = [&](dd a) {
        if (up != 1.0) a = dd{a.hi * up, a.lo * up};
        return dd_div(a, Ts, inv);
    };
    double prev_end = ceil(share(run) * two53);
    if (start + (uint64_t)threadIdx.x * kPer == 0) prev_end = 0.0;
    double s = 0.0, q = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint64_t i = start + (uint64_t)threadIdx.x * kPer + j;
        if (i >= n) break;
        run = dd_add(run, loc[j]);
        const double ci = (i == n - 1) ? 1.0 : share(run);
        const double end = ceil(ci * two53);
        const double p = loc[j] / mass;
        s += fabs((end - prev_end) / two53 - p);
        q = fma(p, p, q);
        prev_end = end;
    }
    const dd tot = block_sum_dd(dd{s, 0.0});
    const dd sq = block_sum_dd(dd{q, 0.0});
    if (threadIdx.x == 0) {
        part[(uint64_t)b * nch + c] = tot.hi + tot.lo;
        sq_part[(uint64_t)b * nch + c] = sq.hi + sq.lo;
    }
    if (c != state[b].chunk) return;
    // element search inside the located chunk: the first i with P_i > target wins
    const double u = res[b].uniform;
    const dd target = dd_mul(T, u);
    int found = -1;
    dd p_before{0, 0}, p_at{0, 0};
    double wi = 0.0;
    run = before;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const dd nxt = dd_add(run, loc[j]);
        if (found < 0 && loc[j] > 0.0 && dd_lt(target, nxt)) {
            found = (int)threadIdx.x * kPer + j;
            p_before = run;
            p_at = nxt;
            wi = loc[j];
        }
        run = nxt;
    }
    __shared__ int best;
    if (threadIdx.x == 0) best = INT32_MAX;
    __syncthreads();
    if (found >= 0) atomicMin(&best, found);
    __syncthreads();
    dcs_draw_result& r = res[b];
    if (found >= 0 && found == best) {
        const uint64_t i = start + found;
        // math.fsum rounds each sum to double before the division (sampling_protocol.py:67-69);
        // a normalised double-double's high word is that rounding
        const double lo = __ddiv_rn(p_before.hi, T.hi), hi = __ddiv_rn(p_at.hi, T.hi);
        r.index = (int64_t)i;
        r.selected_weight = wi;
        r.total_exact = T.hi;
        r.total_cdf = r.total_exact;
        r.cdf_lower_exact = lo;
        r.cdf_upper_exact = hi;
        r.cdf_lower = i ? lo : 0.0;
        r.cdf_upper = (i == n - 1) ? 1.0 : hi;
        // certification against numpy's sequential cumsum (bound on each side + 4 ulp slack)
        const double eps = 1.1102230246251565e-16;  // 2^-53
        const double rel = ((double)i + (double)n + 8.0) * eps;
        const bool low_ok = i == 0 || lo * (1.0 + rel) <= u;
        const bool high_ok = (i == n - 1) || hi * (1.0 - rel) > u;
        r.tie = !(low_ok && high_ok);
        r.status = 0;
    }
    if (threadIdx.x == 0 && best == INT32_MAX) {
        // u*T beyond every accurate prefix (possible only within rounding of T): sequential path decides
        r.tie = 1;
        r.total_exact = T.hi;
    }
}

// Inclusive scan of maps over a warp's lanes (lane 0 first): d0 / d1 become the increments from before lane 0.
__device__ __forceinline__ void map_scan(long long& d0, long long& d1) {
    const int lane = threadIdx.x & 31;
    if (__all_sync(0xffffffffu, d0 == d1)) {  // no ties, as almost always: a sum (a third of the general scan's time)
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const long long a = __shfl_up_sync(0xffffffffu, d0, off);
            if (lane >= off) d0 += a;
        }
        d1 = d0;
        return;
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        long long a0 = __shfl_up_sync(0xffffffffu, d0, off), a1 = __shfl_up_sync(0xffffffffu, d1, off);
        map_then(a0, a1, d0, d1);
        if (lane >= off) {
            d0 = a0;
            d1 = a1;
        }
    }
}
__device__ __forceinline__ int exponent_of(long long bits) { return (int)(bits >> 52) - 1023; }

// S (its bit pattern, the same in every lane) through the maps of lanes pos .. stop - 1, the longest run whose
// maps hold for S's binade; returns stop <= cnt.  `start` receives S before the lane's stretch for lanes pos ..
// stop.  S of one binade is an integer in its bit pattern, so an increment is an integer addition.
__device__ __forceinline__ int seq_run(long long& S, const SeqMap& m, int pos, int cnt, double& start) {
    const int lane = threadIdx.x & 31;
    const int es = exponent_of(S);
    const bool here = lane >= pos && lane < cnt;
    const unsigned bad = __ballot_sync(0xffffffffu, here && m.e != kMapNone && m.e != es);  // kMapWalk: always
    int stop = bad ? __ffs(bad) - 1 : cnt;
    long long d0 = 0, d1 = 0;
    if (here && lane < stop && m.e != kMapNone) {
        d0 = m.d0;
        d1 = m.d1;
    }
    map_scan(d0, d1);
    const long long after = S + ((S & 1) ? d1 : d0);
    long long before = __shfl_up_sync(0xffffffffu, after, 1);
    if (lane == 0) before = S;
    // (maps are made only where S cannot leave the binade; were it to, the stretch would be walked)
    const unsigned left = __ballot_sync(0xffffffffu, here && lane < stop && m.e != kMapNone && exponent_of(after) != es);
    if (left) stop = __ffs(left) - 1;
    if (lane >= pos && lane <= stop) start = __longlong_as_double(before);
    if (stop > pos) S = __shfl_sync(0xffffffffu, after, stop - 1);
    return stop;
}

// S after the weights [i0, i1) of one sub-chunk (one warp, the same S in every lane); out: optional array for S after
// each.  Four consecutive weights per lane; their maps in S's binade are scanned, the first weight that leaves the
// binade is added itself, and the rest goes on in the new one: two scans where 128 dependent additions (2600
// cycles) were.
__device__ __forceinline__ double seq_walk(const double* wb, uint64_t i0, uint64_t i1, double S0, double* out) {
    constexpr int kOwn = kSub / 32;
    const int lane = threadIdx.x & 31;
    const int n = (int)(i1 - i0);
    double v[kOwn];
#pragma unroll
    for (int r = 0; r < kOwn; ++r) {
        const int i = lane * kOwn + r;
        v[r] = i < n ? wb[i0 + i] : 0.0;  // adding zero changes nothing
    }
    int pos = 0;
    if (i0 == 0) {  // the sum of the first few weights leaves a binade with nearly every one
        const int lim = n < 16 ? n : 16;
        for (; pos < lim; ++pos) {
            double w = v[0];
#pragma unroll
            for (int r = 1; r < kOwn; ++r)
                if (r == (pos & (kOwn - 1))) w = v[r];
            S0 = __dadd_rn(S0, __shfl_sync(0xffffffffu, w, pos / kOwn));
            if (out && lane == 0) out[pos] = S0;
        }
    }
    long long S = __double_as_longlong(S0);
    while (pos < n) {
        const int es = exponent_of(S);
        int at = pos;  // the weight to add itself
        if (es < 1000) {
            const double even = __hiloint2double((es + 1023) << 20, 0), odd = __hiloint2double((es + 1023) << 20, 1);
            long long c0[kOwn], c1[kOwn], d0 = 0, d1 = 0;
#pragma unroll
            for (int r = 0; r < kOwn; ++r) {
                if (lane * kOwn + r >= pos)
                    map_then(d0, d1, __double_as_longlong(__dadd_rn(even, v[r])) - __double_as_longlong(even),
                             __double_as_longlong(__dadd_rn(odd, v[r])) - __double_as_longlong(odd));
                c0[r] = d0;
                c1[r] = d1;
            }
            map_scan(d0, d1);
            long long e0 = __shfl_up_sync(0xffffffffu, d0, 1), e1 = __shfl_up_sync(0xffffffffu, d1, 1);
            if (lane == 0) e0 = e1 = 0;
            const long long before = S + ((S & 1) ? e1 : e0);  // before the lane's weights
            long long k[kOwn];
            int first = kOwn;
#pragma unroll
            for (int r = kOwn - 1; r >= 0; --r) {
                k[r] = before + ((before & 1) ? c1[r] : c0[r]);
                const int i = lane * kOwn + r;
                if (i >= pos && i < n && ((v[r] >= even && even > 0.0) || exponent_of(k[r]) != es)) first = r;
            }
            const unsigned any = __ballot_sync(0xffffffffu, first < kOwn);
            const int who = any ? __ffs(any) - 1 : 31;
            const int r0 = __shfl_sync(0xffffffffu, first, who);
            at = any ? who * kOwn + r0 : n;
            if (out) {
#pragma unroll
                for (int r = 0; r < kOwn; ++r) {
                    const int i = lane * kOwn + r;
                    if (i >= pos && i < at && i < n) out[i] = __longlong_as_double(k[r]);
                }
            }
            // S before the weight `at` (after all of them when there is none)
            long long prev = before;
#pragma unroll
            for (int r = 0; r < kOwn; ++r)
                if (r < r0) prev = k[r];
            S = __shfl_sync(0xffffffffu, prev, who);
        }
        if (at < n) {
            double w = 0.0;
#pragma unroll
            for (int r = 0; r < kOwn; ++r)
                if (r == (at & (kOwn - 1))) w = v[r];
            w = __shfl_sync(0xffffffffu, w, at / kOwn);
            const double s = __dadd_rn(__longlong_as_double(S), w);
            if (out && lane == 0) out[at] = s;
            S = __double_as_longlong(s);
        }
        pos = at + 1;
    }
    return __longlong_as_double(S);
}

// S after chunk c from S before it (one warp); sub_start: optional array for S before each of its sub-chunks
__device__ __forceinline__ double seq_chunk(const double* wb, uint64_t n, uint64_t c, const SeqMap* sub_map, double S0, double* sub_start) {
    const int lane = threadIdx.x & 31;
    const uint64_t g0 = c * kSubs;
    const uint64_t left = ((n - c * kChunk) + kSub - 1) / kSub;
    const int cnt = left < kSubs ? (int)left : kSubs;
    SeqMap mine{0, 0, kMapNone, 0};
    if (lane < cnt) mine = sub_map[g0 + lane];
    long long S = __double_as_longlong(S0);
    double start = 0.0;
    for (int pos = 0; pos < cnt;) {
        const int stop = seq_run(S, mine, pos, cnt, start);
        if (stop < cnt) {
            const uint64_t i0 = (g0 + stop) * kSub;
            S = __double_as_longlong(seq_walk(wb, i0, i0 + kSub < n ? i0 + kSub : n, __longlong_as_double(S), nullptr));
        }
        pos = stop + 1;
    }
    if (sub_start && lane < cnt) sub_start[lane] = start;
    return __longlong_as_double(S);
}

// 4. totals of the chunk sums, and the exact sequential FP64 CDF (numpy's operation order) for blocks
//    flagged as ties, or for every block when `force` (one CTA per block).  Warp 0 carries S over runs of
//    chunks by scanning their maps; chunks that cross a binade (about log2 of the block size of them) go through
//    their sub-chunks' maps, and the one or two sub-chunks that cross through their weights'.
//    The chain of n dependent additions this replaces took 10.9 ms for 2^20 weights; chunk by chunk, with
//    dependent additions in the sub-chunks that cross, the kernel took 93 us, and by runs and scans 53.  The
//    selected chunk (and sub-chunk) is the last one whose starting value satisfies fl(start / S_n) <= u
//    (fl(x / S_n) is non-decreasing in x), and only the selected sub-chunk is replayed.  The compensated
//    interval of the selected index is checked against u as the reference's independent check does
//    (sampling_protocol.py:67-72).
__global__ void __launch_bounds__(kThreads)
k_finish(const double* w, int k, const dd* chunk_sum, int nch, const BlockState* state, dcs_draw_result* res,
         const double* part, const double* sq_part, SeqChunk* chunk_map, SeqMap* sub_map, int force) {
    after_previous();
    const int b = blockIdx.x;
    const int lane = threadIdx.x & 31;
    dcs_draw_result& r = res[b];
    if (state[b].status) return;
    double s = 0.0, q = 0.0;
    for (int c = threadIdx.x; c < nch; c += kThreads) {
        s += part[(uint64_t)b * nch + c];
        q += sq_part[(uint64_t)b * nch + c];
    }
    const dd ts = block_sum_dd(dd{s, 0.0}), tq = block_sum_dd(dd{q, 0.0});
    if (threadIdx.x == 0) {
        r.tv53 = 0.5 * (ts.hi + ts.lo);
        r.weight_l2 = tq.hi + tq.lo;
    }
    if (!(r.tie || force)) return;
    const uint64_t n = 1ull << k;
    const double* wb = w + ((uint64_t)b << k);
    const dd* cs = chunk_sum + (uint64_t)b * nch;
    SeqChunk* cm = chunk_map + (uint64_t)b * nch;
    SeqMap* sb = sub_map + (uint64_t)b * (n >= (uint64_t)kSub ? n / kSub : 1);
    __shared__ double s_total, sub_start[kSubs], seq[kSub];
    __shared__ int at;
    if (!force) {  // a tie found by the search: the maps were not made with the chunk sums
        for (int c = 0; c < nch; ++c) {
            double loc[kPer];
            dd acc{0.0, 0.0};
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const uint64_t i = (uint64_t)c * kChunk + (uint64_t)threadIdx.x * kPer + j;
                loc[j] = i < n ? wb[i] : 0.0;
                acc = dd_add(acc, loc[j]);
            }
            dd total;
            const dd before = block_scan_dd(acc, cs[c], &total);
            chunk_maps(loc, before.hi, n, c, nch, cm, sb);
        }
    }
    if (threadIdx.x == 0) at = 0;
    __syncthreads();
    if (threadIdx.x < 32) {
        long long S = 0;
        SeqMap next{0, 0, kMapNone, 0};
        if (lane < nch) next = cm[lane].map;
        for (int c0 = 0; c0 < nch; c0 += 32) {
            const SeqMap mine = next;
            if (c0 + 32 + lane < nch) next = cm[c0 + 32 + lane].map;  // on its way while these are scanned
            double start = 0.0;
            const int cnt = nch - c0 < 32 ? nch - c0 : 32;
            for (int pos = 0; pos < cnt;) {
                const int stop = seq_run(S, mine, pos, cnt, start);
                if (stop < cnt)
                    S = __double_as_longlong(seq_chunk(wb, n, c0 + stop, sb, __longlong_as_double(S), nullptr));
                pos = stop + 1;
            }
            if (c0 + lane < nch) cm[c0 + lane].start = start;
        }
        if (lane == 0) s_total = __longlong_as_double(S);
    }
    __syncthreads();
    const double S = s_total;
    if (!(S > 0.0) || !isfinite(S)) {
        if (threadIdx.x == 0) r.status = DCS_E_CDF;
        return;
    }
    const double u = r.uniform;
    // last chunk whose starting value's quotient is <= u (chunk 0 starts at 0)
    int mine = 0;
    for (int c = threadIdx.x; c < nch; c += kThreads)
        if (__ddiv_rn(cm[c].start, S) <= u) mine = c;
    if (mine) atomicMax(&at, mine);
    __syncthreads();
    const uint64_t c = at;
    __shared__ int64_t s_idx;
    if (threadIdx.x < 32) {
        seq_chunk(wb, n, c, sb, cm[c].start, sub_start);
        __syncwarp();
        const bool is = lane < kSubs && (c * kSubs + lane) * kSub < n && __ddiv_rn(sub_start[lane], S) <= u;
        const unsigned m = __ballot_sync(0xffffffffu, is);
        const int j = m ? 31 - __clz(m) : 0;
        // replay the sub-chunk; the last element's value is forced to 1 (numpy: cumulative[-1] = 1)
        const uint64_t i0 = (c * kSubs + j) * kSub, i1 = i0 + kSub < n ? i0 + kSub : n;
        const double S0 = sub_start[j];
        seq_walk(wb, i0, i1, S0, seq);
        __syncwarp();
        int hit = kSub;
#pragma unroll
        for (int p = kSub / 32 - 1; p >= 0; --p) {
            const uint64_t i = i0 + p * 32 + lane;
            if (i < i1 && u < ((i == n - 1) ? 1.0 : __ddiv_rn(seq[p * 32 + lane], S))) hit = p * 32 + lane;
        }
        for (int off = 16; off > 0; off >>= 1) hit = min(hit, __shfl_xor_sync(0xffffffffu, hit, off));
        if (lane == 0) {
            const uint64_t idx = hit < kSub ? i0 + hit : n - 1;
            double prev = 0.0, upper = 1.0;
            if (hit < kSub) {
                prev = __ddiv_rn(hit ? seq[hit - 1] : S0, S);
                upper = (idx == n - 1) ? 1.0 : __ddiv_rn(seq[hit], S);
            } else {
                prev = __ddiv_rn(seq[i1 - 1 - i0], S);
            }
            s_idx = (int64_t)idx;
            r.cdf_lower = idx ? prev : 0.0;
            r.cdf_upper = upper;
        }
    }
    __syncthreads();
    const uint64_t idx = (uint64_t)s_idx;
    // compensated prefix before idx: the scan's chunk prefix plus the chunk's elements before idx
    const uint64_t ci = idx / kChunk;
    dd acc{0.0, 0.0};
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const uint64_t i = ci * kChunk + (uint64_t)threadIdx.x * kPer + j;
        if (i < idx) acc = dd_add(acc, wb[i]);
    }
    const dd pre = dd_add(cs[ci], block_sum_dd(acc));
    if (threadIdx.x) return;
    const double wi = wb[idx];
    const dd T = state[b].total;
    r.cdf_lower_exact = __ddiv_rn(pre.hi, T.hi);
    r.cdf_upper_exact = __ddiv_rn(dd_add(pre, wi).hi, T.hi);
    r.index = (int64_t)idx;
    r.total_cdf = S;
    r.total_exact = T.hi;
    r.selected_weight = wi;
    if (!(wi > 0.0)) r.status = DCS_E_CDF;
    // the reference's independent check of the interval (a disagreement is an error, never a resample)
    else if (!(r.cdf_lower_exact <= u && u < r.cdf_upper_exact)) r.status = DCS_E_CDF;
}

// ---------------------------------------------------------------- audit overlap
constexpr int kOverlapParts = kThreads;  // partial sums, one CTA each: 16 KiB of scratch

__global__ void __launch_bounds__(kThreads)
k_overlap(const double2* __restrict__ ref, const double2* __restrict__ ap, uint64_t len, dd* __restrict__ part) {
    let_next_start();
    constexpr int kIn = 4;  // entries in flight per thread: one at a time left the loads' latency exposed
    dd rr{0, 0}, aa{0, 0}, re{0, 0}, im{0, 0};
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += kIn * stride) {
        double2 r[kIn], a[kIn];
#pragma unroll
        for (int j = 0; j < kIn; ++j)
            if (i + j * stride < len) {
                r[j] = ref[i + j * stride];
                a[j] = ap[i + j * stride];
            }
#pragma unroll
        for (int j = 0; j < kIn; ++j)
            if (i + j * stride < len) {
                rr = dd_add(rr, r[j].x * r[j].x + r[j].y * r[j].y);
                aa = dd_add(aa, a[j].x * a[j].x + a[j].y * a[j].y);
                re = dd_add(re, r[j].x * a[j].x + r[j].y * a[j].y);   // <ref, ap> = sum conj(ref) * ap
                im = dd_add(im, r[j].x * a[j].y - r[j].y * a[j].x);
            }
    }
    rr = block_sum_dd(rr);
    aa = block_sum_dd(aa);
    re = block_sum_dd(re);
    im = block_sum_dd(im);
    if (threadIdx.x == 0) {
        part[4 * blockIdx.x + 0] = rr;
        part[4 * blockIdx.x + 1] = aa;
        part[4 * blockIdx.x + 2] = re;
        part[4 * blockIdx.x + 3] = im;
    }
}

// A thread per partial sum (four threads walking the 256 of them took 24 us, the first pass 9).
__global__ void __launch_bounds__(kThreads)
k_overlap_final(const dd* part, double* out) {
    after_previous();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const dd s = block_sum_dd(part[4 * threadIdx.x + q]);
        if (threadIdx.x == 0) out[q] = s.hi + s.lo;
    }
}

}  // namespace

extern "C" size_t dcs_draw_scratch_bytes(int k, int nblocks) {
    if (k < 0 || k > 30 || nblocks < 1) return 0;
    return layout(k, nblocks).bytes;
}

namespace {
// the draw kernels on a scratch area laid out by layout(k, nblocks)
int enqueue_draw(const double* blocks, int k, int nblocks, const double* uniforms, unsigned flags, void* scratch,
                 dcs_draw_result* results, cudaStream_t s) {
    const Layout L = layout(k, nblocks);
    char* base = (char*)scratch;
    double* w = (double*)(base + L.w);
    dd* cs = (dd*)(base + L.chunk_sum);
    BlockState* st = (BlockState*)(base + L.state);
    double* part = (double*)(base + L.tv_part);
    double* sq = (double*)(base + L.sq_part);
    SeqChunk* cm = (SeqChunk*)(base + L.chunk_map);
    SeqMap* sm = (SeqMap*)(base + L.sub_map);
    const uint64_t n = 1ull << k;
    const int nch = (int)(n >= (uint64_t)kChunk ? n / kChunk : 1);
    const int force = (flags & DCS_DRAW_SEQUENTIAL) ? 1 : 0;
    k_weights<<<dim3(nch, nblocks), kThreads, 0, s>>>((const double2*)blocks, k, w, cs, part);
    DCS_CHECK_LAUNCH("k_weights");
    // (what these read is written by the launch before, which may still run when they start: none of their
    // pointers is declared read-only)
    using dcs_host::check_cuda;
    using dcs_host::launch_after;
    int rc = check_cuda(launch_after(k_scan_locate, dim3(nblocks), dim3(kThreads), 0, s, cs, nch, uniforms, st, results, part),
                        "k_scan_locate");
    if (!rc)
        rc = check_cuda(launch_after(k_chunk, dim3(nch, nblocks), dim3(kThreads), 0, s, w, k, cs, nch, st, results, part, sq, cm,
                                     sm, force),
                        "k_chunk");
    if (!rc)
        rc = check_cuda(launch_after(k_finish, dim3(nblocks), dim3(kThreads), 0, s, w, k, cs, nch, st, results, part, sq, cm, sm,
                                     force),
                        "k_finish");
    return rc;
}
}  // namespace

extern "C" int dcs_draw_ex(const double* blocks, int k, int nblocks, const double* uniforms, unsigned flags,
                           void* scratch, dcs_draw_result* results, void* stream) {
    if (!blocks || !uniforms || !scratch || !results || k < 0 || k > 30 || nblocks < 1 || nblocks > 65535 ||
        (flags & ~(unsigned)DCS_DRAW_SEQUENTIAL)) {
        dcs_host::set_error("dcs_draw: invalid arguments");
        return DCS_E_ARG;
    }
    return enqueue_draw(blocks, k, nblocks, uniforms, flags, scratch, results, (cudaStream_t)stream);
}

extern "C" int dcs_draw(const double* blocks, int k, int nblocks, const double* uniforms, void* scratch,
                        dcs_draw_result* results, void* stream) {
    return dcs_draw_ex(blocks, k, nblocks, uniforms, 0u, scratch, results, stream);
}

extern "C" int dcs_overlap(const double* ref, const double* ap, uint64_t len, double* out, void* scratch,
                           void* stream) {
    if (!ref || !ap || !out || !scratch || len == 0) {
        dcs_host::set_error("dcs_overlap: invalid arguments");
        return DCS_E_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    k_overlap<<<kOverlapParts, kThreads, 0, s>>>((const double2*)ref, (const double2*)ap, len, (dd*)scratch);
    DCS_CHECK_LAUNCH("k_overlap");
    return dcs_host::check_cuda(dcs_host::launch_after(k_overlap_final, dim3(1), dim3(kThreads), 0, s, (const dd*)scratch, out),
                                "k_overlap_final");
}

// ---------------------------------------------------------------- draw without allocation
//
// For callers that cannot allocate device memory at the point where they draw: code that runs
// while a CUDA stream is being captured (cudaMalloc cannot be captured), host runtimes that
// hand the library only the buffers they own and forbid allocation in their sampling loop, and
// latency-sensitive loops where an allocation would synchronise the device.  The scratch lives
// in a file-scope device array of fixed size, so this entry point allocates nothing.
//
// Limit: one block of up to 2^20 amplitudes per call (DCS_DRAW_STATIC_MAX_K); every GPU that
// loads the library holds the array (about 8.3 MiB) until the process exits.
namespace {
constexpr size_t kStaticDrawBytes = layout(DCS_DRAW_STATIC_MAX_K, 1).bytes;
static __device__ __align__(256) unsigned char g_draw_scratch[kStaticDrawBytes];

// The device address of g_draw_scratch, looked up once per device with that device current,
// and the context it was looked up in: a new context on the device (after cudaDeviceReset, or
// a context torn down and created again) loads the module elsewhere, so the lookup is redone.
std::mutex g_static_mutex;
void* g_static_ptr[64] = {nullptr};
void* g_static_ctx[64] = {nullptr};
typedef CUresult (*ctx_get_current_fn)(CUcontext*);

int current_context(void** ctx) {
    static ctx_get_current_fn fn = nullptr;
    if (!fn) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !f) {
            dcs_host::set_error("dcs_draw_static: cuCtxGetCurrent is not available");
            return DCS_E_CUDA;
        }
        fn = (ctx_get_current_fn)f;
    }
    CUcontext c = nullptr;
    if (fn(&c) != CUDA_SUCCESS) {
        dcs_host::set_error("dcs_draw_static: cuCtxGetCurrent failed");
        return DCS_E_CUDA;
    }
    *ctx = (void*)c;
    return DCS_OK;
}
}  // namespace

extern "C" int dcs_draw_static(const double* blocks, int k, const double* uniform, dcs_draw_result* result,
                               void* stream) {
    if (!blocks || !uniform || !result || k < 0 || k > 30) {
        dcs_host::set_error("dcs_draw_static: invalid arguments");
        return DCS_E_ARG;
    }
    const Layout L = layout(k, 1);
    if (k > DCS_DRAW_STATIC_MAX_K || L.bytes > kStaticDrawBytes) {
        dcs_host::set_error("dcs_draw_static: block of 2^%d amplitudes exceeds the static maximum of 2^%d", k,
                            DCS_DRAW_STATIC_MAX_K);
        return DCS_E_ARG;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return dcs_host::check_cuda(e, "dcs_draw_static: cudaGetDevice");
    if (dev < 0 || dev >= 64) {
        dcs_host::set_error("dcs_draw_static: device index %d out of range", dev);
        return DCS_E_ARG;
    }
    void* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_mutex);
        void* ctx = nullptr;
        const int rc = current_context(&ctx);
        if (rc != DCS_OK) return rc;
        if (!g_static_ptr[dev] || g_static_ctx[dev] != ctx) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_draw_scratch);
            if (e != cudaSuccess) return dcs_host::check_cuda(e, "dcs_draw_static: cudaGetSymbolAddress");
            g_static_ptr[dev] = p;
            g_static_ctx[dev] = ctx;
        }
        scratch = g_static_ptr[dev];
    }
    return enqueue_draw(blocks, k, 1, uniform, 0u, scratch, result, (cudaStream_t)stream);
}
