// Groups of vertex steps over coset tiles in shared memory, for every work item of a batch
// (complex64 tables with FP32 arithmetic, complex128 tables with FP64 arithmetic; sm_100a).
//
// One launch = one group of consecutive vertex steps (fused.py has the tile algebra) on nitems tables
// that share the plan.  A CTA holds one tile of one item in shared memory: the tile's entries
// that are active before the group come in once, every step of the group runs on them, and the
// entries active after the group go out once.  This is the executor of the engine's "device" mode:
// one launch per vertex step (k_step) costs a pass over the table, a launch and the gap to the
// next one for each of the 30 to 400 steps of a plan, and most plans' tables are so small that the
// launch and the gap are most of it.
//
// Bound: instruction issue (68% of the issue slots on 16 items of 1024 tiles of 2^12 entries, 22 instructions per
// active entry and step); with a tile per SM or less, the latency of a step (two shared-memory accesses, the
// products and a barrier).  A slice, device work and enqueueing, against one launch per step: 40 qubits (2^22
// entries, 213 steps in 13 groups) 911 -> 281 us, 48 qubits (2^24) 1414 -> 560 us, in complex128 2044 ->
// 703 us; 16 slices of 40 qubits in one batch 4545 -> 1563 us.
//
// The orbit formulas are k_step's operation by operation (same products, same fused multiply-adds,
// same order of additions).  The power of two of the renormalisation is applied once per group (exact).
// In complex64 every step's maximum is taken all the same, and the exponents that one launch per
// step would have used follow from them (e of step t = exponent of the maximum before it minus that of
// the step before), are added to the item's logscale in step order, and the part that the table does not
// have goes into table_exp: a block has the bits of the per-step executor's (13% of a group's time), and
// so have the draws and the 53-bit distances that depend on every bit of it.  In complex128 a group takes one
// maximum (per-step ones cost 18%); the logscale then is a shorter sum of the same numbers, and the block
// differs from the per-step executor's in that factor's rounding only.  Cancellation in a group can take the
// squares of a table that is not zero below their type's range: that sets kFlagRange, and the host runs the batch
// again with a launch per step.  The host keeps step weights out of
// here that could let a group's entries, or in complex64 their squares, overflow (engine.tile_weights_ok,
// tile_growth_ok).
#include <string.h>

#include "common.cuh"

using namespace dcs;

namespace {

constexpr int kMaxSteps = 24;
constexpr int kMaxDim = 12;   // 32 KiB (complex64) or 64 KiB per tile
constexpr int kManyTiles = 4;  // tiles per SM from which on 128 threads take one (run_groups)
constexpr int kHalfDim = 13;  // binary16 tables: 32 KiB

struct TileStep {
    uint64_t beta, cskip;
    uint32_t tK, tKa, tpiv, tbeta;
    uint8_t kind, sK, sKa, nins;
    uint8_t ins[16];
};

struct TileArgs {
    int32_t count, first, tile_dim, low_bits, coset_m, ncoset_runs;
    int32_t prev_first;  // first step of the group before (-1: none)
    int32_t last;        // the plan's last group
    uint64_t in_inactive, out_inactive;
    uint64_t basis[16];
    uint32_t coset_runs[DCS_MAX_RUNS];
    TileStep st[kMaxSteps];
};

__device__ __forceinline__ uint32_t insert0(uint32_t o, int p) {
    return ((o >> p) << (p + 1)) | (o & ((1u << p) - 1u));
}

__device__ __forceinline__ float2 c2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 c2(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
template <class S> __device__ __forceinline__ S zadd(S a, S b) { return c2(radd(a.x, b.x), radd(a.y, b.y)); }
// a + g b, g = +-1 (one rounding, as the addition of the negated value)
template <class S, class R> __device__ __forceinline__ S zaddg(S a, R g, S b) { return c2(rfma(g, b.x, a.x), rfma(g, b.y, a.y)); }
// f x, with the roundings that k_step's products have
template <class S> __device__ __forceinline__ S zmul(S f, S x) {
    return c2(rfma(f.x, x.x, -rmul(f.y, x.y)), rfma(f.y, x.x, rmul(f.x, x.y)));
}
// the same for a fixed step without a sum, whose product k_step rounds the other way round in the imaginary part
template <class S> __device__ __forceinline__ S zmulf(S f, S x) {
    return c2(rfma(f.x, x.x, -rmul(f.y, x.y)), rfma(f.x, x.y, rmul(f.y, x.x)));
}

template <class S> struct Weights {
    S f0, f1, fp, fm;  // f0 + f1, f0 - f1
};

// whether every step's maximum is taken (else the group's)
template <class M> constexpr bool kStepMax = sizeof(M) <= 8;

constexpr uint32_t kSign = 0x80000000u;
// +-1 by bit 31 of x
__device__ __forceinline__ float sign_of(uint32_t x, float) { return __uint_as_float((x & kSign) | 0x3f800000u); }
__device__ __forceinline__ double sign_of(uint32_t x, double) { return __hiloint2double((int)((x & kSign) | 0x3ff00000u), 0); }
// a with its sign flipped where m has bit 31
__device__ __forceinline__ float flip1(float a, uint32_t m) { return __uint_as_float(__float_as_uint(a) ^ m); }
__device__ __forceinline__ double flip1(double a, uint32_t m) {
    return __hiloint2double(__double2hiint(a) ^ (int)m, __double2loint(a));
}
// zero only for +-0
__device__ __forceinline__ uint32_t nonzero_bits(float2 v) { return (__float_as_uint(v.x) | __float_as_uint(v.y)) & ~kSign; }
__device__ __forceinline__ uint32_t nonzero_bits(double2 v) {
    return ((uint32_t)(__double2hiint(v.x) | __double2hiint(v.y)) & ~kSign) | (uint32_t)(__double2loint(v.x) | __double2loint(v.y));
}
template <class S> __device__ __forceinline__ S flip(S a, uint32_t m) { return c2(flip1(a.x, m), flip1(a.y, m)); }

// Words per step of the spread tables: 16 for bits 0-3 of the thread, then its other bits, then the orbit
// slots of a thread.
template <int NT, int DIM = kMaxDim> struct Tab {
    static constexpr int kHi = 16, kOrb = kHi + NT / 16, kWords = kOrb + (1 << DIM) / NT;
};

// One vertex step over the active orbit representatives of the tile.  Representatives are the tile
// indices with zero bits at ins[]: the role slots and the tile bits of slots inactive at this step.  The
// index o = thread + NT u is spread over the other bits, a linear map, and so is the sign
// parity(t & beta): `tab` has both for parts of o (byte offset, sign in bit 31), and one XOR of three words
// gives an orbit's offset and sign.  (Spreading and counting bits per orbit took 31 instructions per entry
// and step instead of 20.)  Signs enter as factors +-1 of a fused multiply-add, which round as the
// addition of the negated value does.
template <class S, int KIND, int NT, class M = S>
__device__ __forceinline__ typename Mem<S, M>::Q run_step(unsigned char* __restrict__ sh, int T, const TileStep& st,
                                                         const uint32_t* __restrict__ tab, const Weights<S>& w,
                                                         uint32_t cs, int y) {
    using R = typename Store<S>::R;
    using IO = Mem<S, M>;
    constexpr int SH = sizeof(M) == 4 ? 2 : (sizeof(M) == 8 ? 3 : 4);
    const int nrep = T >> st.nins;
    if ((int)threadIdx.x >= nrep) return 0;
    const uint32_t tp = tab[threadIdx.x & 15] ^ tab[Tab<NT>::kHi + (threadIdx.x >> 4)] ^ (cs << 31);
    const uint32_t tK = st.tK << SH, tKa = st.tKa << SH, tpiv = st.tpiv << SH;
    const int niter = nrep > NT ? nrep / NT : 1;
    const R gK = st.sK ? (R)-1 : (R)1;
    const S f0 = w.f0, f1 = w.f1;
    const S f1a = flip(f1, st.sKa ? kSign : 0u);  // f1 (-1)^sKa
    const S fp = w.fp, fm = w.fm, fp2 = st.sK ? fm : fp, fm2 = st.sK ? fp : fm;
    const S fy = y ? f1 : f0;  // a fixed step: the weight that its value selects
    const R gy = y ? gK : (R)1;
    const uint32_t my = y ? kSign : 0u;
    auto ld = [&](uint32_t o) { return IO::ld(*reinterpret_cast<const M*>(sh + o)); };
    typename IO::Q lm = 0;
    auto stv = [&](uint32_t o, S v) {
        const typename IO::Q q = IO::st(reinterpret_cast<M*>(sh + o), 0, v);
        if constexpr (kStepMax<M>) lm = fmax(lm, q);
    };
#pragma unroll 4
    for (int u = 0; u < niter; ++u) {
        const uint32_t x = tp ^ tab[Tab<NT>::kOrb + u];
        const uint32_t t = x & ~kSign;
        const R sg = sign_of(x, (R)0);
        const S a = ld(t);
        if constexpr (KIND == DCS_KIND_GROW) {
            stv(t, zmul(f0, a));
            stv(t ^ tpiv, flip(zmul(f1, a), x & kSign));
        } else if constexpr (KIND == DCS_KIND_MIX) {
            const S b = ld(t ^ tKa);
            stv(t, zaddg(zmul(f0, a), sg, zmul(f1a, b)));
            stv(t ^ tKa, zaddg(zmul(f0, b), sg, zmul(f1, a)));
        } else if constexpr (KIND == DCS_KIND_DIAG) {
            stv(t, zmul(x & kSign ? fm : fp, a));
        } else if constexpr (KIND == DCS_KIND_REPLACE) {
            const S b = ld(t ^ tK);
            stv(t, zmul(f0, zadd(a, b)));
            stv(t ^ tK, flip(zmul(f1, zaddg(a, gK, b)), x & kSign));
        } else if constexpr (KIND == DCS_KIND_FIXED) {
            stv(t, flip(zmulf(fy, a), x & my));
        } else if constexpr (KIND == DCS_KIND_FIXED_SHRINK) {
            const S b = ld(t ^ tK);
            stv(t, flip(zmul(fy, zaddg(a, gy, b)), x & my));
        } else if constexpr (KIND == DCS_KIND_SHRINK4) {
            const S b = ld(t ^ tK), g = ld(t ^ tKa), h = ld(t ^ tK ^ tKa);
            stv(t, zaddg(zmul(f0, zadd(a, b)), sg, zmul(f1a, zaddg(g, gK, h))));
            stv(t ^ tKa, zaddg(zmul(f0, zadd(g, h)), sg, zmul(f1, zaddg(a, gK, b))));
        } else {  // DCS_KIND_SHRINK2
            const S b = ld(t ^ tK);
            stv(t, zadd(zmul(x & kSign ? fm : fp, a), zmul(x & kSign ? fm2 : fp2, b)));
        }
    }
    return lm;
}

// Adds the exponents of steps lo .. lo + n - 1 to the item's scale (one warp, n <= look <= 32): word t is the
// maximum before step t, in one scale for all of them, in which the word before lo is 1.  Words lo .. lo + look - 1
// are looked at for maxima that left the range of their type: a group is renormalised at its start only, so
// cancellation in its steps can take squares of entries that are not zero below it.
template <class R>
__device__ __forceinline__ int add_exponents(const unsigned long long* mb, int lo, int n, int look, dcs_scale* sp) {
    const int lane = threadIdx.x & 31;
    double m2 = 1.0;
    if (lane < look) m2 = (double)bits_to_m2<R>(__ldcg(mb + lo + lane));
    const int x = exponent_of_max<R>(m2);
    int e = x - __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) e = x;
    const unsigned none = __ballot_sync(0xffffffffu, m2 == 0.0);
    const unsigned some = __ballot_sync(0xffffffffu, lane < look && m2 != 0.0);
    const unsigned bad = __ballot_sync(0xffffffffu, lane < n && !isfinite(m2)), zero = n < 32 ? none & ((1u << n) - 1u) : none;
    // (a table of zeros stays one: a maximum after a zero one means that only the squares were zero)
    const bool lost = __any_sync(0xffffffffu, m2 > 0.0 && m2 < kLeastMax<R>) ||
                      (some && none & ((1u << (31 - __clz(some))) - 1u));
    double lg = sp->logscale;
    int sum = 0;
    for (int j = 0; j < n; ++j) {
        const int ej = __shfl_sync(0xffffffffu, e, j);
        lg += (double)ej * 0.69314718055994530942;  // ln 2, as the reference's e*log(2.)
        sum += ej;
    }
    if (lane == 0) {
        sp->logscale = lg;
        sp->exponent_sum += sum;
        if (bad) sp->flags |= 1u;
        if (zero) sp->flags |= 2u;
        if (lost) sp->flags |= kFlagRange;
    }
    return sum;
}

// The spread tables of every step, and the table addresses of the tile's high coordinates.
template <int NT, int DIM, int SH>
__device__ __forceinline__ void fill_tables(const TileArgs& A, uint32_t (*tab)[Tab<NT, DIM>::kWords], uint64_t* hi_tab) {
    constexpr int kTab = Tab<NT, DIM>::kWords, kHi = Tab<NT, DIM>::kHi, kOrb = Tab<NT, DIM>::kOrb;
    const uint32_t in_tile = (1u << A.tile_dim) - 1u;
    for (int i = threadIdx.x; i < A.count * kTab; i += NT) {
        const TileStep& st = A.st[i / kTab];
        const uint32_t j = i % kTab;
        uint32_t o = j < kHi ? j : j < kOrb ? (j - kHi) << 4 : (j - kOrb) * NT;
        for (int q = 0; q < st.nins; ++q) o = insert0(o, st.ins[q]);
        o &= in_tile;  // bits past the tile belong to idle threads and orbit slots
        tab[i / kTab][j] = (o << SH) | (uint32_t)(__popc(o & st.tbeta) << 31);
    }
    for (int h = threadIdx.x; h < (1 << (A.tile_dim - A.low_bits)); h += NT) {
        uint64_t a = 0;
        for (int i = 0; i < A.tile_dim - A.low_bits; ++i)
            if ((h >> i) & 1) a ^= A.basis[i];
        hi_tab[h] = a;
    }
}

template <class S, int NT>
__global__ void __launch_bounds__(NT, (sizeof(S) == 8 ? 1280 : 768) / NT)
k_tiles(S* __restrict__ table, uint64_t table_stride, const __grid_constant__ TileArgs A,
        const dcs_param* __restrict__ params, uint64_t param_stride, unsigned long long* __restrict__ maxbits,
        uint64_t maxbits_stride, dcs_scale* __restrict__ scale) {
    using R = typename Store<S>::R;
    constexpr int SH = sizeof(S) == 8 ? 3 : 4;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t tab[kMaxSteps][Tab<NT>::kWords];
    __shared__ Weights<S> fw[kMaxSteps];
    __shared__ int ovy[kMaxSteps];
    __shared__ uint32_t smax[kMaxSteps];  // per step: the CTA's maximum |x|^2 (max_key)
    const int item = blockIdx.y;
    const int T = 1 << A.tile_dim;
    const int low = A.low_bits;
    uint64_t* hi_tab = reinterpret_cast<uint64_t*>(smem + ((size_t)T << SH));
    S* E = table + (uint64_t)item * table_stride;
    unsigned long long* mb = maxbits + (uint64_t)item * maxbits_stride;

    let_next_start();
    fill_tables<NT, kMaxDim, SH>(A, tab, hi_tab);
    after_previous();  // the tables above are the plan's
    const int e = exponent_of_max<R>((double)bits_to_m2<R>(mb[A.first]));
    if (threadIdx.x < A.count) {
        const dcs_param p = params[(uint64_t)item * param_stride + A.first + threadIdx.x];
        // the pass's power of two goes into the first step's weights (exact)
        const R sc = threadIdx.x ? (R)1 : (R)exp2_neg(e);
        Weights<S> w;
        w.f0 = cscale(Store<S>::make((R)p.f0r, (R)p.f0i), sc);
        w.f1 = cscale(Store<S>::make((R)p.f1r, (R)p.f1i), sc);
        w.fp = zadd(w.f0, w.f1);
        w.fm = zadd(w.f0, c2(-w.f1.x, -w.f1.y));
        fw[threadIdx.x] = w;
        ovy[threadIdx.x] = (p.ov & 1) | ((p.y & 1) << 1);
        smax[threadIdx.x] = 0;
    }
    __syncthreads();

    const uint64_t lowmask = (1ull << low) - 1;
    const uint64_t ntiles = 1ull << A.coset_m;
    // complex64 entries t, t + 1 (t even) are one aligned 16-byte word when slot 0 is a row bit, and are
    // active together when it is active
    const bool pair = sizeof(S) == 8 && low >= 1;
    const bool pair_in = pair && !(A.in_inactive & 1), pair_out = pair && !(A.out_inactive & 1);
    R gm = 0;
    uint32_t left = 0;  // zero if every entry written is
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint64_t base = deposit(tile, A.coset_runs, A.ncoset_runs);
        auto addr = [&](int t) { return base ^ hi_tab[t >> low] ^ ((uint64_t)t & lowmask); };
        // entries active before the group (the others are written by a grow before any step reads them)
        if (pair_in) {
            for (int t = 2 * threadIdx.x; t < T; t += 2 * NT) {
                const uint64_t a = addr(t);
                if (a & A.in_inactive) continue;
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem + ((size_t)t << SH));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(E + a) : "memory");
            }
        } else {
            for (int t = threadIdx.x; t < T; t += NT) {
                const uint64_t a = addr(t);
                if (a & A.in_inactive) continue;
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem + ((size_t)t << SH));
                if constexpr (sizeof(S) == 16)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(E + a) : "memory");
                else
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(E + a) : "memory");
            }
        }
        if (tile == 0 && threadIdx.x < 32) {  // (one CTA, once, while its entries are on their way)
            const int lo = kStepMax<S> ? A.prev_first + 1 : A.first;
            add_exponents<R>(mb, lo, A.first - lo + 1, A.first - lo + 1, scale + item);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        for (int s = 0; s < A.count; ++s) {
            const TileStep& st = A.st[s];
            if (!(base & st.cskip)) {
                const uint32_t cs = (uint32_t)__popcll(base & st.beta) ^ (uint32_t)ovy[s];
                const int y = ovy[s] >> 1;
                const Weights<S>& w = fw[s];
                R lm = 0;
                switch (st.kind) {
#define DCS_CASE(K) \
    case K: lm = run_step<S, K, NT>(smem, T, st, tab[s], w, cs, y); break;
                    DCS_CASE(DCS_KIND_GROW)
                    DCS_CASE(DCS_KIND_MIX)
                    DCS_CASE(DCS_KIND_DIAG)
                    DCS_CASE(DCS_KIND_REPLACE)
                    DCS_CASE(DCS_KIND_FIXED)
                    DCS_CASE(DCS_KIND_FIXED_SHRINK)
                    DCS_CASE(DCS_KIND_SHRINK4)
                    DCS_CASE(DCS_KIND_SHRINK2)
#undef DCS_CASE
                }
                if constexpr (kStepMax<S>) {
                    const uint32_t key = __reduce_max_sync(0xffffffffu, __float_as_uint(lm));
                    if ((threadIdx.x & 31) == 0 && key) atomicMax(&smax[s], key);
                }
            }
            __syncthreads();
        }
        if (pair_out) {
            for (int t = 2 * threadIdx.x; t < T; t += 2 * NT) {
                const uint64_t a = addr(t);
                if (a & A.out_inactive) continue;
                const uint4 v = *reinterpret_cast<const uint4*>(smem + ((size_t)t << SH));
                left |= (v.x | v.y | v.z | v.w) & ~kSign;
                *reinterpret_cast<uint4*>(E + a) = v;
            }
        } else {
            for (int t = threadIdx.x; t < T; t += NT) {
                const uint64_t a = addr(t);
                if (a & A.out_inactive) continue;
                const S v = *reinterpret_cast<const S*>(smem + ((size_t)t << SH));
                if constexpr (!kStepMax<S>) gm = fmax(gm, v.x * v.x + v.y * v.y);
                left |= nonzero_bits(v);
                E[a] = v;
            }
        }
        __syncthreads();
    }
    // (a maximum that is zero although entries are not gets the least number there is, which sets kFlagRange)
    if constexpr (!kStepMax<S>) {
        const unsigned long long bm = block_max_u64(gm == 0 && left ? 1ull : max_bits(gm));
        if (threadIdx.x == 0 && bm) atomicMax(&mb[A.first + A.count], bm);
        return;
    }
    if (left && !smax[A.count - 1]) atomicMax(&mb[A.first + A.count], 1ull);
    if (threadIdx.x < A.count && smax[threadIdx.x])
        atomicMax(&mb[A.first + threadIdx.x + 1], (unsigned long long)smax[threadIdx.x]);
    if (!A.last) return;
    // the item's last CTA adds the exponents of the last group's inner steps, and notes them as the
    // power of two that the table still has (table_exp counts the CTAs until then)
    __shared__ int s_end;
    __threadfence();
    __syncthreads();
    dcs_scale* sp = scale + item;
    if (threadIdx.x == 0) s_end = atomicAdd(&sp->table_exp, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_end || threadIdx.x >= 32) return;
    __threadfence();
    const int rest = add_exponents<R>(mb, A.first + 1, A.count - 1, A.count, sp);
    if (threadIdx.x == 0) sp->table_exp = rest;
}

// Bytes of a binary16 tile, with its end where 8-byte words can follow (a plan that starts with fixed or isolated
// vertices has tiles of one 4-byte entry).
__host__ __device__ constexpr size_t half_tile_bytes(int tile_dim) {
    return tile_dim ? sizeof(ushort2) << tile_dim : sizeof(uint64_t);
}

// A group whose table is one tile, on binary16 tables with FP64 arithmetic (the half-storage tier): one CTA
// per item.  Every step rounds what it stores, scaled by the exponent of the maximum before it, so the
// scale is taken step by step here, too; the CTA holds the whole table, so its maximum is at hand.
// One launch for up to 24 steps instead of a launch each: see run_half_groups.
template <int NT>
__global__ void __launch_bounds__(NT)
k_tile_half(ushort2* __restrict__ table, uint64_t table_stride, const __grid_constant__ TileArgs A,
            const dcs_param* __restrict__ params, uint64_t param_stride, unsigned long long* __restrict__ maxbits,
            uint64_t maxbits_stride, dcs_scale* __restrict__ scale) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t tab[kMaxSteps][Tab<NT, kHalfDim>::kWords];
    __shared__ dcs_param prm[kMaxSteps];
    __shared__ uint32_t smax[kMaxSteps];
    const int item = blockIdx.y;
    const int T = 1 << A.tile_dim;
    const int low = A.low_bits;
    uint64_t* hi_tab = reinterpret_cast<uint64_t*>(smem + half_tile_bytes(A.tile_dim));
    ushort2* E = table + (uint64_t)item * table_stride;
    unsigned long long* mb = maxbits + (uint64_t)item * maxbits_stride;
    let_next_start();
    fill_tables<NT, kHalfDim, 2>(A, tab, hi_tab);
    after_previous();
    if (threadIdx.x < A.count) {
        prm[threadIdx.x] = params[(uint64_t)item * param_stride + A.first + threadIdx.x];
        smax[threadIdx.x] = 0;
    }
    __syncthreads();
    const uint64_t lowmask = (1ull << low) - 1;
    const uint64_t base = deposit(0, A.coset_runs, A.ncoset_runs);
    ushort2* sh = reinterpret_cast<ushort2*>(smem);
    for (int t = threadIdx.x; t < T; t += NT) {
        const uint64_t a = base ^ hi_tab[t >> low] ^ ((uint64_t)t & lowmask);
        if (!(a & A.in_inactive)) sh[t] = E[a];
    }
    __syncthreads();
    double m2 = __longlong_as_double((long long)mb[A.first]);
    dcs_scale sc = scale[item];
    for (int s = 0; s < A.count; ++s) {
        const TileStep& st = A.st[s];
        const dcs_param p = prm[s];
        const int e = exponent_of_max<float>(m2);
        sc.logscale += (double)e * 0.69314718055994530942;  // ln 2, as the reference's e*log(2.)
        sc.exponent_sum += e;
        if (!isfinite(m2)) sc.flags |= 1u;
        else if (m2 == 0.0) sc.flags |= 2u;
        const double f = exp2_neg(e);
        Weights<double2> w;
        w.f0 = cscale(make_double2(p.f0r, p.f0i), f);
        w.f1 = cscale(make_double2(p.f1r, p.f1i), f);
        w.fp = zadd(w.f0, w.f1);
        w.fm = zadd(w.f0, c2(-w.f1.x, -w.f1.y));
        const uint32_t cs = (uint32_t)__popcll(base & st.beta) ^ (uint32_t)(p.ov & 1);
        float lm = 0.f;
        switch (st.kind) {
#define DCS_CASE(K) \
    case K: lm = run_step<double2, K, NT, ushort2>(smem, T, st, tab[s], w, cs, p.y & 1); break;
            DCS_CASE(DCS_KIND_GROW)
            DCS_CASE(DCS_KIND_MIX)
            DCS_CASE(DCS_KIND_DIAG)
            DCS_CASE(DCS_KIND_REPLACE)
            DCS_CASE(DCS_KIND_FIXED)
            DCS_CASE(DCS_KIND_FIXED_SHRINK)
            DCS_CASE(DCS_KIND_SHRINK4)
            DCS_CASE(DCS_KIND_SHRINK2)
#undef DCS_CASE
        }
        const uint32_t key = __reduce_max_sync(0xffffffffu, __float_as_uint(lm));
        if ((threadIdx.x & 31) == 0 && key) atomicMax(&smax[s], key);
        __syncthreads();
        m2 = (double)__uint_as_float(smax[s]);
        if (threadIdx.x == 0) mb[A.first + s + 1] = max_bits(m2);
    }
    for (int t = threadIdx.x; t < T; t += NT) {
        const uint64_t a = base ^ hi_tab[t >> low] ^ ((uint64_t)t & lowmask);
        if (!(a & A.out_inactive)) E[a] = sh[t];
    }
    if (threadIdx.x == 0) scale[item] = sc;
}

bool fill_args(TileArgs& A, int max_dim, const dcs_group* groups, int gi, int ngroups, const dcs_step* steps, int nsteps,
               const dcs_tile_step* tile_steps) {
    const dcs_group& g = groups[gi];
    // the groups follow one another from the first step to the last
    if (g.first != (gi ? groups[gi - 1].first + groups[gi - 1].count : 0) ||
        (gi == ngroups - 1 && g.first + g.count != nsteps))
        return false;
    if (g.count < 1 || g.count > kMaxSteps || g.first < 0 || g.first + g.count > nsteps || g.tile_dim < 0 ||
        g.tile_dim > max_dim || g.low_bits < 0 || g.low_bits > g.tile_dim || g.ncoset_runs < 0 ||
        g.ncoset_runs > DCS_MAX_RUNS || g.coset_m < 0 || g.coset_m > DCS_MAX_SLOTS || g.tile_dim - g.low_bits > 16)
        return false;
    memset(&A, 0, sizeof(A));
    A.count = g.count;
    A.first = g.first;
    A.tile_dim = g.tile_dim;
    A.low_bits = g.low_bits;
    A.coset_m = g.coset_m;
    A.ncoset_runs = g.ncoset_runs;
    A.prev_first = gi ? groups[gi - 1].first : -1;
    A.last = gi == ngroups - 1;
    A.in_inactive = ~steps[g.first].in_mask;
    A.out_inactive = ~g.out_mask;
    memcpy(A.basis, g.basis, sizeof(A.basis));
    memcpy(A.coset_runs, g.coset_runs, sizeof(A.coset_runs));
    for (int s = 0; s < g.count; ++s) {
        const dcs_step& d = steps[g.first + s];
        const dcs_tile_step& ts = tile_steps[g.step_tile_off + s];
        TileStep& f = A.st[s];
        f.beta = d.beta;
        f.cskip = ts.cskip;
        f.tK = ts.tK; f.tKa = ts.tKa; f.tpiv = ts.tpiv; f.tbeta = ts.tbeta;
        if (d.kind < 0 || d.kind > 7 || ts.nins > 16 || ts.nins > g.tile_dim ||
            (f.tK | f.tKa | f.tpiv | f.tbeta) >> g.tile_dim)
            return false;
        f.kind = (uint8_t)d.kind;
        f.sK = ts.sK & 1; f.sKa = ts.sKa & 1; f.nins = ts.nins;
        for (int i = 0; i < f.nins; ++i) {
            f.ins[i] = ts.ins[i];
            if (ts.ins[i] >= g.tile_dim || (i && ts.ins[i] <= ts.ins[i - 1])) return false;
        }
    }
    return true;
}

template <class S, int NT>
int launch_group(S* table, uint64_t table_stride, const TileArgs& A, const dcs_param* params, uint64_t param_stride,
                 unsigned long long* maxbits, uint64_t maxbits_stride, dcs_scale* scale, int nitems, int sms, int dev,
                 cudaStream_t st) {
    static bool smem_set[64] = {false};
    if (!smem_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(k_tiles<S, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
        if (e != cudaSuccess) return dcs_host::check_cuda(e, "k_tiles smem attribute");
        smem_set[dev] = true;
    }
    const size_t smem = sizeof(S) * ((size_t)1 << A.tile_dim) + sizeof(uint64_t) * ((size_t)1 << (A.tile_dim - A.low_bits));
    uint64_t grid = 1ull << A.coset_m;
    if (grid * nitems > (uint64_t)sms) {  // more tiles than SMs: at most one wave of resident CTAs
        int per_sm = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tiles<S, NT>, NT, smem);
        if (e != cudaSuccess) return dcs_host::check_cuda(e, "k_tiles occupancy");
        if (per_sm < 1) per_sm = 1;
        uint64_t wave = (uint64_t)sms * per_sm / nitems;
        if (wave < 1) wave = 1;
        if (grid > wave) {  // the same number of tiles for every CTA, as nearly as it goes
            const uint64_t each = (grid + wave - 1) / wave;
            grid = (grid + each - 1) / each;
        }
    }
    return dcs_host::check_cuda(dcs_host::launch_after(k_tiles<S, NT>, dim3((unsigned)grid, (unsigned)nitems), dim3(NT), smem,
                                                       st, table, table_stride, A, params, param_stride, maxbits,
                                                       maxbits_stride, scale),
                                "k_tiles launch");
}

template <class S>
int run_groups(S* table, uint64_t table_stride, const dcs_step* steps, int nsteps, const dcs_group* groups,
               int ngroups, const dcs_tile_step* tile_steps, const dcs_param* params, uint64_t param_stride,
               unsigned long long* maxbits, uint64_t maxbits_stride, dcs_scale* scale, int nitems, cudaStream_t st) {
    const int sms = dcs_host::sm_count();
    int dev = 0;
    if (sms <= 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        dcs_host::set_error("dcs_tile_groups: no current device");
        return DCS_E_CUDA;
    }
    TileArgs A;
    for (int gi = 0; gi < ngroups; ++gi) {
        if (!fill_args(A, kMaxDim, groups, gi, ngroups, steps, nsteps, tile_steps)) {
            dcs_host::set_error("dcs_tile_groups: malformed group %d", gi);
            return DCS_E_ARG;
        }
        // A tile per SM at most: 512 threads share it (a slice of 2^22 entries 5% faster than with 256).  More: CTAs
        // of 256 hide each other's latencies (512 for them: 2 to 15% slower).  Complex64 with many tiles per SM
        // is bound by issue slots, and 128 threads spend fewer on each step's preparation (2^22 entries, 16
        // slices: 1562 us against 1727; 512 tiles of 2^11: 146 against 138); the five 32 KiB tiles that an SM
        // holds have warps enough then, the three 64 KiB ones of complex128 do not (3014 against 2156).
        const uint64_t tiles = (uint64_t)nitems << A.coset_m;
        const auto launch = tiles <= (uint64_t)sms                               ? launch_group<S, 512>
                            : sizeof(S) == 8 && tiles > (uint64_t)kManyTiles * sms ? launch_group<S, 128>
                                                                                  : launch_group<S, 256>;
        const int rc = launch(table, table_stride, A, params, param_stride, maxbits, maxbits_stride, scale, nitems, sms, dev,
                              st);
        if (rc) return rc;
    }
    return DCS_OK;
}

// Binary16 tables: groups whose table is one tile in one launch, the others a launch per step.  A block with a
// launch per step / so: 16 qubits (31 steps, 2 launches) 301 / 191 us, 24 qubits (72, 3) 452 / 230, 32 qubits
// (97, 25; 2^16 entries at the largest) 583 / 377.
int run_half_groups(ushort2* table, uint64_t table_stride, const dcs_step* steps, int nsteps, const dcs_group* groups,
                    int ngroups, const dcs_tile_step* tile_steps, const dcs_param* params, uint64_t param_stride,
                    uint64_t* maxbits, dcs_scale* scale, int nitems, cudaStream_t st) {
    constexpr int NT = 512;
    const uint64_t mstride = (uint64_t)nsteps + 1;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        dcs_host::set_error("dcs_tile_groups: no current device");
        return DCS_E_CUDA;
    }
    static bool smem_set[64] = {false};
    if (!smem_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(k_tile_half<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
        if (e != cudaSuccess) return dcs_host::check_cuda(e, "k_tile_half smem attribute");
        smem_set[dev] = true;
    }
    TileArgs A;
    for (int gi = 0; gi < ngroups; ++gi) {
        const dcs_group& g = groups[gi];
        int rc;
        if (g.coset_m != 0 || g.tile_dim > kHalfDim) {
            rc = dcs_slice_steps_batched(DCS_H16, table, table_stride, steps, params, param_stride, nsteps, g.first, g.count,
                                         maxbits, scale, nitems, st);
        } else {
            if (!fill_args(A, kHalfDim, groups, gi, ngroups, steps, nsteps, tile_steps)) {
                dcs_host::set_error("dcs_tile_groups: malformed group %d", gi);
                return DCS_E_ARG;
            }
            const size_t smem = half_tile_bytes(A.tile_dim) + sizeof(uint64_t) * ((size_t)1 << (A.tile_dim - A.low_bits));
            rc = dcs_host::check_cuda(
                dcs_host::launch_after(k_tile_half<NT>, dim3(1, (unsigned)nitems), dim3(NT), smem, st, table, table_stride, A,
                                       params, param_stride, (unsigned long long*)maxbits, mstride, scale),
                "k_tile_half launch");
        }
        if (rc) return rc;
    }
    return DCS_OK;
}

}  // namespace

extern "C" int dcs_tile_groups(int dtype, void* table, uint64_t table_stride, const dcs_step* steps, int nsteps,
                               const dcs_group* groups, int ngroups, const dcs_tile_step* tile_steps,
                               const dcs_param* params, uint64_t param_stride, uint64_t* maxbits,
                               uint64_t maxbits_stride, dcs_scale* scale, int nitems, void* stream) {
    if (!table || !steps || !groups || !tile_steps || !params || !maxbits || !scale || ngroups < 0 || nitems < 1 ||
        nitems > 65535 || maxbits_stride < (uint64_t)nsteps + 1 || (dtype != DCS_C64 && dtype != DCS_C128 && dtype != DCS_H16) ||
        (dtype == DCS_H16 && maxbits_stride != (uint64_t)nsteps + 1)) {
        dcs_host::set_error("dcs_tile_groups: invalid arguments");
        return DCS_E_ARG;
    }
    // rows of complex64 entries move in 16-byte words
    const bool aligned = ((uintptr_t)table & 15) == 0 && (nitems == 1 || !(table_stride & 1));
    for (int gi = 0; gi < ngroups && dtype == DCS_C64 && !aligned; ++gi)
        if (groups[gi].low_bits >= 1) {
            dcs_host::set_error("dcs_tile_groups: complex64 tables must be 16-byte aligned (an even table_stride)");
            return DCS_E_ARG;
        }
    if (dtype == DCS_H16)
        return run_half_groups((ushort2*)table, table_stride, steps, nsteps, groups, ngroups, tile_steps, params,
                               param_stride, maxbits, scale, nitems, (cudaStream_t)stream);
    if (dtype == DCS_C64)
        return run_groups((float2*)table, table_stride, steps, nsteps, groups, ngroups, tile_steps, params, param_stride,
                          (unsigned long long*)maxbits, maxbits_stride, scale, nitems, (cudaStream_t)stream);
    return run_groups((double2*)table, table_stride, steps, nsteps, groups, ngroups, tile_steps, params, param_stride,
                      (unsigned long long*)maxbits, maxbits_stride, scale, nitems, (cudaStream_t)stream);
}
