// Block assembly: terminal gather + syndrome scatter + coherent slice sum, then the
// Walsh-Hadamard / open-edge phase / U_open tail (sm_100a).
//
// Reference: source/kernel_opt/inplace_gpu.py:124 (terminal gather),
// source/sampling/conditional_block_gpu.py:155-158 (scatter-add, coefficient
// coef * exp(logscale - (N_full - n + k)/2 ln 2)), :159-171 (tail).
//
// The scatter `total[synd(i) ^ xor] += env(i) * coef` is evaluated as a gather over the
// output index t: i = L(t ^ xor) when t ^ xor lies in the image of the syndrome map
// (parity checks H), with L a left inverse.  Every output entry is owned by one thread and
// the slices of one block are summed in slice order, so the sum is deterministic.
#include <string.h>

#include "common.cuh"

using namespace dcs;

namespace {

struct TermMap {
    uint32_t runs[DCS_MAX_RUNS];  // deposit of i into the terminal slots
    uint32_t linv[32];            // i_j = parity(s & linv[j])
    uint32_t check[32];           // s in image iff parity(s & check[r]) == 0 for all r
    int nruns, tr, nchecks, k;
};

// What an item adds, the same for every entry of its block.
struct ItemTerm {
    double cr, ci, p2;  // coefficient; power of two that its table still has
    uint64_t xor_;
    int on;
};

template <class S>
__global__ void __launch_bounds__(256)
k_accumulate(const S* table, uint64_t table_stride, const __grid_constant__ TermMap tm, const uint64_t* xors,
             const double* coefs, const int32_t* item_begin, double log_shift, dcs_scale* scale,
             const unsigned long long* maxbits_final, uint64_t mstride, int is64, int fresh, int use_exp, double2* total) {
    let_next_start();
    after_previous();
    // grid.y = output block; items item_begin[b] .. item_begin[b+1]-1 belong to block b
    constexpr int kTerms = 64;  // items whose terms sit in shared memory at a time
    __shared__ ItemTerm terms[kTerms];
    const int blk = blockIdx.y;
    const int i0 = item_begin[blk], i1 = item_begin[blk + 1];
    double2* out = total + ((uint64_t)blk << tm.k);
    const uint64_t n = 1ull << tm.k;
    int c0 = i0;
    do {  // (a block without items is written once, too, when it starts at zero)
        const int cn = i1 - c0 < kTerms ? i1 - c0 : kTerms;
        __syncthreads();
        // an exponential and a sine per item and CTA; per item and entry they were most of the kernel
        if ((int)threadIdx.x < cn) {
            const int it = c0 + threadIdx.x;
            const dcs_scale sc = scale[it];
            const unsigned long long mf = maxbits_final[(uint64_t)it * mstride];
            const double m2 = is64 ? __longlong_as_double((long long)mf) : (double)__uint_as_float((uint32_t)mf);
            ItemTerm t;
            // a zero table (skipped slice: at some step, or after the last one) or one that was nonfinite before the
            // last step adds nothing; one that the last step made nonfinite shows in the block, too
            t.on = mf != 0 && (!(sc.flags & 3u) || (sc.flags & kFlagLast));
            // the reference checks every step's max, including the last (kFlagLast: the launch's other CTAs may
            // read the flags before or after this)
            if (blockIdx.x == 0) {
                if (!isfinite(m2)) scale[it].flags = sc.flags | (sc.flags & 1u ? 0u : 1u | kFlagLast);
                else if (m2 > 0.0 && m2 < (is64 ? kLeastMax<double> : kLeastMax<float>)) scale[it].flags = sc.flags | kFlagRange;
            }
            const double m = exp(sc.logscale - log_shift);
            double cr = coefs[2 * it] * m, ci = coefs[2 * it + 1] * m;
            if (sc.phase != 0.0) {  // step factors divided out by the plan-specialised kernels
                double sp, cp;
                sincos(sc.phase, &sp, &cp);
                const double r = __fma_rn(cr, cp, -__dmul_rn(ci, sp));
                ci = __fma_rn(cr, sp, __dmul_rn(ci, cp));
                cr = r;
            }
            t.cr = cr;
            t.ci = ci;
            t.p2 = use_exp ? ldexp(1.0, -sc.table_exp) : 1.0;
            t.xor_ = xors[it];
            terms[threadIdx.x] = t;
        }
        __syncthreads();
        for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x) {
            double2 acc = fresh && c0 == i0 ? make_double2(0.0, 0.0) : out[t];
            for (int q = 0; q < cn; ++q) {
                const ItemTerm& term = terms[q];
                if (!term.on) continue;
                const uint32_t sv = (uint32_t)(t ^ term.xor_);
                bool in = true;
                for (int r = 0; r < tm.nchecks; ++r) in &= !(__popc(sv & tm.check[r]) & 1);
                if (!in) continue;
                uint32_t i = 0;
                for (int j = 0; j < tm.tr; ++j) i |= (uint32_t)(__popc(sv & tm.linv[j]) & 1) << j;
                const uint64_t c = deposit(i, tm.runs, tm.nruns);
                const double2 v = entry_f64(table[(uint64_t)(c0 + q) * table_stride + c]);
                const double vr = v.x * term.p2, vi = v.y * term.p2;  // exact
                // (roundings fixed here and above: the draws' 53-bit distances depend on every bit of a block)
                acc.x = __dadd_rn(acc.x, __fma_rn(vr, term.cr, -__dmul_rn(vi, term.ci)));
                acc.y = __dadd_rn(acc.y, __fma_rn(vi, term.cr, __dmul_rn(vr, term.ci)));
            }
            out[t] = acc;
        }
        c0 += kTerms;
    } while (c0 < i1);
}

// ---------------------------------------------------------------- tail
struct TailParams {
    double u[32][8];     // per physical bit: 2x2 complex row-major (re, im)
    uint32_t adj_hi[32]; // open-edge adjacency, b > a
    int k;
};

constexpr int kTailLog = 12;  // 4096 complex128 = 64 KiB of shared memory per tile
enum { kTailWht = 0, kTailPhaseU = 1, kTailU = 2, kTailAll = 3 };

// 16-byte entries, eight of them per 128-byte row of banks: the XOR keeps the eight lanes of an access apart both
// when they hold neighbours and when each holds a run of eight
__device__ __forceinline__ int swz(int i) { return i ^ ((i >> 3) & 7); }

// sign of the open-edge phase at index ad
__device__ __forceinline__ bool open_phase(uint32_t ad, const TailParams& tp) {
    uint32_t par = 0;
    for (int q = 0; q < tp.k; ++q)
        if ((ad >> q) & 1) par ^= ad & tp.adj_hi[q];
    return __popc(par) & 1;
}

// NB consecutive tile bits from bit j on, one after the other, on 2^NB entries per thread
template <int NB, bool U>
__device__ __forceinline__ void tail_round(double2* sh, int tsize, int j, int q0, const TailParams& tp, bool phase) {
    constexpr int N = 1 << NB;
    for (int g = threadIdx.x; g < (tsize >> NB); g += blockDim.x) {
        const int i0 = ((g >> j) << (j + NB)) | (g & ((1 << j) - 1));
        double2 x[N];
#pragma unroll
        for (int e = 0; e < N; ++e) {
            x[e] = sh[swz(i0 | e << j)];
            if (U && phase && open_phase((uint32_t)(i0 | e << j), tp)) x[e] = make_double2(-x[e].x, -x[e].y);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const double* m = tp.u[q0 + b];
#pragma unroll
            for (int e = 0; e < N; ++e) {
                if (e >> b & 1) continue;
                const double2 x0 = x[e], x1 = x[e | 1 << b];
                if constexpr (U) {
                    x[e] = make_double2(m[0] * x0.x - m[1] * x0.y + m[2] * x1.x - m[3] * x1.y,
                                        m[0] * x0.y + m[1] * x0.x + m[2] * x1.y + m[3] * x1.x);
                    x[e | 1 << b] = make_double2(m[4] * x0.x - m[5] * x0.y + m[6] * x1.x - m[7] * x1.y,
                                                 m[4] * x0.y + m[5] * x0.x + m[6] * x1.y + m[7] * x1.x);
                } else {
                    x[e] = make_double2(x0.x + x1.x, x0.y + x1.y);
                    x[e | 1 << b] = make_double2(x0.x - x1.x, x0.y - x1.y);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < N; ++e) sh[swz(i0 | e << j)] = x[e];
    }
    __syncthreads();
}

// tile bits [lo, hi), three per round (one round trip through shared memory for three of them); `a`: the tile
// bits below it are the physical bits, the others start at physical bit b_lo
template <bool U>
__device__ __forceinline__ void tail_bits(double2* sh, int tsize, int lo, int hi, int a, int b_lo, const TailParams& tp,
                                          bool phase) {
    for (int j = lo; j < hi;) {
        const int q0 = j < a ? j : b_lo + (j - a);  // physical bit
        const int nb = hi - j < 3 ? hi - j : 3;
        if (nb == 3) tail_round<3, U>(sh, tsize, j, q0, tp, phase);
        else if (nb == 2) tail_round<2, U>(sh, tsize, j, q0, tp, phase);
        else tail_round<1, U>(sh, tsize, j, q0, tp, phase);
        phase = false;
        j += nb;
    }
}

// Apply per-bit 2x2 transforms over the tile bits [tb_lo, tb_hi) of tiles made of
// physical bits [0, a) (contiguous) and [b_lo, b_hi).  kTailWht: Walsh-Hadamard; kTailPhaseU: multiply by
// the open-edge phase on load, then U_open; kTailU: U_open; kTailAll (one tile per block): all of it.
template <int MODE>
__global__ void __launch_bounds__(512)
k_tail(double2* __restrict__ total, const __grid_constant__ TailParams tp, int a, int b_lo, int b_hi, int tb_lo,
       int tb_hi) {
    extern __shared__ double2 sh[];
    const int k = tp.k;
    let_next_start();
    after_previous();
    const int tile_log = a + (b_hi - b_lo);
    const int tsize = 1 << tile_log;
    const uint64_t nblk_elems = 1ull << k;
    const uint64_t ntiles_per_block = nblk_elems >> tile_log;
    const uint64_t blk = blockIdx.x / ntiles_per_block;
    const uint64_t g = blockIdx.x % ntiles_per_block;
    double2* v = total + (blk << k);
    // complement bits: [a, b_lo) then [b_hi, k)
    const int mid = b_lo - a;
    const uint64_t g_lo = g & ((1ull << mid) - 1), g_hi = g >> mid;
    const uint64_t gbase = (g_lo << a) | (g_hi << b_hi);
    auto addr = [&](int t) -> uint64_t {
        const uint64_t lo = (uint64_t)t & ((1ull << a) - 1);
        const uint64_t hi = (uint64_t)t >> a;
        return gbase | lo | (hi << b_lo);
    };
#pragma unroll 4
    for (int t = threadIdx.x; t < tsize; t += blockDim.x) {
        const uint64_t ad = addr(t);
        double2 x = v[ad];
        if (MODE == kTailPhaseU && open_phase((uint32_t)ad, tp)) x = make_double2(-x.x, -x.y);
        sh[swz(t)] = x;
    }
    __syncthreads();
    if constexpr (MODE == kTailWht || MODE == kTailAll) tail_bits<false>(sh, tsize, tb_lo, tb_hi, a, b_lo, tp, false);
    if constexpr (MODE != kTailWht) tail_bits<true>(sh, tsize, tb_lo, tb_hi, a, b_lo, tp, MODE == kTailAll);
#pragma unroll 4
    for (int t = threadIdx.x; t < tsize; t += blockDim.x) v[addr(t)] = sh[swz(t)];
}

template <int MODE>
int tail_pass(double2* total, const TailParams& tp, int a, int b_lo, int b_hi, int tb_lo, int tb_hi, int nblocks,
              cudaStream_t st) {
    const int tile_log = a + (b_hi - b_lo);
    const uint64_t tiles = (uint64_t)nblocks << (tp.k - tile_log);
    if (tiles > 0x7fffffffull) {
        dcs_host::set_error("dcs_block_tail: too many tiles");
        return DCS_E_ARG;
    }
    const int threads = tile_log >= kTailLog ? 512 : 1 << (tile_log > 8 ? tile_log - 3 : 5);  // eight entries each
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        dcs_host::set_error("dcs_block_tail: no current device");
        return DCS_E_CUDA;
    }
    static int attr_set[64] = {0};
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_tail<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(sizeof(double2) << kTailLog));
        if (e != cudaSuccess) return dcs_host::check_cuda(e, "k_tail smem attribute");
        attr_set[dev] = 1;
    }
    // (a swizzled index stays inside its row of eight)
    const size_t smem = sizeof(double2) << (tile_log > 3 ? tile_log : 3);
    return dcs_host::check_cuda(dcs_host::launch_after(k_tail<MODE>, dim3((unsigned)tiles), dim3(threads), smem, st, total, tp, a,
                                                       b_lo, b_hi, tb_lo, tb_hi),
                                "k_tail launch");
}

}  // namespace

static int build_termmap(TermMap& tm, int tr, const uint32_t* runs, int nruns, const uint64_t* tbasis_host, int k) {
    if (tr < 0 || tr > 31 || k < 0 || k > 31 || tr > k || nruns < 0 || nruns > DCS_MAX_RUNS) {
        dcs_host::set_error("dcs_accumulate: tr=%d k=%d nruns=%d out of range", tr, k, nruns);
        return DCS_E_ARG;
    }
    memset(&tm, 0, sizeof(tm));
    tm.tr = tr; tm.k = k; tm.nruns = nruns;
    for (int r = 0; r < nruns; ++r) tm.runs[r] = runs[r];
    // Gauss-Jordan on the tr basis vectors (k bits each): rows = basis, track combinations.
    uint32_t row[32], comb[32];
    int piv[32];
    for (int j = 0; j < tr; ++j) {
        if (tbasis_host[j] >> k) { dcs_host::set_error("dcs_accumulate: basis vector wider than k"); return DCS_E_ARG; }
        row[j] = (uint32_t)tbasis_host[j];
        comb[j] = 1u << j;
    }
    for (int j = 0; j < tr; ++j) {
        if (!row[j]) { dcs_host::set_error("dcs_accumulate: dependent terminal basis"); return DCS_E_ARG; }
        piv[j] = 31 - __builtin_clz(row[j]);
        for (int o = 0; o < tr; ++o)
            if (o != j && ((row[o] >> piv[j]) & 1)) { row[o] ^= row[j]; comb[o] ^= comb[j]; }
    }
    // now row[j] has a 1 at piv[j] and 0 at every other pivot; s = sum_j i_j basis_j means
    // reduced coordinates: s in image iff s == XOR_{j: s_piv[j]} row[j]; then i = XOR comb[j].
    // i_bit = parity(s & linv[bit]) with linv[bit] = {piv[j] : comb[j] has bit}
    for (int bit = 0; bit < tr; ++bit) {
        uint32_t m = 0;
        for (int j = 0; j < tr; ++j)
            if ((comb[j] >> bit) & 1) m |= 1u << piv[j];
        tm.linv[bit] = m;
    }
    // parity checks: for every non-pivot bit q, s_q == XOR_j s_piv[j] * row[j]_q
    uint32_t pivmask = 0;
    for (int j = 0; j < tr; ++j) pivmask |= 1u << piv[j];
    int nc = 0;
    for (int q = 0; q < k; ++q) {
        if ((pivmask >> q) & 1) continue;
        uint32_t m = 1u << q;
        for (int j = 0; j < tr; ++j)
            if ((row[j] >> q) & 1) m |= 1u << piv[j];
        tm.check[nc++] = m;
    }
    tm.nchecks = nc;
    return DCS_OK;
}

static int accumulate(int dtype, const void* table, uint64_t table_stride, int tr, const uint32_t* terminal_runs, int nruns,
                      const uint64_t* tbasis, const uint64_t* xors, const double* coefs, const int32_t* item_begin,
                      int nblocks, double log_shift, dcs_scale* scale, const uint64_t* maxbits_final, uint64_t mstride,
                      double* total, int k, int nitems, unsigned flags, bool use_exp, void* stream) {
    if (!table || !xors || !coefs || !item_begin || !scale || !maxbits_final || !total || nblocks < 1 ||
        nblocks > 65535 || nitems < 0 || (flags & ~(unsigned)DCS_ACCUMULATE_FRESH)) {
        dcs_host::set_error("dcs_accumulate: invalid arguments");
        return DCS_E_ARG;
    }
    TermMap tm;
    int rc = build_termmap(tm, tr, terminal_runs, nruns, tbasis, k);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t n = 1ull << k;
    uint64_t bx = (n + 255) / 256;
    const uint64_t cap = (uint64_t)dcs_host::sm_count() * 8;
    if (bx > cap) bx = cap;
    dim3 grid((unsigned)bx, (unsigned)nblocks);
    auto run = [&](auto kernel, auto t) {
        return dcs_host::check_cuda(
            dcs_host::launch_after(kernel, grid, dim3(256), 0, st, t, table_stride, tm, xors, coefs, item_begin, log_shift, scale,
                                   (const unsigned long long*)maxbits_final, mstride, dtype != DCS_C64 ? 1 : 0,  // (binary16: FP64 arithmetic)
                                   (flags & DCS_ACCUMULATE_FRESH) ? 1 : 0, use_exp ? 1 : 0, (double2*)total),
            "k_accumulate launch");
    };
    if (dtype == DCS_C64) return run(k_accumulate<float2>, (const float2*)table);
    if (dtype == DCS_C128) return run(k_accumulate<double2>, (const double2*)table);
    if (dtype == DCS_H16) return run(k_accumulate<ushort2>, (const ushort2*)table);
    dcs_host::set_error("dcs_accumulate: unknown dtype %d", dtype);
    return DCS_E_ARG;
}

extern "C" int dcs_accumulate_batched(int dtype, const void* table, uint64_t table_stride, int tr,
                                      const uint32_t* terminal_runs, int nruns, const uint64_t* tbasis,
                                      const uint64_t* xors, const double* coefs, const int32_t* item_begin,
                                      int nblocks, double log_shift, dcs_scale* scale, const uint64_t* maxbits_final,
                                      uint64_t mstride, double* total, int k, int nitems, void* stream) {
    // (callers of the step and fused kernels need not set table_exp)
    return accumulate(dtype, table, table_stride, tr, terminal_runs, nruns, tbasis, xors, coefs, item_begin, nblocks, log_shift,
                      scale, maxbits_final, mstride, total, k, nitems, 0u, false, stream);
}

extern "C" int dcs_accumulate_ex(int dtype, const void* table, uint64_t table_stride, int tr,
                                 const uint32_t* terminal_runs, int nruns, const uint64_t* tbasis, const uint64_t* xors,
                                 const double* coefs, const int32_t* item_begin, int nblocks, double log_shift,
                                 dcs_scale* scale, const uint64_t* maxbits_final, uint64_t mstride, double* total, int k,
                                 int nitems, unsigned flags, void* stream) {
    return accumulate(dtype, table, table_stride, tr, terminal_runs, nruns, tbasis, xors, coefs, item_begin, nblocks, log_shift,
                      scale, maxbits_final, mstride, total, k, nitems, flags, true, stream);
}

extern "C" int dcs_block_tail(double* total, int k, const uint32_t* adj_hi, const double* u_open, int nblocks,
                              void* stream) {
    if (!total || k < 0 || k > 30 || nblocks < 1 || (k > 0 && (!adj_hi || !u_open))) {
        dcs_host::set_error("dcs_block_tail: invalid arguments");
        return DCS_E_ARG;
    }
    if (k == 0) return DCS_OK;
    TailParams tp;
    memset(&tp, 0, sizeof(tp));
    tp.k = k;
    for (int q = 0; q < k; ++q) {
        tp.adj_hi[q] = adj_hi[q];
        for (int e = 0; e < 8; ++e) tp.u[q][e] = u_open[8 * q + e];
    }
    cudaStream_t st = (cudaStream_t)stream;
    double2* v = (double2*)total;
    int rc;
    if (k <= kTailLog)  // one tile per block: everything in one pass
        return tail_pass<kTailAll>(v, tp, k, k, k, 0, k, nblocks, st);
    // low tile: bits [0, L); high tile: 3 contiguous low bits + bits [L, k).  The two sizes are as near as they
    // get, so that a 2^17 block has 128 tiles in every pass: with 2^12-entry low tiles it had 32, and a
    // shared-memory round trip per bit, and took 39 us for the four passes.
    int L = (k + 3) / 2;
    if (L < k + 3 - kTailLog) L = k + 3 - kTailLog;
    if (L > kTailLog) {
        dcs_host::set_error("dcs_block_tail: k=%d too large for the two-pass tail", k);
        return DCS_E_ARG;
    }
    const int hb = k - L;  // high bits
    if ((rc = tail_pass<kTailWht>(v, tp, L, L, L, 0, L, nblocks, st))) return rc;
    if ((rc = tail_pass<kTailWht>(v, tp, 3, L, k, 3, 3 + hb, nblocks, st))) return rc;
    if ((rc = tail_pass<kTailPhaseU>(v, tp, L, L, L, 0, L, nblocks, st))) return rc;
    return tail_pass<kTailU>(v, tp, 3, L, k, 3, 3 + hb, nblocks, st);
}
