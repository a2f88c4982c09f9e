// Gather-form vertex step on two tables (sm_100a): the executor of the reference's
// ConditionalBlockGPU (source/dcs_rankwidth/gpu_kernel.py:58-103, scan_step_scaled, driven by
// source/sampling/conditional_block_gpu.py:92-126).  It is not the production path (the in-place
// executor is), but keeps the reference's second engine available on the B200.
//
// Per output c' of 2^r_out: p0 = XOR over the bytes of c' of the step's byte table (the right
// inverse L applied to c'), then the sum over the kernel combinations p = p0 ^ combo of
// E[p & mask_in] times f_v(y) with sign (-1)^(y * (parity(c & beta) ^ ov)), y = bit r_in of p for a
// free step, else the fixed value.  Sums are FP64 for both storages (as the reference's kernel),
// written scaled by 2^-e.  Differences by design: e is derived on the device from the previous
// step's max (no host sync); the byte tables and combinations of the step sit in shared memory;
// several work items (slices) per launch (blockIdx.y).
#include "common.cuh"

using namespace dcs;

namespace {

constexpr int kThreads = 256;
constexpr int kMaxTableWords = 8 * 256;  // up to 64-bit outputs
constexpr int kMaxCombos = 64;

// Output cp of a step: the sum over the kernel combinations, in FP64, scaled.
template <class S>
__device__ __forceinline__ S gather_entry(const S* E, uint64_t cp, const dcs_gather_step& st, const uint64_t* T,
                                          const uint64_t* C, uint64_t mask, uint64_t beta, int ov, int y_fixed, double w0r,
                                          double w0i, double w1r, double w1i, double sc) {
    using R = typename Store<S>::R;
    uint64_t p0 = 0;
    for (int b = 0; b < st.nbytes; ++b) p0 ^= T[b * 256 + (int)((cp >> (8 * b)) & 255)];
    double ar = 0.0, ai = 0.0;
    for (int k = 0; k < st.ncombos; ++k) {
        const uint64_t q = p0 ^ C[k];
        const uint64_t c = q & mask;
        const int par = neg_sign(c, beta, ov);
        const int y = st.free_ ? (int)((q >> st.r_in) & 1ull) : y_fixed;
        double wr = y ? w1r : w0r, wi = y ? w1i : w0i;
        if (y & par) {
            wr = -wr;
            wi = -wi;
        }
        const double2 v = entry_f64(E[c]);
        ar += v.x * wr - v.y * wi;
        ai += v.x * wi + v.y * wr;
    }
    return Store<S>::make((R)(ar * sc), (R)(ai * sc));
}

// (Ein is what the launch before writes, which may still run when this one starts: no read-only loads of it)
template <class S>
__global__ void __launch_bounds__(kThreads)
k_gather(const S* Ein, S* Eout, uint64_t stride, const __grid_constant__ dcs_gather_step st,
         const uint64_t* __restrict__ words, int s, const dcs_param* __restrict__ params, uint64_t param_stride,
         unsigned long long* __restrict__ maxbits, uint64_t maxbits_stride, dcs_scale* __restrict__ scale) {
    using R = typename Store<S>::R;
    __shared__ uint64_t T[kMaxTableWords];
    __shared__ uint64_t C[kMaxCombos];
    const int item = blockIdx.y;
    const S* E = Ein + (uint64_t)item * stride;
    S* out = Eout + (uint64_t)item * stride;
    let_next_start();
    // the step's tables are the plan's: nothing in the stream writes them
    for (int i = threadIdx.x; i < st.nbytes * 256; i += kThreads) T[i] = words[st.table_off + i];
    for (int i = threadIdx.x; i < st.ncombos; i += kThreads) C[i] = words[st.combo_off + i];
    after_previous();
    const dcs_param p = params[(uint64_t)item * param_stride + s];
    unsigned long long* mb = maxbits + (uint64_t)item * maxbits_stride;
    const double m2prev = (double)bits_to_m2<R>(mb[s]);
    const int e = exponent_of_max<R>(m2prev);
    const double sc = exp2_neg(e);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        dcs_scale* sp = scale + item;
        sp->logscale += (double)e * 0.69314718055994530942;
        sp->exponent_sum += e;
        if (!isfinite(m2prev)) sp->flags |= 1u;
        else if (m2prev == 0.0) sp->flags |= 2u;
    }
    __syncthreads();
    const uint64_t mask = st.r_in >= 64 ? ~0ull : ((1ull << st.r_in) - 1ull);
    const uint64_t n_out = 1ull << st.r_out;
    const uint64_t beta = st.beta;
    const int ov = p.ov & 1, y_fixed = p.y & 1;
    // the two weights with their sign applied, as FP64
    const double w0r = p.f0r, w0i = p.f0i, w1r = p.f1r, w1i = p.f1i;
    R lm = 0;
    for (uint64_t cp = (uint64_t)blockIdx.x * kThreads + threadIdx.x; cp < n_out; cp += (uint64_t)gridDim.x * kThreads) {
        const S o = gather_entry(E, cp, st, T, C, mask, beta, ov, y_fixed, w0r, w0i, w1r, w1i, sc);
        out[cp] = o;
        lm = fmax(lm, o.x * o.x + o.y * o.y);
    }
    const unsigned long long mx = block_max_u64(max_bits(lm));
    if (threadIdx.x == 0 && mx) atomicMax(&mb[s + 1], mx);
}

// A stretch of steps whose tables both fit shared memory: one CTA per item takes all of them, the two
// tables there, the byte table and combinations of the next step on their way while a step runs.
// Renormalisation is step by step as in k_gather, from the CTA's own maximum.  Bound by the latency of a step.
// A block with a launch per step / with these: 16 qubits (all 31 steps) 240 / 204 us, 24 qubits (70 of 72) 352 /
// 255, 32 qubits (51 of 97) 450 / 405; with tables of up to 2^12 entries 32 qubits take 435 again.
constexpr int kSmallThreads = 512;
constexpr int kSmallSteps = 48;
constexpr int kSmallRank = 11;  // two tables of 2^11 entries; beyond, one SM takes longer over a step than a launch does
constexpr int kSmallBytes = 2;  // bytes of an output index of up to 16 bits

struct GatherRun {
    int32_t count, s0, rank, pad;
    dcs_gather_step st[kSmallSteps];
};

template <class S>
__global__ void __launch_bounds__(kSmallThreads)
k_gather_small(const S* Ein, S* Eout, uint64_t stride, const __grid_constant__ GatherRun G,
               const uint64_t* __restrict__ words, const dcs_param* __restrict__ params, uint64_t param_stride,
               unsigned long long* __restrict__ maxbits, uint64_t maxbits_stride, dcs_scale* __restrict__ scale) {
    using R = typename Store<S>::R;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t T[2][kSmallBytes * 256];
    __shared__ uint64_t C[2][kMaxCombos];
    __shared__ uint32_t smax[kSmallSteps], slow[kSmallSteps];
    __shared__ dcs_param prm[kSmallSteps];
    const int item = blockIdx.y;
    S* tab[2] = {reinterpret_cast<S*>(smem), reinterpret_cast<S*>(smem) + ((size_t)1 << G.rank)};
    unsigned long long* mb = maxbits + (uint64_t)item * maxbits_stride;
    auto fetch = [&](int i) {  // the tables of step i, on their way
        const dcs_gather_step& st = G.st[i];
        for (int j = threadIdx.x; j < st.nbytes * 256 + st.ncombos; j += kSmallThreads) {
            const bool t = j < st.nbytes * 256;
            const uint64_t* src = words + (t ? st.table_off + j : st.combo_off + (j - st.nbytes * 256));
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(t ? &T[i & 1][j] : &C[i & 1][j - st.nbytes * 256]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    let_next_start();
    fetch(0);
    if (threadIdx.x < kSmallSteps) smax[threadIdx.x] = slow[threadIdx.x] = 0;
    after_previous();
    if (threadIdx.x < G.count) prm[threadIdx.x] = params[(uint64_t)item * param_stride + G.s0 + threadIdx.x];
    for (uint32_t i = threadIdx.x; i < (1u << G.st[0].r_in); i += kSmallThreads)
        tab[0][i] = Ein[(uint64_t)item * stride + i];
    double m2 = (double)bits_to_m2<R>(mb[G.s0]);
    dcs_scale rec = scale[item];
    for (int i = 0; i < G.count; ++i) {
        const dcs_gather_step& st = G.st[i];
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();  // this step's tables and input; the step before is done with the other buffers
        if (i + 1 < G.count) fetch(i + 1);
        const dcs_param p = prm[i];
        const int e = scale_exponent_fast(m2);
        const double sc = exp2_neg(e);
        rec.logscale += (double)e * 0.69314718055994530942;
        rec.exponent_sum += e;
        if (!isfinite(m2)) rec.flags |= 1u;
        else if (m2 == 0.0) rec.flags |= 2u;
        const uint64_t mask = (1ull << st.r_in) - 1ull;
        const S* E = tab[i & 1];
        S* out = tab[(i & 1) ^ 1];
        const double w0r = p.f0r, w0i = p.f0i, w1r = p.f1r, w1i = p.f1i;
        R lm = 0;
        for (uint32_t cp = threadIdx.x; cp < (1u << st.r_out); cp += kSmallThreads) {
            const S o = gather_entry(E, cp, st, T[i & 1], C[i & 1], mask, st.beta, p.ov & 1, p.y & 1, w0r, w0i, w1r, w1i, sc);
            out[cp] = o;
            lm = fmax(lm, o.x * o.x + o.y * o.y);
        }
        // 32 bits that order like the maximum and keep its exponent, all that the scale takes from it; in FP64 the
        // low half counts only for a maximum below 2^-1042, whose high half is zero
        uint32_t key = sizeof(R) == 4 ? __float_as_uint((float)lm) : (uint32_t)__double2hiint((double)lm);
        key = __reduce_max_sync(0xffffffffu, key);
        if ((threadIdx.x & 31) == 0 && key) atomicMax(&smax[i], key);
        if (sizeof(R) == 8 && !key) {
            key = __reduce_max_sync(0xffffffffu, (uint32_t)__double2loint((double)lm));
            if ((threadIdx.x & 31) == 0 && key) atomicMax(&slow[i], key);
        }
        __syncthreads();
        const unsigned long long word = sizeof(R) == 4 ? (unsigned long long)smax[i]
                                        : smax[i]      ? (unsigned long long)smax[i] << 32 : slow[i];
        m2 = (double)bits_to_m2<R>(word);
        if (threadIdx.x == 0) mb[G.s0 + i + 1] = word;
    }
    const S* fin = tab[G.count & 1];
    for (uint32_t i = threadIdx.x; i < (1u << G.st[G.count - 1].r_out); i += kSmallThreads)
        Eout[(uint64_t)item * stride + i] = fin[i];
    if (threadIdx.x == 0) scale[item] = rec;
}

template <class S>
int run_steps(void* a, void* b, uint64_t stride, const dcs_gather_step* steps, const uint64_t* words,
              const dcs_param* params, uint64_t param_stride, int s0, int count, unsigned long long* maxbits,
              uint64_t maxbits_stride, dcs_scale* scale, int n_items, cudaStream_t stream) {
    const int sms = dcs_host::sm_count();
    int dev = 0;
    if (sms <= 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        dcs_host::set_error("dcs_gather_steps: no current device");
        return DCS_E_CUDA;
    }
    static bool smem_set[64] = {false};
    if (!smem_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(k_gather_small<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(2 * sizeof(S) << kSmallRank));
        if (e != cudaSuccess) return dcs_host::check_cuda(e, "k_gather_small smem attribute");
        smem_set[dev] = true;
    }
    S* bufs[2] = {(S*)a, (S*)b};
    GatherRun G;
    for (int s = s0; s < s0 + count; ++s) {
        const dcs_gather_step& st = steps[s];
        // steps from here on whose tables fit shared memory (two at least: one alone is a launch either way)
        G.count = 0;
        G.s0 = s;
        G.rank = 0;
        while (G.count < kSmallSteps && s + G.count < s0 + count) {
            const dcs_gather_step& t = steps[s + G.count];
            if (t.r_in < 0 || t.r_out < 0 || t.r_in > kSmallRank || t.r_out > kSmallRank || t.nbytes < 1 ||
                t.nbytes > kSmallBytes || t.ncombos < 1 || t.ncombos > kMaxCombos)
                break;
            if (t.r_in > G.rank) G.rank = t.r_in;
            if (t.r_out > G.rank) G.rank = t.r_out;
            G.st[G.count++] = t;
        }
        if (G.count >= 2) {
            const int k = s - s0;
            const int rc = dcs_host::check_cuda(
                dcs_host::launch_after(k_gather_small<S>, dim3(1, n_items), dim3(kSmallThreads), 2 * sizeof(S) << G.rank, stream,
                                       bufs[k & 1], bufs[(k + G.count) & 1], stride, G, words, params, param_stride, maxbits,
                                       maxbits_stride, scale),
                "k_gather_small");
            if (rc) return rc;
            s += G.count - 1;
            continue;
        }
        if (st.nbytes < 1 || st.nbytes > 8 || st.ncombos < 1 || st.ncombos > kMaxCombos || st.r_out > 62 ||
            st.r_in > 62) {
            dcs_host::set_error("dcs_gather_steps: step %d outside the kernel's limits", s);
            return DCS_E_ARG;
        }
        const uint64_t n_out = 1ull << st.r_out;
        const uint64_t want = (n_out + kThreads - 1) / kThreads;
        const unsigned grid = (unsigned)(want < (uint64_t)sms * 8 ? want : (uint64_t)sms * 8);
        const int k = s - s0;
        const int rc = dcs_host::check_cuda(
            dcs_host::launch_after(k_gather<S>, dim3(grid, n_items), dim3(kThreads), 0, stream, bufs[k & 1],
                                   bufs[(k & 1) ^ 1], stride, st, words, s, params, param_stride, maxbits, maxbits_stride,
                                   scale),
            "k_gather");
        if (rc) return rc;
    }
    return DCS_OK;
}

}  // namespace

extern "C" int dcs_gather_steps(int dtype, void* table_a, void* table_b, uint64_t stride, const dcs_gather_step* steps,
                                const uint64_t* words, const dcs_param* params, uint64_t param_stride, int s0,
                                int count, unsigned long long* maxbits, uint64_t maxbits_stride, dcs_scale* scale,
                                int n_items, void* stream) {
    if (!table_a || !table_b || !steps || !words || !params || !maxbits || !scale || s0 < 0 || count < 0 ||
        n_items < 1 || n_items > 65535 || (dtype != DCS_C64 && dtype != DCS_C128)) {
        dcs_host::set_error("dcs_gather_steps: invalid arguments");
        return DCS_E_ARG;
    }
    if (dtype == DCS_C64)
        return run_steps<float2>(table_a, table_b, stride, steps, words, params, param_stride, s0, count, maxbits,
                                 maxbits_stride, scale, n_items, (cudaStream_t)stream);
    return run_steps<double2>(table_a, table_b, stride, steps, words, params, param_stride, s0, count, maxbits,
                              maxbits_stride, scale, n_items, (cudaStream_t)stream);
}
