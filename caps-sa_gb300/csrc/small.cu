// small.cu — suffix arrays of small plain texts in one launch.
//
// A text of a few thousand symbols is all launches and read-backs on the
// general path (ten kernels, three waits: 143 us for 4,099 DNA symbols, of
// which the kernels run 55).  Here one block does all of it in shared memory:
// order-preserving codes of the symbols present (as Packer::new assigns them,
// src/pack.rs:103-167), the bit-packed text, a placement of every suffix by its
// leading 13 bits, and exact comparisons (suffix_cmp_with, src/lcp.rs:184-201)
// inside each bin.  Bound by the latency of one SM and the call's one wait:
// 40 us for the whole call at 4,099 symbols, where the general path takes 143.
// The limit is where the 13-bit bins still hold a record each: 11,389 symbols
// take 159 us on the general path, and would take one SM about twice the
// comparisons of 8,192.
//
// A thread compares at most kBudget windows; a text that needs more (long
// repeats, very uneven symbols) reports it and takes the general path.
#include "small.cuh"

namespace capssa {

namespace {

constexpr int kThreads = 1024;
constexpr int kPer = (int)kSmallText / kThreads;
constexpr int kLogBins = 13;
constexpr uint32_t kBins = 1u << kLogBins;
constexpr uint32_t kBudget = 384;
constexpr uint32_t kPackWords = kSmallText + 4;  // 32-bit words, codes of up to 32 bits

// Exclusive prefix of one value per thread over the block.
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t *s_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = s_w[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        s_w[lane] = w;  // inclusive
    }
    __syncthreads();
    return (warp ? s_w[warp - 1] : 0u) + x - v;
}

// 64 bits of the packed text from bit `at` (big-endian 32-bit words).
__device__ __forceinline__ uint64_t bits_at(const uint32_t *pk, uint32_t at) {
    const uint32_t *w = pk + (at >> 5);
    const uint32_t sh = at & 31;
    const uint32_t hi = __funnelshift_l(w[1], w[0], sh), lo = __funnelshift_l(w[2], w[1], sh);
    return (uint64_t)hi << 32 | lo;
}

template <typename S, typename IT>
__global__ void __launch_bounds__(kThreads)
    small_kernel(const S *__restrict__ text, uint32_t n, int lf, IT *__restrict__ out,
                 int *__restrict__ gave_up) {
    extern __shared__ __align__(16) unsigned char sm[];
    uint32_t *pk = reinterpret_cast<uint32_t *>(sm);                   // packed text
    uint32_t *bins = pk + kPackWords;                                   // counts, then starts
    uint16_t *ord = reinterpret_cast<uint16_t *>(bins + kBins + 4);     // suffix by slot
    uint32_t *abc = reinterpret_cast<uint32_t *>(ord + kSmallText);     // symbols present (bits)
    uint32_t *pre = abc + 2048;                                         // ... before each word
    __shared__ uint32_t s_w[32], s_lo, s_hi, s_sigma;
    const uint32_t tid = threadIdx.x;
    constexpr uint32_t kAbcWords = sizeof(S) == 1 ? 8 : 2048;

    // symbols, and the order-preserving code of each
    S sym[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        const uint32_t i = j * kThreads + tid;
        if (i < n) sym[j] = text[i];
    }
    if (tid == 0) {
        s_lo = 0xFFFFFFFFu;
        s_hi = 0;
    }
    if (sizeof(S) <= 2)
        for (uint32_t i = tid; i < kAbcWords; i += kThreads) abc[i] = 0;
    for (uint32_t i = tid; i < kPackWords; i += kThreads) pk[i] = 0;
    for (uint32_t i = tid; i <= kBins; i += kThreads) bins[i] = 0;
    __syncthreads();
    if (sizeof(S) <= 2) {
#pragma unroll
        for (int j = 0; j < kPer; j++)
            if (j * kThreads + tid < n) {
                const uint32_t v = (uint32_t)sym[j];
                if (!((abc[v >> 5] >> (v & 31)) & 1u)) atomicOr(&abc[v >> 5], 1u << (v & 31));
            }
        __syncthreads();
        // two words a thread
        const uint32_t a = 2 * tid < kAbcWords ? __popc(abc[2 * tid]) : 0u;
        const uint32_t b2 = 2 * tid < kAbcWords ? __popc(abc[2 * tid + 1]) : 0u;
        const uint32_t before = block_prefix(a + b2, s_w);
        if (2 * tid < kAbcWords) {
            pre[2 * tid] = before;
            pre[2 * tid + 1] = before + a;
        }
        if (tid == kThreads - 1) s_sigma = before + a + b2;
        __syncthreads();
    } else {
        uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
        for (int j = 0; j < kPer; j++)
            if (j * kThreads + tid < n) {
                lo = min(lo, (uint32_t)sym[j]);
                hi = max(hi, (uint32_t)sym[j]);
            }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if ((tid & 31) == 0) {
            atomicMin(&s_lo, lo);
            atomicMax(&s_hi, hi);
        }
        __syncthreads();
    }
    const uint32_t top = sizeof(S) <= 2 ? s_sigma - 1 : s_hi - s_lo;  // largest code
    const int b = top ? 32 - __clz((int)top) : 1;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        const uint32_t i = j * kThreads + tid;
        if (i < n) {
            const uint32_t v = (uint32_t)sym[j];
            uint32_t code;
            if (sizeof(S) <= 2)
                code = pre[v >> 5] + __popc(abc[v >> 5] & ((1u << (v & 31)) - 1u));
            else
                code = v - s_lo;
            const uint32_t at = i * (uint32_t)b, sh = at & 31;
            const uint64_t x = (uint64_t)code << (64 - b - (int)sh);  // b + sh <= 63
            if (x >> 32) atomicOr(&pk[at >> 5], (uint32_t)(x >> 32));
            if ((uint32_t)x) atomicOr(&pk[(at >> 5) + 1], (uint32_t)x);
        }
    }
    __syncthreads();

    // placement by the leading bits, truncated at the text's end and padded low
    // (ShorterFirst) or high (LongerFirst): a smaller bin is a smaller suffix
    auto bin_of = [&](uint32_t p) -> uint32_t {
        const uint32_t *w = pk + ((p * (uint32_t)b) >> 5);
        uint32_t k = __funnelshift_l(w[1], w[0], (p * (uint32_t)b) & 31) >> (32 - kLogBins);
        const uint32_t have = (n - p) * (uint32_t)b;
        if (have < (uint32_t)kLogBins) {
            const uint32_t low = (1u << (kLogBins - have)) - 1u;
            k = lf ? (k | low) : (k & ~low);
        }
        return k;
    };
    uint16_t rk[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        const uint32_t p = j * kThreads + tid;
        if (p < n) rk[j] = (uint16_t)atomicAdd(&bins[bin_of(p)], 1u);
    }
    __syncthreads();
    {
        constexpr int kB = (int)kBins / kThreads;
        uint32_t c[kB], sum = 0;
#pragma unroll
        for (int q = 0; q < kB; q++) {
            c[q] = bins[tid * kB + q];
            sum += c[q];
        }
        uint32_t run = block_prefix(sum, s_w);
#pragma unroll
        for (int q = 0; q < kB; q++) {
            bins[tid * kB + q] = run;
            run += c[q];
        }
        if (tid == kThreads - 1) bins[kBins] = n;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        const uint32_t p = j * kThreads + tid;
        if (p < n) ord[bins[bin_of(p)] + rk[j]] = (uint16_t)p;
    }
    __syncthreads();

    // exact order inside the bins: a suffix's place is the number before it
    const uint32_t spw = 64u / (uint32_t)b;
    const uint64_t mask = spw * (uint32_t)b >= 64 ? ~0ull : ~0ull << (64 - spw * (uint32_t)b);
    uint32_t budget = kBudget;
    bool over = false;
    for (uint32_t i = tid; i < n; i += kThreads) {
        const uint32_t p = ord[i], bin = bin_of(p);
        const uint32_t s = bins[bin], e = bins[bin + 1];
        uint32_t place = s;
        for (uint32_t u = s; u < e && !over; u++) {
            const uint32_t q = ord[u];
            if (q == p) continue;
            // q before p?  the later position is the shorter suffix
            const uint32_t lim = n - max(p, q);
            bool q_first = lf ? q < p : q > p;  // one is the other's prefix
            for (uint32_t t = 0; t < lim; t += spw) {
                if (budget-- == 0) {
                    over = true;
                    break;
                }
                const uint64_t x = bits_at(pk, (p + t) * (uint32_t)b) & mask;
                const uint64_t y = bits_at(pk, (q + t) * (uint32_t)b) & mask;
                if (x != y) {
                    const uint32_t d = (uint32_t)__clzll((long long)(x ^ y)) / (uint32_t)b;
                    if (t + d < lim) q_first = y < x;
                    break;
                }
            }
            place += q_first ? 1u : 0u;
        }
        if (over) {
            atomicExch(gave_up, 1);
            break;
        }
        out[place] = (IT)p;
    }
}

template <typename S, typename IT>
cudaError_t launch(Ctx &c, const void *text, uint32_t n, int lf, void *out, int *flag) {
    constexpr size_t smem = kPackWords * 4 + (kBins + 4) * 4 + kSmallText * 2 + 2048 * 8;
    cudaFuncSetAttribute(small_kernel<S, IT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    small_kernel<S, IT><<<1, kThreads, smem, c.stream>>>((const S *)text, n, lf, (IT *)out, flag);
    return cudaGetLastError();
}

template <typename IT>
cudaError_t launch_sym(Ctx &c, const void *text, int sym_bytes, uint32_t n, int lf, void *out,
                       int *flag) {
    if (sym_bytes == 1) return launch<uint8_t, IT>(c, text, n, lf, out, flag);
    if (sym_bytes == 2) return launch<uint16_t, IT>(c, text, n, lf, out, flag);
    return launch<uint32_t, IT>(c, text, n, lf, out, flag);
}

}  // namespace

capssa_status small_build(Ctx &c, const void *text, int sym_bytes, uint32_t n, int longer_first,
                          void *out_sa, int out_bytes, bool *done) {
    *done = false;
    int *flag = c.d_flags + 3;  // cleared at the start of the call
    const cudaError_t e = out_bytes == 4
                              ? launch_sym<uint32_t>(c, text, sym_bytes, n, longer_first, out_sa, flag)
                              : launch_sym<uint64_t>(c, text, sym_bytes, n, longer_first, out_sa, flag);
    c.launches++;
    if (e != cudaSuccess) return cuda_err(c, e, "small text");
    int *h = (int *)c.h_scratch;
    CAPSSA_CUDA(c, cudaEventRecord(c.ev1, c.stream));
    CAPSSA_CUDA(c, cudaMemcpyAsync(h, flag, 4, cudaMemcpyDeviceToHost, c.stream));
    CAPSSA_CUDA(c, cudaStreamSynchronize(c.stream));
    *done = *h == 0;
    return CAPSSA_OK;
}

}  // namespace capssa
