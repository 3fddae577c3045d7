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
// A text whose comparisons come to more than kWork windows of 64 bits over the
// block (long repeats, very uneven symbols) is left to the general path: at once
// where the bins alone show it, else when the count passes kWork.  A bound of 384
// windows for each thread, as before, let all of them run to it: 8,000 symbols in
// two equal halves took 0.86 ms, twice the 0.40 of the general path they then
// took, and 1,000 equal symbols 0.71 ms; 0.37 and 0.52 now.
#include "small.cuh"

namespace capssa {

namespace {

constexpr int kThreads = 1024;
constexpr int kPer = (int)kSmallText / kThreads;
constexpr int kLogBins = 13;
constexpr uint32_t kBins = 1u << kLogBins;
constexpr uint32_t kWork = 1u << 17;
constexpr uint32_t kWorkStep = 16;  // windows a thread compares between looks at the count
constexpr uint32_t kPackWords = kSmallText + 16;  // 32-bit words, codes of up to 32 bits

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

// First bit, of the 32 * W from bits x and y of the packed text (big-endian
// 32-bit words), at which the two differ (32 * W: none), and whether y's is the
// smaller there.
template <int W>
__device__ __forceinline__ uint32_t differ_at(const uint32_t *pk, uint32_t x, uint32_t y,
                                              bool *y_less) {
    const uint32_t *wx = pk + (x >> 5), *wy = pk + (y >> 5);
    uint32_t a[W + 1], b[W + 1];
#pragma unroll
    for (int i = 0; i <= W; i++) {
        a[i] = wx[i];
        b[i] = wy[i];
    }
    uint32_t d = 32 * W;
#pragma unroll
    for (int i = W - 1; i >= 0; i--) {
        const uint32_t u = __funnelshift_l(a[i + 1], a[i], x & 31);
        const uint32_t v = __funnelshift_l(b[i + 1], b[i], y & 31);
        if (u != v) {
            d = 32 * i + (uint32_t)__clz((int)(u ^ v));
            *y_less = v < u;
        }
    }
    return d;
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
    __shared__ uint32_t s_w[32], s_lo, s_hi, s_sigma, s_least, s_work;
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
        s_least = s_work = 0;
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
        uint32_t c[kB], sum = 0, pairs = 0;
#pragma unroll
        for (int q = 0; q < kB; q++) {
            c[q] = bins[tid * kB + q];
            sum += c[q];
            pairs += c[q] * (c[q] - 1);  // (8,192 records: below 2^26 in all)
        }
        pairs = __reduce_add_sync(0xffffffffu, pairs);
        if ((tid & 31) == 0 && pairs) atomicAdd(&s_least, pairs);
        uint32_t run = block_prefix(sum, s_w);
#pragma unroll
        for (int q = 0; q < kB; q++) {
            bins[tid * kB + q] = run;
            run += c[q];
        }
        if (tid == kThreads - 1) bins[kBins] = n;
    }
    __syncthreads();
    if (s_least > kWork) {  // a window for every pair of a bin
        if (tid == 0) *gave_up = 1;
        return;
    }
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        const uint32_t p = j * kThreads + tid;
        if (p < n) ord[bins[bin_of(p)] + rk[j]] = (uint16_t)p;
    }
    __syncthreads();

    // exact order inside the bins: a suffix's place is the number before it.
    // The first 64 bits decide most pairs, and the next 64 most others; further
    // ones go by 256 (zeros past the text's end, where the shorter suffix has
    // decided).
    uint32_t used = 0;  // windows since the last look at the count
    bool over = false;
    for (uint32_t i = tid; i < n; i += kThreads) {
        const uint32_t p = ord[i], bin = bin_of(p);
        const uint32_t s = bins[bin], e = bins[bin + 1];
        uint32_t place = s;
        for (uint32_t u = s; u < e && !over; u++) {
            const uint32_t q = ord[u];
            if (q == p) continue;
            // q before p?  the later position is the shorter suffix
            const uint32_t end = (n - max(p, q)) * (uint32_t)b;
            const uint32_t x = p * (uint32_t)b, y = q * (uint32_t)b;
            bool less = false;
            uint32_t t = differ_at<2>(pk, x, y, &less);
            used++;
            if (t == 64 && t < end) {
                t += differ_at<2>(pk, x + 64, y + 64, &less);
                used++;
            }
            if (t == 128) {
                while (t < end && !over) {
                    const uint32_t d = differ_at<8>(pk, x + t, y + t, &less);
                    t += d;
                    used += 4;
                    if (used >= kWorkStep) {
                        over = atomicAdd(&s_work, used) > kWork;
                        used = 0;
                    }
                    if (d < 256) break;
                }
            }
            // one is the other's prefix, or they differ inside both
            place += (t < end ? less : lf ? q < p : q > p) ? 1u : 0u;
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
