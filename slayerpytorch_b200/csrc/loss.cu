// Spike-count loss (forward value and gradient) in one pass.
//
// For output spikes s[row, t] (rows = batch x classes) with a target region [lo, hi) and a
// desired number of spikes per row:
//   count      = Ts * sum_{t in region} s[t]
//   c          = float( (double(count) - desired) / (stop - start) * scale )        (one rounding)
//   e[t]       = psp(s outside the region)[t] + (t in region ? c : 0)               (psp = causal FIR, x Ts)
//   loss       = Ts / 2 * sum_{rows, t} e[t]^2
//   dloss/ds   = psp_adjoint(Ts * e)                                                (corr, x Ts)
// which is spikeLoss.numSpikes of the reference with its backward pass (the part of the output
// inside the region enters as a constant).  The reference builds the terms on the host with
// NumPy; a tensor-expression version costs about twenty small launches.  Here one CTA has one
// row: the row, its error signal and the taps sit in shared memory, a warp takes 128 time steps, four
// per lane.  An output layer has a few hundred rows, so what bounds the kernel is the length of one
// row's filters, a chain of loads and FMAs per tap: four chains per lane hide each other's latency, and
// zeros around the row let all lanes run the same taps.  A CTA has four warps; where the rows are short and
// fill the chip by themselves, one, which needs no barrier.
// psp and its adjoint are the same fp32 fused-multiply-add chains as the conv / corr operators
// (ascending taps, x Ts last).  The kernel leaves sum_t e^2 per row (double); the caller adds the
// rows up.
#include "common.cuh"

namespace sb200 {

// out(k, sum) for the N groups of 32 steps behind x, lane by lane; the sum runs over the taps in ascending
// order: x[32 k - i] * f[i] (DIR = -1) or x[32 k + i] * f[i] (DIR = 1), i < K
template <int DIR, int N, class Out>
__device__ __forceinline__ void loss_filter(const float *x, const float *f, int K, Out out)
{
    float acc[N] = {};
#pragma unroll 4
    for (int i = 0; i < K; ++i) {
        const float fi = f[i];
#pragma unroll
        for (int k = 0; k < N; ++k) acc[k] = fmaf(x[32 * k + DIR * i], fi, acc[k]);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) out(k, acc[k]);
}

// One warp's pass over up to 128 steps from t0 on.  Inside the row: four chains and all taps (a trip count
// that no pass changes: 8 rows x 6000 62 us, 71 with the count below).  At its ends: as many chains as there
// are groups of 32 steps left, and no taps that reach only the zeros around the row (65536 x 129: 256 -> 229).
template <int DIR, class Out>
__device__ __forceinline__ void loss_pass(const float *x, const float *f, int K, int t0, int T, int lane, Out out)
{
    const int left = T - t0;
    x += t0 + lane;
    if (left >= 128 && (DIR > 0 || t0 >= K)) {
        loss_filter<DIR, 4>(x, f, K, out);
        return;
    }
    const int taps = min(K, DIR < 0 ? t0 + min(left, 128) : left);
    if (left > 96) loss_filter<DIR, 4>(x, f, taps, out);
    else if (left > 64) loss_filter<DIR, 3>(x, f, taps, out);
    else if (left > 32) loss_filter<DIR, 2>(x, f, taps, out);
    else loss_filter<DIR, 1>(x, f, taps, out);
}

// words of shared memory of a CTA: the taps, the row with K zeros in front, the error signal with
// K zeros behind; both arrays to a whole number of 32 steps
static __host__ __device__ __forceinline__ int loss_span(int T) { return (T + 31) / 32 * 32; }

// WARPS per row
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
num_spikes_loss_kernel(float *__restrict__ grad, double *__restrict__ row_sq, const float *__restrict__ s,
                       const float *__restrict__ desired_count, const float *__restrict__ filt,
                       int64_t rows, int T, int K, int lo, int hi, int span, float Ts, float scale)
{
    extern __shared__ __align__(16) float smem[];
    __shared__ float warp_cnt[WARPS];
    __shared__ double warp_sq[WARPS];
    auto sync = [] {
        if constexpr (WARPS == 1) __syncwarp();
        else __syncthreads();
    };
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int Tp = loss_span(T);
    float *fs = smem;                                    // K taps
    float *x = fs + 2 * K;                               // the row outside the region (K zeros in front)
    float *e = x + Tp;                                   // Ts * e (zeros behind)
    for (int i = threadIdx.x; i < K; i += blockDim.x) {
        fs[i] = filt[i];
        fs[K + i] = 0.0f;
    }
    for (int i = T + threadIdx.x; i < Tp; i += blockDim.x) x[i] = 0.0f;
    for (int i = T + threadIdx.x; i < Tp + K; i += blockDim.x) e[i] = 0.0f;

    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        const float *sr = s + row * (int64_t)T;
        float cnt = 0.0f;
        for (int t = threadIdx.x; t < T; t += blockDim.x) {
            const float v = sr[t];
            const bool in = t >= lo && t < hi;
            x[t] = in ? 0.0f : v;
            if (in) cnt += v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) warp_cnt[warp] = cnt;
        sync();
        cnt = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) cnt += warp_cnt[w];
        const float actual = cnt * Ts;
        const float c = (float)(((double)actual - (double)desired_count[row]) / (double)span * (double)scale);
        double sq = 0.0;
        for (int t0 = warp * 128; t0 < T; t0 += WARPS * 128)
            loss_pass<-1>(x, fs, K, t0, T, lane, [&](int k, float sum) {
                const int t = t0 + 32 * k + lane;
                if (t < T) {
                    const float err = sum * Ts + ((t >= lo && t < hi) ? c : 0.0f);
                    e[t] = err * Ts;
                    sq += (double)err * (double)err;
                }
            });
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) warp_sq[warp] = sq;
        sync();
        if (threadIdx.x == 0) {
            double total = 0.0;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) total += warp_sq[w];
            row_sq[row] = total;
        }
        float *gr = grad + row * (int64_t)T;
        for (int t0 = warp * 128; t0 < T; t0 += WARPS * 128)
            loss_pass<1>(e, fs, K, t0, T, lane, [&](int k, float sum) {
                const int t = t0 + 32 * k + lane;
                if (t < T) gr[t] = sum * Ts;
            });
        sync();
    }
}

}  // namespace sb200

extern "C" int slayer_b200_num_spikes_loss(float *grad, double *row_sq, const float *s, const float *desired_count,
                                           const float *filter, int64_t rows, int64_t T, int64_t K,
                                           int64_t start, int64_t stop, float Ts, float scale, void *stream)
{
    using namespace sb200;
    clear_error();
    SB200_REQUIRE(rows >= 0 && T >= 0 && K >= 0, "num_spikes_loss: negative size");
    SB200_REQUIRE(stop != start, "num_spikes_loss: empty target region");
    if (rows == 0 || T == 0) return SLAYER_B200_OK;
    SB200_REQUIRE(grad && row_sq && s && desired_count && (filter || K == 0), "num_spikes_loss: null pointer");
    SB200_REQUIRE(grad != s, "num_spikes_loss: grad must not alias s");
    const int64_t Keff = K < T ? K : T;
    // taps and zeros, the row, the error signal and zeros
    const size_t smem = T < (1 << 24) ? sizeof(float) * (3 * (size_t)Keff + 2 * (size_t)loss_span((int)T)) : SIZE_MAX;
    if (smem > 200 * 1024) {
        set_error("num_spikes_loss: rows of %lld steps do not fit the kernel's shared memory", (long long)T);
        return SLAYER_B200_EUNSUPPORTED;
    }
    // the slice [start:stop] of a row of T samples, as Python slicing resolves it
    int64_t lo = start < 0 ? start + T : start, hi = stop < 0 ? stop + T : stop;
    lo = lo < 0 ? 0 : (lo > T ? T : lo);
    hi = hi < 0 ? 0 : (hi > T ? T : hi);
    // us with one warp per row / four: 65536 x 50 84 / 113, 131072 x 10 64 / 129, 3200 x 20 10 / 12, 16384 x 256 102 / 105,
    // but 640 x 300 21 / 14, 2368 x 100 16 / 14, 3200 x 130 21 / 20, 16384 x 500 193 / 188, 3200 x 2000 203 / 151
    const int64_t sms = sm_count();
    const bool one = T <= 32 || (T <= 256 && rows >= 32 * sms);
    auto kern = one ? num_spikes_loss_kernel<1> : num_spikes_loss_kernel<4>;
    int rc = reserve_dynamic_smem((const void *)kern, smem);
    if (rc) return rc;
    const int64_t cap = sms * (one ? 32 : 16);
    kern<<<(unsigned)(rows < cap ? rows : cap), one ? 32 : 128, smem, (cudaStream_t)stream>>>(
        grad, row_sq, s, desired_count, filter, rows, (int)T, (int)Keff, (int)lo, (int)hi, (int)(stop - start), Ts, scale);
    return check_launch("num_spikes_loss kernel launch");
}
