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
// zeros around the row let all lanes run the same taps.  (640 rows x 300: 26.1 -> 11.4 us; 3200 x 2000: 303 -> 144 us,
// with one warp per row before, the sum over the rows included.)
// psp and its adjoint are the same fp32 fused-multiply-add chains as the conv / corr operators
// (ascending taps, x Ts last).  The kernel leaves sum_t e^2 per row (double); the caller adds the
// rows up.
#include "common.cuh"

namespace sb200 {

constexpr int kLossWarps = 4;

// sum over taps, ascending: acc[k] += x[32 k - i] * f[i] (DIR = -1) or x[32 k + i] * f[i] (DIR = 1)
template <int DIR>
__device__ __forceinline__ void loss_filter(float (&acc)[4], const float *x, const float *f, int K)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = 0.0f;
#pragma unroll 4
    for (int i = 0; i < K; ++i) {
        const float fi = f[i];
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = fmaf(x[32 * k + DIR * i], fi, acc[k]);
    }
}

// words of shared memory of a CTA: the taps, the row with K zeros in front, the error signal with
// K zeros behind; both arrays to a whole number of 128 steps
static __host__ __device__ __forceinline__ int loss_span(int T) { return (T + 127) / 128 * 128; }

__global__ void __launch_bounds__(kLossWarps * 32)
num_spikes_loss_kernel(float *__restrict__ grad, double *__restrict__ row_sq, const float *__restrict__ s,
                       const float *__restrict__ desired_count, const float *__restrict__ filt,
                       int64_t rows, int T, int K, int lo, int hi, int span, float Ts, float scale)
{
    extern __shared__ __align__(16) float smem[];
    __shared__ float warp_cnt[kLossWarps];
    __shared__ double warp_sq[kLossWarps];
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
        __syncthreads();
        cnt = 0.0f;
#pragma unroll
        for (int w = 0; w < kLossWarps; ++w) cnt += warp_cnt[w];
        const float actual = cnt * Ts;
        const float c = (float)(((double)actual - (double)desired_count[row]) / (double)span * (double)scale);
        double sq = 0.0;
        float acc[4];
        for (int t0 = warp * 128; t0 < T; t0 += kLossWarps * 128) {
            loss_filter<-1>(acc, x + t0 + lane, fs, K);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int t = t0 + 32 * k + lane;
                if (t < T) {
                    const float err = acc[k] * Ts + ((t >= lo && t < hi) ? c : 0.0f);
                    e[t] = err * Ts;
                    sq += (double)err * (double)err;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) warp_sq[warp] = sq;
        __syncthreads();
        if (threadIdx.x == 0) {
            double total = 0.0;
#pragma unroll
            for (int w = 0; w < kLossWarps; ++w) total += warp_sq[w];
            row_sq[row] = total;
        }
        float *gr = grad + row * (int64_t)T;
        for (int t0 = warp * 128; t0 < T; t0 += kLossWarps * 128) {
            loss_filter<1>(acc, e + t0 + lane, fs, K);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int t = t0 + 32 * k + lane;
                if (t < T) gr[t] = acc[k] * Ts;
            }
        }
        __syncthreads();
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
    int rc = reserve_dynamic_smem((const void *)num_spikes_loss_kernel, smem);
    if (rc) return rc;
    int64_t blocks = rows;
    const int64_t cap = (int64_t)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    num_spikes_loss_kernel<<<(unsigned)blocks, kLossWarps * 32, smem, (cudaStream_t)stream>>>(
        grad, row_sq, s, desired_count, filter, rows, (int)T, (int)Keff, (int)lo, (int)hi, (int)(stop - start), Ts, scale);
    return check_launch("num_spikes_loss kernel launch");
}
