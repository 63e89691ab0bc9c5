// Gradient of the loss with respect to the per-neuron axonal delays, one fused pass:
//   gradDelay[n] = Ts * sum_{b,t} g[b,n,t] * diff[b,n,t],
//   diff[b,n,t]  = out[b,n,t] * (-1/Ts) + out[b,n,t-1] * (1/Ts)      (out[.., -1] = 0)
// where `out` is the delayed signal the forward pass produced and g the gradient arriving at
// it.  The reference composes this from a two-tap conv, an elementwise product and a tensor
// reduction, writing two full-size temporaries; here g and out are read once (8 algorithmic
// bytes per element, bound by HBM) and nothing but the [nNeurons] result is written.
//
// One CTA of 1, 4, 8 or 16 warps per neuron.  Its samples (all rows of the batch) are one sequence of
// chunks of V samples dealt to the threads in turn, so that no lane idles at a row's end whatever T is; a
// thread asks for kDelayGradAhead chunks of both arrays before it uses the first.  What bounds the pass
// is how many requests are in flight: a CTA large enough that a layer of a few hundred neurons fills
// the chip, but no larger than the neuron's chunks and the other neurons leave work for (delay_grad_warps).
// The sample in front of a chunk is the neighbouring lane's last one.  Partial sums are combined by warp
// shuffles and a fixed-order pass over the warps' sums, so the result does not depend on scheduling.
#include "common.cuh"

namespace sb200 {

constexpr int kDelayGradAhead = 4;

template <int V>
__device__ __forceinline__ void load_chunk(float (&v)[V], const float *p)
{
    if constexpr (V == 4) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        v[0] = __ldg(p);
    }
}

// V = 4: rows on 16-byte boundaries (T % 4 == 0 and aligned arrays); V = 1: any
template <int V, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 32 / WARPS)
delay_grad_kernel(float *__restrict__ grad_delay, const float *__restrict__ g, const float *__restrict__ out,
                  int64_t nBatch, int64_t nNeurons, int T, float Ts)
{
    constexpr int kThreads = WARPS * 32;
    __shared__ float warp_sum[WARPS];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const float f0 = -1.0f / Ts, f1 = 1.0f / Ts;
    const unsigned per_row = (unsigned)T / V;                         // chunks of a row
    const int64_t chunks = nBatch * per_row;
    const unsigned step_b = per_row ? kThreads / per_row : 0;    // kThreads chunks further on: rows and chunks
    const unsigned step_q = per_row ? kThreads % per_row : 0;
    const unsigned b0 = per_row ? threadIdx.x / per_row : 0;     // this thread's first chunk of a neuron
    const unsigned q0 = per_row ? threadIdx.x % per_row : 0;

    for (int64_t n = blockIdx.x; n < nNeurons; n += gridDim.x) {
        float acc[kDelayGradAhead] = {};
        int64_t b = b0;
        unsigned q = q0;
        for (int64_t c = warp * 32; c < chunks; c += kThreads * kDelayGradAhead) {      // uniform over the warp
            float gv[kDelayGradAhead][V], ov[kDelayGradAhead][V], before[kDelayGradAhead];
            bool ok[kDelayGradAhead], first[kDelayGradAhead];
#pragma unroll
            for (int k = 0; k < kDelayGradAhead; ++k) {
                ok[k] = b < nBatch;
                first[k] = q == 0;
                before[k] = 0.0f;
#pragma unroll
                for (int i = 0; i < V; ++i) gv[k][i] = ov[k][i] = 0.0f;
                if (ok[k]) {
                    const int64_t at = (b * nNeurons + n) * (int64_t)T + (int64_t)q * V;
                    load_chunk<V>(gv[k], g + at);
                    load_chunk<V>(ov[k], out + at);
                    if (lane == 0 && q > 0) before[k] = __ldg(out + at - 1);
                }
                b += step_b;
                q += step_q;
                if (q >= per_row) { q -= per_row; ++b; }
            }
#pragma unroll
            for (int k = 0; k < kDelayGradAhead; ++k) {
                float prev = __shfl_up_sync(0xffffffffu, ov[k][V - 1], 1);
                if (lane == 0) prev = before[k];
                if (first[k]) prev = 0.0f;
                if (ok[k]) {
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        acc[k] = fmaf(gv[k][i], fmaf(prev, f1, ov[k][i] * f0), acc[k]);
                        prev = ov[k][i];
                    }
                }
            }
        }
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < kDelayGradAhead; ++k) sum += acc[k];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if constexpr (WARPS == 1) {
            if (lane == 0) grad_delay[n] = sum * Ts;
        } else {
            if (lane == 0) warp_sum[warp] = sum;
            __syncthreads();
            if (threadIdx.x == 0) {
                float total = 0.0f;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) total += warp_sum[w];
                grad_delay[n] = total * Ts;
            }
            __syncthreads();
        }
    }
}

// Warps per neuron (one warp: no barrier, 32 neurons at a time on an SM).  chunks: of one neuron.
// Times in us with 1 / 4 / 8 / 16 warps (neurons: samples of each):
//   16384: 1 x 300       14 /  27 /  43 /  80       one pass of a warp
//   4096: 8 x 300        23 /  27 /  27 /  39       enough neurons, few passes
//   512: 4 x 300         10 /   8 /   8 /  10       one pass of four warps
//   8192: 8 x 1450      211 / 186 / 201 / 219       enough neurons, many passes
//   512: 64 x 300        49 /  25 /  23 /  25       a few neurons per SM, a few passes
//   512: 512 x 300      305 / 121 / 123 / 113       (5.6 TB/s)
//   256: 32 x 2000      131 /  51 /  37 /  33       fewer than two neurons per SM
static int delay_grad_warps(int64_t nNeurons, int64_t chunks)
{
    const int64_t sms = sm_count();
    if (chunks <= 128 || (nNeurons >= 16 * sms && chunks <= 2048)) return 1;
    if (chunks <= 1024 || nNeurons >= 8 * sms) return 4;
    if (chunks <= 8192 && nNeurons >= 2 * sms) return 8;
    return 16;
}

template <int V>
static void launch_delay_grad(float *grad_delay, const float *g, const float *out, int64_t nBatch, int64_t nNeurons,
                              int T, float Ts, cudaStream_t stream)
{
    const int warps = delay_grad_warps(nNeurons, nBatch * (T / V));
    auto kern = warps == 1 ? delay_grad_kernel<V, 1> : warps == 4 ? delay_grad_kernel<V, 4>
              : warps == 8 ? delay_grad_kernel<V, 8> : delay_grad_kernel<V, 16>;
    const int64_t cap = (int64_t)sm_count() * 32;
    kern<<<(unsigned)(nNeurons < cap ? nNeurons : cap), warps * 32, 0, stream>>>(grad_delay, g, out, nBatch, nNeurons, T, Ts);
}

}  // namespace sb200

extern "C" int slayer_b200_delay_grad(float *grad_delay, const float *grad_output, const float *output,
                                      int64_t nBatch, int64_t nNeurons, int64_t T, float Ts, void *stream)
{
    using namespace sb200;
    clear_error();
    SB200_REQUIRE(nBatch >= 0 && nNeurons >= 0 && T >= 0, "delay_grad: negative size");
    SB200_REQUIRE(T < (1LL << 31) - 256, "delay_grad: T=%lld too large", (long long)T);
    if (nNeurons == 0) return SLAYER_B200_OK;
    SB200_REQUIRE(grad_delay != nullptr, "delay_grad: null pointer");
    SB200_REQUIRE(nBatch == 0 || T == 0 || (grad_output && output), "delay_grad: null pointer");
    const bool vec = (T % 4 == 0) && aligned16(grad_output) && aligned16(output);
    (vec ? launch_delay_grad<4> : launch_delay_grad<1>)(grad_delay, grad_output, output, nBatch, nNeurons, (int)T, Ts,
                                                        (cudaStream_t)stream);
    return check_launch("delay_grad kernel launch");
}
