// Gradient of the loss with respect to the per-neuron axonal delays, one fused pass:
//   gradDelay[n] = Ts * sum_{b,t} g[b,n,t] * diff[b,n,t],
//   diff[b,n,t]  = out[b,n,t] * (-1/Ts) + out[b,n,t-1] * (1/Ts)      (out[.., -1] = 0)
// where `out` is the delayed signal the forward pass produced and g the gradient arriving at
// it.  The reference composes this from a two-tap conv, an elementwise product and a tensor
// reduction, writing two full-size temporaries; here g and out are read once (8 algorithmic
// bytes per element, bound by HBM) and nothing but the [nNeurons] result is written.
//
// One CTA per neuron.  Its samples (all rows of the batch) are one sequence of chunks of V samples
// dealt to the threads in turn, so that no lane idles at a row's end whatever T is; a thread asks for
// kDelayGradAhead chunks of both arrays before it uses the first.  What bounds the pass is how many
// requests are in flight: a layer has a few hundred neurons, two CTAs per SM at most.  The sample in
// front of a chunk is the neighbouring lane's last one.  Partial sums are combined by warp shuffles
// and a fixed-order pass over the warps' sums, so the result does not depend on scheduling.
// (256 neurons, 32 x 2000 samples each: 51.7 -> 21.4 us; 512 neurons, 64 x 300: 20.1 -> 16.0 us, with one
// CTA of eight warps per neuron and a row per warp before.)
#include "common.cuh"

namespace sb200 {

constexpr int kDelayGradWarps = 16;
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
template <int V>
__global__ void __launch_bounds__(kDelayGradWarps * 32, 2)
delay_grad_kernel(float *__restrict__ grad_delay, const float *__restrict__ g, const float *__restrict__ out,
                  int64_t nBatch, int64_t nNeurons, int T, float Ts)
{
    constexpr int kThreads = kDelayGradWarps * 32;
    __shared__ float warp_sum[kDelayGradWarps];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const float f0 = -1.0f / Ts, f1 = 1.0f / Ts;
    const unsigned per_row = (unsigned)T / V;                         // chunks of a row
    const int64_t chunks = nBatch * per_row;
    const unsigned step_b = per_row ? kThreads / per_row : 0;    // kThreads chunks further on: rows and chunks
    const unsigned step_q = per_row ? kThreads % per_row : 0;

    for (int64_t n = blockIdx.x; n < nNeurons; n += gridDim.x) {
        float acc[kDelayGradAhead] = {};
        int64_t b = per_row ? threadIdx.x / per_row : 0;
        unsigned q = per_row ? threadIdx.x % per_row : 0;
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
        if (lane == 0) warp_sum[warp] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            float total = 0.0f;
#pragma unroll
            for (int w = 0; w < kDelayGradWarps; ++w) total += warp_sum[w];
            grad_delay[n] = total * Ts;
        }
        __syncthreads();
    }
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
    int64_t grid = nNeurons;
    const int64_t cap = (int64_t)sm_count() * 32;
    if (grid > cap) grid = cap;
    const bool vec = (T % 4 == 0) && aligned16(grad_output) && aligned16(output);
    if (vec)
        delay_grad_kernel<4><<<(unsigned)grid, kDelayGradWarps * 32, 0, (cudaStream_t)stream>>>(
            grad_delay, grad_output, output, nBatch, nNeurons, (int)T, Ts);
    else
        delay_grad_kernel<1><<<(unsigned)grid, kDelayGradWarps * 32, 0, (cudaStream_t)stream>>>(
            grad_delay, grad_output, output, nBatch, nNeurons, (int)T, Ts);
    return check_launch("delay_grad kernel launch");
}
