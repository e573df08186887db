// BF16 weight copies.
//
// The engine keeps FP32 masters (Tensor::cuda_data) for AdamW and checkpoints
// (optimisers/AdamWOptimiser.h:24-36, GPT.cpp:128-206); the tensor-core products read BF16 copies.  Each expert weight
// is kept once, transposed and tile-major (common.cuh): the forward products read it with the reduction dimension
// contiguous, the data gradients (dHh = dYg*Wd^T, dXg = dG*Wg^T + dU*Wu^T) read the same blocks the other way round.
#include "common.cuh"

namespace mgpt {

namespace {

// Everything BF16 that is made from the router's weight, one block per expert column: Wr [C,E] fp32 -> [C,E8] bf16 (zero
// in the padding columns; backward) and, where pieces is set, the transposed BF16 pieces [2][NE][C] (hi = bf16(w),
// mid = bf16(w - hi)) with the largest column norm / bias magnitude for the error bound of the screened router.
__global__ void __launch_bounds__(256)
router_copies_kernel(const float* Wr, const float* br, int C, int E, int E8, int NE,
                     bf16* out, bf16* pieces, float* rstat)
{
    pdl_wait();
    __shared__ float red[8];
    const int e = blockIdx.x;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        const float w = e < E ? Wr[(size_t)c * E + e] : 0.0f;
        const bf16 hi = __float2bfloat16(w);
        out[(size_t)c * E8 + e] = hi;
        if (pieces && e < E) {
            pieces[(size_t)e * C + c] = hi;
            pieces[((size_t)NE + e) * C + c] = __float2bfloat16(w - __bfloat162float(hi));
            ss = fmaf(w, w, ss);
        }
    }
    if (!pieces || e >= E) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int i = 0; i < 8; ++i) t += red[i];
        // non-negative floats order like their bit patterns; a NaN (bits above +inf) stays the maximum, so a
        // poisoned weight makes every token take the exact pass
        atomicMax(reinterpret_cast<int*>(rstat), __float_as_int(sqrtf(t) * 1.001f));
        atomicMax(reinterpret_cast<int*>(rstat) + 1, __float_as_int(fabsf(br[e])));
    }
}

}  // namespace

// stat_clear: a kernel before this one on the stream has cleared the statistics
int launch_router_copies(mgpt_moe_layer* L, bool stat_clear, cudaStream_t st)
{
    const Dims& d = L->d;
    const int E8 = (d.E + 7) / 8 * 8;
    if (L->d_rstat && !stat_clear) MGPT_CUDA(cudaMemsetAsync(L->d_rstat, 0, 2 * sizeof(float), st));
    MGPT_CUDA(launch_pdl(router_copies_kernel, E8, 256, 0, st, L->p_data[0], L->p_data[1], d.C, d.E, E8, L->router_ne, L->sWr,
                         L->sWrT2, L->d_rstat));
    MGPT_LAUNCHED("router_copies_kernel");
    return 0;
}

int launch_sync_weights(mgpt_moe_layer* L, cudaStream_t st)
{
    if (L->d.mode != MGPT_MOE_BF16) return 0;
    if (L->router_bound) MGPT_TRY(launch_router_copies(L, false, st));
    if (L->experts_bound) MGPT_TRY(launch_weight_copies(L, st));
    L->shadows_fresh = true;
    return 0;
}

}  // namespace mgpt
