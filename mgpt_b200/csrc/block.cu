// The transformer block's glue around the MoE layer, fused:
//
//   forward   x2 = x1 + moe(rmsnorm(x1) * scale)            layers/TransformerBlock.cpp:42-46
//   backward  d_x1 = dout + rmsnorm_backward(d_moe_in)      layers/TransformerBlock.cpp:80-84
//
// The reference runs these as separate passes over [N, C]: rms_norm_into writes the normalised rows twice (x_hat
// and the scaled output, utils/Tensor.cpp:785-800), add_into makes the skip connection, rms_norm_backward_into
// reads x_hat back (utils/Tensor.cpp:1674-1690) and another add_into forms d_x1.  Here the norm writes only the
// layer's input (in the tokens' dtype) and one float per token; the skip connection is folded into the combine
// write; backward recomputes x_hat from x1 and the saved 1/rms and forms d_x1 in the same pass that adds dout.
#include "common.cuh"

namespace mgpt {

namespace {

__device__ __forceinline__ float ld_f32(const float* p) { return *p; }
__device__ __forceinline__ float ld_f32(const bf16* p) { return __bfloat162float(*p); }

// V consecutive elements, V = 1 or 8
template <int V> __device__ __forceinline__ void ld_v(const float* p, float (&v)[V])
{
    if constexpr (V == 1) {
        v[0] = *p;
    } else {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}
template <int V> __device__ __forceinline__ void ld_v(const bf16* p, float (&v)[V])
{
    if constexpr (V == 1) {
        v[0] = __bfloat162float(*p);
    } else {
        const uint4 u = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
}
template <int V> __device__ __forceinline__ void st_v(float* p, const float (&v)[V])
{
    if constexpr (V == 1) {
        *p = v[0];
    } else {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
}
template <int V> __device__ __forceinline__ void st_v(bf16* p, const float (&v)[V])
{
    if constexpr (V == 1) {
        *p = __float2bfloat16(v[0]);
    } else {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// one warp per token: r = 1/sqrt(mean(x^2) + eps), out = (x*r)*scale.  Bound by latency: eight loads in flight in the sum
// (whose order of additions fixes r, and with it the routing), 16-byte accesses in the second pass where the pointers allow
// (V = 8).  8.0 -> 7.3 us for 6000 x 768 BF16.
template <typename TIo, int V>
__global__ void __launch_bounds__(256)
block_rmsnorm_fwd_kernel(const TIo* x, const float* scale, float eps, int N, int C,
                         TIo* out, float* rs)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int tok = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tok >= N) return;
    const TIo* xr = x + (size_t)tok * C;
    float ss = 0.0f;
#pragma unroll 8
    for (int c = lane; c < C; c += 32) {
        const float v = ld_f32(xr + c);
        ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)C), eps)));
    if (lane == 0) rs[tok] = r;
    TIo* orow = out + (size_t)tok * C;
#pragma unroll 2
    for (int c = lane * V; c < C; c += 32 * V) {
        float xv[V], sv[V];
        ld_v<V>(xr + c, xv);
        ld_v<V>(scale + c, sv);
#pragma unroll
        for (int i = 0; i < V; ++i) xv[i] = __fmul_rn(__fmul_rn(xv[i], r), sv[i]);
        st_v<V>(orow + c, xv);
    }
}

// d_x1 = dout + r*(g*scale - x_hat*<g*scale, x_hat>/C), x_hat = x1*r, g = d_in;  d_scale[c] += sum over tokens of g*x_hat.
// A group of GW warps per token, tokens grid-strided.  A thread always has the same columns, so each group sums d_scale in
// a shared row of its own with plain loads and stores (one row for the CTA took shared FP32 atomics, a compare-and-swap
// loop: with them and 2-byte accesses 37.5 us for 6000 x 768 BF16, now 14.6); one atomic per column and CTA at the end.
// GW is the smallest power of two whose 8 / GW rows of C floats fit the 48 KiB that need no opt-in (less `dots`).
constexpr size_t BWD_PART = 48 * 1024 - 32;
template <typename TIo, int V, int GW>
__global__ void __launch_bounds__(256)
block_bwd_kernel(const TIo* x1, const float* scale, const float* rs,
                 const TIo* g_in, const TIo* dout, int N, int C, TIo* d_x1,
                 float* d_scale)
{
    pdl_wait();
    constexpr int GROUPS = 8 / GW, GT = 32 * GW;    // threads of a group
    extern __shared__ __align__(16) float part[];   // [GROUPS][C]
    __shared__ float dots[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = threadIdx.x / GT, gt = threadIdx.x % GT;
    float* mine = part + (size_t)group * C;
    for (int c = gt; c < C; c += GT) mine[c] = 0.0f;
    __syncthreads();
    const int stride = gridDim.x * GROUPS;
    for (int tok0 = blockIdx.x * GROUPS; tok0 < N; tok0 += stride) {
        const int tok = tok0 + group;
        const bool have = tok < N;                  // (the barriers below are everyone's)
        const size_t o = (size_t)tok * C;
        const float r = have ? rs[tok] : 0.0f;
        float dot = 0.0f;
        if (have)
#pragma unroll 2
            for (int c = gt * V; c < C; c += GT * V) {
                float xv[V], gv[V], sv[V];
                prefetch_l1(dout + o + c);
                ld_v<V>(x1 + o + c, xv);
                ld_v<V>(g_in + o + c, gv);
                ld_v<V>(scale + c, sv);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const float xh = __fmul_rn(xv[i], r);
                    dot = fmaf(__fmul_rn(gv[i], sv[i]), xh, dot);
                    xv[i] = gv[i] * xh;
                }
                if (d_scale) {
                    float pv[V];
                    ld_v<V>(mine + c, pv);
#pragma unroll
                    for (int i = 0; i < V; ++i) pv[i] += xv[i];
                    st_v<V>(mine + c, pv);
                }
            }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, s);
        if constexpr (GW > 1) {
            if (lane == 0) dots[warp] = dot;
            __syncthreads();
            dot = 0.0f;
#pragma unroll
            for (int i = 0; i < GW; ++i) dot += dots[group * GW + i];
            __syncthreads();
        }
        const float m = dot / (float)C;
        if (have)
#pragma unroll 2
            for (int c = gt * V; c < C; c += GT * V) {
                float xv[V], gv[V], sv[V], dv[V];
                if (tok + stride < N) {
                    prefetch_l1(x1 + o + (size_t)stride * C + c);
                    prefetch_l1(g_in + o + (size_t)stride * C + c);
                }
                ld_v<V>(x1 + o + c, xv);
                ld_v<V>(g_in + o + c, gv);
                ld_v<V>(scale + c, sv);
                ld_v<V>(dout + o + c, dv);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const float xh = __fmul_rn(xv[i], r);
                    const float dxh = __fmul_rn(gv[i], sv[i]);
                    const float dn = r * (dxh - xh * m);
                    dv[i] += dn;
                }
                st_v<V>(d_x1 + o + c, dv);
            }
    }
    __syncthreads();
    if (d_scale)
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            float t = 0.0f;
#pragma unroll
            for (int i = 0; i < GROUPS; ++i) t += part[(size_t)i * C + c];
            atomicAdd(d_scale + c, t);
        }
}

template <typename TIo>
cudaError_t launch_block_bwd(const TIo* x1, const float* scale, const float* rs, const TIo* g_in, const TIo* dout, int n, int C,
                             TIo* d_x1, float* d_scale, int sms, cudaStream_t st)
{
    const bool vec = (((uintptr_t)x1 | (uintptr_t)scale | (uintptr_t)dout | (uintptr_t)d_x1) & 15) == 0;      // (C: a multiple of 8)
    int gw = 1;
    while (gw < 8 && (size_t)(8 / gw) * C * sizeof(float) > BWD_PART) gw *= 2;
    const int groups = 8 / gw, blocks = (n + groups - 1) / groups, grid = blocks < 4 * sms ? blocks : 4 * sms;
    const size_t sm = (size_t)groups * C * sizeof(float);
    if (sm > BWD_PART)                               // one row of 12281..12288 columns
        for (const void* f : {(const void*)block_bwd_kernel<TIo, 8, 8>, (const void*)block_bwd_kernel<TIo, 1, 8>}) {
            const cudaError_t err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            if (err != cudaSuccess) return err;
        }
#define MGPT_BWD(GW)                                                                                                       \
    (vec ? launch_pdl(block_bwd_kernel<TIo, 8, GW>, grid, 256, sm, st, x1, scale, rs, g_in, dout, n, C, d_x1, d_scale)     \
         : launch_pdl(block_bwd_kernel<TIo, 1, GW>, grid, 256, sm, st, x1, scale, rs, g_in, dout, n, C, d_x1, d_scale))
    return gw == 1 ? MGPT_BWD(1) : gw == 2 ? MGPT_BWD(2) : gw == 4 ? MGPT_BWD(4) : MGPT_BWD(8);
#undef MGPT_BWD
}

template <typename TIo>
cudaError_t launch_block_fwd(const TIo* x, const float* scale, float eps, int n, int C, TIo* out, float* rs, cudaStream_t st)
{
    const bool vec = (((uintptr_t)x | (uintptr_t)scale) & 15) == 0;
    return vec ? launch_pdl(block_rmsnorm_fwd_kernel<TIo, 8>, (n + 7) / 8, 256, 0, st, x, scale, eps, n, C, out, rs)
               : launch_pdl(block_rmsnorm_fwd_kernel<TIo, 1>, (n + 7) / 8, 256, 0, st, x, scale, eps, n, C, out, rs);
}

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

struct BlockWs {
    size_t ln2, rs, d_in, moe, total;
};
BlockWs block_ws(const mgpt_moe_layer* L, int n, int io)
{
    const size_t el = io == MGPT_MOE_IO_BF16 ? 2 : 4;
    BlockWs b;
    size_t off = 0;
    b.ln2 = off; off = align256(off + (size_t)n * L->d.C * el + 1);
    b.rs = off; off = align256(off + (size_t)n * 4 + 1);
    b.d_in = off; off = align256(off + (size_t)n * L->d.C * el + 1);
    b.moe = off;
    b.total = off + mgpt_moe_workspace_bytes(L, n);
    return b;
}

}  // namespace

}  // namespace mgpt

using namespace mgpt;

extern "C" {

size_t mgpt_moe_block_workspace_bytes(const mgpt_moe_layer* L, int n_tokens, int io)
{
    if (!L || n_tokens < 0) return 0;
    return block_ws(L, n_tokens, io).total;
}

int mgpt_moe_block_forward(mgpt_moe_layer* L, const void* x1, const float* rms_scale, float eps, void* x2, int n_tokens,
                           int io, void* workspace, size_t ws_bytes, mgpt_stream_t stream)
{
    if (!L || !rms_scale) return fail(MGPT_MOE_EINVAL, "null argument");
    if (n_tokens <= 0 || !x1 || !x2) return fail(MGPT_MOE_EINVAL, "bad token buffer");
    if (io != MGPT_MOE_IO_F32 && io != MGPT_MOE_IO_BF16) return fail(MGPT_MOE_EINVAL, "unknown io dtype");
    if (!workspace || ((uintptr_t)workspace & 255)) return fail(MGPT_MOE_EINVAL, "workspace must be 256-byte aligned");
    const BlockWs b = block_ws(L, n_tokens, io);
    if (ws_bytes < b.total) return fail(MGPT_MOE_ENOMEM, "workspace smaller than mgpt_moe_block_workspace_bytes()");
    MGPT_CUDA(cudaSetDevice(L->device));
    cudaStream_t st = (cudaStream_t)stream;
    char* ws = (char*)workspace;
    float* rs = (float*)(ws + b.rs);
    if (io == MGPT_MOE_IO_F32)
        MGPT_CUDA(launch_block_fwd((const float*)x1, rms_scale, eps, n_tokens, L->d.C, (float*)(ws + b.ln2), rs, st));
    else
        MGPT_CUDA(launch_block_fwd((const bf16*)x1, rms_scale, eps, n_tokens, L->d.C, (bf16*)(ws + b.ln2), rs, st));
    MGPT_LAUNCHED("block_rmsnorm_fwd_kernel");
    // x2 = x1 + moe(ln2): the skip connection rides on the combine write
    return mgpt_moe_forward_residual(L, ws + b.ln2, x1, x2, n_tokens, io, ws + b.moe, ws_bytes - b.moe, stream);
}

int mgpt_moe_block_backward(mgpt_moe_layer* L, const void* x1, const float* rms_scale, float* d_rms_scale,
                            const void* dout, void* d_x1, int io, void* workspace, size_t ws_bytes, mgpt_stream_t stream)
{
    if (!L || !rms_scale) return fail(MGPT_MOE_EINVAL, "null argument");
    if (!L->fwd_done) return fail(MGPT_MOE_ESTATE, "backward without a forward");
    if (!x1 || !dout || !d_x1) return fail(MGPT_MOE_EINVAL, "null token buffer");
    const int n = L->last_n;
    const BlockWs b = block_ws(L, n, io);
    if (ws_bytes < b.total) return fail(MGPT_MOE_ENOMEM, "workspace smaller than mgpt_moe_block_workspace_bytes()");
    char* ws = (char*)workspace;
    if (ws + b.moe != (char*)L->last_ws) return fail(MGPT_MOE_ESTATE, "backward must reuse the forward's workspace");
    if (n == 0) return 0;
    MGPT_CUDA(cudaSetDevice(L->device));
    cudaStream_t st = (cudaStream_t)stream;
    // the layer's backward: input ln2 (kept by forward), upstream gradient dout, gradient w.r.t. ln2 into the block's buffer
    MGPT_TRY(mgpt_moe_backward(L, ws + b.ln2, dout, ws + b.d_in, io, ws + b.moe, ws_bytes - b.moe, stream));
    int sms = 0;
    MGPT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, L->device));
    if ((size_t)L->d.C * sizeof(float) > 48 * 1024) return fail(MGPT_MOE_EINVAL, "embed_dim above 12288 is not supported by the block glue");
    const float* rs = (const float*)(ws + b.rs);
    if (io == MGPT_MOE_IO_F32)
        MGPT_CUDA(launch_block_bwd((const float*)x1, rms_scale, rs, (const float*)(ws + b.d_in), (const float*)dout, n, L->d.C,
                                   (float*)d_x1, d_rms_scale, sms, st));
    else
        MGPT_CUDA(launch_block_bwd((const bf16*)x1, rms_scale, rs, (const bf16*)(ws + b.d_in), (const bf16*)dout, n, L->d.C,
                                   (bf16*)d_x1, d_rms_scale, sms, st));
    MGPT_LAUNCHED("block_bwd_kernel");
    return 0;
}

}  // extern "C"
