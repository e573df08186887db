// AdamW over the layer's own parameters, fused with the refresh of the BF16 weight copies.
//
// The reference's optimiser calls Tensor::adamw_step once per parameter tensor
// (optimisers/AdamWOptimiser.h:24-36; CPU arithmetic utils/Tensor.cpp:683-699, GPU kernel
// utils/cuda_ops.cu:723-738) and the tensor-core products would then need a separate pass that
// re-reads every FP32 master to rebuild its BF16 copy.  Here one launch updates w, m, v of every
// tensor and writes the copy from the value it just computed, so an optimiser step costs the
// AdamW traffic plus 2 bytes per weight.
//
// Arithmetic: the CPU arm's, operation for operation (separate FP32 roundings, IEEE sqrt and
// divide), so w, m, v match the reference bit for bit:
//   m = b1*m + (1-b1)*g;  v = b2*v + ((1-b2)*g)*g;  w = w - (lr*wd)*w;
//   w = w - (lr*(m*ms)) / (sqrt(v*vs) + eps),   ms = 1/(1-b1^t), vs = 1/(1-b2^t)  (host, powf)
#include <cmath>

#include "common.cuh"

namespace mgpt {

namespace {

struct AdamwScalars {
    float b1, b2, omb1, omb2, eps, lr, lrwd, ms, vs;
    float clip;       // > 0: the gradient is clamped to [-clip, clip] first (the GPU arm's 10, utils/cuda_ops.cu:728)
    int skip_bad;     // != 0: an element whose gradient is NaN or Inf is left as it is (utils/cuda_ops.cu:727)
};

__device__ __forceinline__ void adamw_elem(float& w, float g, float& m, float& v, const AdamwScalars& a)
{
    if (a.skip_bad && !isfinite(g)) return;
    if (a.clip > 0.0f) g = fminf(fmaxf(g, -a.clip), a.clip);
    m = __fadd_rn(__fmul_rn(a.b1, m), __fmul_rn(a.omb1, g));
    v = __fadd_rn(__fmul_rn(a.b2, v), __fmul_rn(__fmul_rn(a.omb2, g), g));
    const float mh = __fmul_rn(m, a.ms), vh = __fmul_rn(v, a.vs);
    w = __fsub_rn(w, __fmul_rn(a.lrwd, w));
    w = __fsub_rn(w, __fdiv_rn(__fmul_rn(a.lr, mh), __fadd_rn(__fsqrt_rn(vh), a.eps)));
}

// The expert matrices and their BF16 copies.  One block = one 64 x 128 tile of one expert's [rows, cols] matrix, which is
// exactly one 16 KiB block of the transposed tile-major copy (common.cuh); the tile's 16 float4 per thread are all in
// flight at once, rows are touched 512 bytes at a time and the transposition goes through shared memory as packed row
// pairs in 16-byte pieces.  Bound by HBM: 16 bytes read, 12 + 2 written per weight.  (32 x 32 tiles of scalars, 16 bytes in
// flight per thread and two copies: 5.4 TB/s of 32 bytes per weight, 549 us per 92 M weights.)
// The block of tile 0 also takes the bias vector that goes with the matrix; blockIdx.y = 3E is the router.
struct WeightsArgs {
    float* const* w[6];                  // Wg Wu Wd bg bu bd, per expert
    const float* const* g[6];
    float* const* m[6];
    float* const* v[6];
    float* const* router[4];             // {w, g, m, v}[2]: Wr, br; null: not bound
    bf16* copyT[3];                      // transposed tile-major copies (tensor-core products)
    bf16* copy[3];                       // or copies as stored (CUDA-core products on BF16 data)
    int C, H, E;
    float* rstat;                        // the router's error-bound statistics, cleared for the kernel that follows
};

// ADAM: update in place, else only the copies are written from w.
template <bool ADAM, bool VEC>
__global__ void __launch_bounds__(256, 2) expert_weights_kernel(const WeightsArgs p, const AdamwScalars a)
{
    pdl_wait();
    __shared__ __align__(16) uint32_t S[32 * 128];
    const int tid = threadIdx.x;
    if (blockIdx.y == 3 * p.E) {
        if (ADAM) {
            if (blockIdx.x == 0 && tid < 2 && p.rstat) p.rstat[tid] = 0.0f;
            if (p.router[0])
                for (int j = 0; j < 2; ++j) {
                    float *w = p.router[0][j], *m = p.router[2][j], *v = p.router[3][j];
                    const float* g = p.router[1][j];
                    const int len = j == 0 ? p.C * p.E : p.E;
                    for (int i = blockIdx.x * 256 + tid; i < len; i += gridDim.x * 256) {
                        float wv = w[i], mv = m[i], vv = v[i];
                        adamw_elem(wv, g[i], mv, vv, a);
                        w[i] = wv; m[i] = mv; v[i] = vv;
                    }
                }
        }
        return;
    }
    const int e = blockIdx.y / 3, which = blockIdx.y % 3;
    const int rows = which == 2 ? p.H : p.C, cols = which == 2 ? p.C : p.H;
    const int ct = (cols + 127) / 128, rt = (rows + 63) / 64;
    if ((int)blockIdx.x >= ct * rt) return;
    const int c0 = blockIdx.x % ct * 128, r0 = blockIdx.x / ct * 64;
    float* w = p.w[which][e];
    const float* g = ADAM ? p.g[which][e] : nullptr;
    float* m = ADAM ? p.m[which][e] : nullptr;
    float* v = ADAM ? p.v[which][e] : nullptr;
    if (ADAM && blockIdx.x == 0) {
        float *bw = p.w[3 + which][e], *bm = p.m[3 + which][e], *bv = p.v[3 + which][e];
        const float* bg = p.g[3 + which][e];
        for (int i = tid; i < cols; i += 256) {
            float wv = bw[i], mv = bm[i], vv = bv[i];
            adamw_elem(wv, bg[i], mv, vv, a);
            bw[i] = wv; bm[i] = mv; bv[i] = vv;
        }
    }
    auto ld = [](const float* q) {
        if constexpr (VEC) return *reinterpret_cast<const float4*>(q);
        else return make_float4(q[0], q[1], q[2], q[3]);
    };
    auto st = [](float* q, const float (&x)[4]) {
        if constexpr (VEC) *reinterpret_cast<float4*>(q) = make_float4(x[0], x[1], x[2], x[3]);
        else { q[0] = x[0]; q[1] = x[1]; q[2] = x[2]; q[3] = x[3]; }
    };
    bf16* copyT = p.copyT[which];
    bf16* copy = p.copy[which];
    const int q4 = tid & 31, c = c0 + q4 * 4;          // this thread's four columns; rows 2*(tid/32), +1, +16 each step
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        float4 wv[4], gv[4], mv[4], vv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + (tid >> 5) * 2 + (half * 2 + (i >> 1)) * 16 + (i & 1);
            wv[i] = gv[i] = mv[i] = vv[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r < rows && c < cols) {
                const size_t o = (size_t)r * cols + c;
                wv[i] = ld(w + o);
                if (ADAM) { gv[i] = ld(g + o); mv[i] = ld(m + o); vv[i] = ld(v + o); }
            }
        }
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) {
            uint32_t pack[4];
            __nv_bfloat162 h[4];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = pr * 2 + k;
                const int r = r0 + (tid >> 5) * 2 + (half * 2 + pr) * 16 + k;
                float ww[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
                if (ADAM) {
                    const float gg[4] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w};
                    float mm[4] = {mv[i].x, mv[i].y, mv[i].z, mv[i].w}, v4[4] = {vv[i].x, vv[i].y, vv[i].z, vv[i].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) adamw_elem(ww[j], gg[j], mm[j], v4[j], a);
                    if (r < rows && c < cols) {
                        const size_t o = (size_t)r * cols + c;
                        st(w + o, ww); st(m + o, mm); st(v + o, v4);
                    }
                }
                if (copy && r < rows && c < cols) {
                    __nv_bfloat162 x0 = __floats2bfloat162_rn(ww[0], ww[1]), x1 = __floats2bfloat162_rn(ww[2], ww[3]);
                    *reinterpret_cast<uint2*>(copy + (size_t)e * rows * cols + (size_t)r * cols + c) =
                        make_uint2(*reinterpret_cast<uint32_t*>(&x0), *reinterpret_cast<uint32_t*>(&x1));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (k == 0) h[j].x = (r < rows && c < cols) ? __float2bfloat16(ww[j]) : __float2bfloat16(0.0f);
                    else h[j].y = (r < rows && c < cols) ? __float2bfloat16(ww[j]) : __float2bfloat16(0.0f);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) pack[j] = *reinterpret_cast<uint32_t*>(&h[j]);
            const int rp = (tid >> 5) + (half * 2 + pr) * 8;                // row pair of the tile
            *reinterpret_cast<uint4*>(S + rp * 128 + ((q4 ^ (rp >> 2)) << 2)) = make_uint4(pack[0], pack[1], pack[2], pack[3]);
        }
    }
    if (!copyT) return;
    __syncthreads();
    // the block of the transposed copy: 128 rows (source columns) x 64 (source rows), a 128-byte row per 8 lanes
    bf16* blk = copyT + (size_t)e * tile_major_elems(cols, rows) + tile_major_index(rows, c0, r0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int hrow = (tid >> 3) + 32 * i, c8 = tid & 7;
        uint32_t x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = S[(c8 * 4 + j) * 128 + (((hrow >> 2) ^ c8) << 2) + (hrow & 3)];
        *reinterpret_cast<uint4*>(blk + hrow * 64 + c8 * 8) = make_uint4(x[0], x[1], x[2], x[3]);
    }
}

template <bool ADAM> int launch_expert_weights(mgpt_moe_layer* L, const WeightsArgs& p, const AdamwScalars& a, bool vec, cudaStream_t st)
{
    const Dims& d = L->d;
    const int tCH = (d.C + 63) / 64 * ((d.H + 127) / 128), tHC = (d.H + 63) / 64 * ((d.C + 127) / 128);
    const dim3 grid(tCH > tHC ? tCH : tHC, 3 * d.E + (ADAM ? 1 : 0));
    if (vec) MGPT_CUDA(launch_pdl(expert_weights_kernel<ADAM, true>, grid, 256, 0, st, p, a));
    else MGPT_CUDA(launch_pdl(expert_weights_kernel<ADAM, false>, grid, 256, 0, st, p, a));
    MGPT_LAUNCHED("expert_weights_kernel");
    return 0;
}

WeightsArgs weights_args(const mgpt_moe_layer* L)
{
    WeightsArgs p = {};
    const ExpertPtrs& t = L->master;
    p.w[0] = (float* const*)t.Wg; p.w[1] = (float* const*)t.Wu; p.w[2] = (float* const*)t.Wd;
    p.w[3] = (float* const*)t.bg; p.w[4] = (float* const*)t.bu; p.w[5] = (float* const*)t.bd;
    p.g[0] = (const float* const*)t.gWg; p.g[1] = (const float* const*)t.gWu; p.g[2] = (const float* const*)t.gWd;
    p.g[3] = (const float* const*)t.gbg; p.g[4] = (const float* const*)t.gbu; p.g[5] = (const float* const*)t.gbd;
    p.C = L->d.C; p.H = L->d.H; p.E = L->d.E;
    p.copyT[0] = L->sWgT; p.copyT[1] = L->sWuT; p.copyT[2] = L->sWdT;
    p.copy[0] = L->sWg; p.copy[1] = L->sWu; p.copy[2] = L->sWd;
    return p;
}

// Router tensors alone (a layer whose experts live elsewhere).
__global__ void __launch_bounds__(256)
adamw_router_kernel(float* const* w_ptrs, const float* const* g_ptrs,
                    float* const* m_ptrs, float* const* v_ptrs, int len0, int len1,
                    float* rstat, const AdamwScalars a)
{
    pdl_wait();
    if (rstat && blockIdx.x == 0 && threadIdx.x < 2) rstat[threadIdx.x] = 0.0f;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, t = i < len0 ? 0 : 1, o = i - t * len0;
    if (i >= len0 + len1) return;
    float wv = w_ptrs[t][o], mv = m_ptrs[t][o], vv = v_ptrs[t][o];
    adamw_elem(wv, g_ptrs[t][o], mv, vv, a);
    w_ptrs[t][o] = wv; m_ptrs[t][o] = mv; v_ptrs[t][o] = vv;
}

}  // namespace

// Rebuilds the BF16 copies of the expert weights from the FP32 masters.
int launch_weight_copies(mgpt_moe_layer* L, cudaStream_t st)
{
    return launch_expert_weights<false>(L, weights_args(L), AdamwScalars{}, L->masters_aligned, st);
}

int launch_adamw(mgpt_moe_layer* L, float lr, float beta1, float beta2, float eps, float weight_decay, int t,
                 cudaStream_t st, float grad_clip, int skip_nonfinite)
{
    const Dims& d = L->d;
    AdamwScalars a;
    a.b1 = beta1; a.b2 = beta2; a.omb1 = 1.0f - beta1; a.omb2 = 1.0f - beta2; a.eps = eps; a.lr = lr;
    a.lrwd = lr * weight_decay;
    a.ms = 1.0f / (1.0f - std::pow(beta1, (float)t));
    a.vs = 1.0f / (1.0f - std::pow(beta2, (float)t));
    a.clip = grad_clip;
    a.skip_bad = skip_nonfinite;
    void** tab = (void**)L->d_opt;     // [m: Wg Wu Wd bg bu bd | v: same | router: w g m v for Wr, br][E]
    const int E = d.E, S = E < 2 ? 2 : E;          // table stride (the router rows hold two entries)
    auto T = [&](int i) { return tab + (size_t)i * S; };
    // router tables: rows 12..15 hold {w, g, m, v}, entry 0 = Wr, entry 1 = br
    if (L->experts_bound) {
        WeightsArgs p = weights_args(L);
        for (int i = 0; i < 6; ++i) {
            p.m[i] = (float* const*)T(i);
            p.v[i] = (float* const*)T(6 + i);
        }
        for (int i = 0; i < 4; ++i) p.router[i] = L->router_bound ? (float* const*)T(12 + i) : nullptr;
        p.rstat = L->d_rstat;
        MGPT_TRY((launch_expert_weights<true>(L, p, a, L->masters_aligned && L->opt_aligned, st)));
    } else if (L->router_bound) {
        MGPT_CUDA(launch_pdl(adamw_router_kernel, (d.C * E + E + 255) / 256, 256, 0, st, (float* const*)T(12),
                             (const float* const*)T(13), (float* const*)T(14), (float* const*)T(15), d.C * E, E, L->d_rstat, a));
        MGPT_LAUNCHED("adamw_router_kernel");
    }
    // the copies of the expert weights are current; the router's small BF16 copies are rebuilt from the new Wr
    L->shadows_fresh = false;
    if (d.mode == MGPT_MOE_BF16 && L->router_bound) MGPT_TRY(launch_router_copies(L, true, st));
    L->shadows_fresh = true;
    return 0;
}

}  // namespace mgpt
