// Grouped expert products on CUDA cores (FP32 accumulate).
//
// This is the FP32 validation mode of the layer (the reference's own dtype,
// parity bar 1e-5) and, with BF16 operands, the cross-check for the tcgen05
// path in gemm_tc.cu.  Same math as the reference's per-expert loop
// (layers/MoELayer.cpp:94-118, 159-181; layers/SwiGLU.cpp:23-50, 57-96;
// layers/LinearLayer.cpp:36-80) but grouped: one launch covers every expert,
// reading the row tiles and the tile->expert table built by the plan.
#include "tc_common.cuh"

namespace mgpt {

namespace {

// One CTA: a 64 x 64 output tile, 128 threads per K group, 8 rows x 4 columns per thread; operands go through two
// shared-memory buffers of 16 k each, the next one loaded into registers with 16-byte accesses while this one is worked
// on.  What bounds these products at the reference's default size (2048 routed rows, C = 128, H = 512) is not the
// 0.13-0.27 GFMA but how many warps are in flight and how long one CTA's k loop is: the products over H with C = 128
// columns are 72 tiles for 148 SMs.  KS groups of 128 threads therefore split a tile's k loop and are added up, in
// order, through shared memory (KS by split_k below).  One 64 x 64 tile per 256 threads with scalar loads and nothing in
// flight between two barriers took 49 / 74 / 25 / 73 us for gate-up / down / dHh / dXg and 27 us for each weight
// gradient there.
constexpr int TM = 64, TN = 64, TK = 16;
constexpr int GT = 128;                       // threads per K group
constexpr int SROW = TM + 4;                  // padded row of a staged operand (floats)
constexpr int OPER = TK * SROW;               // one staged operand

// four consecutive elements (VEC: the address is aligned to four elements)
template <bool VEC> __device__ __forceinline__ float4 load4(const float* p)
{
    if constexpr (VEC) return *reinterpret_cast<const float4*>(p);
    else return make_float4(p[0], p[1], p[2], p[3]);
}
template <bool VEC> __device__ __forceinline__ float4 load4(const bf16* p)
{
    if constexpr (!VEC) return make_float4(__bfloat162float(p[0]), __bfloat162float(p[1]), __bfloat162float(p[2]), __bfloat162float(p[3]));
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ float round_to(float v, float) { return v; }
__device__ __forceinline__ float round_to(float v, bf16) { return __bfloat162float(__float2bfloat16(v)); }
template <bool VEC> __device__ __forceinline__ void store4(float* p, float4 v)
{
    if constexpr (VEC) *reinterpret_cast<float4*>(p) = v;
    else { p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w; }
}
template <bool VEC> __device__ __forceinline__ void store4(bf16* p, float4 v)
{
    if constexpr (!VEC) {
        p[0] = __float2bfloat16(v.x); p[1] = __float2bfloat16(v.y); p[2] = __float2bfloat16(v.z); p[3] = __float2bfloat16(v.w);
        return;
    }
    __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&h0), *reinterpret_cast<uint32_t*>(&h1));
}
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(GT) : "memory"); }

// A staged operand is [TK][SROW]: element (k, m) at k*SROW + m.  Thread t of a group fetches two pieces of four
// elements: along k for a matrix whose k is contiguous (KMAJOR), along m otherwise; out of range reads as zero.
template <typename T, bool KMAJOR, bool VEC>
__device__ __forceinline__ void fetch(const T* P, long ld, int m0, int M, int k0, int K, int t, float4 (&r)[2])
{
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int m = m0 + (KMAJOR ? (t >> 2) + 32 * i : (t & 15) * 4);
        const int k = k0 + (KMAJOR ? (t & 3) * 4 : (t >> 4) + 8 * i);
        r[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (m < M && k < K) r[i] = load4<VEC>(KMAJOR ? P + (long)m * ld + k : P + (long)k * ld + m);
    }
}
template <bool KMAJOR>
__device__ __forceinline__ void put(float* S, int t, const float4 (&r)[2])
{
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (KMAJOR) {
            float* d = S + (t & 3) * 4 * SROW + (t >> 2) + 32 * i;
            d[0] = r[i].x; d[SROW] = r[i].y; d[2 * SROW] = r[i].z; d[3 * SROW] = r[i].w;
        } else {
            *reinterpret_cast<float4*>(S + ((t >> 4) + 8 * i) * SROW + (t & 15) * 4) = r[i];
        }
    }
}
// Two FP32 multiply-adds in one instruction: they take the FMA pipe as long as two would and leave every other issue slot to
// the loads.  Worth it where an SM has 16 warps to issue from (KS > 1: dXg 38 -> 33 us, down 20 -> 19); with half of them
// the pairs' register moves cost more (gate-up 24 -> 26).
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b)
{
    asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %4};\n mov.b64 rd, {%0, %1};\n"
        " fma.rn.f32x2 rd, ra, rb, rd;\n mov.b64 {%0, %1}, rd;\n}" : "+f"(d0), "+f"(d1) : "f"(a0), "f"(a1), "f"(b));
}
// acc[8][4] += rows ty*8.. x columns tx*4.. over the TK staged k
template <bool PACK>
__device__ __forceinline__ void mac(const float* As, const float* Bs, int ty, int tx, float (&acc)[8][4])
{
#pragma unroll
    for (int k = 0; k < TK; ++k) {
        const float4 a0 = *reinterpret_cast<const float4*>(As + k * SROW + ty * 8);
        const float4 a1 = *reinterpret_cast<const float4*>(As + k * SROW + ty * 8 + 4);
        const float4 b = *reinterpret_cast<const float4*>(Bs + k * SROW + tx * 4);
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; i += 2)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (PACK) {
                    fma2(acc[i][j], acc[i + 1][j], av[i], av[i + 1], bv[j]);
                } else {
                    acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
                    acc[i + 1][j] = fmaf(av[i + 1], bv[j], acc[i + 1][j]);
                }
            }
    }
}
// The groups' sums, added to group 0's in group order.  S: shared memory of 64*64 floats per group beyond the first.
template <int KS>
__device__ __forceinline__ void fold(float* S, int group, int t, float (&acc)[8][4])
{
    if constexpr (KS > 1) {
        __syncthreads();                      // every group is done with its operand buffers
        float4* mine = reinterpret_cast<float4*>(S) + (group - 1) * 1024;
        if (group > 0)
#pragma unroll
            for (int i = 0; i < 8; ++i) mine[i * GT + t] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        __syncthreads();
        if (group == 0)
            for (int g = 1; g < KS; ++g)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 v = reinterpret_cast<const float4*>(S)[(g - 1) * 1024 + i * GT + t];
                    acc[i][0] += v.x; acc[i][1] += v.y; acc[i][2] += v.z; acc[i][3] += v.w;
                }
    }
}

// The sums of the CTAs of a cluster that share a tile's k loop, added to the first CTA's in rank order through distributed shared
// memory.  S: shared memory of 64*64 floats; `adds`: this thread holds sums (group 0).
__device__ __forceinline__ void fold_cluster(float* S, int ctas, int rank, bool adds, int t, float (&acc)[8][4])
{
    float4* mine = reinterpret_cast<float4*>(S);
    __syncthreads();                          // what S held has been read
    if (rank > 0 && adds)
#pragma unroll
        for (int i = 0; i < 8; ++i) mine[i * GT + t] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    tcx::cluster_sync();
    if (rank == 0 && adds)
        for (int r = 1; r < ctas; ++r) {
            const uint32_t peer = tcx::mapa((uint32_t)__cvta_generic_to_shared(S), r);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float4 v;
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer + (i * GT + t) * 16) : "memory");
                acc[i][0] += v.x; acc[i][1] += v.y; acc[i][2] += v.z; acc[i][3] += v.w;
            }
        }
    tcx::cluster_sync();                      // nobody leaves, or writes S again, while it is being read
}

enum { EPI_GATEUP = 0, EPI_DOWN = 1, EPI_DHH = 2, EPI_DXG = 3 };

struct RowsArgs {
    const void* A;  const void* A2;            // activations [rows, K]
    const void* const* B; const void* const* B2;   // per-expert weights
    const float* const* bias; const float* const* bias2;
    void* D; void* D2; void* D3;               // outputs [rows, Nout]
    const void* G; const void* U;              // saved pre-activations (EPI_DHH)
    const int32_t* tile_expert; const int32_t* n_tiles;
    // real rows of an expert and its first row: 64-row pieces of a tile that hold padding only are left out (nothing
    // reads them: the weight gradients below stop at the last real row).  Null where rows come in segments.
    const int32_t* counts; const int32_t* padded_offsets;
    int K, Nout;
};

template <int EPI, int KS> constexpr size_t rows_smem()
{
    constexpr size_t ops = (size_t)KS * 2 * (EPI == EPI_GATEUP ? 3 : 2) * OPER * sizeof(float);
    constexpr size_t red = (size_t)(KS - 1) * (EPI == EPI_GATEUP ? 2 : 1) * TM * TN * sizeof(float);
    return ops > red ? ops : red;
}

// VEC: weights and their gradients, AVEC: rows, start on boundaries of four elements.
// CL: a cluster of CTAs per tile.
template <typename TAct, typename TW, int EPI, int KS, bool VEC, bool AVEC, bool CL>
__global__ void __launch_bounds__(GT * KS) simt_rows_kernel(RowsArgs a)
{
    extern __shared__ __align__(16) float sm[];
    pdl_wait();
    constexpr bool BK_MAJOR = EPI == EPI_DHH || EPI == EPI_DXG;      // B(k, n) at n*K + k
    constexpr int NOP = EPI == EPI_GATEUP ? 3 : 2;
    const int m0 = (CL ? blockIdx.x / tcx::cluster_size() : blockIdx.x) * TM, n0 = blockIdx.y * TN;
    const int rows = *a.n_tiles * ROW_TILE;
    if (m0 >= rows) return;
    const int e = a.tile_expert[m0 / ROW_TILE];
    if (a.counts && m0 - a.padded_offsets[e] >= a.counts[e]) return;
    const int group = threadIdx.x / GT, t = threadIdx.x % GT;
    const int tx = t & 15, ty = t >> 4;
    const int K = a.K, N = a.Nout;
    float* S = sm + (size_t)group * 2 * NOP * OPER;
    float acc[8][4] = {}, acc2[8][4] = {};
    // this group's steps of TK; EPI_DXG runs through dG*Wg^T and then dU*Wu^T
    const int per = (K + TK - 1) / TK, steps = EPI == EPI_DXG ? 2 * per : per;
    int s0 = (int)((long)steps * group / KS), s1 = (int)((long)steps * (group + 1) / KS), rank = 0;
    if constexpr (CL) {
        rank = (int)tcx::cluster_ctarank();
        const int part = rank * KS + group, parts = KS * (int)tcx::cluster_size();
        s0 = (int)((long)steps * part / parts);
        s1 = (int)((long)steps * (part + 1) / parts);
    }
    const TW *B1 = (const TW*)a.B[e], *B2 = NOP == 3 || EPI == EPI_DXG ? (const TW*)a.B2[e] : nullptr;
    float4 ra[2], rb[2], rc[2];
    auto gload = [&](int s) {
        const bool second = EPI == EPI_DXG && s >= per;
        const int k0 = (second ? s - per : s) * TK;
        fetch<TAct, true, AVEC>((const TAct*)(second ? a.A2 : a.A), K, m0, rows, k0, K, t, ra);
        fetch<TW, BK_MAJOR, VEC>(second ? B2 : B1, BK_MAJOR ? K : N, n0, N, k0, K, t, rb);
        if (NOP == 3) fetch<TW, BK_MAJOR, VEC>(B2, N, n0, N, k0, K, t, rc);
    };
    auto sstore = [&](int buf) {
        float* d = S + buf * NOP * OPER;
        put<true>(d, t, ra);
        put<BK_MAJOR>(d + OPER, t, rb);
        if (NOP == 3) put<BK_MAJOR>(d + 2 * OPER, t, rc);
    };
    if (s0 < s1) {
        gload(s0);
        sstore(0);
    }
    group_sync(group);
    for (int s = s0; s < s1; ++s) {
        const int buf = (s - s0) & 1;
        if (s + 1 < s1) gload(s + 1);
        const float* c = S + buf * NOP * OPER;
        mac<(KS > 1)>(c, c + OPER, ty, tx, acc);
        if (NOP == 3) mac<(KS > 1)>(c, c + 2 * OPER, ty, tx, acc2);
        if (s + 1 < s1) sstore(buf ^ 1);
        group_sync(group);
    }
    fold<KS>(sm, group, t, acc);
    if (NOP == 3) fold<KS>(sm + (KS - 1) * TM * TN, group, t, acc2);
    if constexpr (CL) {
        fold_cluster(sm, tcx::cluster_size(), rank, group == 0, t, acc);
        if (NOP == 3) fold_cluster(sm, tcx::cluster_size(), rank, group == 0, t, acc2);
        if (rank > 0) return;
    }
    const int n = n0 + tx * 4;
    if (group > 0 || n >= N) return;
    float b1[4] = {}, b2[4] = {};
    if (EPI == EPI_GATEUP || EPI == EPI_DOWN)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            b1[j] = a.bias[e][n + j];
            if (EPI == EPI_GATEUP) b2[j] = a.bias2[e][n + j];
        }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const size_t o = (size_t)(m0 + ty * 8 + i) * N + n;
        float d[4], d2[4], d3[4];
        float4 g4, u4;
        if (EPI == EPI_DHH) {
            g4 = load4<true>((const TAct*)a.G + o);
            u4 = load4<true>((const TAct*)a.U + o);
        }
        const float gs[4] = {g4.x, g4.y, g4.z, g4.w}, us[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (EPI == EPI_GATEUP) {
                // layers/SwiGLU.cpp:32-40, utils/Tensor.cpp:1997-2002; downstream stages read the stored (rounded)
                // values, so round first
                d[j] = round_to(acc[i][j] + b1[j], TAct());
                d2[j] = round_to(acc2[i][j] + b2[j], TAct());
                d3[j] = __fdiv_rn(d[j], 1.0f + expf(-d[j])) * d2[j];
            } else if (EPI == EPI_DOWN) {
                d[j] = acc[i][j] + b1[j];
            } else if (EPI == EPI_DHH) {
                // utils/Tensor.cpp:2020-2027
                const float dd = acc[i][j], g = gs[j], u = us[j];
                const float sig = 1.0f / (1.0f + expf(-g));
                d[j] = (dd * u) * (sig * (1.0f + g * (1.0f - sig)));      // dG
                d2[j] = dd * (g * sig);                                   // dU
            } else {
                d[j] = acc[i][j];
            }
        }
        store4<AVEC>((TAct*)a.D + o, make_float4(d[0], d[1], d[2], d[3]));
        if (EPI == EPI_GATEUP || EPI == EPI_DHH) store4<true>((TAct*)a.D2 + o, make_float4(d2[0], d2[1], d2[2], d2[3]));
        if (EPI == EPI_GATEUP) store4<true>((TAct*)a.D3 + o, make_float4(d3[0], d3[1], d3[2], d3[3]));
    }
}

// grad[e][m,n] += sum over the expert's rows p of A[p,m] * B[p,n], and the bias gradient that is the column sum of B
// (layers/LinearLayer.cpp:56-66: dW = X^T * dOut, db = sum of dOut, accumulated like Tensor::add_grad).  One launch for
// the three weights of every expert: gWg = Xg^T dG, gWu = Xg^T dU, gWd = Hh^T dYg.
struct WgradArgs {
    const void* Xg; const void* Hh; const void* dG; const void* dU; const void* dYg;
    float* const* grad[3];       // per expert: gWg, gWu [C,H], gWd [H,C]
    float* const* gb[3];         // per expert: gbg, gbu [H], gbd [C]
    const int32_t* padded_offsets;
    const int32_t* counts;       // real rows per expert; null: every row of the padded segment is summed (zeros add nothing)
    int C, H;
    const int32_t* seg;          // [E][n_seg][2] {first row, rows} when an expert's rows come in several segments
    int n_seg;
};

template <int KS> constexpr size_t wgrad_smem()
{
    constexpr size_t ops = (size_t)KS * 4 * OPER * sizeof(float);
    constexpr size_t red = ((size_t)(KS - 1) * TM * TN + KS * TN) * sizeof(float);
    return ops > red ? ops : red;
}

template <typename TAct, int KS, bool VEC, bool AVEC>
__global__ void __launch_bounds__(GT * KS) simt_wgrad_kernel(WgradArgs a)
{
    extern __shared__ __align__(16) float sm[];
    pdl_wait();
    const int e = blockIdx.y / 3, which = blockIdx.y % 3;
    const int M = which == 2 ? a.H : a.C, N = which == 2 ? a.C : a.H;
    const int mt = (M + TM - 1) / TM, m0 = blockIdx.x % mt * TM, n0 = blockIdx.x / mt * TN;
    const TAct* A = (const TAct*)(which == 2 ? a.Hh : a.Xg);
    const TAct* B = (const TAct*)(which == 0 ? a.dG : which == 1 ? a.dU : a.dYg);
    const int group = threadIdx.x / GT, t = threadIdx.x % GT;
    const int tx = t & 15, ty = t >> 4;
    const bool bias = m0 == 0;                 // this CTA also sums its columns of B
    float* S = sm + (size_t)group * 4 * OPER;
    float acc[8][4] = {}, bs[4] = {};
    const int nseg = a.n_seg > 0 ? a.n_seg : 1;
    int total = 0;
    for (int sgi = 0; sgi < nseg; ++sgi) {
        const int r0 = a.n_seg > 0 ? a.seg[(e * a.n_seg + sgi) * 2] : a.padded_offsets[e];
        const int len = a.n_seg > 0 ? a.seg[(e * a.n_seg + sgi) * 2 + 1] : a.counts ? a.counts[e] : a.padded_offsets[e + 1] - r0;
        if (len <= 0) continue;               // uniform over the CTA
        total += len;
        const int steps = (len + TK - 1) / TK;
        const int s0 = (int)((long)steps * group / KS), s1 = (int)((long)steps * (group + 1) / KS);
        const TAct *As = A + (size_t)r0 * M, *Bs = B + (size_t)r0 * N;
        float4 ra[2], rb[2];
        auto gload = [&](int s) {
            fetch<TAct, false, AVEC>(As, M, m0, M, s * TK, len, t, ra);
            fetch<TAct, false, AVEC>(Bs, N, n0, N, s * TK, len, t, rb);
        };
        auto sstore = [&](int buf) {
            put<false>(S + buf * 2 * OPER, t, ra);
            put<false>(S + buf * 2 * OPER + OPER, t, rb);
        };
        if (s0 < s1) {
            gload(s0);
            sstore(0);
        }
        group_sync(group);
        for (int s = s0; s < s1; ++s) {
            const int buf = (s - s0) & 1;
            if (s + 1 < s1) gload(s + 1);
            const float* c = S + buf * 2 * OPER;
            mac<(KS > 1)>(c, c + OPER, ty, tx, acc);
            if (bias && ty == 0)
#pragma unroll
                for (int k = 0; k < TK; ++k) {
                    const float4 b = *reinterpret_cast<const float4*>(c + OPER + k * SROW + tx * 4);
                    bs[0] += b.x; bs[1] += b.y; bs[2] += b.z; bs[3] += b.w;
                }
            if (s + 1 < s1) sstore(buf ^ 1);
            group_sync(group);
        }
    }
    if (total == 0) return;
    fold<KS>(sm, group, t, acc);
    const int n = n0 + tx * 4;
    if (bias) {
        float* sb = sm + (KS - 1) * TM * TN;
        if (KS == 1) __syncthreads();         // (more groups: fold has waited for the last reads of the operand buffers)
        if (ty == 0) *reinterpret_cast<float4*>(sb + group * TN + tx * 4) = make_float4(bs[0], bs[1], bs[2], bs[3]);
        __syncthreads();
        if (threadIdx.x < TN && n0 + (int)threadIdx.x < N) {
            float v = 0.0f;
            for (int g = 0; g < KS; ++g) v += sb[g * TN + threadIdx.x];
            (which == 0 ? a.gb[0] : which == 1 ? a.gb[1] : a.gb[2])[e][n0 + threadIdx.x] += v;
        }
    }
    if (group > 0 || n >= N) return;
    float* g = (which == 0 ? a.grad[0] : which == 1 ? a.grad[1] : a.grad[2])[e];      // (a dynamic index would copy the arguments to local memory)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty * 8 + i;
        if (m >= M) break;
        float* p = g + (size_t)m * N + n;
        if (VEC) {
            float4 v = *reinterpret_cast<const float4*>(p);
            v.x += acc[i][0]; v.y += acc[i][1]; v.z += acc[i][2]; v.w += acc[i][3];
            *reinterpret_cast<float4*>(p) = v;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] += acc[i][j];
        }
    }
}

// K groups per tile: enough that ~8 warps (four per group) fall to every SM, at most four, and no group with less than
// two steps.
int split_k(int tiles, int k)
{
    int ks = tiles * 4 < 400 ? 4 : tiles * 4 < 800 ? 2 : 1;
    while (ks > 1 && k < ks * 2 * TK) ks /= 2;
    return ks;
}

// CTAs per tile where four groups each leave SMs without one: a cluster of two, four or eight, no group with less than two steps.
// Stage times without -> with, us: 1024 tokens, C=128, H=512, E=8, top-2 (two CTAs) down 23 -> 19, dXg 37 -> 27, the step 149 ->
// 135; 64 tokens, C=256, H=1024 (four) 35 -> 20 and 66 -> 29, the step 172 -> 120; 256 tokens, C=256, H=1024, E=16, top-1 234
// -> 203.  A few clusters more than the SMs hold are a second round, which takes the gain and more (the step of 564 tokens,
// C=192, H=152, E=13, top-2, 108 without, 113 with 25 row tiles instead of the 24 that were expected), so `tiles` is a number that
// the routing seldom exceeds.
int split_ctas(double tiles, int k)
{
    int ctas = 1;
    while (ctas < 8 && tiles * ctas * 2 <= 148 && k >= ctas * 2 * 4 * 2 * TK) ctas *= 2;
    return ctas;
}

// The row buffers of an expert side are the caller's, at any address; those in the workspace are aligned.
template <typename TAct> bool rows_aligned(const mgpt_moe_layer* L)
{
    const uintptr_t any = (uintptr_t)L->ext_Xg | (uintptr_t)L->ext_Yg | (uintptr_t)L->ext_dYg | (uintptr_t)L->ext_dXg;
    return (any & (4 * sizeof(TAct) - 1)) == 0;
}

template <typename TAct, typename TW, int EPI, int KS, bool CL>
int launch_rows_ks(const mgpt_moe_layer* L, const RowsArgs& a, dim3 grid, int ctas, cudaStream_t st)
{
    constexpr size_t smem = rows_smem<EPI, KS>();
    auto* kernel = !rows_aligned<TAct>(L) ? simt_rows_kernel<TAct, TW, EPI, KS, false, false, CL>
                   : L->masters_aligned   ? simt_rows_kernel<TAct, TW, EPI, KS, true, true, CL>
                                          : simt_rows_kernel<TAct, TW, EPI, KS, false, true, CL>;
    if (smem > 48 * 1024) MGPT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (CL) MGPT_CUDA(launch_pdl_cluster(kernel, grid, ctas, GT * KS, smem, st, a));
    else MGPT_CUDA(launch_pdl(kernel, grid, GT * KS, smem, st, a));
    return 0;
}
template <typename TAct, typename TW, int EPI>
int launch_rows(const mgpt_moe_layer* L, const Workspace& w, const RowsArgs& a, cudaStream_t st, const char* what)
{
    const int cols = (a.Nout + TN - 1) / TN;
    // tiles with real rows: about R/64 and half a tile per expert
    const int tiles = (w.R / TM + (L->d.E + 1) / 2) * cols, k = EPI == EPI_DXG ? 2 * a.K : a.K;
    // (each expert's last tile is filled by chance: that half has a standard deviation of sqrt(E / 12))
    const double most = (w.R / (double)TM + L->d.E / 2.0 + sqrt(L->d.E / 12.0)) * cols;
    const int ks = split_k(tiles, k), ctas = ks == 4 ? split_ctas(most, k) : 1;
    const dim3 grid(w.row_cap / TM * ctas, cols);
    if (ctas > 1) MGPT_TRY((launch_rows_ks<TAct, TW, EPI, 4, true>(L, a, grid, ctas, st)));
    else if (ks == 4) MGPT_TRY((launch_rows_ks<TAct, TW, EPI, 4, false>(L, a, grid, ctas, st)));
    else if (ks == 2) MGPT_TRY((launch_rows_ks<TAct, TW, EPI, 2, false>(L, a, grid, ctas, st)));
    else MGPT_TRY((launch_rows_ks<TAct, TW, EPI, 1, false>(L, a, grid, ctas, st)));
    MGPT_LAUNCHED(what);
    return 0;
}
template <typename TAct, int KS>
int launch_wgrad_ks(const mgpt_moe_layer* L, const WgradArgs& a, dim3 grid, cudaStream_t st)
{
    constexpr size_t smem = wgrad_smem<KS>();
    auto* kernel = !rows_aligned<TAct>(L) ? simt_wgrad_kernel<TAct, KS, false, false>
                   : L->masters_aligned   ? simt_wgrad_kernel<TAct, KS, true, true>
                                          : simt_wgrad_kernel<TAct, KS, false, true>;
    if (smem > 48 * 1024) MGPT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    MGPT_CUDA(launch_pdl(kernel, grid, GT * KS, smem, st, a));
    return 0;
}

// Real rows per expert and the start of its segment, for the kernels that leave padding out: in FP32 mode, where an
// expert's rows are one padded segment.  (With BF16 data these products are the cross-check of the tensor-core ones and
// compute the padding rows as those do.)
void rows_of_experts(const mgpt_moe_layer* L, const Workspace& w, char* ws, const int32_t*& counts, const int32_t*& padded_offsets)
{
    if (w.act_bytes != 4 || L->n_seg > 0) return;
    counts = (const int32_t*)(ws + w.counts);
    padded_offsets = (const int32_t*)(ws + w.padded_offsets);
}

template <typename TAct, typename TW>
int experts_forward_t(mgpt_moe_layer* L, const ExpertPtrs& P, const Workspace& w, char* ws, cudaStream_t st)
{
    const Dims& d = L->d;
    RowsArgs a = {};
    a.tile_expert = (const int32_t*)(ws + w.tile_expert);
    a.n_tiles = (const int32_t*)(ws + w.n_tiles);
    rows_of_experts(L, w, ws, a.counts, a.padded_offsets);
    // gate/up + SwiGLU
    a.A = buf_Xg(L, w, ws); a.B = P.Wg; a.B2 = P.Wu; a.bias = P.bg; a.bias2 = P.bu;
    a.D = ws + w.G; a.D2 = ws + w.U; a.D3 = ws + w.Hh; a.K = d.C; a.Nout = d.H;
    L->stage_begin(ST_GATEUP, st);
    MGPT_TRY((launch_rows<TAct, TW, EPI_GATEUP>(L, w, a, st, "simt_rows_kernel<gateup>")));
    L->stage_end(ST_GATEUP, st);
    // down
    a.A = ws + w.Hh; a.B = P.Wd; a.bias = P.bd; a.D = buf_Yg(L, w, ws); a.K = d.H; a.Nout = d.C;
    L->stage_begin(ST_DOWN, st);
    MGPT_TRY((launch_rows<TAct, TW, EPI_DOWN>(L, w, a, st, "simt_rows_kernel<down>")));
    L->stage_end(ST_DOWN, st);
    return 0;
}

template <typename TAct, typename TW>
int experts_backward_t(mgpt_moe_layer* L, const ExpertPtrs& P, const Workspace& w, char* ws, cudaStream_t st)
{
    const Dims& d = L->d;
    RowsArgs a = {};
    a.tile_expert = (const int32_t*)(ws + w.tile_expert);
    a.n_tiles = (const int32_t*)(ws + w.n_tiles);
    rows_of_experts(L, w, ws, a.counts, a.padded_offsets);
    // dHh = dYg * Wd^T, fused SwiGLU backward -> dG, dU
    a.A = buf_dYg(L, w, ws); a.B = P.Wd; a.G = ws + w.G; a.U = ws + w.U; a.D = ws + w.dG; a.D2 = ws + w.dU;
    a.K = d.C; a.Nout = d.H;
    L->stage_begin(ST_DHH, st);
    MGPT_TRY((launch_rows<TAct, TW, EPI_DHH>(L, w, a, st, "simt_rows_kernel<dhh>")));
    L->stage_end(ST_DHH, st);
    // dXg = dG * Wg^T + dU * Wu^T
    a.A = ws + w.dG; a.A2 = ws + w.dU; a.B = P.Wg; a.B2 = P.Wu; a.D = buf_dXg(L, w, ws); a.K = d.H; a.Nout = d.C;
    L->stage_begin(ST_DXG, st);
    MGPT_TRY((launch_rows<TAct, TW, EPI_DXG>(L, w, a, st, "simt_rows_kernel<dxg>")));
    L->stage_end(ST_DXG, st);
    if (!L->has_grad) return 0;
    L->stage_begin(ST_WGRAD, st);
    WgradArgs g = {};
    g.Xg = buf_Xg(L, w, ws); g.Hh = ws + w.Hh; g.dG = ws + w.dG; g.dU = ws + w.dU; g.dYg = buf_dYg(L, w, ws);
    g.grad[0] = L->master.gWg; g.grad[1] = L->master.gWu; g.grad[2] = L->master.gWd;
    g.gb[0] = L->master.gbg; g.gb[1] = L->master.gbu; g.gb[2] = L->master.gbd;
    g.padded_offsets = (const int32_t*)(ws + w.padded_offsets);
    const int32_t* ignored = nullptr;
    rows_of_experts(L, w, ws, g.counts, ignored);
    g.C = d.C; g.H = d.H;
    g.seg = (const int32_t*)(ws + w.seg); g.n_seg = L->n_seg;
    const int per = ((d.C + TM - 1) / TM) * ((d.H + TM - 1) / TM);
    const dim3 grid(per, 3 * d.E);
    const int ks = split_k(per * 3 * d.E, w.R / d.E);
    if (ks == 4) MGPT_TRY((launch_wgrad_ks<TAct, 4>(L, g, grid, st)));
    else if (ks == 2) MGPT_TRY((launch_wgrad_ks<TAct, 2>(L, g, grid, st)));
    else MGPT_TRY((launch_wgrad_ks<TAct, 1>(L, g, grid, st)));
    MGPT_LAUNCHED("simt_wgrad_kernel");
    L->stage_end(ST_WGRAD, st);
    return 0;
}

}  // namespace

int simt_experts_forward(mgpt_moe_layer* L, const Workspace& w, char* ws, cudaStream_t st)
{
    if (w.act_bytes == 4) return experts_forward_t<float, float>(L, L->master, w, ws, st);
    return experts_forward_t<bf16, bf16>(L, L->shadow, w, ws, st);
}

int simt_experts_backward(mgpt_moe_layer* L, const Workspace& w, char* ws, cudaStream_t st)
{
    if (w.act_bytes == 4) return experts_backward_t<float, float>(L, L->master, w, ws, st);
    return experts_backward_t<bf16, bf16>(L, L->shadow, w, ws, st);
}

}  // namespace mgpt
