// Expert forward for few rows per expert (generation: pipeline/Generator.cpp:10-31 runs the layer forward only).
//
// With a handful of rows per expert the products cost nothing beside reading each touched expert's weights once from
// HBM, so these kernels are built around the weight stream and nothing else: every warp reads weights with 16-byte loads
// straight into mma.sync A fragments (no shared memory, no barrier between warps), four 64-wide k-blocks = 8 KiB in
// flight per warp, 16 warps per SM = 128 KiB per SM where ~55 KiB cover HBM's latency at full rate.  The rows are the
// N side, eight per MMA; their B fragments come through L1 straight from x (no dispatch pass) or from Hh.
//
//   gate/up   task = 8 hidden units of one row group: the 16 MMA rows are 8 gate rows and the 8 up rows of the same
//             units, so a thread ends up with gate and up of the same (unit, row) and applies SwiGLU in registers
//   down      task = 16 output columns of one row group
//
// A k-block's order of k within the fragments is chosen so that one 16-byte load feeds two MMAs (A and B agree on it, so
// the sum is the same set of products).  A row group is up to 16 rows of one expert (the plan lists them); more rows
// read the weights again, mostly from L2.  KS = 4 warps share a task's k-blocks and add up, in order, through shared
// memory; where a product has fewer than eight k-blocks one warp does it alone.  The widths alone decide that: a row's bits
// depend neither on the other rows of the call, nor on how many there are, nor on the number of SMs.  (One warp per task
// from two tasks per warp on, which adds up in another order, was as fast at 20 and 32 tokens, C=1024, H=2816, E=32, 124
// and 134 us for the call, slower at 16 with C=2048, H=1408, E=64, 155 against 142, and ahead only at 64, 138 against 144,
// which tiles do in 141.  One warp that keeps the four parts' sums apart: 130, 138, 155 and 142.)
//
// tcgen05 is no help here: its M side is 128 rows whatever the number of tokens, and with the weights on the M side
// instead an MMA of N = 16 still took ~120 cycles for 4 KiB of weights (1000 cycles per 32 KiB stage, 135 us for the
// products of 64 tokens at C=1024, H=2816, E=32 against 102 us with 128-row token tiles).
#include <type_traits>

#include "common.cuh"

namespace mgpt {

namespace {

constexpr int DW = 16;                 // warps per CTA, one CTA per SM
constexpr int DEPTH = 4;               // k-blocks in flight per warp

struct DecP {
    const void* x;                     // tokens (gathered), or the permuted rows where they have been kept
    const bf16 *WgT, *WuT, *WdT;       // tile-major copies
    const int4* groups;                // {expert, first padded row, rows, 0}
    const int32_t* n_groups;
    const int32_t* row_src;            // padded row -> flat index (null: x holds permuted rows)
    const float* const* b0;            // bias tables
    const float* const* b1;
    const bf16* A;                     // down: Hh
    bf16 *out, *G, *U;
    int C, H, k, hb, cb, kb1, kb2;
    int release;                       // phase 1: let phase 2's blocks in early
};

__device__ __forceinline__ uint4 ld_weights(const bf16* p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_row(const bf16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint4 ld_row(const float* p)
{
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    __nv_bfloat162 h0 = __floats2bfloat162_rn(a.x, a.y), h1 = __floats2bfloat162_rn(a.z, a.w);
    __nv_bfloat162 h2 = __floats2bfloat162_rn(b.x, b.y), h3 = __floats2bfloat162_rn(b.z, b.w);
    return make_uint4(*reinterpret_cast<uint32_t*>(&h0), *reinterpret_cast<uint32_t*>(&h1), *reinterpret_cast<uint32_t*>(&h2),
                      *reinterpret_cast<uint32_t*>(&h3));
}

// The weights of k-block kb for one lane (rows a are MMA rows 0..7, rows b 8..15; k-blocks are 8192 elements apart):
// 16-byte pieces (row a, k 0..31), (a, 32..63), (b, 0..31), (b, 32..63).
struct Frag {
    uint4 v[4];
};
__device__ __forceinline__ void ld_frag(Frag& f, const bf16* ra, const bf16* rb, int kb)
{
    const size_t o = (size_t)kb * 8192;
    f.v[0] = ld_weights(ra + o);
    f.v[1] = ld_weights(ra + o + 32);
    f.v[2] = ld_weights(rb + o);
    f.v[3] = ld_weights(rb + o + 32);
}

// acc[nn] += the task's weights x rows nn*8.. over the k-blocks [k0, k1).  `w` holds the first DEPTH of them, already
// requested.
template <int NN, typename TRow>
__device__ __forceinline__ void run_task(Frag (&w)[DEPTH], const bf16* ra, const bf16* rb, const TRow* const (&src)[NN], int k0, int k1,
                                         int K, int t4, float (&acc)[NN][4])
{
    for (int kb = k0; kb < k1; kb += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            if (kb + u < k1) {
                uint4 b[NN][2];
#pragma unroll
                for (int n = 0; n < NN; ++n)
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int k = (kb + u) * 64 + s * 32 + t4 * 8;
                        b[n][s] = k < K ? ld_row(src[n] + k) : make_uint4(0, 0, 0, 0);
                    }
                const Frag f = w[u];
                if (kb + u + DEPTH < k1) ld_frag(w[u], ra, rb, kb + u + DEPTH);
#pragma unroll
                for (int s = 0; s < 2; ++s)
#pragma unroll
                    for (int n = 0; n < NN; ++n) {
                        mma16816(acc[n], f.v[s].x, f.v[2 + s].x, f.v[s].y, f.v[2 + s].y, b[n][s].x, b[n][s].y);
                        mma16816(acc[n], f.v[s].z, f.v[2 + s].z, f.v[s].w, f.v[2 + s].w, b[n][s].z, b[n][s].w);
                    }
            }
        }
    }
}

// PHASE 1: gate/up, 2: down.  F32: the rows are FP32 tokens.
template <int PHASE, int KS, bool F32>
__global__ void __launch_bounds__(32 * DW, 1) decode_kernel(const DecP p)
{
    typedef typename std::conditional<F32, float, bf16>::type TRow;
    constexpr int NG = DW / KS;                            // task groups per CTA
    __shared__ float red[KS > 1 ? NG : 1][KS > 1 ? KS - 1 : 1][KS > 1 ? 8 : 1][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t4 = lane & 3, group = warp / KS, ks = warp % KS;
    const int K = PHASE == 1 ? p.C : p.H, kbs = PHASE == 1 ? p.kb1 : p.kb2, width = PHASE == 1 ? p.H : p.C;
    constexpr int ROWS = PHASE == 1 ? 8 : 16;              // weight rows (of each matrix) per task
    const int per = (width + ROWS - 1) / ROWS, blocks = PHASE == 1 ? p.hb : p.cb;
    const int k0 = kbs * ks / KS, k1 = kbs * (ks + 1) / KS;
    // Without an SM budget phase 1 lets phase 2's blocks in as SMs run out of work: those request their first weights and wait.  (They may
    // read the plan before they wait: it was complete before phase 1 came this far.)
    if (PHASE == 1) {
        pdl_wait();
        if (p.release) pdl_release();
    }
    const int total = __ldcg(p.n_groups) * per;
    bool waited = PHASE == 1;
    // Tasks are dealt out one by one.  (With a contiguous range per CTA the CTAs' streams run at a common distance from
    // each other: 64 tokens' down product 44 -> 53 us.)
    for (int t = blockIdx.x + gridDim.x * group; t < total; t += gridDim.x * NG) {
        const int gi = t / per, w0 = (t - gi * per) * ROWS;
        const int4 gr = __ldcg(p.groups + gi);
        const int e = gr.x, rows = gr.z;
        // tile-major: row r of this expert's 128-row block
        const size_t base = ((size_t)(e * blocks + (w0 >> 7)) * kbs * 128 + (w0 & 127) + g) * 64 + t4 * 8;
        const bf16* ra = (PHASE == 1 ? p.WgT : p.WdT) + base;
        const bf16* rb = PHASE == 1 ? p.WuT + base : ra + 8 * 64;
        Frag w[DEPTH];
#pragma unroll
        for (int u = 0; u < DEPTH; ++u)
            if (k0 + u < k1) ld_frag(w[u], ra, rb, k0 + u);
        if (!waited) {
            pdl_wait();
            waited = true;
        }
        auto source = [&](int j) -> const TRow* {           // this lane's row j of the group (past the end: the last one)
            const int pr = gr.y + min(j, rows - 1);
            if (PHASE == 2) return (const TRow*)(const void*)p.A + (size_t)pr * K;
            return (const TRow*)p.x + (size_t)(p.row_src ? p.row_src[pr] / p.k : pr) * K;
        };
        const int wa = w0 + g, wb = wa + 8;                 // hidden unit, or output columns
        auto task = [&](auto nn) {
            constexpr int NN = decltype(nn)::value;
            const TRow* src[NN];
#pragma unroll
            for (int n = 0; n < NN; ++n) src[n] = source(n * 8 + g);
            float acc[NN][4];
#pragma unroll
            for (int n = 0; n < NN; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[n][i] = 0.0f;
            run_task<NN, TRow>(w, ra, rb, src, k0, k1, K, t4, acc);
            if constexpr (KS > 1) {
                if (ks > 0)
#pragma unroll
                    for (int n = 0; n < NN; ++n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) red[group][ks - 1][n * 4 + i][lane] = acc[n][i];
                __syncwarp();
                asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(32 * KS) : "memory");
                if (ks == 0)
#pragma unroll
                    for (int s = 0; s < KS - 1; ++s)
#pragma unroll
                        for (int n = 0; n < NN; ++n)
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[n][i] += red[group][s][n * 4 + i][lane];
                __syncwarp();
                asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(32 * KS) : "memory");       // red is free again
                if (ks > 0) return;
            }
            if (wa >= width) return;
            if (PHASE == 1) {
                const float bg = __ldg(p.b0[e] + wa), bu = __ldg(p.b1[e] + wa);
#pragma unroll
                for (int n = 0; n < NN; ++n)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int j = n * 8 + t4 * 2 + i;
                        if (j < rows) {
                            const size_t row = (size_t)gr.y + j;
                            const float gt = acc[n][i] + bg, up = acc[n][2 + i] + bu;
                            const float sig = __fdividef(1.0f, 1.0f + __expf(-gt)), q = gt * sig;
                            p.out[row * p.H + wa] = __float2bfloat16(q * up);
                            if (p.G) {      // what backward needs of gate and up, in the layout gemm_tc.cu reads
                                const size_t o = ((row / ROW_TILE * (size_t)(p.H >> 3) + (wa >> 3)) * ROW_TILE + row % ROW_TILE) * 8 + (wa & 7);
                                p.G[o] = __float2bfloat16((up * sig) * (1.0f + (gt - q)));
                                p.U[o] = __float2bfloat16(q);
                            }
                        }
                    }
            } else {
                const float ba = __ldg(p.b0[e] + wa), bb = wb < width ? __ldg(p.b0[e] + wb) : 0.0f;
#pragma unroll
                for (int n = 0; n < NN; ++n)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int j = n * 8 + t4 * 2 + i;
                        if (j < rows) {
                            bf16* o = p.out + ((size_t)gr.y + j) * p.C;
                            o[wa] = __float2bfloat16(acc[n][i] + ba);
                            if (wb < width) o[wb] = __float2bfloat16(acc[n][2 + i] + bb);
                        }
                    }
            }
        };
        if (rows <= 8) task(std::integral_constant<int, 1>());
        else task(std::integral_constant<int, 2>());
    }
    if (!waited) pdl_wait();
}

template <int PHASE, bool F32>
int launch_phase(const DecP& p, int sms, cudaStream_t st)
{
    if ((PHASE == 1 ? p.kb1 : p.kb2) >= 8) MGPT_CUDA(launch_pdl(decode_kernel<PHASE, 4, F32>, sms, 32 * DW, 0, st, p));
    else MGPT_CUDA(launch_pdl(decode_kernel<PHASE, 1, F32>, sms, 32 * DW, 0, st, p));
    MGPT_LAUNCHED(PHASE == 1 ? "decode_kernel<gateup>" : "decode_kernel<down>");
    return 0;
}

}  // namespace

// Which forward calls take these kernels, training forwards like inference, so that both give the same bits: few rows, and
// either so few column tiles that the 128-row tcgen05 tiles' down product leaves half of the 148 SMs without one, or few
// weight bytes times rows.  These kernels save about 15 us of a call (no dispatch where nothing is kept, no first tile to
// wait for) and lose the more, the more weights stream by and the more rows meet each of them (B fragments and MMAs per
// weight, and a crowded expert's weights again for every 16 rows).  Inference calls, us with tiles / with these kernels, L2
// flushed (training steps at the same sizes, for which the rows are copied all the same: with these kernels up to 5 % slower where
// the routing is even, 3 % faster to 7 % slower where it is crowded):
//   tokens                           1       8       16       24       32       48       64      128
//   C=1024 H=2816 E=32 top-2     51/34   78/67   102/97  121/120  127/130  130/134  129/136  131/146
//     a few experts take most    51/36   55/38    54/40    54/42    57/48    57/52    57/65    61/97
//   C=2048 H=1408 E=64 top-2     57/40   98/87  134/124  143/146  173/174  186/202  213/224  227/254
//     a few experts take most    57/40   62/44    65/52    65/56    68/62    68/66    70/77   73/106
//   C=1024 H= 512 E=64 top-4     41/30   53/46    68/58    72/60    74/71    76/75    76/76    78/80
//   C=2048 H=2816 E= 8 top-2     65/46   98/83    98/83    97/85    97/87        .        .        .
//   C= 768 H=2048 E=16 top-2     43/29   64/52    64/56    66/58    66/58    66/59    66/60        .
// At the line in weight bytes times rows (32 tokens of the first width) an even routing loses 2 % and a crowded one gains 16 %;
// further on (64) both lose.  Which of the two a call has is not known here.
bool decode_usable(const Dims& d, int n_tokens)
{
    const double rows = (double)n_tokens * d.k, experts = rows < d.E ? rows : d.E;
    if (d.mode != MGPT_MOE_BF16 || d.gemm_impl != 0 || rows > 8.0 * d.E) return false;
    if (experts * ((d.C + 255) / 256) <= 74.0) return true;
    return experts * 6.0 * d.C * d.H * (1.0 + rows / d.E) <= 1.7e9;
}
// Room in the workspace, also where these kernels are not taken: a workspace never shrinks as the tokens grow.
int decode_max_groups(const Dims& d, int n_tokens)
{
    if (d.mode != MGPT_MOE_BF16 || d.gemm_impl != 0) return 0;
    const long long rows = (long long)n_tokens * d.k, most = 8ll * d.E;
    return d.E + (int)((rows < most ? rows : most) / DECODE_GROUP);
}

// gate/up and down; x: the tokens, or (from_rows) the permuted rows in the workspace.
int launch_decode_forward(mgpt_moe_layer* L, const Workspace& w, char* ws, const void* x, int io, bool from_rows, cudaStream_t st)
{
    const Dims& d = L->d;
    DecP p = {};
    p.WgT = L->sWgT; p.WuT = L->sWuT; p.WdT = L->sWdT;
    p.groups = (const int4*)(ws + w.groups);
    p.n_groups = (const int32_t*)(ws + w.n_groups);
    p.C = d.C; p.H = d.H; p.k = d.k;
    p.hb = (d.H + 127) / 128; p.cb = (d.C + 127) / 128; p.kb1 = (d.C + 63) / 64; p.kb2 = (d.H + 63) / 64;
    int sms = 0;
    MGPT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, L->device));
    p.release = 1;
    if (L->sm_budget > 0 && L->sm_budget < sms) {
        sms = L->sm_budget;
        p.release = 0;
    }
    p.x = from_rows ? (const void*)(ws + w.Xg) : x;
    p.row_src = from_rows ? nullptr : (const int32_t*)(ws + w.row_src);
    p.out = (bf16*)(ws + w.Hh);
    p.G = w.inference ? nullptr : (bf16*)(ws + w.G);
    p.U = w.inference ? nullptr : (bf16*)(ws + w.U);
    p.b0 = L->master.bg; p.b1 = L->master.bu;
    L->stage_begin(ST_GATEUP, st);
    if (from_rows || io == MGPT_MOE_IO_BF16) MGPT_TRY((launch_phase<1, false>(p, sms, st)));
    else MGPT_TRY((launch_phase<1, true>(p, sms, st)));
    L->stage_end(ST_GATEUP, st);
    p.A = (const bf16*)(ws + w.Hh);
    p.out = (bf16*)(ws + w.Yg);
    p.b0 = L->master.bd;
    L->stage_begin(ST_DOWN, st);
    MGPT_TRY((launch_phase<2, false>(p, sms, st)));
    L->stage_end(ST_DOWN, st);
    return 0;
}

}  // namespace mgpt
