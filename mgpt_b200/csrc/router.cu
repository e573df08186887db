// Router of the MoE layer: gating product, clamped softmax and top-k fused in
// one pass over x, and the matching backward kernels.
//
// Reference semantics reproduced here (paths relative to the reference's
// src/main/):
//   logits = x*Wr + br      layers/LinearLayer.cpp:23-28, utils/Tensor.cpp:567-577
//   P = clamp(softmax)      utils/Tensor.cpp:850-883 (inv = 1/max(sum,1e-15), clamp [1e-7,1])
//   top-k, strict '>'       utils/Tensor.cpp:1296-1334 (ties keep the lowest index)
//   backward                layers/MoELayer.cpp:189-218, utils/Tensor.cpp:885-909
//
// Routing must equal the CPU reference bit for bit, so the gating product is
// accumulated per (token, expert) sequentially over channels with a separate
// FP32 multiply and add, exactly the order of the reference's i-k-j loop.
#include <atomic>

#include "plan_block.cuh"

namespace mgpt {

namespace {

constexpr int R_WARPS = 4;     // warps per CTA of the kernel for any shape
constexpr int R_CK = 32;       // channels staged per step
constexpr int R_XPAD = 36;     // padded row of the staged x tile (floats): rows land in distinct banks

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(bf16 v) { return __bfloat162float(v); }

// Bias, softmax with the reference's summation order, clamp and top-k for the TPW token groups of a warp whose
// logit sums are in acc (layers/MoELayer.cpp:96-131).
template <int EL, int EPL, int TPW>
__device__ __forceinline__ void router_finish(const float (&acc)[TPW][EPL], const int* stok, int warp, int sub, int el,
                                              int E, int k, const float* br, float* logits,
                                              float* probs, int32_t* top_idx,
                                              float* top_p)
{
    constexpr int SUB = 32 / EL;
    constexpr int TOK_W = TPW * SUB;
    float bias[EPL];
#pragma unroll
    for (int i = 0; i < EPL; ++i) bias[i] = (el + 32 * i < E) ? br[el + 32 * i] : 0.0f;

    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int t = 0; t < TPW; ++t) {
        // every lane runs the warp-level steps (tokens past N compute on zeros and store nothing)
        const int tok = stok[warp * TOK_W + t * SUB + sub];
        const bool live = tok >= 0;
        float lg[EPL], p[EPL];
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
            lg[i] = __fadd_rn(acc[t][i], bias[i]);
            if (el + 32 * i < E) mx = fmaxf(mx, lg[i]);
        }
#pragma unroll
        for (int o = EL / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(full, mx, o));
        // exp through double and one rounding: agrees with a correctly rounded expf
#pragma unroll
        for (int i = 0; i < EPL; ++i) p[i] = (el + 32 * i < E) ? (float)exp((double)__fsub_rn(lg[i], mx)) : 0.0f;
        // the reference adds the E terms in index order
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
            const int lim = min(EL, E - 32 * i);
            for (int l = 0; l < lim; ++l) sum = __fadd_rn(sum, __shfl_sync(full, p[i], l, EL));
        }
        const float inv = __fdiv_rn(1.0f, fmaxf(sum, 1e-15f));
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
            p[i] = fminf(fmaxf(__fmul_rn(p[i], inv), 1e-7f), 1.0f);
            const int e = el + 32 * i;
            if (live && e < E) {
                probs[(size_t)tok * E + e] = p[i];
                if (logits) logits[(size_t)tok * E + e] = lg[i];
            }
        }
        // k rounds of (value desc, index asc) arg-max == the reference's stable insertion
        unsigned taken = 0;
        int my_idx = -1;
        float my_val = 0.0f;
        for (int r = 0; r < k; ++r) {
            float bv = -INFINITY;
            int bi = 0x7fffffff;
#pragma unroll
            for (int i = 0; i < EPL; ++i) {
                const int e = el + 32 * i;
                if (e < E && !(taken & (1u << i)) && p[i] > bv) {
                    bv = p[i];
                    bi = e;
                }
            }
#pragma unroll
            for (int o = EL / 2; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(full, bv, o);
                const int oi = __shfl_xor_sync(full, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            if ((bi & 31) == el && bi != 0x7fffffff) taken |= 1u << (bi >> 5);
            if (el == r) {
                my_idx = bi;
                my_val = bv;
            }
        }
        if (live && el < k) {
            top_idx[(size_t)tok * k + el] = my_idx;
            top_p[(size_t)tok * k + el] = my_val;
        }
    }
}

// The exact router.  What bounds it at scale is FP32 issue (one multiply and one add per token, expert and channel) and
// for small batches the addition chain of one (token, expert) pair, C additions of four cycles.
//
// ET lanes of one warp share a token, each with TE neighbouring experts of up to TM tokens (rows tt, tt + 256 / ET, ...: a
// warp works on the rows that it has tokens for), and read the next operands while they work on these.  RS = ET * TE, the
// experts rounded up, is the row length of the staged Wr, so that a thread's operands lie at constant offsets.  Wr and the tokens' rows stream through a ring that four warps fill with cp.async (one
// bulk copy per stage cost its issuing thread ~500 cycles, more than a small batch spends on the stage); the eight
// compute warps never wait for each other.  Softmax and top-k stay with the lanes that hold the logits: maximum and
// arg-max by shuffles, the sum -- sequential in the reference -- by every lane of the token from shared memory.  With
// plan.top_idx set, the last block to finish also builds the dispatch plan (one launch less for small batches).
//
// In a kernel of 128 compute threads with row lengths only known at run time, one thread per token for sum and top-k and stages of
// 128 channels, a channel took 14 cycles with one pair per thread and 38 with eight, the top-k 4000 cycles and the plan 7000-
// 17000.  Stage times before -> now, us: 1 token, C=1024, E=32, with the plan 22.4 -> 16.2; 64 tokens 28.7 -> 18.5; 256 tokens,
// without, 18.6 -> 15; 1777 tokens 26.4 -> 22.6; 5003 FP32 tokens, C=512, E=16 28.5 -> 20.7; both passes of the screened
// router, 16384 skewed tokens, C=1024, E=64, 91 -> 79.
//
// With RS a power of two from 16 on, numbers of experts between two of them paid for up to twice theirs, and rows of Wr off 16-byte
// boundaries were copied with two divisions per element: slower than the kernel of 128 threads.  FP32 tokens, C=512, us, that
// kernel / RS a power of two / now: 8 experts 32851 tokens 38 / 47 / 35; 24 experts 5619 tokens 18 / 21 / 16; 31 experts 291 tokens
// 8.9 / 11.8 / 6.4; 48 experts 5619 tokens 25 / 38 / 21; 80 experts 32851 tokens 265 / 266 / 163; 127 experts 504 / 572 / 235.
struct RouterArgs {
    const void* x;
    const float *Wr, *br;
    int N, C, E, k;
    int ck, stages, tok;    // channels (a power of two) and stages of the ring, tokens per CTA and round
    float *logits, *probs;
    int32_t* top_idx;
    float* top_p;
    const int32_t *list, *list_count;
    int32_t* status;        // error word (null: none)
    int32_t* done;          // blocks finished, zero between launches (with a plan)
    PlanArgs plan;
};

constexpr int RX_COMPUTE = 256, RX_PRODUCE = 128, RX_THREADS = RX_COMPUTE + RX_PRODUCE, RX_MAX_STAGES = 16;
__host__ __device__ inline uint32_t rx_x_row(int ck, int elt) { return (uint32_t)(ck * elt + 16); }      // padded: rows in distinct banks
__host__ __device__ inline uint32_t rx_stage(int ck, int rs, int tok, int elt)
{
    return ((uint32_t)ck * rs * 4 + tok * rx_x_row(ck, elt) + 127u) & ~127u;
}
constexpr uint32_t rx_tail(int et, int te, int tm) { return (uint32_t)(RX_COMPUTE / et) * tm * (et * te + 4) * 4; }      // exponentials, a row per token

// Loads with a 32-bit shared address: through pointers into the ring the compiler lost the address space, and a channel of one
// pair took 13 cycles instead of 8.
__device__ __forceinline__ uint4 lds128(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
template <int TE> __device__ __forceinline__ void lds_weights(float (&w)[TE], uint32_t a)
{
    if constexpr (TE == 4)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]) : "r"(a));
    else if constexpr (TE % 2 == 0)
#pragma unroll
        for (int j = 0; j < TE; j += 2) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(w[j]), "=f"(w[j + 1]) : "r"(a + 4 * j));
    else
#pragma unroll
        for (int j = 0; j < TE; ++j) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(w[j]) : "r"(a + 4 * j));
}
// L consecutive channels (4 or 8) of a staged row
template <typename TIn, int L> struct Row;
template <int L> struct Row<bf16, L> {
    uint32_t u[L / 2];
    __device__ __forceinline__ void load(uint32_t a)
    {
        if constexpr (L == 8) {
            const uint4 v = lds128(a);
            u[0] = v.x; u[1] = v.y; u[2] = v.z; u[3] = v.w;
        } else {
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(u[0]), "=r"(u[1]) : "r"(a));
        }
    }
    __device__ __forceinline__ float get(int i) const { return __uint_as_float((i & 1) ? u[i >> 1] & 0xffff0000u : u[i >> 1] << 16); }
};
template <int L> struct Row<float, L> {
    uint4 u[L / 4];
    __device__ __forceinline__ void load(uint32_t a)
    {
#pragma unroll
        for (int i = 0; i < L / 4; ++i) u[i] = lds128(a + 16 * i);
    }
    __device__ __forceinline__ float get(int i) const
    {
        const uint4& f = u[i >> 2];
        return __uint_as_float((i & 3) == 0 ? f.x : (i & 3) == 1 ? f.y : (i & 3) == 2 ? f.z : f.w);
    }
};

template <typename TIn, int ET, int TE, int TM>
__global__ void __launch_bounds__(RX_THREADS, 1) router_exact_kernel(const RouterArgs p)
{
    extern __shared__ __align__(128) uint8_t rx_smem[];
    __shared__ __align__(8) uint64_t bars[2 * RX_MAX_STAGES];
    __shared__ int last;
    constexpr int RS = ET * TE, GROUPS = RX_COMPUTE / ET;
    static_assert(TM >= 1 && TM <= 4, "rows of a warp");
    static_assert((ET & (ET - 1)) == 0 && ET <= 32 && RS % 4 == 0, "a token's lanes lie in one warp");
    const int tid = threadIdx.x, lane = tid & 31;
    const int C = p.C, E = p.E, CK = p.ck, ST = p.stages;
    const uint32_t x_row = rx_x_row(CK, sizeof(TIn)), x_off = (uint32_t)CK * RS * 4, stage = rx_stage(CK, RS, p.tok, sizeof(TIn));
    const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(rx_smem);
    const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (RX_MAX_STAGES + s); };
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full(s)), "r"(RX_PRODUCE));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty(s)), "r"(RX_COMPUTE / 32));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    // as few rounds as the CTAs can do it in, all alike
    const int n_active = p.list ? *p.list_count : p.N, rounds = max(1, (n_active + (int)gridDim.x * p.tok - 1) / ((int)gridDim.x * p.tok));
    const int TOK = max(1, (n_active + (int)gridDim.x * rounds - 1) / ((int)gridDim.x * rounds)), n_tiles = (n_active + TOK - 1) / TOK;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        for (uint32_t i = 0; i < (1u << 20); ++i) {
            uint32_t ok;
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                         : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
            if (ok) return;
        }
        if (p.status) atomicOr(p.status, ST_FULL_WAIT);
    };

    if (tid >= RX_COMPUTE) {
        // fills the ring
        constexpr int XV = 16 / sizeof(TIn);
        const int per_log = __ffs(CK / XV) - 1, pt = tid - RX_COMPUTE;        // 16-byte pieces per row and chunk
        // A row of Wr may be shorter than the staged one: piece pt, pt + 128, ... of the rows, column and row by addition.  (A column
        // per thread leaves up to half of them without: 296 tokens, C=1024, 4 experts 10.7 us; two divisions per element before
        // that, 127 experts 572 us for 32851 tokens.)
        const bool wide = (E & 3) == 0;
        int per = 1, r0 = 0, q0 = 0, dr = 0, dq = 0;
        if (E != RS) {
            per = wide ? E >> 2 : E;
            r0 = pt / per;
            q0 = pt % per;
            dr = RX_PRODUCE / per;
            dq = RX_PRODUCE % per;
        }
        auto step = [&](int& r, int& q) {
            r += dr;
            q += dq;
            if (q >= per) {
                q -= per;
                ++r;
            }
        };
        int s = 0;
        uint32_t round = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const int n = min(TOK, n_active - tile * TOK);
            for (int c0 = 0; c0 < C; c0 += CK) {
                if (round > 0) wait(empty(s), (round - 1) & 1);
                const int len = min(CK, C - c0), pieces = len / XV;
                const uint32_t dst = ring0 + s * stage;
                const float* src = p.Wr + (size_t)c0 * E;
                if (E == RS) {
                    for (int v = pt; v < len * (RS / 4); v += RX_PRODUCE)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + v * 16), "l"(src + v * 4) : "memory");
                } else if (wide) {
                    for (int v = pt, r = r0, q = q0; v < len * per; v += RX_PRODUCE) {
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (r * RS + q * 4) * 4), "l"(src + v * 4) : "memory");
                        step(r, q);
                    }
                } else {
                    for (int v = pt, r = r0, q = q0; v < len * per; v += RX_PRODUCE) {
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + (r * RS + q) * 4), "l"(src + v) : "memory");
                        step(r, q);
                    }
                }
                for (int v = pt; v < n << per_log; v += RX_PRODUCE) {
                    const int i = v >> per_log, q = v & ((1 << per_log) - 1);
                    if (q < pieces) {
                        const int tok = p.list ? p.list[tile * TOK + i] : tile * TOK + i;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                     ::"r"(dst + x_off + i * x_row + q * 16), "l"((const TIn*)p.x + (size_t)tok * C + c0 + q * XV) : "memory");
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full(s)) : "memory");
                if (++s == ST) {
                    s = 0;
                    ++round;
                }
            }
        }
    } else {
        const int te = tid % ET, tt = tid / ET, e0 = te * TE;
        float* const ex = reinterpret_cast<float*>(rx_smem + ST * stage) + (size_t)tt * TM * (RS + 4);
        float bias[TE];
#pragma unroll
        for (int j = 0; j < TE; ++j) bias[j] = e0 + j < E ? p.br[e0 + j] : 0.0f;
        int s = 0;
        uint32_t round = 0;
        // one tile of n tokens, of which this warp has R rows (tt, tt + GROUPS, ...), or none
        auto work_tile = [&](auto rows, bool works, int tile, int n) {
            constexpr int R = decltype(rows)::value;
            uint32_t xr[R];
#pragma unroll
            for (int t = 0; t < R; ++t) xr[t] = x_off + min(tt + t * GROUPS, p.tok - 1) * x_row;      // (past the end: not stored)
            float acc[R][TE];
#pragma unroll
            for (int t = 0; t < R; ++t)
#pragma unroll
                for (int j = 0; j < TE; ++j) acc[t][j] = 0.0f;
            for (int c0 = 0; c0 < C; c0 += CK) {
                const int len = min(CK, C - c0);
                wait(full(s), round & 1);
                if (works) {
                    const uint32_t base = ring0 + s * stage, ws = base + e0 * 4;
                    // U channels' operands at a time; two sets, the next one on its way.  (More pairs need fewer channels to hide a
                    // load behind, and longer sets cost them registers: 16 x 3 x 4 BF16 tokens 57 -> 50 us with 4.  One pair of
                    // BF16 tokens: 8.2 -> 7.9 us for 100 tokens, C=1024, 16 experts with 32; FP32 tokens 3 % slower,
                    // 32 experts no faster, and 1 us slower in a call whose instructions come from HBM.)
                    constexpr int U = TE * R == 1 && sizeof(TIn) == 2 && ET <= 16 ? 32 : TE * R <= 2 ? 16 : TE * R <= (sizeof(TIn) == 2 ? 8 : 4) ? 8 : 4, L = U < 8 ? U : 8;
                    struct Ops {
                        float w[U][TE];
                        Row<TIn, L> x[R][U / L];
                    };
                    auto load = [&](Ops& o, int c) {
                        const uint32_t wc = ws + c * (RS * 4);
#pragma unroll
                        for (int t = 0; t < R; ++t)
#pragma unroll
                            for (int i = 0; i < U / L; ++i) o.x[t][i].load(base + xr[t] + (c + L * i) * sizeof(TIn));
#pragma unroll
                        for (int u = 0; u < U; ++u) lds_weights<TE>(o.w[u], wc + u * (RS * 4));
                    };
                    // acc = fadd(acc, fmul(x, w)) in channel order, the reference's order; four channels' products first, so
                    // that no addition waits for its product
                    auto work = [&](const Ops& o) {
#pragma unroll
                        for (int h = 0; h < U; h += 4) {
                            float pr[4][R][TE];
#pragma unroll
                            for (int u = 0; u < 4; ++u)
#pragma unroll
                                for (int t = 0; t < R; ++t) {
                                    const float xv = o.x[t][(h + u) / L].get((h + u) % L);
#pragma unroll
                                    for (int j = 0; j < TE; ++j) pr[u][t][j] = __fmul_rn(xv, o.w[h + u][j]);
                                }
#pragma unroll
                            for (int u = 0; u < 4; ++u)
#pragma unroll
                                for (int t = 0; t < R; ++t)
#pragma unroll
                                    for (int j = 0; j < TE; ++j) acc[t][j] = __fadd_rn(acc[t][j], pr[u][t][j]);
                        }
                    };
                    Ops a, b;
                    int c = 0;
                    if (len >= 2 * U) {
                        load(a, 0);
#pragma unroll 1
                        for (; c + 2 * U <= len; c += 2 * U) {
                            load(b, c + U);
                            work(a);
                            load(a, min(c + 2 * U, len - U));       // (the last one again: no branch)
                            work(b);
                        }
                    }
#pragma unroll 1
                    for (; c < len; c += 8) {                       // the rest of a last chunk, eight channels at a time
                        float w[8][TE];
#pragma unroll
                        for (int u = 0; u < 8; ++u) lds_weights<TE>(w[u], ws + (c + u) * (RS * 4));
#pragma unroll
                        for (int t = 0; t < R; ++t) {
                            Row<TIn, 8> x;
                            x.load(base + xr[t] + c * sizeof(TIn));
#pragma unroll
                            for (int u = 0; u < 8; ++u)
#pragma unroll
                                for (int j = 0; j < TE; ++j) acc[t][j] = __fadd_rn(acc[t][j], __fmul_rn(x.get(u), w[u][j]));
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty(s)) : "memory");
                if (++s == ST) {
                    s = 0;
                    ++round;
                }
            }
            if (works) {
                // clamped softmax (utils/Tensor.cpp:850-883) and top-k, strict '>' (utils/Tensor.cpp:1296-1334)
                const unsigned all = 0xffffffffu;
                float lg[R][TE], pr[R][TE];
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    float mx = -INFINITY;
#pragma unroll
                    for (int j = 0; j < TE; ++j) {
                        lg[t][j] = __fadd_rn(acc[t][j], bias[j]);
                        if (e0 + j < E) mx = fmaxf(mx, lg[t][j]);
                    }
#pragma unroll
                    for (int o = ET / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(all, mx, o));
                    // exp through double and one rounding: agrees with a correctly rounded expf
#pragma unroll
                    for (int j = 0; j < TE; ++j) pr[t][j] = e0 + j < E ? (float)exp((double)__fsub_rn(lg[t][j], mx)) : 0.0f;
#pragma unroll
                    for (int j = 0; j < TE; ++j) ex[t * (RS + 4) + e0 + j] = pr[t][j];
                }
                __syncwarp();
                float sum[R] = {};
                for (int e = 0; e < E; e += 4)                      // in index order (zeros past the last: they add nothing)
#pragma unroll
                    for (int t = 0; t < R; ++t) {
                        const float4 v = *reinterpret_cast<const float4*>(ex + t * (RS + 4) + e);
                        sum[t] = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum[t], v.x), v.y), v.z), v.w);
                    }
                __syncwarp();
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    const int i = tt + t * GROUPS;
                    const bool live = i < n;
                    const size_t tok = live ? (p.list ? p.list[tile * TOK + i] : tile * TOK + i) : 0;
                    const float inv = __fdiv_rn(1.0f, fmaxf(sum[t], 1e-15f));
#pragma unroll
                    for (int j = 0; j < TE; ++j) {
                        pr[t][j] = fminf(fmaxf(__fmul_rn(pr[t][j], inv), 1e-7f), 1.0f);
                        if (live && e0 + j < E) {
                            p.probs[tok * E + e0 + j] = pr[t][j];
                            if (p.logits) p.logits[tok * E + e0 + j] = lg[t][j];
                        }
                    }
                    // k rounds of (value desc, index asc) arg-max == the reference's stable insertion
                    unsigned taken = 0;
                    for (int r = 0; r < p.k; ++r) {
                        float bv = -INFINITY;
                        int bi = 0x7fffffff;
#pragma unroll
                        for (int j = 0; j < TE; ++j)
                            if (e0 + j < E && !(taken >> j & 1u) && pr[t][j] > bv) {
                                bv = pr[t][j];
                                bi = e0 + j;
                            }
#pragma unroll
                        for (int o = ET / 2; o > 0; o >>= 1) {
                            const float ov = __shfl_xor_sync(all, bv, o);
                            const int oi = __shfl_xor_sync(all, bi, o);
                            if (ov > bv || (ov == bv && oi < bi)) {
                                bv = ov;
                                bi = oi;
                            }
                        }
                        if (bi / TE == te) taken |= 1u << (bi % TE);
                        if (live && te == 0) {
                            p.top_idx[tok * p.k + r] = bi;
                            p.top_p[tok * p.k + r] = bv;
                        }
                    }
                }
            }
        };
        const int first = (tid & ~31) / ET;                 // the warp's first token
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const int n = min(TOK, n_active - tile * TOK), rows = n > first ? (n - first + GROUPS - 1) / GROUPS : 0;       // (warp-uniform)
            if (TM == 1 || rows <= 1) work_tile(std::integral_constant<int, 1>(), rows > 0, tile, n);
            else if (TM == 2 || rows == 2) work_tile(std::integral_constant<int, (TM >= 2 ? 2 : 1)>(), true, tile, n);
            else if (TM == 3 || rows == 3) work_tile(std::integral_constant<int, (TM >= 3 ? 3 : 1)>(), true, tile, n);
            else work_tile(std::integral_constant<int, (TM >= 4 ? 4 : 1)>(), true, tile, n);
        }
    }
    if (!p.plan.top_idx) return;
    if (gridDim.x > 1) {
        __threadfence();
        __syncthreads();
        if (tid == 0) last = atomicAdd(p.done, 1) == (int)gridDim.x - 1;
        __syncthreads();
        if (!last) return;
        __threadfence();
        if (tid == 0) *p.done = 0;
    } else {
        __syncthreads();
    }
    plan_block<RX_THREADS / 32>(p.plan, *reinterpret_cast<PlanShared*>(rx_smem));
}

// EL lanes share one token (lane % EL owns experts el, el+32, ...: EPL of them, EPL > 1 only
// with EL = 32); a warp therefore works on 32/EL tokens at once and on TPW such groups in
// sequence, which gives every lane TPW*EPL independent accumulation chains.
// For shapes and addresses the kernel above cannot take (C not a multiple of 8, x or Wr not 16-byte aligned).
template <typename TIn, int EL, int EPL, int TPW>
__global__ void __launch_bounds__(R_WARPS * 32)
router_fwd_kernel(const TIn* x, const float* Wr, const float* br,
                  int N, int C, int E, int k,
                  float* logits, float* probs,
                  int32_t* top_idx, float* top_p,
                  const int32_t* list, const int32_t* list_count)
{
    pdl_wait();
    constexpr int SUB = 32 / EL;                    // tokens per warp pass
    constexpr int TOK_W = TPW * SUB;                // tokens per warp
    constexpr int TOK = R_WARPS * TOK_W;            // tokens per CTA
    constexpr int WCOLS = EPL * EL;                 // staged expert columns
    constexpr int THREADS = R_WARPS * 32;
    __shared__ __align__(16) float xs[TOK][R_XPAD];
    __shared__ __align__(16) float wsm[R_CK][WCOLS];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane / EL, el = lane % EL;
    const int tok0 = blockIdx.x * TOK;

    // The CTA's tokens: a contiguous range, or -- second pass of the screened router -- entries of a list of
    // token indices whose length is only known on the device (CTAs beyond it leave at once).
    __shared__ int stok[TOK];
    const int n_active = list ? *list_count : N;
    if (tok0 >= n_active) return;
    for (int i = tid; i < TOK; i += THREADS) {
        const int idx = tok0 + i;
        stok[i] = idx < n_active ? (list ? list[idx] : idx) : -1;
    }
    __syncthreads();
    float acc[TPW][EPL];
#pragma unroll
    for (int t = 0; t < TPW; ++t)
#pragma unroll
        for (int i = 0; i < EPL; ++i) acc[t][i] = 0.0f;

    // sequential over the 32 staged channels: acc = fadd(acc, fmul(x, w)), the reference's order
    auto compute = [&]() {
#pragma unroll 2
        for (int j = 0; j < R_CK; j += 4) {
            float4 xv[TPW];
#pragma unroll
            for (int t = 0; t < TPW; ++t)
                xv[t] = *reinterpret_cast<const float4*>(&xs[warp * TOK_W + t * SUB + sub][j]);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                float w[EPL];
#pragma unroll
                for (int i = 0; i < EPL; ++i) w[i] = wsm[j + jj][el + 32 * i];
#pragma unroll
                for (int t = 0; t < TPW; ++t) {
                    const float xe = jj == 0 ? xv[t].x : jj == 1 ? xv[t].y : jj == 2 ? xv[t].z : xv[t].w;
#pragma unroll
                    for (int i = 0; i < EPL; ++i) acc[t][i] = __fadd_rn(acc[t][i], __fmul_rn(xe, w[i]));
                }
            }
        }
    };

    for (int c0 = 0; c0 < C; c0 += R_CK) {
        // stage x[tok0.., c0..c0+31] and Wr[c0..c0+31, :] (zero padded: adding 0*w is exact)
#pragma unroll 4
        for (int i = tid; i < TOK * R_CK; i += THREADS) {
            const int t = i / R_CK, j = i % R_CK;
            const int tok = stok[t], c = c0 + j;
            xs[t][j] = (tok >= 0 && c < C) ? to_f32(x[(size_t)tok * C + c]) : 0.0f;
        }
#pragma unroll 4
        for (int i = tid; i < R_CK * WCOLS; i += THREADS) {
            const int j = i / WCOLS, e = i % WCOLS;
            const int c = c0 + j;
            wsm[j][e] = (c < C && e < E) ? Wr[(size_t)c * E + e] : 0.0f;
        }
        __syncthreads();
        compute();
        __syncthreads();
    }

    router_finish<EL, EPL, TPW>(acc, stok, warp, sub, el, E, k, br, logits, probs, top_idx, top_p);
}

// dlogits = P * (dP - <dP,P>),  dP = scatter(d_top_p) + alpha*E*f_e/N
// (layers/MoELayer.cpp:189-210).  One warp for four tokens at a time, grid-stride.  The sum over the experts has the
// reference's order, a chain of E additions: the products cross through shared memory, and four lanes run the chains of
// the four tokens (one shuffle per expert and token instead was the kernel: 27 -> 14 us at 32768 tokens, E=64).
// Optionally also writes a bf16 copy with rows padded to E8 columns (for the tensor-core backward) and adds
// the column sums to gbr (layers/LinearLayer.cpp:56-57).
template <int EPL>
__global__ void __launch_bounds__(256)
router_dlogits_kernel(const float* probs, const int32_t* top_idx,
                      const float* d_top_p, const int32_t* counts,
                      int N, int E, int k, float alpha, float* dlogits,
                      bf16* dl16, int E8, float* gbr)
{
    pdl_wait();
    constexpr int T = 4;
    __shared__ float bred[8][EPL * 32];
    __shared__ __align__(16) float prods[8][T][EPL * 32 + 4];     // (+ 4: the rows of a 16-byte read in different banks)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    float lb[EPL], bsum[EPL];
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
        const int e = lane + 32 * i;
        bsum[i] = 0.0f;
        lb[i] = 0.0f;
        if (e < E) {
            const float f = __fdiv_rn((float)counts[e], (float)N);
            lb[i] = __fdiv_rn(__fmul_rn(__fmul_rn(alpha, (float)E), f), (float)N);
        }
    }
    for (int tok0 = (blockIdx.x * 8 + warp) * T; tok0 < N; tok0 += gridDim.x * 8 * T) {
        float p[T][EPL], dp[T][EPL];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int tok = tok0 + t;
            // lane j < k has the token's j-th choice
            const bool mine = tok < N && lane < k;
            const int idx = mine ? top_idx[(size_t)tok * k + lane] : -1;
            const float d = mine ? d_top_p[(size_t)tok * k + lane] : 0.0f;
#pragma unroll
            for (int i = 0; i < EPL; ++i) {
                const int e = lane + 32 * i;
                p[t][i] = tok < N && e < E ? probs[(size_t)tok * E + e] : 0.0f;
                dp[t][i] = 0.0f;
            }
            for (int j = 0; j < k; ++j) {
                const int e = __shfl_sync(full, idx, j);
                const float v = __shfl_sync(full, d, j);
#pragma unroll
                for (int i = 0; i < EPL; ++i)
                    if (e == lane + 32 * i) dp[t][i] = v;
            }
#pragma unroll
            for (int i = 0; i < EPL; ++i) dp[t][i] = lane + 32 * i < E ? __fadd_rn(dp[t][i], lb[i]) : 0.0f;
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < T; ++t)
#pragma unroll
            for (int i = 0; i < EPL; ++i) prods[warp][t][lane + 32 * i] = __fmul_rn(dp[t][i], p[t][i]);
        __syncwarp();
        float chain = 0.0f;                                       // (the products past E are zeros)
        if (lane < T)
#pragma unroll 8
            for (int e = 0; e < E; e += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&prods[warp][lane][e]);
                chain = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(chain, v.x), v.y), v.z), v.w);
            }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int tok = tok0 + t;
            const float dot = __shfl_sync(full, chain, t);
            if (tok >= N) continue;
#pragma unroll
            for (int i = 0; i < EPL; ++i) {
                const int e = lane + 32 * i;
                const float v = e < E ? __fmul_rn(p[t][i], __fsub_rn(dp[t][i], dot)) : 0.0f;
                if (e < E) dlogits[(size_t)tok * E + e] = v;
                if (dl16 && e < E8) dl16[(size_t)tok * E8 + e] = __float2bfloat16(v);
                bsum[i] += v;
            }
        }
    }
    if (gbr) {
#pragma unroll
        for (int i = 0; i < EPL; ++i) bred[warp][lane + 32 * i] = bsum[i];
        __syncthreads();
        for (int e = threadIdx.x; e < E; e += blockDim.x) {
            float t = 0.0f;
#pragma unroll
            for (int wv = 0; wv < 8; ++wv) t += bred[wv][e];
            atomicAdd(&gbr[e], t);
        }
    }
}

// dx[tok,:] = sum_j dXg[pos(tok,j),:] (ascending slot order, as the reference's
// scatter-add visits them, utils/Tensor.cpp:1451-1458) + dlogits[tok,:] * Wr^T
// (layers/LinearLayer.cpp:68-69, layers/MoELayer.cpp:217).
// One CTA: 64 channels of 32*TPT tokens, a thread owns 8 consecutive channels of TPT tokens; Wr^T of the channels and
// dlogits^T of the tokens in shared memory.  TPT = 4 where that still gives every SM two CTAs (the products are then 32
// multiply-adds per three 16-byte shared-memory reads), else 1.  (Whole rows of 64 tokens per CTA left most SMs idle:
// 25 us at 1024 tokens, C = 128, E = 8 and 30 us at 5003 tokens, C = 512, E = 16.)
constexpr int DX_CH = 64;
template <typename TAct> __device__ __forceinline__ void add_row8(float (&s)[8], const TAct* r)
{
    if constexpr (sizeof(TAct) == 2) {
        const uint4 u = *reinterpret_cast<const uint4*>(r);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s[2 * i] = __fadd_rn(s[2 * i], __uint_as_float(w[i] << 16));
            s[2 * i + 1] = __fadd_rn(s[2 * i + 1], __uint_as_float(w[i] & 0xffff0000u));
        }
    } else {
        const float4 a = *reinterpret_cast<const float4*>(r), b = *reinterpret_cast<const float4*>(r + 4);
        s[0] = __fadd_rn(s[0], a.x); s[1] = __fadd_rn(s[1], a.y); s[2] = __fadd_rn(s[2], a.z); s[3] = __fadd_rn(s[3], a.w);
        s[4] = __fadd_rn(s[4], b.x); s[5] = __fadd_rn(s[5], b.y); s[6] = __fadd_rn(s[6], b.z); s[7] = __fadd_rn(s[7], b.w);
    }
}
template <int TPT> constexpr size_t dx_smem(int E) { return (size_t)E * (DX_CH + 4 + 32 * TPT) * sizeof(float); }

template <typename TAct, typename TIo, int TPT>
__global__ void __launch_bounds__(256)
router_dx_kernel(const TAct* dXg, const int32_t* pos, const float* dlogits,
                 const float* Wr, int N, int C, int E, int k, TIo* dx)
{
    pdl_wait();
    constexpr int TOK = 32 * TPT, WS = DX_CH + 4;       // padded row: transposed staging without 32-way conflicts
    extern __shared__ __align__(16) float sm_dx[];
    float* wt = sm_dx;                                  // [E][DX_CH+4]  (Wr^T of these channels)
    float* dlT = sm_dx + E * WS;                        // [E][TOK]  (dlogits^T of these tokens)
    __shared__ int spos[TOK][MAX_TOPK];
    const int tok0 = blockIdx.x * TOK, c_base = blockIdx.y * DX_CH;
    for (int i = threadIdx.x; i < DX_CH * E; i += blockDim.x) {
        const int c = i / E, e = i % E;
        wt[e * WS + c] = (c_base + c < C) ? Wr[(size_t)c_base * E + i] : 0.0f;
    }
    for (int i = threadIdx.x; i < TOK * E; i += blockDim.x) {
        const int t = i / E, e = i % E;
        dlT[e * TOK + t] = (tok0 + t < N) ? dlogits[(size_t)tok0 * E + i] : 0.0f;
    }
    if (threadIdx.x < TOK) {
        const int tok = tok0 + threadIdx.x;
        int v[MAX_TOPK];
#pragma unroll
        for (int j = 0; j < MAX_TOPK; ++j) v[j] = (j < k && tok < N) ? pos[(size_t)tok * k + j] : 0x7fffffff;
#pragma unroll
        for (int a = 0; a < MAX_TOPK - 1; ++a)
#pragma unroll
            for (int b = 0; b < MAX_TOPK - 1 - a; ++b)
                if (v[b] > v[b + 1]) {
                    const int tmp = v[b];
                    v[b] = v[b + 1];
                    v[b + 1] = tmp;
                }
#pragma unroll
        for (int j = 0; j < MAX_TOPK; ++j) spos[threadIdx.x][j] = v[j];
    }
    __syncthreads();
    const int g = threadIdx.x & 7, tl0 = (threadIdx.x >> 3) * TPT;
    const int c = c_base + g * 8;
    if (c >= C) return;
    float acc[TPT][8];
#pragma unroll
    for (int t = 0; t < TPT; ++t)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[t][i] = 0.0f;
#pragma unroll 4
    for (int e = 0; e < E; ++e) {
        const float4 w0 = *reinterpret_cast<const float4*>(&wt[e * WS + g * 8]);
        const float4 w1 = *reinterpret_cast<const float4*>(&wt[e * WS + g * 8 + 4]);
        const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
        float dv[TPT];
        if constexpr (TPT == 4) {
            const float4 d = *reinterpret_cast<const float4*>(&dlT[e * TOK + tl0]);
            dv[0] = d.x; dv[1] = d.y; dv[2] = d.z; dv[3] = d.w;
        } else {
            dv[0] = dlT[e * TOK + tl0];
        }
#pragma unroll
        for (int t = 0; t < TPT; ++t)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[t][i] = fmaf(dv[t], wv[i], acc[t][i]);
    }
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        const int tl = tl0 + t, tok = tok0 + tl;
        if (tok >= N) break;
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int j = 0; j < k; ++j) add_row8(s, dXg + (size_t)spos[tl][j] * C + c);
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = __fadd_rn(s[i], acc[t][i]);
        TIo* o = dx + (size_t)tok * C + c;
        if constexpr (sizeof(TIo) == 4) {
            *reinterpret_cast<float4*>(o) = make_float4(s[0], s[1], s[2], s[3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(s[4], s[5], s[6], s[7]);
        } else {
            uint4 u;
            __nv_bfloat162 h0 = __floats2bfloat162_rn(s[0], s[1]), h1 = __floats2bfloat162_rn(s[2], s[3]);
            __nv_bfloat162 h2 = __floats2bfloat162_rn(s[4], s[5]), h3 = __floats2bfloat162_rn(s[6], s[7]);
            u.x = *reinterpret_cast<uint32_t*>(&h0); u.y = *reinterpret_cast<uint32_t*>(&h1);
            u.z = *reinterpret_cast<uint32_t*>(&h2); u.w = *reinterpret_cast<uint32_t*>(&h3);
            *reinterpret_cast<uint4*>(o) = u;
        }
    }
}

// Router weight gradient in two deterministic steps (layers/LinearLayer.cpp:56-66):
//   part[chunk][c][e] = sum over the chunk's tokens of x[tok,c]*dlogits[tok,e]   (and column sums of dlogits)
//   gWr[c,e] += sum_chunk part[chunk][c][e];  gbr[e] += sum_chunk partb[chunk][e]
// A thread keeps a 4 channel x 4 expert block of accumulators.
template <typename TIo>
__global__ void __launch_bounds__(256)
router_wgrad_partial_kernel(const TIo* x, const float* dlogits, int N, int C, int E,
                            int tok_per_chunk, float* part, float* partb)
{
    pdl_wait();
    const int E4 = (E + 3) / 4;                         // expert groups of 4
    const int cg_per_cta = 256 / E4;                    // channel groups of 4 handled by this CTA
    const int eg = threadIdx.x % E4, cgi = threadIdx.x / E4;
    if (cgi >= cg_per_cta) return;
    const int c = (blockIdx.x * cg_per_cta + cgi) * 4, e0 = eg * 4;
    const int t0 = blockIdx.y * tok_per_chunk, t1 = min(N, t0 + tok_per_chunk);
    const bool c_ok = c < C;
    float acc[4][4] = {};
    float bs[4] = {0, 0, 0, 0};
    constexpr int UN = 8;                               // tokens in flight per thread
    const bool e_vec = (E & 3) == 0;                    // dlogits in 16-byte pieces
    for (int tb = t0; tb < t1; tb += UN) {
        float xv[UN][4], dv[UN][4];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int tok = tb + u;
            const bool ok = tok < t1;
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[u][i] = 0.0f;
            if (ok && c_ok) {
                if constexpr (sizeof(TIo) == 2) {
                    const uint2 w = *reinterpret_cast<const uint2*>(x + (size_t)tok * C + c);
                    xv[u][0] = __uint_as_float(w.x << 16); xv[u][1] = __uint_as_float(w.x & 0xffff0000u);
                    xv[u][2] = __uint_as_float(w.y << 16); xv[u][3] = __uint_as_float(w.y & 0xffff0000u);
                } else {
                    const float4 f = *reinterpret_cast<const float4*>(x + (size_t)tok * C + c);
                    xv[u][0] = f.x; xv[u][1] = f.y; xv[u][2] = f.z; xv[u][3] = f.w;
                }
            }
            if (e_vec) {
                const float4 f = ok ? *reinterpret_cast<const float4*>(dlogits + (size_t)tok * E + e0) : make_float4(0, 0, 0, 0);
                dv[u][0] = f.x; dv[u][1] = f.y; dv[u][2] = f.z; dv[u][3] = f.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) dv[u][j] = (ok && e0 + j < E) ? dlogits[(size_t)tok * E + e0 + j] : 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[u][i], dv[u][j], acc[i][j]);
#pragma unroll
            for (int j = 0; j < 4; ++j) bs[j] += dv[u][j];
        }
    }
    if (c_ok) {
        float* dst = part + ((size_t)blockIdx.y * C + c) * E;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (e0 + j < E) dst[(size_t)i * E + e0 + j] = acc[i][j];
    }
    if (blockIdx.x == 0 && cgi == 0)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (e0 + j < E) partb[(size_t)blockIdx.y * E + e0 + j] = bs[j];
}

// 32 elements per CTA, the chunks shared out over 8 threads per element (one thread per element walked up to 64 chunks
// one after another: 6 us for 1024 elements)
__global__ void __launch_bounds__(256)
router_wgrad_reduce_kernel(const float* part, const float* partb, int n_chunks, int CE, int E,
                           float* gWr, float* gbr)
{
    pdl_wait();
    __shared__ float red[8][32];
    const int x = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + x;                  // elements CE .. CE+E-1 are the bias gradient
    const bool bias = i >= CE;
    const float* src = bias ? partb + (i - CE) : part + i;
    const size_t stride = bias ? E : CE;
    float s = 0.0f;
    if (i < CE + E)
#pragma unroll 8
        for (int ch = slice; ch < n_chunks; ch += 8) s += src[(size_t)ch * stride];
    red[slice][x] = s;
    __syncthreads();
    if (slice == 0 && i < CE + E) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red[w][x];
        if (bias) gbr[i - CE] += t;
        else gWr[i] += t;
    }
}

template <typename TIn, int ET, int TE, int TM>
int router_exact_launch(RouterArgs p, int device, cudaStream_t st)
{
    auto* kernel = router_exact_kernel<TIn, ET, TE, TM>;
    constexpr int RS = ET * TE;
    // Every SM its share of the tokens (a list's length is only known on the device: two rows per warp), in the rounds that cost
    // least (one of 1, 2, 3, 4 rows of 16 tokens x 64 experts x 1024 channels: 20, 28, 41, 55 us; the other forms alike).
    constexpr int GROUPS = RX_COMPUTE / ET;
    const int share = p.list ? GROUPS * (TM < 2 ? TM : 2) : (p.N + 147) / 148;
    int rounds = 0, least = 0;
    for (int r = 1; r <= TM; ++r) {
        const int n = (share + GROUPS * r - 1) / (GROUPS * r), cost = n * (r == 1 ? 10 : 6 * r + 3);
        if (!rounds || cost < least) {
            rounds = n;
            least = cost;
        }
    }
    p.tok = (share + rounds - 1) / rounds;
    // A stage's beginning and end cost 650 cycles (one warp per scheduler hides no instruction fetch), so stages are long: 512
    // channels with a few tokens, whose loads are all on their way at once, 256 with more; two of them fit.
    for (p.ck = p.tok <= 4 ? 512 : 256; p.ck > 16 && rx_stage(p.ck, RS, p.tok, sizeof(TIn)) > 90u * 1024u;) p.ck /= 2;
    const int ctas = (p.N + p.tok - 1) / p.tok, grid = ctas < 148 ? ctas : 148;
    const uint32_t stage = rx_stage(p.ck, RS, p.tok, sizeof(TIn)), tail = rx_tail(ET, TE, TM);
    int stages = (int)((200u * 1024u - tail) / stage);
    const int chunks = (p.C + p.ck - 1) / p.ck;
    if (stages > RX_MAX_STAGES) stages = RX_MAX_STAGES;
    if (ctas <= 148 && stages > chunks) stages = chunks;
    p.stages = stages < 2 ? 2 : stages;
    size_t smem = (size_t)p.stages * stage + tail;
    if (p.plan.top_idx && smem < sizeof(PlanShared)) smem = sizeof(PlanShared);
    static std::atomic<uint64_t> opted{0};             // devices that have the shared-memory opt-in (bit per ordinal)
    if (device >= 64 || !(opted.load(std::memory_order_relaxed) >> device & 1)) {
        MGPT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024));
        if (device < 64) opted.fetch_or(1ull << device);
    }
    MGPT_CUDA(launch_pdl(kernel, grid, RX_THREADS, smem, st, p));
    MGPT_LAUNCHED("router_exact_kernel");
    return 0;
}

// Lanes per token x experts per lane x most rows per warp, by the experts and by an SM's share of the tokens: few pairs per
// thread while an SM has few tokens (a channel's step is bound by latency), more where it is bound by issue, and as few idle
// experts as possible.  The lines lie where the forms cross, us for C=1024, BF16 tokens, by the share:
//   16 experts   16x1 8.5, 8x2 9.6 at 8; 10.9, 10.2 at 12; 8x2 33, 4x4 35 at 96; 40, 36 at 112
//   32           32x1 8.9, 16x2 9.2 at 4; 11.3, 10.9 at 8; 16x2 30, 8x4 33 at 48; 39, 34 at 64
//   64           32x2 29, 16x4 32 at 24; 40, 32 at 28
//    8           8x1 11.6, 2x4 14 at 32; 20, 16 at 40
//   20           8x3 32, 4x5 32 at 64; 49, 45 at 104; 70, 55 at 144
//   40           16x3 31, 8x5 32 at 32; 41, 39 at 46; 68, 54 at 72
//   80           32x3 29, 16x5 30 at 12; 53, 49 at 32; 120, 107 at 72
// One row has a kernel of its own for small shares: in a call whose instructions come from HBM the kernels for several rows cost
// up to 4 us more.
template <typename TIn>
int router_exact_dispatch(const RouterArgs& p, int device, cudaStream_t st)
{
    const int E = p.E, share = p.list ? 1 << 30 : (p.N + 147) / 148;
    if (E <= 8) {
        if (share <= 32) return router_exact_launch<TIn, 8, 1, 1>(p, device, st);
        if (E <= 4) return router_exact_launch<TIn, 1, 4, 2>(p, device, st);
        return router_exact_launch<TIn, 2, 4, 2>(p, device, st);
    }
    if (E <= 16) {
        if (share <= 8) return router_exact_launch<TIn, 16, 1, 1>(p, device, st);
        if (share <= (E > 12 ? 32 : 16)) return router_exact_launch<TIn, 8, 2, 1>(p, device, st);
        if (E <= 12) return router_exact_launch<TIn, 4, 3, 3>(p, device, st);
        if (share <= 96) return router_exact_launch<TIn, 8, 2, 3>(p, device, st);
        return router_exact_launch<TIn, 4, 4, 3>(p, device, st);
    }
    if (E <= 32) {
        if (share <= (E > 24 ? 8 : 4)) return router_exact_launch<TIn, 32, 1, 1>(p, device, st);
        if (share <= (E > 24 ? 16 : 8)) return router_exact_launch<TIn, 16, 2, 1>(p, device, st);
        if (E <= 20 && share > 64) return router_exact_launch<TIn, 4, 5, 3>(p, device, st);
        if (E <= 24) return router_exact_launch<TIn, 8, 3, 4>(p, device, st);
        if (share <= 48) return router_exact_launch<TIn, 16, 2, 3>(p, device, st);
        return router_exact_launch<TIn, 8, 4, 3>(p, device, st);
    }
    if (E <= 64) {
        if (share <= (E > 48 ? 8 : 4)) return router_exact_launch<TIn, 32, 2, 1>(p, device, st);
        if (E <= 40 && share > 40) return router_exact_launch<TIn, 8, 5, 3>(p, device, st);
        if (E <= 48) return router_exact_launch<TIn, 16, 3, 4>(p, device, st);
        if (share <= 24) return router_exact_launch<TIn, 32, 2, 3>(p, device, st);
        return router_exact_launch<TIn, 16, 4, 3>(p, device, st);
    }
    if (share <= (E > 96 ? 8 : 4)) return router_exact_launch<TIn, 32, 4, 1>(p, device, st);
    if (E <= 80 && share > 16) return router_exact_launch<TIn, 16, 5, 3>(p, device, st);
    if (E <= 96) return router_exact_launch<TIn, 32, 3, 4>(p, device, st);
    return router_exact_launch<TIn, 32, 4, 4>(p, device, st);
}

template <typename TIn, int EL, int EPL, int TPW>
int router_any_launch(const RouterArgs& p, cudaStream_t st)
{
    constexpr int TOK = R_WARPS * TPW * (32 / EL);
    MGPT_CUDA(launch_pdl(router_fwd_kernel<TIn, EL, EPL, TPW>, (p.N + TOK - 1) / TOK, R_WARPS * 32, 0, st, (const TIn*)p.x, p.Wr, p.br, p.N,
                         p.C, p.E, p.k, p.logits, p.probs, p.top_idx, p.top_p, p.list, p.list_count));
    MGPT_LAUNCHED("router_fwd_kernel");
    return 0;
}

// Routed rows up to which the router's last block builds the plan (with 512 or 1024 the plan's own kernel, which starts while the
// router drains, is as fast: 256 tokens, top-2, 116.4 against 116.7 us for the call).
constexpr int ROUTER_PLAN_ROWS = 256;

template <typename TIn>
int router_fwd_dispatch(const RouterArgs& p, int device, bool fast, cudaStream_t st)
{
    if (fast) return router_exact_dispatch<TIn>(p, device, st);
    if (p.E <= 32) return router_any_launch<TIn, 32, 1, 2>(p, st);
    if (p.E <= 64) return router_any_launch<TIn, 32, 2, 2>(p, st);
    return router_any_launch<TIn, 32, 4, 2>(p, st);
}

}  // namespace

// list / list_count (device): run only on the tokens list[0 .. *list_count), at most N of them.  plan / done: the last
// block builds the plan too; *planned says whether this launch does.
int launch_router_fwd(const void* x, int io, const float* Wr, const float* br, int N, int C, int E, int k,
                      float* logits, float* probs, int32_t* top_idx, float* top_p, cudaStream_t st,
                      const int32_t* list, const int32_t* list_count, int32_t* status, const PlanArgs* plan, int32_t* done, bool* planned)
{
    if (planned) *planned = false;
    if (N <= 0) return 0;
    RouterArgs p = {};
    p.x = x; p.Wr = Wr; p.br = br; p.N = N; p.C = C; p.E = E; p.k = k;
    p.logits = logits; p.probs = probs; p.top_idx = top_idx; p.top_p = top_p;
    p.list = list; p.list_count = list_count; p.status = status;
    const bool fast = C % 8 == 0 && (((uintptr_t)x | (uintptr_t)Wr) & 15) == 0;
    if (fast && plan && plan->R <= ROUTER_PLAN_ROWS) {
        p.plan = *plan;
        p.done = done;
        *planned = true;
    }
    int device = 0;
    MGPT_CUDA(cudaGetDevice(&device));
    if (io == MGPT_MOE_IO_F32) return router_fwd_dispatch<float>(p, device, fast, st);
    return router_fwd_dispatch<bf16>(p, device, fast, st);
}

template <int TPT>
static int launch_router_dx(mgpt_moe_layer* L, const void* dXg, size_t act_bytes, int io, const int32_t* pos, const float* dl,
                            const float* Wr, int N, int C, int E, int k, void* dx, cudaStream_t st)
{
    const dim3 grid((N + 32 * TPT - 1) / (32 * TPT), (C + DX_CH - 1) / DX_CH);
    const size_t sm = dx_smem<TPT>(E);
    if (!L->router_dx_attr[TPT == 4]) {             // a per-device attribute: one opt-in per layer (layers live on one device)
        const int most = (int)dx_smem<TPT>(MAX_EXPERTS);
        MGPT_CUDA(cudaFuncSetAttribute(router_dx_kernel<float, float, TPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        MGPT_CUDA(cudaFuncSetAttribute(router_dx_kernel<bf16, float, TPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        MGPT_CUDA(cudaFuncSetAttribute(router_dx_kernel<bf16, bf16, TPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        L->router_dx_attr[TPT == 4] = true;
    }
    if (act_bytes == 4)
        MGPT_CUDA(launch_pdl(router_dx_kernel<float, float, TPT>, grid, 256, sm, st, (const float*)dXg, pos, dl, Wr, N, C, E, k, (float*)dx));
    else if (io == MGPT_MOE_IO_F32)
        MGPT_CUDA(launch_pdl(router_dx_kernel<bf16, float, TPT>, grid, 256, sm, st, (const bf16*)dXg, pos, dl, Wr, N, C, E, k, (float*)dx));
    else
        MGPT_CUDA(launch_pdl(router_dx_kernel<bf16, bf16, TPT>, grid, 256, sm, st, (const bf16*)dXg, pos, dl, Wr, N, C, E, k, (bf16*)dx));
    return 0;
}

int launch_router_bwd(mgpt_moe_layer* L, const Workspace& w, char* ws, const void* x, int io,
                      void* dx, cudaStream_t st, const void* dXg_rows, const int32_t* pos_rows)
{
    const Dims& d = L->d;
    const int N = w.n_tokens, C = d.C, E = d.E, k = d.k;
    if (N <= 0) return 0;
    const float* probs = (const float*)(ws + w.probs);
    const int32_t* top_idx = (const int32_t*)(ws + w.top_idx);
    const float* dtp = (const float*)(ws + w.d_top_p);
    const int32_t* counts = (const int32_t*)(ws + w.counts);
    const int32_t* pos = pos_rows ? pos_rows : (const int32_t*)(ws + w.pos);
    const void* dXg = dXg_rows ? dXg_rows : (const void*)(ws + w.dXg);
    float* dl = (float*)(ws + w.dlogits);
    const float* Wr = L->p_data[0];
    // Tensor-core path: BF16 mode with BF16 tokens (x, dx are TMA operands); gWr rows need 16-byte pieces.
    const bool tc = d.mode == MGPT_MOE_BF16 && d.gemm_impl == 0 && io == MGPT_MOE_IO_BF16;
    const bool tc_wgrad = tc && L->has_grad && E % 4 == 0;
    const int E8 = (E + 7) / 8 * 8;
    {
        const int grid = min((N + 31) / 32, 592);
        bf16* dl16 = tc ? (bf16*)(ws + w.dl16) : nullptr;
        float* gbr = tc_wgrad ? L->p_grad[1] : nullptr;
        if (E <= 32) MGPT_CUDA(launch_pdl(router_dlogits_kernel<1>, grid, 256, 0, st, probs, top_idx, dtp, counts, N, E, k, d.alpha, dl, dl16, E8, gbr));
        else if (E <= 64) MGPT_CUDA(launch_pdl(router_dlogits_kernel<2>, grid, 256, 0, st, probs, top_idx, dtp, counts, N, E, k, d.alpha, dl, dl16, E8, gbr));
        else MGPT_CUDA(launch_pdl(router_dlogits_kernel<4>, grid, 256, 0, st, probs, top_idx, dtp, counts, N, E, k, d.alpha, dl, dl16, E8, gbr));
        MGPT_LAUNCHED("router_dlogits_kernel");
    }
    if (tc) {
        MGPT_TRY(tc_router_dx(L, w, ws, dXg, pos, dx, st));
    } else {
        const int cols = (C + DX_CH - 1) / DX_CH;
        if ((N + 127) / 128 * cols >= 2 * 148) MGPT_TRY(launch_router_dx<4>(L, dXg, w.act_bytes, io, pos, dl, Wr, N, C, E, k, dx, st));
        else MGPT_TRY(launch_router_dx<1>(L, dXg, w.act_bytes, io, pos, dl, Wr, N, C, E, k, dx, st));
        MGPT_LAUNCHED("router_dx_kernel");
    }
    if (tc_wgrad) {
        MGPT_TRY(tc_router_wgrad(L, w, ws, x, st));
    } else if (L->has_grad) {
        const int E4 = (E + 3) / 4, ch_per_cta = (256 / E4) * 4;
        const int cblocks = (C + ch_per_cta - 1) / ch_per_cta;
        float* part = (float*)(ws + w.rw_part);
        float* partb = part + (size_t)w.rw_chunks * C * E;
        const int tpc = (N + w.rw_chunks - 1) / w.rw_chunks;
        dim3 grid(cblocks, w.rw_chunks);
        if (io == MGPT_MOE_IO_F32)
            MGPT_CUDA(launch_pdl(router_wgrad_partial_kernel<float>, grid, 256, 0, st, (const float*)x, dl, N, C, E, tpc, part, partb));
        else
            MGPT_CUDA(launch_pdl(router_wgrad_partial_kernel<bf16>, grid, 256, 0, st, (const bf16*)x, dl, N, C, E, tpc, part, partb));
        MGPT_LAUNCHED("router_wgrad_partial_kernel");
        MGPT_CUDA(launch_pdl(router_wgrad_reduce_kernel, (C * E + E + 31) / 32, 256, 0, st, part, partb, w.rw_chunks, C * E, E,
                                                                      L->p_grad[0], L->p_grad[1]));
        MGPT_LAUNCHED("router_wgrad_reduce_kernel");
    }
    return 0;
}

}  // namespace mgpt
