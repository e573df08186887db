// Grouped SwiGLU expert products on the 5th-generation tensor cores.
//
// BF16 operands, FP32 accumulation in TMEM (tcgen05.mma, one issuing thread
// per CTA), operand tiles staged in shared memory by TMA (cp.async.bulk.tensor,
// 128-byte swizzle), epilogues read the accumulator with tcgen05.ld.  No
// cluster multicast is used anywhere: every CTA loads its own tiles.
//
// What the reference does with ~8 launches per expert forward and ~26 per
// expert backward (layers/MoELayer.cpp:94-118, 159-181; layers/SwiGLU.cpp:23-96;
// layers/LinearLayer.cpp:23-80) becomes seven launches for all experts:
//
//   gate/up : [G|U] = Xg * [Wg|Wu] + [bg|bu],  Hh = silu(G)*U; keeps silu(G) and dHh/dG's factor (epilogue)
//   down    : Yg = Hh * Wd + bd
//   dHh     : dHh = dYg * Wd^T -> dG, dU (SwiGLU backward in the epilogue)
//   dXg     : dXg = dG * Wg^T + dU * Wu^T       (one accumulator, K = 2H)
//   wgrad x3: gWg += Xg^T dG, gWu += Xg^T dU, gWd += Hh^T dYg   (FP32 +=)
//
// Row tiles are whole 128-row tiles of one expert (the dispatch plan pads each
// expert's segment with zero rows), so no tile mixes experts and the reduction
// over rows in the weight gradients needs no masking.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets a bit in the
// workspace status word and the CTA leaves through its normal teardown
// (TMEM is released), so a fault in a descriptor cannot hang the device.
#include "tc_common.cuh"

namespace mgpt {

namespace {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4;
constexpr uint32_t A_BYTES = BM * BK * 2;            // 16 KiB
constexpr uint32_t B_BYTES = BN * BK * 2;            // 32 KiB
constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;  // 48 KiB
constexpr uint32_t HALF_B = B_BYTES / 2;
constexpr uint32_t BOX_BYTES = 64 * BK * 2;          // one {64 MN elements, 64 reduction rows} box of an MN-major operand: 8 KiB
constexpr int EPI_WARPS = 16;                        // four per TMEM lane quarter
constexpr uint32_t STAGING_BYTES = 2048;             // per epilogue warp: 32 rows x 64 B
constexpr uint32_t TMEM_COLS = 2 * BN;               // two accumulators
constexpr uint32_t SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * STAGING_BYTES + 1024 /*align slack*/ + 512 /*barriers, work queue*/;
constexpr int TC_THREADS = 64 + 32 * EPI_WARPS;      // warp0 TMA, warp1 MMA, warps2-17 epilogue
constexpr int ROWS_THREADS = TC_THREADS + 32;        // expert products: warp 18 brings the biases
constexpr int CS_WARPS = 2;                          // weight-gradient kernel only: warps 18-19 sum operand columns (bias gradients)
constexpr int WG_THREADS = TC_THREADS + 32 * CS_WARPS;

constexpr int SCHED_Q = 8;                           // queue entries: the producer runs up to ~4 items ahead of the slowest epilogue warp

using namespace tcx;

// Two FP32 operations per instruction, on registers that lie side by side.
__device__ __forceinline__ uint64_t pk2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpk2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint32_t bf2(uint64_t v)
{
    float a, b;
    unpk2(v, a, b);
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint64_t sigmoid2(uint64_t g)
{
    float e0, e1, d0, d1;
    unpk2(mul2(g, pk2(-1.4426950408889634f, -1.4426950408889634f)), e0, e1);
    unpk2(add2(pk2(ex2(e0), ex2(e1)), pk2(1.0f, 1.0f)), d0, d1);
    return pk2(rcp(d0), rcp(d1));
}

// per half: a where x is infinite, else b
__device__ __forceinline__ uint64_t where_infinite(uint64_t x, uint64_t a, uint64_t b)
{
    float x0, x1, a0, a1, b0, b1;
    unpk2(x, x0, x1);
    unpk2(a, a0, a1);
    unpk2(b, b0, b1);
    return pk2(isinf(x0) ? a0 : b0, isinf(x1) ? a1 : b1);
}

// Shared memory of one CTA: operand ring, one 2 KiB staging tile per epilogue warp, barriers.
struct Pipe {
    uint32_t bars, tmem_slot;          // shared-space addresses
    uint8_t* tiles;
    uint8_t* staging;
    __device__ __forceinline__ uint32_t full(int s) const { return bars + 8u * s; }
    __device__ __forceinline__ uint32_t empty(int s) const { return bars + 8u * (STAGES + s); }
    __device__ __forceinline__ uint32_t acc_full(int b) const { return bars + 8u * (2 * STAGES + b); }
    __device__ __forceinline__ uint32_t acc_empty(int b) const { return bars + 8u * (2 * STAGES + 2 + b); }
    // work-item queue: slot i is full once the producer has written item(i), empty once every consumer has read it
    __device__ __forceinline__ uint32_t sched_full(int i) const { return bars + 8u * (2 * STAGES + 5 + i); }
    __device__ __forceinline__ uint32_t sched_empty(int i) const { return bars + 8u * (2 * STAGES + 5 + SCHED_Q + i); }
    __device__ __forceinline__ uint32_t sched_item(int i) const { return bars + 8u * (2 * STAGES + 5 + 2 * SCHED_Q) + 4u * i; }
};

__device__ __forceinline__ Pipe carve(uint8_t* raw)
{
    Pipe p;
    const uint32_t base = smem_u32(raw);
    const uint32_t pad = (1024u - (base & 1023u)) & 1023u;
    p.tiles = raw + pad;
    p.staging = p.tiles + STAGES * STAGE_BYTES;
    p.bars = smem_u32(p.staging + EPI_WARPS * STAGING_BYTES);
    p.tmem_slot = p.bars + 8u * (2 * STAGES + 4);
    return p;
}

// Common prologue: barriers, TMEM (both accumulators), returns the TMEM base address.
// `extra`: warps besides the MMA thread that read every operand stage and every work item (and release both).
__device__ __forceinline__ uint32_t cta_setup(const Pipe& pipe, int warp, int extra = 0)
{
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(pipe.full(s), 1);
            mbar_init(pipe.empty(s), 1 + extra);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            mbar_init(pipe.acc_full(b), 1);
            mbar_init(pipe.acc_empty(b), EPI_WARPS);
        }
#pragma unroll
        for (int i = 0; i < SCHED_Q; ++i) {
            mbar_init(pipe.sched_full(i), 1);
            mbar_init(pipe.sched_empty(i), 1 + EPI_WARPS + extra);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(pipe.tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(pipe.tmem_slot));
    return tmem_base;
}

__device__ __forceinline__ void cta_teardown(uint32_t tmem_base, int warp)
{
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---- work distribution ---------------------------------------------------------
// Items are handed out by a device-wide counter instead of a fixed stride, so a CTA that starts late (its SM
// was busy with another stream's kernel) or meets longer items simply takes fewer of them.  The producer thread
// fetches the CTA's n-th item and passes it to the MMA thread and the epilogue warps through a small queue in
// shared memory.  counter[0] = next item, counter[1] = CTAs that have finished; the last CTA to finish clears
// both, so the pair is ready for the next launch on the stream without a memset.
// The value returned by the counter is first looked at in sched_publish (item >= total: no work left, published
// as -1 so that the other roles stop at this entry too); between request and use lie an item's loads.
// A CTA's first item is its own index (no round trip before the first loads); the counter hands out the rest.
__device__ __forceinline__ int sched_fetch(int32_t* counter) { return (int)gridDim.x + atomicAdd(counter, 1); }
// Hands the CTA's n-th item to the other roles.  False: the wait for a free queue slot ran out.
__device__ __forceinline__ bool sched_publish(const Pipe& pipe, uint32_t n, int& item, int total, int32_t* status)
{
    const int slot = n % SCHED_Q;
    if (item >= total) item = -1;
    if (n >= SCHED_Q && !mbar_wait(pipe.sched_empty(slot), ((n / SCHED_Q) - 1) & 1, status, ERR_SCHED_WAIT)) return false;
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(pipe.sched_item(slot)), "r"(item) : "memory");
    mbar_arrive(pipe.sched_full(slot));
    return true;
}
// The caller reads with every thread that needs the item, then one thread per consumer calls sched_release.
__device__ __forceinline__ int sched_consume(const Pipe& pipe, uint32_t n, int32_t* status)
{
    const int slot = n % SCHED_Q;
    if (!mbar_wait(pipe.sched_full(slot), (n / SCHED_Q) & 1, status, ERR_SCHED_WAIT)) return -1;
    int item;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(item) : "r"(pipe.sched_item(slot)) : "memory");
    return item;
}
__device__ __forceinline__ void sched_release(const Pipe& pipe, uint32_t n) { mbar_arrive(pipe.sched_empty(n % SCHED_Q)); }
// Once per CTA of the grid (CTA pair: by the leader), by the producer thread after its last fetch.
__device__ __forceinline__ void sched_finish(int32_t* counter, int callers)
{
    __threadfence();
    if (atomicAdd(counter + 1, 1) == callers - 1) {
        counter[0] = 0;
        counter[1] = 0;
        __threadfence();
    }
}

// Epilogue warp -> accumulator buffer is free again (all its tcgen05.ld of this tile are done).
__device__ __forceinline__ void release_acc(uint32_t bar, int lane)
{
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// Writes this thread's row of a [32 rows x 32 bf16] tile into the warp's staging tile in the
// 64-byte swizzle a TMA store with SWIZZLE_64B expects (16-byte chunk j of row r at j ^ ((r >> 1) & 3)).
__device__ __forceinline__ void stage_row_bf16(uint8_t* stage, int lane, const uint32_t (&packed)[16])
{
    // the previous TMA store out of this tile must have finished reading it
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
    const uint32_t row = smem_u32(stage) + lane * 64;
    const uint32_t sw = ((uint32_t)lane >> 1) & 3u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t a = row + (((uint32_t)j ^ sw) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(packed[4 * j]), "r"(packed[4 * j + 1]),
                     "r"(packed[4 * j + 2]), "r"(packed[4 * j + 3]) : "memory");
    }
}
// The staged tile -> global through TMA (columns beyond the tensor are clipped by the hardware).
__device__ __forceinline__ void flush_stage(uint8_t* stage, const CUtensorMap* map, int x, int y, int lane)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        tma_store_2d(map, x, y, smem_u32(stage));
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
}
// The two saved activation-derivative arrays (buffers "G" and "U") are private to the gate/up and dHh epilogues, so they are kept in the layout
// both epilogues touch with full-width accesses: [row tile][8-column chunk][128 rows][8 bf16].  A thread owns one
// row (its TMEM lane); the 32 lanes of a warp then read or write 512 contiguous bytes per instruction.
// `chunk0` points at this thread's row in the first chunk of its 32 columns; `valid` = columns left in the tensor.
__device__ __forceinline__ void load_blocked32(const uint4* chunk0, uint32_t (&w)[16], int valid)
{
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint4 u = make_uint4(0, 0, 0, 0);
        if (q * 8 < valid)
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(chunk0 + q * BM));
        w[4 * q] = u.x; w[4 * q + 1] = u.y; w[4 * q + 2] = u.z; w[4 * q + 3] = u.w;
    }
}
// this thread's row in chunk n/8 of row tile `row_tile` (n_out columns, a multiple of 8)
__device__ __forceinline__ size_t blocked_index(int row_tile, int n_out, int n, int row_in_tile)
{
    return ((size_t)row_tile * (n_out >> 3) + (n >> 3)) * BM + row_in_tile;
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// ---- token-major products ------------------------------------------------------
enum { MODE_GATEUP = 0, MODE_DOWN = 1, MODE_DHH = 2, MODE_DXG = 3 };

__host__ __device__ constexpr int rows_groups(int mode) { return mode == MODE_DHH ? 1 : 2; }
struct RowsP {
    const int32_t* tile_expert;
    const int32_t* tile_order;  // optional: i-th row tile to work on (expert-major order over scattered tiles)
    const int32_t* n_tiles;
    int32_t* status;
    int32_t* sched;         // {next item, finished CTAs}, both zero between launches
    int kblocks;            // k-blocks (of 64) per operand pair
    int n_out;              // output columns (H or C)
    int n_col_tiles;        // column tiles per row tile
    int early;              // plan and weights were complete before the kernel before this one on the stream went past its pdl_wait
    int release;            // MODE_GATEUP: let the next kernel's CTAs in early
    bf16 *G, *U;            // P and Q (see the gate/up epilogue) in the blocked layout (written by MODE_GATEUP, read by MODE_DHH)
    const float* const* bias0;
    const float* const* bias1;
    // tc_dx_kernel only: row tiles are token tiles (no experts); the epilogue adds the expert rows of each token
    int fixed_tiles;            // number of 128-token tiles
    int n_valid_rows;           // tokens
    // The B operand of the expert products is a tile-major weight copy (common.cuh): block (expert e, row block rb, column block
    // cb) is block (e * b_row_blocks + rb) * b_col_blocks + cb of the copy.
    // MODE_GATEUP / MODE_DOWN: rows are output columns, block columns the reduction (whole blocks of 128 rows, K-major);
    // MODE_DHH / MODE_DXG: rows are the reduction, block columns output columns (half blocks of 64 rows, MN-major).
    int b_row_blocks, b_col_blocks;
    const bf16* gather_src;     // dXg rows [*, n_out]
    const int32_t* gather_pos;  // [tokens, gather_k] row of dXg for (token, j)
    int gather_k;
    bf16* dx;                   // tc_dx_kernel: the output
};

// What follows the operand ring and the staging tiles of the four expert products.
struct RowsItem {
    int row_tile, n0, e, pad;       // row_tile < 0: no work left
};
struct RowsShared {
    float bias[2][BN];              // per accumulator: the biases of its columns
    RowsItem item[SCHED_Q];
    uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], bias_full[2], item_full[SCHED_Q], item_empty[SCHED_Q];
    uint32_t tmem;
};
constexpr int ROWS_CLAIM = 4;       // the next item is claimed this many k-blocks before the last one's loads end
constexpr uint32_t ROWS_SMEM = STAGES * STAGE_BYTES + EPI_WARPS * STAGING_BYTES + sizeof(RowsShared);
static_assert(ROWS_SMEM <= 232448, "shared memory of one CTA");

// The epilogue of every second item of a CTA for one of the eight warps of its group: TMEM lane quarter q (rows q*32..+31 of
// the row tile), column half h.  `next(n, w)`: the CTA's n-th item, false: no more.
// KEEP (gate/up): a backward pass follows, which needs the saved factors; inference keeps nothing.
template <int MODE, bool KEEP, class Next>
__device__ __forceinline__ void rows_epilogue(const RowsP& p, RowsShared& sh, uint32_t tmem_base, int group, int q, int h, int lane,
                                              uint8_t* stage, const CUtensorMap* tmD0, const CUtensorMap* tmD1, Next next)
{
    const uint32_t acc_full = smem_u32(&sh.acc_full[group]), acc_empty = smem_u32(&sh.acc_empty[group]), bias_full = smem_u32(&sh.bias_full[group]);
    const uint32_t t_lane = tmem_base + group * BN + ((uint32_t)(q * 32) << 16);
    const float* bias = sh.bias[group];
    const int ld = p.n_out;
    uint32_t phase = 0;
    RowsItem w = {};
    auto store = [&](const uint32_t (&pk)[16], const CUtensorMap* tm, int n) {
        stage_row_bf16(stage, lane, pk);
        flush_stage(stage, tm, n, w.row_tile * BM + q * 32, lane);
    };
    if (MODE == MODE_GATEUP) {
        for (uint32_t t = group; next(t, w); t += 2, phase ^= 1) {
            if (!mbar_wait(acc_full, phase, p.status, ERR_ACC_WAIT)) return;
            if (!mbar_wait(bias_full, phase, p.status, ERR_ACC_WAIT)) return;
            tc_fence_after();
#pragma unroll 1
            for (int un = 0; un < 2; ++un) {
                // hidden units n0 + col .. +31: gate columns col.., up columns 128 + col..
                const int col = h * 64 + un * 32, n = w.n0 + col, valid = ld - n;
                float a[32], b[32];
                tmem_ld32(t_lane + col, a);
                tmem_ld32(t_lane + BN / 2 + col, b);
                tmem_ld_wait();
                uint64_t g2[16], u2[16];
                const float4 *b0 = reinterpret_cast<const float4*>(bias + col), *b1 = b0 + BN / 8;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 x = b0[i], y = b1[i];
                    g2[2 * i] = add2(pk2(a[4 * i], a[4 * i + 1]), pk2(x.x, x.y));
                    g2[2 * i + 1] = add2(pk2(a[4 * i + 2], a[4 * i + 3]), pk2(x.z, x.w));
                    u2[2 * i] = add2(pk2(b[4 * i], b[4 * i + 1]), pk2(y.x, y.y));
                    u2[2 * i + 1] = add2(pk2(b[4 * i + 2], b[4 * i + 3]), pk2(y.z, y.w));
                }
                if (un == 1) release_acc(acc_empty, lane);
                if (valid <= 0) continue;
                // What backward needs of G and U is not the values themselves but
                //   Q = silu(G)                       (dU = dHh * Q)
                //   P = U * sigmoid(G) * (1 + G * (1 - sigmoid(G)))      (dG = dHh * P)
                // (utils/Tensor.cpp:2020-2027), so those are what is kept: the sigmoid is evaluated once, here,
                // in FP32 on the unrounded sums, and the dHh epilogue is left with two multiplies per element.
                uint32_t hp[16];
                const size_t o = blocked_index(w.row_tile, ld, n, q * 32 + lane);
                uint4 *gp = reinterpret_cast<uint4*>(p.G) + o, *up = reinterpret_cast<uint4*>(p.U) + o;
                auto work = [&](auto infinite) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {          // 8 hidden units at a time
                        uint32_t pp[4], qp[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint64_t g = g2[4 * c + j], u = u2[4 * c + j], sig = sigmoid2(g), qv = mul2(g, sig), us = mul2(u, sig);
                            const uint64_t d = fma2(qv, pk2(-1.0f, -1.0f), g), v = fma2(us, d, us);
                            hp[4 * c + j] = bf2(mul2(qv, u));
                            qp[j] = bf2(qv);
                            pp[j] = bf2(decltype(infinite)::value ? where_infinite(us, mul2(us, add2(d, pk2(1.0f, 1.0f))), v) : v);
                        }
                        if (KEEP && c * 8 < valid) {
                            gp[c * BM] = make_uint4(pp[0], pp[1], pp[2], pp[3]);
                            up[c * BM] = make_uint4(qp[0], qp[1], qp[2], qp[3]);
                        }
                    }
                };
                if constexpr (KEEP) {
                    // us + us * (g - q) is NaN where us is infinite and g - q negative or zero.  (The sum of products is finite
                    // unless a value is not, or values are huge: 8 instructions for the 32 that a test of each took.)
                    uint64_t sum[2] = {};
#pragma unroll
                    for (int i = 0; i < 8; ++i) sum[i & 1] = fma2(u2[2 * i], u2[2 * i + 1], sum[i & 1]);
                    float s0, s1;
                    unpk2(add2(sum[0], sum[1]), s0, s1);
                    if (__builtin_expect(__any_sync(0xffffffffu, !(fabsf(s0) + fabsf(s1) < INFINITY)), 0)) work(std::true_type());
                    else work(std::false_type());
                } else {
                    work(std::false_type());
                }
                store(hp, tmD0, n);
            }
        }
    } else if (MODE == MODE_DHH) {
        // The saved factors of a 32-column unit are requested while the unit before it is worked on, an item's first ones
        // when the group is done with its item before.  (Not before a TMEM load: its wait would cover them.)
        constexpr int GROUPS = rows_groups(MODE), UNITS = 2 * GROUPS;
        const int c0 = h * 32 * UNITS;
        uint32_t P[2][16], Q[2][16];
        auto fetch = [&](int un, uint32_t (&pv)[16], uint32_t (&qv)[16]) {
            const int n = w.n0 + c0 + un * 32;
            const size_t o = blocked_index(w.row_tile, ld, n, q * 32 + lane);
            load_blocked32(reinterpret_cast<const uint4*>(p.G) + o, pv, ld - n);
            load_blocked32(reinterpret_cast<const uint4*>(p.U) + o, qv, ld - n);
        };
        bool more = next(group, w);
        if (more) fetch(0, P[0], Q[0]);
        for (uint32_t t = group; more; t += GROUPS) {
            const uint32_t buf = GROUPS == 2 ? 0 : t & 1u;
            if (!mbar_wait(acc_full + 8 * buf, (t >> 1) & 1, p.status, ERR_ACC_WAIT)) return;
            tc_fence_after();
#pragma unroll
            for (int un = 0; un < UNITS; ++un) {
                const int n = w.n0 + c0 + un * 32;
                uint32_t (&pv)[16] = P[un & 1];
                uint32_t (&qv)[16] = Q[un & 1];
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    float v[16];
                    tmem_ld16(t_lane + buf * BN + c0 + un * 32 + hf * 16, v);
                    tmem_ld_wait();
                    if (hf == 1 && un == UNITS - 1) release_acc(acc_empty + 8 * buf, lane);
                    if (hf == 1 && un < UNITS - 1) fetch(un + 1, P[(un + 1) & 1], Q[(un + 1) & 1]);
                    // utils/Tensor.cpp:2020-2027 with dd = dHh: dG = dd * P, dU = dd * Q (P, Q saved by the forward epilogue)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint64_t d = pk2(v[2 * i], v[2 * i + 1]);
                        uint32_t &pw = pv[hf * 8 + i], &qw = qv[hf * 8 + i];
                        pw = bf2(mul2(d, pk2(bf_lo(pw), bf_hi(pw))));      // dG, packed in place
                        qw = bf2(mul2(d, pk2(bf_lo(qw), bf_hi(qw))));      // dU
                    }
                }
                if (n < ld) {
                    store(pv, tmD0, n);
                    store(qv, tmD1, n);
                }
            }
            more = next(t + GROUPS, w);
            if (more) fetch(0, P[0], Q[0]);
        }
    } else {
        for (uint32_t t = group; next(t, w); t += 2, phase ^= 1) {
            if (!mbar_wait(acc_full, phase, p.status, ERR_ACC_WAIT)) return;
            if (MODE == MODE_DOWN && !mbar_wait(bias_full, phase, p.status, ERR_ACC_WAIT)) return;
            tc_fence_after();
#pragma unroll 1
            for (int un = 0; un < 4; ++un) {               // columns n0 + h*128 .. +127, four units of 32
                const int col = h * 128 + un * 32, n = w.n0 + col;
                float v[32];
                tmem_ld32(t_lane + col, v);
                tmem_ld_wait();
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint64_t x = pk2(v[4 * i], v[4 * i + 1]), y = pk2(v[4 * i + 2], v[4 * i + 3]);
                    if (MODE == MODE_DOWN) {
                        const float4 b = *reinterpret_cast<const float4*>(bias + col + 4 * i);
                        x = add2(x, pk2(b.x, b.y));
                        y = add2(y, pk2(b.z, b.w));
                    }
                    pk[2 * i] = bf2(x);
                    pk[2 * i + 1] = bf2(y);
                }
                if (un == 3) release_acc(acc_empty, lane);
                if (n < ld) store(pk, tmD0, n);
            }
        }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // stores landed before exit
}

// dx = dlogits * Wr^T (the accumulator) + the token's expert rows in ascending order: the epilogue of all of a CTA's items.
// Bound by the gather of those rows.  With a lane per token every 16-byte load touched 32 lines, one cycle of the L1 each
// (155 us for 402 MB at 32768 tokens, C=2048, top-2), with four lanes per row half of a line (144 us); so eight lanes read
// a line of 128 bytes, four rows per load (123-132 us; 50 us at E=64 and 16384 tokens, before 70).  The accumulator crosses
// to that order through `stage` (32 rows x 64 columns FP32, padded).  Each load is requested right after the registers it
// fills have been added, before the results are written, and the positions of an item while the one before it is worked on:
// that is why this mode deals its items out by stride instead of the queue.
constexpr int DX_LD = 68;                            // floats per staged row
constexpr uint32_t DX_STAGING = 32 * DX_LD * 4 + MAX_TOPK * 32 * 4;     // per epilogue warp: that tile and the positions of 32 tokens
static_assert(EPI_WARPS * DX_STAGING <= (STAGES - 1) * STAGE_BYTES + EPI_WARPS * STAGING_BYTES, "the staging of dx lies behind one stage");
__device__ __forceinline__ void dx_epilogue(const RowsP& p, const Pipe& pipe, uint32_t tmem_base, int total_items, int q, int h,
                                            int lane, float* stage)
{
    const int rsub = lane >> 3, c8 = (lane & 7) * 8, k = p.gather_k;
    bf16* __restrict__ dx = p.dx;
    int* pos = reinterpret_cast<int*>(stage + 32 * DX_LD);       // [j][token]: the item's rows, ascending in j
    int ps[MAX_TOPK];                                // rows of this lane's token
    auto positions = [&](int item) {
        const int tok = item / p.n_col_tiles * BM + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < MAX_TOPK; ++j)
            ps[j] = j < k && item < total_items && tok < p.n_valid_rows ? __ldg(p.gather_pos + (size_t)tok * k + j) : 0x7fffffff;
    };
    auto keep_positions = [&]() {
        __syncwarp();                                // the ones before have been read
#pragma unroll
        for (int a = 0; a < MAX_TOPK - 1; ++a)
            if (a < k - 1)
#pragma unroll
                for (int b = 0; b < MAX_TOPK - 1 - a; ++b)
                    if (b < k - 1 - a) {
                        const int lo = min(ps[b], ps[b + 1]);
                        ps[b + 1] = max(ps[b], ps[b + 1]);
                        ps[b] = lo;
                    }
#pragma unroll
        for (int j = 0; j < MAX_TOPK; ++j)
            if (j < k) pos[j * 32 + lane] = ps[j];
        __syncwarp();
    };
    // rows r16 + 4g + rsub, eight columns from n + c8, of the j-th expert row (0x7fffffff: no such token)
    auto fetch = [&](uint4 (&v)[4], int j, int r16, int n) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int row = pos[j * 32 + r16 + 4 * g + rsub];
            v[g] = make_uint4(0, 0, 0, 0);
            if (row != 0x7fffffff && n + c8 < p.n_out)
                v[g] = __ldg(reinterpret_cast<const uint4*>(p.gather_src + (size_t)row * p.n_out + n + c8));
        }
    };
    const int stride = gridDim.x;
    int item = blockIdx.x;
    positions(item);
    keep_positions();
    uint4 r0[4], r1[4];
    fetch(r0, 0, 0, item % p.n_col_tiles * BN + h * 64);
    if (k > 1) fetch(r1, 1, 0, item % p.n_col_tiles * BN + h * 64);
    for (uint32_t t = 0; item < total_items; ++t, item += stride) {
        const uint32_t buf = t & 1u;
        const int row_w = item / p.n_col_tiles * BM + q * 32, n = item % p.n_col_tiles * BN + h * 64;
        if (!mbar_wait(pipe.acc_full(buf), (t >> 1) & 1, p.status, ERR_ACC_WAIT)) return;
        tc_fence_after();
        __syncwarp();                                // the tile staged before has been read
#pragma unroll
        for (int un = 0; un < 2; ++un) {
            float v[32];
            tmem_ld32(tmem_base + buf * BN + ((uint32_t)(q * 32) << 16) + h * 64 + un * 32, v);
            tmem_ld_wait();
            if (un == 1) release_acc(pipe.acc_empty(buf), lane);
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(stage + lane * DX_LD + un * 32 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        __syncwarp();
#pragma unroll
        for (int r16 = 0; r16 < 32; r16 += 16) {
            if (r16) positions(item + stride);
            float s[4][8];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float* src = stage + (r16 + 4 * g + rsub) * DX_LD + c8;
                const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
                s[g][0] = a.x; s[g][1] = a.y; s[g][2] = a.z; s[g][3] = a.w; s[g][4] = b.x; s[g][5] = b.y; s[g][6] = b.z; s[g][7] = b.w;
            }
            auto add = [&](const uint4 (&r)[4]) {
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const uint32_t w[4] = {r[g].x, r[g].y, r[g].z, r[g].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        s[g][2 * i] += bf_lo(w[i]);
                        s[g][2 * i + 1] += bf_hi(w[i]);
                    }
                }
            };
            add(r0);
            if (k > 1) add(r1);
#pragma unroll
            for (int j = 2; j < MAX_TOPK; j += 2)
                if (j < k) {
                    fetch(r0, j, r16, n);
                    if (j + 1 < k) fetch(r1, j + 1, r16, n);
                    add(r0);
                    if (j + 1 < k) add(r1);
                }
            uint4 o[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    __nv_bfloat162 x = __floats2bfloat162_rn(s[g][2 * i], s[g][2 * i + 1]);
                    w[i] = *reinterpret_cast<uint32_t*>(&x);
                }
                o[g] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            // what the next half or the next item adds first
            if (r16) keep_positions();
            const int n_next = r16 ? (item + stride) % p.n_col_tiles * BN + h * 64 : n;
            fetch(r0, 0, r16 ^ 16, n_next);
            if (k > 1) fetch(r1, 1, r16 ^ 16, n_next);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int tok = row_w + r16 + 4 * g + rsub;
                if (tok < p.n_valid_rows && n + c8 < p.n_out) *reinterpret_cast<uint4*>(dx + (size_t)tok * p.n_out + n + c8) = o[g];
            }
        }
    }
}

// Persistent over items = row_tile * n_col_tiles + col_tile.  Two 256-column accumulators in TMEM alternate, so the epilogue
// of one item runs while the tensor core works on the next.
//
// The producer decodes an item once, while the loads of the one before are still going out, and hands it on through a queue; a
// warp of its own brings the biases of the item's columns into shared memory.  (Every epilogue warp used to look up the
// tile's expert, its bias pointers and then the biases, one load after another: 3000 of the 9800 cycles that an item of 8 k-blocks
// took in gate/up.)  Us for 8192 tokens, C=512, H=1376, E=16, before -> now: gate/up 73 -> 66, dHh 60 -> 54.
//
// What bounds it with few k-blocks: operands, factors and results share the way between L2 and the SM, 512 KiB an item in dHh
// against 4096 cycles of MMAs.  Ring depth counts (three stages instead of four: dXg 54 -> 62 us, gate/up of 1777 tokens 74 ->
// 78), so it is not given up for a second staging tile per epilogue warp; all results by TMA store, the factors too, from such
// tiles: no gain.  dHh's results through 16-byte stores from registers instead of TMA: 54 -> 70 us.  Its factors sent to L2
// an item ahead: 54 -> 56.  More weights sent to L2 before pdl_wait (8 or 16 k-blocks behind the ring): 120.0 -> 120.7 and
// 121.2 us for 256 tokens, C=1024, H=2816, E=32.
template <int MODE, bool KEEP = true>
__global__ void __launch_bounds__(ROWS_THREADS, 1)
tc_rows_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
               const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
               const __grid_constant__ CUtensorMap tmD0, const __grid_constant__ CUtensorMap tmD1, const RowsP p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];       // (the swizzled tiles start on 1024-byte boundaries)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int COLS_PER_ITEM = MODE == MODE_GATEUP ? BN / 2 : BN;
    constexpr int ST = STAGES;
    constexpr bool DATA_GRAD = MODE == MODE_DHH || MODE == MODE_DXG, BIAS = MODE == MODE_GATEUP || MODE == MODE_DOWN;
    const int kb_per_item = (MODE == MODE_DXG ? 2 : 1) * p.kblocks;
    RowsShared& sh = *reinterpret_cast<RowsShared*>(smem_raw + STAGES * STAGE_BYTES + EPI_WARPS * STAGING_BYTES);
    const uint32_t full = smem_u32(sh.full), empty = smem_u32(sh.empty), acc_full = smem_u32(sh.acc_full), acc_empty = smem_u32(sh.acc_empty);
    const uint32_t item_full = smem_u32(sh.item_full), item_empty = smem_u32(sh.item_empty);
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full + 8 * b, 1);
            mbar_init(acc_empty + 8 * b, (EPI_WARPS / rows_groups(MODE)));
            mbar_init(smem_u32(sh.bias_full) + 8 * b, 1);
        }
        for (int i = 0; i < SCHED_Q; ++i) {
            mbar_init(item_full + 8 * i, 1);
            mbar_init(item_empty + 8 * i, 1 + (BIAS ? 1 : 0) + (EPI_WARPS / rows_groups(MODE)));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(&sh.tmem), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = sh.tmem;
    // The setup above overlaps the end of the kernel before, and so do the producer's first loads of weights.
    if (warp > 0) {
        pdl_wait();
        if (MODE == MODE_GATEUP && p.release) pdl_release();
    }

    auto consume = [&](uint32_t n, RowsItem& w) -> bool {
        const int slot = n % SCHED_Q;
        if (!mbar_wait(item_full + 8 * slot, (n / SCHED_Q) & 1, p.status, ERR_SCHED_WAIT)) return false;
        w = sh.item[slot];
        return w.row_tile >= 0;
    };
    auto release = [&](uint32_t n) { mbar_arrive(item_empty + 8 * (n % SCHED_Q)); };

    if (warp == 0) {
        if (elect_one()) {
            int s = 0, claimed = 0;
            uint32_t free_phase = 1;                    // (the first round finds every stage free)
            bool ok = true;
            const uint32_t tile0 = smem_u32(smem_raw);
            RowsItem w = {}, next = {};
            int total_items = 0;
            auto decode = [&](int item) {               // (a CTA beyond the last item hands on "no work" and leaves through the teardown)
                next.row_tile = -1;
                if (item >= total_items) return;
                const int row_i = item / p.n_col_tiles;
                next.n0 = (item - row_i * p.n_col_tiles) * COLS_PER_ITEM;
                next.row_tile = p.tile_order ? p.tile_order[row_i] : row_i;
                next.e = p.tile_expert[next.row_tile];
            };
            auto load_b = [&](int kb, uint32_t b_dst, uint32_t bar) {
                const bool second = MODE == MODE_DXG && kb >= p.kblocks;
                const int kx = (second ? kb - p.kblocks : kb) * BK, e_rows = w.e * p.b_row_blocks;       // row blocks before this expert's
                // One load for the whole 32 KiB of B: a k-block of two loads costs the producer ~230 cycles, one of five
                // (B in 8 KiB pieces) made dXg 14 % slower
                if (MODE == MODE_GATEUP)                // gate block and up block of the same hidden units
                    tma_load_4d(b_dst, &tmB0, 0, 0, (e_rows + (w.n0 >> 7)) * p.b_col_blocks + kb, 0, bar);
                else if (MODE == MODE_DOWN)             // two row blocks
                    tma_load_4d(b_dst, &tmB0, 0, 0, kb, e_rows + (w.n0 >> 7), bar);
                else                                    // four half blocks side by side (past the last column block: columns that are not computed)
                    tma_load_3d(b_dst, second ? &tmB1 : &tmB0, 0, kx & 64, (e_rows + (kx >> 7)) * p.b_col_blocks + (w.n0 >> 6), bar);
            };
            int ahead = 0;                              // k-blocks of the first item whose B is on its way
            if (p.early) {
                total_items = *p.n_tiles * p.n_col_tiles;
                decode(blockIdx.x);
                w = next;
                if (w.row_tile >= 0)
                    for (; ahead < min(ST, kb_per_item); ++ahead) {
                        mbar_expect_tx(full + 8 * ahead, STAGE_BYTES);
                        load_b(ahead, tile0 + ahead * STAGE_BYTES + A_BYTES, full + 8 * ahead);
                    }
            }
            pdl_wait();
            if (MODE == MODE_GATEUP && p.release) pdl_release();
            if (!p.early) {
                total_items = *p.n_tiles * p.n_col_tiles;
                decode(blockIdx.x);
            }
            // the next item is claimed, then decoded, some k-blocks before this one's loads end: not earlier, or the claim would
            // sit behind this CTA's unfinished work while others run dry
            const int claim = max(0, kb_per_item - ROWS_CLAIM), look = max(0, kb_per_item - 2);
            for (uint32_t n = 0; ok; ++n) {
                const int slot = n % SCHED_Q;
                w = next;
                if (!mbar_wait(item_empty + 8 * slot, ((n / SCHED_Q) & 1) ^ 1, p.status, ERR_SCHED_WAIT)) break;
                sh.item[slot] = w;
                mbar_arrive(item_full + 8 * slot);
                if (w.row_tile < 0) {                   // one end for each group of the epilogue
                    const int after = (n + 1) % SCHED_Q;
                    if (!mbar_wait(item_empty + 8 * after, (((n + 1) / SCHED_Q) & 1) ^ 1, p.status, ERR_SCHED_WAIT)) break;
                    sh.item[after].row_tile = -1;
                    mbar_arrive(item_full + 8 * after);
                    break;
                }
                const int row0 = w.row_tile * BM;
                for (int kb = 0; kb < kb_per_item; ++kb) {
                    if (kb == claim) claimed = atomicAdd(p.sched, 1);
                    if (!mbar_wait(empty + 8 * s, free_phase, p.status, ERR_EMPTY_WAIT)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a_dst = tile0 + s * STAGE_BYTES, bar = full + 8 * s;
                    const bool second = MODE == MODE_DXG && kb >= p.kblocks, loaded = n == 0 && kb < ahead;
                    if (!loaded) mbar_expect_tx(bar, STAGE_BYTES);
                    tma_load_2d(a_dst, second ? &tmA1 : &tmA0, (second ? kb - p.kblocks : kb) * BK, row0, bar);
                    if (!loaded) load_b(kb, a_dst + A_BYTES, bar);
                    if (++s == ST) {
                        s = 0;
                        free_phase ^= 1;
                    }
                    if (kb == look) decode(gridDim.x + claimed);
                }
            }
            sched_finish(p.sched, gridDim.x);           // this CTA asks for no more items
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            const uint64_t a0 = make_desc(smem_u32(smem_raw), 16, 1024);
            // MN-major: 16 reduction rows = two 8-row groups (1 KiB each), 64-column blocks BOX_BYTES apart
            const uint64_t b0 = DATA_GRAD ? make_desc(smem_u32(smem_raw) + A_BYTES, BOX_BYTES, 1024) : make_desc(smem_u32(smem_raw) + A_BYTES, 16, 1024);
            constexpr uint32_t B_STEP = (DATA_GRAD ? 2048 : 32) >> 4;       // (the address field: 16-byte units)
            RowsItem w;
            for (uint32_t t = 0; ok && consume(t, w); ++t) {
                release(t);
                const uint32_t buf = t & 1u;
                if (!mbar_wait(acc_empty + 8 * buf, ((t >> 1) & 1) ^ 1, p.status, ERR_ACC_WAIT)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                // a narrower product where the last item of a row tile has fewer columns
                const uint32_t idesc = make_idesc(BM, DATA_GRAD ? min(BN, 64 * p.b_col_blocks - w.n0) : BN, 0, DATA_GRAD ? 1 : 0);
                for (int kb = 0; kb < kb_per_item; ++kb) {
                    if (!mbar_wait(full + 8 * s, phase, p.status, ERR_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t ad = a0 + s * (STAGE_BYTES >> 4), bd = b0 + s * (STAGE_BYTES >> 4);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_bf16(d_tmem, ad + k * (32 >> 4), bd + k * B_STEP, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit(empty + 8 * s);         // frees the stage once these MMAs have read it
                    if (++s == STAGES) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                umma_commit(acc_full + 8 * buf);        // accumulator of this item complete
            }
        }
    } else if (warp == 2 + EPI_WARPS) {
        if (BIAS && elect_one()) {
            RowsItem w;
            for (uint32_t t = 0; consume(t, w); ++t) {
                release(t);
                const uint32_t buf = t & 1u, bar = smem_u32(&sh.bias_full[buf]);
                const int cols = min(COLS_PER_ITEM, p.n_out - w.n0);
                const float *g0 = p.bias0[w.e] + w.n0, *g1 = MODE == MODE_GATEUP ? p.bias1[w.e] + w.n0 : nullptr;
                // (the epilogue has read this buffer's biases of two items ago: it arrives on acc_empty after that)
                if (!mbar_wait(acc_empty + 8 * buf, ((t >> 1) & 1) ^ 1, p.status, ERR_ACC_WAIT)) break;
                if (p.n_out >= 32) {
                    mbar_expect_tx(bar, (MODE == MODE_GATEUP ? 2 : 1) * cols * 4);
                    bulk_load(smem_u32(sh.bias[buf]), g0, cols * 4, bar);
                    if (MODE == MODE_GATEUP) bulk_load(smem_u32(sh.bias[buf] + BN / 2), g1, cols * 4, bar);
                } else {                                // (fewer may start anywhere)
                    for (int i = 0; i < cols; ++i) {
                        sh.bias[buf][i] = g0[i];
                        if (MODE == MODE_GATEUP) sh.bias[buf][BN / 2 + i] = g1[i];
                    }
                    mbar_arrive(bar);
                }
            }
        }
    } else {
        // 16 epilogue warps in two groups, one per accumulator, so that one group computes while the other one's stores drain:
        // TMEM lane quarter q = warp % 4, column half h
        constexpr int PER = EPI_WARPS / rows_groups(MODE);
        const int i = warp - 2;
        rows_epilogue<MODE, KEEP>(p, sh, tmem_base, i / PER, warp & 3, i % PER / 4, lane, smem_raw + STAGES * STAGE_BYTES + i * STAGING_BYTES, &tmD0, &tmD1,
                            [&](uint32_t n, RowsItem& w) -> bool {
                                const bool more = __any_sync(0xffffffffu, consume(n, w));       // (warp-uniform)
                                if (more && lane == 0) release(n);
                                return more;
                            });
    }
    cta_teardown(tmem_base, warp);
}

// dx: dlogits * Wr^T, an item of one or two k-blocks; one stage, and the epilogue's staging lies where the others would.
// Its items are all alike: by stride, no queue.
__global__ void __launch_bounds__(TC_THREADS, 1)
tc_dx_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const RowsP p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Pipe pipe = carve(smem_raw);
    const uint32_t tmem_base = cta_setup(pipe, warp);
    pdl_wait();
    const int total_items = p.fixed_tiles * p.n_col_tiles;
    if (warp == 0) {
        if (elect_one()) {
            uint32_t it = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
                const int row0 = item / p.n_col_tiles * BM, n0 = item % p.n_col_tiles * BN;
                for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
                    if (it >= 1 && !mbar_wait(pipe.empty(0), (it - 1) & 1, p.status, ERR_EMPTY_WAIT)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a_dst = smem_u32(pipe.tiles), b_dst = a_dst + A_BYTES;
                    mbar_expect_tx(pipe.full(0), STAGE_BYTES);
                    tma_load_2d(a_dst, &tmA, kb * BK, row0, pipe.full(0));
                    tma_load_2d(b_dst, &tmB, kb * BK, n0, pipe.full(0));
                    tma_load_2d(b_dst + HALF_B, &tmB, kb * BK, n0 + BN / 2, pipe.full(0));
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            uint32_t it = 0, t = 0;
            bool ok = true;
            for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x, ++t) {
                const uint32_t buf = t & 1u;
                if (t >= 2 && !mbar_wait(pipe.acc_empty(buf), ((t >> 1) - 1) & 1, p.status, ERR_ACC_WAIT)) break;
                tc_fence_after();
                for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
                    if (!mbar_wait(pipe.full(0), it & 1, p.status, ERR_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(pipe.tiles), b_addr = a_addr + A_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_bf16(tmem_base + buf * BN, make_desc(a_addr + k * 32, 16, 1024), make_desc(b_addr + k * 32, 16, 1024),
                                  make_idesc(BM, BN, 0, 0), (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit(pipe.empty(0));
                }
                umma_commit(pipe.acc_full(buf));
            }
        }
    } else {
        dx_epilogue(p, pipe, tmem_base, total_items, warp & 3, (warp - 2) >> 2, lane,
                    reinterpret_cast<float*>(pipe.tiles + STAGE_BYTES + (warp - 2) * DX_STAGING));
    }
    cta_teardown(tmem_base, warp);
}

// ---- weight gradients: grad[e][M,N] += A_e^T * B_e over the expert's rows ---------
// One weight-gradient problem: grad[e][M,N] += A_e^T * B_e over the rows of "expert" e.
struct WgradProb {
    float* const* grad;     // per-expert output [M,N]
    float* single_grad;     // or one output all chunks add into (router gradient)
    int M, N, n_tiles_m, n_tiles_n;
    int n_groups;           // experts, or uniform token chunks
    int uniform_rows;       // > 0: group g covers rows [g*uniform_rows, +uniform_rows) instead of an expert's rows
    int item_begin;         // first item index of this problem
    int transposed;         // the tile is grad^T: element (m, n) of the product belongs at grad[n*M + m]
};
struct WgradP {
    const int32_t* padded_offsets;
    const int32_t* seg;     // [E][n_seg][2] {first row, rows}: an expert's rows in n_seg segments (0 = one padded range)
    int n_seg;
    int32_t* status;
    int32_t* sched;         // {next item, finished CTAs}, both zero between launches
    WgradProb prob[3];
    int n_probs, total_items;
    int overwrite;          // grad = product (zeros for experts without rows) instead of grad += product
    int block_loads;        // the tensor maps are the column-block form: one load per operand tile and stage
    int b_boxes;            // > 0: B has no more than this many 64-column boxes, loaded one by one (block_loads: A's form only)
    // bias gradients from the same operand tiles (null: none): gb[pr][e][col] += column sums, over the expert's
    // rows, of the operand of problem pr whose columns are that bias's (the A operand when the problem is
    // computed transposed, else the B operand)
    float* const* gb[3];
};
struct WgradItem {
    int pr, e, m0, n0, r0, nkb;
};
__device__ __forceinline__ WgradItem wgrad_item(const WgradP& p, int item)
{
    WgradItem w;
    w.pr = (p.n_probs > 2 && item >= p.prob[2].item_begin) ? 2 : (p.n_probs > 1 && item >= p.prob[1].item_begin) ? 1 : 0;
    const WgradProb& q = p.prob[w.pr];
    const int local = item - q.item_begin, per = q.n_tiles_m * q.n_tiles_n;
    w.e = local / per;
    const int r = local % per;
    w.m0 = (r / q.n_tiles_n) * BM;
    w.n0 = (r % q.n_tiles_n) * BN;
    if (q.uniform_rows) {
        w.r0 = w.e * q.uniform_rows;
        w.nkb = q.uniform_rows / BK;
    } else if (p.n_seg > 0) {
        w.r0 = 0;
        w.nkb = 0;
        for (int sg = 0; sg < p.n_seg; ++sg) w.nkb += p.seg[(w.e * p.n_seg + sg) * 2 + 1] / BK;
    } else {
        w.r0 = p.padded_offsets[w.e];
        w.nkb = (p.padded_offsets[w.e + 1] - w.r0) / BK;
    }
    return w;
}

// Persistent over items (problem, expert, m tile, n tile); experts without rows are skipped.
__global__ void __launch_bounds__(WG_THREADS, 1)
tc_wgrad_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0,
                const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1,
                const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2, const WgradP p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total_items = p.total_items;
    const Pipe pipe = carve(smem_raw);
    const uint32_t tmem_base = cta_setup(pipe, warp, CS_WARPS);
    pdl_wait();
    constexpr uint32_t BOX = BOX_BYTES;

    if (warp == 0) {
        if (elect_one()) {
            uint32_t it = 0;
            bool ok = true;
            int item = blockIdx.x;
            ok = sched_publish(pipe, 0, item, total_items, p.status);
            for (uint32_t nf = 1; ok && item >= 0; ++nf) {
                const WgradItem w = wgrad_item(p, item);
                const CUtensorMap* mA = w.pr == 0 ? &tmA0 : w.pr == 1 ? &tmA1 : &tmA2;
                const CUtensorMap* mB = w.pr == 0 ? &tmB0 : w.pr == 1 ? &tmB1 : &tmB2;
                const bool segmented = p.n_seg > 0 && !p.prob[w.pr].uniform_rows;
                const int nseg = segmented ? p.n_seg : 1;
                for (int sg = 0; sg < nseg && ok; ++sg) {
                    const int seg_r0 = segmented ? p.seg[(w.e * p.n_seg + sg) * 2] : w.r0;
                    const int seg_kb = segmented ? p.seg[(w.e * p.n_seg + sg) * 2 + 1] / BK : w.nkb;
                    for (int kb = 0; kb < seg_kb; ++kb, ++it) {
                        const int s = it % STAGES;
                        if (it >= STAGES && !mbar_wait(pipe.empty(s), ((it / STAGES) - 1) & 1, p.status, ERR_EMPTY_WAIT)) {
                            ok = false;
                            break;
                        }
                        const uint32_t a_dst = smem_u32(pipe.tiles + s * STAGE_BYTES), b_dst = a_dst + A_BYTES;
                        const int row = seg_r0 + kb * BK;
                        if (p.b_boxes > 0) {
                            mbar_expect_tx(pipe.full(s), A_BYTES + p.b_boxes * BOX);
                            if (p.block_loads) tma_load_3d(a_dst, mA, 0, row, w.m0 / 64, pipe.full(s));
                            else
                                for (int i = 0; i < BM / 64; ++i) tma_load_2d(a_dst + i * BOX, mA, w.m0 + 64 * i, row, pipe.full(s));
                            for (int i = 0; i < p.b_boxes; ++i) tma_load_2d(b_dst + i * BOX, mB, 64 * i, row, pipe.full(s));
                            continue;
                        }
                        mbar_expect_tx(pipe.full(s), STAGE_BYTES);
                        if (p.block_loads) {
                            // two loads per stage instead of six: with 64-row stages this kernel waits for the
                            // producer thread's issue rate as much as for the bytes (measured: 1.44 -> 1.39 ms)
                            tma_load_3d(a_dst, mA, 0, row, w.m0 / 64, pipe.full(s));
                            tma_load_3d(b_dst, mB, 0, row, w.n0 / 64, pipe.full(s));
                            continue;
                        }
#pragma unroll
                        for (int i = 0; i < BM / 64; ++i) tma_load_2d(a_dst + i * BOX, mA, w.m0 + 64 * i, row, pipe.full(s));
#pragma unroll
                        for (int i = 0; i < BN / 64; ++i) tma_load_2d(b_dst + i * BOX, mB, w.n0 + 64 * i, row, pipe.full(s));
                    }
                }
                // the next item is claimed as late as possible (the ring is full by now, so the round trip to the
                // counter does not starve the tensor core): early claims would sit behind this CTA's unfinished work
                int next = sched_fetch(p.sched);
                if (ok) ok = sched_publish(pipe, nf, next, total_items, p.status);
                item = next;
            }
            sched_finish(p.sched, gridDim.x);            // this CTA asks for no more items
        }
    } else if (warp == 1) {
        if (elect_one()) {
            uint32_t it = 0, t = 0;
            bool ok = true;
            for (uint32_t nf = 0; ok; ++nf) {
                const int item = sched_consume(pipe, nf, p.status);
                if (item < 0) break;
                sched_release(pipe, nf);
                const WgradItem w = wgrad_item(p, item);
                if (w.nkb <= 0) continue;
                // no more 64-column boxes than the product has
                const uint32_t idesc = make_idesc(BM, min(BN, (p.prob[w.pr].N - w.n0 + 63) / 64 * 64), 1, 1);
                const uint32_t buf = t & 1u;
                if (t >= 2 && !mbar_wait(pipe.acc_empty(buf), ((t >> 1) - 1) & 1, p.status, ERR_ACC_WAIT)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int kb = 0; kb < w.nkb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(pipe.full(s), (it / STAGES) & 1, p.status, ERR_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(pipe.tiles + s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        // 16 reduction rows = two 8-row groups (1 KiB each); 64-element MN blocks are BOX apart
                        const uint64_t ad = make_desc(a_addr + k * 2048, BOX, 1024);
                        const uint64_t bd = make_desc(b_addr + k * 2048, BOX, 1024);
                        umma_bf16(d_tmem, ad, bd, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit(pipe.empty(s));
                }
                umma_commit(pipe.acc_full(buf));
                ++t;
            }
        }
    } else if (warp >= 2 + EPI_WARPS) {
        // Column sums of an operand over the expert's rows = a bias gradient (layers/LinearLayer.cpp:56-57).  The tiles
        // are in shared memory anyway, so these two warps add rows up while the tensor core works on the same stage.
        // The operand tile whose columns are the bias's is made of 64-column boxes, and it is loaded once per tile of
        // the OTHER output dimension: box b is summed by the item whose other-dimension tile index is b modulo the
        // number of such tiles, so the work is spread over items (at most two boxes each; the host falls back to a
        // separate kernel for shapes where that does not cover every box).  The two warps split a box's 64 rows.
        // They take part in every stage and every item (fixed barrier counts), summing or not.
        const int cw = warp - (2 + EPI_WARPS);
        const int c8 = lane & 7, rg = lane >> 3;           // 16-byte piece of a 128-byte row; rows rg + 4i
        uint32_t it = 0;
        bool ok = true;
        for (uint32_t nf = 0; ok; ++nf) {
            const int item = __shfl_sync(0xffffffffu, sched_consume(pipe, nf, p.status), 0);
            if (item < 0) break;
            if (lane == 0) sched_release(pipe, nf);
            const WgradItem w = wgrad_item(p, item);
            if (w.nkb <= 0) continue;
            const WgradProb& pb = p.prob[w.pr];
            float* const* gbt = p.gb[w.pr];
            // boxes of the operand tile, tiles of the other dimension, this item's index among them
            const int nbox = pb.transposed ? BM / 64 : BN / 64;
            const int other_tiles = pb.transposed ? pb.n_tiles_n : pb.n_tiles_m;
            const int other = pb.transposed ? w.n0 / BN : w.m0 / BM;
            int box0 = -1, box1 = -1;                       // the (at most two) boxes this item sums
            if (gbt) {
                if (other < nbox) box0 = other;
                if (other + other_tiles < nbox) box1 = other + other_tiles;
            }
            float acc[2][8];
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[b][i] = 0.0f;
            for (int kb = 0; kb < w.nkb; ++kb, ++it) {
                const int s = it % STAGES;
                if (!mbar_wait(pipe.full(s), (it / STAGES) & 1, p.status, ERR_FULL_WAIT)) {
                    ok = false;
                    break;
                }
                if (box0 >= 0) {
                    const uint32_t tile = smem_u32(pipe.tiles + s * STAGE_BYTES) + (pb.transposed ? 0 : A_BYTES);
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const int bx = b ? box1 : box0;
                        if (bx >= 0) {
                            const uint32_t box = tile + (uint32_t)bx * BOX;
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const uint32_t r = (uint32_t)(rg + 32 * cw + 4 * i);
                                uint32_t w0, w1, w2, w3;
                                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                                             : "=r"(w0), "=r"(w1), "=r"(w2), "=r"(w3)
                                             : "r"(box + r * 128u + ((((uint32_t)c8) ^ (r & 7u)) << 4)));
                                acc[b][0] += bf_lo(w0); acc[b][1] += bf_hi(w0); acc[b][2] += bf_lo(w1); acc[b][3] += bf_hi(w1);
                                acc[b][4] += bf_lo(w2); acc[b][5] += bf_hi(w2); acc[b][6] += bf_lo(w3); acc[b][7] += bf_hi(w3);
                            }
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(pipe.empty(s));
            }
            if (box0 >= 0 && ok) {
                float* gbe = gbt[w.e];
                const int limit = pb.transposed ? pb.M : pb.N;
                const int col0 = pb.transposed ? w.m0 : w.n0;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int bx = b ? box1 : box0;
                    if (bx >= 0) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float v = acc[b][i];
                            v += __shfl_xor_sync(0xffffffffu, v, 8);
                            v += __shfl_xor_sync(0xffffffffu, v, 16);
                            const int col = col0 + bx * 64 + c8 * 8 + i;
                            if (rg == 0 && col < limit) atomicAdd(gbe + col, v);      // two partial sums per column: one per warp
                        }
                    }
                }
            }
        }
    } else {
        const int q = warp & 3, h = (warp - 2) >> 2;
        float* stage = reinterpret_cast<float*>(pipe.staging + (warp - 2) * STAGING_BYTES);   // [32 rows][16 floats]
        uint32_t t = 0;
        for (uint32_t nf = 0;; ++nf) {
            const int item = __shfl_sync(0xffffffffu, sched_consume(pipe, nf, p.status), 0);  // warp-uniform
            if (item < 0) break;
            if (lane == 0) sched_release(pipe, nf);
            const WgradItem w = wgrad_item(p, item);
            const WgradProb& pb = p.prob[w.pr];
            float* g = pb.single_grad ? pb.single_grad : pb.grad[w.e];
            const int M = pb.M, N = pb.N;
            const int m_w = w.m0 + q * 32;             // first product row of this warp
            const int n_w = w.n0 + h * 64;             // first product column of this warp
            if (w.nkb <= 0) {
                // an expert without rows: nothing to add; when gradients are overwritten its tile is zeros
                if (p.overwrite) {
                    const int m = m_w + lane;
                    if (pb.transposed) {
                        for (int j = 0; j < 64; ++j)
                            if (m < M && n_w + j < N) g[(size_t)(n_w + j) * M + m] = 0.0f;
                    } else {
                        for (int r = 0; r < 32; ++r)
                            for (int j = lane; j < 64; j += 32)
                                if (m_w + r < M && n_w + j < N) g[(size_t)(m_w + r) * N + n_w + j] = 0.0f;
                    }
                }
                continue;
            }
            const uint32_t buf = t & 1u;
            if (!mbar_wait(pipe.acc_full(buf), (t >> 1) & 1, p.status, ERR_ACC_WAIT)) break;
            tc_fence_after();
            const uint32_t t_lane = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16) + h * 64;
            float v[2][32];
            tmem_ld32(t_lane, v[0]);
            tmem_ld32(t_lane + 32, v[1]);
            tmem_ld_wait();
            release_acc(pipe.acc_empty(buf), lane);
            if (pb.transposed) {
                // this thread's product row m is a COLUMN of grad: for one register the 32 lanes cover 32
                // consecutive floats of one grad row, so every scalar instruction is one full 128-byte line
                const int m = m_w + lane;
                if (m < M) {
                    float* gm = g + m;
#pragma unroll
                    for (int j = 0; j < 64; ++j) {
                        const int n = n_w + j;
                        if (n < N) {
                            if (p.overwrite) gm[(size_t)n * M] = v[j >> 5][j & 31];
                            else red_add(gm + (size_t)n * M, v[j >> 5][j & 31]);
                        }
                    }
                }
                ++t;
                continue;
            }
            const uint32_t sw_w = ((uint32_t)lane >> 1) & 3u;            // writer: row = lane
            const int sub = lane >> 2, piece = lane & 3;                 // reader: 8 rows x 4 pieces per pass
#pragma unroll
            for (int c = 0; c < 4; ++c) {                                // four groups of 16 columns
                const int n = n_w + c * 16;
                if (n >= N) break;
                // transpose through shared memory (16-byte pieces, XOR-swizzled by row) so that one vector
                // RED instruction covers eight full 64-byte row segments
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int s0 = (c & 1) * 16 + 4 * j;
                    *reinterpret_cast<float4*>(&stage[lane * 16 + (((uint32_t)j ^ sw_w) << 2)]) =
                        make_float4(v[c >> 1][s0], v[c >> 1][s0 + 1], v[c >> 1][s0 + 2], v[c >> 1][s0 + 3]);
                }
                __syncwarp();
                const int col = n + piece * 4;
#pragma unroll
                for (int rr = 0; rr < 4; ++rr) {
                    const int row = rr * 8 + sub, m = m_w + row;
                    const float4 x = *reinterpret_cast<const float4*>(
                        &stage[row * 16 + (((uint32_t)piece ^ (((uint32_t)row >> 1) & 3u)) << 2)]);
                    if (m < M && col < N) {
                        if (p.overwrite) *reinterpret_cast<float4*>(g + (size_t)m * N + col) = x;
                        else red_add_v4(g + (size_t)m * N + col, x);
                    }
                }
                __syncwarp();
            }
            ++t;
        }
    }
    cta_teardown(tmem_base, warp);
}

// ---- the three weight gradients on CTA pairs ---------------------------------------
// A cluster of two CTAs computes 256 x 256 of a gradient: each CTA loads 128 of the 256 columns of both operands (32 KiB
// per 64 rows instead of the 48 KiB of a 128 x 256 tile alone), the leader issues tcgen05.mma.cta_group::2, and each
// CTA writes back the 128 rows whose sums lie in its TMEM.
//
// All three are computed transposed, with the gradient's contiguous dimension on the M side, so that the 32 lanes of a
// TMEM row group are one line of the gradient:
//   gWg, gWu [C,H]: M = H, N = C.  They share B (Xg), so their 128-column tiles are paired across the two: 2 ceil(H/128)
//                   tiles, never an odd one.
//   gWd [H,C]     : M = C, N = H.
// A last column tile of 128 or less is an MMA of N = 128.
//
// Items are numbered expert by expert, most rows first: the longest items start first (a skewed routing's crowded expert
// used to be the tail of every problem), and an expert's rows are read for all three at about the same time.  Experts
// without rows have items only where gradients are stored instead of added to (zeros).
//
// The leader's producer takes an item and passes it to the peer's; each decodes it once and hands its own CTA's
// roles what they need, pointers from tables in shared memory.  (Decoded by every warp, with loads from global memory that
// queue behind the reductions, an item cost 6.7 us however few rows it had: 793 us where gradients of 64 experts, C=2048,
// H=1408, are stored, now 498.)
//
// Bound by the sums: 128 KiB of `+=` per CTA and item, which the memory takes at 2.6 TB/s whatever sends them (reductions
// of 4 or 16 bytes, bulk reductions; read-add-write is faster alone, 3.0, and slower here), so 0.85 ms for 64 experts,
// C=2048, H=1408, whose MMAs take 0.7 ms at 1.9 GHz.  Against the kernel above, us, gradients added / stored:
//   rows per expert          256          512          768          1024         2048
//   C=2048 H=1408 E=64   828/600      988/793      1262/1062    1498/1263      .          tc_wgrad_kernel
//                        873/609      953/770      1087/911     1322/1126      .          this one
//   C=1024 H=1408 E=32   218/150      247/195      297/250      340/304      547/512
//                        226/158      242/191      275/232      308/275      492/457
//   C= 512 H=1376 E=16    64/52        72/62        84/76        97/91       148/140
//                         68/52        74/64        84/74        95/84       136/127
//   C=1024 H= 512 E=64   166/121      189/162      228/201      263/240        .
//                        172/125      191/152      211/181      236/207        .
// Few rows leave nothing for a pair to save, and its CTAs wait for one another; hence the line at 512 (pair_wgrad_usable).
// The line is drawn for evenly spread rows.  Where a few experts take most rows pairs are faster on both sides of it, for their
// longest items come first; the step, this kernel / the other one: C=2048 H=1408 E=64 256 rows on average 979/1061, 768
// 2412/2475; C=1024 H=1408 E=32 512 495/513, 768 678/706; C=512 H=1376 E=16 512 184/193, 768 248/256.
//
// The bias gradients are column sums of the A tiles.  Two warps of the LEADER add them up (the peer has no barrier that
// says when its tiles are there: all bytes are counted on the leader's); the pair swaps its two A tiles from one column
// tile to the next, so that the leader has each of them in turn.
struct PairWgradP {
    const int32_t* padded_offsets;
    const int32_t* seg;     // as in WgradP
    int n_seg;
    int32_t *status, *sched;
    int C, H, E;
    float* const* grad[3];  // gWg, gWu, gWd per expert
    float* const* gb[3];
    int overwrite;
    int c_blocks;           // the maps of Xg and dYg are the column-block form (C a multiple of 64)
};
constexpr int WP_STAGES = 6;
constexpr uint32_t WP_STAGE = 2 * A_BYTES;
constexpr int WP_CLAIM = 6;                     // the next item is claimed this many stages before the last one's loads end
struct PairWgradItem {      // one CTA's share of an item
    float* g;               // its first element of the gradient
    float* gb;              // bias gradient of its first column
    int M, rows, cols;      // leading dimension of the gradient; rows and columns from g to its end
    int nkb, half;          // 64-row blocks of the reduction; columns of B per CTA
    int sum;                // leader: which of the A tile's two 64-column boxes to add up (bits)
};
static_assert(sizeof(PairWgradItem) == 40, "read in 8-byte pieces");
struct PairWgradShared {
    PairWgradItem item[SCHED_Q];
    float* grad[3][MAX_EXPERTS];
    float* gb[3][MAX_EXPERTS];
    int rows[MAX_EXPERTS], row0[MAX_EXPERTS];
    int order[MAX_EXPERTS];                     // experts, most rows first
    int passed[SCHED_Q];                        // peer: items from the leader
    uint64_t full[WP_STAGES], empty[WP_STAGES], acc_full[2], acc_empty[2];
    uint64_t item_full[SCHED_Q], item_empty[SCHED_Q], passed_full[SCHED_Q], passed_empty[SCHED_Q];
    uint32_t tmem;
};
constexpr uint32_t WP_SMEM = WP_STAGES * WP_STAGE + 1024 + sizeof(PairWgradShared);
static_assert(WP_SMEM <= 232448, "shared memory of one CTA");
// Rows per expert on average from which pairs are the faster form (table above); both widths need two column tiles, over
// which a bias gradient is summed.
inline bool pair_wgrad_usable(const Dims& d, int R) { return d.C > BN && d.H > BN && R >= 512 * d.E; }
__host__ __device__ inline int pair_wgrad_items(int C, int H)       // of one expert
{
    const int mh = (H + BM - 1) / BM, mc = (C + BM - 1) / BM;
    return mh * ((C + BN - 1) / BN) + (mc + 1) / 2 * ((H + BN - 1) / BN);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WG_THREADS, 1)
tc_wgrad_pair_kernel(const __grid_constant__ CUtensorMap tmXg, const __grid_constant__ CUtensorMap tmdYg,
                     const __grid_constant__ CUtensorMap tmdG, const __grid_constant__ CUtensorMap tmdU,
                     const __grid_constant__ CUtensorMap tmHh, const PairWgradP p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    uint8_t* const tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    PairWgradShared& sh = *reinterpret_cast<PairWgradShared*>(tiles + WP_STAGES * WP_STAGE);
    const uint32_t full = smem_u32(sh.full), empty = smem_u32(sh.empty), acc_full = smem_u32(sh.acc_full), acc_empty = smem_u32(sh.acc_empty);
    const uint32_t item_full = smem_u32(sh.item_full), item_empty = smem_u32(sh.item_empty);
    const uint32_t passed_full = smem_u32(sh.passed_full), passed_empty = smem_u32(sh.passed_empty);
    if (threadIdx.x == 0) {
        for (int s = 0; s < WP_STAGES; ++s) {
            mbar_init(full + 8 * s, 1);                     // (the leader's; the peer's loads count on it too)
            mbar_init(empty + 8 * s, rank == 0 ? 1 + CS_WARPS : 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full + 8 * b, 1);
            mbar_init(acc_empty + 8 * b, 2 * EPI_WARPS);
        }
        for (int i = 0; i < SCHED_Q; ++i) {
            mbar_init(item_full + 8 * i, 1);
            mbar_init(item_empty + 8 * i, rank == 0 ? EPI_WARPS + 1 + CS_WARPS : EPI_WARPS);
            mbar_init(passed_full + 8 * i, 1);
            mbar_init(passed_empty + 8 * i, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(smem_u32(&sh.tmem), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                         // the peer's barriers exist before anything is sent to them
    tc_fence_after();
    const uint32_t tmem_base = sh.tmem;
    pdl_wait();
    int mine = 0;
    if (threadIdx.x < p.E) {
        const int e = threadIdx.x;
        sh.row0[e] = p.n_seg > 0 ? 0 : p.padded_offsets[e];
        if (p.n_seg > 0)
            for (int i = 0; i < p.n_seg; ++i) mine += p.seg[(e * p.n_seg + i) * 2 + 1];
        else
            mine = p.padded_offsets[e + 1] - sh.row0[e];
        sh.rows[e] = mine;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            sh.grad[i][e] = p.grad[i][e];
            sh.gb[i][e] = p.gb[i][e];
        }
    }
    const int busy = __syncthreads_count(mine > 0);
    if (threadIdx.x < p.E) {
        int before = 0;
        for (int e = 0; e < p.E; ++e) before += sh.rows[e] > mine || (sh.rows[e] == mine && e < (int)threadIdx.x);
        sh.order[before] = threadIdx.x;
    }
    __syncthreads();

    // the CTA's n-th item; false: no more
    auto consume = [&](uint32_t n, PairWgradItem& w) -> bool {
        const int slot = n % SCHED_Q;
        if (!mbar_wait(item_full + 8 * slot, (n / SCHED_Q) & 1, p.status, ERR_SCHED_WAIT)) return false;
        w = sh.item[slot];
        return w.nkb >= 0;
    };
    auto release = [&](uint32_t n) { mbar_arrive(item_empty + 8 * (n % SCHED_Q)); };

    if (warp == 0) {
        if (elect_one()) {
            const int mh = (p.H + BM - 1) / BM, nc = (p.C + BN - 1) / BN, nh = (p.H + BN - 1) / BN, per = pair_wgrad_items(p.C, p.H);
            const int total_items = (p.overwrite ? p.E : busy) * per, grid = gridDim.x >> 1;
            int s = 0, item = blockIdx.x >> 1, next = 0;
            uint32_t free_phase = 1;                        // (the first round finds every stage free)
            const uint32_t lead_full = mapa(full, 0), tile0 = smem_u32(tiles);
            const uint32_t peer_passed = mapa(smem_u32(sh.passed), 1), peer_passed_full = mapa(passed_full, 1), lead_passed_empty = mapa(passed_empty, 0);
            for (uint32_t n = 0;; ++n) {
                const int slot = n % SCHED_Q;
                const uint32_t round = (n / SCHED_Q) & 1;
                if (rank == 0) {
                    if (item >= total_items) item = -1;
                    if (!mbar_wait_cluster(passed_empty + 8 * slot, round ^ 1, p.status, ERR_SCHED_WAIT)) break;
                    st_cluster_u32(peer_passed + 4 * slot, (uint32_t)item);
                    mbar_arrive_cluster(peer_passed_full + 8 * slot);       // (release at cluster scope: the item is visible)
                } else {
                    if (!mbar_wait_cluster(passed_full + 8 * slot, round, p.status, ERR_SCHED_WAIT)) break;
                    item = sh.passed[slot];
                    mbar_arrive_cluster(lead_passed_empty + 8 * slot);
                }
                if (!mbar_wait(item_empty + 8 * slot, round ^ 1, p.status, ERR_SCHED_WAIT)) break;
                PairWgradItem& w = sh.item[slot];
                if (item < 0) {
                    w.nkb = -1;
                    mbar_arrive(item_full + 8 * slot);
                    break;
                }
                const int e = sh.order[item / per];
                int r = item % per;
                const bool down = r >= mh * nc;
                if (down) r -= mh * nc;
                const int others = down ? nh : nc, other = r % others, M = down ? p.C : p.H, N = down ? p.H : p.C;
                int tile = r / others * 2 + ((other & 1) ^ rank);
                const int mat = down ? 2 : tile >= mh ? 1 : 0;
                if (mat == 1) tile -= mh;
                const int m0 = tile * BM, n0 = other * BN, half = N - n0 <= BN / 2 ? BN / 4 : BN / 2, nkb = sh.rows[e] / BK;
                // the leader has this A tile in every second column tile: of these visits the first sums the tile's first 64
                // columns and the second the other 64, or one visit both
                const int visit = other >> 1, visits = (others - (other & 1) + 1) >> 1;
                w.g = sh.grad[mat][e] + (size_t)n0 * M + m0;
                w.gb = sh.gb[mat][e] + m0;
                w.M = M; w.rows = N - n0; w.cols = M - m0; w.nkb = nkb; w.half = half;
                w.sum = visits > 1 ? (visit == 0 ? 1 : visit == 1 ? 2 : 0) : 3;
                mbar_arrive(item_full + 8 * slot);
                // this CTA's loads; the leader arms its barrier with both CTAs' bytes
                const CUtensorMap *mA = down ? &tmdYg : mat ? &tmdU : &tmdG, *mB = down ? &tmHh : &tmXg;
                const int colB = n0 + rank * half;
                const bool a_blocks = !down || p.c_blocks, b_blocks = down || p.c_blocks;
                int left = nkb;
                if (rank == 0 && left <= WP_CLAIM) next = atomicAdd(p.sched, 1);
                bool ok = true;
                for (int sg = 0; ok && sg < (p.n_seg > 0 ? p.n_seg : 1); ++sg) {
                    int row = sh.row0[e], end = row + sh.rows[e];
                    if (p.n_seg > 0) {
                        row = p.seg[(e * p.n_seg + sg) * 2];
                        end = row + p.seg[(e * p.n_seg + sg) * 2 + 1];
                    }
                    for (; row < end; row += BK, --left) {
                        if (rank == 0 && left == WP_CLAIM + 1) next = atomicAdd(p.sched, 1);
                        if (!mbar_wait_cluster(empty + 8 * s, free_phase, p.status, ERR_EMPTY_WAIT)) {
                            ok = false;
                            break;
                        }
                        const uint32_t a_dst = tile0 + s * WP_STAGE, b_dst = a_dst + A_BYTES, bar = lead_full + 8 * s;
                        if (rank == 0) mbar_expect_tx(full + 8 * s, 2 * WP_STAGE);
                        if (a_blocks) {
                            tma_load_3d_pair(a_dst, mA, 0, row, m0 / 64, bar);
                        } else {
                            tma_load_2d_pair(a_dst, mA, m0, row, bar);
                            tma_load_2d_pair(a_dst + BOX_BYTES, mA, m0 + 64, row, bar);
                        }
                        if (b_blocks) {
                            tma_load_3d_pair(b_dst, mB, 0, row, colB / 64, bar);
                        } else {
                            tma_load_2d_pair(b_dst, mB, colB, row, bar);
                            tma_load_2d_pair(b_dst + BOX_BYTES, mB, colB + 64, row, bar);
                        }
                        if (++s == WP_STAGES) {
                            s = 0;
                            free_phase ^= 1;
                        }
                    }
                }
                if (!ok) break;
                item = grid + next;
            }
            if (rank == 0) sched_finish(p.sched, grid);
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            uint32_t t = 0, phase = 0;
            int s = 0;
            bool ok = true;
            const uint32_t peer_empty = mapa(empty, 1), peer_acc_full = mapa(acc_full, 1);
            const uint64_t desc0 = make_desc(smem_u32(tiles), BOX_BYTES, 1024);
            PairWgradItem w;
            for (uint32_t n = 0; ok && consume(n, w); ++n) {
                release(n);
                if (w.nkb == 0) continue;
                const uint32_t idesc = make_idesc(2 * BM, 2 * w.half, 1, 1), buf = t & 1u;
                if (!mbar_wait_cluster(acc_empty + 8 * buf, ((t >> 1) & 1) ^ 1, p.status, ERR_ACC_WAIT)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int kb = 0; kb < w.nkb; ++kb) {
                    if (!mbar_wait_cluster(full + 8 * s, phase, p.status, ERR_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t ad = desc0 + s * (WP_STAGE >> 4), bd = ad + (A_BYTES >> 4);      // (the address field: 16-byte units)
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_bf16_pair(d_tmem, ad + k * (2048 >> 4), bd + k * (2048 >> 4), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(empty + 8 * s);
                    umma_commit_pair(peer_empty + 8 * s);
                    if (++s == WP_STAGES) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                if (ok) {
                    umma_commit_pair(acc_full + 8 * buf);
                    umma_commit_pair(peer_acc_full + 8 * buf);
                }
                ++t;
            }
        }
    } else if (warp >= 2 + EPI_WARPS) {
        if (rank == 0) {                                   // column sums of the leader's A tile
            const int cw = warp - (2 + EPI_WARPS);
            const int c8 = lane & 7, rg = lane >> 3;       // 16-byte piece of a 128-byte row; rows rg + 4i
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            PairWgradItem w;
            for (uint32_t n = 0; ok && __any_sync(0xffffffffu, consume(n, w)); ++n) {
                __syncwarp();
                if (lane == 0) release(n);
                float acc[2][8] = {};
                for (int kb = 0; kb < w.nkb; ++kb) {
                    if (!mbar_wait(full + 8 * s, phase, p.status, ERR_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    const uint32_t tile = smem_u32(tiles + s * WP_STAGE);
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                        if (w.sum >> b & 1) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const uint32_t r = (uint32_t)(rg + 32 * cw + 4 * i);
                                uint32_t w0, w1, w2, w3;
                                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                                             : "=r"(w0), "=r"(w1), "=r"(w2), "=r"(w3)
                                             : "r"(tile + b * BOX_BYTES + r * 128u + ((((uint32_t)c8) ^ (r & 7u)) << 4)));
                                acc[b][0] += bf_lo(w0); acc[b][1] += bf_hi(w0); acc[b][2] += bf_lo(w1); acc[b][3] += bf_hi(w1);
                                acc[b][4] += bf_lo(w2); acc[b][5] += bf_hi(w2); acc[b][6] += bf_lo(w3); acc[b][7] += bf_hi(w3);
                            }
                        }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty + 8 * s);
                    if (++s == WP_STAGES) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                if (w.nkb > 0)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                        if (w.sum >> b & 1) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                float v = acc[b][i];
                                v += __shfl_xor_sync(0xffffffffu, v, 8);
                                v += __shfl_xor_sync(0xffffffffu, v, 16);
                                const int col = b * 64 + c8 * 8 + i;
                                if (rg == 0 && col < w.cols) red_add(w.gb + col, v);      // two partial sums per column: one per warp
                            }
                        }
            }
        }
    } else {
        // 16 epilogue warps: TMEM lane quarter q (columns of the gradient), 64 of the product's columns (its rows) each
        const int q = warp & 3, h = (warp - 2) >> 2;
        const uint32_t acc_free = rank == 0 ? acc_empty : mapa(acc_empty, 0);
        uint32_t t = 0;
        PairWgradItem w;
        for (uint32_t n = 0; __any_sync(0xffffffffu, consume(n, w)); ++n) {
            __syncwarp();
            if (lane == 0) release(n);
            const int cols = min(32, w.cols - q * 32), rows = cols > 0 ? min(64, w.rows - h * 64) : 0;
            float* const g = w.g + (size_t)(h * 64) * w.M + q * 32;
            if (w.nkb == 0) {                              // an expert without rows
                if (lane < cols)
                    for (int j = 0; j < rows; ++j) g[(size_t)j * w.M + lane] = 0.0f;
                continue;
            }
            const uint32_t buf = t & 1u;
            if (!mbar_wait_cluster(acc_full + 8 * buf, (t >> 1) & 1, p.status, ERR_ACC_WAIT)) break;
            tc_fence_after();
            const uint32_t t_lane = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16) + h * 64;
            float* d = g + lane;                           // one line of the gradient per instruction
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float v[16];
                tmem_ld16(t_lane + c * 16, v);
                tmem_ld_wait();
                if (c == 3) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (rank == 0) mbar_arrive(acc_free + 8 * buf);
                        else mbar_arrive_cluster(acc_free + 8 * buf);
                    }
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (16 * c + j < rows && lane < cols) {
                        if (p.overwrite) *d = v[j];
                        else red_add(d, v[j]);
                    }
                    d += w.M;
                }
            }
            ++t;
        }
    }
    // neither CTA may leave (or give its TMEM back) while the other can still read its shared memory or signal it
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

}  // namespace

// ---- host side: tensor maps ------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// 2-D row-major bf16 tensor [rows, cols].  Loads: box = {64 columns (128 B), box_rows}, 128-byte swizzle,
// OOB reads 0.  Stores (box_rows == 32): box = {32 columns (64 B), 32 rows}, 64-byte swizzle.
int make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows)
{
    return make_map_kind(m, base, rows, cols, box_rows, box_rows == 32);
}

int make_map_kind(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, bool store)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(MGPT_MOE_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * sizeof(bf16)};
    cuuint32_t box[2] = {store ? 32u : 64u, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, store ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MGPT_MOE_ECUDA, "cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
    return 0;
}

int make_map_blocks(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t n_blocks)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(MGPT_MOE_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[3] = {64, rows, (cols + 63) / 64};
    cuuint64_t strides[2] = {cols * sizeof(bf16), 64 * sizeof(bf16)};
    cuuint32_t box[3] = {64, box_rows, n_blocks};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MGPT_MOE_ECUDA, "cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
    return 0;
}

// A tile-major weight copy as {64 columns, 128 rows, n2 blocks at stride2 elements, n3 at stride3}, box {64, rows, b2, b3}.
static int make_map_weights(CUtensorMap* m, const void* base, uint64_t n2, uint64_t stride2, uint64_t n3, uint64_t stride3,
                            uint32_t rows, uint32_t b2, uint32_t b3)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(MGPT_MOE_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[4] = {64, 128, n2, n3};
    cuuint64_t strides[3] = {64 * sizeof(bf16), stride2 * sizeof(bf16), stride3 * sizeof(bf16)};
    cuuint32_t box[4] = {64, rows, b2, b3};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, n3 ? 4 : 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(MGPT_MOE_ECUDA, "cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
    return 0;
}

namespace {

int cdiv(int a, int b) { return (a + b - 1) / b; }

struct TcState {
    const void* ws = nullptr;
    const void *xg = nullptr, *yg = nullptr, *dyg = nullptr, *dxg = nullptr;
    int n_tokens = -1;
    bool attr_set = false;
    int sms = 0;
    int32_t* sched = nullptr;    // device: one {next item, finished CTAs} pair per kind of launch, zero between launches
    // K-major operand loads (box 64 x 128 rows)
    CUtensorMap Xg, Hh, dYg, dG, dU;
    // weight copies: two whole blocks (gate and up; two row blocks of Wd) per load
    CUtensorMap WguT, WdT;
    CUtensorMap Wg_h, Wu_h, Wd_h;      // the same weight copies in half blocks (box 64 columns x 64 rows x 4 blocks)
    // reduction-over-rows operand loads (box 64 x 64 rows)
    CUtensorMap Xg_t, Hh_t, dYg_t, dG_t, dU_t;
    // the same operands by column blocks (one load per operand tile): A side {64, 64 rows, 2}, B side {64, 64 rows, 4}
    CUtensorMap Xg_b4, dYg_b4, dG_b2, dU_b2, Hh_b2;
    CUtensorMap Xg_b2, dYg_b2;
    // epilogue stores (box 32 x 32 rows, 64-byte swizzle)
    CUtensorMap Hh_s, Yg_s, dG_s, dU_s, dXg_s;
    bool c_blocks = false;       // the maps of Xg and dYg are there (C a multiple of 64); those of dG, dU, Hh always are
};

int prepare_attrs(mgpt_moe_layer* L);

int prepare(mgpt_moe_layer* L, const Workspace& w, char* ws)
{
    MGPT_TRY(prepare_attrs(L));
    TcState* s = (TcState*)L->tc_state;
    const void *xg = buf_Xg(L, w, ws), *yg = buf_Yg(L, w, ws), *dyg = buf_dYg(L, w, ws), *dxg = buf_dXg(L, w, ws);
    if (s->ws == ws && s->n_tokens == w.n_tokens && s->xg == xg && s->yg == yg && s->dyg == dyg && s->dxg == dxg) return 0;
    const Dims& d = L->d;
    const uint64_t rc = w.row_cap, C = d.C, H = d.H, E = d.E;
    MGPT_TRY(make_map(&s->Xg, xg, rc, C, 128));
    MGPT_TRY(make_map(&s->Hh, ws + w.Hh, rc, H, 128));
    MGPT_TRY(make_map(&s->dYg, dyg, rc, C, 128));
    MGPT_TRY(make_map(&s->dG, ws + w.dG, rc, H, 128));
    MGPT_TRY(make_map(&s->dU, ws + w.dU, rc, H, 128));
    // tile-major weight copies, 16 KiB (8192 elements) per block
    const uint64_t BLK = 128 * 64, eCH = E * tile_major_elems(d.H, d.C), eHC = E * tile_major_elems(d.C, d.H);
    const uint64_t cb = cdiv(d.H, 64);
    MGPT_TRY(make_map_weights(&s->WguT, L->sWgT, eCH / BLK, BLK, 2, eCH, 128, 1, 2));            // Wu's copy follows Wg's
    MGPT_TRY(make_map_weights(&s->WdT, L->sWdT, cb, BLK, eHC / BLK / cb, cb * BLK, 128, 1, 2));
    MGPT_TRY(make_map_weights(&s->Wg_h, L->sWgT, eCH / BLK, BLK, 0, 0, 64, BN / 64, 1));
    MGPT_TRY(make_map_weights(&s->Wu_h, L->sWuT, eCH / BLK, BLK, 0, 0, 64, BN / 64, 1));
    MGPT_TRY(make_map_weights(&s->Wd_h, L->sWdT, eHC / BLK, BLK, 0, 0, 64, BN / 64, 1));
    MGPT_TRY(make_map(&s->Xg_t, xg, rc, C, 64));
    MGPT_TRY(make_map(&s->Hh_t, ws + w.Hh, rc, H, 64));
    MGPT_TRY(make_map(&s->dYg_t, dyg, rc, C, 64));
    MGPT_TRY(make_map(&s->dG_t, ws + w.dG, rc, H, 64));
    MGPT_TRY(make_map(&s->dU_t, ws + w.dU, rc, H, 64));
    s->c_blocks = C % 64 == 0;
    if (s->c_blocks) {
        MGPT_TRY(make_map_blocks(&s->Xg_b4, xg, rc, C, 64, BN / 64));
        MGPT_TRY(make_map_blocks(&s->dYg_b4, dyg, rc, C, 64, BN / 64));
        MGPT_TRY(make_map_blocks(&s->Xg_b2, xg, rc, C, 64, BM / 64));
        MGPT_TRY(make_map_blocks(&s->dYg_b2, dyg, rc, C, 64, BM / 64));
    }
    // (the last block may reach up to 112 bytes past the buffer: other buffers of the workspace follow all three)
    MGPT_TRY(make_map_blocks(&s->dG_b2, ws + w.dG, rc, H, 64, BM / 64));
    MGPT_TRY(make_map_blocks(&s->dU_b2, ws + w.dU, rc, H, 64, BM / 64));
    MGPT_TRY(make_map_blocks(&s->Hh_b2, ws + w.Hh, rc, H, 64, BM / 64));
    MGPT_TRY(make_map(&s->Hh_s, ws + w.Hh, rc, H, 32));
    MGPT_TRY(make_map(&s->Yg_s, yg, rc, C, 32));
    MGPT_TRY(make_map(&s->dG_s, ws + w.dG, rc, H, 32));
    MGPT_TRY(make_map(&s->dU_s, ws + w.dU, rc, H, 32));
    MGPT_TRY(make_map(&s->dXg_s, dxg, rc, C, 32));
    s->ws = ws;
    s->n_tokens = w.n_tokens;
    s->xg = xg; s->yg = yg; s->dyg = dyg; s->dxg = dxg;
    return 0;
}

int prepare_attrs(mgpt_moe_layer* L)
{
    if (!L->tc_state) L->tc_state = new TcState();
    TcState* s = (TcState*)L->tc_state;
    if (!s->attr_set) {
        MGPT_CUDA(cudaFuncSetAttribute(tc_rows_kernel<MODE_GATEUP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM));
        MGPT_CUDA(cudaFuncSetAttribute((tc_rows_kernel<MODE_GATEUP, false>), cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM));
        MGPT_CUDA(cudaFuncSetAttribute(tc_rows_kernel<MODE_DOWN>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM));
        MGPT_CUDA(cudaFuncSetAttribute(tc_rows_kernel<MODE_DHH>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM));
        MGPT_CUDA(cudaFuncSetAttribute(tc_rows_kernel<MODE_DXG>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM));
        MGPT_CUDA(cudaFuncSetAttribute(tc_dx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        MGPT_CUDA(cudaFuncSetAttribute(tc_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        MGPT_CUDA(cudaFuncSetAttribute(tc_wgrad_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WP_SMEM));
        MGPT_CUDA(cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, L->device));
        // the work-item counters must read zero before the first launch on any stream: allocate and clear them
        // here, at layer creation, and wait for the clear (nothing orders the legacy stream with a caller's
        // non-blocking stream)
        MGPT_CUDA(cudaMalloc(&s->sched, 64 * sizeof(int32_t)));
        MGPT_CUDA(cudaMemset(s->sched, 0, 64 * sizeof(int32_t)));
        MGPT_CUDA(cudaDeviceSynchronize());
        s->attr_set = true;
    }
    return 0;
}

int imin(int a, int b) { return a < b ? a : b; }
// persistent CTAs to launch: every SM, or the caller's budget when other kernels must stay resident beside these
int grid_sms(const mgpt_moe_layer* L, const TcState* s) { return L->sm_budget > 0 ? imin(L->sm_budget, s->sms) : s->sms; }

}  // namespace

// The weight-gradient kernel also sums the bias gradients when every 64-column box of its operand tiles finds an
// item to sum it: the B tile of gWd has four boxes and is loaded once per 128-row tile of H, two boxes per item.
bool tc_fused_bias_grads(const Dims& d) { return cdiv(d.H, BM) >= 2; }

namespace {
// One of the four token-major products.
template <int MODE, bool KEEP = true>
int launch_rows(mgpt_moe_layer* L, TcState* s, const Workspace& w, const RowsP& p, const CUtensorMap& a0, const CUtensorMap& a1,
                const CUtensorMap& b0, const CUtensorMap& b1, const CUtensorMap& d0, const CUtensorMap& d1, cudaStream_t st, const char* what)
{
    MGPT_CUDA(launch_pdl(tc_rows_kernel<MODE, KEEP>, imin(grid_sms(L, s), w.max_tiles * p.n_col_tiles), ROWS_THREADS, ROWS_SMEM, st, a0, a1, b0, b1, d0, d1, p));
    MGPT_LAUNCHED(what);
    return 0;
}
}  // namespace

int tc_experts_forward(mgpt_moe_layer* L, const Workspace& w, char* ws, cudaStream_t st)
{
    if (!L->biases_aligned) return fail(MGPT_MOE_EINVAL, "the expert biases must be 16-byte aligned");
    MGPT_TRY(prepare(L, w, ws));
    TcState* s = (TcState*)L->tc_state;
    const Dims& d = L->d;
    RowsP p = {};
    p.tile_expert = (const int32_t*)(ws + w.tile_expert);
    p.tile_order = L->n_seg > 0 ? (const int32_t*)(ws + w.tile_order) : nullptr;
    p.n_tiles = (const int32_t*)(ws + w.n_tiles);
    p.status = L->d_status;
    // gate/up + SwiGLU: K = C, 128 hidden units per item
    p.kblocks = cdiv(d.C, BK); p.n_out = d.H; p.n_col_tiles = cdiv(d.H, BN / 2);
    p.b_row_blocks = cdiv(d.H, 128); p.b_col_blocks = cdiv(d.C, BK);
    p.bias0 = L->master.bg; p.bias1 = L->master.bu;
    p.early = L->ext_Xg == nullptr;                     // behind dispatch (an expert side's tiles are the kernel's before)
    // Under an SM budget down's CTAs, an SM each, would wait on the very SMs that the caller keeps free.
    p.release = grid_sms(L, s) == s->sms;
    p.G = w.inference ? nullptr : (bf16*)(ws + w.G);
    p.U = w.inference ? nullptr : (bf16*)(ws + w.U);
    L->stage_begin(ST_GATEUP, st);
    p.sched = s->sched + 0;
    if (w.inference) MGPT_TRY((launch_rows<MODE_GATEUP, false>(L, s, w, p, s->Xg, s->Xg, s->WguT, s->WguT, s->Hh_s, s->Hh_s, st, "tc_rows<gateup>")));
    else MGPT_TRY(launch_rows<MODE_GATEUP>(L, s, w, p, s->Xg, s->Xg, s->WguT, s->WguT, s->Hh_s, s->Hh_s, st, "tc_rows<gateup>"));
    L->stage_end(ST_GATEUP, st);
    // down: K = H
    p.kblocks = cdiv(d.H, BK); p.n_out = d.C; p.n_col_tiles = cdiv(d.C, BN);
    p.b_row_blocks = cdiv(d.C, 128); p.b_col_blocks = cdiv(d.H, BK);
    p.bias0 = L->master.bd; p.bias1 = nullptr;
    p.early = 1;
    L->stage_begin(ST_DOWN, st);
    p.sched = s->sched + 2;
    MGPT_TRY(launch_rows<MODE_DOWN>(L, s, w, p, s->Hh, s->Hh, s->WdT, s->WdT, s->Yg_s, s->Yg_s, st, "tc_rows<down>"));
    L->stage_end(ST_DOWN, st);
    return 0;
}

// phase: 1 = gradients w.r.t. the rows (dHh, dXg), 2 = gradients w.r.t. the parameters, 3 = both
int tc_experts_backward(mgpt_moe_layer* L, const Workspace& w, char* ws, cudaStream_t st, int phase)
{
    if (L->has_grad && !L->grad_wd_aligned) return fail(MGPT_MOE_EINVAL, "the gradients of Wd must be 16-byte aligned");
    MGPT_TRY(prepare(L, w, ws));
    TcState* s = (TcState*)L->tc_state;
    const Dims& d = L->d;
    RowsP p = {};
    if (phase & 1) {
    p.tile_expert = (const int32_t*)(ws + w.tile_expert);
    p.tile_order = L->n_seg > 0 ? (const int32_t*)(ws + w.tile_order) : nullptr;
    p.n_tiles = (const int32_t*)(ws + w.n_tiles);
    p.status = L->d_status;
    // dHh = dYg * Wd^T  (K = C), SwiGLU backward in the epilogue
    p.kblocks = cdiv(d.C, BK); p.n_out = d.H; p.n_col_tiles = cdiv(d.H, BN);
    p.b_row_blocks = cdiv(d.C, 128); p.b_col_blocks = cdiv(d.H, BK);
    p.G = (bf16*)(ws + w.G); p.U = (bf16*)(ws + w.U);
    L->stage_begin(ST_DHH, st);
    p.sched = s->sched + 4;
    MGPT_TRY(launch_rows<MODE_DHH>(L, s, w, p, s->dYg, s->dYg, s->Wd_h, s->Wd_h, s->dG_s, s->dU_s, st, "tc_rows<dhh>"));
    L->stage_end(ST_DHH, st);
    // dXg = dG * Wg^T + dU * Wu^T  (K = 2H)
    p.kblocks = cdiv(d.H, BK); p.n_out = d.C; p.n_col_tiles = cdiv(d.C, BN);
    p.b_row_blocks = cdiv(d.H, 128); p.b_col_blocks = cdiv(d.C, BK);
    L->stage_begin(ST_DXG, st);
    p.sched = s->sched + 6;
    MGPT_TRY(launch_rows<MODE_DXG>(L, s, w, p, s->dG, s->dU, s->Wg_h, s->Wu_h, s->dXg_s, s->dXg_s, st, "tc_rows<dxg>"));
    L->stage_end(ST_DXG, st);
    }
    if (!L->has_grad || !(phase & 2)) return 0;

    if (pair_wgrad_usable(d, w.R) && grid_sms(L, s) >= 2) {
        PairWgradP g = {};
        g.padded_offsets = (const int32_t*)(ws + w.padded_offsets);
        g.seg = (const int32_t*)(ws + w.seg);
        g.n_seg = L->n_seg;
        g.status = L->d_status;
        g.sched = s->sched + 8;
        g.C = d.C; g.H = d.H; g.E = d.E;
        g.grad[0] = L->master.gWg; g.grad[1] = L->master.gWu; g.grad[2] = L->master.gWd;
        g.gb[0] = L->master.gbg; g.gb[1] = L->master.gbu; g.gb[2] = L->master.gbd;
        g.overwrite = L->bwd_overwrite ? 1 : 0;
        g.c_blocks = s->c_blocks ? 1 : 0;
        const int pairs = imin(grid_sms(L, s) / 2, d.E * pair_wgrad_items(d.C, d.H));
        L->stage_begin(ST_WGRAD, st);
        MGPT_CUDA(launch_pdl(tc_wgrad_pair_kernel, 2 * pairs, WG_THREADS, WP_SMEM, st, g.c_blocks ? s->Xg_b2 : s->Xg_t,
                             g.c_blocks ? s->dYg_b2 : s->dYg_t, s->dG_b2, s->dU_b2, s->Hh_b2, g));
        MGPT_LAUNCHED("tc_wgrad_pair_kernel");
        L->stage_end(ST_WGRAD, st);
        return 0;
    }

    // all three weight gradients in one launch:
    //   gWg += Xg^T dG, gWu += Xg^T dU   [C,H];   gWd += Hh^T dYg   [H,C]
    // The first two are computed transposed, (dG^T Xg) [H,C]: H = 1408 splits into eleven 128-row tiles and C into
    // whole 256-column tiles, where the direct form leaves the last of six 256-column tiles over H half empty.
    // Writing the tile back transposed costs nothing: a thread's row index runs along a row of the gradient.
    WgradP g = {};
    g.padded_offsets = (const int32_t*)(ws + w.padded_offsets);
    g.seg = (const int32_t*)(ws + w.seg);
    g.n_seg = L->n_seg;
    g.status = L->d_status;
    g.n_probs = 3;
    g.overwrite = L->bwd_overwrite ? 1 : 0;
    float* const* grads[3] = {L->master.gWg, L->master.gWu, L->master.gWd};
    int items = 0;
    for (int i = 0; i < 3; ++i) {
        WgradProb& q = g.prob[i];
        q.grad = grads[i];
        q.M = d.H;
        q.N = d.C;
        q.transposed = i < 2 ? 1 : 0;
        q.n_tiles_m = cdiv(q.M, BM);
        q.n_tiles_n = cdiv(q.N, BN);
        q.n_groups = d.E;
        q.item_begin = items;
        items += d.E * q.n_tiles_m * q.n_tiles_n;
    }
    g.total_items = items;
    L->stage_begin(ST_WGRAD, st);
    g.sched = s->sched + 8;
    if (tc_fused_bias_grads(d)) {
        g.gb[0] = L->master.gbg; g.gb[1] = L->master.gbu; g.gb[2] = L->master.gbd;
    }
    g.block_loads = s->c_blocks ? 1 : 0;
    if (g.block_loads)
        MGPT_CUDA(launch_pdl(tc_wgrad_kernel, imin(grid_sms(L, s), items), WG_THREADS, SMEM_BYTES, st, s->dG_b2, s->Xg_b4, s->dU_b2, s->Xg_b4,
                                                                           s->Hh_b2, s->dYg_b4, g));
    else
        MGPT_CUDA(launch_pdl(tc_wgrad_kernel, imin(grid_sms(L, s), items), WG_THREADS, SMEM_BYTES, st, s->dG_t, s->Xg_t, s->dU_t, s->Xg_t, s->Hh_t,
                                                                           s->dYg_t, g));
    MGPT_LAUNCHED("tc_wgrad_kernel");
    L->stage_end(ST_WGRAD, st);
    return 0;
}

// dx[N,C] (bf16) = gather-sum of the tokens' expert rows + dlogits * Wr^T on the tensor cores
// (K = experts, so the product is a single k-block; the kernel is bound by the row gather).
int tc_router_dx(mgpt_moe_layer* L, const Workspace& w, char* ws, const void* dXg, const int32_t* pos, void* dx,
                 cudaStream_t st)
{
    MGPT_TRY(prepare_attrs(L));
    TcState* s = (TcState*)L->tc_state;
    const Dims& d = L->d;
    const int E8 = (d.E + 7) / 8 * 8;
    CUtensorMap mA, mB;
    MGPT_TRY(make_map(&mA, ws + w.dl16, (uint64_t)w.n_tokens, (uint64_t)E8, 128));
    MGPT_TRY(make_map(&mB, L->sWr, (uint64_t)d.C, (uint64_t)E8, 128));
    RowsP p = {};
    p.n_tiles = (const int32_t*)(ws + w.n_tiles);
    p.tile_expert = (const int32_t*)(ws + w.tile_expert);
    p.status = L->d_status;
    p.kblocks = cdiv(E8, BK); p.n_out = d.C; p.n_col_tiles = cdiv(d.C, BN);
    p.fixed_tiles = cdiv(w.n_tokens, BM); p.n_valid_rows = w.n_tokens;
    p.gather_src = (const bf16*)dXg; p.gather_pos = pos; p.gather_k = d.k;
    p.dx = (bf16*)dx;
    MGPT_CUDA(launch_pdl(tc_dx_kernel, imin(grid_sms(L, s), p.fixed_tiles * p.n_col_tiles), TC_THREADS, SMEM_BYTES, st, mA, mB, p));
    MGPT_LAUNCHED("tc_dx_kernel");
    return 0;
}

// gWr[C,E] += x^T * dlogits on the tensor cores, split over uniform token chunks (RED accumulation).  Bound by the stream of
// x; but a producer thread spends 250-500 cycles on a TMA load, and with six per 64 tokens (all of a 256-column tile, mostly
// zero fill) that was the kernel: two now where the channels come in whole blocks of 64 and E <= 64.  As many chunks as
// make one wave: 51-57 -> 39 us at 32768 tokens, C=2048, E=64 (8.8 and 15 us at 8192 x 512 and 16384 x 1024: unchanged).
int tc_router_wgrad(mgpt_moe_layer* L, const Workspace& w, char* ws, const void* x, cudaStream_t st)
{
    MGPT_TRY(check_aligned(L->p_grad[0], "the gradient of Wr"));
    MGPT_TRY(prepare_attrs(L));
    TcState* s = (TcState*)L->tc_state;
    const Dims& d = L->d;
    const int E8 = (d.E + 7) / 8 * 8;
    CUtensorMap mA, mB;
    WgradP g = {};
    g.block_loads = d.C % 64 == 0 ? 1 : 0;
    if (g.block_loads) MGPT_TRY(make_map_blocks(&mA, x, (uint64_t)w.n_tokens, (uint64_t)d.C, 64, BM / 64));
    else MGPT_TRY(make_map(&mA, x, (uint64_t)w.n_tokens, (uint64_t)d.C, 64));
    MGPT_TRY(make_map(&mB, ws + w.dl16, (uint64_t)w.n_tokens, (uint64_t)E8, 64));
    g.b_boxes = cdiv(E8, 64);
    g.status = L->d_status;
    g.n_probs = 1;
    WgradProb& q = g.prob[0];
    q.M = d.C; q.N = d.E; q.n_tiles_m = cdiv(d.C, BM); q.n_tiles_n = cdiv(d.E, BN);
    const int per_chunk = q.n_tiles_m * q.n_tiles_n;
    int chunks = imin(64, per_chunk < s->sms ? s->sms / per_chunk : 1);
    int rows = cdiv(cdiv(w.n_tokens, chunks), BK) * BK;           // tokens per chunk, whole k-blocks
    chunks = cdiv(w.n_tokens, rows);
    q.n_groups = chunks; q.uniform_rows = rows; q.single_grad = L->p_grad[0]; q.item_begin = 0;
    g.total_items = chunks * per_chunk;
    g.sched = s->sched + 10;
    MGPT_CUDA(launch_pdl(tc_wgrad_kernel, imin(grid_sms(L, s), g.total_items), WG_THREADS, SMEM_BYTES, st, mA, mB, mA, mB, mA, mB, g));
    MGPT_LAUNCHED("tc_wgrad_kernel<Wr>");
    return 0;
}

// One barrier nothing ever arrives on, waited for with the kernels' own bounded wait and a short limit: the wait
// runs out after a few thousand polls, the error bit is set and the kernel returns normally.
__global__ void bounded_wait_selftest_kernel(int32_t* status)
{
    __shared__ __align__(8) uint64_t bar;
    pdl_wait();
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_wait(smem_u32(&bar), 0, status, ERR_FULL_WAIT, 1u << 12);
    }
}

int tc_selftest_bounded_wait(mgpt_moe_layer* L, cudaStream_t st)
{
    MGPT_CUDA(launch_pdl(bounded_wait_selftest_kernel, 1, 32, 0, st, L->d_status));
    MGPT_LAUNCHED("bounded_wait_selftest_kernel");
    L->last_stream = st;
    return 0;
}

// Called once from mgpt_moe_create (the layer's device is current): function attributes, SM count, work counters.
int tc_init(mgpt_moe_layer* L) { return prepare_attrs(L); }

void tc_destroy(mgpt_moe_layer* L)
{
    TcState* s = (TcState*)L->tc_state;
    if (s && s->sched) cudaFree(s->sched);
    delete s;
    L->tc_state = nullptr;
}

}  // namespace mgpt
