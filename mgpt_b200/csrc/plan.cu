// Dispatch plan, token permutation and combine of the MoE layer.
//
// Reference semantics (paths relative to the reference's src/main/):
//   counts / offsets   utils/Tensor.cpp:1336-1352, layers/MoELayer.cpp:61-80
//   slot assignment    utils/Tensor.cpp:1368-1381 (flat index ascending => stable)
//   combine            utils/Tensor.cpp:1398-1406
//   combine backward   utils/Tensor.cpp:1424-1436
//
// The reference claims slots with a float atomicAdd on the GPU and a host
// round trip for the prefix sum.  Here the plan is built on the device with
// no atomics on the slot order and no host synchronisation: block histograms,
// one scan, then a stable rank per flat index.  The slot map therefore equals
// the CPU reference's bit for bit.
//
// Rows are stored expert-major with every expert's segment padded to a
// multiple of ROW_TILE rows; padding rows are zero.  Every product tile is
// then a full tile of one expert, and zero rows contribute nothing to the
// weight gradients.
#include <mutex>

#include "plan_block.cuh"

namespace mgpt {

namespace {

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(bf16 v) { return __bfloat162float(v); }

// (1) per-block expert histogram
__global__ void __launch_bounds__(PLAN_BLOCK)
plan_count_kernel(const int32_t* top_idx, int R, int E, int32_t* blk_cnt, int32_t* status)
{
    pdl_wait();
    __shared__ int cnt[MAX_EXPERTS];
    if (threadIdx.x < E) cnt[threadIdx.x] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    __syncthreads();
    const int i = blockIdx.x * PLAN_BLOCK + threadIdx.x;
    if (i < R) {
        const int e = top_idx[i];
        if ((unsigned)e < (unsigned)E) atomicAdd(&cnt[e], 1);      // ids outside [0, E) are reported by plan_assign_kernel
    }
    __syncthreads();
    if (threadIdx.x < E) blk_cnt[(size_t)blockIdx.x * E + threadIdx.x] = cnt[threadIdx.x];
}

// (2) for many blocks only: the histograms become, in place, the rows of an expert in the blocks before; totals -> counts.
// One block per 32 experts (lane = expert), each warp a contiguous share of the blocks, walked twice.
__global__ void __launch_bounds__(1024) plan_scan_kernel(int32_t* blk_cnt, int n_blocks, int E, int32_t* counts)
{
    pdl_wait();
    __shared__ int part[32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, x = blockIdx.x * 32 + lane;
    const int b0 = (int)((long long)n_blocks * warp / 32), b1 = (int)((long long)n_blocks * (warp + 1) / 32);
    int sum = 0;
    if (x < E)
#pragma unroll 8
        for (int b = b0; b < b1; ++b) sum += blk_cnt[(size_t)b * E + x];
    part[warp][lane] = sum;
    __syncthreads();
    int run = 0;
    for (int w = 0; w < warp; ++w) run += part[w][lane];
    if (x >= E) return;
    if (warp == 31) counts[x] = run + sum;
    for (int b = b0; b < b1; b += 8) {
        int c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) c[u] = b + u < b1 ? blk_cnt[(size_t)(b + u) * E + x] : 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (b + u < b1) blk_cnt[(size_t)(b + u) * E + x] = run;
            run += c[u];
        }
    }
}

// (3) everything else: the sums of the histograms over all blocks and over those before this one, a scan of the experts, and
// the stable rank of the block's own rows -> map / pos / row_src; block 0 also writes what is not per row.  SCANNED: the
// sums are plan_scan_kernel's; else each block makes them itself (8 slices of blocks x 128 experts; n_blocks * E integers
// out of L2), which saves the launch but grows with the square of the rows.
template <bool SCANNED>
__global__ void __launch_bounds__(PLAN_BLOCK) plan_assign_kernel(const PlanArgs p, int n_blocks, const int32_t* blk_cnt)
{
    pdl_wait();
    __shared__ int warp_cnt[PLAN_SEGS][MAX_EXPERTS];
    __shared__ int part[2][8][MAX_EXPERTS];
    __shared__ int tot[MAX_EXPERTS], base[MAX_EXPERTS], off[MAX_EXPERTS], tile0[MAX_EXPERTS + 1], goff[MAX_EXPERTS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = blockIdx.x * PLAN_BLOCK + tid;
    bool valid = i < p.R;
    int e = valid ? p.top_idx[i] : 0;
    if (!SCANNED) {
        const int x = tid & (MAX_EXPERTS - 1), slice = tid / MAX_EXPERTS;
        int before = 0, all = 0;
        if (x < p.E) {
#pragma unroll 8
            for (int b = slice; b < n_blocks; b += 8) {
                const int c = blk_cnt[(size_t)b * p.E + x];
                all += c;
                if (b < (int)blockIdx.x) before += c;
            }
        }
        part[0][slice][x] = before;
        part[1][slice][x] = all;
    }
    for (int j = tid; j < PLAN_SEGS * MAX_EXPERTS; j += PLAN_BLOCK) (&warp_cnt[0][0])[j] = 0;
    __syncthreads();
    if (tid < MAX_EXPERTS) {
        int before = 0, all = 0;
        if (SCANNED) {
            if (tid < p.E) {
                before = blk_cnt[(size_t)blockIdx.x * p.E + tid];
                all = p.counts[tid];
            }
        } else {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                before += part[0][s][tid];
                all += part[1][s][tid];
            }
        }
        base[tid] = before;
        tot[tid] = all;
    }
    if (valid && (unsigned)e >= (unsigned)p.E) {                  // an id no expert has: no slot, and the caller is told
        atomicOr(p.status, ST_BAD_EXPERT);
        if (p.sticky) atomicOr(p.sticky, ST_BAD_EXPERT);
        valid = false;
    }
    if (!valid) e = -1 - lane;                                    // distinct keys for idle lanes
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
    if (valid && rank_in_warp == 0) warp_cnt[warp][e] = __popc(peers);
    __syncthreads();
    if (warp == 0) {
        int nt, ng;
        plan_scan_experts(tot, p.E, lane, off, tile0, goff, nt, ng);
        if (lane == 0) {
            tile0[p.E] = nt;
            if (blockIdx.x == 0) {
                *p.n_tiles = nt;
                p.padded_offsets[p.E] = nt * ROW_TILE;
                if (p.groups) *p.n_groups = ng;
                if (nt > p.max_tiles) {                           // cannot happen: max_tiles bounds sum(ceil)
                    atomicOr(p.status, ST_PLAN_OVERFLOW);
                    if (p.sticky) atomicOr(p.sticky, ST_PLAN_OVERFLOW);
                }
            }
        }
    }
    __syncthreads();
    if (valid) {
        int r = base[e] + rank_in_warp;
        for (int w = 0; w < warp; ++w) r += warp_cnt[w][e];
        const int slot = off[e] + r, q = tile0[e] * ROW_TILE + r;
        p.map[slot] = i;
        p.pos[i] = q;
        p.row_src[q] = i;
        if (p.slot_of) p.slot_of[i] = slot;
    }
    if (blockIdx.x != 0) return;
    for (int x = warp; x < p.E; x += PLAN_SEGS) {
        const int t0 = tile0[x], t1 = tile0[x + 1], n = tot[x];
        if (lane == 0) {
            if (!SCANNED) p.counts[x] = n;
            p.offsets[x] = off[x];
            p.padded_offsets[x] = t0 * ROW_TILE;
        }
        for (int t = t0 + lane; t < t1 && t < p.max_tiles; t += 32) p.tile_expert[t] = x;
        // padding rows of the expert's segment carry no source
        for (int q = t0 * ROW_TILE + n + lane; q < t1 * ROW_TILE; q += 32) p.row_src[q] = -1;
        if (p.groups)
            for (int g = lane; g * DECODE_GROUP < n; g += 32)
                p.groups[goff[x] + g] = make_int4(x, t0 * ROW_TILE + g * DECODE_GROUP, min(DECODE_GROUP, n - g * DECODE_GROUP), 0);
    }
}

// The whole plan in one block, for up to PLAN_BLOCK routed rows: one launch instead of two.
__global__ void __launch_bounds__(512) plan_small_kernel(const PlanArgs p)
{
    pdl_wait();
    __shared__ PlanShared sh;
    plan_block<16>(p, sh);
}

// 8 consecutive elements <-> 8 floats (16 bytes of bf16, 32 bytes of float)
template <typename T> __device__ __forceinline__ void load8(const T* p, float (&v)[8]);
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&v)[8])
{
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void load8<bf16>(const bf16* p, float (&v)[8])
{
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float (&v)[8]);
template <> __device__ __forceinline__ void store8<float>(float* p, const float (&v)[8])
{
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
template <> __device__ __forceinline__ void store8<bf16>(bf16* p, const float (&v)[8])
{
    uint4 u;
    __nv_bfloat162 h0 = __floats2bfloat162_rn(v[0], v[1]), h1 = __floats2bfloat162_rn(v[2], v[3]);
    __nv_bfloat162 h2 = __floats2bfloat162_rn(v[4], v[5]), h3 = __floats2bfloat162_rn(v[6], v[7]);
    u.x = *reinterpret_cast<uint32_t*>(&h0); u.y = *reinterpret_cast<uint32_t*>(&h1);
    u.z = *reinterpret_cast<uint32_t*>(&h2); u.w = *reinterpret_cast<uint32_t*>(&h3);
    *reinterpret_cast<uint4*>(p) = u;
}

// The rows of a token: lane j < k gets the padded row of the token's j-th choice, or -1 (a choice without a slot: an id no
// expert has, which the plan has reported).
__device__ __forceinline__ int token_row(const int32_t* pos, const int32_t* row_src, int row_cap, int tok,
                                         int k, int lane)
{
    if (lane >= k) return -1;
    const int q = pos[(size_t)tok * k + lane];
    return (unsigned)q < (unsigned)row_cap && row_src[q] == tok * k + lane ? q : -1;
}

// Zeros in those of the PAD_ROWS rows of group `g` that carry no token, eight rows to a warp.  (With 32 rows to a warp,
// and these blocks behind the tokens', an expert's last tile was the end of the launch: 2-4 us more at 8192 tokens.)
constexpr int PAD_ROWS = 64;
template <typename TAct>
__device__ __forceinline__ void zero_padding(const int32_t* row_src, int rows, int g, int C, TAct* dst)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q0 = g * PAD_ROWS + warp * 8;
    unsigned m = __ballot_sync(0xffffffffu, lane < 8 && q0 + lane < rows && row_src[q0 + lane] < 0);
    const float z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (; m; m &= m - 1) {
        TAct* row = dst + (size_t)(q0 + __ffs(m) - 1) * C;
        for (int c = lane * 8; c < C; c += 256) store8(row + c, z);
    }
}

// The same in one of the buffers that backward reads beside Xg where the decode kernels, which leave padding rows alone,
// make the forward: 0: Hh, 1 and 2: the saved SwiGLU factors ([row tile][8-column chunk][128 rows][8], gemm_tc.cu).  Four
// times the blocks of Xg's instead of a memset of the three whole buffers, which broke the chain of launches and cleared
// what the worst routing would need (a training step of 1 token, C=1024, H=2816, E=32: 222 -> 214 us; 16 tokens, C=2048,
// H=1408, E=64: 747 -> 739).
__device__ __forceinline__ void zero_padding_kept(const int32_t* row_src, int rows, int g, const PaddingZeros& z, int which)
{
    if (which == 0) {
        zero_padding(row_src, rows, g, z.H, z.Hh);
        return;
    }
    const int lane = threadIdx.x & 31, q0 = g * PAD_ROWS + (threadIdx.x >> 5) * 8, row = q0 + (lane & 7);
    if (row >= rows || row_src[row] >= 0) return;
    uint4* chunk = reinterpret_cast<uint4*>(which == 1 ? z.G : z.U) + (size_t)(q0 / ROW_TILE) * (z.H >> 3) * ROW_TILE + row % ROW_TILE;
    for (int c = lane >> 3; c < z.H >> 3; c += 4) chunk[(size_t)c * ROW_TILE] = make_uint4(0, 0, 0, 0);
}

// Xg[pos(tok,j),:] = x[tok,:] for every choice j; the blocks before the tokens' write the padding rows' zeros (none are
// launched where nothing reads those rows: the products of inference keep rows apart).  Bound by HBM: one warp per token
// reads its row once, four 16-byte loads per lane in flight, and writes it k times.  (A warp per padded row read every
// token k times and wrote padding by single elements: 104 -> 79-94 us at 32768 tokens, C=2048, top-2; 14.4 -> 3.2 us
// at 256 tokens and 32 experts, where seven of eight rows are padding.)
template <typename TIn, typename TAct, bool VEC>
__global__ void __launch_bounds__(256)
dispatch_kernel(const TIn* x, const int32_t* pos, const int32_t* row_src,
                const int32_t* n_tiles, int row_cap, int N, int C, int k, int pad_blocks, TAct* Xg, PaddingZeros kept)
{
    pdl_wait();
    if constexpr (sizeof(TAct) == 2) pdl_release();  // the tensor-core product that follows requests its first weights
    const int lane = threadIdx.x & 31, all_pads = kept.Hh ? 4 * pad_blocks : pad_blocks;
    if ((int)blockIdx.x < all_pads) {
        const int rows = *n_tiles * ROW_TILE;
        if ((int)blockIdx.x < pad_blocks) zero_padding(row_src, rows, blockIdx.x, C, Xg);
        else zero_padding_kept(row_src, rows, blockIdx.x % pad_blocks, kept, blockIdx.x / pad_blocks - 1);
        return;
    }
    const int tok = (blockIdx.x - all_pads) * 8 + (threadIdx.x >> 5);
    if (tok >= N) return;
    const int mine = token_row(pos, row_src, row_cap, tok, k, lane);
    const TIn* s = x + (size_t)tok * C;
    constexpr int U = sizeof(TIn) == sizeof(TAct) && sizeof(TIn) == 2 ? 4 : 2;
    for (int c0 = lane * 8; c0 - lane * 8 < C; c0 += 256 * U) {
        float v[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + 256 * u < C) {
                if constexpr (VEC) {
                    load8(s + c0 + 256 * u, v[u]);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[u][i] = to_f32(s[c0 + 256 * u + i]);
                }
            }
        for (int j = 0; j < k; ++j) {
            const int q = __shfl_sync(0xffffffffu, mine, j);
            if (q < 0) continue;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (c0 + 256 * u < C) store8(Xg + (size_t)q * C + c0 + 256 * u, v[u]);
        }
    }
}

// y[tok,:] = sum_j p[tok,j] * Yg[pos(tok,j),:], slots visited in ascending order
// like the reference's scatter-add.  One warp per token, 8 channels per lane per step; K = top-k rounded up
// to a power of two, so the sort is a fixed network and the kernel fits 32 registers (all 64 warps resident).
// Few tokens: the 256-channel pieces of a token go to blocks of their own (grid.y) while those fit the chip at once; in one
// warp they follow each other, each a trip to L2 (C=1024: 4.7 -> 2.5 us for one token, 5.4 -> 2.9 for 256, 5.7 -> 3.7 for 1777).
template <typename TAct, typename TIo, int K>
__global__ void __launch_bounds__(256, 8)
combine_fwd_kernel(const TAct* Yg, const int32_t* pos, const float* top_p,
                   int N, int C, int k, const TIo* residual, TIo* y)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int tok = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tok >= N) return;
    int ps[K];
    float pr[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        ps[j] = j < k ? pos[(size_t)tok * k + j] : 0x7fffffff;
        pr[j] = j < k ? top_p[(size_t)tok * k + j] : 0.0f;
    }
#pragma unroll
    for (int a = 0; a < K - 1; ++a)                 // tiny sorting network (bubble), static indices
#pragma unroll
        for (int b = 0; b < K - 1 - a; ++b)
            if (ps[b] > ps[b + 1]) {
                int ti = ps[b]; ps[b] = ps[b + 1]; ps[b + 1] = ti;
                float tf = pr[b]; pr[b] = pr[b + 1]; pr[b + 1] = tf;
            }
    for (int c = (blockIdx.y * 32 + lane) * 8; c < C; c += gridDim.y * 256) {
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < K; ++j) {
            if (j < k) {
                float v[8];
                load8(Yg + (size_t)ps[j] * C + c, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(acc[i], __fmul_rn(v[i], pr[j]));
            }
        }
        if (residual) {                 // y = residual + moe(x): the block's skip connection (TransformerBlock.cpp:44)
            float r[8];
            load8(residual + (size_t)tok * C + c, r);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = __fadd_rn(r[i], acc[i]);
        }
        store8(y + (size_t)tok * C + c, acc);
    }
}

// dYg[q,:] = p * dy[tok,:],  d_top_p[flat] = <Yg[q,:], dy[tok,:]> for the rows q of every token; padding rows -> 0 (the
// blocks before the tokens').  Bound by HBM: one warp per token, which reads dy once for all its K >= k rows (a warp per
// padded row read it k times: 124 -> 110-115 us at 32768 tokens, C=2048, top-2; 56 -> 47 us at 16384, C=1024, top-4).
template <typename TAct, typename TIo, int K>
__global__ void __launch_bounds__(256)
combine_bwd_kernel(const TIo* dy, const TAct* Yg, const int32_t* pos,
                   const int32_t* row_src, const float* top_p, const int32_t* n_tiles,
                   int row_cap, int N, int C, int k, int pad_blocks, TAct* dYg, float* d_top_p)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    if ((int)blockIdx.x < pad_blocks) {
        zero_padding(row_src, *n_tiles * ROW_TILE, blockIdx.x, C, dYg);
        return;
    }
    const int tok = (blockIdx.x - pad_blocks) * 8 + (threadIdx.x >> 5);
    if (tok >= N) return;
    const int mine = token_row(pos, row_src, row_cap, tok, k, lane);
    const float prob = lane < k ? top_p[(size_t)tok * k + lane] : 0.0f;
    int q[K];
    float pr[K], dot[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        q[j] = __shfl_sync(0xffffffffu, mine, j);
        pr[j] = __shfl_sync(0xffffffffu, prob, j);
        dot[j] = 0.0f;
    }
    const TIo* g = dy + (size_t)tok * C;
    constexpr int KB = K < 4 ? K : 4;                // rows in flight
    for (int c = lane * 8; c < C; c += 256) {
        float gv[8];
        load8(g + c, gv);
#pragma unroll
        for (int j0 = 0; j0 < K; j0 += KB) {
            float yv[KB][8];
#pragma unroll
            for (int j = 0; j < KB; ++j) load8(Yg + (size_t)max(q[j0 + j], 0) * C + c, yv[j]);
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                float o[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    o[i] = __fmul_rn(gv[i], pr[j0 + j]);
                    dot[j0 + j] = fmaf(yv[j][i], gv[i], dot[j0 + j]);
                }
                if (q[j0 + j] >= 0) store8(dYg + (size_t)q[j0 + j] * C + c, o);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot[j] += __shfl_xor_sync(0xffffffffu, dot[j], o);
        if (lane == 0 && q[j] >= 0) d_top_p[(size_t)tok * k + j] = dot[j];
    }
}

// Column sums over each expert's rows, for the three bias gradients in one launch:
// gbd[e] += colsum(dYg), gbg[e] += colsum(dG), gbu[e] += colsum(dU)  (layers/LinearLayer.cpp:56-57).
// One CTA = one 128-row tile (one expert) x 256 columns; a thread reads 8 columns (16 bytes) of
// every 8th row, the 8 row lanes are folded in shared memory, then one atomicAdd per column.
struct BiasGradArgs {
    const void* M[3];
    float* const* gb[3];
    int cols[3];
    const int32_t* tile_expert;
    const int32_t* n_tiles;
};

__global__ void __launch_bounds__(256) bias_grad_kernel(BiasGradArgs a)
{
    pdl_wait();
    __shared__ float red[8][256 + 8];
    const int tile = blockIdx.x, which = blockIdx.z;
    if (tile >= *a.n_tiles) return;
    const int cols = a.cols[which];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c = blockIdx.y * 256 + tx * 8;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (c < cols) {
        const bf16* base = (const bf16*)a.M[which] + (size_t)tile * ROW_TILE * cols + c;
#pragma unroll 4
        for (int r = ty; r < ROW_TILE; r += 8) {
            const bf16* p = base + (size_t)r * cols;
            const uint4 u = *reinterpret_cast<const uint4*>(p);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[2 * i] += __uint_as_float(w[i] << 16);
                s[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) red[ty][tx * 8 + i] = s[i];
    __syncthreads();
    const int col = blockIdx.y * 256 + threadIdx.x;
    if (col < cols) {
        float t = 0.0f;
#pragma unroll
        for (int r = 0; r < 8; ++r) t += red[r][threadIdx.x];
        atomicAdd(&a.gb[which][a.tile_expert[tile]][col], t);
    }
}

}  // namespace

// A copy within the device as one of the step's kernels: cudaMemcpyAsync, a copy of its own, breaks the chain of launches
// that overlap each other's start and end (0.6 MB of routing: 1.7-2.4 us and 1.5-2.2 us before it, now 1.9-2.2 us and none; 2 us of a checkpointed step of 718).
static __global__ void __launch_bounds__(256) copy_kernel(const uint4* src, uint4* dst, size_t n)
{
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) dst[i] = src[i];
}

int copy_on_device(void* dst, const void* src, size_t bytes, cudaStream_t st)
{
    if ((((uintptr_t)dst | (uintptr_t)src | bytes) & 15) || bytes == 0) {
        MGPT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st));
        return 0;
    }
    const size_t n = bytes / 16, blocks = (n + 255) / 256;
    MGPT_CUDA(launch_pdl(copy_kernel, (int)(blocks < 1184 ? blocks : 1184), 256, 0, st, (const uint4*)src, (uint4*)dst, n));
    MGPT_LAUNCHED("copy_kernel");
    return 0;
}

// Blocks from which the histograms are scanned by a kernel of their own.  Call us without / with it (E = 64): 128 blocks
// 13 / 14, 256 16 / 13, 512 25 / 18, 1024 59 / 29, 16384 8846 / 404; E = 8 meets at 512 (17 / 17), E = 128 at 128 (16 / 15).
constexpr int PLAN_SCAN_FROM = 256;

// The plan on explicit buffers.  `blk` is scratch of plan_blocks*E ints: every element is written by plan_count_kernel
// before it is read, so it needs no clearing.  (Rows beyond the plan's tiles are never read.)
static int run_plan_args(const PlanArgs& p, int32_t* blk, cudaStream_t st)
{
    if (p.R <= PLAN_BLOCK) {
        MGPT_CUDA(launch_pdl(plan_small_kernel, 1, 512, 0, st, p));
        MGPT_LAUNCHED("plan_small_kernel");
        return 0;
    }
    const int plan_blocks = (p.R + PLAN_BLOCK - 1) / PLAN_BLOCK;
    MGPT_CUDA(launch_pdl(plan_count_kernel, plan_blocks, PLAN_BLOCK, 0, st, p.top_idx, p.R, p.E, blk, p.status));
    MGPT_LAUNCHED("plan_count_kernel");
    if (plan_blocks >= PLAN_SCAN_FROM) {
        MGPT_CUDA(launch_pdl(plan_scan_kernel, (p.E + 31) / 32, 1024, 0, st, blk, plan_blocks, p.E, p.counts));
        MGPT_LAUNCHED("plan_scan_kernel");
        MGPT_CUDA(launch_pdl(plan_assign_kernel<true>, plan_blocks, PLAN_BLOCK, 0, st, p, plan_blocks, blk));
    } else {
        MGPT_CUDA(launch_pdl(plan_assign_kernel<false>, plan_blocks, PLAN_BLOCK, 0, st, p, plan_blocks, blk));
    }
    MGPT_LAUNCHED("plan_assign_kernel");
    return 0;
}

PlanArgs plan_args(const Dims& d, const Workspace& w, char* ws, int32_t* sticky)
{
    auto I = [&](size_t o) { return (int32_t*)(ws + o); };
    return PlanArgs{I(w.top_idx), w.R, d.E, I(w.counts), I(w.offsets), I(w.padded_offsets), I(w.tile_expert), I(w.n_tiles), w.max_tiles,
                    I(w.map), I(w.pos), I(w.row_src), I(w.slot), I(w.status), sticky, w.decode ? (int4*)(ws + w.groups) : nullptr,
                    I(w.n_groups)};
}

int launch_plan(const Dims& d, const Workspace& w, char* ws, cudaStream_t st, int32_t* sticky)
{
    return run_plan_args(plan_args(d, w, ws, sticky), (int32_t*)(ws + w.blk_cnt), st);
}

// dst[pos(tok,j),:] = src[tok,:]; with `zero_pad`, zeros in every other row of the plan's tiles
// (there, and in the buffers of `kept` if given)
int dispatch_rows(const Workspace& w, char* ws, const void* src, int src_io, int C, int k, void* dst, bool zero_pad, cudaStream_t st,
                  PaddingZeros kept)
{
    if (w.n_tokens <= 0) return 0;
    const int32_t* pos = (const int32_t*)(ws + w.pos);
    const int32_t* row_src = (const int32_t*)(ws + w.row_src);
    const int32_t* n_tiles = (const int32_t*)(ws + w.n_tiles);
    const int N = w.n_tokens, pad_blocks = zero_pad ? (w.row_cap + PAD_ROWS - 1) / PAD_ROWS : 0;
    const int grid = (kept.Hh ? 4 * pad_blocks : pad_blocks) + (N + 7) / 8;
    const bool vec = ((uintptr_t)src & 15) == 0;
#define MGPT_DISPATCH(TIN, TACT)                                                                                          \
    do {                                                                                                                  \
        auto* kernel = vec ? dispatch_kernel<TIN, TACT, true> : dispatch_kernel<TIN, TACT, false>;                        \
        MGPT_CUDA(launch_pdl(kernel, grid, 256, 0, st, (const TIN*)src, pos, row_src, n_tiles, w.row_cap, N, C, k, pad_blocks, (TACT*)dst, kept)); \
    } while (0)
    if (w.act_bytes == 4) {
        if (src_io != MGPT_MOE_IO_F32) return fail(MGPT_MOE_EINVAL, "FP32 mode takes FP32 rows");
        MGPT_DISPATCH(float, float);
    } else if (src_io == MGPT_MOE_IO_F32) {
        MGPT_DISPATCH(float, bf16);
    } else {
        MGPT_DISPATCH(bf16, bf16);
    }
#undef MGPT_DISPATCH
    MGPT_LAUNCHED("dispatch_kernel");
    return 0;
}

int launch_dispatch(const Dims& d, const Workspace& w, char* ws, const void* x, int io, bool zero_pad, cudaStream_t st)
{
    PaddingZeros kept = {};
    if (zero_pad && w.decode) kept = PaddingZeros{(bf16*)(ws + w.Hh), (bf16*)(ws + w.G), (bf16*)(ws + w.U), d.H};
    return dispatch_rows(w, ws, x, io, d.C, d.k, ws + w.Xg, zero_pad, st, kept);
}

// y = weighted gather-sum of rows[pos[tok,j]]
int combine_rows(const void* rows, const int32_t* pos, const float* top_p, int N, int C, int k, void* y, int io,
                 size_t act_bytes, cudaStream_t st, const void* residual)
{
    if (N <= 0) return 0;
    const int blocks = (N + 7) / 8, pieces = (C + 255) / 256, room = 148 * 8 / blocks;
    const dim3 grid(blocks, room < 1 ? 1 : room < pieces ? room : pieces);
#define MGPT_COMBINE(KK)                                                                                                  \
    do {                                                                                                                  \
        if (act_bytes == 4)                                                                                               \
            MGPT_CUDA(launch_pdl(combine_fwd_kernel<float, float, KK>, grid, 256, 0, st, (const float*)rows, pos, top_p, N, C, k, (const float*)residual, (float*)y)); \
        else if (io == MGPT_MOE_IO_F32)                                                                                   \
            MGPT_CUDA(launch_pdl(combine_fwd_kernel<bf16, float, KK>, grid, 256, 0, st, (const bf16*)rows, pos, top_p, N, C, k, (const float*)residual, (float*)y)); \
        else                                                                                                              \
            MGPT_CUDA(launch_pdl(combine_fwd_kernel<bf16, bf16, KK>, grid, 256, 0, st, (const bf16*)rows, pos, top_p, N, C, k, (const bf16*)residual, (bf16*)y));   \
    } while (0)
    if (k <= 1) MGPT_COMBINE(1);
    else if (k <= 2) MGPT_COMBINE(2);
    else if (k <= 4) MGPT_COMBINE(4);
    else MGPT_COMBINE(8);
#undef MGPT_COMBINE
    MGPT_LAUNCHED("combine_fwd_kernel");
    return 0;
}

int launch_combine_fwd(const Dims& d, const Workspace& w, char* ws, void* y, int io, cudaStream_t st, const void* residual)
{
    return combine_rows(ws + w.Yg, (const int32_t*)(ws + w.pos), (const float*)(ws + w.top_p), w.n_tokens, d.C, d.k, y,
                        io, w.act_bytes, st, residual);
}

// d_rows[pos(tok,j)] = top_p * dy[tok] (other rows of the plan's tiles: 0), d_top_p[flat] = <rows[pos(tok,j)], dy[tok]>
int combine_rows_backward(const Workspace& w, char* ws, const void* dy, int io, const void* rows, int C, int k, void* d_rows, cudaStream_t st)
{
    if (w.n_tokens <= 0) return 0;
    const int N = w.n_tokens, pad_blocks = (w.row_cap + PAD_ROWS - 1) / PAD_ROWS, grid = pad_blocks + (N + 7) / 8;
#define MGPT_COMBINE(TACT, TIO, KK)                                                                                       \
    MGPT_CUDA(launch_pdl(combine_bwd_kernel<TACT, TIO, KK>, grid, 256, 0, st, (const TIO*)dy, (const TACT*)rows,          \
                         (const int32_t*)(ws + w.pos), (const int32_t*)(ws + w.row_src), (const float*)(ws + w.top_p),    \
                         (const int32_t*)(ws + w.n_tiles), w.row_cap, N, C, k, pad_blocks, (TACT*)d_rows, (float*)(ws + w.d_top_p)))
#define MGPT_COMBINE_K(KK)                                                                                                \
    do {                                                                                                                  \
        if (w.act_bytes == 4) MGPT_COMBINE(float, float, KK);                                                             \
        else if (io == MGPT_MOE_IO_F32) MGPT_COMBINE(bf16, float, KK);                                                    \
        else MGPT_COMBINE(bf16, bf16, KK);                                                                                \
    } while (0)
    if (k <= 1) MGPT_COMBINE_K(1);
    else if (k <= 2) MGPT_COMBINE_K(2);
    else if (k <= 4) MGPT_COMBINE_K(4);
    else MGPT_COMBINE_K(8);
#undef MGPT_COMBINE_K
#undef MGPT_COMBINE
    MGPT_LAUNCHED("combine_bwd_kernel");
    return 0;
}

int launch_combine_bwd(const Dims& d, const Workspace& w, char* ws, const void* dy, int io, cudaStream_t st)
{
    return combine_rows_backward(w, ws, dy, io, ws + w.Yg, d.C, d.k, ws + w.dYg, st);
}

int launch_bias_grads(const mgpt_moe_layer* L, const Workspace& w, char* ws, cudaStream_t st)
{
    const Dims& d = L->d;
    BiasGradArgs a;
    a.M[0] = buf_dYg(L, w, ws); a.M[1] = ws + w.dG; a.M[2] = ws + w.dU;
    a.gb[0] = L->master.gbd; a.gb[1] = L->master.gbg; a.gb[2] = L->master.gbu;
    a.cols[0] = d.C; a.cols[1] = d.H; a.cols[2] = d.H;
    a.tile_expert = (const int32_t*)(ws + w.tile_expert);
    a.n_tiles = (const int32_t*)(ws + w.n_tiles);
    const int mc = d.C > d.H ? d.C : d.H;
    dim3 grid(w.max_tiles, (mc + 255) / 256, 3);
    MGPT_CUDA(launch_pdl(bias_grad_kernel, grid, 256, 0, st, a));
    MGPT_LAUNCHED("bias_grad_kernel");
    return 0;
}

// Expert side of an expert-parallel layer: rows arrive as one block per source rank, inside it one
// 128-row-padded segment per local expert.  From the [n_src][E] real row counts this builds the tile ->
// expert table in arrival order, the per-expert segment list {first row, padded rows} and the totals.
__global__ void __launch_bounds__(256)
segment_tiles_kernel(const int32_t* seg_counts, int n_src, int E, int32_t* counts,
                     int32_t* tile_expert, int32_t* tile_order,
                     int32_t* n_tiles, int max_tiles, int32_t* seg,
                     int32_t* status, int32_t* sticky)
{
    pdl_wait();
    __shared__ int first_tile[MAX_SEGMENTS + 1];     // in arrival order (s, e)
    __shared__ int first_item[MAX_SEGMENTS];         // in processing order (e, s)
    const int n = n_src * E;
    if (threadIdx.x == 0) {
        int t = 0;
        for (int i = 0; i < n; ++i) {            // i = s*E + e, arrival order
            first_tile[i] = t;
            t += (seg_counts[i] + ROW_TILE - 1) / ROW_TILE;
        }
        first_tile[n] = t;
        *n_tiles = t;
        *status = t > max_tiles ? ST_PLAN_OVERFLOW : 0;
        if (sticky && t > max_tiles) atomicOr(sticky, ST_PLAN_OVERFLOW);
        int it = 0;
        for (int e = 0; e < E; ++e)
            for (int s_ = 0; s_ < n_src; ++s_) {
                first_item[e * n_src + s_] = it;
                it += (seg_counts[s_ * E + e] + ROW_TILE - 1) / ROW_TILE;
            }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int s_ = i / E, e = i % E;
        const int t0 = first_tile[i], t1 = first_tile[i + 1];
        seg[(e * n_src + s_) * 2] = t0 * ROW_TILE;
        seg[(e * n_src + s_) * 2 + 1] = (t1 - t0) * ROW_TILE;
        const int o0 = first_item[e * n_src + s_];
        for (int t = t0; t < t1 && t < max_tiles; ++t) {
            tile_expert[t] = e;
            // tiles are worked on expert after expert (one expert's weights stay in L2), wherever they landed
            if (o0 + (t - t0) < max_tiles) tile_order[o0 + (t - t0)] = t;
        }
    }
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        int c = 0;
        for (int s_ = 0; s_ < n_src; ++s_) c += seg_counts[s_ * E + e];
        counts[e] = c;
    }
}

int launch_segment_tiles(const Dims& d, const Workspace& w, char* ws, const int32_t* seg_counts, int n_src, cudaStream_t st,
                         int32_t* sticky)
{
    if (n_src * d.E > MAX_SEGMENTS) return fail(MGPT_MOE_EINVAL, "sources x local experts must not exceed 4096");
    MGPT_CUDA(launch_pdl(segment_tiles_kernel, 1, 256, 0, st, seg_counts, n_src, d.E, (int32_t*)(ws + w.counts),
                                            (int32_t*)(ws + w.tile_expert), (int32_t*)(ws + w.tile_order),
                                            (int32_t*)(ws + w.n_tiles), w.max_tiles, (int32_t*)(ws + w.seg),
                                            (int32_t*)(ws + w.status), sticky));
    MGPT_LAUNCHED("segment_tiles_kernel");
    return 0;
}

static int check_plan_args(const int32_t* top_idx, int n_rows, int E, const void* const* outs, int n_outs,
                           int row_cap)
{
    if (!top_idx) return fail(MGPT_MOE_EINVAL, "null top_idx");
    for (int i = 0; i < n_outs; ++i)
        if (!outs[i]) return fail(MGPT_MOE_EINVAL, "null output buffer");
    if (E <= 0 || E > MAX_EXPERTS) return fail(MGPT_MOE_EINVAL, "num_experts must be in 1..128");
    if (n_rows < 0) return fail(MGPT_MOE_EINVAL, "negative row count");
    const long long need = ((long long)n_rows + (long long)E * (ROW_TILE - 1)) / ROW_TILE * ROW_TILE;
    if (row_cap < need || row_cap % ROW_TILE) return fail(MGPT_MOE_EINVAL, "row_cap too small or not a multiple of 128");
    return 0;
}

}  // namespace mgpt

using namespace mgpt;

extern "C" size_t mgpt_moe_op_plan_scratch_bytes(int n_rows, int E)
{
    if (n_rows < 0 || E <= 0) return 0;
    const size_t blocks = n_rows > 0 ? ((size_t)n_rows + PLAN_BLOCK - 1) / PLAN_BLOCK : 1;
    return blocks * (size_t)E * sizeof(int32_t);
}

extern "C" int mgpt_moe_op_plan(const int32_t* top_idx, int n_rows, int E, int32_t* counts, int32_t* offsets,
                                int32_t* padded_offsets, int32_t* tile_expert, int32_t* n_tiles, int32_t* map,
                                int32_t* pos, int32_t* row_src, int row_cap, int32_t* status, void* scratch,
                                size_t scratch_bytes, mgpt_stream_t stream)
{
    const void* outs[] = {counts, offsets, padded_offsets, tile_expert, n_tiles, map, pos, row_src, status, scratch};
    MGPT_TRY(check_plan_args(top_idx, n_rows, E, outs, 10, row_cap));
    if (scratch_bytes < mgpt_moe_op_plan_scratch_bytes(n_rows, E))
        return fail(MGPT_MOE_ENOMEM, "scratch smaller than mgpt_moe_op_plan_scratch_bytes()");
    return run_plan_args(PlanArgs{top_idx, n_rows, E, counts, offsets, padded_offsets, tile_expert, n_tiles, row_cap / ROW_TILE, map, pos,
                                  row_src, nullptr, status, nullptr, nullptr, nullptr}, (int32_t*)scratch, (cudaStream_t)stream);
}

// ---- dispatch plan without any allocation ------------------------------------------
// Some callers cannot give the plan scratch memory of their own and cannot let the
// library allocate it either: an engine that has already handed all device memory to
// its own arena (the reference sizes its Scratchpad from a footprint predictor and
// leaves nothing over), or a step loop that must not meet cudaMalloc's device-wide
// synchronisation.  For them the per-block histogram lives in a fixed array inside the
// library image.  Every GPU that loads the library holds these 512 KiB until exit.
#define PLAN_STATIC_BLOCKS (MGPT_MOE_PLAN_NOALLOC_MAX_ROWS / 1024)
static __device__ __align__(256) int32_t g_plan_scratch[PLAN_STATIC_BLOCKS * mgpt::MAX_EXPERTS];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
int32_t* g_scratch_dev_ptr[kMaxDevices] = {};   // device address of g_plan_scratch, per device

// In host code `g_plan_scratch` names a host-side shadow, not device memory; the
// address a kernel may use has to be asked for, on the device that will run it.
int plan_static_scratch(int32_t** out)
{
    int dev = -1;
    MGPT_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(MGPT_MOE_EINVAL, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_dev_ptr[dev]) {
        void* p = nullptr;
        MGPT_CUDA(cudaGetSymbolAddress(&p, g_plan_scratch));
        if (!p) return fail(MGPT_MOE_ECUDA, "cudaGetSymbolAddress returned a null address");
        g_scratch_dev_ptr[dev] = (int32_t*)p;
    }
    *out = g_scratch_dev_ptr[dev];
    return 0;
}
}  // namespace

extern "C" int mgpt_moe_op_plan_noalloc(const int32_t* top_idx, int n_rows, int E, int32_t* counts, int32_t* offsets,
                                        int32_t* padded_offsets, int32_t* tile_expert, int32_t* n_tiles,
                                        int32_t* map, int32_t* pos, int32_t* row_src, int row_cap, int32_t* status,
                                        mgpt_stream_t stream)
{
    if (n_rows > MGPT_MOE_PLAN_NOALLOC_MAX_ROWS)
        return fail(MGPT_MOE_EINVAL, "mgpt_moe_op_plan_noalloc handles at most " +
                                         std::to_string(MGPT_MOE_PLAN_NOALLOC_MAX_ROWS) + " routed rows, got " +
                                         std::to_string(n_rows) + "; use mgpt_moe_op_plan with your own scratch");
    const void* outs[] = {counts, offsets, padded_offsets, tile_expert, n_tiles, map, pos, row_src, status};
    MGPT_TRY(check_plan_args(top_idx, n_rows, E, outs, 9, row_cap));
    int32_t* scratch = nullptr;
    MGPT_TRY(plan_static_scratch(&scratch));
    // The array still holds the previous call's block bases.  Nothing has to be cleared:
    // plan_count_kernel writes all plan_blocks*E entries this call reads before they are read.
    return run_plan_args(PlanArgs{top_idx, n_rows, E, counts, offsets, padded_offsets, tile_expert, n_tiles, row_cap / ROW_TILE, map, pos,
                                  row_src, nullptr, status, nullptr, nullptr, nullptr}, scratch, (cudaStream_t)stream);
}
