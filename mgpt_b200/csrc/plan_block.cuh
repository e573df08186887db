// The dispatch plan of up to 1024 routed rows by one thread block (plan.cu states what a plan is): histogram, prefix sums,
// tile and row-group lists and the stable slot assignment without leaving the SM.  Run by a kernel of its own, or by the
// last block of the router.
#pragma once

#include "common.cuh"

namespace mgpt {

constexpr int PLAN_BLOCK = 1024;            // flat indices one block plans
constexpr int PLAN_SEGS = PLAN_BLOCK / 32;  // in segments of one warp's width

struct PlanArgs {
    const int32_t* top_idx;
    int R, E;
    int32_t *counts, *offsets, *padded_offsets, *tile_expert, *n_tiles;
    int max_tiles;
    int32_t *map, *pos, *row_src, *slot_of, *status, *sticky;
    int4* groups;           // null: no decode kernels follow
    int32_t* n_groups;
};

struct PlanShared {
    int seg[PLAN_SEGS][MAX_EXPERTS];        // rows of an expert in a segment, then in the segments before it
    int tot[MAX_EXPERTS], off[MAX_EXPERTS], poff[MAX_EXPERTS + 1], goff[MAX_EXPERTS];
    int bad;
};

// Exclusive sums over the experts by one warp, lane l having experts 4l .. 4l+3: first compact slot, first row tile, first
// row group; and the totals of the last two.
__device__ __forceinline__ void plan_scan_experts(const int* tot, int E, int lane, int* off, int* tile0, int* group0, int& n_tiles, int& n_groups)
{
    int o = 0, t = 0, g = 0, v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[j] = 4 * lane + j < E ? tot[4 * lane + j] : 0;
        o += v[j];
        t += (v[j] + ROW_TILE - 1) / ROW_TILE;
        g += (v[j] + DECODE_GROUP - 1) / DECODE_GROUP;
    }
    const int o0 = o, t0 = t, g0 = g;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, o, d), b = __shfl_up_sync(0xffffffffu, t, d), c = __shfl_up_sync(0xffffffffu, g, d);
        if (lane >= d) { o += a; t += b; g += c; }
    }
    n_tiles = __shfl_sync(0xffffffffu, t, 31);
    n_groups = __shfl_sync(0xffffffffu, g, 31);
    o -= o0; t -= t0; g -= g0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int x = 4 * lane + j;
        if (x < E) { off[x] = o; tile0[x] = t; group0[x] = g; }
        o += v[j];
        t += (v[j] + ROW_TILE - 1) / ROW_TILE;
        g += (v[j] + DECODE_GROUP - 1) / DECODE_GROUP;
    }
}

// WARPS warps of one block, all of them; top_idx may have been written by other blocks of the same kernel (read past L1).
template <int WARPS>
__device__ __forceinline__ void plan_block(const PlanArgs& p, PlanShared& sh)
{
    constexpr int PER = (PLAN_SEGS + WARPS - 1) / WARPS, THREADS = 32 * WARPS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int segs = (p.R + 31) >> 5;
    for (int i = tid; i < segs * MAX_EXPERTS; i += THREADS) (&sh.seg[0][0])[i] = 0;
    if (tid == 0) sh.bad = 0;
    int e[PER], rank[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = (warp + j * WARPS) * 32 + lane;
        e[j] = i < p.R ? __ldcg(p.top_idx + i) : 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int s = warp + j * WARPS;
        rank[j] = 0;
        if (s < segs) {                                               // warp-uniform
            const bool row = s * 32 + lane < p.R;
            const bool known = (unsigned)e[j] < (unsigned)p.E;
            if (row && !known) sh.bad = 1;                            // an id no expert has: no slot, and the caller is told
            if (!row || !known) e[j] = -1 - lane;                     // distinct keys for lanes without a row
            const unsigned peers = __match_any_sync(0xffffffffu, e[j]);
            rank[j] = __popc(peers & ((1u << lane) - 1u));
            if (e[j] >= 0 && rank[j] == 0) sh.seg[s][e[j]] = __popc(peers);
        }
    }
    __syncthreads();
    for (int x = tid; x < p.E; x += THREADS) {
        int run = 0;
        for (int s = 0; s < segs; ++s) {
            const int c = sh.seg[s][x];
            sh.seg[s][x] = run;
            run += c;
        }
        sh.tot[x] = run;
        p.counts[x] = run;
    }
    __syncthreads();
    if (warp == 0) {
        int nt, ng;
        plan_scan_experts(sh.tot, p.E, lane, sh.off, sh.poff, sh.goff, nt, ng);
        __syncwarp();
        for (int x = lane; x < p.E; x += 32) {
            sh.poff[x] *= ROW_TILE;
            p.offsets[x] = sh.off[x];
            p.padded_offsets[x] = sh.poff[x];
        }
        if (lane == 0) {
            sh.poff[p.E] = nt * ROW_TILE;
            p.padded_offsets[p.E] = nt * ROW_TILE;
            *p.n_tiles = nt;
            if (p.groups) *p.n_groups = ng;
            const int st = (nt > p.max_tiles ? ST_PLAN_OVERFLOW : 0) | (sh.bad ? ST_BAD_EXPERT : 0);
            *p.status = st;
            if (p.sticky && st) atomicOr(p.sticky, st);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int s = warp + j * WARPS, i = s * 32 + lane;
        if (s < segs && e[j] >= 0) {
            const int r = sh.seg[s][e[j]] + rank[j];
            const int slot = sh.off[e[j]] + r, q = sh.poff[e[j]] + r;
            p.map[slot] = i;
            p.pos[i] = q;
            p.row_src[q] = i;
            if (p.slot_of) p.slot_of[i] = slot;
        }
    }
    for (int x = tid; x < p.E; x += THREADS) {
        for (int t = sh.poff[x] / ROW_TILE; t < sh.poff[x + 1] / ROW_TILE && t < p.max_tiles; ++t) p.tile_expert[t] = x;
        if (p.groups)
            for (int g = 0; g * DECODE_GROUP < sh.tot[x]; ++g)
                p.groups[sh.goff[x] + g] = make_int4(x, sh.poff[x] + g * DECODE_GROUP, min(DECODE_GROUP, sh.tot[x] - g * DECODE_GROUP), 0);
    }
    // padding rows: the end of an expert's last tile
    for (int x = warp; x < p.E; x += WARPS) {
        const int end = sh.poff[x + 1];
#pragma unroll
        for (int i = 0; i < ROW_TILE / 32; ++i) {
            const int q = end - ROW_TILE + 32 * i + lane;
            if (q >= sh.poff[x] + sh.tot[x]) p.row_src[q] = -1;
        }
    }
}

}  // namespace mgpt
