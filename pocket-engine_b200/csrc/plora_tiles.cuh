// Tensor-core tiles of the cluster kernel's expand (one kernel per layer): S as bf16 terms in shared memory times rows of B in
// shared memory, y updated in global memory. Tiles of the warp-level instruction (m16n8k16, bf16 in, f32 accumulate); the
// f32 intermediate enters as three bf16 terms (high, middle, low part), whose products with bf16 B are exact in
// f32, so no precision is given up against an f32 multiply-add chain.
#pragma once
#include <cuda_bf16.h>

#include "plora_device.cuh"

#define PLORA_TILE_WARPS 8  // warps of a block that share the columns of an expand

namespace {

typedef __nv_bfloat16 bf16;

// D (16 x 8, f32) += A (16 x 16, bf16, row-major) . B (16 x 8, bf16, column-major)
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Four adjacent columns of one token's y. load, add_to: as one aligned piece; the _pairs forms: the first `n` of them (2 or 4: widths
// and pitches are even) in pieces of two, for shares or rows of y that do not come in aligned pieces of four
template <bool F32>
struct YQuad;
template <>
struct YQuad<true> {
    float4 v;
    __device__ __forceinline__ void clear() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load(const void* p) { v = __ldcg(reinterpret_cast<const float4*>(p)); }
    __device__ __forceinline__ void load_pairs(const void* p, int n) {
        const float2 a = __ldcg(reinterpret_cast<const float2*>(p));
        v.x = a.x, v.y = a.y;
        if (n > 2) {
            const float2 b = __ldcg(reinterpret_cast<const float2*>(p) + 1);
            v.z = b.x, v.w = b.y;
        }
    }
    __device__ __forceinline__ void add_to(void* p, const float (&d)[4]) const {
        *reinterpret_cast<float4*>(p) = make_float4(v.x + d[0], v.y + d[1], v.z + d[2], v.w + d[3]);
    }
    __device__ __forceinline__ void add_to_pairs(void* p, const float (&d)[4], int n) const {
        *reinterpret_cast<float2*>(p) = make_float2(v.x + d[0], v.y + d[1]);
        if (n > 2) *(reinterpret_cast<float2*>(p) + 1) = make_float2(v.z + d[2], v.w + d[3]);
    }
};
template <>
struct YQuad<false> {
    uint2 v;
    __device__ __forceinline__ void clear() { v = make_uint2(0u, 0u); }
    __device__ __forceinline__ void load(const void* p) { v = __ldcg(reinterpret_cast<const uint2*>(p)); }
    __device__ __forceinline__ void load_pairs(const void* p, int n) {
        v.x = __ldcg(reinterpret_cast<const uint32_t*>(p));
        if (n > 2) v.y = __ldcg(reinterpret_cast<const uint32_t*>(p) + 1);
    }
    __device__ __forceinline__ uint2 plus(const float (&d)[4]) const {
        const __nv_bfloat162 a = __floats2bfloat162_rn(__uint_as_float(v.x << 16) + d[0], __uint_as_float(v.x & 0xffff0000u) + d[1]);
        const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(v.y << 16) + d[2], __uint_as_float(v.y & 0xffff0000u) + d[3]);
        return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
    __device__ __forceinline__ void add_to(void* p, const float (&d)[4]) const { *reinterpret_cast<uint2*>(p) = plus(d); }
    __device__ __forceinline__ void add_to_pairs(void* p, const float (&d)[4], int n) const {
        const uint2 o = plus(d);
        *reinterpret_cast<uint32_t*>(p) = o.x;
        if (n > 2) *(reinterpret_cast<uint32_t*>(p) + 1) = o.y;
    }
};

// How a part's rank is walked. Lane t of four holds 4 t .. 4 t + 3 of 16 ranks (one multiply) or 8 t .. 8 t + 7 of 32 (two): the
// multiply's 16 input slots may be permuted freely as long as both operands agree, and operands are then plain loads of 8 or 16
// bytes. A rank that is an odd multiple of 16 goes 16 at a time (R16: 16 itself, its operand of S in registers; ODD: any), the
// others 32 at a time (R32, EVEN).
enum RankWalk { R16, ODD, R32, EVEN };

// The steps of 32 columns c and, with STEPS 2, c + 256 for four tokens. The 16 rows of a
// token tile are four tokens' high, middle and low terms of S and four rows of zeros, so the three terms take one multiply per
// 8-column tile. A lane holds one term's 8 columns of one token (rows g and g + 8: high + low, or middle + zero); with the
// lane 16 further on it trades half of them, and each adds up and moves 4 columns.
// brow: bytes of this lane's rows of B in the tiles 0..3 from row 0 of the step on; swap: its tiles come in the order 1, 0, 3, 2.
// have: how many of the lane's four columns there are in each step (WHOLE: whether).
template <RankWalk W, bool F32, bool WHOLE, int STEPS>
__device__ __forceinline__ void quad_step(const uint4& sa0, const uint4& sa1, uint32_t a0, uint32_t a1, uint32_t b, const uint32_t (&brow)[4],
                                          uint32_t step_bytes, int r, bool upper, bool swap, const YQuad<F32> (&y)[STEPS], unsigned char* yp,
                                          const int (&have)[STEPS], uint32_t ystep) {
    constexpr bool BY16 = W == R16 || W == ODD;
    float d[STEPS][4][4];
#pragma unroll
    for (int i = 0; i < STEPS; i++)
#pragma unroll
        for (int n = 0; n < 4; n++) d[i][n][0] = d[i][n][1] = d[i][n][2] = d[i][n][3] = 0.f;
    auto walk = [&](uint32_t at) {  // the ranks whose bytes in a row are at, at + 1, ...
        uint4 lo = sa0, hi = sa1;   // rows g and g + 8 of the token tile
        if (W == ODD) {
            const uint2 u = lds64(a0 + at), v = lds64(a1 + at);
            lo = make_uint4(u.x, u.y, 0u, 0u);
            hi = make_uint4(v.x, v.y, 0u, 0u);
        } else if (W == EVEN) {
            lo = lds128(a0 + at);
            hi = lds128(a1 + at);
        }
        const uint32_t m0[4] = {lo.x, hi.x, lo.y, hi.y}, m1[4] = {lo.z, hi.z, lo.w, hi.w};
        if (BY16) {
            uint2 bv[STEPS][4];
#pragma unroll
            for (int s = 0; s < STEPS; s++)
#pragma unroll
                for (int n = 0; n < 4; n++) bv[s][n] = lds64(b + brow[n] + (uint32_t)s * step_bytes + at);
#pragma unroll
            for (int s = 0; s < STEPS; s++)
#pragma unroll
                for (int n = 0; n < 4; n++) mma_16816(d[s][n], m0, bv[s][n].x, bv[s][n].y);
        } else {
#pragma unroll
            for (int s = 0; s < STEPS; s++) {
                uint4 bv[4];
#pragma unroll
                for (int n = 0; n < 4; n++) bv[n] = lds128(b + brow[n] + (uint32_t)s * step_bytes + at);
#pragma unroll
                for (int n = 0; n < 4; n++) mma_16816(d[s][n], m0, bv[n].x, bv[n].y);
#pragma unroll
                for (int n = 0; n < 4; n++) mma_16816(d[s][n], m1, bv[n].z, bv[n].w);
            }
        }
    };
    if (W == R16 || W == R32) walk(0u);
    else
#pragma unroll 1
        for (int k = 0; k < r; k += BY16 ? 16 : 32) walk((uint32_t)k * 2u);
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float f = d[i][e >> 1][e & 1] + d[i][e >> 1][2 + (e & 1)], h = d[i][2 + (e >> 1)][e & 1] + d[i][2 + (e >> 1)][2 + (e & 1)];
            const float got = __shfl_xor_sync(0xffffffffu, upper ? f : h, 16);
            o[e] = (upper ? h : f) + got;
        }
        if (BY16) {
            const float t0 = o[0], t1 = o[1];
            o[0] = swap ? o[2] : o[0];
            o[1] = swap ? o[3] : o[1];
            o[2] = swap ? t0 : o[2];
            o[3] = swap ? t1 : o[3];
        }
        if (have[i] > 0) {
            if (WHOLE) y[i].add_to(yp + (size_t)i * ystep, o);
            else y[i].add_to_pairs(yp + (size_t)i * ystep, o, have[i]);
        }
    }
}

// The same for up to four tokens tok[0..n_tok) over all columns of a share: 32 columns per step, at 16 ranks a walk and bf16 two steps at a time (a step is a chain of latencies, and a few warps per scheduler do not
// cover it). The B rows are fed to the step's four tiles in an order that leaves a lane and its partner with 8 adjacent
// columns of their token row: y is read and written in pieces of 4 columns, 64 contiguous bytes per row and instruction (bf16).
// In shared memory that order would put four of a tile's eight rows on the same banks where the rank is an odd multiple of 16:
// there the lanes of odd t take the tiles 1, 0, 3, 2 (64 tokens of 16 adapters, 16 layers: 101 us through four-matrix loads of that
// order, 95 so).
// WHOLE: y moves in aligned pieces of four columns (the common case). Otherwise in pairs; nothing else differs, so that a column's
// sum is the same whichever way its share is cut. y0, y1: this lane's y of the first two steps, if `have` (WHOLE). Few registers beside those of a step: whatever spills goes to L2 and back,
// since these kernels leave L1 no room.
template <RankWalk W, bool F32, bool WHOLE>
__device__ __forceinline__ void expand_quads(uint32_t s3, uint32_t sp_pad, uint32_t plane_bytes, uint32_t b, int r, int ncols, void* Y, int ldy,
                                             size_t ycol, const int* tok, int n_tok, int warp, int lane, bool have, const YQuad<F32>& y0, const YQuad<F32>& y1) {
    constexpr int ES = F32 ? 4 : 2;
    constexpr bool BY16 = W == R16 || W == ODD;
    constexpr bool PAIRS = BY16 && !F32;         // (f32 pieces of two steps and the next two take too many registers)
    constexpr int WIDE = PLORA_TILE_WARPS * 32;  // columns between a warp's steps
    if (W == R16) r = 16;
    if (W == R32) r = 32;
    const int g = lane >> 2, t4 = lane & 3, qtok = g & 3;
    const bool upper = g >= 4, swap = (t4 & 1) != 0, live = qtok < n_tok;
    const uint32_t r2 = (uint32_t)r * 2u, piece = (uint32_t)t4 * (BY16 ? 8u : 16u);
    // row i of the token tile: term i / 4 of token i % 4
    const uint32_t a0 = s3 + (upper ? plane_bytes : 0u) + (uint32_t)qtok * sp_pad + piece, a1 = a0 + 2u * plane_bytes;
    uint4 sa0 = make_uint4(0u, 0u, 0u, 0u), sa1 = sa0;
    if (W == R16) {
        const uint2 u = lds64(a0), v = lds64(a1);
        sa0 = make_uint4(u.x, u.y, 0u, 0u);
        sa1 = make_uint4(v.x, v.y, 0u, 0u);
    } else if (W == R32) {
        sa0 = lds128(a0);
        sa1 = lds128(a1);
    }
    // row j of tile n is column 8 (j / 2) + 2 n + (j % 2) of the step, n ^ 1 in place of n where j / 2 is odd (BY16)
    uint32_t brow[4];
#pragma unroll
    for (int n = 0; n < 4; n++) brow[n] = (uint32_t)(8 * (g >> 1) + 2 * (BY16 ? n ^ ((g >> 1) & 1) : n) + (g & 1)) * r2;
    b += (uint32_t)(warp * 32) * r2 + piece;
    const int mycol = 8 * t4 + (upper ? 4 : 0);
    unsigned char* yp = reinterpret_cast<unsigned char*>(Y) + ((size_t)(live ? tok[qtok] : 0) * ldy + ycol + mycol + warp * 32) * ES;
    int left = ncols - warp * 32;  // columns from this warp's step on
    auto mine = [&](int ahead) {  // ... of this lane's four (none if not above 0)
        if (WHOLE) return (int)(live && left > ahead + mycol);
        return live ? min(4, left - ahead - mycol) : 0;
    };
    YQuad<F32> q[2], n[2];
    auto fetch = [&](YQuad<F32>& y, int ahead) {
        y.clear();
        const int have = mine(ahead);
        if (have > 0) {
            if (WHOLE) y.load(yp + ahead * ES);
            else y.load_pairs(yp + ahead * ES, have);
        }
    };
    if (WHOLE && have) {
        q[0] = y0;
        q[1] = y1;
    } else {
        fetch(q[0], 0);
        fetch(q[1], WIDE);
    }
    if (PAIRS) {
        for (; left > WIDE; left -= 2 * WIDE) {
            fetch(n[0], 2 * WIDE);
            fetch(n[1], 3 * WIDE);
            const int on[2] = {mine(0), mine(WIDE)};
            quad_step<W, F32, WHOLE, 2>(sa0, sa1, a0, a1, b, brow, WIDE * r2, r, upper, swap, q, yp, on, WIDE * ES);
            b += 2 * WIDE * r2;
            yp += 2 * WIDE * ES;
            q[0] = n[0];
            q[1] = n[1];
        }
    }
    for (; left > 0; left -= WIDE) {  // the last one, or all of them where they do not go in pairs
        if (!PAIRS) fetch(n[0], 2 * WIDE);
        const int on[1] = {mine(0)};
        YQuad<F32> one[1] = {q[0]};
        quad_step<W, F32, WHOLE, 1>(sa0, sa1, a0, a1, b, brow, 0u, r, upper, swap, one, yp, on, 0u);
        b += WIDE * r2;
        yp += WIDE * ES;
        q[0] = q[1];
        q[1] = n[0];
    }
}

}  // namespace
