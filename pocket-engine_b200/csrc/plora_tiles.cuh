// Tensor-core tiles of the cluster kernel's expand (one kernel per layer): S as bf16 terms in shared memory times rows of B in
// shared memory, y updated in global memory. Tiles of the warp-level instruction (m16n8k16, bf16 in, f32 accumulate); the
// f32 intermediate enters as three bf16 terms (high, middle, low part), whose products with bf16 B are exact in
// f32, so no precision is given up against an f32 multiply-add chain.
#pragma once
#include <cuda_bf16.h>

#include <type_traits>

#include "plora_device.cuh"

#define PLORA_TILE_WARPS 8  // warps of a block that share the columns of an expand

namespace {

typedef __nv_bfloat16 bf16;

// four 8x8 bf16 matrices from shared memory: lane l gives the address of row (l % 8) of matrix l / 8
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// D (16 x 8, f32) += A (16 x 16, bf16, row-major) . B (16 x 8, bf16, column-major)
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// y of one 16-column step: the lane's two token rows (g and g + 8) times its two column pairs
template <bool F32>
struct YStep {
    float2 v[2][2];
};

// One part's share of the output columns: y[tok, off + lo + c] += S3[tok, r_off ..] . B[c, :]^T for c in [0, ncols).
// NK: 16-wide steps over the part's rank held as fragments in registers (0: fetched from shared memory per step).
template <int NK, bool F32>
__device__ __forceinline__ void expand_part(uint32_t s3_part, uint32_t plane_bytes, uint32_t bs_lane, int r, int ncols,
                                            void* Y, int ldy, size_t ybase, int tok0, int tok1, int warp, int t2) {
    typedef typename std::conditional<F32, float, bf16>::type ytype;
    const int nk = NK > 0 ? NK : r >> 4;
    uint32_t sa[NK > 0 ? NK : 1][3][4];
    if (NK > 0) {
#pragma unroll
        for (int ks = 0; ks < NK; ks++)
#pragma unroll
            for (int pl = 0; pl < 3; pl++) ldmatrix_x4(sa[ks][pl], s3_part + (uint32_t)pl * plane_bytes + (uint32_t)ks * 32u);
    }
    ytype* y0 = tok0 >= 0 ? reinterpret_cast<ytype*>(Y) + (size_t)tok0 * ldy + ybase + t2 : nullptr;
    ytype* y1 = tok1 >= 0 ? reinterpret_cast<ytype*>(Y) + (size_t)tok1 * ldy + ybase + t2 : nullptr;
    auto load = [&](YStep<F32>& q, int c) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const ytype* yp = h ? y1 : y0;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                if (yp != nullptr && c + n * 8 + t2 < ncols) {
                    if (F32) q.v[h][n] = *reinterpret_cast<const float2*>(yp + c + n * 8);
                    else q.v[h][n] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(yp + c + n * 8));
                }
            }
        }
    };
    // 16 columns (two tiles of 8) per step; warp q takes the steps q, q + 8, ...; y is fetched two steps ahead
    int c = warp * 16;
    YStep<F32> q0, q1, q2;
    load(q0, c);
    load(q1, c + PLORA_TILE_WARPS * 16);
    for (; c < ncols; c += PLORA_TILE_WARPS * 16) {
        load(q2, c + 2 * PLORA_TILE_WARPS * 16);
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < (NK > 0 ? NK : 8); ks++) {
            if (ks < nk) {
                uint32_t bb[4];
                ldmatrix_x4(bb, bs_lane + (uint32_t)c * (uint32_t)r * 2u + (uint32_t)ks * 32u);
                // low, middle, high term: the small ones first
#pragma unroll
                for (int pl = 2; pl >= 0; pl--) {
                    if (NK > 0) {
                        mma_16816(d0, sa[ks][pl], bb[0], bb[1]);
                        mma_16816(d1, sa[ks][pl], bb[2], bb[3]);
                    } else {
                        uint32_t st[4];
                        ldmatrix_x4(st, s3_part + (uint32_t)pl * plane_bytes + (uint32_t)ks * 32u);
                        mma_16816(d0, st, bb[0], bb[1]);
                        mma_16816(d1, st, bb[2], bb[3]);
                    }
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            ytype* yp = h ? y1 : y0;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                if (yp != nullptr && c + n * 8 + t2 < ncols) {
                    const float* d = n ? d1 : d0;
                    const float v0 = q0.v[h][n].x + d[2 * h], v1 = q0.v[h][n].y + d[2 * h + 1];
                    if (F32) *reinterpret_cast<float2*>(yp + c + n * 8) = make_float2(v0, v1);
                    else *reinterpret_cast<__nv_bfloat162*>(yp + c + n * 8) = __floats2bfloat162_rn(v0, v1);
                }
            }
        }
        q0 = q1;
        q1 = q2;
    }
}

// Four adjacent columns of one token's y
template <bool F32>
struct YQuad;
template <>
struct YQuad<true> {
    float4 v;
    __device__ __forceinline__ void clear() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load(const void* p) { v = __ldcg(reinterpret_cast<const float4*>(p)); }
    __device__ __forceinline__ void add_to(void* p, const float (&d)[4]) const {
        *reinterpret_cast<float4*>(p) = make_float4(v.x + d[0], v.y + d[1], v.z + d[2], v.w + d[3]);
    }
};
template <>
struct YQuad<false> {
    uint2 v;
    __device__ __forceinline__ void clear() { v = make_uint2(0u, 0u); }
    __device__ __forceinline__ void load(const void* p) { v = __ldcg(reinterpret_cast<const uint2*>(p)); }
    __device__ __forceinline__ void add_to(void* p, const float (&d)[4]) const {
        const __nv_bfloat162 a = __floats2bfloat162_rn(__uint_as_float(v.x << 16) + d[0], __uint_as_float(v.x & 0xffff0000u) + d[1]);
        const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(v.y << 16) + d[2], __uint_as_float(v.y & 0xffff0000u) + d[3]);
        *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
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
template <RankWalk W, bool F32, int STEPS>
__device__ __forceinline__ void quad_step(const uint4& sa0, const uint4& sa1, uint32_t a0, uint32_t a1, uint32_t b, const uint32_t (&brow)[4],
                                          uint32_t step_bytes, int r, bool upper, bool swap, const YQuad<F32> (&y)[STEPS], unsigned char* yp,
                                          const bool (&live)[STEPS], uint32_t ystep) {
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
        if (live[i]) y[i].add_to(yp + (size_t)i * ystep, o);
    }
}

// The same for up to four tokens tok[0..n_tok) whose y rows can move in whole pieces (the common decoding case): 32 columns per
// step, at 16 ranks a walk and bf16 two steps at a time (a step is a chain of latencies, and a few warps per scheduler do not
// cover it). The B rows are fed to the step's four tiles in an order that leaves a lane and its partner with 8 adjacent
// columns of their token row: y is read and written in pieces of 4 columns, 64 contiguous bytes per row and instruction (bf16).
// In shared memory that order would put four of a tile's eight rows on the same banks where the rank is an odd multiple of 16:
// there the lanes of odd t take the tiles 1, 0, 3, 2 (64 tokens of 16 adapters, 16 layers: 101 us through four-matrix loads of that
// order, 95 so).
// y0, y1: this lane's y of the first two steps, if `have`. Few registers beside those of a step: whatever spills goes to L2 and back,
// since these kernels leave L1 no room.
template <RankWalk W, bool F32>
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
    int left = ncols - warp * 32;  // columns from this warp's step on; the lane's four are there if left > mycol
    YQuad<F32> q[2], n[2];
    auto fetch = [&](YQuad<F32>& y, int ahead) {
        y.clear();
        if (live && left > ahead + mycol) y.load(yp + ahead * ES);
    };
    if (have) {
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
            const bool on[2] = {live, live && left > WIDE + mycol};
            quad_step<W, F32, 2>(sa0, sa1, a0, a1, b, brow, WIDE * r2, r, upper, swap, q, yp, on, WIDE * ES);
            b += 2 * WIDE * r2;
            yp += 2 * WIDE * ES;
            q[0] = n[0];
            q[1] = n[1];
        }
    }
    for (; left > 0; left -= WIDE) {  // the last one, or all of them where they do not go in pairs
        if (!PAIRS) fetch(n[0], 2 * WIDE);
        const bool on[1] = {live && left > mycol};
        YQuad<F32> one[1] = {q[0]};
        quad_step<W, F32, 1>(sa0, sa1, a0, a1, b, brow, 0u, r, upper, swap, one, yp, on, 0u);
        b += WIDE * r2;
        yp += WIDE * ES;
        q[0] = q[1];
        q[1] = n[0];
    }
}

}  // namespace
