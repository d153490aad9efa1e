// Tensor-core tile path for long runs of contiguous tokens of one slot (prefill segments): tcgen05.mma with
// the accumulator in tensor memory, 128 tokens per tile.
//
//   plora_shrink_mma_kernel  S[128, R] = X[128, K] . A_slot[R, K]^T   x tiles and slab tiles by TMA (128-byte
//                            swizzle) from a producer thread, MMAs from another, a ring of stages, f32 in TMEM
//   plora_expand_mma_kernel  y[128, 128-column block] += S[128, r] . B_p[block, r]^T   S split into a bf16 high
//                            and low part (two accumulating MMAs, so S keeps ~16 bits of mantissa), operands in
//                            the unswizzled core-matrix layout, y read-modify-written from registers
//
// Every wait is bounded (mbar_wait); on a timeout the block records PLORA_ERR_TIMEOUT, frees its tensor
// memory and leaves. Replaces the reference's mma.sync tiles of 16 tokens (src/kernels/lora.cuh:23-126).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "plora_internal.h"
#include "plora_device.cuh"
#include "plora_tc.cuh"

typedef __nv_bfloat16 bf16;

namespace {

// ---- tcgen05 ----

// D (tensor memory) (+)= A (tensor memory: lane = row, two bf16 per column) . B (shared), f32 accumulate
__device__ __forceinline__ void umma_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
// 8 consecutive columns of this warp's 32 lanes; to be followed by tmem_st_wait
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 8 consecutive columns, without the wait (several loads, then one tmem_ld_wait)
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

// v[0] = balanced binary tree sum of v[0..n), n a power of two <= 8 (W values per item)
template <int W>
__device__ __forceinline__ void tree_sum(float (&v)[PLORA_TILE_SPLIT_MAX][W], int n) {
#pragma unroll
    for (int stride = 1; stride < PLORA_TILE_SPLIT_MAX; stride <<= 1)
#pragma unroll
        for (int a = 0; a < PLORA_TILE_SPLIT_MAX; a += 2 * stride)
            if (a + stride < n)
#pragma unroll
                for (int q = 0; q < W; q++) v[a][q] += v[a + stride][q];
}

// Instruction descriptor, kind::f16: f32 accumulator, bf16 A and B, both K-major, M rows by N columns.
__device__ __forceinline__ uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const uint32_t n = valid ? 16u : 0u;  // a zero source size fills the 16 bytes with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Makes a tensor map that sits in global memory (written by a copy earlier in the stream) visible to this
// thread's tensor copies.
__device__ __forceinline__ void tmap_acquire(const CUtensorMap* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
}

#define MMA_M 128
#define EXP_TPAD 66  // floats per row of the epilogue's transpose tile (64 columns + 2 of padding)

// ------------------------------------------------------------------------------------------------------
// Shrink of one 128-token tile. Grid (split, rank groups, tiles); 128 threads. The slot's K chunks (plora_tile_chunks) are
// shared evenly by min(split, chunks) blocks; each block accumulates its chunks in separate accumulators, adds
// them as a tree and writes plane blockIdx.x of S. K is walked in steps of 64 inputs through a ring of stages
// with two roles and no block-wide synchronisation in the loop: one thread of warp 0 issues, per step, the x
// tile and the slab's rows for the same 64 inputs as tensor copies (both in the 128-byte swizzle; the slab
// through the tensor map plora_upload encoded for the slot), waiting for a stage's MMAs before it refills it;
// one thread of warp 1 waits for a stage to land, issues its MMAs and commits them to the stage's "empty"
// barrier. Once the last MMAs are complete the f32 result leaves tensor memory one token row per thread.
#define SHR_KSTEP 64
#define SHR_X_BYTES (MMA_M * SHR_KSTEP * 2)
#define SHR_MAX_STAGES 8
// A block walks its K ranges at the rate at which copies of 128-byte rows arrive at one SM (0.3 us per 64 inputs for x and 64
// rows of A, 0.5 us with 192 rows, 0.9 with 384), and a total rank over 256 leaves K a single range, since accumulators
// share tensor memory. So where a step's tiles, 128 rows each, leave SMs idle, the rows of A go to one block for each SHR_GROUP of them
// (RSPLIT); x is then read again for each group, from L2, which a step with tiles for every SM could not afford. The sums of
// an element stay the same. 300 tokens, 4 layers: rank 64 169 -> 149 us, rank 128 262 -> 183 us; 2,000 tokens of one
// adapter: rank 64 228 -> 213 us, rank 128 327 -> 259 us.
#define SHR_GROUP PLORA_TILE_GROUP

template <bool RSPLIT>
__global__ void __launch_bounds__(128) plora_shrink_mma_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                const PloraSlabMaps* __restrict__ smaps, int K,
                                                                const int* __restrict__ segs, SegLayout lay,
                                                                const plora_desc* __restrict__ table,
                                                                float* __restrict__ S, size_t s_stride, int lds,
                                                                int ksplit, int fit, int nstage, int stage_bytes, int sub,
                                                                int late, int* __restrict__ status) {
    // late != 0: the kernel launched right before this one is the same layer's gather shrink, whose blocks let
    // this grid start only after they have themselves waited for the kernels before (or whose caller vouches
    // that x is older than those). x is then complete when this grid starts, the gather shrink writes other
    // rows of S, and only this grid's stores have to come after the dependency wait: the whole main loop runs
    // beside the gather shrink instead of behind it.
    // `sub` steps of 64 inputs share a stage (1 or 2): with two, a token row's two adjacent 128-byte pieces are
    // requested together. A stage is then [x box][x box][slab box][slab box] and stage_bytes covers all of it.
    extern __shared__ unsigned char dsm_raw[];
    __shared__ __align__(8) uint64_t full[SHR_MAX_STAGES], empty[SHR_MAX_STAGES], acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int tile = blockIdx.z;
    const int n_mma = segs[SEG_N_MMA];
    const int* mt = segs + lay.mma() + 3 * tile;
    const int start = mt[0], len = mt[1], slot = mt[2];
    if (tile >= n_mma) return pdl_exit_idle();
    const plora_desc& d = table[slot];
    const int R_all = d.rank;
    // this block's rows of the stacked A: all of them, or SHR_GROUP from r0 on
    const int r0 = RSPLIT ? (int)blockIdx.y * SHR_GROUP : 0, R = RSPLIT ? SHR_GROUP : R_all;
    const int R_out = RSPLIT ? min(SHR_GROUP, R_all - r0) : R_all;
    if (R_out <= 0) return pdl_exit_idle();
    const int n_chunks = plora_tile_chunks(K, R_all);
    const int s_eff = plora_tile_blocks(ksplit, fit, n_mma, K, R_all);
    if ((int)blockIdx.x >= s_eff) return pdl_exit_idle();
    const int n_acc = n_chunks / s_eff;  // accumulators (chunks) of this block
    const CUtensorMap* amap = reinterpret_cast<const CUtensorMap*>(RSPLIT ? &smaps[slot].a64 : &smaps[slot].a);
    const int tid = threadIdx.x, warp = tid >> 5;
    // 1024-byte aligned stage ring: [x tile 16 KB][slab rows R x 128 B]
    unsigned char* ring = dsm_raw + ((1024u - (smem_u32(dsm_raw) & 1023u)) & 1023u);
    const uint32_t acc_cols = (uint32_t)plora_tile_cols(R);
    const uint32_t ncols = acc_cols * (uint32_t)n_acc;
    if (tid == 0) {
        for (int i = 0; i < nstage; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&acc_bar, 1);
        mbar_fence_init();
        s_fail = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_slot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int nk_all = (K + SHR_KSTEP - 1) / SHR_KSTEP;
    const int spc = (nk_all + n_chunks - 1) / n_chunks;  // steps per chunk
    const int k_first = (int)blockIdx.x * n_acc * spc;
    const int nk1 = min(nk_all, k_first + n_acc * spc) - k_first;  // this block's steps of 64 inputs
    const int nk = (nk1 + sub - 1) / sub;                          // and its stages
    const uint32_t a_box_bytes = (uint32_t)R * 128u;
    // the slab's rows arrive as one box of R rows, or two of R / 2 when R is over the 256-row limit of a box
    const int nbox = R > 256 ? 2 : 1, box_rows = R / nbox;
    if (!late) pdl_wait();  // x comes from the kernels before
    pdl_trigger();

    if (warp == 0) {
        // producer: one thread feeds the ring, waiting for a stage's MMAs before refilling it
        if (elect_one()) {
            tmap_acquire(amap);
            // (both role threads are single threads whose instruction latencies are on the critical path: stage
            // index, barrier parity and chunk position are carried along instead of divided out every step)
            int st = 0;
            uint32_t par = 0;  // parity of the "empty" phase to wait for, from the ring's second round on
            bool round2 = false;
            int k0 = k_first * SHR_KSTEP;
            const uint32_t tx = (uint32_t)sub * (SHR_X_BYTES + a_box_bytes);
            for (int ks = 0; ks < nk; ks++) {
                if (ks >= nstage && !mbar_wait(&empty[st], par, status)) {
                    s_fail = 1;
                    break;
                }
                unsigned char* xs = ring + (size_t)st * stage_bytes;
                unsigned char* as = xs + (size_t)sub * SHR_X_BYTES;
                mbar_expect_tx(&full[st], tx);
                for (int u = 0; u < sub; u++)  // a step past the block's range reads zeros or unused columns
                    tma_load_2d(xs + (size_t)u * SHR_X_BYTES, &xmap, k0 + u * SHR_KSTEP, start, &full[st]);
                for (int u = 0; u < sub; u++)
                    for (int b = 0; b < nbox; b++)
                        tma_load_2d(as + (size_t)u * a_box_bytes + (size_t)b * box_rows * 128, amap, k0 + u * SHR_KSTEP,
                                    r0 + b * box_rows, &full[st]);
                k0 += sub * SHR_KSTEP;
                if (++st == nstage) {
                    st = 0;
                    if (round2) par ^= 1;
                    round2 = true;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // MMA issuer: a chunk of K starts a fresh accumulator
        if (elect_one()) {
            const uint32_t idesc_lo = umma_idesc_bf16(MMA_M, R > 256 ? 256 : R);
            const uint32_t idesc_hi = umma_idesc_bf16(MMA_M, R > 256 ? R - 256 : 16);
            // descriptors of stage 0's first x and slab boxes; every other operand is a constant number of 16-byte
            // units further on (the address field is the low 14 bits: shared memory is under 256 KB)
            const uint64_t dx0 = umma_desc(smem_u32(ring), 16, 1024, 2);
            const uint64_t da0 = umma_desc(smem_u32(ring) + (uint32_t)sub * SHR_X_BYTES, 16, 1024, 2);
            const uint32_t stage16 = (uint32_t)stage_bytes >> 4, abox16 = a_box_bytes >> 4;
            int st = 0, step = 0, first = 0;  // stage, 64-input step of this block, position inside the K chunk
            uint32_t par = 0, st16 = 0;
            uint32_t dacc = tmem;
            for (int it = 0; it < nk; it++) {
                if (!mbar_wait(&full[st], par, status)) {
                    s_fail = 1;
                    break;
                }
                tc_fence_after();
                for (int u = 0; u < sub && step < nk1; u++, step++) {
                    const uint64_t dx = dx0 + st16 + (uint32_t)u * (SHR_X_BYTES >> 4);
                    const uint64_t da = da0 + st16 + (uint32_t)u * abox16;
#pragma unroll
                    for (int kk = 0; kk < SHR_KSTEP / 16; kk++) {
                        umma<1>(dacc, dx + 2 * kk, da + 2 * kk, idesc_lo, (first | kk) != 0);
                        if (R > 256) umma<1>(dacc + 256, dx + 2 * kk, da + (256 * 128 >> 4) + 2 * kk, idesc_hi, (first | kk) != 0);
                    }
                    if (++first == spc) {  // the next step starts the next chunk's accumulator
                        first = 0;
                        dacc += acc_cols;
                    }
                }
                umma_commit(&empty[st]);
                if (it == nk - 1) umma_commit(&acc_bar);
                st16 += stage16;
                if (++st == nstage) {
                    st = 0;
                    st16 = 0;
                    par ^= 1;
                }
            }
        }
        __syncwarp();
    }
    // everyone: the accumulators are complete once the last commit has arrived
    bool ok = mbar_wait_long(&acc_bar, 0, status);
    __syncthreads();
    if (late) pdl_wait();  // before any store, and on every path: this grid must outlast the ones before it
    if (ok && !s_fail) {
        tc_fence_after();
        const int row = tid;
        float* out = S + (size_t)blockIdx.x * s_stride + (size_t)(start + row) * lds + r0;
        const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
        for (int c = 0; n_acc > 1 && c < R_out; c += 8) {
            float v[PLORA_TILE_SPLIT_MAX][8];
#pragma unroll
            for (int a = 0; a < PLORA_TILE_SPLIT_MAX; a++)
                if (a < n_acc) tmem_ld8_nowait(lane_base + (uint32_t)a * acc_cols + c, v[a]);
            tmem_ld_wait();
            tree_sum<8>(v, n_acc);
            if (row < len) {
                *reinterpret_cast<float4*>(out + c) = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
                *reinterpret_cast<float4*>(out + c + 4) = make_float4(v[0][4], v[0][5], v[0][6], v[0][7]);
            }
        }
        for (int c = 0; n_acc == 1 && c < R_out; c += 32) {
            uint32_t v[32];
            tmem_ld32(lane_base + c, v);
            if (row < len) {
#pragma unroll
                for (int q = 0; q < 32; q += 4)
                    if (c + q < R_out)
                        *reinterpret_cast<float4*>(out + c + q) =
                            make_float4(__uint_as_float(v[q]), __uint_as_float(v[q + 1]), __uint_as_float(v[q + 2]),
                                        __uint_as_float(v[q + 3]));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// ------------------------------------------------------------------------------------------------------
// Expand of one 128-token tile over `nb_per_cta` blocks of 128 output columns of one part. Grid (column
// groups, parts, tiles); 128 threads, thread t owns token row t. Operand layout: 8 x 16-byte core matrices,
// K direction 128 bytes apart, 8-row groups r * 16 bytes apart.
// 32 row segments of this lane's two columns, all requested before any is used
__device__ __forceinline__ void load_rows_bf16(uint32_t (&raw)[32], const bf16* y, int ldy, int nrows, bool colok) {
#pragma unroll
    for (int rr = 0; rr < 32; rr++)
        if (colok && rr < nrows) raw[rr] = *reinterpret_cast<const uint32_t*>(y + (size_t)rr * ldy);
}
__device__ __forceinline__ void load_rows_f32(float2 (&raw)[32], const float* y, int ldy, int nrows, bool colok) {
#pragma unroll
    for (int rr = 0; rr < 32; rr++)
        if (colok && rr < nrows) raw[rr] = *reinterpret_cast<const float2*>(y + (size_t)rr * ldy);
}

template <bool F32>
__global__ void __launch_bounds__(128) plora_expand_mma_kernel(const float* __restrict__ S, size_t s_stride, int lds,
                                                                int K, int ksplit, int fit,
                                                                const int* __restrict__ segs, SegLayout lay,
                                                                const plora_desc* __restrict__ table, void* Y,
                                                                int ldy, int nb_per_cta, int op_bytes,
                                                                int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ __align__(8) uint64_t done;
    __shared__ uint32_t tmem_slot;
    const int tile = blockIdx.z;
    const int n_mma = segs[SEG_N_MMA];
    const int* mt = segs + lay.mma() + 3 * tile;
    const int start = mt[0], len = mt[1], slot = mt[2];
    if (tile >= n_mma) return pdl_exit_idle();
    const plora_desc& d = table[slot];
    const int p = blockIdx.y, r = d.r[p];
    if (r == 0) return pdl_exit_idle();
    const int rows = d.rows[p];
    const int cb0 = blockIdx.x * nb_per_cta;
    if (cb0 * 128 >= rows) return pdl_exit_idle();
    const int nblk = min(nb_per_cta, (rows - cb0 * 128 + 127) / 128);
    const int tid = threadIdx.x, warp = tid >> 5;
    unsigned char* Ahi = dsm;
    unsigned char* Alo = dsm + op_bytes;
    unsigned char* Bs[2] = {dsm + 2 * (size_t)op_bytes, dsm + 3 * (size_t)op_bytes};
    const bf16* B = reinterpret_cast<const bf16*>(d.b[p]);
    const uint32_t sbo = (uint32_t)r * 16u;  // 8-row group stride
    const int P = r >> 3;

    auto load_b = [&](int cb, unsigned char* dst) {
        const int n = tid;  // row of B = output column of the block
        const bool valid = cb * 128 + n < rows;
        const bf16* src = B + (size_t)(valid ? cb * 128 + n : 0) * r;
        unsigned char* drow = dst + (size_t)(n >> 3) * sbo + (n & 7) * 16;
        for (int j = 0; j < P; j++) cp_async16(drow + j * 128, src + j * 8, valid);
    };

    if (tid == 0) {
        mbar_init(&done, 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 128);
    load_b(cb0, Bs[0]);  // B is a slab: it may be fetched before the kernels ahead have finished
    cp_async_commit();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_wait();
    pdl_trigger();

    // this thread's token row of S, split into a bf16 high part and the bf16 of what is left
    {
        const int row = tid;
        const bool valid = row < len;
        const float* sp = S + (size_t)(start + (valid ? row : 0)) * lds + d.r_off[p];
        const int s_eff = plora_tile_blocks(ksplit, fit, n_mma, K, d.rank);  // planes the shrink wrote for this slot
        unsigned char* ahi = Ahi + (size_t)(row >> 3) * sbo + (row & 7) * 16;
        unsigned char* alo = Alo + (size_t)(row >> 3) * sbo + (row & 7) * 16;
        for (int j = 0; j < P; j++) {
            float f[8];
            if (valid && s_eff > 1) {
                float v[PLORA_TILE_SPLIT_MAX][8];
#pragma unroll
                for (int s = 0; s < PLORA_TILE_SPLIT_MAX; s++)
                    if (s < s_eff) {
                        const float* q = sp + (size_t)s * s_stride + j * 8;
                        const float4 a = __ldcg(reinterpret_cast<const float4*>(q));
                        const float4 b = __ldcg(reinterpret_cast<const float4*>(q + 4));
                        v[s][0] = a.x, v[s][1] = a.y, v[s][2] = a.z, v[s][3] = a.w;
                        v[s][4] = b.x, v[s][5] = b.y, v[s][6] = b.z, v[s][7] = b.w;
                    }
                tree_sum<8>(v, s_eff);
#pragma unroll
                for (int e = 0; e < 8; e++) f[e] = v[0][e];
            } else if (valid) {
                const float4 a = __ldcg(reinterpret_cast<const float4*>(sp + j * 8));
                const float4 b = __ldcg(reinterpret_cast<const float4*>(sp + j * 8 + 4));
                f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
            } else {
#pragma unroll
                for (int e = 0; e < 8; e++) f[e] = 0.f;
            }
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
                const float2 hf = __bfloat1622float2(h);
                const __nv_bfloat162 l = __floats2bfloat162_rn(f[2 * e] - hf.x, f[2 * e + 1] - hf.y);
                hi[e] = *reinterpret_cast<const uint32_t*>(&h);
                lo[e] = *reinterpret_cast<const uint32_t*>(&l);
            }
            *reinterpret_cast<uint4*>(ahi + j * 128) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(alo + j * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
    const uint32_t idesc = umma_idesc_bf16(MMA_M, 128);
    const int lane = tid & 31;
    // Epilogue layout: the accumulator leaves tensor memory one token row per thread, is transposed through a
    // warp-private shared-memory tile, and meets y with one 128-byte (bf16) or 256-byte (f32) row segment per
    // warp instruction: lane l owns columns 2l and 2l+1 of a 64-column chunk for each of the warp's 32 rows.
    float* T = reinterpret_cast<float*>(dsm + 4 * (size_t)op_bytes) + (size_t)warp * 32 * EXP_TPAD;
    const int wrow0 = warp * 32;
    const int nrows = max(0, min(32, len - wrow0));  // live rows of this warp
    const size_t ybase = (size_t)(start + wrow0) * ldy + d.off[p] + 2 * lane;
    bool ok = true;
    for (int nb = 0; nb < nblk; nb++) {
        const int cb = cb0 + nb;
        if (nb + 1 < nblk) load_b(cb + 1, Bs[(nb + 1) & 1]);
        cp_async_commit();
        cp_async_wait<1>();  // everything but the block just requested has landed
        fence_async_smem();
        __syncthreads();
        if (warp == 0) {
            if (elect_one()) {
                tc_fence_after();
                const uint32_t a_hi = smem_u32(Ahi), a_lo = smem_u32(Alo), b = smem_u32(Bs[nb & 1]);
                for (int kk = 0; kk < r / 16; kk++)
                    umma<1>(tmem, umma_desc(a_hi + kk * 256, 128, sbo, 0), umma_desc(b + kk * 256, 128, sbo, 0), idesc,
                              kk != 0);
                for (int kk = 0; kk < r / 16; kk++)
                    umma<1>(tmem, umma_desc(a_lo + kk * 256, 128, sbo, 0), umma_desc(b + kk * 256, 128, sbo, 0), idesc, 1);
                umma_commit(&done);
            }
            __syncwarp();
        }
        const int ncols = min(128, rows - cb * 128);
        // y is requested before the MMAs are waited for, as raw words so that all of a chunk's 32 row
        // segments are in flight together: both 64-column chunks for bf16, the first one for f32
        const size_t yblk = ybase + (size_t)cb * 128;
        uint32_t yb0[32], yb1[32];
        float2 yf[32];
        if (F32) {
            load_rows_f32(yf, reinterpret_cast<const float*>(Y) + yblk, ldy, nrows, 2 * lane < ncols);
        } else {
            load_rows_bf16(yb0, reinterpret_cast<const bf16*>(Y) + yblk, ldy, nrows, 2 * lane < ncols);
            load_rows_bf16(yb1, reinterpret_cast<const bf16*>(Y) + yblk + 64, ldy, nrows, 64 + 2 * lane < ncols);
        }
        ok = mbar_wait(&done, nb & 1, status);
        if (!__syncthreads_and(ok)) {
            ok = false;
            break;
        }
        tc_fence_after();
#pragma unroll
        for (int ch = 0; ch < 2; ch++) {
            if (ch * 64 >= ncols) break;
            {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)wrow0 << 16) + ch * 64, v);
#pragma unroll
                for (int q = 0; q < 32; q++) T[lane * EXP_TPAD + q] = __uint_as_float(v[q]);
                tmem_ld32(tmem + ((uint32_t)wrow0 << 16) + ch * 64 + 32, v);
#pragma unroll
                for (int q = 0; q < 32; q++) T[lane * EXP_TPAD + 32 + q] = __uint_as_float(v[q]);
            }
            __syncwarp();
            const bool colok = ch * 64 + 2 * lane < ncols;
            if (F32) {
                if (ch == 1) load_rows_f32(yf, reinterpret_cast<const float*>(Y) + yblk + 64, ldy, nrows, colok);
                float* yo = reinterpret_cast<float*>(Y) + yblk + ch * 64;
#pragma unroll
                for (int rr = 0; rr < 32; rr++) {
                    if (colok && rr < nrows) {
                        const float2 a = *reinterpret_cast<const float2*>(T + rr * EXP_TPAD + 2 * lane);
                        *reinterpret_cast<float2*>(yo + (size_t)rr * ldy) = make_float2(yf[rr].x + a.x, yf[rr].y + a.y);
                    }
                }
            } else {
                bf16* yo = reinterpret_cast<bf16*>(Y) + yblk + ch * 64;
#pragma unroll
                for (int rr = 0; rr < 32; rr++) {
                    if (colok && rr < nrows) {
                        const float2 a = *reinterpret_cast<const float2*>(T + rr * EXP_TPAD + 2 * lane);
                        const uint32_t raw = ch == 0 ? yb0[rr] : yb1[rr];
                        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw));
                        *reinterpret_cast<__nv_bfloat162*>(yo + (size_t)rr * ldy) = __floats2bfloat162_rn(y.x + a.x, y.y + a.y);
                    }
                }
            }
            __syncwarp();
        }
        tc_fence_before();
        __syncthreads();  // the accumulator and this B buffer are free again
    }
    cp_async_wait<0>();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 128);
}

// ------------------------------------------------------------------------------------------------------
// The same expand with y moved by tensor copies, for outputs whose base, row pitch and part offsets are
// 16-byte aligned (every model width in practice; the kernel above stays for the rest). Eight adding warps and
// one more, two blocks per SM. The last warp copies the blocks' rows of B and issues the MMAs of 64 output columns at a
// time, up to two column blocks ahead (mbarriers tell it when S is staged and when an accumulator has been read); the
// other eight never meet at a block-wide barrier inside the loop. Each of them owns the 32 token rows tensor memory
// gives it (two warps per 32 rows, taking alternate slots of columns) and a private ring of 4 KB slots; a slot holds
// 32 rows x 128 bytes of y (64 bf16 or 32 f32 columns, 128-byte swizzle). Lane 0 keeps the ring full of loads; a landed
// slot gets the accumulator columns added in shared memory (thread = row: with the swizzle, eight rows cover all banks)
// and goes back with a tensor store, whose completion frees the slot for the next load. So the read-modify-write
// of y, which is most of the bytes of a prefill step, is asynchronous on both sides and several slots deep.
//
// S is the A operand in tensor memory (written there row by row by the threads that split it): in shared memory it left
// room for one slot per warp at a rank of 64. B arrives by tensor copies of its own: copied by the lanes of the MMA
// warp, 16 bytes each, it bounded the kernel (435 us for the widest prefill layer, 304 without those copies).
// The accumulator is double-buffered in tensor memory and given back as soon as it is in registers: the MMAs of the next
// column block run during this block's additions. Tensor memory: 2 x 64 accumulator columns, then S high and low
// (r / 2 columns each). Tensor maps are per part and end at the part's last column, so a box at the edge is clipped
// instead of touching the next part's columns. A warp whose 32 rows are not all inside the tile (the tail of
// a run) loads the same way but writes its live rows with plain stores: the other rows belong to other tokens.
struct ExpandYMaps {
    CUtensorMap m[PLORA_MAX_PARTS];
};
#ifndef EXP_RING_MAX
#define EXP_RING_MAX 3
#endif
#define EXP_SLOT_BYTES 4096
#define EXP_BN 64        // output columns per MMA
#define EXP_TMEM_A 128   // first tensor-memory column of S
#define EXP_WARPS 8      // adding warps
#define EXP_B_STAGES 6
// ranks per box of B: a swizzle span of 128, 64 or 32 bytes, whichever divides a row
__host__ __device__ inline int exp_b_width(int r) { return r % 64 == 0 ? 64 : r % 32 == 0 ? 32 : 16; }
#define EXP_TMA_SMEM (113 * 1024)  // two blocks per SM: half of 228 KB, less the 1 KB the system keeps per block
struct ExpandBars {
    uint64_t done[2], acc_free[2], a_full, b_full[EXP_B_STAGES], ybar[EXP_WARPS][EXP_RING_MAX];
    uint32_t tmem_slot;
};

// barrier of the two warps that share a quarter of the tile's rows
__device__ __forceinline__ void pair_sync(int quarter) {
    if (quarter == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
    else if (quarter == 1) asm volatile("bar.sync 2, 64;" ::: "memory");
    else if (quarter == 2) asm volatile("bar.sync 3, 64;" ::: "memory");
    else asm volatile("bar.sync 4, 64;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }

template <bool F32, bool HIGH>
__global__ void __launch_bounds__(32 * (EXP_WARPS + 1), 2) plora_expand_tma_kernel(const float* __restrict__ S, size_t s_stride, int lds, int K,
                                                                int ksplit, int fit, const int* __restrict__ segs, SegLayout lay,
                                                                const plora_desc* __restrict__ table,
                                                                const PloraSlabMaps* __restrict__ smaps,
                                                                const __grid_constant__ ExpandYMaps ymaps, void* Y, int ldy,
                                                                int nb_per_cta, int b_bytes, int nbs, int nst, int late,
                                                                int* __restrict__ status) {
    // late != 0: the kernel launched right before this one is the same layer's gather expand, whose blocks let this grid start
    // only after they have themselves waited for the kernels before. S and y are then complete when this grid starts and the
    // gather expand writes other rows of y: the two run side by side, and this grid waits at its end, to outlast the other.
    // Measured, with the tile shrink of plora_apply started in the same way (512 tokens of mixed run lengths, 4 layers): 209 ->
    // 190 us per step; 2,000 ragged tokens with f32 outputs: 328 -> 314 us.
    extern __shared__ __align__(1024) unsigned char dsm1k[];  // (no static shared memory: the ring starts 1024-byte aligned)
    constexpr int CW = F32 ? 32 : 64;     // y columns per slot
    constexpr int CH = EXP_BN / CW;       // slots per column block
    constexpr int NW = EXP_WARPS, WPQ = NW / 4;
    const int n_mma = segs[SEG_N_MMA], p = blockIdx.y, cb0 = blockIdx.x * nb_per_cta;
    bool begun = false;  // the block has waited for the kernels before it and holds tensor memory
    // The grid is as deep as a step of full tiles needs; a step of many short runs has more tiles, which the blocks then
    // walk in turn. (Sized for the most tiles a step can have, half of the blocks of a prefill step found none and
    // cost 15 us of 780.)
    for (int tile = blockIdx.z; tile < n_mma; tile += gridDim.z) {
        const int* mt = segs + lay.mma() + 3 * tile;
        const int start = mt[0], len = mt[1], slot = mt[2];
        // (all that the block needs of the descriptor at once: fetched where it is used, each field is one more way to L2)
        const plora_desc& d = table[slot];
        const int r = __ldg(&d.r[p]), rows = __ldg(&d.rows[p]), y_off = __ldg(&d.off[p]), r_off = __ldg(&d.r_off[p]), rank = __ldg(&d.rank);
        if (r == 0 || cb0 * EXP_BN >= rows) continue;
        const int nblk = min(nb_per_cta, (rows - cb0 * EXP_BN + EXP_BN - 1) / EXP_BN);
        const int nchunks = min(nblk * CH, (rows - cb0 * EXP_BN + CW - 1) / CW);  // slots this block fills, in column order
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        unsigned char* ring = dsm1k + (size_t)warp * nst * EXP_SLOT_BYTES;  // this warp's slots
        unsigned char* ops = dsm1k + (size_t)NW * nst * EXP_SLOT_BYTES;
        ExpandBars& bars = *reinterpret_cast<ExpandBars*>(ops + nbs * (size_t)b_bytes);
        // warps w and w + 4 read the same 32 lanes of tensor memory (rows 32 (w % 4) ...) and take the even and the odd
        // slots of the block's columns
        const int wq = warp & 3, wh = warp >> 2;
        const CUtensorMap* ymap = &ymaps.m[p];
        const CUtensorMap* bmap = reinterpret_cast<const CUtensorMap*>(&smaps[slot].b[p]);
        // the rows of B of column block nb: r / bw boxes of 64 rows by bw ranks, one after another in stage nb % nbs
        const int bw = exp_b_width(r);
        auto load_b = [&](int nb) {
            const int stg = nb % nbs;
            mbar_expect_tx(&bars.b_full[stg], (uint32_t)(EXP_BN * r * 2));
            for (int q = 0; q < r; q += bw)
                tma_load_2d(ops + (size_t)stg * b_bytes + (size_t)q * EXP_BN * 2, bmap, q, (cb0 + nb) * EXP_BN, &bars.b_full[stg]);
        };

        if (tid == 0) {
            auto start_bar = [&](uint64_t* bar, uint32_t count) {
                if (begun) mbar_inval(bar);
                mbar_init(bar, count);
            };
            start_bar(&bars.done[0], 1);
            start_bar(&bars.done[1], 1);
            // the warps that have rows of the tile and a slot in the accumulator's column blocks: the ones of one parity
            // where a column block is one slot, all where it is two
            const int live_warps = CH * min(4, (len + 31) / 32);
            start_bar(&bars.acc_free[0], live_warps);
            start_bar(&bars.acc_free[1], live_warps);
            start_bar(&bars.a_full, 32 * NW);
            for (int i = 0; i < nbs; i++) start_bar(&bars.b_full[i], 1);
            for (int w = 0; w < NW; w++)
                for (int i = 0; i < nst; i++) start_bar(&bars.ybar[w][i], 1);
            mbar_fence_init();
        }
        if (warp == NW && !begun) tmem_alloc(&bars.tmem_slot, 256);
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t tmem = bars.tmem_slot;
        const bool leader = warp == NW && elect_one();
        if (leader) {
            tmap_acquire(bmap);
            for (int nb = 0; nb < nbs - 2 && nb < nblk; nb++) load_b(nb);  // a slab: it may be fetched before the kernels ahead have finished
        }
        if (!begun) {
            if (!late) pdl_wait();
            pdl_trigger();
            begun = true;
        }

        if (warp == NW) {
            // ---- B copies (nbs - 2 column blocks ahead) and MMAs (up to two column blocks ahead of the additions)
            if (leader) {
                const uint32_t idesc = umma_idesc_bf16(MMA_M, EXP_BN);
                const uint32_t a_hi = tmem + EXP_TMEM_A, a_lo = a_hi + (uint32_t)(r >> 1);
                const uint32_t sw = bw == 64 ? 2u : bw == 32 ? 4u : 6u;
                const uint64_t b0 = umma_desc(smem_u32(ops), 16, (uint32_t)bw * 16u, sw);  // eight rows of a box are bw * 16 bytes
                bool ok = mbar_wait(&bars.a_full, 0, status);  // S staged by the other warps
                int stg = 0;
                uint32_t bpar = 0;
                for (int nb = 0; ok && nb < nblk; nb++) {
                    // the accumulator this block goes to was last read for block nb - 2, whose stage of B is therefore free too
                    if (nb >= 2) ok = mbar_wait_long(&bars.acc_free[nb & 1], ((nb >> 1) - 1) & 1, status);
                    if (!ok) break;
                    if (nb + nbs - 2 < nblk) load_b(nb + nbs - 2);
                    ok = mbar_wait_long(&bars.b_full[stg], bpar, status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t bd = b0 + (uint64_t)((uint32_t)stg * (uint32_t)b_bytes >> 4);
                    const uint32_t acc = tmem + (uint32_t)(nb & 1) * EXP_BN;
                    for (int half = 0; half < 2; half++)
                        for (int k = 0; k < r; k += 16)
                            umma_ta(acc, (half ? a_lo : a_hi) + (uint32_t)(k >> 1), bd + (uint64_t)((k / bw) * (EXP_BN * bw * 2 / 16) + (k % bw) / 8),
                                    idesc, (half | k) != 0);
                    umma_commit(&bars.done[nb & 1]);
                    if (++stg == nbs) {
                        stg = 0;
                        bpar ^= 1;
                    }
                }
                // every MMA has completed before the tensor memory goes back
                if (ok && nblk >= 1) mbar_wait_long(&bars.done[(nblk - 1) & 1], ((nblk - 1) >> 1) & 1, status);
                if (ok && nblk >= 2) mbar_wait_long(&bars.done[(nblk - 2) & 1], ((nblk - 2) >> 1) & 1, status);
            }
            __syncwarp();
        } else {
            const int wrow0 = wq * 32;
            const bool live = wrow0 < len;            // the warp has rows of the tile
            const bool whole = wrow0 + 32 <= len;     // all its 32 rows are: results go back by tensor store
            const int ycol0 = y_off + cb0 * EXP_BN;  // first y column of this block's range
            const uint32_t lane_base = tmem + ((uint32_t)wrow0 << 16);
            // the warp's i-th slot is slot wh + 2 i of the block's column range
            const int my_n = (nchunks - wh + WPQ - 1) / WPQ;
            auto load_y = [&](int i, int at) {        // lane 0 only; `at` = i % nst
                uint64_t* bar = &bars.ybar[warp][at];
                mbar_expect_tx(bar, EXP_SLOT_BYTES);
                tma_load_2d(ring + (size_t)at * EXP_SLOT_BYTES, ymap, ycol0 + (wh + WPQ * i) * CW, start + wrow0, bar);
            };
            // (the last slot of the ring is the staging buffer of S first)
            const int early_y = nst - 1;
            if (live && lane == 0)
                for (int i = 0; i < early_y && i < my_n; i++) load_y(i, i);

            // The quarter's 32 rows of S, 32 ranks at a time: each of its two warps fetches 16 rows, a row's 128 bytes by eight lanes, adds
            // up the planes and leaves the sums in shared memory; there every lane finds its own row, split into a bf16 high part (the
            // first warp) and the bf16 of what is left (the second), and puts it into its lane of tensor memory. With a row
            // per lane from the start, each load touched 32 lines of L1 for 16 bytes each: 7,500 to 16,000 cycles to here, now
            // 4,000 to 8,000 (one prompt of 199 tokens: 157 -> 133 us a step, 512 mixed tokens 194 -> 167, eight prompts of 2048 792 -> 765).
            // HIGH (registries of ranks over 64): where S is one plane, 64 ranks at a time through both buffers, where it is two, both planes at
            // once. With one way to L2 per 32 ranks, one run of 64 tokens of rank 128 over four layers of 1024 inputs took 93 us (88 with a row
            // per lane), 88 so; four prompts of 2048 tokens of rank 128 562 -> 546. Not for the others: the longer code costs more at a
            // block's start than it gives (the prompt of 199 tokens of rank 16: 133 -> 139).
            {
                const int s_eff = plora_tile_blocks(ksplit, fit, n_mma, K, rank);  // planes the shrink wrote for this slot
                const float* sq = S + (size_t)(start + wrow0) * lds + r_off;
                auto buffer = [&](int k) { return dsm1k + (size_t)((wq + (k & 32 ? 4 : 0)) * nst + nst - 1) * EXP_SLOT_BYTES; };
#pragma unroll 1
                for (int k0 = 0; k0 < r;) {
                    const bool wide = HIGH && s_eff == 1 && r - k0 >= 64;
                    const int ls = r - k0 >= 32 ? 3 : 2, rpi = 32 >> ls;  // 1 << ls lanes of a row, rows of an instruction
                    const int row0 = 16 * wh + (lane >> ls), piece = lane & ((1 << ls) - 1);
                    // G groups of 32 ranks, U planes and N instructions' rows from the i0-th on, all of them on their way together
                    auto fetch = [&](auto g_, auto u_, auto n_, int i0) {
                        constexpr int G = decltype(g_)::value, U = decltype(u_)::value, N = decltype(n_)::value;
                        float4 sum[G][N];
                        const float* from = sq + (size_t)(row0 + i0 * rpi) * lds + k0 + 4 * piece;
                        for (int s0 = 0; s0 < (U == 4 ? s_eff : U); s0 += U) {  // (U = 1, 2: as many planes as there are)
                            float4 v[U][G][N];
#pragma unroll
                            for (int u = 0; u < U; u++)
#pragma unroll
                                for (int i = 0; i < N; i++)
#pragma unroll
                                    for (int j = 0; j < G; j++) {
                                        v[u][j][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                                        if ((U < 4 || s0 + u < s_eff) && wrow0 + row0 + (i0 + i) * rpi < len)
                                            v[u][j][i] = __ldcg(reinterpret_cast<const float4*>(from + (size_t)(s0 + u) * s_stride + i * rpi * lds + 32 * j));
                                    }
#pragma unroll
                            for (int j = 0; j < G; j++)
#pragma unroll
                                for (int i = 0; i < N; i++) {  // a balanced tree over the 1, 2, 4 or 8 planes
                                    float4 t = v[0][j][i];
                                    if (U > 1) t = add4(t, v[U > 1 ? 1 : 0][j][i]);
                                    if (U > 2 && (HIGH || s_eff > 2)) t = add4(t, add4(v[U > 2 ? 2 : 0][j][i], v[U > 2 ? 3 : 0][j][i]));
                                    sum[j][i] = s0 == 0 ? t : add4(sum[j][i], t);
                                }
                        }
#pragma unroll
                        for (int j = 0; j < G; j++)
#pragma unroll
                            for (int i = 0; i < N; i++) {
                                const int row = row0 + (i0 + i) * rpi;
                                if (row < 16 * wh + 16) *reinterpret_cast<float4*>(buffer(k0 + 32 * j) + row * 128 + ((piece ^ (row & 7)) << 4)) = sum[j][i];
                            }
                    };
                    const std::integral_constant<int, 1> one;
                    const std::integral_constant<int, 2> two;
                    const std::integral_constant<int, 4> four;
                    if constexpr (HIGH) {
                        if (wide) fetch(two, one, four, 0);
                        else if (s_eff == 2) fetch(one, two, four, 0);
                    }
                    if (s_eff == 1 && !wide) {
                        fetch(one, one, four, 0);
                    } else if (s_eff > (HIGH ? 2 : 1)) {
                        fetch(one, four, two, 0);
                        if (ls == 3) fetch(one, four, two, 2);
                    }
                    pair_sync(wq);
                    auto put = [&](int k) {
                        const unsigned char* buf = buffer(k);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            if (k + 16 * h < r) {
                                uint32_t w[8];
#pragma unroll
                                for (int c = 0; c < 4; c++) {
                                    const float4 f = *reinterpret_cast<const float4*>(buf + lane * 128 + (((4 * h + c) ^ (lane & 7)) << 4));
                                    __nv_bfloat162 a = __floats2bfloat162_rn(f.x, f.y), b = __floats2bfloat162_rn(f.z, f.w);
                                    if (wh == 1) {
                                        const float2 af = __bfloat1622float2(a), bf = __bfloat1622float2(b);
                                        a = __floats2bfloat162_rn(f.x - af.x, f.y - af.y);
                                        b = __floats2bfloat162_rn(f.z - bf.x, f.w - bf.y);
                                    }
                                    w[2 * c] = *reinterpret_cast<const uint32_t*>(&a);
                                    w[2 * c + 1] = *reinterpret_cast<const uint32_t*>(&b);
                                }
                                __syncwarp();
                                tmem_st8(lane_base + EXP_TMEM_A + (wh == 1 ? (uint32_t)(r >> 1) : 0u) + (uint32_t)((k + 16 * h) >> 1), w);
                            }
                        }
                    };
                    put(k0);  // (the buffer of the ranks before stays: the next ones go to the other warp's slot)
                    k0 += 32;
                    if (wide) {
                        put(k0);
                        k0 += 32;
                        if (k0 < r) pair_sync(wq);  // both buffers have been read
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&bars.a_full);  // S is staged
                fence_async_smem();         // the staging buffers, read and written, before the copies of y into them
                pair_sync(wq);
                if (live && lane == 0 && early_y < my_n) load_y(early_y, early_y);
            }

            bool ok = true;
            int at = 0;             // i % nst
            uint32_t ypar = 0;      // (i / nst) & 1
#pragma unroll 1
            for (int i = 0; ok && live && i < my_n; i++) {  // the warp's slots, in column order
                const int q = wh + WPQ * i, nb = q / CH, ch = q % CH;
                ok = mbar_wait_long(&bars.done[nb & 1], (nb >> 1) & 1, status);
                if (!ok) break;
                tc_fence_after();
                // 32 accumulator columns at a time: 64 at once leave too few registers, and what spills goes through to L2 beside y;
                // the accumulator is given back once the last ones are in registers
                uint32_t v[32];
                const uint32_t acc = lane_base + (uint32_t)(nb & 1) * EXP_BN + ch * CW;
                auto fetch = [&](int h) {
                    tmem_ld32(acc + h * 32, v);
                    if (h + 1 == CW / 32) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars.acc_free[nb & 1]);
                    }
                };
                fetch(0);
                unsigned char* sl = ring + (size_t)at * EXP_SLOT_BYTES;
                if (!mbar_wait(&bars.ybar[warp][at], ypar, status)) {
                    ok = false;
                    break;
                }
                unsigned char* myrow = sl + lane * 128;
                const int col0 = (cb0 + nb) * EXP_BN + ch * CW;  // first column of the slot within the part
                const bool mine = wrow0 + lane < len;
                if (F32) {
                    float* yrow = reinterpret_cast<float*>(Y) + (size_t)(start + wrow0 + lane) * ldy + y_off + col0;
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        float4* yp = reinterpret_cast<float4*>(myrow + ((c ^ (lane & 7)) << 4));
                        float4 y = *yp;
                        y.x += __uint_as_float(v[4 * c]), y.y += __uint_as_float(v[4 * c + 1]);
                        y.z += __uint_as_float(v[4 * c + 2]), y.w += __uint_as_float(v[4 * c + 3]);
                        if (whole) {
                            *yp = y;
                        } else if (mine) {
                            if (col0 + 4 * c + 4 <= rows) {
                                *reinterpret_cast<float4*>(yrow + 4 * c) = y;
                            } else {
                                const float e[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                                for (int k = 0; k < 4; k++)
                                    if (col0 + 4 * c + k < rows) yrow[4 * c + k] = e[k];
                            }
                        }
                    }
                } else {
                    bf16* yrow = reinterpret_cast<bf16*>(Y) + (size_t)(start + wrow0 + lane) * ldy + y_off + col0;
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        if (c == 4) fetch(1);
                        uint4* yp = reinterpret_cast<uint4*>(myrow + ((c ^ (lane & 7)) << 4));
                        const uint4 raw = *yp;
                        float f[8];
                        unpack8(raw, f);
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const __nv_bfloat162 b2 = __floats2bfloat162_rn(f[2 * e] + __uint_as_float(v[8 * (c & 3) + 2 * e]),
                                                                            f[2 * e + 1] + __uint_as_float(v[8 * (c & 3) + 2 * e + 1]));
                            o[e] = *reinterpret_cast<const uint32_t*>(&b2);
                        }
                        if (whole) {
                            *yp = make_uint4(o[0], o[1], o[2], o[3]);
                        } else if (mine) {
                            if (col0 + 8 * c + 8 <= rows) {
                                *reinterpret_cast<uint4*>(yrow + 8 * c) = make_uint4(o[0], o[1], o[2], o[3]);
                            } else {
#pragma unroll
                                for (int k = 0; k < 4; k++)  // (a part's width is even)
                                    if (col0 + 8 * c + 2 * k < rows) *reinterpret_cast<uint32_t*>(yrow + 8 * c + 2 * k) = o[k];
                            }
                        }
                    }
                }
                if (whole) fence_async_smem();  // the additions above, before the tensor store reads them
                __syncwarp();
                if (lane == 0) {
                    if (whole) {
                        tma_store_2d(ymap, ycol0 + q * CW, start + wrow0, sl);
                        bulk_commit();
                        if (nst == 1) {  // one slot: wait for this store to have read it, then refill it
                            bulk_wait_read();
                            if (i + 1 < my_n) load_y(i + 1, 0);
                        } else {  // the store before this one has read its slot: refill that slot
                            bulk_wait_read_1();
                            if (i >= 1 && i - 1 + nst < my_n) load_y(i - 1 + nst, at == 0 ? nst - 1 : at - 1);
                        }
                    } else if (i + nst < my_n) {
                        load_y(i + nst, at);  // plain stores: the slot is free at once
                    }
                }
                if (++at == nst) {
                    at = 0;
                    ypar ^= 1;
                }
            }
            if (lane == 0) bulk_wait_all();
        }
        tc_fence_before();
        __syncthreads();
    }
    if (!begun) return pdl_exit_idle();
    if (late) pdl_wait();
    if ((threadIdx.x >> 5) == NW) tmem_dealloc(reinterpret_cast<ExpandBars*>(dsm1k + (size_t)NW * nst * EXP_SLOT_BYTES + nbs * (size_t)b_bytes)->tmem_slot, 256);
}

// cuTensorMapEncodeTiled, fetched from the driver once (no link-time dependency on libcuda)
typedef CUresult (*encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
encode_tiled_fn g_encode = nullptr;

}  // namespace

static int g_sms = 148;

cudaError_t plora_mma_init() {
    if (!g_encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (!fn || q != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
        g_encode = reinterpret_cast<encode_tiled_fn>(fn);
    }
    cudaError_t e;
    if ((e = plora_kernel_shared(reinterpret_cast<const void*>(plora_shrink_mma_kernel<false>), 200 * 1024)) != cudaSuccess) return e;
    if ((e = plora_kernel_shared(reinterpret_cast<const void*>(plora_shrink_mma_kernel<true>), 200 * 1024)) != cudaSuccess) return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    e = plora_kernel_shared(reinterpret_cast<const void*>(plora_expand_mma_kernel<false>), 172 * 1024);
    if (e != cudaSuccess) return e;
    e = plora_kernel_shared(reinterpret_cast<const void*>(plora_expand_mma_kernel<true>), 172 * 1024);
    if (e != cudaSuccess) return e;
    if ((e = plora_kernel_shared(reinterpret_cast<const void*>(plora_expand_tma_kernel<false, false>), EXP_TMA_SMEM))) return e;
    if ((e = plora_kernel_shared(reinterpret_cast<const void*>(plora_expand_tma_kernel<true, false>), EXP_TMA_SMEM))) return e;
    if ((e = plora_kernel_shared(reinterpret_cast<const void*>(plora_expand_tma_kernel<false, true>), EXP_TMA_SMEM))) return e;
    return plora_kernel_shared(reinterpret_cast<const void*>(plora_expand_tma_kernel<true, true>), EXP_TMA_SMEM);
}

namespace {
template <typename... Params, typename... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl,
                       Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
}  // namespace

// The tensor maps of one slot's slabs for one layer. Stacked A [R, K]: boxes of 64 inputs by R rows (R / 2 rows when R
// is over 256, the limit of a box), 128-byte swizzle. B of a part [rows, r]: boxes of 64 output columns by as many ranks
// as exp_b_width says, the swizzle as wide as the box.
cudaError_t plora_mma_encode_slab(PloraSlabMaps* out, const plora_desc& d, int K) {
    static_assert(sizeof(CUtensorMap) == sizeof(PloraTmap), "tensor map size");
    if (!g_encode) return cudaErrorNotSupported;
    auto encode = [](PloraTmap* m, uint64_t base, int inner, int outer, int box_inner, int box_outer) {
        const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
        const cuuint64_t strides[1] = {(cuuint64_t)inner * 2};
        const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
        const cuuint32_t es[2] = {1, 1};
        const CUtensorMapSwizzle sw = box_inner == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
                                      : box_inner == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                        : CU_TENSOR_MAP_SWIZZLE_32B;
        return g_encode(reinterpret_cast<CUtensorMap*>(m), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)(uintptr_t)base, dims, strides, box,
                        es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    bool ok = encode(&out->a, d.a, K, d.rank, SHR_KSTEP, d.rank > 256 ? d.rank / 2 : d.rank);
    ok = ok && encode(&out->a64, d.a, K, d.rank, SHR_KSTEP, SHR_GROUP);  // (rows past the last one arrive as zeros)
    for (int p = 0; p < PLORA_MAX_PARTS; p++)
        if (d.r[p] > 0) ok = ok && encode(&out->b[p], d.b[p], d.r[p], d.rows[p], exp_b_width(d.r[p]), EXP_BN);
    return ok ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t plora_launch_shrink_mma(const void* x, int rows, int ldx, int K, const int32_t* segs, SegLayout lay,
                                    const plora_desc* table, const PloraSlabMaps* smaps, float* S, size_t s_stride_elems, int lds,
                                    int max_rank_total, int tile_cap, int tile_split, int* status, bool pdl, bool late,
                                    cudaStream_t st) {
    if (!g_encode) return cudaErrorNotSupported;
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ldx * 2};
    const cuuint32_t box[2] = {SHR_KSTEP, MMA_M};
    const cuuint32_t es[2] = {1, 1};
    if (g_encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, es,
                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    const int groups = (max_rank_total + SHR_GROUP - 1) / SHR_GROUP;
    const bool rsplit = (tile_split & PLORA_TILE_RSPLIT) != 0;
    int stage_bytes = SHR_X_BYTES + (((rsplit ? SHR_GROUP : max_rank_total) * 128 + 1023) / 1024) * 1024;
    // two steps of 64 inputs per stage where at least three such stages fit
    const int sub = 3 * 2 * stage_bytes <= 190 * 1024 ? 2 : 1;
    stage_bytes *= sub;
    int nstage = (190 * 1024) / stage_bytes;
    nstage = nstage > SHR_MAX_STAGES ? SHR_MAX_STAGES : nstage;
    if (nstage < 2) return cudaErrorInvalidValue;
    const size_t smem = (size_t)nstage * stage_bytes + 1024;
    return launch_pdl(rsplit ? plora_shrink_mma_kernel<true> : plora_shrink_mma_kernel<false>,
                      dim3((unsigned)(tile_split & (PLORA_TILE_RSPLIT - 1)), rsplit ? (unsigned)groups : 1, (unsigned)tile_cap), dim3(128), smem, st, pdl, map, smaps, K, segs, lay, table, S, s_stride_elems, lds,
                      tile_split & (PLORA_TILE_RSPLIT - 1), tile_split / PLORA_TILE_FIT, nstage, stage_bytes, sub, late && pdl ? 1 : 0, status);
}

cudaError_t plora_launch_expand_mma(const float* S, size_t s_stride_elems, int lds, int K, int tile_split,
                                    const int32_t* segs, SegLayout lay, const plora_desc* table, const PloraSlabMaps* smaps, void* y,
                                    int ldy, int f32_out, int parts, const int* part_off, const int* part_rows, int rows_total,
                                    int max_rows, int tile_cap, int* status, bool pdl, bool late, cudaStream_t st) {
    const int max_rank = lds / PLORA_MAX_PARTS;
    const int op_bytes = MMA_M * max_rank * 2;
    // Column blocks per thread block (one staging of its S tile each): the count that minimises waves x (start-up +
    // blocks walked) for the step's estimated tile count, two thread blocks per SM; start-up (tensor-memory allocation,
    // staging S, the first MMAs) costs about as much as walking 320 columns.
    const long long tiles_est = (tile_cap + 1) / 2;  // tile_cap counts 64-token halves
    auto per_cta = [&](int width, int most) {
        int pick = 1;
        double best = 1e30;
        for (int nb = 1; nb <= most; nb++) {
            long long groups = 0;
            for (int p = 0; p < parts; p++) groups += ((part_rows[p] + width - 1) / width + nb - 1) / nb;
            const long long waves = (tiles_est * groups + 2 * g_sms - 1) / (2 * g_sms);
            const double cost = (double)waves * (320.0 + (double)nb * width);
            if (cost < best) {
                best = cost;
                pick = nb;
            }
        }
        return std::min(pick, (max_rows + width - 1) / width);
    };
    // y by tensor copies where its base, pitch and part offsets are 16-byte aligned
    const int elt = f32_out ? 4 : 2;
    bool aligned = g_encode && ((uintptr_t)y & 15) == 0 && ((size_t)ldy * elt) % 16 == 0 && rows_total > 0;
    for (int p = 0; p < parts; p++) aligned = aligned && ((size_t)part_off[p] * elt) % 16 == 0;
    if (aligned) {
        // stages of B of 2 KB (rank 16) to 16 KB (rank 128); two slots per warp fit at every rank
        const int b_bytes = EXP_BN * max_rank * 2, nbs = b_bytes <= 8192 ? EXP_B_STAGES : 3;
        int nst = (int)((EXP_TMA_SMEM - nbs * b_bytes - (int)sizeof(ExpandBars)) / (EXP_WARPS * EXP_SLOT_BYTES));
        nst = nst > EXP_RING_MAX ? EXP_RING_MAX : nst;
        ExpandYMaps maps;
        memset(&maps, 0, sizeof(maps));
        const cuuint32_t es[2] = {1, 1};
        const cuuint32_t box[2] = {(cuuint32_t)(128 / elt), 32};
        const cuuint64_t strides[1] = {(cuuint64_t)ldy * elt};
        for (int p = 0; p < parts && aligned; p++) {
            // the map ends at the part's last column: a box over the edge is clipped
            const cuuint64_t dims[2] = {(cuuint64_t)(part_off[p] + part_rows[p]), (cuuint64_t)rows_total};
            aligned = g_encode(&maps.m[p], f32_out ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, y,
                               dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
        }
        if (aligned && nst >= 1) {
            const size_t smem_tma = (size_t)EXP_WARPS * nst * EXP_SLOT_BYTES + nbs * (size_t)b_bytes + sizeof(ExpandBars);
            const int nb_per_cta = per_cta(EXP_BN, 32);
            const dim3 grid((unsigned)(((max_rows + EXP_BN - 1) / EXP_BN + nb_per_cta - 1) / nb_per_cta), (unsigned)parts,
                            (unsigned)std::min(tile_cap, (rows_total + MMA_M - 1) / MMA_M + 4));
            auto* fn = max_rank > 64 ? (f32_out ? plora_expand_tma_kernel<true, true> : plora_expand_tma_kernel<false, true>)
                                     : (f32_out ? plora_expand_tma_kernel<true, false> : plora_expand_tma_kernel<false, false>);
            return launch_pdl(fn, grid, dim3(32 * (EXP_WARPS + 1)),
                              smem_tma, st, pdl, S, s_stride_elems, lds, K, tile_split & (PLORA_TILE_RSPLIT - 1), tile_split / PLORA_TILE_FIT, segs, lay, table, smaps, maps, y, ldy,
                              nb_per_cta, b_bytes, nbs, nst, late && pdl ? 1 : 0, status);
        }
    }
    const int nb_per_cta = per_cta(128, 16);
    const dim3 grid((unsigned)(((max_rows + 127) / 128 + nb_per_cta - 1) / nb_per_cta), (unsigned)parts, (unsigned)tile_cap);
    // at least 48 KB of shared memory per block: no more than four blocks, 128 tensor-memory columns each,
    // share an SM's 512 columns
    size_t smem = (size_t)4 * op_bytes + (size_t)4 * 32 * EXP_TPAD * sizeof(float);
    if (smem < 48 * 1024) smem = 48 * 1024;
    if (f32_out)
        return launch_pdl(plora_expand_mma_kernel<true>, grid, dim3(128), smem, st, pdl, S, s_stride_elems, lds, K,
                          tile_split & (PLORA_TILE_RSPLIT - 1), tile_split / PLORA_TILE_FIT, segs, lay, table, y, ldy, nb_per_cta, op_bytes, status);
    return launch_pdl(plora_expand_mma_kernel<false>, grid, dim3(128), smem, st, pdl, S, s_stride_elems, lds, K,
                      tile_split & (PLORA_TILE_RSPLIT - 1), tile_split / PLORA_TILE_FIT, segs, lay, table, y, ldy, nb_per_cta, op_bytes, status);
}
