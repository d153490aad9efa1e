// One layer for prefill-sized steps as a single tensor-core kernel: the base matrix multiply (FP8 with
// per-token and per-output-channel scales, or bf16) and the adapter term of every long run of tokens, both on
// tcgen05 with accumulators in tensor memory, y written once (no read-modify-write). No counterpart in
// pocket-engine, whose expand is always a separate kernel after the layer's own GEMM (src/linear.rs:889-921).
//
// A pair of blocks (a cluster of two, cta_group::2) computes tiles of 256 tokens x BN output columns (256, or 192 or 128
// where that fills the device better); as many pairs as fit walk the tiles. Each block holds half of the tile's tokens and
// half of its rows of W; the MMAs of the leading block read both, so a byte that enters an SM is used twice as often
// as in a tile of one block's own: the single-block 128 x 256 kernel before this one moved 48 KB per SM and step of 128
// bytes of K where this one moves 32. 320 threads per block:
//   warp 0      producer: per step of 128 bytes of K, the block's x rows (16 KB) and W rows (BN / 2 x 128 bytes) as tensor
//               copies into a ring of four stages (128-byte swizzle); both blocks' copies report to the leader
//   warp 1      (leader) issues the MMAs and tells both blocks when a stage, an accumulator or the adapter operands are free
//   warps 2..9  stage the adapter passes of the next tile, then run its epilogue. A pass = one tensor-core tile of the
//               step's grouping (a run of one slot's tokens) that meets the pair's rows x 64 columns of the slot's rank:
//               S rows (plane 0, other rows zero) split into bf16 high and low parts, and the block's rows of B_p, in
//               rows of 128 bytes with the 128-byte swizzle (the same products from unswizzled operands, whose rows
//               collide in shared memory, took a fifth of the FP8 layer's time). The MMA warp takes a pass as soon as it is staged, in the middle of
//               the main loop.
// The adapter term has an accumulator of its own, added once in the epilogue: when a pass is taken depends on timing, so in
// the base product's accumulator the order of the sums, and with it the last bits of y, would differ from run to run.
// bf16: two accumulators of BN columns, so the epilogue of a tile without passes runs under the next tile's main loop. A
// tile with passes has them in the other one (BN over 128; with 128 columns there is room for two of each), and the next
// tile starts when both have been read into registers. FP8: base product in columns 0 .., adapter term in columns BN ..
// Epilogue: y = s_t s_n acc + adapter (or acc), staged in 128-byte-swizzled slots and written by tensor stores.
//
// Tokens outside long runs (decode tokens, short prompts) get only the base product here; the gather expand
// kernel adds their adapter term afterwards. Needs y 16-byte aligned with a 16-byte multiple pitch, and part
// boundaries at multiples of 256 columns (a tile lies in one part). Every wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "plora_internal.h"
#include "plora_device.cuh"
#include "plora_tc.cuh"

typedef __nv_bfloat16 bf16;

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const uint32_t n = valid ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- the two blocks of a pair ----
__device__ __forceinline__ uint32_t pair_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address, in the cluster's shared memory, of the leading block's copy of a shared variable
__device__ __forceinline__ uint32_t at_leader(const void* p) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
    return a;
}
__device__ __forceinline__ void arrive_at(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// tiled load into this block's shared memory whose bytes are counted on a barrier of either block of the pair
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* slot) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(taddr) : "memory");
}
template <int KIND>
__device__ __forceinline__ void pair_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    if (KIND == 0)
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc)
            : "memory");
}
// arrives on the barrier at this address in both blocks once this thread's earlier MMAs are complete
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}

#define G_BM 128   // token rows per block
#define G_BKB 128  // bytes of K per stage row
#define G_STAGES 4
#define G_RC 64  // rank columns per adapter pass
#define G_AOP (G_BM * G_RC * 2)
#define G_MAX_PASS 16
#define G_SLOT 4096  // 32 rows x 128 bytes of y
#define G_EPI_WARPS 8
#define G_EPI (32 * G_EPI_WARPS)
#define G_GROUP_M 8  // tiles of tokens that are walked together: neighbouring pairs share rows of x and of W in L2

__device__ __forceinline__ void epi_sync_all() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

struct GemmParts {
    int n;
    int off[PLORA_MAX_PARTS];
    int rows[PLORA_MAX_PARTS];
};

struct GemmShared {
    uint64_t full[G_STAGES], empty[G_STAGES], acc_full[2], acc_empty[2], meta, ad_full, ad_empty;
    uint32_t tmem_slot;
    int npass, row0[G_MAX_PASS], row1[G_MAX_PASS], slot[G_MAX_PASS], rc0[G_MAX_PASS], rw[G_MAX_PASS];
};

// rows of W per block; the adapter operands are the pairs' only
__host__ __device__ constexpr int gemm_w_rows(int bn, bool two) { return two ? bn / 2 : bn; }
__host__ __device__ constexpr size_t gemm_stage_bytes(int bn, bool two) { return G_BM * G_BKB + gemm_w_rows(bn, two) * G_BKB; }
__host__ __device__ constexpr size_t gemm_operands(int bn, bool two) { return two ? 2 * G_AOP + (size_t)bn / 2 * G_RC * 2 : 0; }
constexpr size_t gemm_smem(int bn, bool two) {
    return 1024 + G_STAGES * gemm_stage_bytes(bn, two) + gemm_operands(bn, two) + G_EPI_WARPS * G_SLOT + bn * sizeof(float);
}

// TWO: a pair of blocks per tile (above). Otherwise a block has a tile of 128 tokens x BN columns to itself and there are no
// adapter passes: for steps of up to 128 tokens without long runs, in which the second block of a pair would have no tokens
// and its MMAs no use.
template <int KIND, bool F32, int BN, bool TWO>
__global__ void __cluster_dims__(TWO ? 2 : 1, 1, 1) __launch_bounds__(64 + G_EPI, 1)
    plora_gemm_fused_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                            const __grid_constant__ CUtensorMap ymap, const float* __restrict__ st, const float* __restrict__ sn, int T,
                            int N, int K, const int* __restrict__ segs, SegLayout lay, const plora_desc* __restrict__ table,
                            GemmParts parts, const float* __restrict__ S, int lds, int* __restrict__ status) {
    extern __shared__ unsigned char dsm_raw[];
    __shared__ __align__(8) GemmShared sh;
    constexpr uint32_t STAGE = (uint32_t)gemm_stage_bytes(BN, TWO);
    constexpr int BLOCKS = TWO ? 2 : 1, TM = BLOCKS * G_BM;  // blocks and tokens of a tile
    constexpr int WR = gemm_w_rows(BN, TWO);
    constexpr int HALF = BN == 192 ? 128 : BN / 2;  // columns of the first four epilogue warps (whole slots of 64)
    constexpr int NBUF = KIND == 0 ? 1 : 2;               // accumulators of the base product
    constexpr bool SHARED = KIND == 1 && BN > 128;        // the adapter term uses the other one of them
    // first column of the adapter term of a tile whose base product is in accumulator `buf`
    auto ad_col = [](int buf) { return (uint32_t)(KIND == 0 ? BN : SHARED ? (buf ^ 1) * BN : (2 + buf) * BN); };
    constexpr int KEL = KIND == 0 ? G_BKB : G_BKB / 2;    // elements of K per step
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = TWO ? pair_rank() : 0;
    unsigned char* ring = dsm_raw + ((1024u - (smem_u32(dsm_raw) & 1023u)) & 1023u);
    unsigned char* Ahi = ring + G_STAGES * STAGE;
    unsigned char* Alo = Ahi + G_AOP;
    unsigned char* Bop = Alo + G_AOP;
    unsigned char* slots = ring + G_STAGES * STAGE + gemm_operands(BN, TWO);
    float* sn_s = reinterpret_cast<float*>(slots + G_EPI_WARPS * G_SLOT);  // the tile's column scales
    if (tid == 0) {
        for (int i = 0; i < G_STAGES; i++) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&sh.acc_full[i], 1);
            mbar_init(&sh.acc_empty[i], BLOCKS * G_EPI_WARPS);
        }
        mbar_init(&sh.meta, 1);
        mbar_init(&sh.ad_full, 2);
        mbar_init(&sh.ad_empty, 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        if (TWO) pair_tmem_alloc(&sh.tmem_slot);
        else tmem_alloc(&sh.tmem_slot, 512);
    }
    tc_fence_before();
    __syncthreads();
    if (TWO) pair_sync();  // the other block's barriers exist
    tc_fence_after();
    const uint32_t tmem = sh.tmem_slot;
    const int nk = ((KIND == 0 ? K : 2 * K) + G_BKB - 1) / G_BKB;
    // tiles in groups of G_GROUP_M tiles of tokens; within a group, tokens first
    const int mt = (T + TM - 1) / TM, nt = (N + BN - 1) / BN, tiles = mt * nt;
    const int pair = blockIdx.x / BLOCKS, pairs = gridDim.x / BLOCKS;
    auto place = [&](int t, int& m0, int& n0) {
        const int per = G_GROUP_M * nt, g = t / per, in = t - g * per, gm = min(G_GROUP_M, mt - g * G_GROUP_M);
        m0 = (g * G_GROUP_M + in % gm) * TM;
        n0 = in / gm * BN;
    };
    pdl_wait();  // S, x and the scales come from the kernels before
    pdl_trigger();

    if (warp == 0) {
        if (elect_one()) {
            int stg = 0;
            uint32_t par = 0;
            bool ok = true, round2 = false;
            for (int t = pair; ok && t < tiles; t += pairs) {
                int m0, n0;
                place(t, m0, n0);
                for (int ks = 0; ks < nk; ks++) {
                    if (round2) ok = mbar_wait_long(&sh.empty[stg], par ^ 1, status);
                    if (!ok) break;
                    unsigned char* xs = ring + (size_t)stg * STAGE;
                    if (rank == 0) mbar_expect_tx(&sh.full[stg], BLOCKS * STAGE);
                    if (TWO) {
                        const uint32_t bar = at_leader(&sh.full[stg]);
                        tma_load_2d_pair(xs, &xmap, ks * KEL, m0 + (int)rank * G_BM, bar);
                        tma_load_2d_pair(xs + G_BM * G_BKB, &wmap, ks * KEL, n0 + (int)rank * WR, bar);
                    } else {
                        tma_load_2d(xs, &xmap, ks * KEL, m0, &sh.full[stg]);
                        tma_load_2d(xs + G_BM * G_BKB, &wmap, ks * KEL, n0, &sh.full[stg]);
                    }
                    if (++stg == G_STAGES) {
                        stg = 0;
                        par ^= 1;
                        round2 = true;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // M TM, N BN, f32 accumulator, K-major operands; kind::f16 carries the bf16 formats in bits 7 and 10
            const uint32_t idesc_ad = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
            const uint32_t idesc = KIND == 0 ? (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24) : idesc_ad;
            const uint64_t dx0 = umma_desc(smem_u32(ring), 16, 1024, 2), dw0 = umma_desc(smem_u32(ring) + G_BM * G_BKB, 16, 1024, 2);
            int stg = 0, i = 0;
            uint32_t par = 0, apar = 0;  // parities of the stages and of the adapter operands
            int before = 0;              // passes of the tile before
            bool ok = true;
            for (int t = pair; ok && t < tiles; t += pairs, i++) {
                const int buf = KIND == 0 ? 0 : i & 1;
                const uint32_t acc = tmem + (uint32_t)buf * BN, ad = tmem + ad_col(buf);
                // Whoever last had this tile's accumulator has been read: the tile NBUF before, or the one before, whose
                // adapter term was in it (its warps have then read the earlier tile too). The adapter term's needs no wait of
                // its own: the warps that stage a pass have finished the tile before.
                if (SHARED && before > 0) ok = mbar_wait_long(&sh.acc_empty[buf ^ 1], (i - 1) / NBUF & 1, status);
                else if (i >= NBUF) ok = mbar_wait_long(&sh.acc_empty[buf], (i / NBUF - 1) & 1, status);
                tc_fence_after();
                int npass = TWO ? -1 : 0, ps = 0;  // npass: not known before the other warps have written the list
                auto pass = [&]() {
                    tc_fence_after();
                    const int rw = sh.rw[ps];
                    const uint64_t a_hi = umma_desc(smem_u32(Ahi), 16, 1024, 2), a_lo = umma_desc(smem_u32(Alo), 16, 1024, 2);
                    const uint64_t b = umma_desc(smem_u32(Bop), 16, 1024, 2);
                    for (int kk = 0; kk < rw / 16; kk++) pair_umma<1>(ad, a_hi + 2 * kk, b + 2 * kk, idesc_ad, (ps | kk) != 0);
                    for (int kk = 0; kk < rw / 16; kk++) pair_umma<1>(ad, a_lo + 2 * kk, b + 2 * kk, idesc_ad, 1);
                    pair_commit(&sh.ad_empty);
                    ps++;
                    apar ^= 1;
                };
                for (int ks = 0; ok && ks < nk; ks++) {
                    ok = mbar_wait_long(&sh.full[stg], par, status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t dx = dx0 + (uint64_t)((uint32_t)stg * STAGE >> 4), dw = dw0 + (uint64_t)((uint32_t)stg * STAGE >> 4);
#pragma unroll
                    for (int kk = 0; kk < G_BKB / 32; kk++) {
                        if (TWO) pair_umma<KIND>(acc, dx + 2 * kk, dw + 2 * kk, idesc, (ks | kk) != 0);
                        else umma<KIND>(acc, dx + 2 * kk, dw + 2 * kk, idesc, (ks | kk) != 0);
                    }
                    if (TWO) pair_commit(&sh.empty[stg]);
                    else umma_commit(&sh.empty[stg]);
                    if (++stg == G_STAGES) {
                        stg = 0;
                        par ^= 1;
                    }
                    if (TWO && npass < 0 && mbar_test(&sh.meta, i & 1)) npass = sh.npass;
                    if (TWO && ps < npass && mbar_test(&sh.ad_full, apar)) pass();
                }
                if (TWO && ok && npass < 0) {
                    ok = mbar_wait_long(&sh.meta, i & 1, status);
                    npass = ok ? sh.npass : 0;
                }
                while (TWO && ok && ps < npass) {
                    ok = mbar_wait_long(&sh.ad_full, apar, status);
                    if (ok) pass();
                }
                before = ps;
                if (ok && TWO) pair_commit(&sh.acc_full[buf]);
                if (ok && !TWO) umma_commit(&sh.acc_full[buf]);
            }
        }
        __syncwarp();
    } else {
        const int e = tid - 64;                  // 0..255
        const int ew = warp - 2, wq = warp & 3;  // tensor-memory lanes 32 wq .. 32 wq + 31, columns of half ew / 4
        unsigned char* slot = slots + ew * G_SLOT;
        const uint32_t ad_full = at_leader(&sh.ad_full);
        uint32_t apar = 0;
        bool staged = false;  // the adapter operands have been used before
        bool ok = true;  // (of this warp: after a wait that ran out it goes on meeting the barriers, and does nothing else)
        int i = 0;
        for (int t = pair; t < tiles; t += pairs, i++) {
            int m0, n0;
            place(t, m0, n0);
            int part = 0;  // the part the tile's columns lie in
#pragma unroll
            for (int q = 1; q < PLORA_MAX_PARTS; q++)
                if (q < parts.n && n0 >= parts.off[q]) part = q;
            const int n_local = n0 - parts.off[part] + (int)rank * WR;  // this block's first row of B_p
            // ---- the tile's adapter passes: tensor-core tiles of the grouping that meet the pair's rows
            if (TWO && ew == 0) {
                const int n_mma = segs[SEG_N_MMA];
                const int* ml = segs + lay.mma();
                // the first tile that ends after the first row: 32 probes a round
                int lo = 0, n = n_mma;
                while (n > 0) {
                    const int step = (n + 31) >> 5, at = lo + lane * step;
                    const unsigned past = __ballot_sync(0xffffffffu, lane * step >= n || ml[3 * at] + ml[3 * at + 1] > m0);
                    const int q = past ? __ffs(past) - 1 : 32;  // tile lo + q * step is past, the one a step before is not
                    if (q == 0) break;
                    const int from = (q - 1) * step + 1, to = min(n, q * step);
                    lo += from;
                    n = to - from;
                }
                if (lane == 0) {
                    int np = 0;
                    for (int q = lo; q < n_mma && ml[3 * q] < m0 + TM; q++) {
                        const int start = ml[3 * q], len = ml[3 * q + 1], slot_id = ml[3 * q + 2];
                        const int r = table[slot_id].r[part];
                        for (int rc0 = 0; rc0 < r; rc0 += G_RC) {
                            if (np == G_MAX_PASS) {
                                atomicMax(status, PLORA_ERR_CAPACITY);
                                break;
                            }
                            sh.row0[np] = max(start, m0) - m0;
                            sh.row1[np] = min(start + len, m0 + TM) - m0;
                            sh.slot[np] = slot_id;
                            sh.rc0[np] = rc0;
                            sh.rw[np] = min(G_RC, r - rc0);
                            np++;
                        }
                    }
                    sh.npass = np;
                }
                __syncwarp();
            }
            if (KIND == 0)
                for (int c = e; c < BN; c += G_EPI) sn_s[c] = n0 + c < N ? sn[n0 + c] : 0.f;
            epi_sync_all();
            const int npass = TWO ? sh.npass : 0;
            if (TWO && e == 0) mbar_arrive(&sh.meta);
            for (int ps = 0; ps < npass; ps++) {
                if (staged) {  // the operands of the pass before are still being read until its MMAs complete
                    if (ok) ok = mbar_wait_long(&sh.ad_empty, apar, status);
                    apar ^= 1;
                }
                staged = true;
                if (!ok) {
                    epi_sync_all();
                    continue;
                }
                const plora_desc& d = table[sh.slot[ps]];
                const int rc0 = sh.rc0[ps], r = d.r[part], P = sh.rw[ps] >> 3;
                // eight threads a row, one 16-byte piece of 8 ranks each: rows of B_p for the block's half of the columns
                const int j = e & 7;
                const bf16* B = reinterpret_cast<const bf16*>(d.b[part]) + rc0 + j * 8;
#pragma unroll
                for (int h = 0; h < BN / 64; h++) {
                    const int n = (e >> 3) + 32 * h;
                    const bool valid = n_local + n < d.rows[part];
                    if (j < P) cp_async16(Bop + (size_t)n * 128 + ((j ^ (n & 7)) << 4), B + (size_t)(valid ? n_local + n : 0) * r, valid);
                }
                // ... and this block's token rows of S (zero outside the pass's rows), as bf16 high and low parts
                const float* sp = S + d.r_off[part] + rc0 + j * 8;
                float4 f[4][2];
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const int rel = (e >> 3) + 32 * h + (int)rank * G_BM;
                    f[h][0] = f[h][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (j < P && rel >= sh.row0[ps] && rel < sh.row1[ps]) {
                        f[h][0] = __ldcg(reinterpret_cast<const float4*>(sp + (size_t)(m0 + rel) * lds));
                        f[h][1] = __ldcg(reinterpret_cast<const float4*>(sp + (size_t)(m0 + rel) * lds + 4));
                    }
                }
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const int row = (e >> 3) + 32 * h;
                    const float v[8] = {f[h][0].x, f[h][0].y, f[h][0].z, f[h][0].w, f[h][1].x, f[h][1].y, f[h][1].z, f[h][1].w};
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                        const float2 hf = __bfloat1622float2(h2);
                        const __nv_bfloat162 l2 = __floats2bfloat162_rn(v[2 * q] - hf.x, v[2 * q + 1] - hf.y);
                        hi[q] = *reinterpret_cast<const uint32_t*>(&h2);
                        lo[q] = *reinterpret_cast<const uint32_t*>(&l2);
                    }
                    const uint32_t at = (uint32_t)row * 128u + (uint32_t)((j ^ (row & 7)) << 4);
                    if (j < P) {
                        *reinterpret_cast<uint4*>(Ahi + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                        *reinterpret_cast<uint4*>(Alo + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                    }
                }
                cp_async_wait_all();
                fence_async_smem();
                epi_sync_all();
                if (e == 0) arrive_at(ad_full);
            }
            // ---- epilogue: the warp's 32 rows of its half of the columns, scaled and added, into a swizzled slot of 128
            // bytes a row, then a tensor store (clipped at the edges of y by the tensor map)
            const int buf = KIND == 0 ? 0 : i & 1;
            if (ok) ok = mbar_wait_long(&sh.acc_full[buf], (i / NBUF) & 1, status);
            if (!ok) {
                epi_sync_all();
                continue;
            }
            tc_fence_after();
            const int row = m0 + (int)rank * G_BM + wq * 32 + lane;
            constexpr int CW = F32 ? 32 : 64;  // y columns per slot
            const int c0 = (ew >> 2) * HALF, groups = (ew >> 2 ? BN - HALF : HALF) / 32;
            const float srow = KIND == 0 ? (row < T ? __ldcg(st + row) : 0.f) : 1.f;
            const uint32_t lanes = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)c0;
            const uint32_t base = lanes + (uint32_t)buf * BN, ad = lanes + ad_col(buf);
            constexpr int NW = F32 ? 32 : 16;  // words of 32 columns
            auto fetch = [&](int g, uint32_t (&w)[NW]) {  // 32 accumulator columns, as they go to y
                uint32_t vb[32], va[32];
                tmem_ld32_nowait(base + g * 32, vb);
                if (npass > 0) tmem_ld32_nowait(ad + g * 32, va);
                tmem_ld_wait();
                float o[32];
#pragma unroll
                for (int q = 0; q < 32; q++) {
                    const float v = KIND == 0 ? __uint_as_float(vb[q]) * (srow * sn_s[c0 + g * 32 + q]) : __uint_as_float(vb[q]);
                    o[q] = npass > 0 ? v + __uint_as_float(va[q]) : v;
                }
#pragma unroll
                for (int q = 0; q < NW; q++) {
                    const __nv_bfloat162 b2 = __floats2bfloat162_rn(o[(2 * q) % 32], o[(2 * q + 1) % 32]);
                    w[q] = F32 ? __float_as_uint(o[q]) : *reinterpret_cast<const uint32_t*>(&b2);
                }
            };
            auto release = [&]() {  // everything this warp reads is in registers: the accumulator is free
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (TWO) arrive_at(at_leader(&sh.acc_empty[buf]));
                    else mbar_arrive(&sh.acc_empty[buf]);
                }
            };
            auto put = [&](int g, const uint32_t (&w)[NW]) {
                if (F32 || (g & 1) == 0) {  // a new slot: the store before has to have read it
                    if (lane == 0) bulk_wait_read();
                    __syncwarp();
                }
                unsigned char* myrow = slot + lane * 128;
#pragma unroll
                for (int q = 0; q < NW / 4; q++) {
                    const int c = F32 ? q : (g & 1) * 4 + q;
                    *reinterpret_cast<uint4*>(myrow + ((c ^ (lane & 7)) << 4)) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
                }
                if (F32 || (g & 1) == 1) {
                    fence_async_smem();
                    __syncwarp();
                    const int col = n0 + c0 + (F32 ? g : g >> 1) * CW;
                    if (lane == 0) {
                        if (col < N && m0 + (int)rank * G_BM + wq * 32 < T) tma_store_2d(&ymap, col, m0 + (int)rank * G_BM + wq * 32, slot);
                        bulk_commit();
                    }
                }
            };
            // Where the next tile waits for both accumulators, all columns come to registers (as bf16 they fit) before any goes on
            if (SHARED && TWO && !F32) {
                constexpr int NG = SHARED && TWO && !F32 ? HALF / 32 : 1;
                uint32_t w[NG][NW];
#pragma unroll
                for (int g = 0; g < NG; g++)
                    if (g < groups) fetch(g, w[g]);
                release();
#pragma unroll
                for (int g = 0; g < NG; g++)
                    if (g < groups) put(g, w[g]);
            } else {
#pragma unroll 1
                for (int g = 0; g < groups; g++) {
                    uint32_t w[NW];
                    fetch(g, w);
                    if (g == groups - 1) release();
                    put(g, w);
                }
            }
            epi_sync_all();  // the list of passes and the column scales are overwritten for the next tile
        }
        if (lane == 0) bulk_wait_all();
    }
    tc_fence_before();
    __syncthreads();
    if (TWO) pair_sync();  // neither block leaves while the other may still signal it or read its operands
    if (warp == 1) {
        if (TWO) pair_tmem_dealloc(tmem);
        else tmem_dealloc(tmem, 512);
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
encode_tiled_fn g_encode = nullptr;

int g_pairs = 74;  // pairs of blocks the device runs at once

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

bool encode2d(CUtensorMap* m, CUtensorMapDataType dt, const void* base, uint64_t inner, uint64_t outer, uint64_t pitch_bytes,
              uint32_t box_inner, uint32_t box_outer) {
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {pitch_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t es[2] = {1, 1};
    return g_encode(m, dt, 2, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cudaError_t plora_gemm_init() {
    if (!g_encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (!fn || q != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
        g_encode = reinterpret_cast<encode_tiled_fn>(fn);
    }
    cudaError_t e;
    auto init = [](auto* kernel, size_t smem) { return plora_kernel_shared(reinterpret_cast<const void*>(kernel), (int)smem); };
#define PLORA_GEMM_INIT(KIND, F32)                                                                                                         \
    if ((e = init(plora_gemm_fused_kernel<KIND, F32, 256, true>, gemm_smem(256, true)))) return e;   \
    if ((e = init(plora_gemm_fused_kernel<KIND, F32, 192, true>, gemm_smem(192, true)))) return e;   \
    if ((e = init(plora_gemm_fused_kernel<KIND, F32, 128, true>, gemm_smem(128, true)))) return e;   \
    if ((e = init(plora_gemm_fused_kernel<KIND, F32, 256, false>, gemm_smem(256, false)))) return e; \
    if ((e = init(plora_gemm_fused_kernel<KIND, F32, 192, false>, gemm_smem(192, false)))) return e
    PLORA_GEMM_INIT(0, false);
    PLORA_GEMM_INIT(0, true);
    PLORA_GEMM_INIT(1, false);
    PLORA_GEMM_INIT(1, true);
#undef PLORA_GEMM_INIT
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sms & ~1));
    cfg.blockDim = dim3(64 + G_EPI);
    cfg.dynamicSmemBytes = gemm_smem(256, true);
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, plora_gemm_fused_kernel<0, false, 256, true>, &cfg);
    if (e != cudaSuccess) return e;
    if (n < 1) return cudaErrorInvalidConfiguration;
    g_pairs = n;
    return cudaSuccess;
}

// Whether a layer's shapes fit the kernel: parts starting at multiples of 256 columns (so does every block),
// and x, W, y meeting the alignment of tensor copies. kind 0 = e4m3 x and W with scales, 1 = bf16.
bool plora_gemm_fits(int kind, const void* x, const void* w, const void* y, int ldy, int f32_out, int K, int n_parts,
                     const int* part_off) {
    if (!g_encode) return false;
    const int el = kind == 0 ? 1 : 2, yel = f32_out ? 4 : 2;
    if (((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)y & 15)) return false;
    if (((size_t)K * el) % 16 || ((size_t)ldy * yel) % 16) return false;
    for (int p = 0; p < n_parts; p++)
        if (part_off[p] % 256) return false;
    return true;
}

cudaError_t plora_launch_gemm_fused(int kind, const void* x, const float* st_, const void* w, const float* sn, int T, int N,
                                    int K, const int32_t* segs, SegLayout lay, const plora_desc* table, int n_parts,
                                    const int* part_off, const int* part_rows, const float* S, int lds, void* y, int ldy,
                                    int f32_out, bool tiles, int* status, bool pdl, cudaStream_t stream) {
    if (!g_encode) return cudaErrorNotSupported;
    CUtensorMap xmap, wmap, ymap;
    const CUtensorMapDataType dt = kind == 0 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int el = kind == 0 ? 1 : 2;
    // 256 output columns per tile, or fewer where that makes the rounds of the pairs shorter: a step of few tokens has few
    // tiles, and a round that is nearly empty costs as much as a full one. A step of K costs what it moves into an SM,
    // G_BM rows of x and the block's rows of W, of 128 bytes each. Tiles of 192 columns may span two parts, which adapter
    // passes do not, so they are for steps that cannot have long runs: begun as decoding steps, or of fewer
    // rows (FP8, 256 tokens, 24,576 columns, shrink and layer: 77.3 -> 74.9 us). Up to 128 tokens of such a step, blocks on their own take tiles of 256 or 192 columns where that costs less: layers too wide for
    // one round of pairs. FP8, 24,576 columns: 36 us in two rounds of pairs, 24 in one round of blocks (shrink and layer at
    // 70 tokens: 65 -> 53 us, at 128: 69 -> 57); the bf16 layers of a block at 70 tokens: 238 -> 218 us.
    const int blocks = 2 * g_pairs;
    int bn = 0;
    bool two = true;
    long long best = 0;
    auto consider = [&](int width, bool pair) {
        const int tm = pair ? 2 * G_BM : G_BM, places = pair ? g_pairs : blocks;
        const long long n = (long long)((T + tm - 1) / tm) * ((N + width - 1) / width);
        const long long cost = (n + places - 1) / places * (G_BM + gemm_w_rows(width, pair));
        if (bn != 0 && cost >= best) return;
        bn = width;
        two = pair;
        best = cost;
    };
    consider(256, true);
    if (!tiles) consider(192, true);
    consider(128, true);
    if (!tiles && T <= G_BM) {
        consider(256, false);
        consider(192, false);
    }
    if (!encode2d(&xmap, dt, x, (uint64_t)K, (uint64_t)T, (uint64_t)K * el, G_BKB / el, G_BM)) return cudaErrorInvalidValue;
    if (!encode2d(&wmap, dt, w, (uint64_t)K, (uint64_t)N, (uint64_t)K * el, G_BKB / el, (uint32_t)gemm_w_rows(bn, two))) return cudaErrorInvalidValue;
    if (!encode2d(&ymap, f32_out ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, y, (uint64_t)N,
                  (uint64_t)T, (uint64_t)ldy * (f32_out ? 4 : 2), f32_out ? 32 : 64, 32))
        return cudaErrorInvalidValue;
    GemmParts parts;
    parts.n = n_parts;
    for (int p = 0; p < PLORA_MAX_PARTS; p++) {
        parts.off[p] = p < n_parts ? part_off[p] : 0;
        parts.rows[p] = p < n_parts ? part_rows[p] : 0;
    }
    const int tm = two ? 2 * G_BM : G_BM;
    const long long n_tiles = (long long)((T + tm - 1) / tm) * ((N + bn - 1) / bn);
    const dim3 grid(two ? 2u * (unsigned)std::min<long long>(n_tiles, g_pairs) : (unsigned)std::min<long long>(n_tiles, blocks)), block(64 + G_EPI);
    auto launch = [&](auto* kernel) {
        return launch_pdl(kernel, grid, block, gemm_smem(bn, two), stream, pdl, xmap, wmap, ymap, st_, sn, T, N, K, segs, lay, table, parts, S, lds,
                          status);
    };
#define PLORA_GEMM_LAUNCH(KIND, F32)                                                  \
    return two ? launch(bn == 256   ? plora_gemm_fused_kernel<KIND, F32, 256, true>   \
                        : bn == 192 ? plora_gemm_fused_kernel<KIND, F32, 192, true>   \
                                    : plora_gemm_fused_kernel<KIND, F32, 128, true>)  \
               : launch(bn == 256 ? plora_gemm_fused_kernel<KIND, F32, 256, false>    \
                                  : plora_gemm_fused_kernel<KIND, F32, 192, false>)
    if (kind == 0) {
        if (f32_out) PLORA_GEMM_LAUNCH(0, true);
        PLORA_GEMM_LAUNCH(0, false);
    }
    if (f32_out) PLORA_GEMM_LAUNCH(1, true);
    PLORA_GEMM_LAUNCH(1, false);
#undef PLORA_GEMM_LAUNCH
}
