// One kernel per layer for the few-token work items: a thread-block cluster of 8 blocks takes one work item (up
// to 16 tokens of one slot, 8 at a time) and one group of its output columns. Block q of the cluster shrinks over the q-th
// eighth of the input features; the partial sums meet through distributed shared memory (no trip through global
// memory, no second launch); every block then expands its eighth of the cluster's columns. Replaces the
// lora_shrink + lora_expand pair of src/kernels/lora.cuh:23-126 when x and y are both ready at the call (after
// the layer's own matrix multiply).
//
// A layer is a chain of latencies from the dependency wait to the last store of y, and everything that can be known early is
// done before that wait. Order of events in a block:
//   1. one fetch of the work item's launch record (descriptor and token rows, written once per step);
//   2. bulk async copies of the block's inputs of the rows of A and of its share of B into shared memory, L2 prefetch hints
//      for the x and y lines it will touch (and, when asked for, an L2 prefetch of the same work item's slabs of
//      the next layer); addresses and predicates of the loads to come; A has landed;
//   3. the dependency wait (the kernel before, typically the layer's matrix multiply, wrote y);
//   4. x from L2 straight into operand registers, y of the first two steps of columns behind it; the next kernel of the stream
//      is released (its steps 1 and 2 then overlap the rest of this one);
//   5. shrink, exchange (the summed partials are stored into all eight blocks, with their own completion), expand.
// Nothing before step 3 binds a value of x or y, unless the caller vouched for x (early_x; the next kernel is then released at
// once). Cycles from the wait to the end of a block, one token of rank 16: 5,100 with the parts and shares walked after the wait, 3,300
// so; one layer then takes 2.9 us against 4.8 (x through bulk copies, partials fetched from the other blocks, y and S in
// tiles of 8 tokens), 64 tokens of 16 adapters 5.2 against 7.0. The release point, one token / 64 tokens, us per 16 layers: at kernel
// start 57 / 96, after the loads 57 / 95, after the shrink 69 / 106.
//
// Column groups: a cluster loads and multiplies the rows of A of the parts its columns meet, no others. A step of many work items
// takes as few groups as fit, since a B200 holds 33 clusters of such blocks; one of few items takes more, up to a
// step of columns per warp: one token over 24,576 columns goes to 96 blocks instead of 16.
//
// Arithmetic: tiles of the warp-level tensor-core instruction (m16n8k16, bf16 in, f32 accumulate), the shape the
// engine's own kernels use for their 16-token tiles; here the shrink has 16 rows of A by 8 tokens in a tile, the expand four tokens'
// three terms of S by 8 columns (plora_tiles.cuh). On the CUDA cores the step is bound by
// instruction issue (one conversion per bf16 element plus one multiply-add per token), not by memory; a 128-row
// tcgen05 tile would spend 1/8 or less of its rows on a work item. The f32 intermediate enters the expand as
// three bf16 terms (high, middle, low part), whose products with bf16 B are exact in f32, so no precision is
// given up against an f32 multiply-add chain.
//
// No registers spill, and none may: these kernels leave L1 no room, so a spilled value comes back from L2 (300 bytes of them
// doubled the time of a layer).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "plora_internal.h"
#include "plora_device.cuh"
#include "plora_tiles.cuh"

#define SITE_CLUSTER 8
#define SITE_THREADS 256
#define SITE_WARPS PLORA_TILE_WARPS
#define SITE_TOK 8  // tokens per pass over a work item
#define SITE_SMEM (112 * 1024)  // two blocks per SM: half of 228 KB, less the 1 KB the system keeps per block and the static part

namespace {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// a block's columns of one part, which it expands in one go
struct alignas(16) Seg {
    int r, ncols, boff, soff;  // ranks, columns; bytes to its rows of B and to the first of its ranks in a row of S
    long long ycol;            // first column of y
    int fast, pad;             // y rows that move in pieces of 4 columns, 16-byte aligned every eighth
};

// Columns per block when `pieces` blocks share `ntot` output columns: in eights, so that y moves in whole pieces
__host__ __device__ inline int site_share(int ntot, int pieces) { return ((ntot + pieces - 1) / pieces + 7) & ~7; }

// The slot's output columns, over the targeted parts laid end to end (rec.cat, rec.ntot), are cut into even shares of
// `share` columns, one per block of the layer's clusters. One warp: lane p finds what of part p falls into the block's share, and
// asks for its rows of B.
__device__ __forceinline__ void block_segs(const PloraRec& rec, int share, int piece, int ja, const void* Y, int ldy, int esize, int lane, Seg* segs,
                                           int* n_segs, unsigned char* Bs, uint64_t* bar) {
    const int p = lane & (PLORA_MAX_PARTS - 1);
    const int c_lo = min(rec.ntot, piece * share), c_hi = min(rec.ntot, c_lo + share);
    const int lo = max(c_lo, rec.cat[p]) - rec.cat[p];
    const int hi = rec.r[p] > 0 ? min(c_hi, rec.cat[p] + rec.rows[p]) - rec.cat[p] : 0;
    const int ncols = max(0, hi - lo), bytes = ncols * rec.r[p] * 2;
    // where the part's rows of B start in shared memory: the bytes of the parts before it
    int off = 0, total = 0;
#pragma unroll
    for (int q = 0; q < PLORA_MAX_PARTS; q++) {
        const int b = __shfl_sync(0xffffffffu, bytes, q);
        if (q < p) off += b;
        total += b;
    }
    const unsigned have = __ballot_sync(0xffffffffu, lane < PLORA_MAX_PARTS && ncols > 0);
    if (lane == 0) {
        *n_segs = __popc(have);
        if (have == 0) segs[0] = Seg{};
        if (total > 0) mbar_expect_tx(bar, (uint32_t)total);
    }
    __syncwarp();
    if (lane < PLORA_MAX_PARTS && ncols > 0) {
        bulk_g2s(Bs + off, reinterpret_cast<const bf16*>(rec.b[p]) + (size_t)lo * rec.r[p], (uint32_t)bytes, bar);
        Seg s;
        s.r = rec.r[p];
        s.ncols = ncols;
        s.boff = off;
        s.soff = (rec.r_off[p] - ja) * 2;
        s.ycol = (long long)rec.off[p] + lo;
        s.fast = (ncols & 7) == 0 && ((reinterpret_cast<uintptr_t>(Y) | ((size_t)ldy * esize) | (size_t)(s.ycol * esize)) & 15) == 0;
        s.pad = 0;
        segs[__popc(have & ((1u << lane) - 1u))] = s;
    }
}

// L2 prefetch of this block's eighth of `bytes` at `base` (both multiples of 16), 32 KB per request, one warp
__device__ __forceinline__ void prefetch_eighth(uint64_t base, uint64_t bytes, uint32_t crank, int lane) {
    const uint64_t per = ((bytes / SITE_CLUSTER) + 15) & ~(uint64_t)15;
    const uint64_t lo = min(bytes, per * crank), hi = min(bytes, lo + per);
    for (uint64_t o = lo + (uint64_t)lane * 32768; o < hi; o += 32 * 32768) {
        const uint32_t n = (uint32_t)min((uint64_t)32768, hi - o) & ~15u;
        if (n) bulk_prefetch_l2(reinterpret_cast<const unsigned char*>(base) + o, n);
    }
}

// 16 bytes to the same shared-memory offset in block `rank` of the cluster, counted on the same barrier there
__device__ __forceinline__ void st_async_peer(const void* p, float4 v, const uint64_t* bar, uint32_t rank) {
    uint32_t a, m;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(smem_u32(bar)), "r"(rank));
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(m)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status) {
    for (int i = 0; i < (1 << 20); i++)
        if (mbar_try_wait_cluster(bar, parity)) return true;
    atomicMax(status, PLORA_ERR_TIMEOUT);
    return false;
}
// "my reads of your shared memory are done": no memory ordering is asked of the arrival itself
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }

#define SITE_XSTEPS 8  // steps of 32 inputs per warp whose x is held in registers at a time

// The shrink's inner loop for one warp: acc (16 rows of A x 8 tokens per tile) += A . x over the steps of 32 inputs whose x is
// in registers. Rows of A are the multiply's 16-row operand and tokens its 8 columns. Its 16 input slots may be permuted freely as
// long as both operands agree: lane t of four holds inputs 8 t .. 8 t + 7 of a step, two multiplies' worth, as one
// 16-byte piece of either. a0: this lane's row and piece of the first of n steps; the lane has inputs in the first `mine` of them.
template <int TILES>
__device__ __forceinline__ void shrink_steps(float (&acc)[2][4], const uint4 (&xr)[SITE_XSTEPS], uint32_t a0, uint32_t kb_pad, int n, int mine) {
    // A step's rows of A are fetched before the multiplies of the step before (those of the first while x is on its way), and its
    // two multiplies of a tile go to accumulators of their own: half as long a chain of dependent multiplies.
    float odd[TILES][4];
#pragma unroll
    for (int i = 0; i < TILES; i++) odd[i][0] = odd[i][1] = odd[i][2] = odd[i][3] = 0.f;
    uint4 lo[TILES], hi[TILES];
    auto fetch = [&](int s) {
#pragma unroll
        for (int i = 0; i < TILES; i++) {
            const uint32_t at = a0 + (uint32_t)(i * 16) * kb_pad + (uint32_t)s * (SITE_WARPS * 64u);
            lo[i] = hi[i] = make_uint4(0u, 0u, 0u, 0u);
            if (s < mine) {  // (shared memory behind the inputs may hold anything)
                lo[i] = lds128(at);
                hi[i] = lds128(at + 8u * kb_pad);
            }
        }
    };
    fetch(0);
#pragma unroll
    for (int s = 0; s < SITE_XSTEPS; s++) {
        if (s >= n) break;
        uint32_t m[TILES][2][4];
#pragma unroll
        for (int i = 0; i < TILES; i++) {
            m[i][0][0] = lo[i].x, m[i][0][1] = hi[i].x, m[i][0][2] = lo[i].y, m[i][0][3] = hi[i].y;
            m[i][1][0] = lo[i].z, m[i][1][1] = hi[i].z, m[i][1][2] = lo[i].w, m[i][1][3] = hi[i].w;
        }
        if (s + 1 < SITE_XSTEPS) fetch(s + 1);
#pragma unroll
        for (int i = 0; i < TILES; i++) mma_16816(acc[i], m[i][0], xr[s].x, xr[s].y);
#pragma unroll
        for (int i = 0; i < TILES; i++) mma_16816(odd[i], m[i][1], xr[s].z, xr[s].w);
    }
#pragma unroll
    for (int i = 0; i < TILES; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][e] += odd[i][e];
}

template <RankWalk W>
using Walk = std::integral_constant<RankWalk, W>;

template <bool F32>
__global__ void __cluster_dims__(SITE_CLUSTER, 1, 1) __launch_bounds__(SITE_THREADS, 2)
    plora_site_gather_kernel(const bf16* __restrict__ X, int ldx, int K, const PloraRec* recs, int rec_cap,
                             const PloraRec* next_recs, void* Y, int ldy, PloraSiteShape sh, int mode,
                             int* __restrict__ status PLORA_BOUNDS_PARAM) {
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ __align__(8) uint64_t bars[3];  // A rows, B rows, the cluster's partials
    __shared__ PloraRec srec;
    __shared__ __align__(16) Seg segs[PLORA_MAX_PARTS];
    __shared__ int n_segs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t crank = cluster_rank();
    unsigned char* As = dsm;                                                 // this block's inputs of the cluster's rows of A, kb_pad apart
    float* Ps = reinterpret_cast<float*>(As + sh.a_bytes);                   // the warps' partial sums [warp][token][rc + 4]
    float* Rs = reinterpret_cast<float*>(As + sh.a_bytes + sh.p_bytes);      // the blocks' partial sums [block][token][rc]
    unsigned char* Bs = As + sh.a_bytes + sh.p_bytes + sh.r_bytes;           // this block's rows of B, part after part
    // the summed S as three bf16 planes [8][sp_pad] (high, middle, low term) and a fourth plane that stays zero
    unsigned char* S3 = Bs + sh.b_bytes;
    const uint32_t plane_bytes = SITE_TOK * (uint32_t)sh.sp_pad;
    for (uint32_t i = tid * 16u; i < plane_bytes; i += SITE_THREADS * 16u)
        *reinterpret_cast<uint4*>(S3 + 3u * plane_bytes + i) = make_uint4(0u, 0u, 0u, 0u);
    // The kernels after this one may start their prologues now: before their own waits they touch slabs and
    // launch records only (and x, where their caller vouched for it); every store of the path comes after a
    // wait, and every grid waits for its predecessor before it completes.
    // mode: bit 0 = the caller vouched for x; bits 1-3 = when the next kernel of the stream is released (0: at
    // once, 1: after the shrink, 2: after the exchange, 3: after the loads of x and y); bit 4 = ask L2 for the next layer's slabs too
    const int early_x = mode & 1, release_at = (mode >> 1) & 7;
    // bit 5 = the kernel before is the step's grouping, which writes the records: nothing is read, and nothing
    // released, before the dependency wait (the launch itself overlaps the grouping)
    const bool late = (mode & 32) != 0;
    bool triggered = release_at == 0 && !late;
    if (triggered) pdl_trigger();
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_init(&bars[2], 1);  // this block's own arrival; the bytes of all eight blocks' partials complete it
        mbar_fence_init();
    }
    cluster_arrive_relaxed();  // the barriers exist (published by the init fence); met before the first remote store
    bool met = false, waited = false, hints = true;
    if (late) {
        pdl_wait();
        waited = true;
        if (release_at == 0) {
            pdl_trigger();
            triggered = true;
        }
    }
    uint32_t ph_a = 0, ph_b = 0, ph_s = 0;  // barrier phases (each flips only when its barrier was used)
    // false once a bounded wait ran out: the block goes on meeting the cluster and waiting for what is still on its way into its shared
    // memory (copies of its own, the other blocks' partials), which must not arrive after it has left, and does no more work
    bool alive = true;
    const int k0 = (int)crank * sh.kchunk;
    const int klen = max(0, min(sh.kchunk, K - k0));
    const uint32_t kbytes = (uint32_t)klen * 2u;
    const int esize = F32 ? 4 : 2;
    // fragment coordinates of the tensor-core tile: this lane holds rows g and g + 8, columns 2 t and 2 t + 1
    const int g = lane >> 2, t4 = lane & 3, t2 = t4 * 2;
    // shrink: warp q takes the steps of 32 inputs q, q + 8, ...; a lane has no inputs in a last one that ends before its piece
    const int w_steps = (((klen + 31) >> 5) - warp + SITE_WARPS - 1) / SITE_WARPS;
    const int w_mine = ((klen - 8 * t4 + 31) >> 5) - warp > 0 ? (((klen - 8 * t4 + 31) >> 5) - warp + SITE_WARPS - 1) / SITE_WARPS : 0;
    const uint32_t a_lane = smem_u32(As) + (uint32_t)g * (uint32_t)sh.kb_pad + (uint32_t)warp * 64u + (uint32_t)t4 * 16u;
    for (int w = blockIdx.z; w < rec_cap; w += gridDim.z) {
        // ---- the one metadata fetch: the record's 208 live bytes into shared memory
        if (tid < 13) reinterpret_cast<uint4*>(&srec)[tid] = reinterpret_cast<const uint4*>(recs + w)[tid];
        __syncthreads();
        const int cnt = srec.cnt;
        if (cnt == 0) break;  // end of the list: the same decision in every block of the cluster
#ifdef PLORA_BOUNDS
        if (!rec_in_bounds(srec, bnd, K) || srec.cols != K) {  // the same decision in every block that reads this record
            if (tid == 0) atomicMax(status, PLORA_ERR_ARG);
            __syncthreads();
            continue;
        }
#endif
        // the rows of A of the parts that the cluster's columns meet: [ja, ja + R)
        const int share = site_share(srec.ntot, SITE_CLUSTER * (int)gridDim.y);
        const int c_lo = (int)blockIdx.y * SITE_CLUSTER * share, c_hi = min(srec.ntot, c_lo + SITE_CLUSTER * share);
        int ja = srec.rank, jb = 0;
#pragma unroll
        for (int p = 0; p < PLORA_MAX_PARTS; p++)
            if (srec.r[p] > 0 && srec.cat[p] < c_hi && srec.cat[p] + srec.rows[p] > c_lo) {
                ja = min(ja, srec.r_off[p]);
                jb = max(jb, srec.r_off[p] + srec.r[p]);
            }
        const int R = jb - ja;
        if (R <= 0) {  // the slot's adapter skips this layer, or its columns end before this cluster's: the same in every block
            __syncthreads();
            continue;
        }
        // quads of a token's partial sums, and the factor that divides by their number (exact for the at most 512 quads)
        const int nq = R >> 2;
        const uint32_t inv = (65536u + (uint32_t)nq - 1u) / (uint32_t)nq;
        // the work item's tokens, 8 at a time (a decoding batch rarely has more of one slot)
        for (int t0 = 0; t0 < cnt; t0 += SITE_TOK) {
            const int cn = min(SITE_TOK, cnt - t0);
            const int* tok = srec.tok + t0;
            // ---- slab requests (before the dependency wait)
            if (t0 == 0) {  // (a second pass finds the slabs in place)
                // the block's inputs of the rows of A, one bulk copy per row. The copies of the lanes of one warp are issued
                // one after another, so the rows go round the warps: row r is lane r / 8 of warp r % 8. (The barrier's one
                // arrival carries the whole byte count; copies that land before it only run the count down early.)
                if (klen > 0) {
                    const bf16* A = reinterpret_cast<const bf16*>(srec.a) + (size_t)ja * K + k0;
                    if (tid == 0) mbar_expect_tx(&bars[0], (uint32_t)R * kbytes);
                    for (int r = warp + SITE_WARPS * lane; r < R; r += SITE_THREADS)
                        bulk_g2s(As + (size_t)r * sh.kb_pad, A + (size_t)r * K, kbytes, &bars[0]);
                }
                // warp 1: the block's share of the output columns (lane p takes part p), and the copies of its rows of B
                if (warp == 1) block_segs(srec, share, (int)blockIdx.y * SITE_CLUSTER + (int)crank, ja, Y, ldy, esize, lane, segs, &n_segs, Bs, &bars[1]);
                __syncthreads();  // the share is known to every warp
            }
            const int nseg = n_segs;
            // ---- hints: the x and y lines this block will touch, and the next layer's slabs of this work item
            if (hints && warp >= 2) {
                const int t1 = tid - 64, n1 = SITE_THREADS - 64;
                if (klen > 0 && !early_x && !waited) {
                    const int lines = (int)((kbytes + 127) / 128);
                    for (int i = t1; i < cn * lines; i += n1) {
                        const int t = i / lines, l = i - t * lines;
                        prefetch_l2(reinterpret_cast<const unsigned char*>(X + (size_t)tok[t] * ldx + k0) + (size_t)l * 128);
                    }
                }
#pragma unroll 1
                for (int q = 0; q < nseg; q++) {
                    const size_t len = (size_t)segs[q].ncols * esize;
                    const int lines = (int)((len + 127) / 128) + 1;
                    for (int i = t1; i < cn * lines; i += n1) {
                        const int t = i / lines, l = i - t * lines;
                        const size_t start = ((size_t)tok[t] * ldy + segs[q].ycol) * esize;
                        const size_t at = (start & ~(size_t)127) + (size_t)l * 128;
                        if (at < start + len) prefetch_l2(reinterpret_cast<const unsigned char*>(Y) + at);
                    }
                }
            }
            if (next_recs != nullptr && warp == 1 && blockIdx.y == 0 && t0 == 0) {
                // the same work item's launch record at the next layer (the records are written for all layers at
                // once) is asked into L2, and, when the caller wants it, an eighth of each of its slabs
                const PloraRec* nr = next_recs + w;
                if (crank == 0 && lane < 2) prefetch_l2(reinterpret_cast<const unsigned char*>(nr) + 128 * lane);
                if (mode & 16) {
                    const int4 head = __ldcg(reinterpret_cast<const int4*>(nr));  // cn, slot, rank, cols
                    if (head.x > 0 && head.z > 0) {
                        prefetch_eighth(__ldcg(&nr->a), (uint64_t)head.z * (uint64_t)head.w * 2u, crank, lane);
#pragma unroll 1
                        for (int p = 0; p < PLORA_MAX_PARTS; p++) {
                            const int rp = __ldcg(&nr->r[p]);
                            if (rp > 0) prefetch_eighth(__ldcg(&nr->b[p]), (uint64_t)__ldcg(&nr->rows[p]) * (uint64_t)rp * 2u, crank, lane);
                        }
                    }
                }
            }
            hints = false;
            // ---- everything that the rest of the pass will need and that is known by now: where this lane's x is (the token of
            // column g of the multiply), and its y of the first two steps of the block's first columns
            const bf16* xrow = X + (size_t)(g < cn ? tok[g] : 0) * ldx + k0 + warp * 32 + 8 * t4;
            const int x_steps = g < cn ? w_mine : 0;
            const Seg first = segs[0];  // (of zeros where the block has no columns)
            const int qtok = g & 3;     // the token whose y this lane moves (of the first four), and its columns of a step
            const int qcol = warp * 32 + 8 * t4 + 4 * (g >> 2);
            const bool ahead = first.fast != 0 && qtok < cn;
            const unsigned char* yahead = reinterpret_cast<const unsigned char*>(Y) + ((size_t)(ahead ? tok[qtok] : 0) * ldy + first.ycol + qcol) * esize;
            const bool ahead0 = ahead && qcol < first.ncols, ahead1 = ahead && qcol + SITE_WARPS * 32 < first.ncols;
            if (klen > 0 && t0 == 0) {
                alive = mbar_wait(&bars[0], ph_a, status) && alive;
                ph_a ^= 1;
            }
            if (!waited && !early_x) {
                pdl_wait();
                waited = true;
            }
            // ---- x straight into operand registers, all steps at once
            uint4 xr[SITE_XSTEPS];
            auto load_x = [&](int s0) {
#pragma unroll
                for (int s = 0; s < SITE_XSTEPS; s++) {
                    xr[s] = make_uint4(0u, 0u, 0u, 0u);
                    if (s0 + s < x_steps) xr[s] = __ldcg(reinterpret_cast<const uint4*>(xrow + (size_t)(s0 + s) * (SITE_WARPS * 32)));
                }
            };
            load_x(0);
            // ... and y, on its way while the shrink and the exchange run
            YQuad<F32> y0, y1;
            y0.clear();
            y1.clear();
            const bool fetched = waited;
            if (fetched) {
                if (ahead0) y0.load(yahead);
                if (ahead1) y1.load(yahead + SITE_WARPS * 32 * esize);
            }
            if (!triggered && release_at == 3) {
                pdl_trigger();
                triggered = true;
            }
            // ---- shrink over this block's eighth of the inputs, 32 rows of A at a time
            for (int j0 = 0; j0 < R; j0 += 32) {
                float acc[2][4];
#pragma unroll
                for (int i = 0; i < 2; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
                const int tiles = min(2, (R - j0) >> 4);
                for (int s0 = 0; alive && s0 < w_steps; s0 += SITE_XSTEPS) {
                    if (s0 > 0 || (j0 > 0 && w_steps > SITE_XSTEPS)) load_x(s0);  // (else still in registers)
                    const uint32_t a0 = a_lane + (uint32_t)j0 * (uint32_t)sh.kb_pad + (uint32_t)s0 * (SITE_WARPS * 64u);
                    if (tiles == 1) shrink_steps<1>(acc, xr, a0, (uint32_t)sh.kb_pad, w_steps - s0, w_mine - s0);
                    else shrink_steps<2>(acc, xr, a0, (uint32_t)sh.kb_pad, w_steps - s0, w_mine - s0);
                }
                float* wp = Ps + (size_t)warp * SITE_TOK * (sh.rc + 4) + j0 + g;
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    if (i < tiles) {
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            if (t2 + e < cn) {
                                wp[(t2 + e) * (sh.rc + 4) + i * 16] = acc[i][e];
                                wp[(t2 + e) * (sh.rc + 4) + i * 16 + 8] = acc[i][2 + e];
                            }
                        }
                    }
                }
            }
            if (tid == 0) mbar_expect_tx(&bars[2], (uint32_t)(SITE_CLUSTER * cn * R * 4));
            __syncthreads();
            if (!triggered && release_at == 1) {
                pdl_trigger();
                triggered = true;
            }
            if (!met) {
                cluster_wait();  // everybody's barriers exist
                met = true;
            }
            // ---- the eight warps' partials are added in warp order, four rows of a token at a time, and every sum goes to all
            // eight blocks at once: a store that arrives with its own completion takes one way through the cluster, where an
            // arrival, a wait and a remote load took three
            for (int i = tid; i < cn * nq * SITE_CLUSTER; i += SITE_THREADS) {
                const int q = i >> 3, t = (int)(((uint32_t)q * inv) >> 16), j = 4 * (q - t * nq);
                const float* p = Ps + (size_t)t * (sh.rc + 4) + j;
                float4 v = *reinterpret_cast<const float4*>(p);
#pragma unroll
                for (int u = 1; u < SITE_WARPS; u++) {
                    const float4 b = *reinterpret_cast<const float4*>(p + (size_t)u * SITE_TOK * (sh.rc + 4));
                    v.x += b.x, v.y += b.y, v.z += b.z, v.w += b.w;
                }
                st_async_peer(Rs + (size_t)(crank * SITE_TOK + t) * sh.rc + j, v, &bars[2], (uint32_t)(i & 7));
            }
            if (nseg > 0 && t0 == 0) {  // (a later pass finds the rows of B in place)
                alive = mbar_wait(&bars[1], ph_b, status) && alive;
                ph_b ^= 1;
            }
            alive = mbar_wait_cluster(&bars[2], ph_s, status) && alive;
            ph_s ^= 1;
            // added in block order, as three bf16 terms whose sum is the f32 value
            for (int i = tid; i < 2 * cn * nq; i += SITE_THREADS) {
                const int t = (int)(((uint32_t)(i >> 1) * inv) >> 16), j = 2 * (i - 2 * t * nq);
                const float* p = Rs + (size_t)t * sh.rc + j;
                float2 v = *reinterpret_cast<const float2*>(p);
#pragma unroll
                for (int q = 1; q < SITE_CLUSTER; q++) {
                    const float2 b = *reinterpret_cast<const float2*>(p + (size_t)q * SITE_TOK * sh.rc);
                    v.x += b.x, v.y += b.y;
                }
                const __nv_bfloat162 hi = __floats2bfloat162_rn(v.x, v.y);
                const float2 hf = __bfloat1622float2(hi);
                const float2 r1 = make_float2(v.x - hf.x, v.y - hf.y);
                const __nv_bfloat162 mid = __floats2bfloat162_rn(r1.x, r1.y);
                const float2 mf = __bfloat1622float2(mid);
                const __nv_bfloat162 lo = __floats2bfloat162_rn(r1.x - mf.x, r1.y - mf.y);
                unsigned char* s3 = S3 + (size_t)t * sh.sp_pad + (size_t)j * 2;
                *reinterpret_cast<__nv_bfloat162*>(s3) = hi;
                *reinterpret_cast<__nv_bfloat162*>(s3 + plane_bytes) = mid;
                *reinterpret_cast<__nv_bfloat162*>(s3 + 2 * plane_bytes) = lo;
            }
            if (!triggered) {
                pdl_trigger();
                triggered = true;
            }
            if (!waited) {             // early_x: everything so far ran ahead of the kernel before; y must not
                pdl_wait();
                waited = true;
            }
            __syncthreads();
            cluster_arrive_relaxed();  // (every warp behind its reads of Rs) the others may send the next pass's partials
            // ---- expand over this block's share of the output columns
            if (alive) {
#pragma unroll 1
                for (int q = 0; q < nseg; q++) {
                    const Seg sg = segs[q];
                    const uint32_t s3 = smem_u32(S3) + (uint32_t)sg.soff, b = smem_u32(Bs) + (uint32_t)sg.boff;
                    auto expand = [&](auto walk, auto whole, int q0) {  // four tokens at a time
                        expand_quads<decltype(walk)::value, F32, decltype(whole)::value>(s3 + (uint32_t)q0 * (uint32_t)sh.sp_pad, (uint32_t)sh.sp_pad, plane_bytes, b, sg.r,
                                                                                         sg.ncols, Y, ldy, sg.ycol, tok + q0, min(4, cn - q0), warp, lane,
                                                                                         fetched && q == 0 && q0 == 0, y0, y1);
                    };
                    if (sg.fast) {
#pragma unroll 1
                        for (int q0 = 0; q0 < cn; q0 += 4) {
                            if (sg.r == 16) expand(Walk<R16>(), std::true_type(), q0);
                            else if (sg.r == 32) expand(Walk<R32>(), std::true_type(), q0);
                            else if (sg.r & 16) expand(Walk<ODD>(), std::true_type(), q0);
                            else expand(Walk<EVEN>(), std::true_type(), q0);
                        }
                    } else {
#pragma unroll 1
                        for (int q0 = 0; q0 < cn; q0 += 4) {
                            if (sg.r & 16) expand(Walk<ODD>(), std::false_type(), q0);
                            else expand(Walk<EVEN>(), std::false_type(), q0);
                        }
                    }
                }
            }
            cluster_wait();   // nobody reads what this block sent any more
            __syncthreads();  // shared memory is reused by the next pass or work item
        }
    }
    if (!met) cluster_wait();  // a block must not leave while a peer may still be arriving at the start-up barrier
    // A grid completes only after the grids before it. Blocks with work have waited; of the blocks that found none,
    // one waits for all (a grid is complete only when every block has left), so that the others give their places
    // on the SMs back at once instead of holding them until the kernel before has finished.
    if (!waited && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) pdl_wait();
}

PloraSiteShape shape_for(int K, int n_parts, const int* part_rows, int max_rank, int nsub) {
    PloraSiteShape s;
    s.kchunk = ((K + SITE_CLUSTER - 1) / SITE_CLUSTER + 31) & ~31;
    s.kb_pad = ((s.kchunk * 2 + 127) & ~127) + 64;
    // Whichever parts an adapter targets: the most of them that one cluster's columns meet, and the widest share
    int most = 1, wide = 0;
    for (int set = 1; set < 1 << n_parts; set++) {
        int ntot = 0;
        for (int p = 0; p < n_parts; p++)
            if (set >> p & 1) ntot += part_rows[p];
        const int share = site_share(ntot, SITE_CLUSTER * nsub);
        wide = std::max(wide, share);
        for (int y = 0; y < nsub; y++) {
            const int lo = y * SITE_CLUSTER * share, hi = std::min(ntot, lo + SITE_CLUSTER * share);
            int met = 0, at = 0;
            for (int p = 0; p < n_parts; p++) {
                if (!(set >> p & 1)) continue;
                met += at < hi && at + part_rows[p] > lo;
                at += part_rows[p];
            }
            most = std::max(most, met);
        }
    }
    s.rc = most * max_rank;
    s.sp_pad = (s.rc + 8) * 2;
    s.a_bytes = s.rc * s.kb_pad;
    s.p_bytes = SITE_WARPS * SITE_TOK * (s.rc + 4) * 4;
    s.r_bytes = SITE_CLUSTER * SITE_TOK * s.rc * 4;
    // the tile loads of the last columns of a part may run up to 31 rows past the share
    s.b_bytes = ((wide + 32 * n_parts) * max_rank * 2 + 127) & ~127;
    return s;
}

int shape_smem(const PloraSiteShape& s) { return s.a_bytes + s.p_bytes + s.r_bytes + s.b_bytes + 4 * SITE_TOK * s.sp_pad; }

// the clusters of such blocks that the device runs at once (0 on failure)
int clusters_at_once(int smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SITE_CLUSTER, 1, 16);
    cfg.blockDim = dim3(SITE_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, plora_site_gather_kernel<false>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace

cudaError_t plora_site_init() {
    // The split of an SM's memory between L1 and shared memory is fixed while any block runs on it. Layers of
    // different widths ask for different amounts of shared memory per block; left to itself the driver would pick
    // a split per launch, and a block of the next layer would then find no room beside the blocks still running
    // under a smaller split. Every launch of this kernel asks for the largest split.
    cudaError_t e = cudaSuccess;
    for (int f32 = 0; f32 < 2 && e == cudaSuccess; f32++) {
        const void* fn = f32 ? reinterpret_cast<const void*>(plora_site_gather_kernel<true>)
                             : reinterpret_cast<const void*>(plora_site_gather_kernel<false>);
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    return e;
}

// Whether the cluster kernel or the shrink / expand pair is the better one for a layer that the cluster kernel could run. It may
// depend on the layer and the largest rank alone: a rule on the step would let a token's result depend on its batch.
// Column groups make ever larger layers fit, but each group repeats the shrink, and 33 clusters run at a time: such layers are faster as
// clusters in steps of few items and slower in steps of many. The line is drawn where a block's inputs of all parts' rows of A
// (every 64 of them at least the eight warps' sums over them), eight tokens of x, its columns of B out of four groups and S leave
// no room for two blocks per SM. Beyond it, four layers, clusters / pairs in us for 1, 8, 16 and 64 tokens of as many adapters and
// 128 tokens of 8:
//   4096 -> 2 x 12288, rank 32   25 / 35   39 / 51   65 / 63   205 / 139   87 / 74
//   2048 -> 2 x 6144,  rank 48   25 / 35   37 / 50   62 / 61   193 / 133   77 / 70
//   1024 -> 2 x 3072,  rank 64   26 / 33   38 / 40   60 / 49   183 /  98   77 / 51
// Within it the most clusters lose is (3072 -> 3072, rank 64)  25 / 35   31 / 40   49 / 48   148 /  85   69 / 53,
// and most layers gain throughout (4096 -> 4096, rank 16       23 / 32   25 / 35   25 / 40    52 /  63   41 / 44).
bool clusters_pay(int K, int n_parts, int total, int max_rank) {
    const int rows = n_parts * max_rank, kchunk = ((K + SITE_CLUSTER - 1) / SITE_CLUSTER + 7) & ~7;
    const size_t pitch = (size_t)kchunk * 2 + (kchunk / 8 % 2 ? 32 : 16), in64 = std::min(rows, 64);
    const size_t a = (std::max(in64 * pitch, in64 * SITE_WARPS * PLORA_WORK_TOKENS * 4) + 127) / 128 * 128 * (size_t)((rows + 63) / 64);
    const size_t x = (SITE_TOK * pitch + 127) / 128 * 128;
    const size_t share = (((size_t)total + 4 * SITE_CLUSTER - 1) / (4 * SITE_CLUSTER) + 1) / 2 * 2;
    const size_t b = ((share + 32 * n_parts) * max_rank * 2 + 127) / 128 * 128;
    const size_t s = (size_t)PLORA_WORK_TOKENS * rows * 4 + (size_t)4 * PLORA_WORK_TOKENS * (rows + 8) * 2;
    return rows <= 256 && a + x + b + s <= 111 * 1024;
}

// Plans of the cluster kernel for one layer, by column groups per work item: those with which two blocks share an SM (one SM
// cannot take a whole cluster of 8, and a B200 has room for only 15 clusters of 8 at one block per SM). Empty where nothing
// fits (13 tokens of 8 adapters at rank 32, four layers: 240 us with one block per SM, 150 as pairs) or clusters do not pay: such
// a layer takes the shrink / expand pair. What does not fit at rank 64 and 4096 inputs are the partial sums of eight tokens; four tokens
// a pass would, but then the pair is the better one from 16 items on. Four layers, clusters so / pairs in us, steps as above:
//   4096 -> 4096, rank 64        27 / 35   39 / 42   61 / 47   197 /  97   95 / 51
//   4096 -> 1024, rank 64        25 / 34   27 / 38   29 / 40    71 /  80   67 / 47
std::vector<PloraSitePlan> plora_site_plans(int K, int n_parts, const int* part_rows, int max_rank) {
    std::vector<PloraSitePlan> out;
    int total = 0;
    for (int p = 0; p < n_parts; p++) total += part_rows[p];
    if (!clusters_pay(K, n_parts, total, max_rank)) return out;
    for (int nsub : {1, 2, 3, 4, 6, 8, 12, 16}) {
        if (nsub > 4 && out.empty()) break;  // (as few clusters as that run at once, and every group reads x again)
        PloraSitePlan pl;
        pl.shape = shape_for(K, n_parts, part_rows, max_rank, nsub);
        if (pl.shape.rc > 256 || shape_smem(pl.shape) > SITE_SMEM) continue;
        pl.nsub = nsub;
        pl.smem = shape_smem(pl.shape);
        pl.max_clusters = clusters_at_once(pl.smem);
        if (pl.max_clusters < nsub) continue;
        out.push_back(pl);
        if (site_share(total, SITE_CLUSTER * nsub) <= SITE_WARPS * 32) break;  // every warp has one step of columns
    }
    return out;
}

cudaError_t plora_launch_site(const void* x, int ldx, int K, const PloraRec* recs, int rec_cap, const PloraRec* next_recs,
                              void* y, int ldy, int f32_out, const PloraSitePlan& plan, int work_cap, int mode, const PloraBounds& bnd,
                              int* status, bool pdl, cudaStream_t st) {
    (void)bnd;
    // one wave: work items beyond the clusters the device runs at once are walked in a loop, so that every block
    // of the grid starts (and releases the next kernel) at once
    const int z = std::min(std::min(work_cap, PLORA_REC_TERM), std::max(1, plan.max_clusters / plan.nsub));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SITE_CLUSTER, (unsigned)plan.nsub, (unsigned)z);
    cfg.blockDim = dim3(SITE_THREADS);
    cfg.dynamicSmemBytes = (size_t)plan.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    if (f32_out)
        return cudaLaunchKernelEx(&cfg, plora_site_gather_kernel<true>, reinterpret_cast<const bf16*>(x), ldx, K, recs, rec_cap,
                                  next_recs, y, ldy, plan.shape, mode, status PLORA_BOUNDS_ARG(bnd));
    return cudaLaunchKernelEx(&cfg, plora_site_gather_kernel<false>, reinterpret_cast<const bf16*>(x), ldx, K, recs, rec_cap,
                              next_recs, y, ldy, plan.shape, mode, status PLORA_BOUNDS_ARG(bnd));
}
