// sm_100a kernels of the adapter path and their launchers.
//
//   plora_meta_tiles_kernel  cu[], seq_slot[] -> the engine's tile words (src/sched.rs:1096-1104), on the device
//   plora_meta_group_kernel  tile words -> tokens regrouped by slot (gather work items) and long runs cut
//                            into tensor-core tiles; stable, so results do not depend on scheduling
//   plora_shrink_gather      S_split[t, :] = x[t, k-chunk] . A_slot[:, k-chunk]^T   (replaces lora.cuh:23-67)
//   plora_expand_gather      y[t, off_p + n] += sum_j S[t, r_off_p + j] B_p[n, j]   (replaces lora.cuh:74-126)
//
// The shrink writes one partial per K-split instead of accumulating with float atomics; the expand adds
// the partials in split order, so S needs no zeroing and the result is reproducible bit for bit.
#include <cuda_bf16.h>

#include "plora_internal.h"
#include "plora_device.cuh"
#include "plora_tc.cuh"
#include "plora_tiles.cuh"


namespace {

// Exclusive scan of one 64-bit word per thread over a block of 1024 threads (several counts packed into one word are
// scanned together). `sh` holds 33 words; it may be used again after the next __syncthreads().
__device__ __forceinline__ unsigned long long block_scan_excl(unsigned long long v, unsigned long long& total, unsigned long long* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const unsigned long long t = sh[lane];
        unsigned long long ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += u;
        }
        sh[lane] = ti - t;
        if (lane == 31) sh[32] = ti;
    }
    __syncthreads();
    total = sh[32];
    return incl - v + sh[warp];
}

// ---------------------------------------------------------------------------------------------
// Tile words from the step's sequences: for each sequence in order with a slot, chunks of 16 tokens
// (start, len, slot); word 0 is the count. One block of 1024 threads.
__global__ void __launch_bounds__(1024) plora_meta_tiles_kernel(const int* __restrict__ cu,
                                                                 const int* __restrict__ seq_slot, int n_seqs,
                                                                 int* __restrict__ tiles, int cap_tiles,
                                                                 int* __restrict__ status) {
    __shared__ unsigned long long sh[33];
    __shared__ int s_first[1024], s_start[1024], s_n[1024], s_slot[1024];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_trigger();  // the grouping kernel waits for this grid before it reads a word
    int carry = 0;
    for (int base = 0; base < n_seqs; base += 1024) {
        const int i = base + tid;
        int start = 0, n = 0, slot = 0, nt = 0;
        if (i < n_seqs) {
            start = cu[i];
            n = cu[i + 1] - start;
            slot = seq_slot[i];
            if (n < 0) n = 0;
            nt = slot != 0 ? (n + PLORA_TILE - 1) / PLORA_TILE : 0;
        }
        unsigned long long total;
        const int excl = (int)block_scan_excl((unsigned long long)nt, total, sh);
        s_first[tid] = carry + excl;
        s_start[tid] = start;
        s_n[tid] = n;
        s_slot[tid] = slot;
        __syncthreads();
        const int here = min(1024, n_seqs - base);
        for (int q = warp; q < here; q += 32) {
            const int qs = s_slot[q];
            if (qs == 0) continue;
            const int qn = s_n[q], q0 = s_start[q], qf = s_first[q];
            const int qt = (qn + PLORA_TILE - 1) / PLORA_TILE;
            for (int k = lane; k < qt; k += 32) {
                const int idx = qf + k;
                if (idx < cap_tiles) {
                    tiles[1 + 3 * idx] = q0 + k * PLORA_TILE;
                    tiles[2 + 3 * idx] = min(qn - k * PLORA_TILE, PLORA_TILE);
                    tiles[3 + 3 * idx] = qs;
                }
            }
        }
        carry += (int)total;
        __syncthreads();
    }
    if (tid == 0) {
        if (carry > cap_tiles) {
            tiles[0] = 0;
            atomicMax(status, PLORA_ERR_CAPACITY);
        } else {
            tiles[0] = carry;
        }
    }
}

// ---------------------------------------------------------------------------------------------
#define SHR_PAD 20  // floats between the token rows of a warp's partial

// One launch record: gather work item w resolved against one layer's descriptor table, so that the kernels of
// that layer make one metadata fetch per block. `o` is the record's 16 uint4.
// Returns the item's units of the few-token kernels (pack_units).
__device__ __forceinline__ unsigned long long write_record(uint4* o, const int* segs, const SegLayout& lay, const plora_desc* table, int w,
                                             int cols, int nsplit, int most) {
    const uint4* work = reinterpret_cast<const uint4*>(segs + lay.work() + PLORA_WORK_WORDS * w);
    const uint4 head = work[0];  // slot, perm start, count, 0
    const int slot = (int)head.x;
    const uint4* d = reinterpret_cast<const uint4*>(table + slot);  // 112 bytes: a, b[4], rank, r, r_off, off, rows
    uint4 dv[7];
#pragma unroll
    for (int i = 0; i < 7; i++) dv[i] = d[i];
    // Desc: a | b0 b1 | b2 b3 | rank r0 r1 r2 | r3 ro0 ro1 ro2 | ro3 o0 o1 o2 | o3 rows0 rows1 rows2 | rows3 pad
    const uint32_t* dw = reinterpret_cast<const uint32_t*>(dv);
    int r[PLORA_MAX_PARTS], rows[PLORA_MAX_PARTS];
#pragma unroll
    for (int p = 0; p < PLORA_MAX_PARTS; p++) r[p] = (int)dw[11 + p], rows[p] = (int)dw[23 + p];
    const unsigned long long units = pack_units(expand_item_units(r, rows, (int)head.z, most), shrink_item_units((int)dw[10], nsplit));
    o[0] = make_uint4(head.z, head.x, dw[10], (uint32_t)cols);  // cnt, slot, rank, cols
    o[1] = make_uint4(dw[0], dw[1], dw[2], dw[3]);              // a, b[0]
    o[2] = make_uint4(dw[4], dw[5], dw[6], dw[7]);              // b[1], b[2]
    o[3] = make_uint4(dw[8], dw[9], dw[11], dw[12]);            // b[3], r[0], r[1]
    o[4] = make_uint4(dw[13], dw[14], dw[15], dw[16]);          // r[2], r[3], r_off[0], r_off[1]
    o[5] = make_uint4(dw[17], dw[18], dw[19], dw[20]);          // r_off[2], r_off[3], off[0], off[1]
    o[6] = make_uint4(dw[21], dw[22], dw[23], dw[24]);          // off[2], off[3], rows[0], rows[1]
    // the slot's output columns over its targeted parts laid end to end
    uint32_t cat[PLORA_MAX_PARTS], ntot = 0;
#pragma unroll
    for (int p = 0; p < PLORA_MAX_PARTS; p++) {
        cat[p] = ntot;
        if ((int)dw[11 + p] > 0) ntot += dw[23 + p];
    }
    o[7] = make_uint4(dw[25], dw[26], ntot, 0u);                // rows[2], rows[3], ntot
    o[8] = work[1];                                             // the token rows
    o[9] = work[2];
    o[10] = work[3];
    o[11] = work[4];
    o[12] = make_uint4(cat[0], cat[1], cat[2], cat[3]);
    return units;
}

// ---------------------------------------------------------------------------------------------
// Regroup the tile words by slot. Runs = maximal ranges of contiguous tokens of one slot. Runs of at
// least lay.run_min tokens become tensor-core tiles; the rest are gathered by slot: perm lists their
// token rows ordered by (slot, position in the tile list), cut into work items of <= 16 tokens.
//
// Every block then writes the launch records of its layers (blockIdx.x, blockIdx.x + gridDim.x, ...): each gather work
// item resolved against the layer's descriptor table. The list of a layer ends with records whose cnt is 0.
//
// The kernel is a chain of latencies (fetch, scans, fetch of the descriptors), not of bytes. So the blocks do not
// share the grouping, which would take a grid-wide wait: each of them does all of it, with the same result, and writes
// the regrouped rows and work items that it will read back itself (the same words from every block); block 0 also
// writes what only later kernels read. Counts that are scanned together share one 64-bit scan. One block wrote the
// records of all layers before: 9 us for a single token over 16 layers, 13 us for 64 tokens, 19-27 us for a prefill
// step, against what bench.py reports as meta_us now.
__global__ void __launch_bounds__(1024) plora_meta_group_kernel(const int* tiles, int* __restrict__ segs,
                                                                 SegLayout lay, int* __restrict__ status,
                                                                 const plora_desc* __restrict__ tables,
                                                                 const int* __restrict__ site_cols, int n_sites,
                                                                 PloraRec* __restrict__ recs, int rec_cap,
                                                                 int* __restrict__ prefix, int expand_grid) {
    extern __shared__ int sm[];
    __shared__ int first_item;  // (thread 0's) units of a layer's first item in the expand
    __shared__ unsigned long long sh[4][33];  // a row per scan in flight: no barrier between one scan and the next
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cap = lay.cap_tiles, S1 = lay.max_slots + 1;
    const bool first = blockIdx.x == 0;
    int* run_tok = sm;  // [cap + 1]: tokens of the runs before; the length of run r is run_tok[r + 1] - run_tok[r]
    int* run_start = run_tok + cap + 1;
    int* run_slot = run_start + cap;
    int* run_pos = run_slot + cap;
    int* cnt = run_pos + cap;
    int* seg_base = cnt + S1;
    int* fill = seg_base + S1;
    int* whist = fill + S1;  // [32][S1]

    // what needs no tile word, under the wait for the kernel before (the tile words, or the step before, which may
    // still be reading the metadata)
    for (int i = tid; i < S1; i += 1024) cnt[i] = fill[i] = seg_base[i] = 0;
    for (int i = tid; i < 32 * S1; i += 1024) whist[i] = 0;
    pdl_trigger();  // (the first kernel of the step waits for this grid before it reads a record)
    pdl_wait();

    // the first tile words are fetched together with their count (`tiles` is not __restrict__: its writer may run when this kernel begins)
    int w0 = 0, w1 = 0, w2 = 0;
    if (tid < cap) {
        w0 = tiles[1 + 3 * tid];
        w1 = tiles[2 + 3 * tid];
        w2 = tiles[3 + 3 * tid];
    }
    int n_tiles = tiles[0];
    bool bad = false;
    if (n_tiles < 0 || n_tiles > cap) {
        n_tiles = 0;
        bad = true;
    }
    if (first)
        for (int i = tid; i < lay.max_tokens; i += 1024) segs[lay.tslot() + i] = 0;
    __syncthreads();

    // runs
    int n_runs = 0, n_tok = 0;
    for (int base = 0; base < n_tiles; base += 1024) {
        const int i = base + tid;
        int head = 0, start = 0, len = 0, slot = 0;
        if (i < n_tiles) {
            if (base > 0) {
                w0 = tiles[1 + 3 * i];
                w1 = tiles[2 + 3 * i];
                w2 = tiles[3 + 3 * i];
            }
            start = w0;
            len = w1;
            slot = w2;
        }
        // the tile before: a neighbour's, or fetched by the first lane of a warp
        int ps = __shfl_up_sync(0xffffffffu, start, 1), pl = __shfl_up_sync(0xffffffffu, len, 1), pslot = __shfl_up_sync(0xffffffffu, slot, 1);
        if (i < n_tiles) {
            if (lane == 0 && i > 0) {
                ps = tiles[1 + 3 * (i - 1)];
                pl = tiles[2 + 3 * (i - 1)];
                pslot = tiles[3 + 3 * (i - 1)];
            }
            if (slot < 0 || slot > lay.max_slots || len < 1 || len > PLORA_TILE || start < 0 ||
                start + len > lay.max_tokens) {
                bad = true;
                slot = 0;
                len = 0;
                start = 0;
            } else if (recs != nullptr && blockIdx.x < (unsigned)n_sites) {
                // the descriptor this block will resolve first
                prefetch_l2(tables + (size_t)blockIdx.x * (size_t)S1 + slot);
            }
            head = i == 0 || !(pslot == slot && ps + pl == start);
        }
        unsigned long long total;
        const unsigned long long excl = block_scan_excl(((unsigned long long)head << 32) | (unsigned)len, total, sh[(base >> 10) & 1]);
        const int rid = n_runs + (int)(excl >> 32);
        if (head) {
            run_start[rid] = start;
            run_slot[rid] = slot;
            run_tok[rid] = n_tok + (int)(excl & 0xffffffffu);
        }
        n_runs += (int)(total >> 32);
        n_tok += (int)(total & 0xffffffffu);
    }
    if (tid == 0) run_tok[n_runs] = n_tok;
    __syncthreads();
    // the slot of every token row: 16 lanes a tile
    if (first)
        for (int i = tid; i < 16 * n_tiles; i += 1024) {
            const int t = i >> 4, k = i & 15;
            const int start = tiles[1 + 3 * t], len = tiles[2 + 3 * t], slot = tiles[3 + 3 * t];
            if (slot >= 0 && slot <= lay.max_slots && len >= 1 && len <= PLORA_TILE && start >= 0 && start + len <= lay.max_tokens && k < len)
                segs[lay.tslot() + start + k] = slot;
        }

    // classify runs; tensor-core tiles (none when every run stays under run_min)
    const bool any_mma = lay.run_min <= n_tok;
    int n_mma = 0;
    for (int base = 0; base < n_runs; base += 1024) {
        const int r = base + tid;
        int nm = 0, len = 0, slot = 0, start = 0;
        if (r < n_runs) {
            len = run_tok[r + 1] - run_tok[r];
            slot = run_slot[r];
            start = run_start[r];
            if (slot == 0 || len == 0) run_pos[r] = -1;
            else if (len >= lay.run_min) {
                nm = (len + PLORA_MMA_TOKENS - 1) / PLORA_MMA_TOKENS;
                run_pos[r] = -1;
            } else {
                run_pos[r] = -2;
                atomicAdd(&cnt[slot], len);
            }
        }
        if (any_mma) {
            unsigned long long total;
            const int excl = (int)block_scan_excl((unsigned long long)nm, total, sh[2 + ((base >> 10) & 1)]);
            int* mma = segs + lay.mma();
            for (int q = 0; first && q < nm; q++) {
                const int at = n_mma + excl + q;
                if (at >= cap) break;  // tiles that overlap can add up to more rows than the step has: flagged below
                mma[3 * at] = start + q * PLORA_MMA_TOKENS;
                mma[3 * at + 1] = min(PLORA_MMA_TOKENS, len - q * PLORA_MMA_TOKENS);
                mma[3 * at + 2] = slot;
            }
            n_mma += (int)total;
        }
    }
    __syncthreads();

    // slots with gather tokens, ascending; their offsets into perm; work items. One scan of (slots, work items, tokens).
    int n_act, n_gather, n_work;
    {
        const int s = tid;
        const int c = (s >= 1 && s < S1) ? cnt[s] : 0;
        const int flag = c > 0;
        const int nw = (c + PLORA_WORK_TOKENS - 1) / PLORA_WORK_TOKENS;
        unsigned long long total;
        const unsigned long long excl =
            block_scan_excl(((unsigned long long)flag << 53) | ((unsigned long long)nw << 29) | (unsigned long long)c, total, sh[0]);
        const int aidx = (int)(excl >> 53), woff = (int)((excl >> 29) & 0xffffffu), off = (int)(excl & 0x1fffffffu);
        n_act = (int)(total >> 53);
        n_work = (int)((total >> 29) & 0xffffffu);
        n_gather = (int)(total & 0x1fffffffu);
        // Tiles that overlap one another pass the per-tile checks but name more token rows than the step has: the
        // regrouped rows would not fit their region. Such a list is refused as a whole.
        const bool over = n_gather > lay.max_tokens || n_work > cap || n_mma > cap;
        if (over) bad = true;
        if (flag && !over) {
            if (first) {
                segs[lay.act() + aidx] = s;
                segs[lay.seg_off() + aidx] = off;
            }
            seg_base[s] = off;
            int* work = segs + lay.work();
            for (int q = 0; q < nw; q++)
                *reinterpret_cast<int4*>(work + PLORA_WORK_WORDS * (woff + q)) =
                    make_int4(s, off + q * PLORA_WORK_TOKENS, min(PLORA_WORK_TOKENS, c - q * PLORA_WORK_TOKENS), 0);
            cnt[s] = woff;  // from here on: the slot's first work item
        }
        if (first && tid == 0 && !over) segs[lay.seg_off() + n_act] = n_gather;
        if (over) n_act = n_gather = n_work = n_mma = n_runs = 0;
    }

    // stable position of every gather run inside its slot's segment: the weights of the same slot in the lanes below,
    // in the warps below (whist), and in the rounds of 1024 runs before (fill)
    for (int base = 0; base < n_runs; base += 1024) {
        const int r = base + tid;
        int key = 0, w = 0;
        if (r < n_runs && run_pos[r] == -2) {
            key = run_slot[r];
            w = run_tok[r + 1] - run_tok[r];
        }
        if (base > 0) {
            for (int i = tid; i < 32 * S1; i += 1024) whist[i] = 0;
            __syncthreads();
        }
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const unsigned below = peers & ((1u << lane) - 1u);
        int sum = 0;
        if (__all_sync(0xffffffffu, w <= 1)) {
            sum = key != 0 ? __popc(below) : 0;
        } else {
#pragma unroll 8
            for (int j = 0; j < 32; j++) {
                const int wj = __shfl_sync(0xffffffffu, w, j);
                if ((below >> j) & 1u) sum += wj;
            }
        }
        if (key != 0 && (peers >> lane) == 1u) whist[warp * S1 + key] = sum + w;  // the slot's last lane of the warp
        __syncthreads();
        if (key != 0) {
            int pre = 0;
            for (int q = 0; q < warp; q++) pre += whist[q * S1 + key];
            run_pos[r] = seg_base[key] + fill[key] + pre + sum;
        }
        if (base + 1024 < n_runs) {
            __syncthreads();
            for (int s = tid; s < S1; s += 1024) {
                int tot = 0;
                for (int q = 0; q < 32; q++) tot += whist[q * S1 + s];
                fill[s] += tot;
            }
            __syncthreads();
        }
    }

    // perm, and the same token rows inside the work items (each thread reads back the positions it wrote)
    int* perm = segs + lay.perm();
    int* work = segs + lay.work();
    for (int r = tid; r < n_runs; r += 1024) {
        const int pos = run_pos[r];
        if (pos < 0) continue;
        const int start = run_start[r], len = run_tok[r + 1] - run_tok[r], slot = run_slot[r];
        const int rel0 = pos - seg_base[slot], w0 = cnt[slot];
        for (int k = 0; k < len; k++) {
            if (first) perm[pos + k] = start + k;
            const int rel = rel0 + k;
            work[PLORA_WORK_WORDS * (w0 + rel / PLORA_WORK_TOKENS) + 4 + rel % PLORA_WORK_TOKENS] = start + k;
        }
    }
    const int any_bad = __syncthreads_or(bad);
    if (first && tid == 0) {
        if (any_bad) atomicMax(status, PLORA_ERR_ARG);
        segs[SEG_N_ACT] = n_act;
        segs[SEG_N_WORK] = n_work;
        segs[SEG_N_MMA] = n_mma;
        segs[SEG_N_GATHER] = n_gather;
        segs[SEG_N_TILES] = n_tiles;
        segs[SEG_STATUS] = any_bad ? PLORA_ERR_ARG : 0;
    }
    // launch records (the barrier above made the work items, written by other threads of this block, visible)
    if (recs != nullptr) {
        const int nw = min(n_work, rec_cap - 1), end = min(rec_cap, nw + PLORA_REC_TERM);
        for (int site = blockIdx.x; site < n_sites; site += gridDim.x) {
            const int cols = site_cols[3 * site], nsplit = site_cols[3 * site + 1], most = site_cols[3 * site + 2];
            int* ps = prefix + (size_t)site * (size_t)unit_words(rec_cap);
            long long* pe = reinterpret_cast<long long*>(ps + unit_expand(rec_cap));
            unsigned long long before = 0;
            for (int base = 0; base < end; base += 1024) {
                const int w = base + tid;
                unsigned long long units = 0, total = 0;
                if (w < end) {
                    uint4* o = reinterpret_cast<uint4*>(recs + (size_t)site * (size_t)rec_cap + w);
                    if (w >= nw) o[0] = make_uint4(0u, 0u, 0u, (uint32_t)cols);
                    else units = write_record(o, segs, lay, tables + (size_t)site * (size_t)S1, w, cols, nsplit, most);
                }
                if (w == 0) first_item = (int)packed_expand(units);
                const unsigned long long at = before + block_scan_excl(units, total, sh[(base >> 10) & 1]);
                if (w < nw) {
                    ps[1 + w] = packed_shrink(at);
                    pe[2 + w] = packed_expand(at);
                }
                before += total;
            }
            if (tid == 0) {
                ps[0] = nw;
                pe[0] = (long long)share_blocks(packed_expand(before), nw, first_item, expand_grid) << 32 | nw;
                ps[1 + nw] = packed_shrink(before);
                pe[1] = pe[2 + nw] = packed_expand(before);
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The few-token kernels below share a form. Their work is a list of equal units over all work items of the layer, found
// through a prefix count per item that the grouping kernel wrote: a step's slots differ up to 8-fold in rank and its
// layers in width, so a grid of (items x most tiles an item can have) is mostly idle blocks next to a few long ones. Two
// blocks per SM take an equal, contiguous range of units each. In a block, a producer warp walks the units ahead of the
// eight computing warps and keeps a ring of pieces full of slab rows by bulk copies, beginning before the
// dependency wait: 130 to 190 KB in flight per SM, where two steps' worth of operand registers per warp were not enough (25 us for
// 52 MB of A, 80 us for 157 MB of B). The products are tiles of the warp-level tensor instruction (m16n8k16; a 128-row tcgen05
// tile would spend 7/8 or more of its rows on tokens that are not there; on the CUDA cores both kernels were bound by
// instructions). Its 16 input slots may be permuted freely as long as both operands agree, so lane t of four holds inputs
// 8 t .. 8 t + 7 of a row's 32 (two multiplies), and operands move in 16-byte pieces.

// The shrink's unit counts of a layer in shared memory: pre[0] = items, pre[1 + w] = units before item w, pre[1 + items] = all
__device__ __forceinline__ int load_prefix(int* pre, const int* __restrict__ src, int rec_cap) {
    for (int i = threadIdx.x; i < min(rec_cap + 2, (int)blockDim.x); i += blockDim.x) pre[i] = __ldcg(src + i);
    __syncthreads();
    const int n = min(pre[0], rec_cap);
    for (int i = (int)blockDim.x + threadIdx.x; i < n + 2; i += blockDim.x) pre[i] = __ldcg(src + i);
    if (n + 2 > (int)blockDim.x) __syncthreads();
    return pre[1 + n];
}
// The same for the expand, and the block's share [u0, u1) of all units. In shared memory the units before an item are
// counted from u0. False where the block has no share.
__device__ __forceinline__ bool load_share(int* pre, const int* __restrict__ src, int rec_cap, int& share) {
    const long long* pe = reinterpret_cast<const long long*>(src);
    const long long head = __ldcg(pe), total = __ldcg(pe + 1);
    const int n = min((int)(head & 0xffffffff), rec_cap);
    long long mine = 0;  // (fetched beside the counts that say how many there are)
    if ((int)threadIdx.x <= rec_cap) mine = __ldcg(pe + 2 + threadIdx.x);
    const int blocks = min((int)(head >> 32), (int)gridDim.x);
    if ((int)blockIdx.x >= blocks || total == 0) return false;
    const long long u0 = share_at(total, blockIdx.x, blocks);
    share = (int)(share_at(total, blockIdx.x + 1, blocks) - u0);
    if (threadIdx.x == 0) pre[0] = n;
    for (int i = threadIdx.x; i <= n; i += blockDim.x) pre[1 + i] = units_from(i == (int)threadIdx.x ? mine : __ldcg(pe + 2 + i), u0);
    __syncthreads();
    return true;
}
// the item that unit u belongs to
__device__ __forceinline__ int find_item(const int* pre, int u) {
    int lo = 0, hi = pre[0];
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[1 + mid] <= u) lo = mid;
        else hi = mid;
    }
    return lo;
}
// barrier among the eight warps that compute (the producer warp does not take part)
__device__ __forceinline__ void gather_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// The barrier behind a unit's waits. A wait that ran out is one warp's; all eight leave for it, or the others would meet the
// next barrier without it. `gave_up` is only set between a barrier before and this one, and only read behind this one.
__device__ __forceinline__ bool gather_sync_ok(bool ok, int* gave_up) {
    if (!ok) *reinterpret_cast<volatile int*>(gave_up) = 1;
    gather_sync();
    return *reinterpret_cast<volatile int*>(gave_up) == 0;
}
// The producer leaves once the last `stages` of its n copies have landed, whoever still wanted them
__device__ __forceinline__ void ring_landed(uint64_t* full, int n, int stages, int* status) {
    for (int m = n > stages ? n - stages : 0; m < n; m++) mbar_wait_long(&full[m % stages], (uint32_t)(m / stages) & 1u, status);
}

#define GATHER_STAGES 3
#define GATHER_THREADS 288  // eight computing warps and the producer

// Shrink: unit = (item, one of the layer's K-splits, 16 rows of the slot's stacked A), in pieces of 1024 inputs. Every warp
// multiplies the item's tokens (16 rows of the tile) by the 16 rows of A over its 128 inputs of each piece, the
// eight partials are added in warp order in shared memory, and every (token, row, split) is written exactly once.
// Bound by the slabs' bytes (A of every slot present once).
#define SHR_PIECE 1024
#define SHR_PITCH (SHR_PIECE * 2 + 64)  // bytes between rows of a piece: eight lanes' 16-byte reads then meet all banks
#define SHR_STAGE (SHR_ROWS * SHR_PITCH)
__global__ void __launch_bounds__(GATHER_THREADS, 2) plora_shrink_gather_kernel(const bf16* __restrict__ X, int ldx, int K,
                                                                      const PloraRec* __restrict__ recs, int rec_cap,
                                                                      const int* __restrict__ prefix, float* __restrict__ S,
                                                                      size_t s_stride, int lds, int kchunk, int nsplit, int early,
                                                                      int early_x, int late, int* __restrict__ status PLORA_BOUNDS_PARAM) {
    // late != 0: the kernel before is the step's grouping, which writes the records: nothing is read, and no dependent
    // released, before the dependency wait. (The launch itself then overlaps the grouping.)
    // early != 0: dependents are released at kernel start (every store of the path comes after a wait).
    // early_x != 0: the caller vouches that x is older than every kernel still in flight, so x is fetched and
    // the partial sums computed before the dependency wait; only the stores into S (which the expand before may
    // still be reading) come after it.
    extern __shared__ __align__(128) unsigned char gsm[];
    __shared__ __align__(16) PloraRec srec[2];
    __shared__ __align__(8) uint64_t full[GATHER_STAGES], empty[GATHER_STAGES];
    __shared__ int gave_up;
    float* red = reinterpret_cast<float*>(gsm + GATHER_STAGES * SHR_STAGE);  // [8 warps][16][SHR_PAD]
    int* pre = reinterpret_cast<int*>(red + 8 * 16 * SHR_PAD);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    if (early && !late) pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < GATHER_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 8);
        }
        gave_up = 0;
        mbar_fence_init();
    }
    bool waited = false;
    if (late) {
        pdl_wait();
        pdl_trigger();
        waited = true;
    }
    const int total = load_prefix(pre, prefix, rec_cap);  // (its barrier publishes the ring's as well)
    const int u0 = (int)((long long)total * blockIdx.x / gridDim.x), u1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
    if (u0 >= u1) {
        if (!waited) pdl_exit_idle();
        return;
    }
    // a unit's place: its item, its split and first row (units of an item go split by split, so that the rows of A of a split
    // find the tokens' x in L2)
    struct Place {
        int item, k0, split, row0;
    };
    auto place = [&](int u, int item) {
        Place q;
        while (pre[2 + item] <= u) item++;  // (items without units are passed over)
        q.item = item;
        const int n = (pre[2 + item] - pre[1 + item]) / nsplit, local = u - pre[1 + item];
        q.split = local / n;
        q.k0 = q.split * kchunk;
        q.row0 = (local - q.split * n) * SHR_ROWS;
        return q;
    };
    auto fine = [&](const PloraRec& rec, const Place& q) {
#ifdef PLORA_BOUNDS
        return rec_in_bounds(rec, bnd, K) && q.row0 + SHR_ROWS <= rec.rank;
#else
        (void)rec, (void)q;
        return true;
#endif
    };
    int item = find_item(pre, u0);
    if (warp == 8) {
        int stg = 0, n = 0;
        uint32_t par = 1;
        bool ok = true;
        for (int u = u0; ok && u < u1; u++) {
            const Place q = place(u, item);
            item = q.item;
            if (!fine(recs[q.item], q)) continue;
            const bf16* A = reinterpret_cast<const bf16*>(__ldcg(&recs[q.item].a)) + (size_t)(q.row0 + (lane & 15)) * K;
            const int kend = min(K, q.k0 + kchunk);
            for (int k = q.k0; k < kend; k += SHR_PIECE, n++) {
                if (n >= GATHER_STAGES) ok = mbar_wait_long(&empty[stg], par, status);
                if (!ok) break;
                const uint32_t bytes = (uint32_t)min(SHR_PIECE, kend - k) * 2u;
                if (lane == 0) mbar_expect_tx(&full[stg], bytes * SHR_ROWS);
                __syncwarp();
                if (lane < SHR_ROWS) bulk_g2s(gsm + (size_t)stg * SHR_STAGE + (size_t)lane * SHR_PITCH, A + k, bytes, &full[stg]);
                if (++stg == GATHER_STAGES) {
                    stg = 0;
                    par ^= 1;
                }
            }
        }
        ring_landed(full, n, GATHER_STAGES, status);
        if (!waited) pdl_wait();
        return;
    }
    // ---- computing warps
    auto fetch = [&](int w, int at) {
        if (tid < 12) reinterpret_cast<uint4*>(&srec[at])[tid] = __ldcg(reinterpret_cast<const uint4*>(recs + w) + tid);
    };
    const bf16 *x0 = nullptr, *x1 = nullptr;
    bool two = false;
    uint4 xv[4][2];
    auto aim = [&](const PloraRec& rec) {
        x0 = X + (size_t)rec.tok[g < rec.cnt ? g : 0] * ldx + warp * 128 + 8 * t4;
        x1 = X + (size_t)rec.tok[g + 8 < rec.cnt ? g + 8 : 0] * ldx + warp * 128 + 8 * t4;
        two = rec.cnt > 8;  // (else rows 8 to 15 of the tile hold zeros, and their results are dropped)
    };
    auto load_x = [&](int k, int kend) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const bool in = k + warp * 128 + 32 * q + 8 * t4 < kend;
            xv[q][0] = in ? __ldcg(reinterpret_cast<const uint4*>(x0 + k + 32 * q)) : make_uint4(0u, 0u, 0u, 0u);
            xv[q][1] = in && two ? __ldcg(reinterpret_cast<const uint4*>(x1 + k + 32 * q)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    Place here = place(u0, item);
    fetch(here.item, 0);
    gather_sync();
    bool good = fine(srec[0], here);
    if (!good && tid == 0) atomicMax(status, PLORA_ERR_ARG);
    aim(srec[0]);
    if (!early_x && !waited) {
        pdl_wait();
        if (!early) pdl_trigger();
        waited = true;
    }
    if (good) load_x(here.k0, min(K, here.k0 + kchunk));
    int stg = 0;
    uint32_t par = 0;
    bool ok = true;
    for (int u = u0, at = 0; ok && u < u1; u++, at ^= 1) {
        Place next = here;
        if (u + 1 < u1) {
            next = place(u + 1, here.item);
            fetch(next.item, at ^ 1);
        }
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        const int kend = min(K, here.k0 + kchunk);
#pragma unroll 1
        for (int k = here.k0; good && k < kend; k += SHR_PIECE) {
            ok = mbar_wait_long(&full[stg], par, status);
            if (!ok) break;
            const uint32_t a = smem_u32(gsm) + (uint32_t)stg * SHR_STAGE + (uint32_t)g * SHR_PITCH + (uint32_t)(warp * 256 + 16 * t4);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (k + warp * 128 + 32 * q < kend) {
                    const uint4 &x = xv[q][0], &z = xv[q][1];
                    const uint32_t f0[4] = {x.x, z.x, x.y, z.y}, f1[4] = {x.z, z.z, x.w, z.w};
                    const bool in = k + warp * 128 + 32 * q + 8 * t4 < kend;
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        uint4 b = make_uint4(0u, 0u, 0u, 0u);
                        if (in) b = lds128(a + (uint32_t)(8 * i) * SHR_PITCH + 64u * q);
                        mma_16816(acc[i], f0, b.x, b.y);
                        mma_16816(acc[i], f1, b.z, b.w);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[stg]);
            if (++stg == GATHER_STAGES) {
                stg = 0;
                par ^= 1;
            }
            if (k + SHR_PIECE < kend) load_x(k + SHR_PIECE, kend);
        }
        float* mine = red + (size_t)warp * 16 * SHR_PAD + g * SHR_PAD + 2 * t4;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            *reinterpret_cast<float2*>(mine + 8 * i) = make_float2(acc[i][0], acc[i][1]);
            if (two) *reinterpret_cast<float2*>(mine + 8 * SHR_PAD + 8 * i) = make_float2(acc[i][2], acc[i][3]);
        }
        ok = gather_sync_ok(ok, &gave_up);  // the partials and the next record are there
        const bool was = good && ok;
        if (u + 1 < u1) {
            good = fine(srec[at ^ 1], next);
            if (!good && tid == 0) atomicMax(status, PLORA_ERR_ARG);
            aim(srec[at ^ 1]);
            if (good && (waited || early_x)) load_x(next.k0, min(K, next.k0 + kchunk));
        }
        if (!waited) {
            pdl_wait();
            if (!early) pdl_trigger();
            waited = true;
        }
        const int t = tid >> 4, c = tid & 15;
        if (was && t < srec[at].cnt) {
            float sum = red[t * SHR_PAD + c];
#pragma unroll
            for (int q = 1; q < 8; q++) sum += red[q * 16 * SHR_PAD + t * SHR_PAD + c];
            S[(size_t)here.split * s_stride + (size_t)srec[at].tok[t] * lds + here.row0 + c] = sum;
        }
        here = next;
        gather_sync();  // shared memory is reused by the next unit
    }
    if (!waited) pdl_wait();
}

// Expand: the units are what the columns cost, so that a block's range is a few stretches of columns of one part for one
// item's tokens, as long as any other block's. The producer copies their rows of B (contiguous) and hints the lines of y that go with
// them to L2. At the start of a stretch the computing warps put the item's S rows (K-split partials, added in split order)
// into shared memory as three bf16 terms (high, middle, low part, whose products with bf16 B are exact in f32, so no
// precision is given up against an f32 multiply-add chain); then each takes its groups of columns of every piece. An item's
// tokens are taken 8 at a time, whatever their number, so that a token's result does not depend on the others: rows 0-7 of
// the token tile carry one term of S and rows 8-15 another, two multiplies per 8 x 16 ranks ([low | zero], then
// [high | middle]), and a lane adds its two rows. The rows of B go to the tiles of a group in an order that leaves every
// lane with 8 adjacent columns of its token: y moves in pieces of 16 bytes.
// Bound by the bytes of B and y.
#define EXP_PIECE 16384
#define EXP_STAGES 5
#define EXP_AHEAD 2     // groups of columns whose y a warp has on its way
#define EXP_Y_BYTES 1024 // ... each: two pieces of 16 bytes per lane (16 tokens of bf16, or 8 of f32)
struct ExpandUnit {
    int r, r_off;          // rank, first column of S
    int c0, c1;            // the stretch of the part's columns
    size_t ybase;          // column of y where the part starts
};
__device__ __forceinline__ int expand_piece_cols(int r) { return r <= 16 ? 512 : r <= 32 ? 256 : r <= 64 ? 128 : 64; }

// 8 tokens' three terms of S over 32 ranks (16 where NARROW), as this lane's operands of a step
template <bool NARROW>
struct SFrag {
    uint32_t h[NARROW ? 2 : 4], m[NARROW ? 2 : 4], l[NARROW ? 2 : 4];
    __device__ __forceinline__ void load(uint32_t sp, uint32_t plane, int k, int t4) {  // (row g of the planes at `sp`, from rank k)
        if (NARROW) {
            const uint2 a = lds64(sp + 8u * t4), b = lds64(sp + plane + 8u * t4), c = lds64(sp + 2 * plane + 8u * t4);
            h[0] = a.x, h[1] = a.y, m[0] = b.x, m[1] = b.y, l[0] = c.x, l[1] = c.y;
        } else {
            constexpr int Z = NARROW ? 0 : 2, W = NARROW ? 1 : 3;
            const uint32_t o = sp + 2u * k + 16u * t4;
            const uint4 a = lds128(o), b = lds128(o + plane), c = lds128(o + 2 * plane);
            h[0] = a.x, h[1] = a.y, h[Z] = a.z, h[W] = a.w;
            m[0] = b.x, m[1] = b.y, m[Z] = b.z, m[W] = b.w;
            l[0] = c.x, l[1] = c.y, l[Z] = c.z, l[W] = c.w;
        }
    }
};

// The products with one group of NT tiles of 8 columns over the same ranks: `col` = this lane's row of B in every tile. Loads
// first, then one term after another over all tiles: a tile's products depend on one another.
template <int NT, bool NARROW>
__device__ __forceinline__ void expand_step(float (&d)[NT][4], const SFrag<NARROW>& s, const uint32_t (&col)[NT], int k, int r, int t4) {
    const uint32_t al[4] = {s.l[0], 0u, s.l[1], 0u}, ah[4] = {s.h[0], s.m[0], s.h[1], s.m[1]};
    if (NARROW) {
        uint2 b[NT];
#pragma unroll
        for (int i = 0; i < NT; i++) b[i] = lds64(col[i] + 8u * t4);
#pragma unroll
        for (int i = 0; i < NT; i++) mma_16816(d[i], al, b[i].x, b[i].y);
#pragma unroll
        for (int i = 0; i < NT; i++) mma_16816(d[i], ah, b[i].x, b[i].y);
    } else {
        constexpr int Z = NARROW ? 0 : 2, W = NARROW ? 1 : 3;
        const bool in = k + 8 * t4 < r;  // (the second half of the last 32 ranks may lie outside)
        uint4 b[NT];
#pragma unroll
        for (int i = 0; i < NT; i++) {
            b[i] = make_uint4(0u, 0u, 0u, 0u);
            if (in) b[i] = lds128(col[i] + 2u * k + 16u * t4);
        }
        const uint32_t bl[4] = {s.l[Z], 0u, s.l[W], 0u}, bh[4] = {s.h[Z], s.m[Z], s.h[W], s.m[W]};
#pragma unroll
        for (int i = 0; i < NT; i++) mma_16816(d[i], al, b[i].x, b[i].y);
#pragma unroll
        for (int i = 0; i < NT; i++) mma_16816(d[i], bl, b[i].z, b[i].w);
#pragma unroll
        for (int i = 0; i < NT; i++) mma_16816(d[i], ah, b[i].x, b[i].y);
#pragma unroll
        for (int i = 0; i < NT; i++) mma_16816(d[i], bh, b[i].z, b[i].w);
    }
}

// A lane's 2 NT adjacent columns of one token of y, in one or two pieces where the row allows it
template <bool F32, int NT>
struct YPiece {
    uint32_t w[F32 ? 2 * NT : NT];
};
template <bool F32, int NT>
__device__ __forceinline__ void y_load(YPiece<F32, NT>& q, const unsigned char* y, int cols, bool wide) {
    constexpr int NW = F32 ? 2 * NT : NT;  // words
    if (cols <= 0) return;
    if (wide && cols >= 2 * NT) {
        if (NW == 2) {
            const uint2 v = __ldcg(reinterpret_cast<const uint2*>(y));
            q.w[0] = v.x, q.w[1] = v.y;
        } else {
#pragma unroll
            for (int i = 0; i < NW / 4; i++) {
                const uint4 v = __ldcg(reinterpret_cast<const uint4*>(y) + i);
                q.w[(4 * i) % NW] = v.x, q.w[(4 * i + 1) % NW] = v.y, q.w[(4 * i + 2) % NW] = v.z, q.w[(4 * i + 3) % NW] = v.w;
            }
        }
    } else {
#pragma unroll
        for (int c = 0; c < NW; c++)  // (widths, offsets and pitches are even)
            if (c * (F32 ? 1 : 2) < cols) q.w[c] = __ldcg(reinterpret_cast<const uint32_t*>(y) + c);
    }
}
template <bool F32, int NT>
__device__ __forceinline__ void y_store(const YPiece<F32, NT>& q, const float (&d)[NT][4], unsigned char* y, int cols, bool wide) {
    constexpr int NW = F32 ? 2 * NT : NT;
    if (cols <= 0) return;
    uint32_t o[NW];
#pragma unroll
    for (int i = 0; i < NT; i++) {
        const float a = d[i][0] + d[i][2], b = d[i][1] + d[i][3];
        if (F32) {
            o[(2 * i) % NW] = __float_as_uint(__uint_as_float(q.w[(2 * i) % NW]) + a);
            o[(2 * i + 1) % NW] = __float_as_uint(__uint_as_float(q.w[(2 * i + 1) % NW]) + b);
        } else {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.w[i]));
            const __nv_bfloat162 s = __floats2bfloat162_rn(f.x + a, f.y + b);
            o[i] = *reinterpret_cast<const uint32_t*>(&s);
        }
    }
    if (wide && cols >= 2 * NT) {
        if (NW == 2) {
            *reinterpret_cast<uint2*>(y) = make_uint2(o[0], o[1]);
        } else {
#pragma unroll
            for (int i = 0; i < NW / 4; i++)
                reinterpret_cast<uint4*>(y)[i] = make_uint4(o[(4 * i) % NW], o[(4 * i + 1) % NW], o[(4 * i + 2) % NW], o[(4 * i + 3) % NW]);
        }
    } else {
#pragma unroll
        for (int c = 0; c < NW; c++)
            if (c * (F32 ? 1 : 2) < cols) reinterpret_cast<uint32_t*>(y)[c] = o[c];
    }
}

// What a stretch needs besides its B: S of the item as planes in shared memory, and y
struct ExpandStep {
    const float* S;
    size_t s_stride;
    int lds, nsplit;
    unsigned char* planes;  // three bf16 planes [16 tokens][s_pad bytes]
    uint32_t s_pad;
    unsigned char* Y;
    int ldy;
};

// One stretch by one warp: every eighth group of 32 columns, wherever the pieces of B end. Full groups of rows that move in
// 16-byte pieces find their y in shared memory, where each lane has asked for its own pieces EXP_AHEAD groups before (in
// registers, one group ahead was all that fitted, and the round trips to L2 were a third of the time). Up to 8 tokens
// keep their operands of S in registers (KEEP steps of 32 ranks, as many as there is room for); the rest reads them again
// for every group. `at` = the ring's stage and, from bit 8 on, the parity of its barriers; returns where the ring then
// stands, or -1 when a wait ran out. (Not inlined: eight of these share a kernel, and each has its own use for 96 registers.)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
template <bool NARROW, int KEEP, bool TWO, bool F32>
__device__ __noinline__ int expand_stretch(unsigned char* pieces, uint64_t* full, uint64_t* empty, int at, ExpandUnit un, ExpandStep st,
                                           const PloraRec& rec, int* status) {
    constexpr int NT = 4, ES = F32 ? 4 : 2, GC = 8 * NT, H = TWO ? 2 : 1, NW = F32 ? 2 * NT : NT, STEP = 8 * GC;
    constexpr bool RING = !(TWO && F32);  // (16 tokens of f32 would take twice the space)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    int stg = at & 0xff;
    uint32_t par = (uint32_t)at >> 8;
    const bool wide = ((reinterpret_cast<uintptr_t>(st.Y) | ((size_t)st.ldy * ES) | (un.ybase * ES)) & 15) == 0;
    const int cnt = rec.cnt, pc = expand_piece_cols(un.r);
    const uint32_t plane = 16u * st.s_pad, planes = smem_u32(st.planes);
    unsigned char* yrow[H];
    uint32_t sp[H];
#pragma unroll
    for (int h = 0; h < H; h++) {
        const int t = min(8 * h + g, cnt - 1);
        yrow[h] = st.Y + ((size_t)rec.tok[t] * st.ldy + un.ybase) * ES;
        sp[h] = planes + (uint32_t)t * st.s_pad;
    }
    constexpr int NK = TWO || KEEP == 0 ? 1 : KEEP;
    SFrag<NARROW> keep[NK];
    if (!TWO && KEEP > 0)
#pragma unroll
        for (int q = 0; q < NK; q++)
            if (32 * q < un.r) keep[q].load(sp[0], plane, 32 * q, t4);
    int p0 = un.c0;        // first column of the ring's current piece
    bool landed = false;   // ... which this warp has waited for
    auto wait = [&]() {
        if (!landed) landed = mbar_wait_long(&full[stg], par, status);
        return landed;
    };
    auto release = [&]() {  // this warp is through with the current piece
        if (!wait()) return false;
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stg]);
        if (++stg == EXP_STAGES) {
            stg = 0;
            par ^= 1;
        }
        p0 += pc;
        landed = false;
        return true;
    };
    const uint32_t r2 = 2u * (uint32_t)un.r, brow = (uint32_t)(2 * NT * (g >> 1) + (g & 1)) * r2;
    const uint32_t ybuf = planes + 3 * plane + (uint32_t)(warp * EXP_AHEAD * EXP_Y_BYTES + lane * 16);
#pragma unroll
    for (int h = 0; h < H; h++) yrow[h] += (un.c0 + warp * GC + 2 * NT * t4) * ES;  // this lane's columns of the warp's first group
    const int full_end = RING && wide ? un.c1 - GC : un.c0 - 1;  // groups that start up to here go through shared memory
    auto ask = [&](int c, int slot, int ahead) {
        if (c <= full_end) {
#pragma unroll
            for (int h = 0; h < H; h++)
                if (8 * h + g < cnt)
#pragma unroll
                    for (int i = 0; i < NW / 4; i++)
                        cp_async16(ybuf + (uint32_t)(slot * EXP_Y_BYTES + (h * (NW / 4) + i) * 512), yrow[h] + (size_t)ahead * ES + 16 * i);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int q = 0; q < EXP_AHEAD; q++) ask(un.c0 + warp * GC + q * STEP, q, q * STEP);
    int slot = 0;
#pragma unroll 1
    for (int c = un.c0 + warp * GC; c < un.c1; c += STEP) {
        while (c >= p0 + pc)
            if (!release()) return -1;
        if (!wait()) return -1;
        // (rows past the last column are whatever the stage holds: their products are dropped)
        const uint32_t rows = smem_u32(pieces) + (uint32_t)stg * EXP_PIECE + (uint32_t)(c - p0) * r2 + brow;
        const uint32_t col[NT] = {rows, rows + 2 * r2, rows + 4 * r2, rows + 6 * r2};
        const int left = un.c1 - c - 2 * NT * t4;  // this lane's columns and those after them
        const bool ringed = c <= full_end;
        cp_async_wait<EXP_AHEAD - 1>();
#pragma unroll
        for (int h = 0; h < H; h++) {
            const bool live = 8 * h + g < cnt;
            YPiece<F32, NT> y;
            if (!ringed) y_load<F32, NT>(y, yrow[h], live ? left : 0, wide);
            float d[NT][4];
#pragma unroll
            for (int i = 0; i < NT; i++) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.f;
            if (TWO || KEEP == 0) {
#pragma unroll 1
                for (int k = 0; k < un.r; k += 32) {
                    SFrag<NARROW> f;
                    f.load(sp[h], plane, k, t4);
                    expand_step<NT, NARROW>(d, f, col, k, un.r, t4);
                }
            } else {
#pragma unroll
                for (int k = 0; k < NK; k++)
                    if (32 * k < un.r) expand_step<NT, NARROW>(d, keep[k], col, 32 * k, un.r, t4);
            }
            if (ringed) {
                if (live) {
#pragma unroll
                    for (int i = 0; i < NW / 4; i++) {
                        const uint4 z = lds128(ybuf + (uint32_t)(slot * EXP_Y_BYTES + (h * (NW / 4) + i) * 512));
                        y.w[4 * i] = z.x, y.w[4 * i + 1] = z.y, y.w[4 * i + 2] = z.z, y.w[4 * i + 3] = z.w;
                    }
                    y_store<F32, NT>(y, d, yrow[h], 2 * NT, true);
                }
            } else {
                y_store<F32, NT>(y, d, yrow[h], live ? left : 0, wide);
            }
        }
        ask(c + EXP_AHEAD * STEP, slot, EXP_AHEAD * STEP);
        slot = slot + 1 == EXP_AHEAD ? 0 : slot + 1;
#pragma unroll
        for (int h = 0; h < H; h++) yrow[h] += STEP * ES;
    }
    while (p0 < un.c1)
        if (!release()) return -1;
    return stg | (int)(par << 8);
}

// The same for ranks above 128, which no piece holds: the rows of B from global memory, 32 ranks at a time, four such loads
// of a row on their way together. (With one, each waited for L2 or memory by itself: a layer block at rank 256, 16 tokens of
// 16 adapters 389 -> 219 us, 2,000 tokens 2900 -> 1950; the CUDA-core kernel before took 291 and 12,200.)
template <bool F32>
__device__ __noinline__ void expand_wide_rank(const bf16* B, ExpandUnit un, ExpandStep st, const PloraRec& rec, int warp, int g, int t4) {
    constexpr int ES = F32 ? 4 : 2, NT = 2, AHEAD = 4;
    const bool wide = ((reinterpret_cast<uintptr_t>(st.Y) | ((size_t)st.ldy * ES) | (un.ybase * ES)) & 15) == 0;
    const uint32_t plane = 16u * st.s_pad;
#pragma unroll 1
    for (int t0 = 0; t0 < rec.cnt; t0 += 8) {
        const int t = min(t0 + g, rec.cnt - 1);
        unsigned char* yrow = st.Y + ((size_t)rec.tok[t] * st.ldy + un.ybase) * ES;
        const uint32_t sp = smem_u32(st.planes) + (uint32_t)t * st.s_pad;
#pragma unroll 1
        for (int c = un.c0 + warp * 8 * NT; c < un.c1; c += 64 * NT) {
            const int mine = c + 2 * NT * t4, cols = t0 + g < rec.cnt ? un.c1 - mine : 0;
            YPiece<F32, NT> y;
            y_load<F32, NT>(y, yrow + (size_t)mine * ES, cols, wide);
            float d[NT][4];
#pragma unroll
            for (int i = 0; i < NT; i++) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.f;
            const bf16* row[NT];
#pragma unroll
            for (int i = 0; i < NT; i++) row[i] = B + (size_t)min(c + 2 * NT * (g >> 1) + 2 * i + (g & 1), un.c1 - 1) * un.r + 8 * t4;
#pragma unroll 1
            for (int k0 = 0; k0 < un.r; k0 += 32 * AHEAD) {
                uint4 b[AHEAD][NT];
#pragma unroll
                for (int q = 0; q < AHEAD; q++)
#pragma unroll
                    for (int i = 0; i < NT; i++) {
                        b[q][i] = make_uint4(0u, 0u, 0u, 0u);
                        if (k0 + 32 * q + 8 * t4 < un.r) b[q][i] = __ldg(reinterpret_cast<const uint4*>(row[i] + k0 + 32 * q));
                    }
#pragma unroll
                for (int q = 0; q < AHEAD; q++) {
                    const int k = k0 + 32 * q;
                    if (k >= un.r) break;
                    const uint32_t o = 2u * k + 16u * t4;
                    const uint4 h = lds128(sp + o), m = lds128(sp + plane + o), l = lds128(sp + 2 * plane + o);
                    const uint32_t al0[4] = {l.x, 0u, l.y, 0u}, ah0[4] = {h.x, m.x, h.y, m.y}, al1[4] = {l.z, 0u, l.w, 0u}, ah1[4] = {h.z, m.z, h.w, m.w};
#pragma unroll
                    for (int i = 0; i < NT; i++) {
                        mma_16816(d[i], al0, b[q][i].x, b[q][i].y);
                        mma_16816(d[i], ah0, b[q][i].x, b[q][i].y);
                        mma_16816(d[i], al1, b[q][i].z, b[q][i].w);
                        mma_16816(d[i], ah1, b[q][i].z, b[q][i].w);
                    }
                }
            }
            y_store<F32, NT>(y, d, yrow + (size_t)mine * ES, cols, wide);
        }
    }
}

// The bf16 high part of a sum, and what the lower parts are to hold. A sum whose nearest bf16 would be infinite is rounded
// towards zero; of an infinite one nothing is left (infinity less itself would be no number).
__device__ __forceinline__ float high_part(float f) {
    const float h = __bfloat162float(__float2bfloat16_rn(f));
    return isinf(h) ? __uint_as_float(__float_as_uint(f) & 0xffff0000u) : h;
}
__device__ __forceinline__ float rest_of(float f, float h) { return isinf(h) ? 0.f : f - h; }

// S of an item's part, four values a thread and step: all planes on their way together, added in split order; the bf16
// planes are filled up with zeros to a multiple of 32 ranks
__device__ __forceinline__ void expand_stage_s(const ExpandUnit& un, const ExpandStep& st, const PloraRec& rec, int tid) {
    const uint32_t plane = 16u * st.s_pad;
    const int r4 = ((un.r + 31) & ~31) >> 2;
    for (int i = tid; i < rec.cnt * r4; i += 256) {
        const int t = i / r4, j = (i - t * r4) * 4;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < un.r) {
            const float* sp = st.S + (size_t)rec.tok[t] * st.lds + un.r_off + j;
            for (int s0 = 0; s0 < st.nsplit; s0 += 4) {
                float4 v[4];
#pragma unroll
                for (int s = 0; s < 4; s++)
                    v[s] = s0 + s < st.nsplit ? __ldcg(reinterpret_cast<const float4*>(sp + (size_t)(s0 + s) * st.s_stride)) : a;
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    if (s0 + s == 0) a = v[0];
                    else if (s0 + s < st.nsplit) a.x += v[s].x, a.y += v[s].y, a.z += v[s].z, a.w += v[s].w;
                }
            }
        }
        const float f[4] = {a.x, a.y, a.z, a.w};
        uint32_t w[3][2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float2 hf = make_float2(high_part(f[2 * e]), high_part(f[2 * e + 1]));
            const __nv_bfloat162 h = __floats2bfloat162_rn(hf.x, hf.y);
            const float m0 = rest_of(f[2 * e], hf.x), m1 = rest_of(f[2 * e + 1], hf.y);
            const __nv_bfloat162 m = __floats2bfloat162_rn(m0, m1);
            const float2 mf = __bfloat1622float2(m);
            const __nv_bfloat162 l = __floats2bfloat162_rn(m0 - mf.x, m1 - mf.y);
            w[0][e] = *reinterpret_cast<const uint32_t*>(&h);
            w[1][e] = *reinterpret_cast<const uint32_t*>(&m);
            w[2][e] = *reinterpret_cast<const uint32_t*>(&l);
        }
#pragma unroll
        for (int q = 0; q < 3; q++) *reinterpret_cast<uint2*>(st.planes + q * plane + (size_t)t * st.s_pad + j * 2) = make_uint2(w[q][0], w[q][1]);
    }
}

// WIDE: for registries whose adapters may have ranks above 128 (the call takes registers that the other form has better uses for)
template <bool F32, bool WIDE>
__global__ void __launch_bounds__(GATHER_THREADS, 2) plora_expand_gather_kernel(const float* __restrict__ S, size_t s_stride, int lds, int nsplit,
                                                                      const PloraRec* __restrict__ recs, int rec_cap,
                                                                      const int* __restrict__ prefix, void* Y, int ldy, int s_pad,
                                                                      int most, int early, int* __restrict__ status PLORA_BOUNDS_PARAM) {
    // early != 0: dependents are released at kernel start. No value of y is bound before the dependency wait
    // (the kernel before, the layer's matrix multiply, may still be writing it): only L2 prefetch hints.
    extern __shared__ __align__(128) unsigned char gsm[];
    __shared__ __align__(16) PloraRec srec;
    __shared__ __align__(8) uint64_t full[EXP_STAGES], empty[EXP_STAGES];
    __shared__ int gave_up;
    unsigned char* planes = gsm + EXP_STAGES * EXP_PIECE;
    int* pre = reinterpret_cast<int*>(planes + 3 * 16 * (size_t)s_pad + 8 * EXP_AHEAD * EXP_Y_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    constexpr int ES = F32 ? 4 : 2;
    if (early) pdl_trigger();
    if (tid == 0) {
        for (int i = 0; i < EXP_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 8);
        }
        gave_up = 0;
        mbar_fence_init();
    }
    int u1;  // the block's share is the units 0 .. u1
    if (!load_share(pre, prefix, rec_cap, u1)) return pdl_exit_idle();  // (its barrier publishes the ring's as well)
    const int w0 = find_item(pre, 0);
    if (warp == 8) {
        // ---- copies of B, and hints for y
        int stg = 0, n = 0;
        uint32_t par = 1;
        bool ok = true;
        for (int u = 0, w = w0; ok && u < u1;) {
            while (pre[2 + w] <= u) w++;  // (items without units are passed over)
            const PloraRec& rec = recs[w];
            int r[PLORA_MAX_PARTS], rows[PLORA_MAX_PARTS], part, c0, c1;
            const int cnt = __ldcg(&rec.cnt), tok = lane < PLORA_WORK_TOKENS ? __ldcg(&rec.tok[lane]) : 0;
#pragma unroll
            for (int p = 0; p < PLORA_MAX_PARTS; p++) r[p] = __ldcg(&rec.r[p]), rows[p] = __ldcg(&rec.rows[p]);
#ifdef PLORA_BOUNDS
            if (!rec_in_bounds(rec, bnd, rec.cols)) {
                u = pre[2 + w];
                continue;
            }
#endif
            u += expand_stretch_at(r, rows, cnt, most, u - pre[1 + w], u1 - u, part, c0, c1);
            const int rp = __ldcg(&rec.r[part]);
            if (c0 >= c1 || (WIDE && rp > 128)) continue;  // (ranks above 128 are read from global memory)
            const bf16* B = reinterpret_cast<const bf16*>(__ldcg(&rec.b[part]));
            const size_t off = (size_t)__ldcg(&rec.off[part]);
            const int pc = expand_piece_cols(rp);
            for (int p0 = c0; p0 < c1; p0 += pc, n++) {
                const int p1 = min(c1, p0 + pc);
                if (n >= EXP_STAGES) ok = mbar_wait_long(&empty[stg], par, status);
                if (!ok) break;
                if (lane == 0) {
                    const uint32_t bytes = (uint32_t)(p1 - p0) * (uint32_t)rp * 2u;
                    mbar_expect_tx(&full[stg], bytes);
                    bulk_g2s(gsm + (size_t)stg * EXP_PIECE, B + (size_t)p0 * rp, bytes, &full[stg]);
                }
                if (++stg == EXP_STAGES) {
                    stg = 0;
                    par ^= 1;
                }
                const size_t len = (size_t)(p1 - p0) * ES;
                const int lines = (int)((len + 127) / 128) + 1;
                for (int i = lane; i < ((cnt * lines + 31) & ~31); i += 32) {
                    const int t = i / lines, l = i - t * lines;
                    const int tk = __shfl_sync(0xffffffffu, tok, t & 15);
                    const size_t start = ((size_t)tk * ldy + off + p0) * ES, at = (start & ~(size_t)127) + (size_t)l * 128;
                    if (t < cnt && at < start + len) prefetch_l2(reinterpret_cast<const unsigned char*>(Y) + at);
                }
            }
        }
        ring_landed(full, n, EXP_STAGES, status);
        pdl_wait();
        return;
    }
    const ExpandStep st = {S, s_stride, lds, nsplit, planes, (uint32_t)s_pad, reinterpret_cast<unsigned char*>(Y), ldy};
    bool waited = false, ok = true;
    int at = 0;  // the ring's position, see expand_stretch
    for (int u = 0, w = w0; ok && u < u1;) {
        while (pre[2 + w] <= u) w++;
        if (tid < 12) reinterpret_cast<uint4*>(&srec)[tid] = __ldcg(reinterpret_cast<const uint4*>(recs + w) + tid);
        gather_sync();
        if (!waited) {
            pdl_wait();
            if (!early) pdl_trigger();
            waited = true;
        }
#ifdef PLORA_BOUNDS
        if (!rec_in_bounds(srec, bnd, srec.cols)) {
            if (tid == 0) atomicMax(status, PLORA_ERR_ARG);
            u = pre[2 + w];
            gather_sync();
            continue;
        }
#endif
        ExpandUnit un;
        int part;
        u += expand_stretch_at(srec.r, srec.rows, srec.cnt, most, u - pre[1 + w], u1 - u, part, un.c0, un.c1);
        if (un.c0 < un.c1) {
            un.r = srec.r[part], un.r_off = srec.r_off[part];
            un.ybase = (size_t)srec.off[part];
            expand_stage_s(un, st, srec, tid);
            gather_sync();
            if (WIDE && un.r > 128) {
                expand_wide_rank<F32>(reinterpret_cast<const bf16*>(srec.b[part]), un, st, srec, warp, g, t4);
            } else {
#define PLORA_STRETCH(NARROW, KEEP)                                                                                     \
    at = srec.cnt > 8 ? expand_stretch<NARROW, KEEP, true, F32>(gsm, full, empty, at, un, st, srec, status)              \
                      : expand_stretch<NARROW, KEEP, false, F32>(gsm, full, empty, at, un, st, srec, status)
                if (un.r <= 16) PLORA_STRETCH(true, 1);
                else if (un.r <= 32) PLORA_STRETCH(false, 1);
                else if (un.r <= 64) PLORA_STRETCH(false, 2);
                else PLORA_STRETCH(false, 0);
#undef PLORA_STRETCH
                ok = at >= 0;
            }
        }
        ok = gather_sync_ok(ok, &gave_up);  // S and the record are replaced for the next stretch
    }
    if (!waited) pdl_wait();
}

}  // namespace

// ---------------------------------------------------------------------------------------------

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

cudaError_t plora_launch_meta_tiles(const int32_t* cu, const int32_t* seq_slot, int n_seqs, int32_t* tiles,
                                    int cap_tiles, int* status, cudaStream_t st) {
    plora_meta_tiles_kernel<<<1, 1024, 0, st>>>(cu, seq_slot, n_seqs, tiles, cap_tiles, status);
    return cudaGetLastError();
}

size_t plora_meta_group_smem(const SegLayout& lay) {
    return (size_t)(4 * lay.cap_tiles + 1 + 3 * (lay.max_slots + 1) + 32 * (lay.max_slots + 1)) * sizeof(int);
}

// One-time function attributes (dynamic shared memory above 48 KB). Called from plora_create, never from
// the launch path, so launches stay legal inside a stream capture.
static int g_sms = 148;  // SMs of the device the kernels were set up for

cudaError_t plora_kernels_init() {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    // (the limit belongs to the kernel, not to a handle: the most that any handle may need)
    cudaError_t e = cudaFuncSetAttribute(plora_meta_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PLORA_GROUP_SMEM_MAX);
    if (e != cudaSuccess) return e;
    // The few-token kernels overlap with their neighbours in the stream (programmatic dependent launch), and an SM's
    // split between L1 and shared memory is fixed while any block runs on it: all of them ask for the largest
    // split, so that a block of the next kernel finds room beside the blocks of this one.
    const void* fns[5] = {reinterpret_cast<const void*>(plora_shrink_gather_kernel),
                          reinterpret_cast<const void*>(plora_expand_gather_kernel<false, false>), reinterpret_cast<const void*>(plora_expand_gather_kernel<true, false>),
                          reinterpret_cast<const void*>(plora_expand_gather_kernel<false, true>), reinterpret_cast<const void*>(plora_expand_gather_kernel<true, true>)};
    for (int i = 0; i < 5 && e == cudaSuccess; i++) e = plora_kernel_shared(fns[i], 220 * 1024);
    return e;
}

cudaError_t plora_launch_meta_group(const int32_t* tiles, int32_t* segs, SegLayout lay, int* status, const plora_desc* tables,
                                    const int32_t* site_cols, int n_sites, PloraRec* recs, int rec_cap, int* prefix, bool pdl,
                                    cudaStream_t st) {
    // a block per layer, up to 64: past that a block has more than one layer's records to write, and every further
    // block repeats the grouping
    const int blocks = recs == nullptr ? 1 : n_sites < 64 ? n_sites : 64;
    return launch_pdl(plora_meta_group_kernel, dim3((unsigned)blocks), dim3(1024), plora_meta_group_smem(lay), st, pdl, tiles, segs, lay,
                      status, tables, site_cols, n_sites, recs, rec_cap, prefix, 2 * g_sms);
}

// Two blocks per SM walk the units; `bound` is the most units a step of this size can have
static unsigned unit_grid(long long bound) { return (unsigned)(bound < 2 * g_sms ? bound : 2 * g_sms); }

cudaError_t plora_launch_shrink(const void* x, int ldx, int K, const PloraRec* recs, int rec_cap, const int* prefix, float* S,
                                size_t s_stride_elems, int lds, int kchunk, int nsplit, int work_cap, int max_rank_total,
                                const PloraBounds& bnd, int* status, bool pdl, bool early, bool early_x, bool late,
                                cudaStream_t st) {
    (void)bnd;
    const unsigned grid = unit_grid((long long)work_cap * ((max_rank_total + SHR_ROWS - 1) / SHR_ROWS) * nsplit);
    const size_t smem = (size_t)GATHER_STAGES * SHR_STAGE + (size_t)8 * 16 * SHR_PAD * sizeof(float) + (size_t)(rec_cap + 2) * sizeof(int);
    return launch_pdl(plora_shrink_gather_kernel, dim3(grid), dim3(GATHER_THREADS), smem, st, pdl, reinterpret_cast<const bf16*>(x), ldx, K, recs,
                      rec_cap, prefix, S, s_stride_elems, lds, kchunk, nsplit, early ? 1 : 0, early_x ? 1 : 0, pdl && late ? 1 : 0,
                      status PLORA_BOUNDS_ARG(bnd));
}

cudaError_t plora_launch_expand(const float* S, size_t s_stride_elems, int lds, int nsplit, const PloraRec* recs,
                                int rec_cap, const int* prefix, void* y, int ldy, int f32_out, int parts, int max_rows, int work_cap,
                                int most, const PloraBounds& bnd, int* status, bool pdl, bool early, cudaStream_t st) {
    (void)bnd;
    const int max_rank = lds / PLORA_MAX_PARTS;
    const int s_pad = ((max_rank + 31) & ~31) * 2 + 16;  // an odd number of 16-byte pieces between the rows of a plane
    const unsigned grid = unit_grid(1 + (long long)work_cap * parts * max_rows * expand_cost(max_rank, PLORA_WORK_TOKENS) / 2048);
    const size_t smem = (size_t)EXP_STAGES * EXP_PIECE + (size_t)3 * 16 * s_pad + (size_t)8 * EXP_AHEAD * EXP_Y_BYTES + (size_t)(rec_cap + 2) * sizeof(int);
    auto* fn = max_rank > 128 ? (f32_out ? plora_expand_gather_kernel<true, true> : plora_expand_gather_kernel<false, true>)
                              : (f32_out ? plora_expand_gather_kernel<true, false> : plora_expand_gather_kernel<false, false>);
    return launch_pdl(fn, dim3(grid), dim3(GATHER_THREADS), smem, st,
                      pdl, S, s_stride_elems, lds, nsplit, recs, rec_cap, prefix, y, ldy, s_pad, most, early ? 1 : 0, status PLORA_BOUNDS_ARG(bnd));
}
