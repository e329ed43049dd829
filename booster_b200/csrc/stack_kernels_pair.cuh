// stack_kernels_pair.cuh — bfloat16 products of prompt portions on pairs of SMs (sm_100a, tcgen05 cta_group::2): Y = X W^T (+ bias), gated units in the epilogue, rows sorted by
// expert (LinArgs::seg), K in parts.
//
// D is formed transposed: a pair's accumulator has 256 rows of W (128 in each block's tensor memory) by up to 256 tokens, two of them side by side where a portion is longer. A row of
// W is then read once for 512 tokens, and a portion of few tokens costs few columns (32 at least) instead of a 128-row tile.
//   warps 0, 1 copy, per slice of 64 k: its block's 128 rows of W, its half of the tokens' rows. The first block's `full` barrier counts both blocks' bytes. The first slices of W are
//              asked for ahead of pdl_wait(): weights depend on no kernel
//   warp 2     of the first block issues 256 x N x 16 MMAs; tcgen05.commit hands the slice's room (`empty`) and the accumulators (`acc_full`) back to both blocks
//   warps 3-10 drain: lane = row of W, so that a token's 32 outputs of a warp are 128 consecutive bytes; two columns at a time make gated units (gate and up are neighbouring lanes:
//              one shuffle gives each lane one unit). They join K parts, segments and the tile after (a second set of accumulators where both fit 512 columns) to one loop
// What bounds it: a pair's slice is 16 KB of W and 16 KB of X per block for 256 x 256 (1024 clocks of MMAs for 512 tokens: 47 bytes a clock and SM out of L2), and W itself from HBM.
// Its predecessor for these shapes, one block per 128 tokens x 256 rows, read 94 bytes a clock and stored a token per lane, 4 bytes of each sector at a time for gated units.
// Measured in a pass (B200, with and without the rounding of X that is now the norm's or the unit's): 512 x 16384 x 2048 gated 81 + 2.7 us then, 42 now (7 of them the units' exponentials and quotients, the same as every other product's); 512 x 2048 x 8192 18 + 4.5 + 3.7
// (parts) and 17 + 3.1; 512 x 2048 x 2048 18 + 2.7 + 3.7 and 10 + 3.4; 2048 rows of 16 experts of 4096 x 2048 106 and 64 (268 MB of weights), 16 tokens x 2048 x 8192 by mma.sync 245, now
// 23 by itself. The MMA loop is at the tensor cores' rate for 512 tokens (1020 clocks a slice); for 64 tokens a slice takes 400 clocks, half of them waits and votes between instructions.
// Every wait on an mbarrier is bounded: on a timeout the block raises *err, skips what is left, and still meets its partner and frees its tensor memory.
#pragma once

namespace b200 {
namespace stk {

constexpr int PG_BK = 64, PG_ROWS = 256, PG_THREADS = 352, PG_DRAIN = 8;                    // rows of W per pair; draining warps
constexpr int PG_W_BYTES = 128 * PG_BK * 2, PG_SMEM = 200 * 1024, PG_MAX_STAGES = 8, PG_SEG_MAX = 512;
struct PairPlan {
    int acc, n;             // accumulators side by side (1 or 2) and columns of each (a multiple of 32, up to 256): acc x n tokens a tile
    int parts;              // K parts (1: whole)
    int stages, sets;       // ring; sets of accumulators (2: a tile is drained while the next one is formed)
    int n_seg;              // segments (0: none)
};
__host__ __device__ inline int pg_stage_bytes(int acc, int n) { return PG_W_BYTES + acc * (n / 2) * PG_BK * 2; }

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t at_rank(uint32_t addr, uint32_t rank) { uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r; }
__device__ __forceinline__ void pair_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// bytes are counted by a barrier that may be the partner's
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap * map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
                 :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_commit(uint32_t bar) {       // to the barrier at this address in both blocks, when the MMAs so far are done
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" :: "r"(bar), "h"((uint16_t) 3) : "memory");
}

__device__ __forceinline__ void pair_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
}
// a piece of work of a pair: rows of W from n0, tokens from t0 of those r0 .. r0 + T - 1, slices kb .. kb + nk - 1
struct PairTile { int n0, t0, r0, T, z, part, kb, nk; };

// SEG: rows sorted by expert (one accumulator a tile). GLU: GLU_*; ROUND: its units go to Yb. map_x: X as bf16 [1][rows][K], box 64 x n / 2 (SEG: 64 x 32); map_w: W [batch][N][K], box 64 x 128
template <bool SEG, int ACC, int GLU, bool ROUND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PG_THREADS, 1) k_gemm_bf16_pair(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                                           const LinArgs a, const PairPlan p, int * err, float * part) {
    extern __shared__ uint8_t pg_raw[];
    __shared__ __align__(8) uint64_t full[PG_MAX_STAGES], empty[PG_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int seg_s[SEG ? PG_SEG_MAX + 1 : 1], before_s[SEG ? PG_SEG_MAX + 1 : 1];      // segments: first rows, tiles in front of each
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t smem0 = (smem_addr(pg_raw) + 1023u) & ~1023u, rank = cluster_rank();
    if (tid == 0) {
        for (int s = 0; s < p.stages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&empty[s])) : "memory");
        }
        for (int s = 0; s < 2; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&acc_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(&acc_empty[s])), "r"(2 * PG_DRAIN) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (SEG) {                                                 // where the segments lie: an earlier kernel's work
        pdl_wait();
        for (int i = tid; i <= p.n_seg; i += PG_THREADS) seg_s[i] = a.seg[i];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_meet();                                               // both blocks' barriers are there before the first copy counts on one
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    const int per = ACC * p.n, nk_all = (a.K + PG_BK - 1) / PG_BK, row_tiles = (a.N + PG_ROWS - 1) / PG_ROWS, tok_tiles = SEG ? 0 : (a.T + per - 1) / per;
    int total;
    if (SEG) {
        if (tid == 0) {
            int n = 0;
            for (int i = 0; i < p.n_seg; i++) { before_s[i] = n; n += (seg_s[i + 1] - seg_s[i] + per - 1) / per * row_tiles; }
            before_s[p.n_seg] = n;
        }
        __syncthreads();
        total = before_s[p.n_seg];
    } else total = row_tiles * tok_tiles * p.parts;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
    // tile v: neighbouring pairs have the same rows of W for other tokens, then other parts of K, then the next rows
    int seg_at = 0;
    const auto tile = [&](int v) {
        PairTile t;
        if (SEG) {
            while (v >= before_s[seg_at + 1]) seg_at++;        // (v only grows; segments without rows have no tiles)
            t.r0 = seg_s[seg_at]; t.T = seg_s[seg_at + 1] - t.r0; t.z = seg_at; t.part = 0; t.kb = 0; t.nk = nk_all;
            const int tt = (t.T + per - 1) / per, i = v - before_s[seg_at];
            t.n0 = i / tt * PG_ROWS; t.t0 = i % tt * per;
            return t;
        }
        t.r0 = 0; t.T = a.T; t.z = 0;
        t.t0 = v % tok_tiles * per; t.part = v / tok_tiles % p.parts; t.n0 = v / tok_tiles / p.parts * PG_ROWS;
        t.kb = (int) ((long long) nk_all * t.part / p.parts); t.nk = (int) ((long long) nk_all * (t.part + 1) / p.parts) - t.kb;      // at least one: parts <= nk_all
        return t;
    };
    const uint32_t stage_bytes = (uint32_t) pg_stage_bytes(ACC, p.n), acc_bytes = (uint32_t) (p.n / 2) * PG_BK * 2;
    // columns of accumulator c that hold a token of the tile
    const auto columns = [&](const PairTile & t, int c) { return min(p.n, max(0, (t.T - t.t0 - c * p.n + 31) / 32 * 32)); };
    bool dead = false;                                         // a wait of this thread ran out
    if (warp == 0) {
        const uint32_t bars = at_rank(smem_addr(&full[0]), 0);
        const auto load = [&](const PairTile & t, int kt, int slot) {
            if (elect_one() && !dead) {
                const uint32_t rows_x = SEG ? (uint32_t) ((columns(t, 0) / 2 + 31) / 32 * 32) * (PG_BK * 2) : ACC * acc_bytes;
                if (rank == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_addr(&full[slot])), "r"(2 * (PG_W_BYTES + rows_x)) : "memory");
                pair_load_3d(smem0 + (uint32_t) slot * stage_bytes, &map_w, (t.kb + kt) * PG_BK, t.n0 + (int) rank * 128, t.z, bars + 8u * (uint32_t) slot);
            }
            __syncwarp();
        };
        int ahead = 0;
        if (!SEG) {
            if (first < total) { const PairTile t = tile(first); for (; ahead < min(p.stages, t.nk); ahead++) load(t, ahead, ahead); }
            pdl_wait();
        }
        int it = 0, slot = 0, turn = 0;                        // slices so far, the ring's slot and round
        for (int v = first; v < total; v += step) {
            const PairTile t = tile(v);
            for (int kt = 0; kt < t.nk; kt++, it++) {
                if (it >= ahead) {
                    if (turn > 0) tc_wait(smem_addr(&empty[slot]), (uint32_t) ((turn - 1) & 1), dead);
                    load(t, kt, slot);
                }
                if (++slot == p.stages) { slot = 0; turn++; }
            }
        }
    } else if (warp == 1) {
        const uint32_t bars = at_rank(smem_addr(&full[0]), 0);
        if (!SEG) pdl_wait();
        asm volatile("fence.proxy.async;" ::: "memory");      // X was written by ordinary stores
        int slot = 0, turn = 0;
        for (int v = first; v < total; v += step) {
            const PairTile t = tile(v);
            const int half = (SEG ? columns(t, 0) : p.n) / 2, y = t.r0 + t.t0 + (int) rank * half;
            for (int kt = 0; kt < t.nk; kt++) {
                if (turn > 0) tc_wait(smem_addr(&empty[slot]), (uint32_t) ((turn - 1) & 1), dead);
                if (elect_one() && !dead) {
                    const uint32_t dst = smem0 + (uint32_t) slot * stage_bytes + PG_W_BYTES, bar = bars + 8u * (uint32_t) slot;
                    const int k = (t.kb + kt) * PG_BK;
                    if (SEG) { for (int i = 0; i < half; i += 32) pair_load_3d(dst + (uint32_t) (i * PG_BK * 2), &map_x, k, y + i, 0, bar); }
                    else {
#pragma unroll
                        for (int c = 0; c < ACC; c++) pair_load_3d(dst + (uint32_t) c * acc_bytes, &map_x, k, y + c * p.n, 0, bar);
                    }
                }
                __syncwarp();
                if (++slot == p.stages) { slot = 0; turn++; }
            }
        }
    } else if (warp == 2) {
        if (!SEG) pdl_wait();
        if (rank == 0) {
            // both operands K-major, 128-byte swizzle: start >> 4 | 8-row group stride 1024 B >> 4 << 32 | version 1 | layout 2; a K = 16 step is 32 bytes along the row
            constexpr uint64_t DESC = ((uint64_t) 1 << 16) | ((uint64_t) (1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
            // D f32, A and B bf16, both K-major, M = 256
            constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (PG_ROWS >> 4) << 24);
            int i = 0, slot = 0, turn = 0;
            for (int v = first; v < total; v += step, i++) {
                const PairTile t = tile(v);
                const int set = p.sets == 2 ? i & 1 : 0, round = p.sets == 2 ? i >> 1 : i;
                if (round > 0) tc_wait(smem_addr(&acc_empty[set]), (uint32_t) ((round - 1) & 1), dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d0 = tmem + (uint32_t) (set * ACC * p.n), idesc = IDESC | ((uint32_t) ((SEG ? columns(t, 0) : p.n) >> 3) << 17);
                const bool second = ACC > 1 && columns(t, 1) > 0;
                for (int kt = 0; kt < t.nk; kt++) {
                    tc_wait(smem_addr(&full[slot]), (uint32_t) (turn & 1), dead);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one() && !dead) {
                        const uint64_t dw = DESC | (uint64_t) ((smem0 + (uint32_t) slot * stage_bytes) >> 4), dx = dw + (PG_W_BYTES >> 4);
#pragma unroll
                        for (int c = 0; c < ACC; c++) {
                            if (c > 0 && !second) break;
#pragma unroll
                            for (int ks = 0; ks < PG_BK / 16; ks++)
                                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                             :: "r"(d0 + (uint32_t) (c * p.n)), "l"(dw + 2u * ks), "l"(dx + (uint64_t) (c * (acc_bytes >> 4)) + 2u * ks), "r"(idesc), "r"((uint32_t) (kt | ks)) : "memory");
                        }
                        pair_commit(smem_addr(&empty[slot]));
                        if (kt == t.nk - 1) pair_commit(smem_addr(&acc_full[set]));
                    }
                    __syncwarp();
                    if (++slot == p.stages) { slot = 0; turn++; }
                }
            }
        }
    } else {
        if (!SEG) pdl_wait();
        const int wq = warp & 3, half = (warp - 3) >> 2;
        const bool parts = p.parts > 1;
        const int ldy = parts ? a.N : a.ldy;
        int i = 0;
        for (int v = first; v < total; v += step, i++) {
            const PairTile t = tile(v);
            const int set = p.sets == 2 ? i & 1 : 0, round = p.sets == 2 ? i >> 1 : i;
            if (lane == 0) {                                   // one lane looks, now and then
                for (uint32_t spins = 0; !dead; spins++) {
                    uint32_t ok;
                    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_addr(&acc_full[set])), "r"((uint32_t) (round & 1)) : "memory");
                    if (ok) break;
                    if (spins >= (1u << 22)) dead = true;
                    __nanosleep(50);
                }
            }
            dead = __shfl_sync(0xffffffffu, dead ? 1 : 0, 0) != 0;
            if (dead) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int n = t.n0 + (int) rank * 128 + 32 * wq + lane, odd = lane & 1;
            const bool in = n < a.N;
            const float b = in && a.bias && !parts ? a.bias[n] : 0.f;
#pragma unroll
            for (int c = 0; c < ACC; c++) {
                const int cols = columns(t, c), use = SEG ? cols : p.n, lo = half * (use / 2), hi = min(cols, lo + use / 2);
                const uint32_t taddr = tmem + ((uint32_t) (32 * wq) << 16) + (uint32_t) ((set * ACC + c) * p.n);
                uint32_t next[16];
                if (lo < hi) pair_ld16(taddr + (uint32_t) lo, next);
#pragma unroll 1
                for (int j = lo; j < hi; j += 16) {
                    uint32_t r[16];
                    tc_ld_ready(next);
#pragma unroll
                    for (int e = 0; e < 16; e++) r[e] = next[e];
                    if (j + 16 < hi) pair_ld16(taddr + (uint32_t) (j + 16), next);      // on its way while these are stored
                    const int tok = t.t0 + c * p.n + j, left = t.T - tok;      // columns of the sixteen that are tokens
                    if constexpr (GLU != GLU_NONE) {
                        float u[8];                                            // even lanes make column e's unit, odd ones column e + 1's
#pragma unroll
                        for (int e = 0; e < 16; e += 2) u[e / 2] = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[e] : r[e + 1]) + b, 1);
#pragma unroll
                        for (int e = 0; e < 16; e += 2) {                      // (stores stand behind: between the units they would put them in a row)
                            const float mine = __uint_as_float(odd ? r[e + 1] : r[e]) + b, gate = odd ? u[e / 2] : mine, up = odd ? mine : u[e / 2];
                            u[e / 2] = GLU == GLU_GELU ? gelu_tanhf_(gate) * up : clamped_glu(gate, up, a.limit, a.alpha, a.up_shift);
                        }
                        const size_t at = (size_t) (t.r0 + tok + odd) * ldy + (n >> 1);
                        const int most = in ? left - odd : 0;
                        if constexpr (ROUND) {
#pragma unroll
                            for (int e = 0; e < 16; e += 2) if (e < most) a.Yb[at + (size_t) e * ldy] = __float2bfloat16_rn(u[e / 2]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 16; e += 2) if (e < most) a.Y[at + (size_t) e * ldy] = u[e / 2];
                        }
                        __syncwarp();
                    } else {
                        float * y = (parts ? part + (size_t) t.part * t.T * a.N : a.Y) + (size_t) (t.r0 + tok) * ldy + n;
                        if (in) {
                            if (left >= 16) {
#pragma unroll
                                for (int e = 0; e < 16; e++) y[(size_t) e * ldy] = __uint_as_float(r[e]) + b;
                            } else {
#pragma unroll
                                for (int e = 0; e < 16; e++) if (e < left) y[(size_t) e * ldy] = __uint_as_float(r[e]) + b;
                            }
                        }
                        __syncwarp();
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(at_rank(smem_addr(&acc_empty[set]), 0)) : "memory");
        }
    }
    pdl_launch_dependents();
    if (dead) {
        atomicExch(err, 1);
        for (int j = 0; j < 1000; j++) __nanosleep(1000);      // copies and MMAs under way end before shared and tensor memory are given back
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_meet();                                               // neither block leaves while the other may still reach its barriers, operands or tensor memory
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace stk
}  // namespace b200
