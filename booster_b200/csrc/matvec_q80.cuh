// matvec_q80.cuh — one token's product with a Q8_0 matrix (Q8_0 x Q8_0), fused like k_matvec: [RMSNorm] + activation quantization, exact W.x, the layer's
// epilogue. BIT-EXACT with the reference's CPU arithmetic (tinyBLAS_Q0_AVX, cpp/ggml/src/llamafile/sgemm.cpp): lane m of a row sums the four products of bytes
// 4m..4m+3 of a 32-weight block and runs acc[m] = fma(d_w d_x, (float) isum[m], acc[m]) block after block.
//
// A thread owns ONE lane of ONE row and walks its blocks in order: the chain never leaves its register, and nothing is exchanged before the row is finished. (k_matvec
// gives a thread all eight lanes of a row and splits K over warps, which hand the chains over after every 32 weights: a bulk copy, a wait and a hand-over per 1088 bytes.)
// 32 rows are 256 threads, a team: warp = eight rows x four lanes, so that a warp's weights are 128 consecutive bytes of the tile.
// What bounds it: HBM where there are several units of 32 rows per SM, else the instructions of the eight warps that a unit has, 9 per weight word.
// Measured (B200, 8 layers of an 8B model, token at 333): 968 us with k_matvec, 515 here; launches of one kind back to back gate|up (125 MB) 37.6 and 22.4 us, down (62 MB)
// 36.1 and 13.1, wo 12.2 and 5.8. Alone and cold under ncu gate|up has DRAM at 57 % and 47 % of the issue slots busy.
// Reading a stage's words ahead of adding the one before: 630 against 607 with stages of eight blocks.
#pragma once
#include "kernels.cuh"

namespace b200 {

static constexpr int QV_WARPS = 16, QV_TEAMS = 2, QV_THREADS = (QV_WARPS + QV_TEAMS) * 32;    // consuming warps, then one copying warp per team
static constexpr int QV_MAX_STAGES = 24;
static constexpr int QV_FIN = 8 * 32;                           // floats: finished chains of one unit
// the quantized vector: words [block / 4][lane m (8)][block % 4] | f32 d[k / 32]
__host__ __device__ __forceinline__ int qv_act_bytes(int k) { return k + k / 32 * 4; }
__host__ __device__ __forceinline__ int qv_fixed_bytes(int k) { return (qv_act_bytes(k) + 127) / 128 * 128 + QV_TEAMS * 2 * QV_FIN * 4; }

// 256 consecutive values (8 per lane) -> eight Q8_0 blocks, AVX path of quantize_row_q8_0 (cpp/ggml/src/ggml-quants.c:936-1000)
__device__ __forceinline__ void qv_quantize(const float (&v)[8], int lane, int b256, uint32_t * q, float * dx) {
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d  = __fdiv_rn(amax, 127.f);
    const float id = amax != 0.f ? __fdiv_rn(127.f, amax) : 0.f;
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; i++) w[i >> 2] |= ((uint32_t) (__float2int_rn(__fmul_rn(v[i], id)) & 0xff)) << (8 * (i & 3));
    const int b = b256 * 8 + (lane >> 2), m = 2 * (lane & 3);
    uint32_t * o = q + (b >> 2) * 32 + m * 4 + (b & 3);
    o[0] = w[0]; o[4] = w[1];
    if ((lane & 3) == 0) dx[b] = __half2float(__float2half_rn(d));
}

// um_wait for a warp that has time: between two looks it sleeps, and leaves its scheduler's issue slots to the warps that add
__device__ __forceinline__ void um_wait_asleep(uint32_t bar, uint32_t parity, volatile int * failed, int * err) {
#pragma unroll 1
    for (uint32_t looks = 0; looks < (1u << 22); looks++) {
        if (um_try(bar, parity) || *failed) return;
        __nanosleep(150);
    }
    *failed = 1;
    atomicExch_system(err, 1);
}
// The copying warp of a team: its units' blocks, NB to a stage, into the team's ring from before the dependency wait on; weights wait for nobody. Passes the block's
// barrier when the ring is full or nothing is left to copy: the consumers may start. full: one arrival and the stage's bytes; empty: one arrival per consuming warp.
template <int NB, int TW>       // TW: consuming warps
__device__ __forceinline__ void qv_copy(const MatvecArgs & a, int lane, bool has_team, int first, int stride, int S, uint32_t slot_bytes, uint32_t dst,
                                        uint32_t b_full, uint32_t b_empty, volatile int * failed) {
    if (lane == 0 && has_team) {
        for (int s = 0; s < S; s++) { mbar_init(b_full + 8 * s, 1); mbar_init(b_empty + 8 * s, TW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    const int n_steps = a.tiles_unit / NB;
    int s = 0, n = 0;
    uint32_t par = 1;
    const uint64_t pol = l2_policy_evict_first();
    bool synced = false;
    if (has_team) {
        for (int u = first; u < a.n_units; u += stride) {
            const UnitDesc ud = describe_unit(a, u);
            const uint32_t bytes = NB * ud.bytes;
            const uint8_t * src = ud.tiles;
#pragma unroll 1
            for (int st = 0; st < n_steps; st++) {
                if (n >= S) {
                    if (!synced) { __syncthreads(); synced = true; }
                    um_wait_asleep(b_empty + 8 * s, par, failed, a.err);
                }
                if (lane == 0 && !(n >= S && *failed)) {
                    mbar_expect_tx(b_full + 8 * s, bytes);
                    bulk_g2s_hint(dst + (uint32_t) s * slot_bytes, src, bytes, b_full + 8 * s, pol);
                }
                __syncwarp();
                src += bytes;
                n++;
                if (++s == S) { s = 0; par ^= 1u; }
            }
        }
    }
    if (!synced) __syncthreads();
    pdl_wait();
    if (*failed) { for (int i = 0; i < 1000; i++) __nanosleep(1000); }      // copies nobody waited for end before the block does
}

// NB: blocks per stage of the ring
template <int NB, bool TR>
__global__ void __launch_bounds__(QV_THREADS, 1) k_matvec_q80(const __grid_constant__ MatvecArgs a) {
    constexpr int STAGE = NB * 1088;
    extern __shared__ __align__(128) uint8_t qv_smem[];
    __shared__ __align__(8) uint64_t bars[QV_TEAMS * 2 * QV_MAX_STAGES];
    __shared__ double red[QV_WARPS];
    __shared__ int failed_s;
    volatile int * failed = &failed_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t * act = reinterpret_cast<uint32_t *>(qv_smem);
    float * dxs = reinterpret_cast<float *>(qv_smem + a.k);
    float * fins = reinterpret_cast<float *>(qv_smem + (qv_act_bytes(a.k) + 127) / 128 * 128);
    uint8_t * ring = qv_smem + qv_fixed_bytes(a.k);
    const int S = a.stages, n_steps = a.tiles_unit / NB, n_teams = a.groups_per_cta;
    const int team = warp >= QV_WARPS ? warp - QV_WARPS : warp >> 3;
    const uint32_t b_full = smem_u32(bars) + (uint32_t) team * (2 * QV_MAX_STAGES * 8), b_empty = b_full + QV_MAX_STAGES * 8;
    uint8_t * slots = ring + (size_t) team * S * STAGE;
    const int first = team * gridDim.x + blockIdx.x, stride = n_teams * gridDim.x;        // unit u: block u % grid, team (u / grid) % teams
    if (tid == 0) failed_s = 0;                                 // (first read behind the block's barrier)
    trace_mark<TR>(a.trace, 0);
    pdl_launch_dependents();
    if (warp >= QV_WARPS)
        return qv_copy<NB, 8>(a, lane, team < n_teams, first, stride, S, STAGE, smem_u32(slots), b_full, b_empty, failed);
    // ---- the vector: norm weights are constants and requested ahead of the wait; four blocks of 256 per warp and pass, their loads together
    const bool norm = a.norm_w != nullptr;
    const int n256 = a.k / 256;
    float ww[PRO_U][8] = {};
    if (norm) {
#pragma unroll
        for (int u = 0; u < PRO_U; u++)
            if (warp + u * QV_WARPS < n256) ldg8(a.norm_w + (warp + u * QV_WARPS) * 256 + lane * 8, ww[u]);
    }
    trace_mark<TR>(a.trace, 1);
    pdl_wait();
    trace_mark<TR>(a.trace, 2);
    int pos = 0, cell = 0;
    if (a.epi == EPI_QKV) {
        const int4 s0 = *reinterpret_cast<const int4 *>(a.st), s1 = *(reinterpret_cast<const int4 *>(a.st) + 1);
        pos = s0.y; cell = s1.x;
    }
#pragma unroll 1
    for (int b0 = warp; b0 < n256 || b0 == warp; b0 += PRO_U * QV_WARPS) {       // (with a norm one pass holds the vector: the host checks)
        float v[PRO_U][8];
#pragma unroll
        for (int u = 0; u < PRO_U; u++) {
            if (b0 + u * QV_WARPS < n256) load8(a.x + (b0 + u * QV_WARPS) * 256 + lane * 8, v[u]);
            else {
#pragma unroll
                for (int i = 0; i < 8; i++) v[u][i] = 0.f;
            }
        }
        if (norm) {
            double s[PRO_U];
#pragma unroll
            for (int u = 0; u < PRO_U; u++) {
                s[u] = 0.0;
#pragma unroll
                for (int i = 0; i < 8; i++) s[u] += (double) __fmul_rn(v[u][i], v[u][i]);
            }
            const double w = warp_sum_d((s[0] + s[1]) + (s[2] + s[3]));
            if (lane == 0) red[warp] = w;
            asm volatile("bar.sync 1, %0;" :: "n"(QV_WARPS * 32) : "memory");
            double tot = red[lane & (QV_WARPS - 1)];
#pragma unroll
            for (int o = 1; o < QV_WARPS; o <<= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
            const float scale = rms_scale(tot, a.k, a.inv_k, a.eps);
#pragma unroll
            for (int u = 0; u < PRO_U; u++) {
#pragma unroll
                for (int i = 0; i < 8; i++) v[u][i] = __fmul_rn(__fmul_rn(v[u][i], scale), ww[u][i]);
            }
        }
#pragma unroll
        for (int u = 0; u < PRO_U; u++)
            if (b0 + u * QV_WARPS < n256) qv_quantize(v[u], lane, b0 + u * QV_WARPS, act, dxs);
    }
    __syncthreads();
    trace_mark<TR>(a.trace, 3);
    if (team >= n_teams) return;

    // ---- the rows
    const int tw = warp & 7, h = tw & 1, row = (tw >> 1) * 8 + (lane >> 2), m = 4 * h + (lane & 3);
    const uint8_t * wp = slots + h * 512 + row * 16 + (lane & 3) * 4, * dp = slots + 1024 + row * 2;
    int s = 0, j = 0;
    uint32_t par = 0;
    for (int u = first; u < a.n_units; u += stride, j++) {
        const UnitDesc ud = describe_unit(a, u);
        const uint32_t * qp = act + m * 4;
        const float * xp = dxs;
        float acc = 0.f;
        float pre0 = 0.f, pre1 = 0.f;
        const bool finisher = tw == (j & 7);                    // the warp that finishes this unit's rows; what it needs comes in meanwhile
        if (finisher) {
            const int prow = ud.row0 + lane;
            if (a.epi == EPI_RESID) pre0 = a.resid[prow];
            if (a.epi == EPI_QKV && prow < a.n_q + a.n_k) {
                const float2 cs2 = a.rope[(size_t) pos * (a.head_dim / 2) + (((prow & ~1) & (a.head_dim - 1)) >> 1)];
                pre0 = cs2.x; pre1 = cs2.y;
            }
        }
#pragma unroll 1
        for (int st = 0; st < n_steps; st++) {
            um_wait(b_full + 8 * s, par, failed, a.err);
            const uint8_t * w = wp + s * STAGE, * dw = dp + s * STAGE;
#pragma unroll
            for (int b4 = 0; b4 < NB / 4; b4++) {
                const int4 q = *reinterpret_cast<const int4 *>(qp + b4 * 32);
                const float4 x = *reinterpret_cast<const float4 *>(xp + b4 * 4);
                float f[4], d[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    // (float) isum, exactly: |isum| <= 4 * 128 * 127 < 2^22 on top of 1.5 * 2^23
                    f[i] = __fadd_rn(__int_as_float(__dp4a((int) lds_u32(w + (4 * b4 + i) * 1088), word_of(q, i), 0x4b400000)), -12582912.f);
                    d[i] = __fmul_rn(__half2float(*reinterpret_cast<const __half *>(dw + (4 * b4 + i) * 1088)), i == 0 ? x.x : i == 1 ? x.y : i == 2 ? x.z : x.w);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) acc = __fmaf_rn(d[i], f[i], acc);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(b_empty + 8 * s);
            qp += NB * 8; xp += NB;
            if (++s == S) { s = 0; par ^= 1u; }
        }
        float * fin = fins + (team * 2 + (j & 1)) * QV_FIN;
        fin[m * 32 + row] = acc;
        asm volatile("bar.sync %0, 256;" :: "r"(2 + team) : "memory");
        if (finisher && !*failed) {
            float c[8];
#pragma unroll
            for (int i = 0; i < 8; i++) c[i] = fin[i * 32 + lane];
            matvec_epilogue(a, finish_row<T_Q8_0>(c), ud.row0 + lane, lane, pre0, pre1, cell);
        }
    }
    trace_mark<TR>(a.trace, 10);
    if (TR) { if (a.trace != nullptr) trace_mark<TR>(a.trace, 4); }
}

}  // namespace b200
