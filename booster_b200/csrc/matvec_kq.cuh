// matvec_kq.cuh — one token's product with K-quant matrices (Q4_K / Q5_K / Q6_K x Q8_K), fused like k_matvec: [RMSNorm] + activation quantization, exact W.x, the
// layer's epilogue. BIT-EXACT with the reference's CPU arithmetic (ggml_vec_dot_q{4,5,6}_K_q8_K, cpp/ggml/src/ggml-quants.c:6914-6977, 7487-7560, 8145-8220).
//
// A thread owns lanes w and w + 4 (bytes 4w..4w+3 and 16 + 4w.. of every 32-weight group) of R rows and walks their super-blocks in order: its chains never leave its
// registers, a row's are in four neighbouring threads, and nothing is exchanged before the row is finished, then by shuffles. A warp is 8 R rows, its weight words are 128
// consecutive bytes of the tile; 32 rows are a team of 4 / R warps with a ring and a copying warp of its own.
// Scales go in pairs: two four-byte sums fit 16 bits each (<= 4 * 32 * 127), one dp2a multiplies both by their scales.
// What bounds it: with several units of 32 rows per SM the issue slots (gate|up of an 8B model, 66 MB: 67 % of them busy, DRAM at 46 %, alone and cold under ncu), with one unit
// the team's four warps, one per scheduler: 300 clocks a super-block of which 105 issue. Copies are 9 KB where two super-blocks make a stage: a bulk copy costs 210 to 230
// clocks of the copy engine however small it is, 4.6 KB ones end at 20 bytes a clock and SM.
// Measured (B200, an 8B model's 8 layers at 2000; launches of one kind back to back, k_matvec, a thread = a row, K split over warps that exchange the integers, and this one): qkv
// 8.5 and 7.3 us, wo 5.2 and 5.5, gate|up 15.8 and 14.9 (4.4 TB/s), down 15.2 and 13.3, head 20.9 and 20.0; the token 509 and 467. Models of width 512 to 8192: tokens 0.77 to
// 0.95 of the time; alone two rows per thread are behind k_matvec at k of 3072 and more (gate|up up to 9 %) and a Q6_K head of 4096 rows at k = 5120 and 6144 (3 to 8 %).
// One lane per thread (eight warps a unit): 507 us a token against 485 when it was tried. Four teams taking a unit's super-blocks in turn and four warps for the
// chains: 521. The next super-block's words read ahead into registers: 510.
#pragma once
#include "matvec_q80.cuh"

namespace b200 {

static constexpr int KV_WARPS = 16, KV_MAX_STAGES = 16;         // consuming warps; stages of a team's ring
__host__ __device__ constexpr int kv_teams(int R) { return KV_WARPS * R / 4; }
__host__ __device__ constexpr int kv_threads(int R) { return (KV_WARPS + kv_teams(R)) * 32; }   // and one copying warp per team
// the quantized vector: words [block][lane m (8)][group of 32 (8)] | with Q6_K: int -32 * (sum of the word's four quants), same order | per block the sums of its
// groups of 32 as four pairs of int16 | f32 d
__host__ __device__ __forceinline__ int kv_act_bytes(int k, bool q6) { return ((q6 ? 2 * k : k) + k / 256 * 20 + 127) / 128 * 128; }

struct KvAct { uint32_t * q; int * as; uint32_t * bp; float * dx; };

// U blocks of 256 consecutive values (8 per lane) go through the steps of quantize_row_q8_K_ref (cpp/ggml/src/ggml-quants.c:3593-3630) together: q8k_blocks_warp has
// the arithmetic. Block u is b + u * KV_WARPS; those from n256 on do not exist.
template <int U>
__device__ __forceinline__ void kv_quantize(const float (&v)[U][8], int lane, int b, int n256, bool q6, const KvAct & A) {
    unsigned top[U], first[U];
    float mval[U], iscale[U], d[U];
    int at[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        float amax = 0.f;
        mval[u] = 0.f; at[u] = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (fabsf(v[u][i]) > amax) { amax = fabsf(v[u][i]); mval[u] = v[u][i]; at[u] = lane * 8 + i; }
        top[u] = __float_as_uint(amax);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const unsigned all = __reduce_max_sync(0xffffffffu, top[u]);
        first[u] = __reduce_min_sync(0xffffffffu, top[u] == all ? (unsigned) at[u] : 0xffffffffu);
        top[u] = all;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        mval[u] = __shfl_sync(0xffffffffu, mval[u], (int) (first[u] >> 3));
        iscale[u] = top[u] != 0u ? __fdiv_rn(-127.f, mval[u]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; u++) d[u] = top[u] != 0u ? __fdiv_rn(1.f, iscale[u]) : 0.f;
#pragma unroll
    for (int u = 0; u < U; u++) {
        uint32_t w[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; i++) w[i >> 2] |= ((uint32_t) (min(127, __float2int_rn(__fmul_rn(iscale[u], v[u][i]))) & 0xff)) << (8 * (i & 3));
        const int s0 = __dp4a((int) w[0], 0x01010101, 0), s1 = __dp4a((int) w[1], 0x01010101, 0);
        int sum = s0 + s1;
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);             // of the group lane / 4
        const int odd = __shfl_down_sync(0xffffffffu, sum, 4);
        const int bb = b + u * KV_WARPS, o = bb * 64 + (lane & 3) * 16 + (lane >> 2);
        if (bb < n256) {
            A.q[o] = w[0]; A.q[o + 8] = w[1];
            if (q6) { A.as[o] = -32 * s0; A.as[o + 8] = -32 * s1; }
            if ((lane & 7) == 0) A.bp[bb * 4 + (lane >> 3)] = ((uint32_t) sum & 0xffffu) | (uint32_t) odd << 16;
            if (lane == 0) A.dx[bb] = d[u];
        }
    }
}

// two sums of four products as the halves of a dp2a operand
__device__ __forceinline__ int kv_pair(int even, int odd) { return (int) __byte_perm((unsigned) even, (unsigned) odd, 0x5410u); }
// word s (0..7) of a lane's eight
__device__ __forceinline__ int kv_word(const int4 (&a)[2], int s) { return word_of(a[s >> 2], s & 3); }

// what a super-block brings to a thread's chains: exact integers as floats and their multipliers
struct KvSums { float s[2], d, p, dmin; };
// a thread's share of one row's super-block. W[h]: its words of lane w + 4h in the order of the arithmetic; H: their high bits
struct KvTile { uint32_t W[2][4], H[2][2]; uint4 sd; float d; };
template <int TYPE>
__device__ __forceinline__ void kv_tile(const uint8_t * t, int w, int row, KvTile & k) {       // t: tile + row * 16
    const uint8_t * wp = t + w * 4;
    k.sd = lds_u4(t + 4096);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        // Q6_K: half n, group g of 32 weights (dequantize_row_q6_K, cpp/ggml/src/ggml-quants.c:2970-3000): ql chunk 4n + 2(g & 1) + h; qh chunk 2n + h
#pragma unroll
        for (int j = 0; j < 4; j++) k.W[h][j] = lds_u32(wp + (2 * j + h) * 512);
        if (TYPE == T_Q5_K) k.H[h][0] = lds_u32(wp + 4608 + h * 512);
        if (TYPE == T_Q6_K) { k.H[h][0] = lds_u32(wp + 4608 + h * 512); k.H[h][1] = lds_u32(wp + 4608 + (2 + h) * 512); }
    }
    if (TYPE == T_Q6_K) k.d = __half2float(*reinterpret_cast<const __half *>(t + 6656 - row * 14));
}
// q[h] / as[h]: the block's words of lane w + 4h; bp: its groups' sums (Q4_K: pair w in .x)
template <int TYPE>
__device__ __forceinline__ void kv_block(const KvTile & k, int w, const int4 (&q)[2][2], const int4 (&as)[2][2], const int4 & bp, float yd, KvSums & o) {
    if (TYPE == T_Q6_K) {
        // group g: nibble g >> 1 of its ql word, bits 2g of its qh word, scale 8n + 2g + h
        o.d = __fmul_rn(yd, k.d);
        o.p = o.dmin = 0.f;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int s = 0;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const int sc = (int) __byte_perm(n ? k.sd.z : k.sd.x, n ? k.sd.w : k.sd.y, h ? 0x7531u : 0x6420u);       // of groups 0..3
                const uint32_t l0 = k.W[h][2 * n], l1 = k.W[h][2 * n + 1], H = k.H[h][n];
                const int p0 = dp4a_us((l0 & 0x0f0f0f0fu) | ((H << 4) & 0x30303030u), q[h][n].x, as[h][n].x);
                const int p1 = dp4a_us((l1 & 0x0f0f0f0fu) | ((H << 2) & 0x30303030u), q[h][n].y, as[h][n].y);
                const int p2 = dp4a_us(((l0 >> 4) & 0x0f0f0f0fu) | (H & 0x30303030u), q[h][n].z, as[h][n].z);
                const int p3 = dp4a_us(((l1 >> 4) & 0x0f0f0f0fu) | ((H >> 2) & 0x30303030u), q[h][n].w, as[h][n].w);
                s = __dp2a_hi(kv_pair(p2, p3), sc, __dp2a_lo(kv_pair(p0, p1), sc, s));
            }
            o.s[h] = (float) s;
        }
    } else {
        const uint4 sd = k.sd;
        // the 8 scale bytes and 8 min bytes: get_scale_min_k4 packing (cpp/ggml/src/ggml-quants.c:1891-1898)
        const uint32_t sc_a = sd.x & 0x3f3f3f3fu, sc_b = (sd.z & 0x0f0f0f0fu) | ((sd.x >> 2) & 0x30303030u);
        const uint32_t m_a = sd.y & 0x3f3f3f3fu, m_b = ((sd.z >> 4) & 0x0f0f0f0fu) | ((sd.y >> 2) & 0x30303030u);
        const __half2 dm = *reinterpret_cast<const __half2 *>(&sd.w);
        o.d = __fmul_rn(yd, __low2float(dm));
        o.dmin = __fmul_rn(-yd, __high2float(dm));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t H = TYPE == T_Q5_K ? k.H[h][0] : 0u;
            int s = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t W = k.W[h][j];
                uint32_t lo = W & 0x0f0f0f0fu, hi = (W >> 4) & 0x0f0f0f0fu;
                if (TYPE == T_Q5_K) {                           // qh bits 2j, 2j + 1: +16 on the low and the high nibble's weight
                    lo |= (j < 2 ? H << (4 - 2 * j) : H >> (2 * j - 4)) & 0x10101010u;
                    hi |= (j < 2 ? H << (3 - 2 * j) : H >> (2 * j - 3)) & 0x10101010u;
                }
                const int p = kv_pair(__dp4a((int) lo, kv_word(q[h], 2 * j), 0), __dp4a((int) hi, kv_word(q[h], 2 * j + 1), 0)), sc = (int) (j < 2 ? sc_a : sc_b);
                s = (j & 1) ? __dp2a_hi(p, sc, s) : __dp2a_lo(p, sc, s);
            }
            o.s[h] = (float) s;
        }
        if (TYPE == T_Q4_K)                                     // lane w of the reference's _mm_madd_epi16(mins, q8s): mins 2w, 2w + 1
            o.p = (float) __dp2a_lo(bp.x, (int) (((w & 2) ? m_b : m_a) >> (16 * (w & 1))), 0);
        else                                                    // summs: the same in a row's four threads
            o.p = (float) __dp2a_hi(bp.w, (int) m_b, __dp2a_lo(bp.z, (int) m_b, __dp2a_hi(bp.y, (int) m_a, __dp2a_lo(bp.x, (int) m_a, 0))));
    }
}
// block b's words of lanes w and w + 4, and its groups' sums
template <int TYPE>
__device__ __forceinline__ void kv_words(const KvAct & A, int b, int w, int4 (&q)[2][2], int4 (&as)[2][2], int4 & bs) {
    bs = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            q[h][i] = *reinterpret_cast<const int4 *>(A.q + b * 64 + w * 8 + h * 32 + i * 4);
            if (TYPE == T_Q6_K) as[h][i] = *reinterpret_cast<const int4 *>(A.as + b * 64 + w * 8 + h * 32 + i * 4);
        }
    }
    if (TYPE == T_Q4_K) bs.x = (int) A.bp[b * 4 + w];
    if (TYPE == T_Q5_K) bs = *reinterpret_cast<const int4 *>(A.bp + b * 4);
}
template <int TYPE>
__device__ __forceinline__ void kv_chain(const KvSums & o, float (&acc)[2], float & accm) {
    acc[0] = __fmaf_rn(o.d, o.s[0], acc[0]);
    acc[1] = __fmaf_rn(o.d, o.s[1], acc[1]);
    if (TYPE == T_Q4_K) accm = __fmaf_rn(o.dmin, o.p, accm);
    if (TYPE == T_Q5_K) accm = __fadd_rn(accm, __fmul_rn(o.dmin, o.p));      // an add of a product, not an fma (ggml-quants.c:7516)
}
// the row's tail over its four threads: finish_row's sums, whose operands may change places. Lanes l and l + 8, ... get row l % 8 of the warp's eight
template <int TYPE>
__device__ __forceinline__ float kv_finish(const float (&acc)[2], float accm, int lane) {
    float v = __fadd_rn(acc[1], acc[0]);
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
    if (TYPE == T_Q4_K) {
        float m = __fadd_rn(accm, __shfl_xor_sync(0xffffffffu, accm, 2));
        m = __fadd_rn(m, __shfl_xor_sync(0xffffffffu, m, 1));
        v = __fadd_rn(v, m);
    }
    if (TYPE == T_Q5_K) v = __fadd_rn(v, accm);
    return __shfl_sync(0xffffffffu, v, (lane & 7) * 4);
}
__device__ __forceinline__ bool kv_has_q6(const MatvecArgs & a) {
    return a.seg[0].type == T_Q6_K || (a.n_seg > 1 && a.seg[1].type == T_Q6_K) || (a.n_seg > 2 && a.seg[2].type == T_Q6_K);
}
__device__ __forceinline__ KvAct kv_act(uint8_t * smem, int k, bool q6) {
    KvAct A;
    A.q = reinterpret_cast<uint32_t *>(smem);
    A.as = reinterpret_cast<int *>(smem + k);
    A.bp = reinterpret_cast<uint32_t *>(smem + (q6 ? 2 * k : k));
    A.dx = reinterpret_cast<float *>(A.bp + k / 256 * 4);
    return A;
}
// what a row's epilogue needs beside its value
__device__ __forceinline__ void kv_epilogue_inputs(const MatvecArgs & a, int row, int pos, float & pre0, float & pre1) {
    pre0 = pre1 = 0.f;
    if (a.epi == EPI_RESID) pre0 = a.resid[row];
    if (a.epi == EPI_QKV && row < a.n_q + a.n_k) {
        const float2 cs = a.rope[(size_t) pos * (a.head_dim / 2) + (((row & ~1) & (a.head_dim - 1)) >> 1)];
        pre0 = cs.x; pre1 = cs.y;
    }
}

// The vector, by the block's first KV_WARPS warps: norm weights are constants and requested ahead of the wait; U blocks of 256 per warp and pass, their loads together.
template <int U, bool TR>
__device__ __forceinline__ void kv_prologue(const MatvecArgs & a, int warp, int lane, int n256, bool q6, const KvAct & A, double * red) {
    const bool norm = a.norm_w != nullptr;
    float ww[U][8] = {};
    if (norm) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (warp + u * KV_WARPS < n256) ldg8(a.norm_w + (warp + u * KV_WARPS) * 256 + lane * 8, ww[u]);
    }
    trace_mark<TR>(a.trace, 1);
    pdl_wait();
    trace_mark<TR>(a.trace, 2);
#pragma unroll 1
    for (int b0 = warp; b0 < n256 || b0 == warp; b0 += U * KV_WARPS) {           // (with a norm one pass holds the vector: the host checks)
        float v[U][8];
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (b0 + u * KV_WARPS < n256) load8(a.x + (b0 + u * KV_WARPS) * 256 + lane * 8, v[u]);
            else {
#pragma unroll
                for (int i = 0; i < 8; i++) v[u][i] = 0.f;
            }
        }
        if (norm) {
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                double p = 0.0;
#pragma unroll
                for (int i = 0; i < 8; i++) p += (double) __fmul_rn(v[u][i], v[u][i]);
                s += p;
            }
            s = warp_sum_d(s);
            if (lane == 0) red[warp] = s;
            asm volatile("bar.sync 1, %0;" :: "n"(KV_WARPS * 32) : "memory");
            double tot = red[lane & (KV_WARPS - 1)];
#pragma unroll
            for (int o = 1; o < KV_WARPS; o <<= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
            const float scale = rms_scale(tot, a.k, a.inv_k, a.eps);
#pragma unroll
            for (int u = 0; u < U; u++) {
#pragma unroll
                for (int i = 0; i < 8; i++) v[u][i] = __fmul_rn(__fmul_rn(v[u][i], scale), ww[u][i]);
            }
        }
        if (b0 < n256) kv_quantize<U>(v, lane, b0, n256, q6, A);
    }
}

// U: blocks of the vector per warp and pass of the prologue; R: rows per thread; NB: super-blocks per stage of the ring
template <int U, int R, int NB, bool TR>
__global__ void __launch_bounds__(kv_threads(R), 1) k_matvec_kq(const __grid_constant__ MatvecArgs a) {
    constexpr int TW = 4 / R;                                   // warps of a team
    extern __shared__ __align__(128) uint8_t kv_smem[];
    __shared__ __align__(8) uint64_t bars[kv_teams(R) * 2 * KV_MAX_STAGES];
    __shared__ double red[KV_WARPS];
    __shared__ int failed_s;
    volatile int * failed = &failed_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool q6 = kv_has_q6(a);
    const int n256 = a.k / 256, S = a.stages, slot = a.stage_bytes, n_steps = a.tiles_unit / NB, n_teams = a.groups_per_cta;
    const KvAct A = kv_act(kv_smem, a.k, q6);
    const int team = warp >= KV_WARPS ? warp - KV_WARPS : warp / TW;
    const uint32_t b_full = smem_u32(bars) + (uint32_t) team * (2 * KV_MAX_STAGES * 8), b_empty = b_full + KV_MAX_STAGES * 8;
    uint8_t * slots = kv_smem + kv_act_bytes(a.k, q6) + (size_t) team * S * slot;
    const int first = team * gridDim.x + blockIdx.x, stride = n_teams * gridDim.x;        // unit u: block u % grid, team (u / grid) % teams
    if (tid == 0) failed_s = 0;                                 // (first read behind the block's barrier)
    trace_mark<TR>(a.trace, 0);
    pdl_launch_dependents();
    if (warp >= KV_WARPS)
        return qv_copy<NB, TW>(a, lane, team < n_teams, first, stride, S, (uint32_t) slot, smem_u32(slots), b_full, b_empty, failed);
    kv_prologue<U, TR>(a, warp, lane, n256, q6, A, red);
    int pos = 0, cell = 0;
    if (a.epi == EPI_QKV) {
        const int4 s0 = *reinterpret_cast<const int4 *>(a.st), s1 = *(reinterpret_cast<const int4 *>(a.st) + 1);
        pos = s0.y; cell = s1.x;
    }
    __syncthreads();
    trace_mark<TR>(a.trace, 3);
    if (team >= n_teams) return;

    // ---- the rows
    const int w = lane & 3, row = (warp % TW) * (8 * R) + (lane >> 2), erow = (warp % TW) * (8 * R) + (lane & (8 * R - 1));      // erow: this lane's row of the epilogue
    int s = 0;
    uint32_t par = 0;
    for (int u = first; u < a.n_units; u += stride) {
        const UnitDesc ud = describe_unit(a, u);
        const int prow = ud.row0 + erow;
        float pre0, pre1;                                       // in flight meanwhile
        kv_epilogue_inputs(a, prow, pos, pre0, pre1);
        float val = 0.f;
        auto walk = [&](auto tag) {
            constexpr int TYPE = decltype(tag)::value;
            float acc[R][2] = {}, accm[R] = {};
#pragma unroll 1
            for (int st = 0; st < n_steps; st++) {
                um_wait(b_full + 8 * s, par, failed, a.err);
                const uint8_t * t = slots + s * slot + row * 16;
#pragma unroll
                for (int b = 0; b < NB; b++) {
                    int4 q[2][2], as[2][2], bs;
                    kv_words<TYPE>(A, st * NB + b, w, q, as, bs);
                    const float yd = A.dx[st * NB + b];
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        KvTile k;
                        KvSums o;
                        kv_tile<TYPE>(t + b * tile_bytes_of(TYPE) + r * 128, w, row + 8 * r, k);
                        kv_block<TYPE>(k, w, q, as, bs, yd, o);
                        kv_chain<TYPE>(o, acc[r], accm[r]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(b_empty + 8 * s);
                if (++s == S) { s = 0; par ^= 1u; }
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float v = kv_finish<TYPE>(acc[r], accm[r], lane);
                if (r == 0 || (lane & 8)) val = v;
            }
        };
        if (ud.type == T_Q4_K) walk(TypeTag<T_Q4_K>{});
        else if (ud.type == T_Q5_K) walk(TypeTag<T_Q5_K>{});
        else walk(TypeTag<T_Q6_K>{});
        matvec_epilogue(a, val, prow, lane, pre0, pre1, cell, lane < 8 * R && !*failed);
    }
    trace_mark<TR>(a.trace, 10);
    if (TR) { if (a.trace != nullptr) trace_mark<TR>(a.trace, 4); }
}

}  // namespace b200
